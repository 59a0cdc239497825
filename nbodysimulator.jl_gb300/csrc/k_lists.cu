// k_lists.cu - cell lists and Verlet lists under cubic periodic boundaries.
//
// The reference evaluates every ordered pair (O(N^2), basic_potentials.jl:
// 253-267, 288-299); these lists only restrict the candidates. A Verlet list
// holds every j with FP32 r^2 < (cutoff + skin)^2 (inflated), so as long as no
// atom moved more than skin/2 since the build it is a superset of the
// reference's pair set; the force kernels then apply the exact test.
//
// Build, skipped on device unless a rebuild is due (host-forced every
// rebuild_every steps, or an atom moved more than skin/2):
//   k_cell_fill        : atom -> cell by its wrapped position (the image taken
//                        at the build is kept for the packing until the
//                        next), slot by atomicAdd
//   k_cell_sort        : each cell's atoms sorted by index (deterministic
//                        lists), counts moved to cell_n and cleared for the
//                        next build
//   k_list_build_cells : (up to 25 cells per SM) blocks per cell; the stencil
//                        cells' atoms are staged in shared memory in scan
//                        order, and a warp per atom of the cell tests 32 of
//                        them at a time
//   k_list_build_warps : (more cells) one warp per 32 atoms of a cell; the
//                        stencil cells' atoms pass through a per-warp buffer
//                        in scan order and every atom of the cell tests them
//                        with broadcast reads. The
//                        list is column-major (nbr[k*n + i]) for
//                        thread-per-atom force kernels and row-major
//                        (nbr[i*cap + k]) for lanes-per-atom kernels.
#include <algorithm>

#include "nbg_internal.cuh"

struct ListCtl {
    StepRef pos;  // time index of the positions: its parity picks the rebuild_flag word
    int force;    // host-forced rebuild
};

__device__ __forceinline__ int read_parity(const ListCtl& L) { return (int)(step_of(L.pos) & 1); }

// Replica r's list is rebuilt when the host forces it or one of its atoms
// moved more than skin/2 (flags per replica, so one fast atom in a batch
// rebuilds only its own replica).
__device__ __forceinline__ bool need_build(const Dev& d, const ListCtl& L, int rep)
{
    return L.force || d.rebuild_flag[read_parity(L) * d.nrep + rep] != 0;
}

__device__ __forceinline__ int cell_coord(float h, const RepDev& R)
{
    int c = (int)floorf(h * (float)R.cell_inv);
    if (c < 0) c = 0;
    if (c >= R.nc) c = R.nc - 1;
    return c;
}

// At a build the atom's periodic image is taken afresh (the wrap into
// [0, L)), stored in d.img and its split position packed with it; until the
// next build the drift packs with that image, so that a replica's lists and
// positions keep one frame.
__global__ void k_cell_fill(Dev d, ListCtl L, const double* X)
{
    // the other parity's flags start clean for the next drift (nothing of
    // this rebuild reads them)
    const int other = (read_parity(L) ^ 1) * d.nrep;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < d.nrep; r += gridDim.x * blockDim.x)
        d.rebuild_flag[other + r] = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < d.n; i += (int64_t)gridDim.x * blockDim.x) {
        if (!need_build(d, L, d.rep_of[i])) continue;
        const RepDev& R = d.reps[d.rep_of[i]];
        if (d.img && d.bc == NBG_BC_CUBIC) {
            double im[3];
            for (int k = 0; k < 3; ++k) {
                const double p = X[3 * i + k];
                double m = floor(p * R.invL);
                const double w = fma(-R.L, m, p);
                if (w < 0.0) m -= 1.0;
                else if (w >= R.L) m += 1.0;
                im[k] = m;
                d.img[3 * i + k] = m;
            }
            const double p[3] = {X[3 * i], X[3 * i + 1], X[3 * i + 2]};
            float hh[3], ll[3];
            split_position_image(R, p, im, hh, ll);
            d.phi[i] = make_float4(hh[0], hh[1], hh[2], d.phi[i].w);
            d.plo[i] = make_float4(ll[0], ll[1], ll[2], d.plo[i].w);
        }
        float4 h = d.phi[i];
        int cx = cell_coord(h.x, R), cy = cell_coord(h.y, R), cz = cell_coord(h.z, R);
        int cell = R.cell0 + (cx * R.nc + cy) * R.nc + cz;
        int slot = atomicAdd(&d.cell_count[cell], 1);
        if (slot < d.cell_cap) d.cell_atoms[(int64_t)cell * d.cell_cap + slot] = (int)i;
        else status_set(d.status, ST_CELL_OVERFLOW);
    }
}

// One block per cell: rank sort of the (distinct) atom indices.
__global__ void k_cell_sort(Dev d, ListCtl L)
{
    extern __shared__ int sh[];
    for (int cell = blockIdx.x; cell < d.ncell_total; cell += gridDim.x) {
        const int rep = d.cell_rep[cell];
        if (!need_build(d, L, rep)) continue;
        if (threadIdx.x == 0 && cell == d.reps[rep].cell0) atomicAdd(d.build_count, 1ull);  // one per replica
        int cnt = d.cell_count[cell];
        if (cnt > d.cell_cap) cnt = d.cell_cap;
        int* src = d.cell_atoms + (int64_t)cell * d.cell_cap;
        for (int k = threadIdx.x; k < cnt; k += blockDim.x) sh[k] = src[k];
        __syncthreads();
        for (int k = threadIdx.x; k < cnt; k += blockDim.x) {
            int v = sh[k];
            int rank = 0;
            for (int m = 0; m < cnt; ++m) rank += (sh[m] < v);
            src[rank] = v;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            d.cell_n[cell] = cnt;
            d.cell_count[cell] = 0;
        }
        __syncthreads();
    }
}

// Blocks per cell (item (cell, c): the cell's atoms from G c in strides of
// G chunks, so that few, full cells spread over many blocks): the stencil's
// cells (125 or 27, or for a one-cell replica 1) are staged into shared
// memory in scan order (cell q = ((ox+ns) w + oy+ns) w + oz+ns, then slot
// order), and a warp per atom tests 32 candidates at a time and appends the
// accepted ones, in order, through a ballot prefix count. Two tests, both
// only the list's superset test (the force kernels classify every pair
// exactly):
//   hi parts   from two cells per SM on: the split-position hi parts, moved by
//              the periodic shift into the cell's frame, as in
//              k_list_build_warps
//   SPLIT      fewer cells: the full split difference
// The rows are those of k_list_build_warps, and of the per-atom builders that
// SPLIT replaces (a thread or lane group per atom gathering its candidates).
//
// A warp per (cell, 32 atoms) with lanes as atoms leaves the chip idle where
// cells are few: with 17 atoms a cell 15 lanes idle, and the 729 warps of
// 12,288-atom water left three SM sub-partitions in four without one that
// could issue. Full builds, us (this kernel / the one it replaces there):
// water 12,288 atoms 52 / 213, 24,000 177 / 292, 98,304 478 / 579; LJ 5,000
// 19 / 28, 11,000 25 / 62, 30,000 38 / 69, 60,000 67 / 73, 100,000 111 / 101
// (staging a 27-cell stencil for 21 atoms then costs more than the idle
// lanes: the line lies at 25 cells per SM).
#define LC_WARPS 8
#define LC_NB 125
#define LC_BYTES 40960       // staged candidates at a time
#define LC_MAX_PER_SM 25     // cells per SM, at most
#define LC_SPLIT_PER_SM 2    // cells per SM below which the split difference is tested

template <bool ONE, bool WATER>
__device__ __forceinline__ bool lc_test(const float4& c, const float4& hi, int i, int mol0, float rl2, const RepDev& R)
{
    float dx = c.x - hi.x, dy = c.y - hi.y, dz = c.z - hi.z;
    if (ONE) {
        // s = rint(d / L) by the 1.5 * 2^23 trick (|d / L| <= 1)
        const float magic = 12582912.0f;
        dx = __fmaf_rn(-__fsub_rn(__fmaf_rn(dx, R.invLf, magic), magic), R.Lh, dx);
        dy = __fmaf_rn(-__fsub_rn(__fmaf_rn(dy, R.invLf, magic), magic), R.Lh, dy);
        dz = __fmaf_rn(-__fsub_rn(__fmaf_rn(dz, R.invLf, magic), magic), R.Lh, dz);
    }
    const float r2 = dx * dx + dy * dy + dz * dz;
    const int j = __float_as_int(c.w);
    return r2 < rl2 && j != i && (!WATER || (unsigned)(j - mol0) >= 3u);
}

template <bool WATER>
__device__ __forceinline__ bool lc_test_split(const float4& c, const float4& cl, const float4& hi, const float4& lo, int i,
                                              int mol0, float rl2, const PairK& K)
{
    const float3 dr = split_diff(hi, lo, c, cl, true, K);
    const float r2 = dr.x * dr.x + dr.y * dr.y + dr.z * dr.z;
    const int j = __float_as_int(c.w);
    return r2 < rl2 && j != i && (!WATER || (unsigned)(j - mol0) >= 3u);
}

// The rows of atoms c0 .. c0 + G - 1, c0 + stride .. of a cell against the m
// staged candidates.
template <bool SPLIT, bool ONE, bool WATER>
__device__ __forceinline__ void lc_rows(const Dev& d, const RepDev& R, const float4* cand, const float4* cand_lo, int m,
                                        const int* atoms, int c0, int G, int stride, int cnt, bool first, int w, int lane)
{
    const float rl2 = R.rl2;
    const PairK K(R);
    for (int b = c0; b < cnt; b += stride)
        for (int a = b + w; a < min(cnt, b + G); a += LC_WARPS) {
#ifdef NBG_DEBUG
            const int i = dbg_index(atoms[a], d.n, -1, d.status);
            if (i < 0) continue;
#else
            const int i = atoms[a];
#endif
            const float4 hi = d.phi[i];
            float4 lo = hi;
            if (SPLIT) lo = d.plo[i];
            const int mol0 = WATER ? 3 * (i / 3) : -8;  // first atom of i's molecule
            int* const row = d.nbr + (int64_t)i * d.nbr_istride;
            int n = first ? 0 : d.nbr_count[i];  // (a pass continues the row of the one before)
            const unsigned below = (1u << lane) - 1u;
            auto step = [&](int k, bool real) {
                const float4 c = cand[k];
                bool take;
                if (SPLIT) take = lc_test_split<WATER>(c, cand_lo[k], hi, lo, i, mol0, rl2, K) && real;
                else take = lc_test<ONE, WATER>(c, hi, i, mol0, rl2, R) && real;
                const unsigned bal = __ballot_sync(0xffffffffu, take);
                const int pos = n + __popc(bal & below);
                if (take && pos < d.nbr_cap) row[(int64_t)pos * d.nbr_kstride] = __float_as_int(c.w);
                n += __popc(bal);
            };
            int k0 = 0;
#pragma unroll 4
            for (; k0 + 32 <= m; k0 += 32) step(k0 + lane, true);
            if (k0 < m) step(k0 + lane < m ? k0 + lane : 0, k0 + lane < m);
            if (lane == 0) d.nbr_count[i] = n;
        }
}

template <bool SPLIT>
__global__ void __launch_bounds__(LC_WARPS * 32) k_list_build_cells(Dev d, ListCtl L, const double* X, int G, int chunks)
{
    constexpr int CAP = LC_BYTES / (SPLIT ? 32 : 16);  // candidates staged at a time
    __shared__ int nb_code[LC_NB];  // stencil cell | (shift + 1) per axis in bits 24-29
    __shared__ int nb_off[LC_NB + 1];
    __shared__ float4 cand[LC_BYTES / 16];
    float4* const cand_lo = cand + (SPLIT ? CAP : 0);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool water = d.kind == NBG_SYSTEM_WATER;
    const int64_t items = (int64_t)d.ncell_total * chunks;
    if (d.nrep == 1 && !need_build(d, L, 0)) return;
    for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
        const int cell = (int)(it / chunks), c0 = (int)(it % chunks) * G;
        const int rep = d.cell_rep[cell];
        if (!need_build(d, L, rep)) continue;
        const int cnt = min(d.cell_n[cell], d.cell_cap);
        if (c0 >= cnt) continue;
        const RepDev& R = d.reps[rep];
        const int nc = R.nc;
        const bool one = R.ns == 0;  // one cell holds the replica: minimum image per pair
        const int sw = 2 * R.ns + 1;  // stencil width (1, 3 or 5)
        const int nnb = sw * sw * sw;
        const int* atoms = d.cell_atoms + (int64_t)cell * d.cell_cap;
        __syncthreads();  // the previous item's tables are consumed
        if (threadIdx.x < nnb) {
            const int lc = cell - R.cell0, q = threadIdx.x;
            const int cx = lc / (nc * nc), cy = (lc / nc) % nc, cz = lc % nc;
            int nx = cx + q / (sw * sw) - R.ns, ny = cy + (q / sw) % sw - R.ns, nz = cz + q % sw - R.ns;
            int sx = 1, sy = 1, sz = 1;
            if (nx < 0) { nx += nc; sx = 0; }
            if (nx >= nc) { nx -= nc; sx = 2; }
            if (ny < 0) { ny += nc; sy = 0; }
            if (ny >= nc) { ny -= nc; sy = 2; }
            if (nz < 0) { nz += nc; sz = 0; }
            if (nz >= nc) { nz -= nc; sz = 2; }
            const int cq = R.cell0 + (nx * nc + ny) * nc + nz;
            nb_code[q] = cq | (sx << 24) | (sy << 26) | (sz << 28);
            nb_off[q + 1] = min(d.cell_n[cq], d.cell_cap);
        }
        __syncthreads();
        if (w == 0) {  // inclusive sums of the counts, four per lane
            int v[4], t = 0;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                t += 4 * lane + e < nnb ? nb_off[4 * lane + e + 1] : 0;
                v[e] = t;
            }
            int x = t;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (4 * lane + e < nnb) nb_off[4 * lane + e + 1] = x - t + v[e];
            if (lane == 0) nb_off[0] = 0;
        }
        __syncthreads();
        const int total = nb_off[nnb];
        const float Lh = R.Lh;
        for (int p0 = 0; p0 < total; p0 += CAP) {
            if (p0 > 0) __syncthreads();  // the previous pass's candidates are tested
            // a warp per stencil cell, four cells' loads in flight
            for (int q0 = w; q0 < nnb; q0 += 4 * LC_WARPS) {
                int m[4], off[4], code[4], most = 0;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int q = q0 + e * LC_WARPS;
                    off[e] = q < nnb ? nb_off[q] - p0 : 0;
                    m[e] = q < nnb ? nb_off[q + 1] - p0 - off[e] : 0;
                    code[e] = q < nnb ? nb_code[q] : 0;
                    if (off[e] >= CAP || off[e] + m[e] <= 0) m[e] = 0;
                    most = max(most, m[e]);
                }
                for (int k0 = 0; k0 < most; k0 += 32) {
                    int j[4];
                    float4 h[4], l[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int k = k0 + lane, s = off[e] + k;
                        j[e] = -1;
                        if (k < m[e] && s >= 0 && s < CAP)
                            j[e] = dbg_index(d.cell_atoms[(int64_t)(code[e] & 0xffffff) * d.cell_cap + k], d.n, 0, d.status);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (j[e] >= 0) {
                            h[e] = d.phi[j[e]];
                            if (SPLIT) l[e] = d.plo[j[e]];
                        }
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if (j[e] < 0) continue;
                        const int s = off[e] + k0 + lane;
                        if (SPLIT) {
                            cand[s] = make_float4(h[e].x, h[e].y, h[e].z, __int_as_float(j[e]));
                            cand_lo[s] = l[e];
                        } else {
                            const float sx = (float)(((code[e] >> 24) & 3) - 1) * Lh;
                            const float sy = (float)(((code[e] >> 26) & 3) - 1) * Lh;
                            const float sz = (float)(((code[e] >> 28) & 3) - 1) * Lh;
                            cand[s] = make_float4(h[e].x + sx, h[e].y + sy, h[e].z + sz, __int_as_float(j[e]));
                        }
                    }
                }
            }
            __syncthreads();
            const int m = min(CAP, total - p0), stride = G * chunks;
            const bool first = p0 == 0;
            if (one && !SPLIT) {
                if (water) lc_rows<SPLIT, true, true>(d, R, cand, cand_lo, m, atoms, c0, G, stride, cnt, first, w, lane);
                else lc_rows<SPLIT, true, false>(d, R, cand, cand_lo, m, atoms, c0, G, stride, cnt, first, w, lane);
            } else {
                if (water) lc_rows<SPLIT, false, true>(d, R, cand, cand_lo, m, atoms, c0, G, stride, cnt, first, w, lane);
                else lc_rows<SPLIT, false, false>(d, R, cand, cand_lo, m, atoms, c0, G, stride, cnt, first, w, lane);
            }
        }
        __syncthreads();  // the rows' counts
        for (int b = c0; b < cnt; b += G * chunks)
            if (threadIdx.x < G && b + threadIdx.x < cnt) {
                const int i = dbg_index(atoms[b + threadIdx.x], d.n, 0, d.status);
                if (d.nbr_count[i] > d.nbr_cap) {
                    status_set(d.status, ST_NBR_OVERFLOW);
                    d.nbr_count[i] = d.nbr_cap;
                }
                d.xref[3 * i] = X[3 * i];
                d.xref[3 * i + 1] = X[3 * i + 1];
                d.xref[3 * i + 2] = X[3 * i + 2];
            }
    }
}

// Warp per (cell, chunk of 32 of its atoms): lane l holds atom l of the
// chunk. The stencil's cells (125 or 27, or for a one-cell replica 1)
// pass their atoms through a per-warp buffer of 32 candidates (split-position
// hi parts moved by the periodic shift into the cell's frame, index in w) read
// back by broadcast; the next chunk's index and position gathers are issued
// before the current chunk's tests. The test r^2 < rl2 on the hi parts is the
// list's superset test (the force kernels classify every pair exactly). The
// candidates come in the stencil order of the per-atom builders (cell q =
// ((ox+ns) w + oy+ns) w + oz+ns, then slot order), so the lists are the same.
#define LW_WARPS 4
#define LW_NB 125

template <bool ONE, bool WATER>
__device__ __forceinline__ int lw_test(const float4* cand, int bn, const float4& hi, int i, int mol0, float rl2,
                                       const RepDev& R, int* row, int64_t kstride, int cap, int lcnt)
{
#pragma unroll 4
    for (int k = 0; k < bn; ++k) {
        const float4 c = cand[k];
        float dx = c.x - hi.x, dy = c.y - hi.y, dz = c.z - hi.z;
        if (ONE) {
            // s = rint(d / L) by the 1.5 * 2^23 trick (|d / L| <= 1)
            const float magic = 12582912.0f;
            dx = __fmaf_rn(-__fsub_rn(__fmaf_rn(dx, R.invLf, magic), magic), R.Lh, dx);
            dy = __fmaf_rn(-__fsub_rn(__fmaf_rn(dy, R.invLf, magic), magic), R.Lh, dy);
            dz = __fmaf_rn(-__fsub_rn(__fmaf_rn(dz, R.invLf, magic), magic), R.Lh, dz);
        }
        const float r2 = dx * dx + dy * dy + dz * dz;
        const int j = __float_as_int(c.w);
        if (r2 < rl2 && j != i && (!WATER || (unsigned)(j - mol0) >= 3u)) {
            if (lcnt < cap) row[(int64_t)lcnt * kstride] = j;
            ++lcnt;
        }
    }
    return lcnt;
}

__global__ void __launch_bounds__(LW_WARPS * 32) k_list_build_warps(Dev d, ListCtl L, const double* X, int chunks)
{
    __shared__ int nb_code[LW_WARPS][LW_NB];  // stencil cell | (shift + 1) per axis in bits 24-29
    __shared__ int nb_cnt[LW_WARPS][LW_NB];
    __shared__ float4 cand[LW_WARPS][32];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool water = d.kind == NBG_SYSTEM_WATER;
    // work item: (cell, c), c < chunks; it takes the cell's atoms from 32 c
    // in strides of 32 chunks, so that cells holding many atoms spread over
    // several warps
    const int64_t items = (int64_t)d.ncell_total * chunks;
    for (int64_t it = blockIdx.x * (int64_t)LW_WARPS + wid; it < items; it += (int64_t)gridDim.x * LW_WARPS) {
        const int cell = (int)(it / chunks);
        const int c0 = (int)(it % chunks) * 32;
        const int rep = d.cell_rep[cell];
        if (!need_build(d, L, rep)) continue;
        const int cnt = min(d.cell_n[cell], d.cell_cap);
        if (c0 >= cnt) continue;
        const RepDev& R = d.reps[rep];
        const int nc = R.nc;
        const int lc = cell - R.cell0;
        const int cx = lc / (nc * nc), cy = (lc / nc) % nc, cz = lc % nc;
        const bool one = R.ns == 0;  // one cell holds the replica: minimum image per pair
        const int w = 2 * R.ns + 1;  // stencil width (1, 3 or 5)
        const int nnb = w * w * w;
        __syncwarp();  // the previous cell's tables are consumed
        for (int q = lane; q < nnb; q += 32) {
            const int ox = q / (w * w) - R.ns, oy = (q / w) % w - R.ns, oz = q % w - R.ns;
            int nx = cx + ox, ny = cy + oy, nz = cz + oz;
            int sx = 1, sy = 1, sz = 1;
            if (nx < 0) { nx += nc; sx = 0; }
            if (nx >= nc) { nx -= nc; sx = 2; }
            if (ny < 0) { ny += nc; sy = 0; }
            if (ny >= nc) { ny -= nc; sy = 2; }
            if (nz < 0) { nz += nc; sz = 0; }
            if (nz >= nc) { nz -= nc; sz = 2; }
            const int cq = R.cell0 + (nx * nc + ny) * nc + nz;
            nb_code[wid][q] = cq | (sx << 24) | (sy << 26) | (sz << 28);
            nb_cnt[wid][q] = min(d.cell_n[cq], d.cell_cap);
        }
        __syncwarp();
        const float Lh = R.Lh, rl2 = R.rl2;
        const int* atoms = d.cell_atoms + (int64_t)cell * d.cell_cap;
        for (int a0 = c0; a0 < cnt; a0 += 32 * chunks) {
            const int a = a0 + lane;
#ifdef NBG_DEBUG
            const int i_read = a < cnt ? atoms[a] : -1;
            const bool active = a < cnt && dbg_index(i_read, d.n, -1, d.status) >= 0;
            const int i = active ? i_read : -1;
#else
            const bool active = a < cnt;
            const int i = active ? atoms[a] : -1;
#endif
            const float4 hi = active ? d.phi[i] : make_float4(0.f, 0.f, 0.f, 0.f);
            const int mol0 = water && active ? 3 * (i / 3) : -8;  // first atom of i's molecule
            int* row = d.nbr + (int64_t)(active ? i : 0) * d.nbr_istride;
            int lcnt = 0;
            // chunk (q, b0): atoms b0 .. b0 + 31 of stencil cell q
            int q = 0;
            while (q < nnb && nb_cnt[wid][q] == 0) ++q;
            int b0 = 0;
            int jn = -1;
            float4 hn = make_float4(0.f, 0.f, 0.f, 0.f);
            if (q < nnb) {
                const int cq = nb_code[wid][q] & 0xffffff;
                if (lane < nb_cnt[wid][q]) {
                    jn = dbg_index(d.cell_atoms[(int64_t)cq * d.cell_cap + lane], d.n, 0, d.status);
                    hn = d.phi[jn];
                }
            }
            while (q < nnb) {
                const int code = nb_code[wid][q];
                const int cn = nb_cnt[wid][q];
                const int bn = min(32, cn - b0);
                const int j = jn;
                const float4 hj = hn;
                // the next chunk's gathers go out before this chunk's tests
                int q2 = q, b2 = b0 + 32;
                if (b2 >= cn) {
                    b2 = 0;
                    ++q2;
                    while (q2 < nnb && nb_cnt[wid][q2] == 0) ++q2;
                }
                if (q2 < nnb) {
                    const int cq2 = nb_code[wid][q2] & 0xffffff;
                    jn = -1;
                    if (b2 + lane < nb_cnt[wid][q2]) {
                        jn = dbg_index(d.cell_atoms[(int64_t)cq2 * d.cell_cap + b2 + lane], d.n, 0, d.status);
                        hn = d.phi[jn];
                    }
                }
                const float sx = (float)(((code >> 24) & 3) - 1) * Lh;
                const float sy = (float)(((code >> 26) & 3) - 1) * Lh;
                const float sz = (float)(((code >> 28) & 3) - 1) * Lh;
                if (lane < bn) cand[wid][lane] = make_float4(hj.x + sx, hj.y + sy, hj.z + sz, __int_as_float(j));
                __syncwarp();
                if (active) {
                    if (one)
                        lcnt = water ? lw_test<true, true>(cand[wid], bn, hi, i, mol0, rl2, R, row, d.nbr_kstride, d.nbr_cap, lcnt)
                                     : lw_test<true, false>(cand[wid], bn, hi, i, mol0, rl2, R, row, d.nbr_kstride, d.nbr_cap, lcnt);
                    else
                        lcnt = water ? lw_test<false, true>(cand[wid], bn, hi, i, mol0, rl2, R, row, d.nbr_kstride, d.nbr_cap, lcnt)
                                     : lw_test<false, false>(cand[wid], bn, hi, i, mol0, rl2, R, row, d.nbr_kstride, d.nbr_cap, lcnt);
                }
                __syncwarp();
                q = q2;
                b0 = b2;
            }
            if (active) {
                if (lcnt > d.nbr_cap) {
                    status_set(d.status, ST_NBR_OVERFLOW);
                    lcnt = d.nbr_cap;
                }
                d.nbr_count[i] = lcnt;
                d.xref[3 * i] = X[3 * i];
                d.xref[3 * i + 1] = X[3 * i + 1];
                d.xref[3 * i + 2] = X[3 * i + 2];
            }
        }
    }
}

#ifdef NBG_DEBUG
// Debug builds only: entry 0 of atom 0's Verlet-list row (nbr[0] in both
// layouts) becomes n + k, an index past every per-atom buffer, so that the
// tests see the list readers' index checks report it (NBG_ERR_INDEX).
__global__ void k_plant_index(Dev d, int k)
{
    if (threadIdx.x == 0 && blockIdx.x == 0 && d.nbr_count[0] > 0) d.nbr[0] = (int)(d.n + k);
}

int launch_plant_index(nbg_ctx* c, int k)
{
    k_plant_index<<<1, 32, 0, c->stream>>>(c->d, k);
    NBG_LAUNCH_CHECK(c, "k_plant_index");
    return NBG_OK;
}
#endif

int launch_list_build(nbg_ctx* c, const StateView& s, bool force, StepRef pos)
{
    NBG_RANGE("launch_list_build");
    c->accel_lists_valid = false;  // the lists follow other positions now
    c->ens_lists_valid = false;
    ListCtl L{pos, force ? 1 : 0};
    // The kernels run at every step of a captured graph and skip the atoms
    // and cells of replicas without a due rebuild. The fill and the sort
    // loop over their items on a few waves of blocks, so that a step with no
    // rebuild (or, in a batch, few) does not schedule a block per cell; the
    // list build keeps a warp per item, whose work is too uneven for a
    // fixed share per warp.
    const int64_t wave = (int64_t)c->sms * 8;
    k_cell_fill<<<(unsigned)std::min<int64_t>(grid_for(c->n, 256), wave), 256, 0, c->stream>>>(c->d, L, s.x);
    NBG_LAUNCH_CHECK(c, "k_cell_fill");
    const int64_t cells = c->d.ncell_total;
    k_cell_sort<<<(unsigned)std::min<int64_t>(cells, 4 * wave), 128, sizeof(int) * c->d.cell_cap, c->stream>>>(c->d, L);
    NBG_LAUNCH_CHECK(c, "k_cell_sort");
    const double occ = (double)c->n / std::max<int64_t>(cells, 1);
    if (cells <= LC_MAX_PER_SM * (int64_t)c->sms) {
        // 32 atoms an item (4 a warp), down to 8 while the items leave an SM
        // under 4 blocks
        int G = 32;
        while (G > LC_WARPS && cells * (int64_t)std::ceil(occ / G) < 4 * (int64_t)c->sms) G /= 2;
        const int chunks = std::max(1, (int)std::ceil(occ / G));
        const int64_t blocks = std::min<int64_t>(cells * chunks, 6 * (int64_t)c->sms);  // (cheap when idle)
        if (cells < LC_SPLIT_PER_SM * (int64_t)c->sms)
            k_list_build_cells<true><<<(unsigned)blocks, LC_WARPS * 32, 0, c->stream>>>(c->d, L, s.x, G, chunks);
        else
            k_list_build_cells<false><<<(unsigned)blocks, LC_WARPS * 32, 0, c->stream>>>(c->d, L, s.x, G, chunks);
    } else {
        // warps per cell from the mean occupancy (with margin); fuller cells loop
        const int chunks = std::max(1, std::min((c->d.cell_cap + 31) / 32, (int)std::ceil(1.5 * occ / 32.0)));
        const int64_t items = cells * chunks;
        const int64_t blocks = std::min<int64_t>((items + LW_WARPS - 1) / LW_WARPS, 1 << 20);
        k_list_build_warps<<<(unsigned)blocks, LW_WARPS * 32, 0, c->stream>>>(c->d, L, s.x, chunks);
    }
    NBG_LAUNCH_CHECK(c, "k_list_build");
    return NBG_OK;
}
