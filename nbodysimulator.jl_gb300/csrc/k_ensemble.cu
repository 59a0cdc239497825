// k_ensemble.cu - replica ensembles as one persistent launch per chunk of
// steps: a CTA per replica, the replica's whole step loop inside it.
//
// The replicas of a batch never interact, so no step needs a grid-wide
// barrier: CTA b runs replica order[b] (largest first, so that the big
// replicas start early and the small ones fill the gaps) for all the steps of
// the launch, synchronising only its own threads. Per step:
//   - integration of its atoms (BAOAB for the Langevin thermostat, velocity
//     Verlet without thermostat; the FP64 arithmetic of k_baoab_drift /
//     k_drift_pack) and their fixed-point box coordinates into shared memory
//     (the whole replica: 16 bytes per atom), with the displacement check
//     against the positions of the last list build (fixed point, no FP64);
//   - when a rebuild is due (an atom moved more than skin/2, or
//     rebuild_every steps passed): a counting sort of the atoms into cells in
//     shared memory, each cell's atoms in index order, then every atom's
//     Verlet-list row from the stencil cells (FP32 superset test on the
//     fixed-point differences), written to the list buffer as 16-bit indices;
//   - the pair forces of each atom from its list row, gathering neighbours
//     from shared memory (fx_pair2: the fixed-point kernels' classification
//     and arithmetic, so the pair set is the reference's), joined over the
//     atom's lanes, and the velocity update by a lane per component.
// The Philox noise is keyed (seed, atom, step) as in the step-graph kernels;
// the lists and each replica's steps since its build carry over to the next
// launch unless another path moved the state.
#include <algorithm>
#include <vector>

#include "fx_pair.cuh"

#define ENS_MAX_ATOMS 9216  // largest replica the loop takes (shared memory)
#define ENS_MAX_CELLS 4096
#define ENS_RANK 3          // atoms per lane of the cell sort (cells of up to 96 atoms)

struct EnsArgs {
    const int* order;
    int* since;     // per replica: steps since its build (-1: build first)
    uint4* pref;    // per atom: fixed-point position at its replica's build
    int reuse;      // the lists and counts are this loop's from the previous launch
    int mode;       // cell width: 0 rl / 3^3 stencil, 1 rl/2 / 5^3
    double dt;
    int nsteps;
    int rebuild_every;
    int64_t step0;
    int save;
    int baoab;
};

__device__ __forceinline__ int ens_cell(const uint4& q, int nc)
{
    const int cx = (int)__umulhi(q.x, (unsigned)nc), cy = (int)__umulhi(q.y, (unsigned)nc),
              cz = (int)__umulhi(q.z, (unsigned)nc);
    return (cx * nc + cy) * nc + cz;
}

// Exclusive prefix sum of cnt[0..m) into out[0..m] (out[m] = total), by the
// whole block: a contiguous chunk per thread, then the chunk totals.
template <int THREADS>
__device__ void ens_scan(const int* cnt, int* out, int m, int* warp_tot)
{
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int per = (m + THREADS - 1) / THREADS;
    const int b0 = min(tid * per, m), b1 = min(b0 + per, m);
    int sum = 0;
    for (int k = b0; k < b1; ++k) sum += cnt[k];
    int x = sum;  // inclusive scan in the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    if (w == 0) {
        int t = lane < THREADS / 32 ? warp_tot[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < THREADS / 32) warp_tot[lane] = t;  // inclusive totals of the warps
    }
    __syncthreads();
    int run = x - sum + (w > 0 ? warp_tot[w - 1] : 0);  // exclusive prefix of this thread's chunk
    for (int k = b0; k < b1; ++k) {
        out[k] = run;
        run += cnt[k];
    }
    if (tid == THREADS - 1) out[m] = run;
    __syncthreads();
}

// Distance along one axis, at least, from a candidate to any of the warp's
// atoms, whose offsets from the reference position lie in [lo, hi]; the
// candidate's offset as the wrapped difference, and its other image.
__device__ __forceinline__ float ens_gap(unsigned off, float lo, float hi)
{
    const float o = (float)(int)off;
    const float here = fmaxf(lo - o, o - hi);
    const float there = o < 0.f ? o + 4294967296.f - hi : lo - (o - 4294967296.f);
    return fmaxf(0.f, fminf(here, there));
}

// Where entry k of a row lies (16-bit units): block of 8 LPA entries, then
// lane k % LPA, then its 8 entries in order.
template <int LPA>
__device__ __forceinline__ int ens_slot(int k)
{
    return (k & ~(8 * LPA - 1)) + (k % LPA) * 8 + (k % (8 * LPA)) / LPA;
}

template <int LPA, int POT, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) k_ensemble(Dev d, StateView s, EnsArgs A)
{
    constexpr int G = THREADS / LPA;  // lane groups (atoms in flight)
    const int r = A.order[blockIdx.x];
    const RepDev& R = d.reps[r];
    const int n = (int)R.n;
    const int64_t a0 = R.atom0;
    const int nc = R.ens_nc[A.mode], ns = R.ens_ns[A.mode];
    const int ncell = nc * nc * nc;
    extern __shared__ uint4 ens_sm[];
    uint4* pos = ens_sm;                                   // [n] fixed-point x, y, z and the charge bits
    int* cstart = reinterpret_cast<int*>(pos + n);         // [ncell + 1]
    int* ccur = cstart + (ncell + 1);                      // [ncell]
    uint16_t* sorted = reinterpret_cast<uint16_t*>(ccur + ncell);  // [n] atoms in cell order
    uint16_t* cnts = sorted + n;                           // [n] list counts
    __shared__ int warp_tot[THREADS / 32];
    __shared__ int next_item;  // the list build's next cell
    __shared__ uint4 cand[THREADS / 32][32];  // its candidates, per warp
    const int tid = threadIdx.x, lane = tid % LPA, g = tid / LPA;
    const double dt = A.dt, hdt = 0.5 * dt, dtsq = dt * dt;
    const double c1 = R.bc1;
    const int cap = d.nbr_cap;

    // the frame sink (trajectory saving), read at a save point
    const int64_t sk_every = A.save ? d.sink->every : 0;
    const int64_t sk_t0 = A.save ? d.sink->t0 : 0;
    // list rows of this loop: replica-local 16-bit indices in the list
    // buffer's memory, 2 cap per atom (nothing else reads them: every other
    // path builds its own lists first). Entry k of a row lies where lane
    // k % LPA finds its 8 entries of a block of 8 LPA in one 16-byte load,
    // four packed steps of the force loop (ens_slot). (Row capacities are
    // whole 16-byte units and hold whole blocks: list_rows.h.)
    uint16_t* const rows = reinterpret_cast<uint16_t*>(d.nbr);
    for (int i = tid; i < n; i += THREADS) {
        pos[i].w = d.pfx[a0 + i].w;
        cnts[i] = A.reuse ? (uint16_t)min(d.nbr_count[a0 + i], cap) : (uint16_t)0;
    }
    int since = A.reuse ? A.since[r] : -1;

    bool range_err = false;
    for (int st = 0; st < A.nsteps; ++st) {
        const int64_t step = A.step0 + st;
        // integration to the step's positions, their fixed-point form, and
        // the displacement since the last build
        bool moved = false;
        for (int i = tid; i < n; i += THREADS) {
            const int64_t gi = a0 + i;
            double* x = s.x + 3 * gi;
            double* v = s.v + 3 * gi;
            const double* ao = s.a_old + 3 * gi;
            if (A.baoab) {
                const double sd = __dmul_rn(R.bsd, d.rsqrt_mass[gi]);
                float z[3];
                philox_normals3<float>(R.seed, (uint64_t)i, (uint64_t)step, z);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const double vh = fma(hdt, ao[k], v[k]);
                    const double xh = fma(hdt, vh, x[k]);
                    const double vo = fma(c1, vh, sd * widen(z[k]));
                    x[k] = fma(hdt, vo, xh);
                    v[k] = vo;
                }
            } else {
#pragma unroll
                for (int k = 0; k < 3; ++k) x[k] = drift1(x[k], v[k], ao[k], dt, dtsq);
            }
            uint4 q = pos[i];
            q.x = fx_coord(x[0], R.fx_scale);
            q.y = fx_coord(x[1], R.fx_scale);
            q.z = fx_coord(x[2], R.fx_scale);
            pos[i] = q;
            if (since >= 0) {
                const uint4 p0 = A.pref[gi];
                float ddx, ddy, ddz;
                const float m2 = fx_r2(q, p0, ddx, ddy, ddz);
                moved |= !(m2 <= R.fx_disp2);
            }
        }
        const bool build = __syncthreads_or(moved ? 1 : 0) || since < 0 ||
                           (A.rebuild_every > 0 && since + 1 >= A.rebuild_every);
        if (build) {
            if (tid == 0) atomicAdd(d.build_count, 1ull);  // the replica's builds, as the graph path counts them
            // counting sort of the atoms into cells, each cell in index order
            for (int c = tid; c < ncell; c += THREADS) ccur[c] = 0;
            __syncthreads();
            for (int i = tid; i < n; i += THREADS) atomicAdd(&ccur[ns > 0 ? ens_cell(pos[i], nc) : 0], 1);
            __syncthreads();
            ens_scan<THREADS>(ccur, cstart, ncell, warp_tot);
            for (int c = tid; c < ncell; c += THREADS) ccur[c] = cstart[c];
            __syncthreads();
            for (int i = tid; i < n; i += THREADS) {
                const int slot = atomicAdd(&ccur[ns > 0 ? ens_cell(pos[i], nc) : 0], 1);
                sorted[slot] = i;
            }
            __syncthreads();
            // each cell's atoms into index order: a warp per cell, every
            // lane counts the smaller indices of its (up to ENS_RANK) atoms
            // and then places them. (A thread per cell by insertion took the
            // whole block's time in a one-cell replica, ~n^2 / 4 dependent
            // shared-memory moves, and kept 1 lane in 32 busy elsewhere.) In
            // a one-cell replica the order is the identity.
            if (ns == 0) {
                for (int i = tid; i < n; i += THREADS) sorted[i] = i;
            } else {
                const int wl = tid & 31;
                for (int c = tid >> 5; c < ncell; c += THREADS / 32) {
                    const int b0 = cstart[c], m = cstart[c + 1] - b0;
                    if (m <= 32 * ENS_RANK) {
                        int v[ENS_RANK], rank[ENS_RANK];
#pragma unroll
                        for (int e = 0; e < ENS_RANK; ++e) {
                            v[e] = wl + 32 * e < m ? sorted[b0 + wl + 32 * e] : 0x7fffffff;
                            rank[e] = 0;
                        }
                        for (int k = 0; k < m; ++k) {
                            const int o = sorted[b0 + k];
#pragma unroll
                            for (int e = 0; e < ENS_RANK; ++e) rank[e] += o < v[e];
                        }
                        __syncwarp();
#pragma unroll
                        for (int e = 0; e < ENS_RANK; ++e)
                            if (wl + 32 * e < m) sorted[b0 + rank[e]] = v[e];
                        __syncwarp();
                    } else if (wl == 0) {  // a collapsed cell: insertion sort
                        for (int k = b0 + 1; k < b0 + m; ++k) {
                            const int v0 = sorted[k];
                            int q = k - 1;
                            while (q >= b0 && sorted[q] > v0) {
                                sorted[q + 1] = sorted[q];
                                --q;
                            }
                            sorted[q + 1] = v0;
                        }
                    }
                }
            }
            if (tid == 0) next_item = 0;
            __syncthreads();
            // list rows: a warp per item, an item a cell (in a one-cell
            // replica 32 of its atoms), taken from a shared counter; lane =
            // one of the cell's atoms (32 at a time). The stencil cells'
            // atoms pass, in stencil then index order, through a per-warp
            // buffer that takes only those within the list radius of the box
            // of the warp's atoms (about 3 in 4), and each lane appends those
            // within the list radius of its own atom to its row. (Items on a
            // counter, so that no warp waits for the one with the fullest
            // cells; a one-cell replica has a warp per 32 atoms instead of
            // one warp in all.)
            {
                const int wl = tid & 31;
                const float rl2 = R.fx_rl2;
                uint4* const buf = cand[tid >> 5];
                const int items = ns > 0 ? ncell : (n + 31) / 32;
                for (;;) {
                    int c = 0;
                    if (wl == 0) c = atomicAdd(&next_item, 1);
                    c = __shfl_sync(0xffffffffu, c, 0);
                    if (c >= items) break;
                    const int cx = ns > 0 ? c / (nc * nc) : 0, cy = ns > 0 ? (c / nc) % nc : 0,
                              cz = ns > 0 ? c % nc : 0;
                    const int c0 = ns > 0 ? cstart[c] : 32 * c, c1 = ns > 0 ? cstart[c + 1] : min(n, 32 * c + 32);
                    for (int a0c = c0; a0c < c1; a0c += 32) {
                        const bool active = a0c + wl < c1;
                        const int i = active ? sorted[a0c + wl] : 0;
                        const uint4 qi = pos[i];
                        const int64_t gi = a0 + i;
                        uint16_t* row = rows + gi * 2 * cap;
                        int cnt = 0;
                        // the box of the warp's atoms, as offsets from the first one's position
                        uint4 ref = qi;
                        ref.x = __shfl_sync(0xffffffffu, qi.x, 0);
                        ref.y = __shfl_sync(0xffffffffu, qi.y, 0);
                        ref.z = __shfl_sync(0xffffffffu, qi.z, 0);
                        const int rx = active ? (int)(qi.x - ref.x) : 0, ry = active ? (int)(qi.y - ref.y) : 0,
                                  rz = active ? (int)(qi.z - ref.z) : 0;
                        const float lox = (float)__reduce_min_sync(0xffffffffu, rx),
                                    hix = (float)__reduce_max_sync(0xffffffffu, rx),
                                    loy = (float)__reduce_min_sync(0xffffffffu, ry),
                                    hiy = (float)__reduce_max_sync(0xffffffffu, ry),
                                    loz = (float)__reduce_min_sync(0xffffffffu, rz),
                                    hiz = (float)__reduce_max_sync(0xffffffffu, rz);
                        int fill = 0;
                        // the m candidates of the buffer: the tests without a
                        // branch into a bit mask, then the lane's hits in order
                        auto test = [&](int m) {
                            unsigned hits = 0u;
#pragma unroll 8
                            for (int k = 0; k < m; ++k) {
                                const uint4 c = buf[k];
                                float ddx, ddy, ddz;
                                const float r2 = fx_r2(qi, c, ddx, ddy, ddz);
                                hits |= (r2 < rl2 && (int)c.w != i) ? 1u << k : 0u;
                            }
                            if (!active) hits = 0u;
                            while (hits) {
                                const int j = (int)buf[__ffs(hits) - 1].w;
                                hits &= hits - 1u;
                                if (cnt < cap) row[ens_slot<LPA>(cnt)] = (uint16_t)j;
                                ++cnt;
                            }
                        };
                        for (int ox = -ns; ox <= ns; ++ox) {
                            int nx = cx + ox;
                            nx += nx < 0 ? nc : 0;
                            nx -= nx >= nc ? nc : 0;
                            for (int oy = -ns; oy <= ns; ++oy) {
                                int ny = cy + oy;
                                ny += ny < 0 ? nc : 0;
                                ny -= ny >= nc ? nc : 0;
                                for (int oz = -ns; oz <= ns; ++oz) {
                                    int nz = cz + oz;
                                    nz += nz < 0 ? nc : 0;
                                    nz -= nz >= nc ? nc : 0;
                                    const int cq = (nx * nc + ny) * nc + nz;
                                    const int q1 = cstart[cq + 1];
                                    for (int kb = cstart[cq]; kb < q1; kb += 32) {
                                        // a candidate per lane; those out of every row's reach are dropped
                                        uint4 qc = qi;
                                        bool keep = kb + wl < q1;
                                        if (keep) {
                                            const int j = sorted[kb + wl];
                                            qc = pos[j];
                                            qc.w = (unsigned)j;
                                            if (ns > 0) {
                                                const float gx = ens_gap(qc.x - ref.x, lox, hix);
                                                const float gy = ens_gap(qc.y - ref.y, loy, hiy);
                                                const float gz = ens_gap(qc.z - ref.z, loz, hiz);
                                                keep = gx * gx + gy * gy + gz * gz < rl2 * 1.0002f;
                                            }
                                        }
                                        const unsigned bal = __ballot_sync(0xffffffffu, keep);
                                        const int at = fill + __popc(bal & ((1u << wl) - 1u));
                                        const int added = __popc(bal);
                                        if (keep && at < 32) buf[at] = qc;
                                        __syncwarp();
                                        fill += added;
                                        if (fill >= 32) {
                                            test(32);
                                            __syncwarp();
                                            if (keep && at >= 32) buf[at - 32] = qc;
                                            fill -= 32;
                                        }
                                    }
                                }
                            }
                        }
                        __syncwarp();
                        test(fill);
                        __syncwarp();  // (the buffer is free for the next chunk)
                        if (active) {
                            if (cnt > cap) {
                                status_set(d.status, ST_NBR_OVERFLOW);
                                cnt = cap;
                            }
                            d.nbr_count[gi] = cnt;
                            cnts[i] = (uint16_t)cnt;
                            A.pref[gi] = qi;
                        }
                    }
                }
            }
            since = 0;
            __syncthreads();  // rows written before they are read (other groups)
        } else {
            ++since;
        }
        // forces from the list rows (neighbours from shared memory), then
        // the velocity update of the atom by a lane per component
        const bool lj_atoms = POT != FX_EL;
        const float lj_lo = R.fx_lj_lo, lj_hi = R.fx_lj_hi, el_lo = R.fx_el_lo, el_hi = R.fx_el_hi;
        const float sig2h = R.fx_sig2_hi, sig2l = R.fx_sig2_lo, krf = R.fx_krf;
        for (int i0 = 0; i0 < n; i0 += G) {
            const int i = i0 + g;
            const bool active = i < n;
            const int64_t gi = a0 + (active ? i : 0);
            const uint4 qi = pos[active ? i : 0];
            const int cnt = active ? cnts[i] : 0;
            const int cmax = __reduce_max_sync(0xffffffffu, cnt);  // the warp's longest row
            const float kqi =
                POT != FX_LJ ? (float)(d.charge[gi] * R.fx_kq) : 0.0f;
            // the velocity update's operands (one lane per component, as
            // lane_sums3 leaves them) are loaded ahead of the pair loop
            const int comp = min(lane / (LPA / 4), 2);
            const bool upd = active && lane == comp * (LPA / 4);
            const int64_t e = 3 * gi + comp;
            const double im = d.inv_mass_fx[gi];
            const double v_in = upd ? s.v[e] : 0.0;
            const double ao_in = upd && !A.baoab ? s.a_old[e] : 0.0;
            const uint4* row = reinterpret_cast<const uint4*>(rows + gi * 2 * cap) + lane;
            float2 px = make_float2(0.f, 0.f), py = px, pz = px;
            // one load holds the lane's entries of four packed steps; the
            // next block's load is issued before this block's arithmetic.
            // An entry past the row's count reads the atom itself and adds
            // zero; steps past the warp's longest row are skipped.
            uint4 nx = lane < cnt ? __ldcg(row) : make_uint4(0u, 0u, 0u, 0u);
            for (int kb = 0; kb < cmax; kb += 8 * LPA) {
                const uint4 cur = nx;
                if (kb + 8 * LPA + lane < cnt) nx = __ldcg(row + (kb / 8 + LPA));
                const unsigned w[4] = {cur.x, cur.y, cur.z, cur.w};
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const int k0 = kb + 2 * m * LPA;
                    if (k0 >= cmax) break;
                    const bool v0 = k0 + lane < cnt, v1 = k0 + LPA + lane < cnt;
                    int j0 = v0 ? (int)(w[m] & 0xffffu) : (active ? i : 0);
                    int j1 = v1 ? (int)(w[m] >> 16) : (active ? i : 0);
                    // (debug builds: an entry outside the replica's atoms is
                    // reported and replaced by its first atom)
                    j0 = dbg_index(j0, n, 0, d.status);
                    j1 = dbg_index(j1, n, 0, d.status);
                    const uint4 q0 = pos[j0], q1 = pos[j1];
                    fx_pair2<POT>(d, s.x, gi, lj_atoms, kqi, qi, (int)a0 + j0, (int)a0 + j1, v0, v1, q0, q1, lj_lo,
                                  lj_hi, el_lo, el_hi, sig2h, sig2l, krf, px, py, pz, range_err);
                }
            }
            float hx = __fadd_rn(px.x, px.y), hy = __fadd_rn(py.x, py.y), hz = __fadd_rn(pz.x, pz.y);
            // a lane per component updates the velocity
            const LaneSum f = lane_sums3<LPA>(hx, hy, hz, lane);
            if (upd) {
                const double an = (widen(f.h) + widen(f.e)) * im;
                if (!finite64(an)) status_set(d.status, ST_NONFINITE);
                const double vn = A.baoab ? __dadd_rn(v_in, __dmul_rn(hdt, an)) : kick1(v_in, ao_in, an, dt);
                s.v[e] = vn;
                s.a_old[e] = an;
                s.a_new[e] = an;
                const int64_t t = step + 1 - sk_t0;  // the frame sink's index of the new state
                if (sk_every > 0 && t % sk_every == 0) {
                    const FrameSink* sk = d.sink;
                    const int64_t slot = t / sk_every - sk->first;
                    if (slot >= 0 && slot < sk->cap) {
                        const size_t o = (size_t)slot * 3 * d.cols + (size_t)e;
                        sk->x[o] = s.x[e];
                        sk->v[o] = vn;
                    }
                }
            }
        }
        __syncthreads();  // the next step's integration overwrites the shared positions
    }
    if (range_err) status_set(d.status, ST_RANGE);
    if (tid == 0) A.since[r] = since;
}

// ---------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------
typedef void (*ens_kernel_t)(Dev, StateView, EnsArgs);

template <int POT, int THREADS>
static ens_kernel_t ens_kernel_lpa(int lpa)
{
    return lpa == 8 ? k_ensemble<8, POT, THREADS> : k_ensemble<4, POT, THREADS>;
}

template <int POT>
static ens_kernel_t ens_kernel_threads(int lpa, int threads)
{
    switch (threads) {
    case 512: return ens_kernel_lpa<POT, 512>(lpa);
    case 1024: return ens_kernel_lpa<POT, 1024>(lpa);
    default: return ens_kernel_lpa<POT, 768>(lpa);
    }
}

static ens_kernel_t ens_kernel(const nbg_ctx* c)
{
    return c->d.pots == NBG_POT_LJ ? ens_kernel_threads<FX_LJ>(c->ens_lpa, c->ens_threads)
                                   : ens_kernel_threads<FX_LJEL>(c->ens_lpa, c->ens_threads);
}

static int ens_mode(const nbg_ctx* c)
{
    return c->ens_cells == 2 ? 1 : 0;
}

// Whether a batch runs the persistent loop, with its form (lanes, threads,
// cell width) and shared memory; per-replica cell grids are set here.
bool ensemble_plan(nbg_ctx* c)
{
    c->ens_ok = false;
    if (c->ens_disabled || c->nrep < 2 || c->path != PATH_LIST || c->d.kind != NBG_SYSTEM_POTENTIAL ||
        c->d.bc != NBG_BC_CUBIC || !c->d.pfx || (c->d.pots & ~(uint32_t)(NBG_POT_LJ | NBG_POT_EL)) ||
        !(c->d.therm == NBG_THERMO_NULL || (c->d.therm == NBG_THERMO_LANGEVIN && c->baoab)))
        return false;
    int64_t nmax = 0;
    int cmax = 1;
    for (int r = 0; r < c->nrep; ++r) {
        RepDev& R = c->reps_h[r];
        nmax = std::max<int64_t>(nmax, R.n);
        const double rl = std::sqrt((double)R.fx_rl2) * (R.L / 4294967296.0);
        const int n1 = (int)std::floor(R.L / (rl * (1.0 + 1e-4)));
        const int n2 = (int)std::floor(R.L / (0.5 * rl * (1.0 + 1e-4)));
        R.ens_nc[0] = n1 >= 3 ? n1 : 1;
        R.ens_ns[0] = n1 >= 3 ? 1 : 0;
        R.ens_nc[1] = n2 >= 5 ? n2 : R.ens_nc[0];
        R.ens_ns[1] = n2 >= 5 ? 2 : R.ens_ns[0];
        for (int m = 0; m < 2; ++m) cmax = std::max(cmax, R.ens_nc[m] * R.ens_nc[m] * R.ens_nc[m]);
    }
    if (nmax > ENS_MAX_ATOMS || cmax > ENS_MAX_CELLS) return false;
    if (cudaMemcpy(const_cast<RepDev*>(c->d.reps), c->reps_h.data(), sizeof(RepDev) * c->nrep,
                   cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    c->ens_smem = sizeof(uint4) * (size_t)nmax + sizeof(int) * (2 * (size_t)cmax + 1) +
                  2 * sizeof(uint16_t) * (size_t)nmax;
    ens_kernel_t k = ens_kernel(c);
    if (!allow_shared((const void*)k, c->device, c->ens_smem)) return false;
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, c->ens_threads, c->ens_smem) != cudaSuccess || occ < 1) {
        cudaGetLastError();
        return false;
    }
    c->ens_ok = true;
    return true;
}

int launch_ensemble(nbg_ctx* c, const StateView& s, double dt, int64_t nsteps, int64_t step0, unsigned* status)
{
    EnsArgs A;
    A.order = c->ens_order;
    A.since = c->ens_since;
    A.pref = c->ens_pref;
    A.reuse = c->ens_lists_valid ? 1 : 0;
    A.mode = ens_mode(c);
    A.dt = dt;
    A.nsteps = (int)nsteps;
    A.rebuild_every = c->desc.rebuild_every;
    A.step0 = step0;
    A.save = c->sink_on ? 1 : 0;
    A.baoab = c->baoab ? 1 : 0;
    Dev d = c->d;
    d.status = status;
    prof_begin(c);
    ens_kernel(c)<<<(unsigned)c->nrep, (unsigned)c->ens_threads, c->ens_smem, c->stream>>>(d, s, A);
    prof_end(c);
    NBG_LAUNCH_CHECK(c, "k_ensemble");
    return NBG_OK;
}
