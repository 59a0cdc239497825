// k_forces.cu - force kernels.
//
//  k_gravity<PLAIN>  all-pairs gravity (gravitational_acceleration!,
//                    basic_potentials.jl:306-331): 128-body j-tiles of split
//                    positions staged in shared memory and read as warp-wide
//                    broadcasts, two bodies i per thread; the j range is cut
//                    into J chunks so the grid fills whole waves of resident
//                    blocks (J partials per body in scratch, reduced in fixed
//                    order by k_gravity_reduce).
//                    Per pair: FP32 differences of hi/lo split positions (exact
//                    to ~2^-24 of |r_ij|, or plain FP32 positions when PLAIN),
//                    one rsqrt, partial sums per tile folded into a compensated
//                    (TwoSum) pair. With tile boxes (bodies sorted along a
//                    Morton curve), a tile pair whose boxes or radial shells
//                    are apart by at least 1/16 of their largest |r| uses the
//                    plain difference: its error, 2^-24 of the coordinates,
//                    is then below 2^-19 of |r_ij|.
//  k_allpairs_cut    LJ and electrostatics on small / unbounded systems under
//                    infinite or cubic boundaries: a cluster of CTAs per 32
//                    bodies, the 128-body j-tiles shared out over its CTAs,
//                    their sums folded in tile order by the first one; two
//                    bodies j per packed instruction.
//  k_allpairs        every other form off the lists (mixed potentials, general
//                    periodic boxes, dipoles, more than 32,768 bodies): 32
//                    bodies a block, a warp per 128-body j-tile.
//  k_force_list      cutoff LJ + reaction-field electrostatics over a Verlet
//                    list (one thread per atom, coalesced column-major list).
//  k_bonded          SPC/Fw harmonic bonds and H-O-H angles, one thread per
//                    molecule (basic_potentials.jl:367-433), FP32 terms from
//                    FP64 intramolecular differences.
#include <algorithm>
#include <type_traits>

#include <cooperative_groups.h>
#include <cub/device/device_radix_sort.cuh>

#include "nbg_internal.cuh"

#define GB 128         // gravity block size = j-tile size
#define GI_MAX (4 * GB)  // bodies i per block at most (TI <= 4)
#define GRAV_SPREAD 2048 // largest padded system whose bodies take a thread each

// Grid: (i-block, j-chunk) units; each thread owns TI bodies i (strided by
// GB within the block) and walks the chunk's j-tiles from shared memory:
// every lane of a warp reads the same body j (one broadcast load serves TI
// pairs). PACKED evaluates the TI bodies two at a time with the packed
// FP32x2 instructions (__ffma2_rn / __fadd2_rn / __fmul2_rn), which halve the
// issued FP32 instructions; both forms round every element identically.
// Per pair: p += m_j (r_i - r_j) |r_i - r_j|^-3 (gravitational_acceleration!,
// basic_potentials.jl:318-324), the j == i term skipped (:318).
// Accumulate one j-tile (sh_hi / sh_lo) into the per-body partials.
// DIAG: the tile holds some of this thread's own bodies (j == i skipped).
template <bool PLAIN, int TI, bool PACKED, bool DIAG, bool UNIFORM>
__device__ __forceinline__ void grav_tile(const float4* sh_hi, const float4* sh_lo, int64_t j0, const int64_t* ii,
                                          const float* hx, const float* hy, const float* hz, const float* lx,
                                          const float* ly, const float* lz, float* px, float* py, float* pz)
{
    constexpr int NP = PACKED ? TI / 2 : 1;
    if (!PACKED) {
#pragma unroll 4
        for (int jj = 0; jj < GB; ++jj) {
            const float4 hj = sh_hi[jj];
            float4 lj = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!PLAIN) lj = sh_lo[jj];
#pragma unroll
            for (int k = 0; k < TI; ++k) {
                float dx = hx[k] - hj.x, dy = hy[k] - hj.y, dz = hz[k] - hj.z;
                if (!PLAIN) {
                    dx += lx[k] - lj.x;
                    dy += ly[k] - lj.y;
                    dz += lz[k] - lj.z;
                }
                float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                float ri = rsqrt_ftz(r2);
                if (DIAG && j0 + jj == ii[k]) ri = 0.0f;
                const float sc = UNIFORM ? __fmul_rn(ri, __fmul_rn(ri, ri)) : __fmul_rn(__fmul_rn(hj.w, ri), __fmul_rn(ri, ri));
                px[k] = fmaf(sc, dx, px[k]);
                py[k] = fmaf(sc, dy, py[k]);
                pz[k] = fmaf(sc, dz, pz[k]);
            }
        }
        return;
    }
    float2 hx2[NP], hy2[NP], hz2[NP], lx2[NP], ly2[NP], lz2[NP], px2[NP], py2[NP], pz2[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        hx2[q] = make_float2(hx[2 * q], hx[2 * q + 1]);
        hy2[q] = make_float2(hy[2 * q], hy[2 * q + 1]);
        hz2[q] = make_float2(hz[2 * q], hz[2 * q + 1]);
        lx2[q] = make_float2(lx[2 * q], lx[2 * q + 1]);
        ly2[q] = make_float2(ly[2 * q], ly[2 * q + 1]);
        lz2[q] = make_float2(lz[2 * q], lz[2 * q + 1]);
        px2[q] = py2[q] = pz2[q] = make_float2(0.f, 0.f);
    }
    const float2 m1 = make_float2(-1.f, -1.f);
#pragma unroll 8
    for (int jj = 0; jj < GB; ++jj) {
        const float4 hj = sh_hi[jj];
        const float2 jx = make_float2(hj.x, hj.x), jy = make_float2(hj.y, hj.y), jz = make_float2(hj.z, hj.z);
        const float2 jm = make_float2(hj.w, hj.w);
        float2 kx = m1, ky = m1, kz = m1;
        if (!PLAIN) {
            const float4 lj = sh_lo[jj];
            kx = make_float2(lj.x, lj.x);
            ky = make_float2(lj.y, lj.y);
            kz = make_float2(lj.z, lj.z);
        }
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            float2 dx = __ffma2_rn(jx, m1, hx2[q]);  // hi_i - hi_j (scaling by -1 is exact)
            float2 dy = __ffma2_rn(jy, m1, hy2[q]);
            float2 dz = __ffma2_rn(jz, m1, hz2[q]);
            if (!PLAIN) {
                dx = __fadd2_rn(dx, __ffma2_rn(kx, m1, lx2[q]));
                dy = __fadd2_rn(dy, __ffma2_rn(ky, m1, ly2[q]));
                dz = __fadd2_rn(dz, __ffma2_rn(kz, m1, lz2[q]));
            }
            float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
            float2 ri = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
            if (DIAG) {
                if (j0 + jj == ii[2 * q]) ri.x = 0.0f;
                if (j0 + jj == ii[2 * q + 1]) ri.y = 0.0f;
            }
            // equal masses: m_j leaves the sum (the reduction multiplies by G m)
            float2 sc = UNIFORM ? __fmul2_rn(ri, __fmul2_rn(ri, ri)) : __fmul2_rn(__fmul2_rn(jm, ri), __fmul2_rn(ri, ri));
            px2[q] = __ffma2_rn(sc, dx, px2[q]);
            py2[q] = __ffma2_rn(sc, dy, py2[q]);
            pz2[q] = __ffma2_rn(sc, dz, pz2[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        px[2 * q] = px2[q].x; px[2 * q + 1] = px2[q].y;
        py[2 * q] = py2[q].x; py[2 * q + 1] = py2[q].y;
        pz[2 * q] = pz2[q].x; pz[2 * q + 1] = pz2[q].y;
    }
}

// Box of a 128-body tile from those of its four runs of 32 bodies:
// (min x, y, z, largest |r|) and (max x, y, z, smallest |r|).
__device__ __forceinline__ void tile_box(const float4* __restrict__ box, int64_t t, float4& lo, float4& hi)
{
    lo = box[8 * t];
    hi = box[8 * t + 1];
#pragma unroll
    for (int q = 1; q < 4; ++q) {
        const float4 a = box[8 * t + 2 * q], b = box[8 * t + 2 * q + 1];
        lo = make_float4(fminf(lo.x, a.x), fminf(lo.y, a.y), fminf(lo.z, a.z), fmaxf(lo.w, a.w));
        hi = make_float4(fmaxf(hi.x, b.x), fmaxf(hi.y, b.y), fmaxf(hi.z, b.z), fminf(hi.w, b.w));
    }
}

// Grid: (i-block, j-chunk) units; each thread owns TI bodies i (strided by
// GB within the block) and walks the chunk's j-tiles from shared memory:
// every lane of a warp reads the same body j (one broadcast load serves TI
// pairs). PACKED evaluates the TI bodies two at a time with the packed
// FP32x2 instructions (__ffma2_rn / __fadd2_rn / __fmul2_rn), which halve the
// issued FP32 instructions; both forms round every element identically.
// Per pair: p += m_j (r_i - r_j) |r_i - r_j|^-3 (gravitational_acceleration!,
// basic_potentials.jl:318-324), the j == i term skipped (:318).
// UNIFORM: every body has the same mass, which the reduction applies.
template <bool PLAIN, int TI, bool PACKED, bool UNIFORM>
__global__ void __launch_bounds__(GB, TI == 2 ? 7 : 1) k_gravity(const float4* __restrict__ phi, const float4* __restrict__ plo,
                                                int64_t n, int64_t npad, int jchunks, double* __restrict__ part,
                                                const float4* __restrict__ box, float far2)
{
    static_assert(TI == 1 || TI == 2 || TI == 4, "TI");
    static_assert(!PACKED || TI >= 2, "packed needs pairs");
    __shared__ float4 sh_hi[GB];
    __shared__ float4 sh_lo[PLAIN ? 1 : GB];
    const int64_t ntile = npad / GB;
    const int64_t iblock = blockIdx.x / jchunks;
    const int jc = (int)(blockIdx.x % jchunks);
    const int64_t t0 = (int64_t)jc * ntile / jchunks;
    const int64_t t1 = (int64_t)(jc + 1) * ntile / jchunks;
    const int64_t ib0 = iblock * (TI * GB);
    // thread t owns bodies ib0 + TI t .. + TI - 1: a warp's bodies lie in one
    // of the block's TI 128-body tiles (its i-tile `it`), so the far test of a
    // tile pair is uniform over the warp
    const int it = (int)((threadIdx.x * TI) / GB);
    float hx[TI], hy[TI], hz[TI], lx[TI], ly[TI], lz[TI];
    int64_t ii[TI];
#pragma unroll
    for (int k = 0; k < TI; ++k) {
        ii[k] = ib0 + (int64_t)threadIdx.x * TI + k;
        float4 h = phi[ii[k]];
        hx[k] = h.x; hy[k] = h.y; hz[k] = h.z;
        float4 l = PLAIN ? make_float4(0.f, 0.f, 0.f, 0.f) : plo[ii[k]];
        lx[k] = l.x; ly[k] = l.y; lz[k] = l.z;
    }
    Acc2 ax[TI], ay[TI], az[TI];
#pragma unroll
    for (int k = 0; k < TI; ++k) ax[k] = ay[k] = az[k] = Acc2{0.f, 0.f};
    // boxes and radial shells of the block's TI i-tiles
    __shared__ float4 ibox_s[2 * TI];
    if (!PLAIN && box && threadIdx.x < TI)
        tile_box(box, ib0 / GB + threadIdx.x, ibox_s[2 * threadIdx.x], ibox_s[2 * threadIdx.x + 1]);
    constexpr unsigned ALL_FAR = (1u << TI) - 1u;
    __shared__ unsigned char far_s[GB];  // per j-tile of the next GB: bit k = far from i-tile k
    for (int64_t t = t0; t < t1; ++t) {
        const int64_t j0 = t * GB;
        // far tile pair: a lower bound g of |r_ij| (the boxes' gap, or the
        // radial shells' gap) with F g >= the largest |r| of both tiles
        // (far2 = F^2; F = 16 by default);
        // flags for GB j-tiles at a time, one j-tile per thread
        if (!PLAIN && box && (t - t0) % GB == 0) {
            __syncthreads();
            const int64_t tt = t + threadIdx.x;
            unsigned f = 0;
            if (tt < t1) {
                float4 lo4, hi4;
                tile_box(box, tt, lo4, hi4);
#pragma unroll
                for (int k = 0; k < TI; ++k) {
                    const float4 a = ibox_s[2 * k], b = ibox_s[2 * k + 1];  // (min x,y,z, max|r|), (max x,y,z, min|r|)
                    const float gx = fmaxf(0.f, fmaxf(a.x - hi4.x, lo4.x - b.x));
                    const float gy = fmaxf(0.f, fmaxf(a.y - hi4.y, lo4.y - b.y));
                    const float gz = fmaxf(0.f, fmaxf(a.z - hi4.z, lo4.z - b.z));
                    const float gr = fmaxf(0.f, fmaxf(b.w - lo4.w, hi4.w - a.w));
                    const float g2 = fmaxf(gx * gx + gy * gy + gz * gz, gr * gr);
                    const float mm = fmaxf(a.w, lo4.w);
                    if (g2 > 0.f && far2 * g2 >= mm * mm) f |= 1u << k;
                }
            }
            far_s[threadIdx.x] = (unsigned char)f;
        }
        __syncthreads();
        const unsigned fl = (!PLAIN && box) ? far_s[(t - t0) % GB] : 0u;
        const bool far = (fl >> it) & 1u;
        sh_hi[threadIdx.x] = phi[j0 + threadIdx.x];
        if (!PLAIN && fl != ALL_FAR) sh_lo[threadIdx.x] = plo[j0 + threadIdx.x];
        __syncthreads();
        float px[TI], py[TI], pz[TI];
#pragma unroll
        for (int k = 0; k < TI; ++k) px[k] = py[k] = pz[k] = 0.f;
        if (!PLAIN && far)
            grav_tile<true, TI, PACKED, false, UNIFORM>(sh_hi, sh_lo, j0, ii, hx, hy, hz, lx, ly, lz, px, py, pz);
        else if ((j0 < ib0 + TI * GB) && (j0 + GB > ib0))
            grav_tile<PLAIN, TI, PACKED, true, UNIFORM>(sh_hi, sh_lo, j0, ii, hx, hy, hz, lx, ly, lz, px, py, pz);
        else
            grav_tile<PLAIN, TI, PACKED, false, UNIFORM>(sh_hi, sh_lo, j0, ii, hx, hy, hz, lx, ly, lz, px, py, pz);
#pragma unroll
        for (int k = 0; k < TI; ++k) {
            ax[k].add(px[k]);
            ay[k].add(py[k]);
            az[k].add(pz[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < TI; ++k) {
        if (ii[k] < n) {
            double* p = part + ((int64_t)jc * n + ii[k]) * 3;
            p[0] = ax[k].value();
            p[1] = ay[k].value();
            p[2] = az[k].value();
        }
    }
}

typedef void (*grav_kernel_t)(const float4*, const float4*, int64_t, int64_t, int, double*, const float4*, float);

// Kernel variants: bodies per thread (TI) x packed FP32x2; index
// 0: TI=2 scalar, 1: TI=2 packed, 2: TI=4 scalar, 3: TI=4 packed, 4: TI=1 scalar.
// uniform (equal masses) selects the forms without m_j in the loop (1, 3, 4).
static grav_kernel_t grav_variant(bool plain, int v, bool uniform)
{
    switch (v) {
    case 0: return plain ? k_gravity<true, 2, false, false> : k_gravity<false, 2, false, false>;
    case 2: return plain ? k_gravity<true, 4, false, false> : k_gravity<false, 4, false, false>;
    case 3:
        if (uniform) return plain ? k_gravity<true, 4, true, true> : k_gravity<false, 4, true, true>;
        return plain ? k_gravity<true, 4, true, false> : k_gravity<false, 4, true, false>;
    case 4:
        if (uniform) return plain ? k_gravity<true, 1, false, true> : k_gravity<false, 1, false, true>;
        return plain ? k_gravity<true, 1, false, false> : k_gravity<false, 1, false, false>;
    default:
        if (uniform) return plain ? k_gravity<true, 2, true, true> : k_gravity<false, 2, true, true>;
        return plain ? k_gravity<true, 2, true, false> : k_gravity<false, 2, true, false>;
    }
}
static bool grav_variant_uniform(int v) { return v != 0 && v != 2; }
static int grav_ti(int v) { return v == 2 || v == 3 ? 4 : (v == 4 ? 1 : 2); }

// a_i = -G sum_chunks partial_i (fixed chunk order); with a permutation the
// partials are in sorted order and body perm[s] receives slot s
__global__ void k_gravity_reduce(const double* __restrict__ part, int64_t n, int jchunks, double G,
                                 double* __restrict__ A, unsigned* status, const int* __restrict__ perm)
{
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < 3 * n; e += (int64_t)gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int c = 0; c < jchunks; ++c) s += part[(int64_t)c * 3 * n + e];
        double a = -G * s;
        if (!finite64(a)) status_set(status, ST_NONFINITE);
        const int64_t slot = e / 3;
        A[perm ? 3 * (int64_t)perm[slot] + (e - 3 * slot) : e] = a;
    }
}

// Morton order of the bodies: 21 bits per dimension of the position in
// [-S, S]^3 (clamped), interleaved (x in the top bit of each triple). The
// fine grid keeps a concentrated core ordered when a few bodies lie far out.
__device__ __forceinline__ unsigned long long spread3(unsigned long long v)
{
    v &= 0x1fffffull;
    v = (v | (v << 32)) & 0x1f00000000ffffull;
    v = (v | (v << 16)) & 0x1f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

// Largest |coordinate| of the finite positions, rounded up to FP32, as the
// bits of a non-negative float (which order like unsigned integers): the
// half-width of the Morton cube. *ext is 0 before (k_grav_pack_sorted clears
// it after its use).
__device__ __forceinline__ void extent_max(double x, unsigned* ext)
{
    const unsigned v = finite64(x) ? __float_as_uint(__double2float_ru(fabs(x))) : 0u;
    const unsigned m = __reduce_max_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(ext, m);
}

__global__ void __launch_bounds__(256) k_grav_extent(const double* __restrict__ X, int64_t m, unsigned* ext)
{
    double v = 0.0;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x) {
        const double a = fabs(X[e]);
        // (non-negative doubles order like integers)
        if (finite64(a) && __double_as_longlong(a) > __double_as_longlong(v)) v = a;
    }
    extent_max(v, ext);
}

// vals: null where the ranks are counted (k_grav_rank)
__global__ void __launch_bounds__(64) k_grav_keys(const double* __restrict__ X, int64_t n,
                                                  const unsigned* __restrict__ ext, unsigned long long* keys, int* vals)
{
    const double cells = 2097152.0;  // 2^21
    __shared__ double scale;         // (one FP64 division per block)
    if (threadIdx.x == 0) {
        const double S = (double)__uint_as_float(*ext) * 1.0001;
        scale = S > 0.0 && isfinite(S) ? 0.5 / S : 0.5;
    }
    __syncthreads();
    const double inv2S = scale;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        unsigned long long q[3];
        for (int k = 0; k < 3; ++k) {
            const double t = (X[3 * i + k] * inv2S + 0.5) * cells;
            // clamped to [0, cells - 1]; not finite: NaN 0, +-Inf at the ends' cells
            const long long b = __double_as_longlong(t);
            int c = 0;
            if (b >= __double_as_longlong(cells - 1.0)) c = t == t ? 2097151 : 0;
            else if (b > 0) c = __double2int_rz(t);
            q[k] = (unsigned long long)c;
        }
        keys[i] = (spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]);
        if (vals) vals[i] = (int)i;
    }
}

// The stable order by counting: the rank of body i is the number of bodies j
// with key_j < key_i, or key_j = key_i and j < i. A block ranks 32 bodies (a
// lane each), its 8 warps count an eighth of the keys each (keys below 2^63:
// "<=" is "< key + 1"). One launch of n^2 / 32 compares instead of a radix
// sort's single block or chain of passes: 1500 bodies 16 -> 5.3 us. Every warp
// reads each staged key once for its 32 bodies: shared-memory loads bound it.
__global__ void __launch_bounds__(256) k_grav_rank(const unsigned long long* __restrict__ keys, int n, int* __restrict__ perm)
{
    constexpr int CH = 2048;  // keys staged at a time
    __shared__ __align__(16) unsigned long long sk[CH];
    __shared__ int rank[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i0 = blockIdx.x * 32, i = i0 + lane;
    if (threadIdx.x < 32) rank[lane] = 0;
    const unsigned long long key = i < n ? keys[i] : 0ull;
    int cnt = 0;
    for (int c0 = 0; c0 < n; c0 += CH) {
        __syncthreads();
        // (the largest key, behind the last, counts for nobody)
        for (int k = threadIdx.x; k < CH; k += 256) sk[k] = c0 + k < n ? keys[c0 + k] : ~0ull;
        __syncthreads();
        const int m = min(CH, n - c0);
        const int per = ((m + 7) / 8 + 1) & ~1;  // even: pairs of keys load as 16 bytes
        const int b = w * per, e = min(m, b + per);
        const int jb = c0 + b, je = c0 + e;
        auto two = [&](int k, unsigned long long t0, unsigned long long t1) {
            const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(sk + k);
            cnt += (q.x < t0) + (q.y < t1);
        };
        if (je <= i0 || jb >= i0 + 32) {  // all before the block's bodies, or all after
            const unsigned long long t = key + (je <= i0 ? 1 : 0);
#pragma unroll 8
            for (int k = b; k < e; k += 2) two(k, t, t);
        } else {
            for (int k = b; k < e; ++k) cnt += sk[k] < key + (c0 + k < i ? 1 : 0);
        }
    }
    atomicAdd(&rank[lane], cnt);
    __syncthreads();
    if (w == 0 && i < n) perm[rank[lane]] = i;
}

// The warp's box: (min x, y, z, largest |r|), (max x, y, z, smallest |r|) of
// 32 bodies' hi positions (a lane without a body: an inverted box)
__device__ __forceinline__ void warp_box(bool real, float x, float y, float z, float4* box)
{
    float v[8];  // minima of x, y, z, -x, -y, -z, |r|, -|r|
    if (real) {
        const float r = sqrtf(x * x + y * y + z * z);
        v[0] = x; v[1] = y; v[2] = z;
        v[3] = -x; v[4] = -y; v[5] = -z;
        v[6] = r; v[7] = -r;
    } else {
        for (int k = 0; k < 8; ++k) v[k] = INFINITY;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        for (int k = 0; k < 8; ++k) v[k] = fminf(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
    if ((threadIdx.x & 31) == 0) {
        box[0] = make_float4(v[0], v[1], v[2], -v[7]);
        box[1] = make_float4(-v[3], -v[4], -v[5], v[6]);
    }
}

// split positions and masses in sorted order (slot s holds body perm[s]), and
// the boxes of each 32 slots (128 threads per block, npad a multiple of 128)
__global__ void __launch_bounds__(GB) k_grav_pack_sorted(const double* __restrict__ X, const double* __restrict__ mass,
                                                         const int* __restrict__ perm, int64_t n, float4* phi, float4* plo,
                                                         float4* box, unsigned* ext)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) *ext = 0u;  // (ready for the next sort)
    const int64_t s = blockIdx.x * (int64_t)GB + threadIdx.x;
    const bool real = s < n;
    float h[3] = {0.f, 0.f, 0.f}, l[3];
    if (real) {
        const int64_t i = perm[s];
        for (int k = 0; k < 3; ++k) {
            const double p = X[3 * i + k];
            h[k] = (float)p;
            l[k] = (float)(p - (double)h[k]);
        }
        phi[s] = make_float4(h[0], h[1], h[2], (float)mass[i]);
        plo[s] = make_float4(l[0], l[1], l[2], 0.f);
    }
    warp_box(real, h[0], h[1], h[2], box + 2 * (s / 32));
}

// One pass over the bodies between two gravity evaluations of a captured run
// of steps: the sum of the chunk partials (KICK; k_gravity_reduce's
// operations) and the kick that ends step sr (k_kick's, no thermostat), the
// saved frame of that state, the next drift (k_drift_pack's), and (PACK: the
// next evaluation keeps the order) the sorted split positions and boxes of
// k_grav_pack_sorted. Block: 32 slots, warp k the component k, so that small
// systems spread their FP64 operations over the chip (1500 bodies: 47 blocks)
// and six launches per step become two.
struct GravStep {
    const double* part;
    const int* perm;  // null: slot = body
    int jchunks;
    double G, dt, dtsq;
    StepRef step;     // KICK: the step that ends
    int save;
    float4* box;      // null: none
    unsigned* ext;    // not PACK: the extent for the sort that follows
};

template <bool KICK, bool PACK>
__global__ void __launch_bounds__(96) k_grav_step(Dev d, StateView s, GravStep A)
{
    __shared__ float sh[3][32];
    const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
    const int64_t slot = blockIdx.x * (int64_t)32 + lane;
    const bool real = slot < d.n;
    float h = 0.f;
    double x = 0.0;
    if (real) {
        const int64_t i = A.perm ? A.perm[slot] : slot;
        const int64_t e = 3 * i + k;
        x = s.x[e];
        double v = s.v[e], a = s.a_old[e];
        if (KICK) {
            double t = 0.0;
            const double* p = A.part + 3 * slot + k;
#pragma unroll 4
            for (int c = 0; c < A.jchunks; ++c) t += p[(int64_t)c * 3 * d.n];
            const double an = -A.G * t;
            if (!finite64(an)) status_set(d.status, ST_NONFINITE);
            v = kick1(v, a, an, A.dt);
            a = an;
            s.a_old[e] = an;
            s.v[e] = v;
            if (A.save) {
                const FrameSink* sink = d.sink;
                const int64_t every = sink->every;
                const int64_t f = step_of(A.step) + 1 - sink->t0;
                if (every > 0 && f % every == 0) {
                    const int64_t q = f / every - sink->first;
                    if (q >= 0 && q < sink->cap) {
                        sink->x[q * 3 * d.cols + e] = x;
                        sink->v[q * 3 * d.cols + e] = v;
                    }
                }
            }
        }
        x = drift1(x, v, a, A.dt, A.dtsq);
        s.x[e] = x;
        if (PACK) {
            h = (float)x;
            reinterpret_cast<float*>(d.phi + slot)[k] = h;
            reinterpret_cast<float*>(d.plo + slot)[k] = (float)(x - widen(h));
        }
    }
    if (!PACK) extent_max(x, A.ext);
    if (!PACK || !A.box) return;
    sh[k][lane] = h;
    __syncthreads();
    if (k == 0) warp_box(real, h, sh[1][lane], sh[2][lane], A.box + 2 * (int64_t)blockIdx.x);
}

// Number of j-chunks: the smallest that makes (i-blocks x chunks) fill the
// resident block slots (SMs x blocks per SM) in near-whole waves.
static int plan_gravity(nbg_ctx* c, int64_t npad)
{
    int dev = c->device, sms = 0, occ = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // small systems: a body per thread spreads the pairs over twice the warps
    // while even those leave SM sub-partitions without one (the packed form's
    // arithmetic body by body, so the same bits): 1500 bodies 8.4 -> 6.5 us; a
    // whole step, packed against spread: 2100 bodies 18.3 and 17.5 us, 3000
    // 19.1 and 20.6.
    // The chunks stay those of the packed form.
    const bool spread = c->grav_variant == 1 && npad <= GRAV_SPREAD;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, grav_variant(c->d.grav_plain, c->grav_variant, c->grav_uniform),
                                                  GB, 0);
    if (sms < 1) sms = 1;
    if (occ < 1) occ = 1;
    const double slots = (double)sms * occ;
    const int64_t ib = npad / (grav_ti(c->grav_variant) * GB);
    const int64_t ntile = npad / GB;
    int best = 1;
    double best_eff = -1.0;
    for (int J = 1; J <= 64 && J <= ntile; ++J) {
        double waves = (double)(ib * J) / slots;
        // whole-wave efficiency, with chunks of ceil(ntile/J) vs ntile/J tiles
        double eff = waves / ceil(waves) * ((double)ntile / J) / (double)((ntile + J - 1) / J);
        if (eff > best_eff + 0.005) {
            best_eff = eff;
            best = J;
        }
        if (eff >= 0.97) break;
    }
    if (spread) c->grav_variant = 4;
    return best;
}

// Up to this many bodies the order is counted (k_grav_rank), above it sorted.
// A whole step, sorted against counted (one sort in 8 to 10 steps): 2000 bodies
// 17.3 and 15.2 us, 8300 69 and 60, 12,000 114 and 106, 16,000 167 and 160;
// the n^2 compares catch up with the sort soon after.
#define GRAV_RANK_MAX 16384
bool gravity_ranks(int64_t n) { return n <= GRAV_RANK_MAX; }

// Whether the next gravity evaluation sorts the bodies afresh (every 8th: the
// bodies move little in between).
static bool grav_sorts(const nbg_ctx* c) { return c->grav_sort && (!c->grav_perm_valid || c->grav_evals % 8 == 0); }

// The order and the sorted split positions and boxes of the next evaluation;
// packed: the positions and boxes are in place for the current order;
// extent: the pass before left the extent of the positions.
static int gravity_order(nbg_ctx* c, const StateView& s, bool packed, bool extent)
{
    if (!c->grav_sort) return NBG_OK;
    if (grav_sorts(c)) {
        packed = false;
        if (!extent) {
            k_grav_extent<<<(unsigned)std::min<int64_t>(grid_for(3 * c->n, 256), 2 * c->sms), 256, 0, c->stream>>>(
                s.x, 3 * c->n, c->grav_extent);
            NBG_LAUNCH_CHECK(c, "k_grav_extent");
        }
        k_grav_keys<<<grid_for(c->n, 64), 64, 0, c->stream>>>(s.x, c->n, c->grav_extent, c->grav_keys[0],
                                                               c->grav_vals[0]);
        NBG_LAUNCH_CHECK(c, "k_grav_keys");
        if (gravity_ranks(c->n)) {
            k_grav_rank<<<(unsigned)((c->n + 31) / 32), 256, 0, c->stream>>>(c->grav_keys[0], (int)c->n, c->grav_vals[1]);
            NBG_LAUNCH_CHECK(c, "k_grav_rank");
        } else {
            size_t bytes = c->grav_sort_bytes;
            cudaError_t e = cub::DeviceRadixSort::SortPairs(c->grav_sort_tmp, bytes, c->grav_keys[0], c->grav_keys[1],
                                                            c->grav_vals[0], c->grav_vals[1], (int)c->n, 0, 63,
                                                            c->stream);
            if (e != cudaSuccess) return cuda_fail(c, e, "gravity Morton sort");
            c->launches += 8;  // the sort's own passes
        }
        c->grav_perm_valid = true;
    }
    ++c->grav_evals;
    if (!packed) {
        k_grav_pack_sorted<<<(unsigned)(c->npad / GB), GB, 0, c->stream>>>(s.x, c->d.mass, c->grav_vals[1], c->n, c->d.phi,
                                                                           c->d.plo, c->grav_box, c->grav_extent);
        NBG_LAUNCH_CHECK(c, "k_grav_pack_sorted");
    }
    return NBG_OK;
}

// the pair sums of the packed positions into c->grav_part (grav_chunks * n * 3 doubles)
static int gravity_pairs(nbg_ctx* c)
{
    int64_t units = (c->npad / (grav_ti(c->grav_variant) * GB)) * c->grav_chunks;
    const bool uniform = c->grav_uniform && grav_variant_uniform(c->grav_variant);
    grav_kernel_t kern = grav_variant(c->d.grav_plain, c->grav_variant, uniform);
    prof_begin(c);
    kern<<<(unsigned)units, GB, 0, c->stream>>>(c->d.phi, c->d.plo, c->n, c->npad, c->grav_chunks, c->grav_part,
                                                c->grav_sort ? c->grav_box : nullptr, c->grav_far2);
    prof_end(c);
    NBG_LAUNCH_CHECK(c, "k_gravity");
    return NBG_OK;
}

static double gravity_factor(const nbg_ctx* c)
{
    return c->grav_uniform && grav_variant_uniform(c->grav_variant) ? c->d.G * c->grav_m0 : c->d.G;
}

static int gravity_reduce(nbg_ctx* c, const StateView& s)
{
    k_gravity_reduce<<<grid_for(3 * c->n, 256), 256, 0, c->stream>>>(c->grav_part, c->n, c->grav_chunks, gravity_factor(c),
                                                                      s.a_new, c->d.status,
                                                                      c->grav_sort ? c->grav_vals[1] : nullptr);
    NBG_LAUNCH_CHECK(c, "k_gravity_reduce");
    return NBG_OK;
}

// Order, pair sums and the chunk reduction into s.a_new.
int launch_gravity(nbg_ctx* c, const StateView& s)
{
    int st;
    if ((st = gravity_order(c, s, false, false))) return st;
    if ((st = gravity_pairs(c))) return st;
    return gravity_reduce(c, s);
}

// The gravity evaluation of step k of a captured run of steps after its
// drift: (first) the drift alone, else the previous evaluation's reduction,
// the kick that ends step sr and the drift in one pass; (last) the reduction
// into s.a_new follows.
int launch_gravity_step(nbg_ctx* c, const StateView& s, double dt, StepRef sr, bool first, bool last)
{
    GravStep A;
    A.part = c->grav_part;
    A.perm = c->grav_sort ? c->grav_vals[1] : nullptr;
    A.jchunks = c->grav_chunks;
    A.G = gravity_factor(c);
    A.dt = dt;
    A.dtsq = dt * dt;
    A.step = sr;
    A.save = c->sink_on ? 1 : 0;
    A.box = c->grav_sort ? c->grav_box : nullptr;
    A.ext = c->grav_extent;
    const bool pack = !grav_sorts(c);
    const unsigned grid = (unsigned)(c->npad / 32);
    if (first && !c->grav_perm_valid) A.perm = nullptr;  // (no order yet: it sorts next)
    if (first) {
        if (pack) k_grav_step<false, true><<<grid, 96, 0, c->stream>>>(c->d, s, A);
        else k_grav_step<false, false><<<grid, 96, 0, c->stream>>>(c->d, s, A);
    } else {
        if (pack) k_grav_step<true, true><<<grid, 96, 0, c->stream>>>(c->d, s, A);
        else k_grav_step<true, false><<<grid, 96, 0, c->stream>>>(c->d, s, A);
    }
    NBG_LAUNCH_CHECK(c, "k_grav_step");
    int st;
    if ((st = gravity_order(c, s, pack, !pack))) return st;
    if ((st = gravity_pairs(c))) return st;
    return last ? gravity_reduce(c, s) : NBG_OK;
}

// scratch of the Morton sort (keys, values and cub's temporary storage) and
// the tile boxes
size_t gravity_sort_bytes(int64_t n)
{
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, bytes, (unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                    (int*)nullptr, (int*)nullptr, (int)n, 0, 63);
    return bytes;
}

int gravity_plan_chunks(nbg_ctx* c, int64_t npad) { return plan_gravity(c, npad); }

// ---------------------------------------------------------------------
// generic all-pairs kernel
// ---------------------------------------------------------------------
#define AT 128        // j-tile: FP32 partials are summed in order over one tile
#define AP_WARPS 10   // general form: j-tiles in flight per block, at most (48 KB of stages and sums)
#define AP_SUB 32     // general form: bodies of a tile staged at a time per warp
#define AP_COOP_TILES 16      // a tile per CTA up to 2048 bodies, then a tile per warp (kernel time, us, at 1000 /
                              // 1500 / 2000 / 2500 bodies: ions 8.3 / 12.3 / 15.1 / 19.8 per CTA, 11.3 / 12.5 /
                              // 12.5 / 15.6 per warp; LJ and charges in a cube 11.9 / 16.4 / 21.2 / 28.6 and
                              // 22 / 22 / 21 / 28)
#define AP_CLUSTER_TILES 256  // most tiles whose sums a CTA holds (96 KB)

// A pair that FP32 leaves open, decided (and its difference taken) in the
// reference's FP64 arithmetic.
struct ApExact {
    float3 dr;
    float r2;
    bool lj_in, el_in, range_err;
};

static __device__ __noinline__ ApExact ap_exact(const Dev& d, const double* X, int i, int j, bool lj_pair, bool el_pair)
{
    ApExact o{make_float3(0.f, 0.f, 0.f), 1.0f, false, false, false};
    Dist64 q;
    if (!distance64(X + 3 * (int64_t)i, X + 3 * (int64_t)j, d.bc, d.reps[0], q)) {
        o.range_err = true;
        return o;
    }
    o.lj_in = lj_pair && (q.r2 < d.lj_R2);
    o.el_in = el_pair && (q.r2 < d.el_R2);
    o.dr = make_float3((float)q.x, (float)q.y, (float)q.z);
    o.r2 = (float)q.r2;
    return o;
}

// Bodies j staged per warp in shared memory, one array per field so that two
// neighbouring bodies load as the two halves of a packed operand and four by
// one load. Positions are stored negated (i - j is then an addition).
template <int SUB>
struct __align__(16) ApStage {
    float f[8][SUB];  // -hi x, y, z; charge; -lo x, y, z; flags
    __device__ __forceinline__ void put(int k, const float4& h, const float4& l)
    {
        f[0][k] = -h.x; f[1][k] = -h.y; f[2][k] = -h.z; f[3][k] = h.w;
        f[4][k] = -l.x; f[5][k] = -l.y; f[6][k] = -l.z; f[7][k] = l.w;
    }
    // slots k .. k + 3 (k a multiple of 4) as two packed operands
    __device__ __forceinline__ void four(int c, int k, float2 (&v)[2]) const
    {
        const float4 q = *reinterpret_cast<const float4*>(&f[c][k]);
        v[0] = make_float2(q.x, q.y);
        v[1] = make_float2(q.z, q.w);
    }
};

// the pair constants and body i of a lane, as packed operands
struct ApOwn {
    float2 hx, hy, hz, lx, ly, lz, invL, Lh, Ll;
    float kqi, lj_lo, lj_hi, el_lo, el_hi;
    int flags;
    __device__ __forceinline__ ApOwn(const RepDev& R, const float4& h, const float4& l, float kq)
        : hx(make_float2(h.x, h.x)), hy(make_float2(h.y, h.y)), hz(make_float2(h.z, h.z)), lx(make_float2(l.x, l.x)),
          ly(make_float2(l.y, l.y)), lz(make_float2(l.z, l.z)), invL(make_float2(R.invLf, R.invLf)),
          Lh(make_float2(-R.Lh, -R.Lh)), Ll(make_float2(-R.Ll, -R.Ll)), kqi(kq), lj_lo(R.lj_lo), lj_hi(R.lj_hi),
          el_lo(R.el_lo), el_hi(R.el_hi)
    {
        flags = __float_as_int(l.w);
    }
};

// The forces on i of AP_G bodies j0 .. j0 + AP_G - 1 (staged from slot k on;
// m of them real), in pair_cutoff's arithmetic and classification, two
// bodies per packed instruction. One branch for the group, to the pairs that
// FP32 does not decide: a branch per pair kept a lane's pairs from
// overlapping. Exactly zero for a pair outside both cutoffs, but NaN (the sum
// is then reported) where a difference is not finite.
// CUT: some cutoff is finite. SKIP: the group may hold i itself, its
// molecule, or slots past the last body.
#define AP_G 4
static_assert(AP_G == 4, "a staged load holds four bodies");

template <bool CUBIC, bool HAS_LJ, bool HAS_EL, bool CUT, bool WATER, bool SKIP, int SUB>
__device__ __forceinline__ void ap_pairs(const Dev& d, const ApOwn& o, const ApStage<SUB>& sh, int i, int j0, int k, int m,
                                         const double* X, float (&fx)[AP_G], float (&fy)[AP_G], float (&fz)[AP_G],
                                         bool& range_err)
{
    // an r^2 that is not below infinity takes the branch where a slot may hold
    // anything; and with both potentials, whose forms then keep their
    // registers (12,000 bodies 346 -> 336 us; one potential is 5 % faster without)
    constexpr bool LOST = SKIP || (CUT && HAS_LJ && HAS_EL);
    float2 dx[AP_G / 2], dy[AP_G / 2], dz[AP_G / 2], r2[AP_G / 2], qj[AP_G / 2], fl[AP_G / 2];
    bool lj_in[AP_G], el_in[AP_G], any = false;
    auto at = [](float2* v, int q) -> float& { return (q & 1) ? v[q >> 1].y : v[q >> 1].x; };
    auto pairs = [&](int q, bool& lj_pair, bool& el_pair) {
        const int j = j0 + q;
        const bool skip = SKIP && (q >= m || j == i);
        lj_pair = HAS_LJ && !skip && (!WATER || (o.flags & __float_as_int(at(fl, q)) & AF_LJ) != 0);
        el_pair = HAS_EL && !skip && !(SKIP && WATER && i / 3 == j / 3);
    };
    float2 jx[2], jy[2], jz[2], kx[2], ky[2], kz[2];
    sh.four(0, k, jx);
    sh.four(1, k, jy);
    sh.four(2, k, jz);
    sh.four(4, k, kx);
    sh.four(5, k, ky);
    sh.four(6, k, kz);
    if (HAS_EL) sh.four(3, k, qj);
    if (WATER) sh.four(7, k, fl);
#pragma unroll
    for (int h = 0; h < AP_G / 2; ++h) {
        dx[h] = __fadd2_rn(o.hx, jx[h]);
        dy[h] = __fadd2_rn(o.hy, jy[h]);
        dz[h] = __fadd2_rn(o.hz, jz[h]);
        float2 ex = __fadd2_rn(o.lx, kx[h]);
        float2 ey = __fadd2_rn(o.ly, ky[h]);
        float2 ez = __fadd2_rn(o.lz, kz[h]);
        if (CUBIC) {  // split_diff's image shift
            const float2 magic = make_float2(12582912.0f, 12582912.0f), back = make_float2(-12582912.0f, -12582912.0f);
            const float2 sx = __fadd2_rn(__ffma2_rn(dx[h], o.invL, magic), back);
            const float2 sy = __fadd2_rn(__ffma2_rn(dy[h], o.invL, magic), back);
            const float2 sz = __fadd2_rn(__ffma2_rn(dz[h], o.invL, magic), back);
            dx[h] = __ffma2_rn(sx, o.Lh, dx[h]);
            dy[h] = __ffma2_rn(sy, o.Lh, dy[h]);
            dz[h] = __ffma2_rn(sz, o.Lh, dz[h]);
            ex = __ffma2_rn(sx, o.Ll, ex);
            ey = __ffma2_rn(sy, o.Ll, ey);
            ez = __ffma2_rn(sz, o.Ll, ez);
        }
        dx[h] = __fadd2_rn(dx[h], ex);
        dy[h] = __fadd2_rn(dy[h], ey);
        dz[h] = __fadd2_rn(dz[h], ez);
        r2[h] = __ffma2_rn(dx[h], dx[h], __ffma2_rn(dy[h], dy[h], __fmul2_rn(dz[h], dz[h])));
    }
#pragma unroll
    for (int q = 0; q < AP_G; ++q) {
        bool lj_pair, el_pair;
        pairs(q, lj_pair, el_pair);
        const float r = at(r2, q);
        lj_in[q] = lj_pair && r < (CUT ? o.lj_lo : INFINITY);
        el_in[q] = el_pair && r < (CUT ? o.el_lo : INFINITY);
        if (CUT) any |= (lj_pair && !lj_in[q] && r < o.lj_hi) || (el_pair && !el_in[q] && r < o.el_hi);
        if (LOST) any |= !(r < INFINITY);
    }
    if (any) {
#pragma unroll
        for (int q = 0; q < AP_G; ++q) {
            bool lj_pair, el_pair;
            pairs(q, lj_pair, el_pair);
            const float r = at(r2, q);
            if (CUT && ((lj_pair && !lj_in[q] && r < o.lj_hi) || (el_pair && !el_in[q] && r < o.el_hi))) {
                const ApExact e = ap_exact(d, X, i, j0 + q, lj_pair, el_pair);
                lj_in[q] = e.lj_in;
                el_in[q] = e.el_in;
                at(dx, q) = e.dr.x;
                at(dy, q) = e.dr.y;
                at(dz, q) = e.dr.z;
                at(r2, q) = e.r2;
                range_err |= e.range_err;
            }
            if (LOST && !(at(r2, q) < INFINITY) && !lj_in[q] && !el_in[q]) {
                at(r2, q) = 1.0f;
                if (SKIP && (q >= m || j0 + q == i)) at(dx, q) = at(dy, q) = at(dz, q) = 0.f;
            }
        }
    }
#pragma unroll
    for (int h = 0; h < AP_G / 2; ++h) {
        float2 f = make_float2(0.f, 0.f);
        // (without cutoffs and skipped bodies every pair is in, but for those
        // with an r^2 past FP32's range: their factors are zero by themselves)
        constexpr bool ALL = !CUT && !SKIP && !WATER;
        const bool in0 = lj_in[2 * h] || el_in[2 * h], in1 = lj_in[2 * h + 1] || el_in[2 * h + 1];
        const float2 rr = make_float2(ALL || in0 ? r2[h].x : 1.f, ALL || in1 ? r2[h].y : 1.f);
        if (HAS_LJ) {
            const float2 ri = make_float2(rcp_ftz(rr.x), rcp_ftz(rr.y));
            const float2 s2 = __fmul2_rn(make_float2(d.lj_sig2, d.lj_sig2), ri);
            const float2 s6 = __fmul2_rn(__fmul2_rn(s2, s2), s2);
            const float2 s12 = __fmul2_rn(s6, s6);
            const float2 t = __ffma2_rn(make_float2(2.f, 2.f), s12, make_float2(-s6.x, -s6.y));
            const float2 g = __fmul2_rn(make_float2(d.lj_eps24, d.lj_eps24), __fmul2_rn(t, ri));
            f = make_float2(ALL || lj_in[2 * h] ? g.x : 0.f, ALL || lj_in[2 * h + 1] ? g.y : 0.f);
        }
        if (HAS_EL) {
            const float2 rb = make_float2(rsqrt_ftz(rr.x), rsqrt_ftz(rr.y));
            const float2 t = __ffma2_rn(__fmul2_rn(rb, rb), rb, make_float2(-d.el_krf2, -d.el_krf2));
            const float2 g = __ffma2_rn(__fmul2_rn(make_float2(o.kqi, o.kqi), qj[h]), t, f);
            f = make_float2(ALL || el_in[2 * h] ? g.x : f.x, ALL || el_in[2 * h + 1] ? g.y : f.y);
        }
        const float2 vx = __fmul2_rn(f, dx[h]), vy = __fmul2_rn(f, dy[h]), vz = __fmul2_rn(f, dz[h]);
        fx[2 * h] = vx.x; fx[2 * h + 1] = vx.y;
        fy[2 * h] = vy.x; fy[2 * h + 1] = vy.y;
        fz[2 * h] = vz.x; fz[2 * h + 1] = vz.y;
    }
}

// Whether a tile may hold a body, or a molecule mate, of block b's 32 bodies
// (a molecule can straddle two tiles), or slots past the last body.
__device__ __forceinline__ bool ap_skips(int t, int b, int n, bool water)
{
    const int mine = b * 32 / AT;
    return (t + 1) * AT > n || t == mine || (water && (t == mine - 1 || t == mine + 1));
}

// Both kernels below: every ordered pair of a system off the list path. The
// FP32 sums of a 128-body tile run over its bodies in order and the tiles'
// sums are folded in tile order into a compensated pair, so the result does
// not depend on how the tiles are shared out. They replace one thread per
// body walking every tile, which left all but n / 128 SMs idle and waited
// ~350 cycles per pair (n = 648 water: 230 us per evaluation; 5000 ions:
// 1.3 ms).

// The cutoff potentials under infinite or cubic boundaries: a cluster of C
// CTAs per 32 bodies i (lane = body), CTA r of it taking tiles r, r + C, ..
// and leaving their sums in the first CTA's shared memory, which folds them
// (the others exit: waiting for the fold held their SM's warp slots for half
// of the kernel).
// COOP, for systems of up to AP_COOP_TILES tiles, which are bound by
// latency: the CTA's 8 warps evaluate 16 bodies j each of one tile into
// shared memory, and three warps then add a component each in body order
// (n = 648 water: 11 us against 22 with a tile per warp; 8.2 to 7.7 in a step
// since the cluster's first barrier orders no memory and ends behind the pairs).
// 16 warps of 8 bodies were slower from 1000 bodies on (18.5 us against 14.5).
// Otherwise a warp takes a whole tile and adds as it evaluates (bound by the
// FP32 pipe: 22 instructions a pair and warp for the bare Coulomb force, 10
// of them packed; an evaluation of 4000 ions 23 us, 35 with COOP; of 12000,
// 126 us = 0.35 of the FP32 rate at 23 flop a pair). Three blocks per SM are
// asked for where 80 registers were measured to be better or as good at all
// of these sizes: the bare Coulomb form (5000 ions 35 -> 33 us when it was
// bounded) and LJ under cubic boundaries (7000 bodies 97 -> 88 us, 12000 232
// -> 221). With both potentials the bound is mixed (spills): 2500 bodies
// 28.0 -> 30.9 us, 7000 130 -> 123, 12000 346 -> 298.
#define APC_WARPS 8

template <bool COOP, bool CUBIC, bool HAS_LJ, bool HAS_EL, bool CUT, bool WATER>
__global__ void __launch_bounds__(APC_WARPS * 32, !COOP && (HAS_EL ? !HAS_LJ && !CUT : CUBIC) ? 3 : 0)
    k_allpairs_cut(Dev d, StateView s, int C)
{
    // every CTA of the cluster runs before its shared memory is written to:
    // waited for before the first such write (no data goes with this barrier)
    asm volatile("barrier.cluster.arrive.relaxed.aligned;");
    extern __shared__ float apc_sm[];
    auto cluster = cooperative_groups::this_cluster();
    float* const sums = cluster.map_shared_rank(apc_sm, 0);   // [tiles][3][32], the first CTA's
    constexpr int SUB = COOP ? AT / APC_WARPS : 32;           // bodies staged at a time per warp
    __shared__ ApStage<SUB> stage[APC_WARPS];
    const int W = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b = blockIdx.x / C, rank = blockIdx.x % C;
    const int n = (int)d.n, tiles = (n + AT - 1) / AT;
    const int i = b * 32 + lane;
    const bool active = i < n;
    const int ii = active ? i : 0;
    const float4 hi_i = d.phi[ii], lo_i = d.plo[ii];
    const ApOwn own(d.reps[0], hi_i, lo_i, HAS_EL ? (float)(d.el_k_d * d.charge[ii]) : 0.0f);
    ApStage<SUB>& sh = stage[w];
    bool range_err = false;
    if constexpr (!COOP) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    // the m staged bodies from j0 on; put(k, the AP_G values from slot k on)
    auto eval = [&](auto skip, int j0, int m, auto put) {
#pragma unroll 2
        for (int k = 0; k < SUB; k += AP_G) {
            if (k >= m) break;
            float fx[AP_G], fy[AP_G], fz[AP_G];
            ap_pairs<CUBIC, HAS_LJ, HAS_EL, CUT, WATER, decltype(skip)::value>(d, own, sh, ii, j0 + k, k, m - k, s.x, fx, fy,
                                                                               fz, range_err);
            put(k, fx, fy, fz);
        }
    };
    if constexpr (COOP) {
        float* const val = apc_sm + tiles * 96;               // [3][AT][32]
        for (int t = rank, ti = 0; t < tiles; t += C, ++ti) {
            const int j0 = t * AT + w * SUB, m = min(SUB, n - j0);
            __syncwarp();
            if (lane < m) sh.put(lane, d.phi[j0 + lane], d.plo[j0 + lane]);
            __syncwarp();
            if (ti > 0) __syncthreads();  // the previous tile's values are added
            auto put = [&](int k, const float* fx, const float* fy, const float* fz) {
#pragma unroll
                for (int q = 0; q < AP_G; ++q) {
                    float* v = val + (w * SUB + k + q) * 32 + lane;
                    v[0] = fx[q];
                    v[AT * 32] = fy[q];
                    v[2 * AT * 32] = fz[q];
                }
            };
            if (ap_skips(t, b, n, WATER)) eval(std::true_type{}, j0, m, put);
            else eval(std::false_type{}, j0, m, put);
            __syncthreads();
            if (ti == 0) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
            if (w < 3) {
                const float* v = val + w * AT * 32 + lane;
                const int mt = min(AT, n - t * AT);
                float p = 0.f;
                if (mt == AT) {
#pragma unroll 32
                    for (int k = 0; k < AT; ++k) p = __fadd_rn(p, v[k * 32]);
                } else {
                    for (int k = 0; k < mt; ++k) p = __fadd_rn(p, v[k * 32]);
                }
                sums[(t * 3 + w) * 32 + lane] = p;
            }
        }
    } else {
        for (int ti = w; ti * C + rank < tiles; ti += W) {
            const int t = ti * C + rank, j1 = min(n, (t + 1) * AT);
            const bool skips = ap_skips(t, b, n, WATER);
            float px = 0.f, py = 0.f, pz = 0.f;
            auto put = [&](int, const float* fx, const float* fy, const float* fz) {
#pragma unroll
                for (int q = 0; q < AP_G; ++q) {
                    px = __fadd_rn(px, fx[q]);
                    py = __fadd_rn(py, fy[q]);
                    pz = __fadd_rn(pz, fz[q]);
                }
            };
            // (the next bodies are loaded before the current ones' arithmetic)
            float4 h = hi_i, l = lo_i;
            if (t * AT + lane < j1) {
                h = d.phi[t * AT + lane];
                l = d.plo[t * AT + lane];
            }
            for (int j0 = t * AT; j0 < j1; j0 += SUB) {
                const int m = min(SUB, j1 - j0);
                __syncwarp();
                sh.put(lane, h, l);
                __syncwarp();
                if (j0 + SUB + lane < j1) {
                    h = d.phi[j0 + SUB + lane];
                    l = d.plo[j0 + SUB + lane];
                }
                if (skips) eval(std::true_type{}, j0, m, put);
                else eval(std::false_type{}, j0, m, put);
            }
            sums[(t * 3) * 32 + lane] = px;
            sums[(t * 3 + 1) * 32 + lane] = py;
            sums[(t * 3 + 2) * 32 + lane] = pz;
        }
    }
    if (range_err) status_set(d.status, ST_RANGE);
    // the tiles' sums, in tile order; the other CTAs have written theirs into
    // the first one's shared memory and leave
    cluster.barrier_arrive();
    if (rank != 0) return;
    cluster.barrier_wait();
    for (int c = w; c < 3; c += W) {
        Acc2 a{0.f, 0.f};
        const float* v = apc_sm + c * 32 + lane;
#pragma unroll 8
        for (int t = 0; t < tiles; ++t) a.add(v[t * 96]);
        if (active) {
            const double acc = a.value() * d.inv_mass[i];
            if (!finite64(acc)) status_set(d.status, ST_NONFINITE);
            s.a_new[3 * (int64_t)i + c] = acc;
        }
    }
}

// Every other form, and systems whose tiles' sums do not fit the cluster's
// shared memory: a block owns 32 bodies i and each of its warps a whole tile
// at a time; after each round of tiles their sums are folded.
__global__ void __launch_bounds__(AP_WARPS * 32) k_allpairs(Dev d, StateView s)
{
    constexpr int NC = 9;  // sums: cutoff force, then gravity and dipoles
    extern __shared__ float4 ap_sm[];
    const int W = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int STAGE = 3 * AP_SUB;  // float4 of one warp's stage
    float4* const sh_hi = ap_sm + w * STAGE;
    float4* const sh_lo = sh_hi + AP_SUB;
    float4* const sh_mm = sh_lo + AP_SUB;                                  // dipole, mass
    float* const part = reinterpret_cast<float*>(ap_sm + W * STAGE);       // [2][W][NC][32]
    float* const acc = part + 2 * W * NC * 32;                             // [2][NC][32]: hi, lo
    const int n = (int)d.n;
    const int i = blockIdx.x * 32 + lane;
    const bool active = i < n;
    const int ii = active ? i : 0;
    const RepDev& R = d.reps[0];
    const float4 hi_i = d.phi[ii], lo_i = d.plo[ii];
    const float kqi = (d.pots & NBG_POT_EL) ? (float)(d.el_k_d * d.charge[ii]) : 0.0f;
    const PairK K(R);
    float3 mi = make_float3(0.f, 0.f, 0.f);
    if (d.pots & NBG_POT_MAG)
        mi = make_float3((float)d.dipole[3 * ii], (float)d.dipole[3 * ii + 1], (float)d.dipole[3 * ii + 2]);
    bool range_err = false;
    const bool cutpots = (d.pots & (NBG_POT_LJ | NBG_POT_EL)) != 0;
    for (int k = threadIdx.x; k < 2 * NC * 32; k += blockDim.x) acc[k] = 0.f;
    const int tiles = (n + AT - 1) / AT;
    const int rounds = (tiles + W - 1) / W;
    __syncthreads();
    for (int r = 0; r <= rounds; ++r) {
        // the previous round's partials, folded in tile order (a warp per sum)
        if (r > 0) {
            const float* pp = part + ((r - 1) & 1) * W * NC * 32;
            for (int c = w; c < NC; c += W) {
                Acc2 a{acc[c * 32 + lane], acc[(NC + c) * 32 + lane]};
                const int m = min(W, tiles - (r - 1) * W);
                for (int k = 0; k < m; ++k) a.add(pp[(k * NC + c) * 32 + lane]);
                acc[c * 32 + lane] = a.hi;
                acc[(NC + c) * 32 + lane] = a.lo;
            }
        }
        const int t = r * W + w;
        if (r < rounds && t < tiles) {
            float p[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) p[c] = 0.f;
            const int j1 = min(n, (t + 1) * AT);
            for (int j0 = t * AT; j0 < j1; j0 += AP_SUB) {
                const int m = min(AP_SUB, j1 - j0);
                __syncwarp();
                if (lane < m) {
                    sh_hi[lane] = d.phi[j0 + lane];
                    sh_lo[lane] = d.plo[j0 + lane];
                    float4 q = make_float4(0.f, 0.f, 0.f, (float)d.mass[j0 + lane]);
                    if (d.pots & NBG_POT_MAG) {
                        q.x = (float)d.dipole[3 * (j0 + lane)];
                        q.y = (float)d.dipole[3 * (j0 + lane) + 1];
                        q.z = (float)d.dipole[3 * (j0 + lane) + 2];
                    }
                    sh_mm[lane] = q;
                }
                __syncwarp();
                for (int k = 0; k < m; ++k) {
                    const int jg = j0 + k;
                    if (jg == ii) continue;
                    const float4 hj = sh_hi[k], lj = sh_lo[k];
                    if (cutpots) {
                        PairOut o = pair_cutoff(d, R, K, ii, jg, hi_i, lo_i, hj, lj, kqi, s.x);
                        range_err |= o.range_err;
                        p[0] += o.fx;
                        p[1] += o.fy;
                        p[2] += o.fz;
                    }
                    if (d.pots & (NBG_POT_GRAV | NBG_POT_MAG)) {
                        // plain differences: gravity and dipoles ignore the boundary
                        float3 dr = split_diff(hi_i, lo_i, hj, lj, false, R);
                        float r2 = fmaf(dr.x, dr.x, fmaf(dr.y, dr.y, dr.z * dr.z));
                        float ri = rsqrtf(r2);
                        const float4 mj = sh_mm[k];
                        if (d.pots & NBG_POT_GRAV) {
                            float sg = mj.w * ri * ri * ri;
                            p[3] = fmaf(sg, dr.x, p[3]);
                            p[4] = fmaf(sg, dr.y, p[4]);
                            p[5] = fmaf(sg, dr.z, p[5]);
                        }
                        if (d.pots & NBG_POT_MAG) {
                            // (mi (mj.r) + mj (mi.r) + r (mi.mj) - 5 r (mi.r)(mj.r)) / |r|^4, r unit
                            float3 u = make_float3(dr.x * ri, dr.y * ri, dr.z * ri);
                            float mir = mi.x * u.x + mi.y * u.y + mi.z * u.z;
                            float mjr = mj.x * u.x + mj.y * u.y + mj.z * u.z;
                            float mimj = mi.x * mj.x + mi.y * mj.y + mi.z * mj.z;
                            float inv4 = (ri * ri) * (ri * ri);
                            p[6] += (mi.x * mjr + mj.x * mir + u.x * mimj - 5.0f * u.x * mir * mjr) * inv4;
                            p[7] += (mi.y * mjr + mj.y * mir + u.y * mimj - 5.0f * u.y * mir * mjr) * inv4;
                            p[8] += (mi.z * mjr + mj.z * mir + u.z * mimj - 5.0f * u.z * mir * mjr) * inv4;
                        }
                    }
                }
            }
            float* pw = part + (r & 1) * W * NC * 32 + w * NC * 32;
#pragma unroll
            for (int c = 0; c < NC; ++c) pw[c * 32 + lane] = p[c];
        }
        __syncthreads();
    }
    if (range_err) status_set(d.status, ST_RANGE);
    // a warp per component (lane = body)
    for (int c = w; c < 3; c += W) {
        if (!active) continue;
        auto value = [&](int q) { return (double)acc[q * 32 + lane] + (double)acc[(NC + q) * 32 + lane]; };
        double a = value(c) * d.inv_mass[i];
        if (d.pots & NBG_POT_GRAV) a += -d.G * value(3 + c);
        if (d.pots & NBG_POT_MAG) a += 3.0 * d.mu4pi / d.mass[i] * value(6 + c);
        if (!finite64(a)) status_set(d.status, ST_NONFINITE);
        s.a_new[3 * (int64_t)i + c] = a;
    }
}

typedef void (*allpairs_cut_t)(Dev, StateView, int);

template <bool COOP, bool CUBIC, bool CUT>
static allpairs_cut_t ap_kernel(const Dev& d)
{
    if (d.kind == NBG_SYSTEM_WATER) return k_allpairs_cut<COOP, CUBIC, true, true, CUT, true>;
    if (d.pots == NBG_POT_LJ) return k_allpairs_cut<COOP, CUBIC, true, false, CUT, false>;
    if (d.pots == NBG_POT_EL) return k_allpairs_cut<COOP, CUBIC, false, true, CUT, false>;
    return k_allpairs_cut<COOP, CUBIC, true, true, CUT, false>;
}

template <bool COOP>
static allpairs_cut_t ap_kernel(const Dev& d)
{
    if (d.bc == NBG_BC_CUBIC) return ap_kernel<COOP, true, true>(d);
    const bool finite = ((d.pots & NBG_POT_LJ) && isfinite(d.lj_R2)) || ((d.pots & NBG_POT_EL) && isfinite(d.el_R2));
    return finite ? ap_kernel<COOP, false, true>(d) : ap_kernel<COOP, false, false>(d);
}

int launch_allpairs(nbg_ctx* c, const StateView& s)
{
    const Dev& d = c->d;
    const int64_t tiles = (c->n + AT - 1) / AT, blocks = (c->n + 31) / 32;
    const uint32_t cut = d.pots & (NBG_POT_LJ | NBG_POT_EL);
    const int C = (int)std::min<int64_t>(tiles, 8);  // CTAs per cluster (8: the portable size)
    const int64_t per = (tiles + C - 1) / C;         // tiles of a CTA
    prof_begin(c);
    if (d.pots == cut && cut != 0 && d.bc != NBG_BC_PERIODIC && tiles <= AP_CLUSTER_TILES) {
        const bool coop = tiles <= AP_COOP_TILES;
        const allpairs_cut_t k = coop ? ap_kernel<true>(d) : ap_kernel<false>(d);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(blocks * C));
        // (a tile per warp: equal rounds of at most APC_WARPS tiles)
        const int64_t rounds = (per + APC_WARPS - 1) / APC_WARPS;
        cfg.blockDim = dim3((unsigned)(32 * (coop ? APC_WARPS : (per + rounds - 1) / rounds)));
        cfg.dynamicSmemBytes = sizeof(float) * 96 * (size_t)(tiles + (coop ? AT : 0));
        cfg.stream = c->stream;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)C;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(float) * 96 * AP_CLUSTER_TILES);
        if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, k, d, s, C);
        if (e != cudaSuccess) return cuda_fail(c, e, "k_allpairs_cut");
    } else {
        // warps per block: the tiles in equal rounds of at most AP_WARPS
        const int64_t rounds = (tiles + AP_WARPS - 1) / AP_WARPS;
        const int W = (int)((tiles + rounds - 1) / rounds);
        const size_t smem = sizeof(float4) * (size_t)W * 3 * AP_SUB + sizeof(float) * 32 * 9 * (2 * (size_t)W + 2);
        k_allpairs<<<(unsigned)blocks, 32 * W, smem, c->stream>>>(d, s);
    }
    prof_end(c);
    NBG_LAUNCH_CHECK(c, "k_allpairs");
    return NBG_OK;
}

// ---------------------------------------------------------------------
// Verlet-list force kernels
// ---------------------------------------------------------------------
// Thread per atom over a column-major list (coalesced across the atoms of a
// warp): for large systems, where every SM has thousands of atoms.
__global__ void __launch_bounds__(128) k_force_list(Dev d, StateView s)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < d.n; i += (int64_t)gridDim.x * blockDim.x) {
        const RepDev& R = d.reps[d.rep_of[i]];
        const PairK K(R);
        const float4 hi_i = d.phi[i], lo_i = d.plo[i];
        const float kqi = (d.pots & NBG_POT_EL) ? (float)(d.el_k_d * d.charge[i]) : 0.0f;
        const int cnt = d.nbr_count[i];
        Acc2 fx{0.f, 0.f}, fy{0.f, 0.f}, fz{0.f, 0.f};
        float px = 0.f, py = 0.f, pz = 0.f;
        bool range_err = false;
        const int* nl = d.nbr + i * d.nbr_istride;
        // the next neighbour's index and split position are loaded one entry
        // ahead, so that their gathers overlap this pair's arithmetic
        int jn = 0;
        float4 hn = make_float4(0.f, 0.f, 0.f, 0.f), ln = hn;
        if (cnt > 0) {
            jn = dbg_index(__ldg(nl), d.n, (int)i, d.status);
            hn = __ldg(&d.phi[jn]);
            ln = __ldg(&d.plo[jn]);
        }
        for (int k = 0; k < cnt; ++k) {
            const int j = jn;
            const float4 hj = hn, lj = ln;
            if (k + 1 < cnt) {
                jn = dbg_index(__ldg(nl + (int64_t)(k + 1) * d.nbr_kstride), d.n, (int)i, d.status);
                hn = __ldg(&d.phi[jn]);
                ln = __ldg(&d.plo[jn]);
            }
            PairOut o = pair_cutoff(d, R, K, i, j, hi_i, lo_i, hj, lj, kqi, s.x);
            range_err |= o.range_err;
            px += o.fx;
            py += o.fy;
            pz += o.fz;
            if ((k & 31) == 31) {
                fx.add(px); fy.add(py); fz.add(pz);
                px = py = pz = 0.f;
            }
        }
        fx.add(px); fy.add(py); fz.add(pz);
        if (range_err) status_set(d.status, ST_RANGE);
        const double im = d.inv_mass[i];
        double a0 = fx.value() * im, a1 = fy.value() * im, a2 = fz.value() * im;
        if (!finite64(a0) || !finite64(a1) || !finite64(a2)) status_set(d.status, ST_NONFINITE);
        s.a_new[3 * i] = a0;
        s.a_new[3 * i + 1] = a1;
        s.a_new[3 * i + 2] = a2;
    }
}

// LPA lanes per atom over a row-major list: the group reads its atom's
// entries coalesced, each lane keeps an FP32 partial of every LPA-th entry,
// and the partials are joined by a compensated FP32 xor butterfly of shuffles
// (a fixed order: deterministic); one FP64 multiply by 1/m per component
// gives the acceleration. For small systems, where one atom per thread
// leaves the GPU waiting on memory latency.
template <int LPA>
__global__ void __launch_bounds__(256) k_force_list_lanes(Dev d, StateView s)
{
    // one atom per group of LPA lanes; groups past n keep running (with no
    // entries) so that every lane of the warp takes part in the shuffles
    const int lane = threadIdx.x % LPA;
    const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / LPA;
    const bool active = i < d.n;
    const int64_t ia = active ? i : 0;
    const RepDev& R = d.reps[d.rep_of[ia]];
    const float4 hi_i = d.phi[ia], lo_i = d.plo[ia];
    const float kqi = (d.pots & NBG_POT_EL) ? (float)(d.el_k_d * d.charge[ia]) : 0.0f;
    const int cnt = active ? d.nbr_count[ia] : 0;
    float px = 0.f, py = 0.f, pz = 0.f;
    bool range_err = false;
    const int* nl = d.nbr + ia * d.nbr_istride;
    // the pair constants in registers pay off for the short lists of 4-lane
    // groups (LJ ensembles); longer lists keep fewer registers (more warps)
    auto pair_loop = [&](const auto& K) {
        for (int k = lane; k < cnt; k += LPA) {
            int j = dbg_index(__ldg(nl + k), d.n, (int)ia, d.status);
            float4 hj = __ldg(&d.phi[j]), lj = __ldg(&d.plo[j]);
            PairOut o = pair_cutoff(d, R, K, ia, j, hi_i, lo_i, hj, lj, kqi, s.x);
            range_err |= o.range_err;
            px += o.fx;
            py += o.fy;
            pz += o.fz;
        }
    };
    if constexpr (LPA <= 4) pair_loop(PairK(R));
    else pair_loop(R);
    const LaneSum f = lane_sums3<LPA>(px, py, pz, lane);
    if (range_err) status_set(d.status, ST_RANGE);
    if (active && f.writer) {
        const double acc = (widen(f.h) + widen(f.e)) * d.inv_mass[i];
        if (!finite64(acc)) status_set(d.status, ST_NONFINITE);
        s.a_new[3 * i + f.comp] = acc;
    }
}

int launch_force_list(nbg_ctx* c, const StateView& s)
{
    if (c->fx_ready) return launch_force_fx(c, s);
    const int lpa = c->list_lpa;
    prof_begin(c);
    if (lpa <= 1) {
        k_force_list<<<grid_for(c->n, 128), 128, 0, c->stream>>>(c->d, s);
    } else {
        const int per_block = 256 / lpa;  // one atom per group, whole groups per block
        int grid = (int)((c->n + per_block - 1) / per_block);
        if (lpa == 4) k_force_list_lanes<4><<<grid, 256, 0, c->stream>>>(c->d, s);
        else if (lpa == 8) k_force_list_lanes<8><<<grid, 256, 0, c->stream>>>(c->d, s);
        else if (lpa == 16) k_force_list_lanes<16><<<grid, 256, 0, c->stream>>>(c->d, s);
        else k_force_list_lanes<32><<<grid, 256, 0, c->stream>>>(c->d, s);
    }
    prof_end(c);
    NBG_LAUNCH_CHECK(c, "k_force_list");
    return NBG_OK;
}

// ---------------------------------------------------------------------
// SPC/Fw bonded terms (FP64), one thread per molecule (O, H1, H2)
// ---------------------------------------------------------------------
// Bonds and angle of one molecule. The intramolecular differences are taken
// in FP64 from the unwrapped positions and rounded once to FP32 (relative
// error 2^-24); the terms themselves are FP32, like the pair forces (the bond
// stretch r - rOH and the angle offset then carry ~1e-6 relative error). The
// accelerations are added to a_new in FP64.
__global__ void k_bonded(Dev d, StateView s)
{
    int64_t nm = d.n / 3;
    const float rOH = (float)d.rOH, kb = (float)d.kbond, ka = (float)d.kangle, a0 = (float)d.aHOH;
    for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m < nm; m += (int64_t)gridDim.x * blockDim.x) {
        int64_t o = 3 * m, h1 = o + 1, h2 = o + 2;
        const double* X = s.x;
        float r1[3], r2[3];  // H1 - O, H2 - O
        for (int k = 0; k < 3; ++k) {
            r1[k] = (float)(X[3 * h1 + k] - X[3 * o + k]);
            r2[k] = (float)(X[3 * h2 + k] - X[3 * o + k]);
        }
        float fO[3], f1[3], f2[3];
        bonded_forces(r1, r2, rOH, kb, ka, a0, fO, f1, f2);
        const double iO = d.inv_mass[o], iH1 = d.inv_mass[h1], iH2 = d.inv_mass[h2];
        for (int k = 0; k < 3; ++k) {
            s.a_new[3 * o + k] = fma(widen(fO[k]), iO, s.a_new[3 * o + k]);
            s.a_new[3 * h1 + k] = fma(widen(f1[k]), iH1, s.a_new[3 * h1 + k]);
            s.a_new[3 * h2 + k] = fma(widen(f2[k]), iH2, s.a_new[3 * h2 + k]);
        }
    }
}

int launch_bonded(nbg_ctx* c, const StateView& s)
{
    k_bonded<<<grid_for(c->n / 3, 64), 64, 0, c->stream>>>(c->d, s);
    NBG_LAUNCH_CHECK(c, "k_bonded");
    return NBG_OK;
}

// ---------------------------------------------------------------------
// Raw launcher of the gravity kernel (default form) and its chunk reduction
// on caller-provided buffers, for entry points that own their scratch.
// ---------------------------------------------------------------------
int gravity_raw_chunks(int device, int64_t npad, int max_chunks)
{
    int sms = 0, occ = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_gravity<false, 2, true, false>, GB, 0);
    if (sms < 1) sms = 1;
    if (occ < 1) occ = 1;
    const double slots = (double)sms * occ;
    const int64_t ib = npad / (2 * GB);
    const int64_t ntile = npad / GB;
    int best = 1;
    double best_eff = -1.0;
    for (int J = 1; J <= max_chunks && J <= ntile; ++J) {
        double waves = (double)(ib * J) / slots;
        double eff = waves / ceil(waves) * ((double)ntile / J) / (double)((ntile + J - 1) / J);
        if (eff > best_eff + 0.005) {
            best_eff = eff;
            best = J;
        }
    }
    return best;
}

cudaError_t gravity_raw_launch(const float4* phi, const float4* plo, int64_t n, int64_t npad, int jchunks,
                               double* part, double G, double* a, unsigned* status, cudaStream_t stream)
{
    int64_t units = (npad / (2 * GB)) * jchunks;
    k_gravity<false, 2, true, false><<<(unsigned)units, GB, 0, stream>>>(phi, plo, n, npad, jchunks, part, nullptr, 0.f);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_gravity_reduce<<<grid_for(3 * n, 256), 256, 0, stream>>>(part, n, jchunks, G, a, status, nullptr);
    return cudaGetLastError();
}
