// k_cluster.cu - velocity Verlet for small systems (up to 2048 atoms) as one
// persistent launch over a thread-block cluster.
//
// A step of a small system is a handful of microsecond kernels, so launches,
// not arithmetic, set its pace. Here the cluster's CTAs (up to 16 SMs) run
// many steps in one launch:
//   - CTA r owns atoms [r per, (r+1) per); its threads drift them (FP64, the
//     reference's velocity-Verlet arithmetic) and write the new positions, split
//     and FP64, to global buffers of the step's parity; a thread per peer then
//     arrives (release) at that CTA's mbarrier of the parity, after setting
//     its rebuild flag where an atom moved too far;
//   - a CTA waits (bounded) for its own mbarrier alone, no barrier of the whole
//     cluster, and reads all split positions through L2 into shared memory.
//     (Sent from SM to SM, as bulk copies into the peers' shared memory, the
//     30 KB per CTA and step at 1000 atoms took 3000 cycles, 10 bytes per
//     cycle, whether one thread issued the copies or seven warps did. Through
//     L2 it is about the same, but the threads' work between runs faster.)
//     With two parity buffers the arrivals order
//     their reuse too: a CTA writes step s+2 after it has received every
//     peer's step s+1, which a peer sends when its threads are done with step s;
//   - each CTA keeps the Verlet lists of its own atoms in shared memory,
//     rebuilt from the shared positions (all atoms scanned, the FP32 superset
//     test of the list builders) when any atom moved more than skin/2 since
//     the last build and every rebuild_every steps; a launch that built
//     them stores them at its end (the steps since the build always), and
//     the next one starts from them unless the host invalidated them (a new
//     state), else it builds first;
//   - at its start a launch writes x, v, a_old of its atoms to the backup,
//     from which the host undoes a launch that timed out or overflowed;
//   - LPA lanes per atom evaluate the pairs (cl_pair: the exact pair set;
//     the ambiguous ones read FP64 positions, which the drift also writes to
//     a global copy of the step's parity, through L2) and join their
//     partials (compensated FP32) into shared memory; the atom's owner thread,
//     which keeps its x, v, a in registers for the whole launch, kicks the
//     velocity at the start of the next step.
// Every thread of every CTA passes the same cluster barriers (no early exit).
//
// Cycles per step and CTA at 1000 LJ atoms (63 per CTA, 16 lanes each), before
// and after the cluster barrier of every step gave way to the arrivals, the
// constants came from the constant bank, the pair lost its branches and the
// build its counts per test: kick and drift 7100 and 3700 (FP64, two warps per
// SM sub-partition), exchange 5100 and 3900 (three L2 round trips), list
// build, over its ~9 steps, 4300 and 2150, forces 7200 and 5000; 200 steps
// 2.24 ms and 1.58.
//
// The same kernel with ACCEL evaluates the right-hand side alone (nbg_accel):
// the positions come from src (pinned host memory read over the CPU-GPU
// link, or device memory), one step of the loop without drift or kick runs
// (exchange, displacement check, list build when needed, forces), and the
// accelerations go to dst; the lists it keeps are its own, built for earlier
// calls' positions, and the resident state is not touched.
#include <algorithm>

#include <cooperative_groups.h>

#include "nbg_internal.cuh"

namespace cg = cooperative_groups;

#define CL_THREADS 1024
#define CL_MAX 16

// mbarrier helpers (shared-memory addresses as 32-bit
// shared-window offsets; remote ones from mapa)
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned cluster_addr(unsigned a, int rank)
{
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}

__device__ __forceinline__ void mbar_init(unsigned a, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned a, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    return ok != 0;
}

// arrival on another CTA's mbarrier: this thread's writes, and those it has
// seen through a block barrier, are visible to who waits for the phase
__device__ __forceinline__ void mbar_arrive_peer(unsigned mbar_cluster)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(mbar_cluster) : "memory");
}

// block barrier of the first `threads` threads, with an OR
__device__ __forceinline__ bool owners_sync_or(unsigned threads, bool v)
{
    unsigned r;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.cta.red.or.pred q, 1, %2, p;\n"
        " selp.u32 %0, 1, 0, q;\n}"
        : "=r"(r)
        : "r"((unsigned)v), "r"(threads)
        : "memory");
    return r != 0;
}

#define CL_WAIT_TRIES (1u << 16)

__device__ __forceinline__ bool mbar_wait(unsigned a, unsigned parity)
{
    unsigned tries = 0;
    while (!mbar_try_wait(a, parity))
        if (++tries >= CL_WAIT_TRIES) return false;
    return true;
}

// The force on i of listed atom j, in pair_cutoff's arithmetic and
// classification without its branches (only a pair that FP32 does not decide
// takes one), added to p. A potential system: every listed pair has both
// potentials of POTS.
template <int POTS>
__device__ __forceinline__ void cl_pair(const Dev& d, const RepDev& R, int i, int j, const float4& hi_i, const float4& lo_i,
                                        const float4& hi_j, const float4& lo_j, float kqi, const double* X, float (&p)[3],
                                        bool& range_err)
{
    constexpr bool LJ = (POTS & NBG_POT_LJ) != 0, EL = (POTS & NBG_POT_EL) != 0;
    float3 dr = split_diff(hi_i, lo_i, hi_j, lo_j, true, R);
    float r2 = __fmaf_rn(dr.x, dr.x, __fmaf_rn(dr.y, dr.y, __fmul_rn(dr.z, dr.z)));
    bool lj = LJ && r2 < R.lj_lo, el = EL && r2 < R.el_lo;
    if ((LJ && !lj && r2 < R.lj_hi) || (EL && !el && r2 < R.el_hi)) {
        Dist64 q;
        if (!distance64<true>(X + 3 * i, X + 3 * j, NBG_BC_CUBIC, R, q)) {
            range_err = true;
            return;
        }
        lj = LJ && q.r2 < d.lj_R2;
        el = EL && q.r2 < d.el_R2;
        dr = make_float3((float)q.x, (float)q.y, (float)q.z);
        r2 = (float)q.r2;
    }
    const float rr = lj || el ? r2 : 1.0f;
    float f = 0.0f;
    if (LJ) {
        const float ri = rcp_ftz(rr);
        const float s2 = __fmul_rn(d.lj_sig2, ri);
        const float s6 = __fmul_rn(__fmul_rn(s2, s2), s2);
        const float s12 = __fmul_rn(s6, s6);
        const float g = __fmul_rn(d.lj_eps24, __fmul_rn(__fmaf_rn(2.0f, s12, -s6), ri));
        f = lj ? g : 0.0f;
    }
    if (EL) {
        const float rb = rsqrt_ftz(rr);
        const float t = __fmaf_rn(__fmul_rn(rb, rb), rb, -d.el_krf2);
        const float g = __fmaf_rn(__fmul_rn(kqi, hi_j.w), t, f);
        f = el ? g : f;
    }
    p[0] = __fadd_rn(p[0], __fmul_rn(f, dr.x));
    p[1] = __fadd_rn(p[1], __fmul_rn(f, dr.y));
    p[2] = __fadd_rn(p[2], __fmul_rn(f, dr.z));
}

// Shared memory (dynamic): split positions [hi, lo][n] (float4), the
// own atoms' positions at the last list build [per][3] (double, padded to a 16-byte end), their lists
// [per][cap], counts [per] (int) and force partials [per][6] (float: h, e per
// component).
static size_t cluster_smem(int n, int per, int cap)
{
    return sizeof(float4) * 2 * (size_t)n + sizeof(double) * (3 * (size_t)per + ((3 * per) & 1)) +
           sizeof(int) * ((size_t)per * cap + per) + sizeof(float) * 6 * (size_t)per;
}

// split_component under cubic boundaries, given the box image img (the floor of
// p / L) of the last step: while the wrapped position keeps clear of both
// faces the image is the same and the floor (with its product a sixth of a
// step's FP64 time per component) is not taken. Images too large for p / L to be
// that exact are not kept (NaN).
__device__ __forceinline__ void split_kept_image(const RepDev& R, double p, double& img, float& h, float& l)
{
    double w = fma(-R.L, img, p);
    // L 2^-20 <= w < L (1 - 2^-21), by the high words (positive doubles order like integers)
    const int hL = __double2hiint(R.L), lo = hL - (20 << 20);
    if ((unsigned)(__double2hiint(w) - lo) >= (unsigned)(hL - 1 - lo)) {
        img = floor(p * R.invL);
        w = fma(-R.L, img, p);
        if (negative64(w)) w += R.L;
        if (__double_as_longlong(w) >= __double_as_longlong(R.L)) w -= R.L;
        if (!(fabs(img) < 1048576.0)) img = __longlong_as_double(0x7ff8000000000000ll);
    }
    grid_split(R, w, h, l);
}

// R: the replica's constants as a kernel argument (operands from the constant
// bank; through d.reps every use was a load again, as the kernel stores).
template <int LPA, bool ACCEL, int POTS>
__global__ void __launch_bounds__(CL_THREADS, 1) k_cluster_vv(Dev d, const __grid_constant__ RepDev R, StateView s, double* xb,
                                                              float4* xs, double dt, int nsteps,
                                                              int rebuild_every, int per, int cap, int* lst_g,
                                                              int* cnt_g, double* xref_g, int* since_g, int reuse,
                                                              int64_t step0, int save, int drop_step,
                                                              double* __restrict__ bk,
                                                              const double* __restrict__ src, double* __restrict__ dst)
{
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int C = (int)cl.num_blocks();
    const int n = (int)d.n;
    extern __shared__ float4 cl_pos[];
    float4* const ph = cl_pos;
    float4* const pl = ph + n;
    double* xref_s = reinterpret_cast<double*>(cl_pos + 2 * (size_t)n);
    int* lst = reinterpret_cast<int*>(xref_s + 3 * (size_t)per + ((3 * per) & 1));  // 16-byte aligned
    int* cnt = lst + (size_t)per * cap;
    float* fsum = reinterpret_cast<float*>(cnt + per);
    __shared__ unsigned flag[2];  // rebuild requests of the step of each parity
    __shared__ __align__(8) unsigned long long mbar[2];  // the CTAs' positions of each parity are written
    const int tid = threadIdx.x;
    const int a0 = rank * per;
    const int na = max(0, min(n - a0, per));
    const int g = tid / LPA, lane = tid % LPA;  // lane group g <-> own atom a0 + g
    const double dtsq = dt * dt;
    const float magic = 12582912.0f;  // 1.5 * 2^23: rint by addition

    // component k of own atom ko keeps its state in the registers of one
    // thread for the whole launch: 10 atoms a warp, lane 3 a + k (a thread
    // per atom had the three components' FP64 in one chain on two warps)
    const int k = (tid & 31) % 3;
    const int ko = (tid >> 5) * 10 + (tid & 31) / 3;
    const bool owner = (tid & 31) < 30 && ko < na;
    const int owners = (per + 9) / 10 * 32;  // threads of the warps that own atoms
    const int io = owner ? a0 + ko : 0;
    const size_t eo = 3 * (size_t)io + k;
    double x = owner ? (ACCEL ? src[eo] : s.x[eo]) : 0.0;
    double v = owner && !ACCEL ? s.v[eo] : 0.0;
    double a = owner && !ACCEL ? s.a_old[eo] : 0.0;
    const double im_o = owner ? d.inv_mass[io] : 0.0;
    if (owner && !ACCEL) {
        // the backup of the launch's start (x, v, a_old segments of 3 cols):
        // a timed-out or overflowed launch is undone from it
        const size_t seg = 3 * (size_t)d.cols;
        bk[eo] = x;
        bk[seg + eo] = v;
        bk[2 * seg + eo] = a;
    }

    // the static w parts (charge, atom flags) of the own atoms in both parities
    for (int t = tid; t < 4 * na; t += CL_THREADS) {
        const int j = a0 + (t >> 2);
        xs[(size_t)(t & 3) * n + j].w = (t & 1) ? d.plo[j].w : d.phi[j].w;
    }
    int since = 0;
    bool built = false;  // a list build ran in this launch (the same in every CTA)
    if (reuse) {
        // the lists, their reference positions and the steps since their
        // build, as the previous launch left them
        // (cap is a multiple of 4: whole 16-byte rows, several loads in flight per thread)
        const int4* src4 = reinterpret_cast<const int4*>(lst_g + (size_t)rank * per * cap);
        int4* dst4 = reinterpret_cast<int4*>(lst);
#pragma unroll 4
        for (int t = tid; t < na * cap / 4; t += CL_THREADS) dst4[t] = src4[t];
        for (int t = tid; t < na; t += CL_THREADS) cnt[t] = cnt_g[(size_t)rank * per + t];
        for (int t = tid; t < 3 * na; t += CL_THREADS) xref_s[t] = xref_g[3 * (size_t)a0 + t];
        since = *since_g;
    }
    if (tid < 2) flag[tid] = 0u;
    if (tid == 0) {
        mbar_init(smem_addr(&mbar[0]), C);  // an arrival per CTA
        mbar_init(smem_addr(&mbar[1]), C);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // every CTA of the cluster is running (and initialised) before any
    // remote shared-memory access
    cl.sync();

    // the frame sink (trajectory saving): state of time index step0 + st;
    // its other fields are read at a save point, `unsaved` steps ahead
    const int64_t sk_every = save && owner ? d.sink->every : 0;
    const int64_t sk_t0 = save && owner ? d.sink->t0 : 0;
    int64_t unsaved = 0;
    if (sk_every > 0) {
        const int64_t over = (step0 - sk_t0) % sk_every;
        unsaved = over < 0 ? -over : sk_every - over;
    }
    // the FP32 sum of squares of a displacement below this is one below
    // (skin/2)^2 in FP64 (the FP32 sum is within 5e-7 of it)
    const float still2 = d.skin_half2 > 1e-30 ? (float)d.skin_half2 * (1.0f - 4e-6f) : 0.0f;
    double img = __longlong_as_double(0x7ff8000000000000ll);  // the component's box image (not known)

    for (int st = 0; st <= nsteps; ++st) {
        // kick of the previous step with the forces its groups left in fsum
        if constexpr (ACCEL) {
            if (owner && st > 0) {
                // the right-hand side: the acceleration of the source positions
                const double an = (widen(fsum[6 * ko + 2 * k]) + widen(fsum[6 * ko + 2 * k + 1])) * im_o;
                if (!finite64(an)) status_set(d.status, ST_NONFINITE);
                dst[eo] = an;
            }
        } else if (owner && st > 0) {
            const double an = (widen(fsum[6 * ko + 2 * k]) + widen(fsum[6 * ko + 2 * k + 1])) * im_o;
            if (!finite64(an)) status_set(d.status, ST_NONFINITE);
            v = kick1(v, a, an, dt);
            a = an;
            if (sk_every > 0 && --unsaved == 0) {
                unsaved = sk_every;
                const FrameSink* sk = d.sink;
                const int64_t slot = (step0 + st - sk_t0) / sk_every - sk->first;
                if (slot >= 0 && slot < sk->cap) {
                    const size_t o = (size_t)slot * 3 * d.cols + eo;
                    sk->x[o] = x;
                    sk->v[o] = v;
                }
            }
        }
        if (st == nsteps) break;  // uniform: every thread leaves after the last kick
        const int par = st & 1;
        float4* const P = xs + (size_t)(2 * par) * n;  // split positions of this step
        double* X = xb + (size_t)par * 3 * n;  // FP64 positions of this step
        const unsigned mb = smem_addr(&mbar[par]);
        // drift, split and displacement check of the own atoms
        if (tid < owners) {
            double dk = 0.0;
            if (owner) {
                if (!ACCEL) x = drift1(x, v, a, dt, dtsq);
                X[eo] = x;
                float h, l;
                split_kept_image(R, x, img, h, l);
                reinterpret_cast<float*>(P + io)[k] = h;
                reinterpret_cast<float*>(P + n + io)[k] = l;
                // (a launch that does not reuse lists builds at step 0, which
                // sets xref_s)
                dk = x - xref_s[3 * ko + k];
            }
            const float fk = (float)dk, fk2 = fk * fk;
            const float f2 = fk2 + __shfl_down_sync(0xffffffffu, fk2, 1) + __shfl_down_sync(0xffffffffu, fk2, 2);
            bool moved = owner && k == 0 && (st > 0 || reuse) && !(f2 < still2);
            if (__any_sync(0xffffffffu, moved)) {
                const double dy = __shfl_down_sync(0xffffffffu, dk, 1), dz = __shfl_down_sync(0xffffffffu, dk, 2);
                moved = moved && !(dk * dk + dy * dy + dz * dz <= d.skin_half2);
            }
            // every thread has read the last step's flag; peers write it again
            // only after this step's arrivals
            if (tid == 0) flag[par ^ 1] = 0u;
            const bool any_moved = owners_sync_or((unsigned)owners, moved);
            // (drop_step: a host-set test of the timeout path; no CTA arrives for
            // that step, so every wait runs out)
            if (tid < C && st != drop_step) {
                if (any_moved) *cl.map_shared_rank(&flag[par], tid) = 1u;
                mbar_arrive_peer(cluster_addr(mb, tid));
            }
        }
        // all positions of this step (the k-th use of mbar[par] completes phase
        // k). A wait that ran out ends this CTA's loop and, as it arrives for
        // no further step, the others' at their next wait
        const bool ok = mbar_wait(mb, (unsigned)((st >> 1) & 1));
        if (ok) {
#pragma unroll 2
            for (int t = tid; t < 2 * n; t += CL_THREADS) cl_pos[t] = __ldcg(P + t);
        }
        if (__syncthreads_or(ok ? 0 : 1)) {
            if (tid == 0) status_set(d.status, ST_TIMEOUT);
            break;
        }
        const bool build = (st == 0 && !reuse) || *(volatile unsigned*)&flag[par] != 0u ||
                           (rebuild_every > 0 && since >= rebuild_every);
        if (build) {
            // lists of the own atoms, entries in j order: a warp tests 32 atoms j
            // at a time against the atoms of its groups, 1024 in a row, and
            // lane t keeps the t-th mask of hits; the masks' entries are then
            // placed by a prefix sum over the lanes (a count per mask and test
            // was a third of the build)
            constexpr int A = 32 / LPA;
            const int ga = (tid >> 5) * A, ln = tid & 31;
            if (ga < na) {
                float hx[A], hy[A], hz[A];
                int c0[A];
#pragma unroll
                for (int q = 0; q < A; ++q) {
                    const float4 h = ph[a0 + min(ga + q, na - 1)];
                    hx[q] = h.x;
                    hy[q] = h.y;
                    hz[q] = h.z;
                    c0[q] = 0;
                }
                for (int j0 = 0; j0 < n; j0 += 1024) {
                    unsigned hits[A];
#pragma unroll
                    for (int q = 0; q < A; ++q) hits[q] = 0u;
                    const int tests = min(32, (n - j0 + 31) >> 5);
#pragma unroll 2
                    for (int t = 0; t < tests; ++t) {
                        const float4 hj = ph[min(j0 + t * 32 + ln, n - 1)];
#pragma unroll
                        for (int q = 0; q < A; ++q) {
                            float dx = hj.x - hx[q], dy = hj.y - hy[q], dz = hj.z - hz[q];
                            dx = __fmaf_rn(-__fsub_rn(__fmaf_rn(dx, R.invLf, magic), magic), R.Lh, dx);
                            dy = __fmaf_rn(-__fsub_rn(__fmaf_rn(dy, R.invLf, magic), magic), R.Lh, dy);
                            dz = __fmaf_rn(-__fsub_rn(__fmaf_rn(dz, R.invLf, magic), magic), R.Lh, dz);
                            const unsigned m = __ballot_sync(0xffffffffu, dx * dx + dy * dy + dz * dz < R.rl2);
                            if (ln == t) hits[q] = m;
                        }
                    }
                    const int jl = j0 + ln * 32;  // the first atom of this lane's masks
#pragma unroll
                    for (int q = 0; q < A; ++q) {
                        unsigned m = hits[q];
                        const int self = a0 + ga + q - jl, left = n - jl;
                        if (self >= 0 && self < 32) m &= ~(1u << self);
                        if (left < 32) m &= left > 0 ? (1u << left) - 1u : 0u;
                        int sum = __popc(m);
                        const int own = sum;
#pragma unroll
                        for (int o = 1; o < 32; o *= 2) {
                            const int up = __shfl_up_sync(0xffffffffu, sum, o);
                            if (ln >= o) sum += up;
                        }
                        int at = c0[q] + sum - own;
                        if (ga + q < na) {
                            for (; m != 0u && at < cap; m &= m - 1u, ++at) lst[(ga + q) * cap + at] = jl + __ffs(m) - 1;
                        }
                        c0[q] += __shfl_sync(0xffffffffu, sum, 31);
                    }
                }
#pragma unroll
                for (int q = 0; q < A; ++q) {
                    if (ln == 0 && ga + q < na) {
                        if (c0[q] > cap) {
                            status_set(d.status, ST_NBR_OVERFLOW);
                            c0[q] = cap;
                        }
                        cnt[ga + q] = c0[q];
                    }
                }
            }
            if (owner) xref_s[3 * ko + k] = x;
            since = 0;
            built = true;
            __syncthreads();
        }
        ++since;
        // forces of the own atoms: FP32 partials joined over the group, left
        // in fsum for the owner's kick
        {
            const bool active = g < na;
            const int i = active ? a0 + g : 0;
            const float4 hi_i = ph[i], lo_i = pl[i];
            const float kqi = (POTS & NBG_POT_EL) ? (float)(d.el_k_d * d.charge[i]) : 0.0f;
            const int c = active ? cnt[g] : 0;
            float p[3] = {0.f, 0.f, 0.f};
            bool range_err = false;
#pragma unroll 2
            for (int k = lane; k < c; k += LPA) {
                const int j = dbg_index(lst[g * cap + k], d.n, i, d.status);
                cl_pair<POTS>(d, R, i, j, hi_i, lo_i, ph[j], pl[j], kqi, X, p, range_err);
            }
            const LaneSum f = lane_sums3<LPA>(p[0], p[1], p[2], lane);
            if (range_err) status_set(d.status, ST_RANGE);
            if (active && f.writer) {
                fsum[6 * g + 2 * f.comp] = f.h;
                fsum[6 * g + 2 * f.comp + 1] = f.e;
            }
        }
        // the next kick and drift touch only this CTA's own atoms: a block
        // barrier, no cluster barrier
        __syncthreads();
    }
    // all flags and arrivals are in: no CTA's shared memory is written to any more
    cl.sync();
    if (owner && !ACCEL) {
        s.x[eo] = x;
        s.v[eo] = v;
        s.a_old[eo] = a;
        d.xref[eo] = xref_s[3 * ko + k];
    }
    // the lists for the next launch, if this one built them (with their own
    // reference positions: d.xref also serves the global lists, which other
    // calls rebuild)
    if (built) {
        for (int t = tid; t < 3 * na; t += CL_THREADS) xref_g[3 * (size_t)a0 + t] = xref_s[t];
        int4* dst4 = reinterpret_cast<int4*>(lst_g + (size_t)rank * per * cap);
        const int4* src4 = reinterpret_cast<const int4*>(lst);
#pragma unroll 4
        for (int t = tid; t < na * cap / 4; t += CL_THREADS) dst4[t] = src4[t];
        for (int t = tid; t < na; t += CL_THREADS) cnt_g[(size_t)rank * per + t] = cnt[t];
    }
    if (!ACCEL && rank == 0 && tid == 0) *since_g = since;
}

typedef void (*cluster_kernel_t)(Dev, RepDev, StateView, double*, float4*, double, int, int, int, int, int*, int*, double*, int*, int, int64_t,
                                 int, int, double*, const double*, double*);

template <int LPA>
static cluster_kernel_t cluster_kernel_pots(int pots, bool accel)
{
    switch (pots & (NBG_POT_LJ | NBG_POT_EL)) {
    case NBG_POT_LJ: return accel ? k_cluster_vv<LPA, true, NBG_POT_LJ> : k_cluster_vv<LPA, false, NBG_POT_LJ>;
    case NBG_POT_EL: return accel ? k_cluster_vv<LPA, true, NBG_POT_EL> : k_cluster_vv<LPA, false, NBG_POT_EL>;
    default:
        return accel ? k_cluster_vv<LPA, true, NBG_POT_LJ | NBG_POT_EL> : k_cluster_vv<LPA, false, NBG_POT_LJ | NBG_POT_EL>;
    }
}

// (at most 128 atoms per CTA: 8 lanes each at least)
static cluster_kernel_t cluster_kernel(const nbg_ctx* c, int lpa, bool accel = false)
{
    switch (lpa) {
    case 8: return cluster_kernel_pots<8>(c->d.pots, accel);
    case 16: return cluster_kernel_pots<16>(c->d.pots, accel);
    default: return cluster_kernel_pots<32>(c->d.pots, accel);
    }
}

// Plan the cluster path for the current list capacity: cluster size (16 where
// the device allows it, else the portable 8), atoms per CTA, lanes per atom
// and shared-memory bytes. Returns false when the system does not qualify
// (one replica of a potential system under cubic boundaries, no
// thermostat, small enough for the shared-memory copies).
bool cluster_plan(nbg_ctx* c)
{
    c->cluster_ok = false;
    if (c->cluster_disabled || c->path != PATH_LIST || c->nrep != 1 || c->d.kind != NBG_SYSTEM_POTENTIAL ||
        c->d.bc != NBG_BC_CUBIC || c->d.therm != NBG_THERMO_NULL || c->baoab || c->n < 64 || c->n > 2048)
        return false;
    // (the cluster lists' rows are whole 16-byte units: cap rounded up to 4)
    const int n = (int)c->n, cap = (c->d.nbr_cap + 3) & ~3;
    for (int C = CL_MAX; C >= 8; C /= 2) {
        const int per = (n + C - 1) / C;
        if (per > 128) continue;  // owner threads: 4 warps x 32 lanes
        int lpa = 32;
        while (lpa > 8 && per * lpa > CL_THREADS) lpa /= 2;
        if (per * lpa > CL_THREADS) continue;
        const size_t bytes = cluster_smem(n, per, cap);
        // (two position buffers' worth: with lists longer than this leaves room
        // for, the step graphs serve the system)
        if (bytes + sizeof(float4) * 2 * (size_t)n > 200 * 1024) continue;
        cluster_kernel_t k = cluster_kernel(c, lpa), ka = cluster_kernel(c, lpa, true);
        bool attrs_ok = true;
        for (cluster_kernel_t f : {k, ka}) {
            attrs_ok = attrs_ok &&
                       cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess &&
                       (C <= 8 || cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                                      cudaSuccess);
        }
        if (!attrs_ok) {
            cudaGetLastError();
            continue;
        }
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = C;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(C);
        cfg.blockDim = dim3(CL_THREADS);
        cfg.dynamicSmemBytes = bytes;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, (const void*)k, &cfg) != cudaSuccess || clusters < 1) {
            cudaGetLastError();
            continue;
        }
        c->cluster_ok = true;
        c->cluster_size = C;
        c->cluster_per = per;
        c->cluster_lpa = lpa;
        c->cluster_bytes = bytes;
        c->cluster_cap = cap;
        return true;
    }
    return false;
}

int launch_cluster_vv(nbg_ctx* c, const StateView& s, double dt, int64_t nsteps, int rebuild_every, int64_t step0,
                      unsigned* status)
{
    cluster_kernel_t k = cluster_kernel(c, c->cluster_lpa);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c->cluster_size;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(c->cluster_size);
    cfg.blockDim = dim3(CL_THREADS);
    cfg.dynamicSmemBytes = c->cluster_bytes;
    cfg.stream = c->stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // a one-shot test of the timeout path (NBG_TEST_CLUSTER_DROP at context
    // creation): the launch drops the position copies of one step
    int drop = -2;
    if (c->cluster_test_drop != -2 && c->cluster_test_skip > 0) {
        --c->cluster_test_skip;
    } else if (c->cluster_test_drop != -2) {
        drop = c->cluster_test_drop < 0 ? (int)nsteps - 1 : std::min<int>(c->cluster_test_drop, (int)nsteps - 1);
        c->cluster_test_drop = -2;
    }
    Dev d = c->d;
    d.status = status;
    prof_begin(c);
    cudaError_t e = cudaLaunchKernelEx(&cfg, k, d, c->reps_h[0], s, c->cluster_x, c->cluster_split, dt, (int)nsteps, rebuild_every,
                                       c->cluster_per, c->cluster_cap, c->cluster_lists, c->cluster_cnt,
                                       c->cluster_xref, c->cluster_since, c->cluster_lists_valid ? 1 : 0, step0,
                                       c->sink_on ? 1 : 0, drop, c->bk, (const double*)nullptr, (double*)nullptr);
    prof_end(c);
    if (e != cudaSuccess) return cuda_fail(c, e, "k_cluster_vv launch");
    NBG_LAUNCH_CHECK(c, "k_cluster_vv");
    return NBG_OK;
}

// The right-hand side of a small system (nbg_accel) as one cluster launch:
// positions from u, accelerations to dv (device addresses: pinned host
// memory mapped into the device's space, or device memory), the launch's
// own lists reused while no atom moved more than skin/2 from their build.
int launch_cluster_accel(nbg_ctx* c, const double* u, double* dv, unsigned* status)
{
    cluster_kernel_t k = cluster_kernel(c, c->cluster_lpa, true);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c->cluster_size;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(c->cluster_size);
    cfg.blockDim = dim3(CL_THREADS);
    cfg.dynamicSmemBytes = c->cluster_bytes;
    cfg.stream = c->stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    Dev d = c->d;
    d.status = status;
    prof_begin(c);
    cudaError_t e = cudaLaunchKernelEx(&cfg, k, d, c->reps_h[0], c->st, c->cluster_x, c->cluster_split, 0.0, 1, 0, c->cluster_per, c->cluster_cap,
                                       c->cla_lists, c->cla_cnt, c->cla_xref, c->cluster_since,
                                       c->cla_valid ? 1 : 0, (int64_t)0, 0, -2, c->bk, u, dv);
    prof_end(c);
    if (e != cudaSuccess) return cuda_fail(c, e, "k_cluster_vv (right-hand side) launch");
    NBG_LAUNCH_CHECK(c, "k_cluster_vv");
    return NBG_OK;
}

// The launch floor of the cluster loop's shape: a kernel with the same CTAs,
// threads, shared memory and cluster that only passes one cluster barrier.
__global__ void __launch_bounds__(CL_THREADS, 1) k_cluster_empty(int* sink)
{
    extern __shared__ float4 ce_s[];
    cg::cluster_group cl = cg::this_cluster();
    if (threadIdx.x == 0) ce_s[0] = make_float4(0.f, 0.f, 0.f, 0.f);
    cl.sync();
    if (threadIdx.x == 0 && ce_s[0].x != 0.f) *sink = 1;  // never: keeps the store live
}

int cluster_launch_floor(nbg_ctx* c, double* us_single, double* us_per_launch)
{
    if (!c->cluster_ok) return NBG_ERR_UNSUPPORTED;
    if (cudaFuncSetAttribute(k_cluster_empty, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c->cluster_bytes) !=
            cudaSuccess ||
        (c->cluster_size > 8 &&
         cudaFuncSetAttribute(k_cluster_empty, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess))
        return cuda_fail(c, cudaGetLastError(), "k_cluster_empty attributes");
    int* sink = nullptr;
    if (cudaMalloc(&sink, sizeof(int)) != cudaSuccess) return cuda_fail(c, cudaGetLastError(), "probe sink");
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c->cluster_size;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(c->cluster_size);
    cfg.blockDim = dim3(CL_THREADS);
    cfg.dynamicSmemBytes = c->cluster_bytes;
    cfg.stream = c->stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < 20 && e == cudaSuccess; ++k) e = cudaLaunchKernelEx(&cfg, k_cluster_empty, sink);
    const int reps = 200;
    float ms = 0.f, single = 0.f;
    if (e == cudaSuccess) {
        // back to back
        cudaEventRecord(e0, c->stream);
        for (int k = 0; k < reps && e == cudaSuccess; ++k) e = cudaLaunchKernelEx(&cfg, k_cluster_empty, sink);
        cudaEventRecord(e1, c->stream);
        if (e == cudaSuccess) e = cudaEventSynchronize(e1);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    }
    // one at a time, the host waiting for each
    for (int k = 0; k < reps && e == cudaSuccess; ++k) {
        float m1 = 0.f;
        cudaEventRecord(e0, c->stream);
        e = cudaLaunchKernelEx(&cfg, k_cluster_empty, sink);
        cudaEventRecord(e1, c->stream);
        if (e == cudaSuccess) e = cudaEventSynchronize(e1);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&m1, e0, e1);
        single += m1;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    if (e != cudaSuccess) return cuda_fail(c, e, "cluster launch floor");
    if (us_per_launch) *us_per_launch = 1e3 * ms / reps;
    if (us_single) *us_single = 1e3 * single / reps;
    return NBG_OK;
}

