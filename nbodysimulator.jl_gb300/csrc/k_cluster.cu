// k_cluster.cu - velocity Verlet for small systems (up to 2048 atoms) as one
// persistent cooperative launch. ("Cluster" in the names is this group of
// CTAs; it is not a thread-block cluster.)
//
// A step of a small system is a handful of microsecond kernels, so launches,
// not arithmetic, set its pace. Here up to 64 co-resident CTAs run many steps
// in one launch:
//   - CTA r owns atoms [r per, (r+1) per); its threads drift them (FP64, the
//     reference's velocity-Verlet arithmetic) and write each atom's new split
//     position as two 16-byte records (hi, tag) and (lo, tag) to the global
//     buffer of the step's parity. The tag is the step's number over all
//     launches and, as its lowest bit, whether the atom moved too far for the
//     lists. FP64 positions follow as records of their own;
//   - every CTA reads all records through L2 into its shared memory, again
//     (bounded) while a tag is not the step's. 16-byte accesses are single
//     ones, so a record with the right tag is whole: no barrier, flag or
//     fence between the CTAs. With two parity buffers their reuse is ordered
//     too: a CTA writes step s+2 after it has read every step s+1 record,
//     and a peer writes those when all its threads are done with step s;
//   - each CTA keeps the Verlet lists of its own atoms in shared memory,
//     rebuilt from the shared positions (all atoms scanned, the FP32 superset
//     test of the list builders) when any atom moved more than skin/2 since
//     the last build and every rebuild_every steps; a launch that built
//     them stores them at its end (the steps since the build always), and
//     the next one starts from them unless the host invalidated them (a new
//     state), else it builds first;
//   - at its start a launch writes x, v, a_old of its atoms to the backup,
//     from which the host undoes a launch that timed out or overflowed;
//   - LPA lanes per atom evaluate the pairs (cl_pairs: the exact pair set;
//     the ambiguous ones read the FP64 records) and join their
//     partials (compensated FP32) into shared memory; the atom's owner thread,
//     which keeps its x, v, a in registers for the whole launch, kicks the
//     velocity at the start of the next step.
//
// Two exchanges were measured before this one, both in a cluster of 16 CTAs:
// bulk copies into the peers' shared memory, and global buffers with an arrival
// (release) at each peer's mbarrier. Either took ~3900 cycles per step at
// 1000 atoms (10 bytes per cycle from SM to SM; three L2 round trips), and 16
// SMs left the pairs 5000 cycles, kick and drift (FP64) 3700 and the list
// build, over its ~9 steps, 2150. The records take 4000 cycles among 63 CTAs
// (two or three rounds of reads), the rest 1800, 2300 and 850. Step times at
// 500, 1000 and 2000 atoms: 128 threads per CTA 3.6, 4.4, 6.9 us, 256: 3.4, 4.3,
// 6.6, 512: 3.8, 4.8, 8.5, 1024: 5.3, 7.6, 14.4. 200 steps of 1000 atoms: 2.24 ms
// with the cluster's barrier in every step, 1.58 with arrivals, 1.09 now.
//
// The same kernel with ACCEL evaluates the right-hand side alone (nbg_accel):
// the positions come from src (pinned host memory read over the CPU-GPU
// link, or device memory), one step of the loop without drift or kick runs
// (exchange, displacement check, list build when needed, forces), and the
// accelerations go to dst; the lists it keeps are its own, built for earlier
// calls' positions, and the resident state is not touched.
#include <algorithm>

#include "nbg_internal.cuh"

#define CL_THREADS 256  // up to 64 CTAs

// A 16-byte record as one access (single-copy atomic), at L2.
__device__ __forceinline__ ulonglong2 rec_load(const ulonglong2* p)
{
    ulonglong2 r;
    asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
                 : "=l"(r.x), "=l"(r.y)
                 : "l"(p)
                 : "memory");
    return r;
}

__device__ __forceinline__ void rec_store(ulonglong2* p, unsigned long long x, unsigned long long y)
{
    asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p), "l"(x),
                 "l"(y)
                 : "memory");
}

// three floats and their record's tag
__device__ __forceinline__ void rec_store3(ulonglong2* p, float x, float y, float z, unsigned tag)
{
    rec_store(p, (unsigned long long)__float_as_uint(x) | (unsigned long long)__float_as_uint(y) << 32,
              (unsigned long long)__float_as_uint(z) | (unsigned long long)tag << 32);
}

#define CL_TRIES (1u << 18)  // reads of a record before a launch gives up

// The FP64 position of an atom of this step (three records (bits, tag)).
__device__ __forceinline__ bool rec_position(const ulonglong2* X, unsigned tag, double (&x)[3])
{
    unsigned tries = 0;
    for (int k = 0; k < 3; ++k) {
        ulonglong2 r = rec_load(X + k);
        while ((unsigned)r.y != tag) {
            if (++tries >= CL_TRIES) return false;
            r = rec_load(X + k);
        }
        x[k] = __longlong_as_double((long long)r.x);
    }
    return true;
}

// A pair that FP32 does not decide, by the FP64 records (out of line: rare).
struct ClExact {
    float x, y, z, r2;
    int in;  // 1: inside lj_R2, 2: inside el_R2, 4: image not found, 8: a record did not come
};

__device__ __noinline__ ClExact cl_exact(const ulonglong2* X, unsigned tag, int i, int j, double L, double lj_R2, double el_R2)
{
    ClExact o = {0.f, 0.f, 0.f, 1.f, 0};
    double xi[3], xj[3];
    if (!rec_position(X + 3 * i, tag, xi) || !rec_position(X + 3 * j, tag, xj)) {
        o.in = 8;
        return o;
    }
    double x = __dsub_rn(xi[0], xj[0]), y = __dsub_rn(xi[1], xj[1]), z = __dsub_rn(xi[2], xj[2]);
    const double radius = __dmul_rn(0.5, L);
    if (!(wrap_cubic64(x, L, radius) && wrap_cubic64(y, L, radius) && wrap_cubic64(z, L, radius))) {
        o.in = 4;
        return o;
    }
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
    o.x = (float)x;
    o.y = (float)y;
    o.z = (float)z;
    o.r2 = (float)r2;
    o.in = (r2 < lj_R2 ? 1 : 0) | (r2 < el_R2 ? 2 : 0);
    return o;
}

// The forces on i of M listed atoms j[] (the first m of them), in
// pair_cutoff's arithmetic and classification, added to p in order. One branch for
// all, to the pairs that FP32 does not decide: with one per pair a lane's
// pairs did not overlap, and there are only two warps per SM sub-partition
// to hide a pair's latency. A potential system: every listed pair has both
// potentials of POTS.
#define CL_M 3
template <int POTS>
__device__ __forceinline__ void cl_pairs(const Dev& d, const RepDev& R, int i, const int (&j)[CL_M], int m, const float4& hi_i,
                                         const float4& lo_i, const float4* ph, const float4* pl, float kqi,
                                         const ulonglong2* X, unsigned tag, float (&p)[3], bool& range_err)
{
    constexpr bool LJ = (POTS & NBG_POT_LJ) != 0, EL = (POTS & NBG_POT_EL) != 0;
    float3 dr[CL_M];
    float r2[CL_M], qj[CL_M];
    bool lj[CL_M], el[CL_M], open[CL_M], any = false;
#pragma unroll
    for (int q = 0; q < CL_M; ++q) {
        const float4 hj = ph[j[q]], lj4 = pl[j[q]];
        qj[q] = hj.w;
        dr[q] = split_diff(hi_i, lo_i, hj, lj4, true, R);
        r2[q] = __fmaf_rn(dr[q].x, dr[q].x, __fmaf_rn(dr[q].y, dr[q].y, __fmul_rn(dr[q].z, dr[q].z)));
        lj[q] = LJ && r2[q] < R.lj_lo;
        el[q] = EL && r2[q] < R.el_lo;
        open[q] = q < m && ((LJ && !lj[q] && r2[q] < R.lj_hi) || (EL && !el[q] && r2[q] < R.el_hi));
        any |= open[q];
    }
    if (any) {
#pragma unroll
        for (int q = 0; q < CL_M; ++q) {
            if (!open[q]) continue;
            const ClExact e = cl_exact(X, tag, i, j[q], R.L, d.lj_R2, d.el_R2);
            lj[q] = LJ && (e.in & 1);
            el[q] = EL && (e.in & 2);
            dr[q] = make_float3(e.x, e.y, e.z);
            r2[q] = e.r2;
            range_err |= (e.in & 4) != 0;
            if (e.in & 8) status_set(d.status, ST_TIMEOUT);
        }
    }
#pragma unroll
    for (int q = 0; q < CL_M; ++q) {
        const float rr = lj[q] || el[q] ? r2[q] : 1.0f;
        float f = 0.0f;
        if (LJ) {
            const float ri = rcp_ftz(rr);
            const float s2 = __fmul_rn(d.lj_sig2, ri);
            const float s6 = __fmul_rn(__fmul_rn(s2, s2), s2);
            const float s12 = __fmul_rn(s6, s6);
            const float g = __fmul_rn(d.lj_eps24, __fmul_rn(__fmaf_rn(2.0f, s12, -s6), ri));
            f = lj[q] ? g : 0.0f;
        }
        if (EL) {
            const float rb = rsqrt_ftz(rr);
            const float t = __fmaf_rn(__fmul_rn(rb, rb), rb, -d.el_krf2);
            const float g = __fmaf_rn(__fmul_rn(kqi, qj[q]), t, f);
            f = el[q] ? g : f;
        }
        if (q < m) {
            p[0] = __fadd_rn(p[0], __fmul_rn(f, dr[q].x));
            p[1] = __fadd_rn(p[1], __fmul_rn(f, dr[q].y));
            p[2] = __fadd_rn(p[2], __fmul_rn(f, dr[q].z));
        }
    }
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
        grid_split(R, w, h, l);
    } else {
        grid_split<true>(R, w, h, l);
    }
}

// R: the replica's constants as a kernel argument (operands from the constant
// bank; through d.reps every use was a load again, as the kernel stores).
template <int LPA, bool ACCEL, int POTS>
__global__ void __launch_bounds__(CL_THREADS, 1) k_cluster_vv(Dev d, const __grid_constant__ RepDev R, StateView s, ulonglong2* xb,
                                                              ulonglong2* xs, unsigned seq, double dt, int nsteps,
                                                              int rebuild_every, int per, int cap, int* lst_g,
                                                              int* cnt_g, double* xref_g, int* since_g, int reuse,
                                                              int64_t step0, int save, int drop_step,
                                                              double* __restrict__ bk,
                                                              const double* __restrict__ src, double* __restrict__ dst)
{
    const int rank = blockIdx.x;
    const int n = (int)d.n;
    extern __shared__ float4 cl_pos[];
    float4* const ph = cl_pos;
    float4* const pl = ph + n;
    double* xref_s = reinterpret_cast<double*>(cl_pos + 2 * (size_t)n);
    int* lst = reinterpret_cast<int*>(xref_s + 3 * (size_t)per + ((3 * per) & 1));  // 16-byte aligned
    int* cnt = lst + (size_t)per * cap;
    float* fsum = reinterpret_cast<float*>(cnt + per);
    __shared__ int gave_up;  // some record of this step did not come
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

    // the charges of all atoms
    if (POTS & NBG_POT_EL)
        for (int j = tid; j < n; j += CL_THREADS) ph[j].w = d.phi[j].w;
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
    if (tid == 0) gave_up = 0;
    __syncthreads();

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
        ulonglong2* const P = xs + (size_t)(2 * par) * n;  // split positions of this step
        ulonglong2* const X = xb + (size_t)par * 3 * n;    // FP64 positions
        const unsigned tag = (seq + (unsigned)st) << 1;
        // drift, split and displacement check of the own atoms
        if (tid < owners) {
            double dk = 0.0;
            float h = 0.f, l = 0.f;
            if (owner) {
                if (!ACCEL) x = drift1(x, v, a, dt, dtsq);
                // (a launch that does not reuse lists builds at step 0, which
                // sets xref_s)
                dk = x - xref_s[3 * ko + k];
                split_kept_image(R, x, img, h, l);
            }
            const float fk = (float)dk, fk2 = fk * fk;
            const int l0 = (tid & 31) - k;  // the atom's first lane
            const float f2 = __shfl_sync(0xffffffffu, fk2, l0) + __shfl_sync(0xffffffffu, fk2, l0 + 1) +
                             __shfl_sync(0xffffffffu, fk2, l0 + 2);
            bool moved = owner && (st > 0 || reuse) && !(f2 < still2);
            if (__any_sync(0xffffffffu, moved)) {
                const double dx = __shfl_sync(0xffffffffu, dk, l0), dy = __shfl_sync(0xffffffffu, dk, l0 + 1),
                             dz = __shfl_sync(0xffffffffu, dk, l0 + 2);
                moved = moved && !(dx * dx + dy * dy + dz * dz <= d.skin_half2);
            }
            // lane 0 of the atom writes the hi record, lane 1 the lo record
            const float hx = __shfl_sync(0xffffffffu, h, l0), hy = __shfl_sync(0xffffffffu, h, l0 + 1),
                        hz = __shfl_sync(0xffffffffu, h, l0 + 2);
            const float lx = __shfl_sync(0xffffffffu, l, l0), ly = __shfl_sync(0xffffffffu, l, l0 + 1),
                        lz = __shfl_sync(0xffffffffu, l, l0 + 2);
            // (drop_step: a host-set test of the timeout path; no CTA writes
            // that step's records, so every wait runs out)
            if (owner && st != drop_step) {
                if (k < 2) rec_store3(P + k * n + io, k ? lx : hx, k ? ly : hy, k ? lz : hz, tag | (moved ? 1u : 0u));
                rec_store(X + eo, (unsigned long long)__double_as_longlong(x), tag);
            }
        }
        // all records of this step, several reads in flight per thread. One that
        // does not come ends this CTA's loop and, as it writes no further
        // step, the others' at their next one
        bool moved = false;
        {
            constexpr int B = 8;
            unsigned tries = 0;
            for (int t0 = tid; t0 < 2 * n; t0 += B * CL_THREADS) {
                // (all that are missing are read again together: one after
                // the other they cost a round trip each)
                ulonglong2 r[B];
                unsigned missing = 0u;
#pragma unroll
                for (int q = 0; q < B; ++q)
                    if (t0 + q * CL_THREADS < 2 * n) missing |= 1u << q;
                while (missing != 0u && tries < CL_TRIES) {
                    ++tries;
#pragma unroll
                    for (int q = 0; q < B; ++q)
                        if (missing >> q & 1u) r[q] = rec_load(P + t0 + q * CL_THREADS);
#pragma unroll
                    for (int q = 0; q < B; ++q) {
                        if ((missing >> q & 1u) && ((unsigned)(r[q].y >> 32) ^ tag) <= 1u) {
                            missing &= ~(1u << q);
                            moved |= ((unsigned)(r[q].y >> 32) & 1u) != 0u;
                            float* o = reinterpret_cast<float*>(cl_pos + t0 + q * CL_THREADS);
                            *reinterpret_cast<float2*>(o) =
                                make_float2(__uint_as_float((unsigned)r[q].x), __uint_as_float((unsigned)(r[q].x >> 32)));
                            o[2] = __uint_as_float((unsigned)r[q].y);
                        }
                    }
                }
                if (missing != 0u) gave_up = 1;
            }
        }
        const int any_moved = __syncthreads_or(moved ? 1 : 0);
        if (gave_up) {
            if (tid == 0) status_set(d.status, ST_TIMEOUT);
            break;
        }
        const bool build = (st == 0 && !reuse) || any_moved ||
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
            for (int k = lane; k < c; k += CL_M * LPA) {
                int j[CL_M];
#pragma unroll
                for (int q = 0; q < CL_M; ++q) j[q] = dbg_index(lst[g * cap + min(k + q * LPA, c - 1)], d.n, i, d.status);
                cl_pairs<POTS>(d, R, i, j, (c - k + LPA - 1) / LPA, hi_i, lo_i, ph, pl, kqi, X, tag, p, range_err);
            }
            const LaneSum f = lane_sums3<LPA>(p[0], p[1], p[2], lane);
            if (range_err) status_set(d.status, ST_RANGE);
            if (active && f.writer) {
                fsum[6 * g + 2 * f.comp] = f.h;
                fsum[6 * g + 2 * f.comp + 1] = f.e;
            }
        }
        __syncthreads();
    }
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

typedef void (*cluster_kernel_t)(Dev, RepDev, StateView, ulonglong2*, ulonglong2*, unsigned, double, int, int, int, int, int*, int*, double*, int*, int, int64_t,
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

static cluster_kernel_t cluster_kernel(const nbg_ctx* c, int lpa, bool accel = false)
{
    switch (lpa) {
    case 8: return cluster_kernel_pots<8>(c->d.pots, accel);
    case 16: return cluster_kernel_pots<16>(c->d.pots, accel);
    default: return cluster_kernel_pots<32>(c->d.pots, accel);
    }
}

// A cooperative launch of the loop's shape: its CTAs wait for one another.
struct ClusterLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    explicit ClusterLaunch(const nbg_ctx* c)
    {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.gridDim = dim3(c->cluster_size);
        cfg.blockDim = dim3(CL_THREADS);
        cfg.dynamicSmemBytes = c->cluster_bytes;
        cfg.stream = c->stream;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    ClusterLaunch(const ClusterLaunch&) = delete;
};

// Plan the loop for the current list capacity: CTAs, atoms per CTA, lanes per
// atom and shared-memory bytes. Returns false when the system does not qualify
// (one replica of a potential system under cubic boundaries, no
// thermostat, small enough for the shared-memory copies).
bool cluster_plan(nbg_ctx* c)
{
    c->cluster_ok = false;
    if (c->cluster_disabled || c->path != PATH_LIST || c->nrep != 1 || c->d.kind != NBG_SYSTEM_POTENTIAL ||
        c->d.bc != NBG_BC_CUBIC || c->d.therm != NBG_THERMO_NULL || c->baoab || c->n < 64 || c->n > 2048)
        return false;
    // (the lists' rows are whole 16-byte units: cap rounded up to 4)
    const int n = (int)c->n, cap = (c->d.nbr_cap + 3) & ~3;
    // the lanes per atom and the line between this loop and the step graphs
    // are those of 1024 threads and 200 KB on each of 16 SMs, so that a
    // system keeps the order of its FP32 sums whatever the CTAs
    const int part = (n + 15) / 16;
    const int lpa = part <= 32 ? 32 : part <= 64 ? 16 : 8;
    if (cluster_smem(n, part, cap) + sizeof(float4) * 2 * (size_t)n > 200 * 1024) return false;
    const int per = CL_THREADS / lpa, C = (n + per - 1) / per;
    const size_t bytes = cluster_smem(n, per, cap);
    for (cluster_kernel_t f : {cluster_kernel(c, lpa), cluster_kernel(c, lpa, true)}) {
        // (the attribute is the function's, for every context of the process)
        int blocks = 0;
        if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, f, CL_THREADS, bytes) != cudaSuccess ||
            blocks * c->sms < C) {
            cudaGetLastError();
            return false;
        }
    }
    c->cluster_ok = true;
    c->cluster_size = C;
    c->cluster_per = per;
    c->cluster_lpa = lpa;
    c->cluster_bytes = bytes;
    c->cluster_cap = cap;
    return true;
}

int launch_cluster_vv(nbg_ctx* c, const StateView& s, double dt, int64_t nsteps, int rebuild_every, int64_t step0,
                      unsigned* status)
{
    cluster_kernel_t k = cluster_kernel(c, c->cluster_lpa);
    ClusterLaunch L(c);
    // a one-shot test of the timeout path (NBG_TEST_CLUSTER_DROP at context
    // creation): the launch drops the position records of one step
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
    cudaError_t e = cudaLaunchKernelEx(&L.cfg, k, d, c->reps_h[0], s, c->cluster_x, c->cluster_split, c->cluster_seq, dt, (int)nsteps, rebuild_every,
                                       c->cluster_per, c->cluster_cap, c->cluster_lists, c->cluster_cnt,
                                       c->cluster_xref, c->cluster_since, c->cluster_lists_valid ? 1 : 0, step0,
                                       c->sink_on ? 1 : 0, drop, c->bk, (const double*)nullptr, (double*)nullptr);
    prof_end(c);
    c->cluster_seq += (unsigned)nsteps;
    if (e != cudaSuccess) return cuda_fail(c, e, "k_cluster_vv launch");
    NBG_LAUNCH_CHECK(c, "k_cluster_vv");
    return NBG_OK;
}

// The right-hand side of a small system (nbg_accel) as one launch:
// positions from u, accelerations to dv (device addresses: pinned host
// memory mapped into the device's space, or device memory), the launch's
// own lists reused while no atom moved more than skin/2 from their build.
int launch_cluster_accel(nbg_ctx* c, const double* u, double* dv, unsigned* status)
{
    cluster_kernel_t k = cluster_kernel(c, c->cluster_lpa, true);
    ClusterLaunch L(c);
    Dev d = c->d;
    d.status = status;
    prof_begin(c);
    cudaError_t e = cudaLaunchKernelEx(&L.cfg, k, d, c->reps_h[0], c->st, c->cluster_x, c->cluster_split, c->cluster_seq, 0.0, 1, 0, c->cluster_per, c->cluster_cap,
                                       c->cla_lists, c->cla_cnt, c->cla_xref, c->cluster_since,
                                       c->cla_valid ? 1 : 0, (int64_t)0, 0, -2, c->bk, u, dv);
    prof_end(c);
    ++c->cluster_seq;
    if (e != cudaSuccess) return cuda_fail(c, e, "k_cluster_vv (right-hand side) launch");
    NBG_LAUNCH_CHECK(c, "k_cluster_vv");
    return NBG_OK;
}

// The launch floor of the loop's shape: a kernel with the same CTAs, threads,
// shared memory and launch attribute that does nothing.
__global__ void __launch_bounds__(CL_THREADS) k_cluster_empty(int* sink)
{
    extern __shared__ float4 ce_s[];
    if (threadIdx.x == 0) ce_s[0] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    if (threadIdx.x == 0 && ce_s[0].x != 0.f) *sink = 1;  // never: keeps the store live
}

int cluster_launch_floor(nbg_ctx* c, double* us_single, double* us_per_launch)
{
    if (!c->cluster_ok) return NBG_ERR_UNSUPPORTED;
    if (cudaFuncSetAttribute(k_cluster_empty, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess)
        return cuda_fail(c, cudaGetLastError(), "k_cluster_empty attributes");
    int* sink = nullptr;
    if (cudaMalloc(&sink, sizeof(int)) != cudaSuccess) return cuda_fail(c, cudaGetLastError(), "probe sink");
    ClusterLaunch L(c);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < 20 && e == cudaSuccess; ++k) e = cudaLaunchKernelEx(&L.cfg, k_cluster_empty, sink);
    const int reps = 200;
    float ms = 0.f, single = 0.f;
    if (e == cudaSuccess) {
        // back to back
        cudaEventRecord(e0, c->stream);
        for (int k = 0; k < reps && e == cudaSuccess; ++k) e = cudaLaunchKernelEx(&L.cfg, k_cluster_empty, sink);
        cudaEventRecord(e1, c->stream);
        if (e == cudaSuccess) e = cudaEventSynchronize(e1);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    }
    // one at a time, the host waiting for each
    for (int k = 0; k < reps && e == cudaSuccess; ++k) {
        float m1 = 0.f;
        cudaEventRecord(e0, c->stream);
        e = cudaLaunchKernelEx(&L.cfg, k_cluster_empty, sink);
        cudaEventRecord(e1, c->stream);
        if (e == cudaSuccess) e = cudaEventSynchronize(e1);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&m1, e0, e1);
        single += m1;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    if (e != cudaSuccess) return cuda_fail(c, e, "launch floor of the small-system loop");
    if (us_per_launch) *us_per_launch = 1e3 * ms / reps;
    if (us_single) *us_single = 1e3 * single / reps;
    return NBG_OK;
}

