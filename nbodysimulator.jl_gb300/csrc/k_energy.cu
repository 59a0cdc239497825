// k_energy.cu - FP64 energy reductions with the reference's definitions and
// the pair-set export used by the parity tests.
//
// Energies (nbody_simulation_result.jl): kinetic sum m v^2 / 2 (:209-212);
// Lennard-Jones 4 eps sum_{i<j} (s^12 - s^6) with r^2 clamped to R^2 beyond
// the cutoff (:293-319); electrostatic k sum_i q_i sum_{j>i, not excluded}
// (q_j / r or q_j / R) (:321-351); bonds sum over directed bonds k d^2 / 4
// (:353-372); angles sum k (theta - theta0)^2 / 2 (:374-397); gravity
// -G sum_{i<j} m_i m_j / r (this project's; the reference has none).
// Per-block partials are summed in a fixed order (deterministic).
#include <algorithm>

#include "fx_pair.cuh"

#define EB 128
#define EJ 32        // bodies j per block of k_energy_pairs
#define EL_WARPS 8   // warps per block of k_energy_list

// These kernels are bound by their count of FP64 instructions.

// 1 / sqrt(x) to ~1 ulp: the FP32 approximation (2^-22) refined by one
// third-order step, y (1 + e/2 + 3 e^2 / 8) with e = 1 - x y^2 (error ~e^3);
// arguments outside FP32's comfortable range take the square root and the
// division (9 against ~40 FP64 instructions).
__device__ __forceinline__ double rsqrt64(double x)
{
    const int hi = __double2hiint(x);
    if (hi < 0x39b00000 || hi > 0x46300000) return 1.0 / sqrt(x);  // 2^-100 .. 2^100
    const double y = widen(rsqrtf(__double2float_rn(x)));
    const double e = fma(-(x * y), y, 1.0);
    return fma(y, e * fma(0.375, e, 0.5), y);
}

// Cubic minimum image of a difference: d - L rint(d / L) (r^2 does not depend
// on the choice at half a box). False where the image number is not a plain
// one (beyond the reference loops' cap, or not finite).
__device__ __forceinline__ bool nearest_image(double& d, double L, double invL)
{
    const double magic = 6755399441055744.0;  // 1.5 * 2^52
    const double t = fma(d, invL, magic);
    const int k = __double2loint(t), h = __double2hiint(t);
    d = fma(-L, t - magic, d);
    return (h == 0x43380000 || h == 0x4337ffff) && k >= -MINIMAGE_MAX_ITERS && k <= MINIMAGE_MAX_ITERS;
}

// x < y for non-negative doubles; a NaN of either sign compares as large (as
// unsigned words: a negative one has the top bit)
__device__ __forceinline__ bool below(double x, double y)
{
    return (unsigned long long)__double_as_longlong(x) < (unsigned long long)__double_as_longlong(y);
}

// Sums over the block of up to 3 values per thread, by warps and then in
// warp order, to out[0..K-1] by the first thread.
template <int K>
__device__ __forceinline__ void block_sums(double (&v)[K], double* out)
{
    __shared__ double sh[32][K];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < K; ++k) sh[threadIdx.x >> 5][k] = v[k];
    __syncthreads();
    if (threadIdx.x < K) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[w][threadIdx.x];
        out[threadIdx.x] = t;
    }
}

// LJ, electrostatic and gravity sums over all pairs j > i: an item is 128
// bodies i (a thread each) and 32 bodies j from shared memory. (A thread per
// body i walking every j > i left n / 128 blocks of very uneven length:
// 8.0 ms for 6429 gravitating bodies, 4.0 ms for 3163 ions.)
template <int BC, bool HAS_LJ, bool HAS_EL, bool HAS_G>
__global__ void __launch_bounds__(EB) k_energy_pairs(Dev d, const double* X, double* out /*[grid][3]*/)
{
    __shared__ double xj[EJ], yj[EJ], zj[EJ], qj[EJ], mj[EJ];
    const RepDev& R = d.reps[0];
    const bool water = d.kind == NBG_SYSTEM_WATER;
    const int64_t jt = (d.n + EJ - 1) / EJ, items = (d.n + EB - 1) / EB * jt;
    const double L = R.L, invL = R.invL, invR = 1.0 / d.el_R;
    const double sR = HAS_LJ ? d.lj_sig2_d / d.lj_R2 : 0.0;  // sigma^2 / r^2 from the cutoff on
    double e[3] = {0.0, 0.0, 0.0};
    bool range_err = false;
    for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
        const int64_t i0 = it / jt * EB, j0 = it % jt * EJ;
        if (j0 + EJ <= i0 + 1) continue;  // no j > i (uniform)
        __syncthreads();
        if (threadIdx.x < EJ && j0 + threadIdx.x < d.n) {
            const int64_t j = j0 + threadIdx.x;
            xj[threadIdx.x] = X[3 * j];
            yj[threadIdx.x] = X[3 * j + 1];
            zj[threadIdx.x] = X[3 * j + 2];
            if (HAS_EL) qj[threadIdx.x] = d.charge[j];
            if (HAS_G) mj[threadIdx.x] = d.mass[j];
        }
        __syncthreads();
        const int64_t i = i0 + threadIdx.x;
        if (i >= d.n) continue;
        const double x = X[3 * i], y = X[3 * i + 1], z = X[3 * i + 2];
        double el = 0.0, g = 0.0;
        const int k0 = (int)max((int64_t)0, i + 1 - j0), k1 = (int)min((int64_t)EJ, d.n - j0);
        for (int k = k0; k < k1; ++k) {
            const int64_t j = j0 + k;
            double dx = x - xj[k], dy = y - yj[k], dz = z - zj[k];
            if (HAS_G) {  // (gravity ignores the boundary)
                const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
                g = fma(mj[k], rsqrt64(r2), g);
            }
            if (!HAS_LJ && !HAS_EL) continue;
            const bool lj = HAS_LJ && (!water || (i % 3 == 0 && j % 3 == 0));
            const bool ep = HAS_EL && !(water && i / 3 == j / 3);
            if (!(lj || ep)) continue;
            double r2;
            bool plain = BC != NBG_BC_PERIODIC;
            if (BC == NBG_BC_CUBIC) {
                const bool px = nearest_image(dx, L, invL), py = nearest_image(dy, L, invL),
                           pz = nearest_image(dz, L, invL);
                plain = px && py && pz;
            }
            if (plain) {
                r2 = fma(dx, dx, fma(dy, dy, dz * dz));
            } else {  // the reference's loops
                Dist64 q;
                if (!distance64(X + 3 * i, X + 3 * j, BC, R, q)) {
                    range_err = true;
                    continue;
                }
                r2 = q.r2;
            }
            const double ri = rsqrt64(r2);
            if (lj) {
                double s6 = below(r2, d.lj_R2) ? d.lj_sig2_d * (ri * ri) : sR;
                s6 = s6 * s6 * s6;
                e[0] += fma(s6, s6, -s6);
            }
            if (ep) {
                double t = ri;  // reaction field: 1/r + k_rf r^2 - c_rf (+ c_rf back, so eps_rf = 1 gives 1/r)
                if (d.el_krf != 0.0) t += fma(d.el_krf, r2, -(d.el_crf - invR));
                el = fma(qj[k], below(r2, d.el_R2) ? t : invR, el);
            }
        }
        if (HAS_EL) e[1] = fma(el, d.charge[i], e[1]);
        if (HAS_G) e[2] = fma(g, d.mass[i], e[2]);
    }
    if (range_err) status_set(d.status, ST_RANGE);
    block_sums<3>(e, out + 3 * (int64_t)blockIdx.x);
}

// The same LJ and electrostatic sums over the Verlet list (built for X):
// for each pair inside a cutoff, its term minus the term the reference gives
// a pair beyond it (LJ at r = R, Coulomb q_i q_j / R); the host adds those
// constant terms for all pairs analytically. O(N x neighbours) instead of
// O(N^2); each pair is taken once (j > i). A warp per atom reads its row,
// keeps the entries j > i that FP32 finds within the largest cutoff (about a
// third), and queues them by the arithmetic they need: the FP64 code then
// runs on full warps of like pairs (14 FP64 instructions for a bare charge
// pair, 30 for an LJ + charge pair across a face). (A thread per atom over its whole row took 1.1 ms at 12,288 atoms.)
__global__ void __launch_bounds__(EL_WARPS * 32) k_energy_list(Dev d, const double* X, double* out /*[grid][3]*/)
{
    __shared__ int2 queue[EL_WARPS][4][64];
    const RepDev& R = d.reps[0];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool water = d.kind == NBG_SYSTEM_WATER;
    const bool has_lj = (d.pots & NBG_POT_LJ) != 0, has_el = (d.pots & NBG_POT_EL) != 0;
    const float reach = fmaxf(has_lj ? R.fx_lj_hi : 0.f, has_el ? R.fx_el_hi : 0.f);
    const double L = R.L, invL = R.invL;
    const double reach2 = 0.25 * L * L;  // (above every cutoff's square on the list path)
    double s6R = d.lj_sig2_d / d.lj_R2;
    s6R = s6R * s6R * s6R;
    const double ljR = fma(s6R, s6R, -s6R);
    const double invR = 1.0 / d.el_R;
    double e[3] = {0.0, 0.0, 0.0};
    bool range_err = false;
    // queues by the arithmetic their pairs need: + 1 for a pair whose bare
    // difference is not its minimum image, + 2 for an LJ pair
    int fill[4] = {0, 0, 0, 0};
    auto take = [&](int2* q, int m, bool image, bool lj) {  // the first m queued pairs, one per lane
        if (lane >= m) return;
        const int64_t i = q[lane].x, j = q[lane].y;
        const double x0 = X[3 * i] - X[3 * j], y0 = X[3 * i + 1] - X[3 * j + 1], z0 = X[3 * i + 2] - X[3 * j + 2];
        double r2 = fma(x0, x0, fma(y0, y0, z0 * z0));
        // (a pair queued as bare may still cross a face by a rounding of the
        // fixed-point positions: its r^2 is then far above the list's)
        if (image || !below(r2, reach2)) {
            double dx = x0, dy = y0, dz = z0;
            const bool px = nearest_image(dx, L, invL), py = nearest_image(dy, L, invL), pz = nearest_image(dz, L, invL);
            r2 = fma(dx, dx, fma(dy, dy, dz * dz));
            if (!(px && py && pz)) {  // the reference's loops
                Dist64 o;
                if (!distance64(X + 3 * i, X + 3 * j, NBG_BC_CUBIC, R, o)) {
                    range_err = true;
                    return;
                }
                r2 = o.r2;
            }
        }
        const double ri = rsqrt64(r2);
        if (lj && below(r2, d.lj_R2)) {
            double s6 = d.lj_sig2_d * (ri * ri);
            s6 = s6 * s6 * s6;
            e[0] += fma(s6, s6, -s6) - ljR;
        }
        if (has_el && below(r2, d.el_R2)) {
            double t = ri - invR;
            if (d.el_krf != 0.0) t += fma(d.el_krf, r2, -(d.el_crf - invR));
            e[1] = fma(d.charge[i] * d.charge[j], t, e[1]);
        }
    };
    const int64_t stride = (int64_t)gridDim.x * EL_WARPS;
    for (int64_t i = blockIdx.x * (int64_t)EL_WARPS + w; i < d.n; i += stride) {
        const bool lj_i = has_lj && (!water || fx_oxygen((int)i));
        if (!lj_i && !has_el) continue;
        const int cnt = min(d.nbr_count[i], d.nbr_cap);
        const uint4 qi = d.pfx ? d.pfx[i] : make_uint4(0u, 0u, 0u, 0u);
        const long long* im = reinterpret_cast<const long long*>(d.img) + 3 * i;
        // an atom over half the minimum-image cap of boxes out (or lost): its
        // row is not screened, for its fixed-point position may mean nothing,
        // and every listed pair has to stay within the cap
        bool far = false;
        if (d.pfx)
            for (int c = 0; c < 3; ++c) far |= (im[c] & 0x7fffffffffffffffll) > 0x40e0000000000000ll;  // |image| > 2^15
        for (int k0 = 0; k0 < cnt; k0 += 32) {
            const int k = k0 + lane;
            int j = 0;
            int cls = -1;
            if (k < cnt) {
                j = dbg_index(d.nbr[(int64_t)k * d.nbr_kstride + i * d.nbr_istride], d.n, (int)i, d.status);
                const bool lj = lj_i && (!water || fx_oxygen(j));
                if ((j > (int)i || far) && (lj || (has_el && !el_excluded(d.kind, i, j)))) {
                    if (j > (int)i) {
                        cls = lj ? 3 : 1;
                    } else {  // (the pair's sums are with the row of j)
                        Dist64 o;
                        range_err |= !distance64(X + 3 * (int64_t)j, X + 3 * i, NBG_BC_CUBIC, R, o);
                    }
                    if (d.pfx && !far) {
                        const uint4 qj = d.pfx[j];
                        float fx, fy, fz;
                        if (fx_r2(qi, qj, fx, fy, fz) >= reach) cls = -1;
                        // bare: the same image, and no wrap of the unsigned positions
                        const long long* jm = reinterpret_cast<const long long*>(d.img) + 3 * (int64_t)j;
                        if (im[0] == jm[0] && im[1] == jm[1] && im[2] == jm[2] && (qi.x >= qj.x) == ((int)(qi.x - qj.x) >= 0) &&
                            (qi.y >= qj.y) == ((int)(qi.y - qj.y) >= 0) && (qi.z >= qj.z) == ((int)(qi.z - qj.z) >= 0))
                            cls &= ~1;
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                int2* const q = queue[w][c];
                const bool mine = cls == c;
                const unsigned bal = __ballot_sync(0xffffffffu, mine);
                if (!bal) continue;
                if (mine) q[fill[c] + __popc(bal & ((1u << lane) - 1u))] = make_int2((int)i, j);
                fill[c] += __popc(bal);
                __syncwarp();
                if (fill[c] >= 32) {
                    take(q, 32, c & 1, c & 2);
                    __syncwarp();
                    if (lane < fill[c] - 32) q[lane] = q[32 + lane];
                    fill[c] -= 32;
                    __syncwarp();
                }
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) take(queue[w][c], fill[c], c & 1, c & 2);
    if (range_err) status_set(d.status, ST_RANGE);
    block_sums<3>(e, out + 3 * (int64_t)blockIdx.x);
}

// kinetic sum (v.v) m/2 and m v.v (temperature): a thread per atom; bonds and
// angles: a thread per molecule
__global__ void __launch_bounds__(EB) k_energy_local(Dev d, const double* X, const double* V, double* out /*[grid][4]*/)
{
    double e[4] = {0.0, 0.0, 0.0, 0.0};
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    for (int64_t i = t0; i < d.n; i += stride) {
        double s = __dadd_rn(__dadd_rn(__dmul_rn(V[3 * i], V[3 * i]), __dmul_rn(V[3 * i + 1], V[3 * i + 1])),
                             __dmul_rn(V[3 * i + 2], V[3 * i + 2]));
        e[0] = __dadd_rn(e[0], __dmul_rn(s, d.mass[i] / 2.0));
        e[1] = __dadd_rn(e[1], __dmul_rn(d.mass[i], s));
    }
    if (d.kind == NBG_SYSTEM_WATER)
        for (int64_t m = t0; m < d.n / 3; m += stride) {
            const double *ro = X + 9 * m, *ra = ro + 3, *rc = ro + 6;
            double b1[3], b2[3];
            for (int k = 0; k < 3; ++k) {
                b1[k] = __dsub_rn(ra[k], ro[k]);
                b2[k] = __dsub_rn(rc[k], ro[k]);
            }
            double n1 = sqrt(__dadd_rn(__dadd_rn(__dmul_rn(b1[0], b1[0]), __dmul_rn(b1[1], b1[1])), __dmul_rn(b1[2], b1[2])));
            double n2 = sqrt(__dadd_rn(__dadd_rn(__dmul_rn(b2[0], b2[0]), __dmul_rn(b2[1], b2[1])), __dmul_rn(b2[2], b2[2])));
            double d1 = __dsub_rn(n1, d.rOH), d2 = __dsub_rn(n2, d.rOH);
            // directed bonds O->H1, O->H2, H1->O, H2->O
            double t1 = __dmul_rn(__dmul_rn(d1, d1), d.kbond), t2 = __dmul_rn(__dmul_rn(d2, d2), d.kbond);
            e[2] = __dadd_rn(e[2], __dadd_rn(__dadd_rn(t1, t2), __dadd_rn(t1, t2)));
            double dot = __dadd_rn(__dadd_rn(__dmul_rn(b1[0], b2[0]), __dmul_rn(b1[1], b2[1])), __dmul_rn(b1[2], b2[2]));
            double th = acos(dot / __dmul_rn(n1, n2));
            double dt = __dsub_rn(th, d.aHOH);
            e[3] = __dadd_rn(e[3], __dmul_rn(__dmul_rn(d.kangle, dt), dt));
        }
    block_sums<4>(e, out + 4 * (int64_t)blockIdx.x);
}

// The sums of the block partials in a fixed order: out[0..2] of a[na][3],
// out[3..6] of b[nb][4]; out[7] the status word.
__global__ void __launch_bounds__(128) k_energy_sum(const double* a, int64_t na, const double* b, int64_t nb,
                                                     const unsigned* status, double* out)
{
    if (threadIdx.x == 0) out[7] = (double)*status;
    double v[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int64_t k = threadIdx.x; k < na; k += blockDim.x)
        for (int c = 0; c < 3; ++c) v[c] += a[3 * k + c];
    for (int64_t k = threadIdx.x; k < nb; k += blockDim.x)
        for (int c = 0; c < 4; ++c) v[3 + c] += b[4 * k + c];
    block_sums<7>(v, out);
}

typedef void (*energy_pairs_t)(Dev, const double*, double*);

template <int BC>
static energy_pairs_t energy_pairs(const Dev& d)
{
    const bool lj = d.pots & NBG_POT_LJ, el = d.pots & NBG_POT_EL, g = d.pots & NBG_POT_GRAV;
    if (g) return lj ? (el ? k_energy_pairs<BC, true, true, true> : k_energy_pairs<BC, true, false, true>)
                     : (el ? k_energy_pairs<BC, false, true, true> : k_energy_pairs<BC, false, false, true>);
    if (lj) return el ? k_energy_pairs<BC, true, true, false> : k_energy_pairs<BC, true, false, false>;
    return k_energy_pairs<BC, false, true, false>;
}

// out_host: kinetic, lj, el, bonds, angles, gravity, sum m v^2, status word
int launch_energy(nbg_ctx* c, const StateView& s, double* out_host)
{
    const Dev& d = c->d;
    const bool list = c->path == PATH_LIST && c->nrep == 1;
    const bool any_pairs = (d.pots & (NBG_POT_LJ | NBG_POT_EL | NBG_POT_GRAV)) != 0;
    // list: four warps per SM sub-partition (FP64 needs few), so that each
    // fills its queue many times; all pairs: a block per item, up to 16 an SM
    const int64_t gp = list ? std::min<int64_t>((c->n + EL_WARPS - 1) / EL_WARPS, 2 * (int64_t)c->sms)
                       : any_pairs ? std::min<int64_t>((c->n + EB - 1) / EB * ((c->n + EJ - 1) / EJ), 16 * (int64_t)c->sms)
                                   : 0;
    const int64_t gl = std::min<int64_t>((c->n + EB - 1) / EB, 2 * (int64_t)c->sms);
    // block partials, then the seven sums
    const int64_t need = 3 * gp + 4 * gl + 8;
    if (c->energy_cap < need) {
        if (c->energy_buf) cudaFree(c->energy_buf);
        c->energy_buf = nullptr;
        c->energy_cap = 0;
        cudaError_t e = cudaMalloc((void**)&c->energy_buf, sizeof(double) * (size_t)need);
        if (e != cudaSuccess) {
            c->energy_buf = nullptr;
            return cuda_fail(c, e, "energy scratch");
        }
        c->energy_cap = need;
    }
    double* const part = c->energy_buf + 8;
    if (list) {
        // a list for exactly these positions
        int st = launch_pack(c, s);
        if (st) return st;
        if ((st = launch_list_build(c, s, true, StepRef{0, nullptr}))) return st;
        k_energy_list<<<(unsigned)gp, EL_WARPS * 32, 0, c->stream>>>(d, s.x, part);
        NBG_LAUNCH_CHECK(c, "k_energy_list");
    } else if (any_pairs) {
        const energy_pairs_t k = d.bc == NBG_BC_CUBIC      ? energy_pairs<NBG_BC_CUBIC>(d)
                                 : d.bc == NBG_BC_PERIODIC ? energy_pairs<NBG_BC_PERIODIC>(d)
                                                           : energy_pairs<NBG_BC_INFINITE>(d);
        k<<<(unsigned)gp, EB, 0, c->stream>>>(d, s.x, part);
        NBG_LAUNCH_CHECK(c, "k_energy_pairs");
    }
    k_energy_local<<<(unsigned)gl, EB, 0, c->stream>>>(d, s.x, s.v, part + 3 * gp);
    NBG_LAUNCH_CHECK(c, "k_energy_local");
    k_energy_sum<<<1, 128, 0, c->stream>>>(part, gp, part + 3 * gp, gl, d.status, c->energy_buf);
    NBG_LAUNCH_CHECK(c, "k_energy_sum");
    double h[8];
    cudaError_t e = cudaMemcpyAsync(h, c->energy_buf, sizeof h, cudaMemcpyDeviceToHost, c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "energy copy");
    e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "energy sync");
    double lj = h[0], el = h[1];
    const double g = h[2], ke = h[3], mv2 = h[4], eb = h[5], ea = h[6];
    if (list) {
        // every pair's beyond-cutoff term: LJ(R) per LJ pair, q_i q_j / R per charge pair
        double s6R = d.lj_sig2_d / d.lj_R2;
        s6R = s6R * s6R * s6R;
        if (d.pots & NBG_POT_LJ) lj += (double)c->lj_pairs * (s6R * s6R - s6R);
        if (d.pots & NBG_POT_EL) el += c->el_pair_qq / d.el_R;
    }
    out_host[0] = ke;
    out_host[1] = (d.pots & NBG_POT_LJ) ? 4.0 * d.lj_eps * lj : 0.0;
    out_host[2] = (d.pots & NBG_POT_EL) ? el * d.el_k_d : 0.0;
    out_host[3] = d.kind == NBG_SYSTEM_WATER ? eb / 4.0 : 0.0;
    out_host[4] = d.kind == NBG_SYSTEM_WATER ? ea / 2.0 : 0.0;
    out_host[5] = (d.pots & NBG_POT_GRAV) ? -d.G * g : 0.0;
    out_host[6] = mv2;
    out_host[7] = h[7];
    return NBG_OK;
}

// Pair-set export: every ordered pair the force kernels count as inside the
// cutoff of `which` (NBG_POT_LJ or NBG_POT_EL), same classification code
// (fx: the fixed-point kernel's, fx_pair.cuh; else pair_cutoff's).
__global__ void k_pairs(Dev d, StateView s, int which, int use_list, int fx, int* out_j, int* out_cnt, int64_t cap)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < d.n; i += (int64_t)gridDim.x * blockDim.x) {
        const RepDev& R = d.reps[d.rep_of[i]];
        float4 hi = d.phi[i], lo = d.plo[i];
        int64_t cnt = 0;
        int64_t m = use_list ? d.nbr_count[i] : (R.atom0 + R.n);
        const bool water = d.kind == NBG_SYSTEM_WATER;
        const bool lj_i = (d.pots & NBG_POT_LJ) && (!water || (i % 3) == 0);
        for (int64_t k = use_list ? 0 : R.atom0; k < m; ++k) {
            int64_t j = use_list ? dbg_index(d.nbr[k * d.nbr_kstride + i * d.nbr_istride], d.n, (int)i, d.status) : k;
            if (j == i) continue;
            bool in;
            if (fx) {
                const bool lp = lj_i && (!water || fx_oxygen((int)j));
                const bool ep = (d.pots & NBG_POT_EL) != 0;
                float dx, dy, dz;
                const float r2 = fx_r2(d.pfx[i], d.pfx[j], dx, dy, dz);
                bool lj_in, el_in, amb;
                fx_classify(r2, lp, ep, R.fx_lj_lo, R.fx_lj_hi, R.fx_el_lo, R.fx_el_hi, lj_in, el_in, amb);
                if (amb) {
                    const FxPair o = fx_pair_fallback(d, s.x, i, j, lp, ep);
                    if (o.range_err) status_set(d.status, ST_RANGE);
                    lj_in = o.lj_in;
                    el_in = o.el_in;
                }
                in = which == NBG_POT_LJ ? lj_in : el_in;
            } else {
                PairOut o = pair_cutoff(d, R, PairK(R), i, j, hi, lo, d.phi[j], d.plo[j], 0.0f, s.x);
                if (o.range_err) status_set(d.status, ST_RANGE);
                in = which == NBG_POT_LJ ? o.lj_in : o.el_in;
            }
            if (in) {
                if (cnt < cap) out_j[i * cap + cnt] = (int)j;
                ++cnt;
            }
        }
        out_cnt[i] = (int)cnt;
    }
}

int launch_pairs(nbg_ctx* c, const StateView& s, int which, int* out_j, int* out_cnt, int64_t cap_per_atom)
{
    k_pairs<<<grid_for(c->n, 128), 128, 0, c->stream>>>(c->d, s, which, c->path == PATH_LIST ? 1 : 0,
                                                        c->fx_ready ? 1 : 0, out_j, out_cnt, cap_per_atom);
    NBG_LAUNCH_CHECK(c, "k_pairs");
    return NBG_OK;
}
