// Neighbour-sum passes of the PBF substep for sm_100a: density and lambda (with
// the warm-start features in the first pass of a substep), the position
// correction, curl, and vorticity confinement + XSPH.
//
// Reference kernels replaced (kernels/cudaPBFSolver.cu): calculateLambda
// :156-180, calculateOffset :182-199, updatePosition :15-22, calculateCurl
// :201-215, calculateVorticityAndViscosity :217-239, applyVorticityAndViscosity
// :24-29.
//
// Pair lanes. A particle's neighbour list is split over P = L * V lanes: L
// consecutive threads of a warp (a team), each evaluating V = 1 or 2 pairs per
// instruction. With V = 2 the pair arithmetic runs on the sm_100 packed FP32
// operations (add/mul/fma.rn.f32x2), each component of which is the scalar
// IEEE operation, so one instruction evaluates two pairs and the
// per-pair results are the scalar ones bit for bit. Lane p = V t + v (thread t,
// component v) takes list entries p, p + P, p + 2P, ... in list order; the lane
// sums are combined by an xor butterfly over distances 1, 2, 4 (first the two
// components of a thread, then across the team by shuffles), which gives
// ((s0 + s1) + (s2 + s3)) + ... on every lane. pair_lanes = P selects
// (L, V): 1 = (1, 1), 2 = (1, 2), 4 = (2, 2), 8 = (4, 2).
//
// The search pads every list to whole batches with the padding slot (KParams::pad_slot,
// a position no particle comes near). A padding entry contributes +0 or -0 to every
// sum, which leaves the sum unchanged: no accumulator is ever -0 (they start at +0,
// and in round-to-nearest x + (-x) = +0 and +0 + (-0) = +0). So no entry is tested
// for the end of its list, but for the correction with an s_corr exponent that is not
// a small whole number: a negative one takes a padding entry's weight of 0 to infinity,
// which times a gradient of 0 is no zero.
#include "pbf_kernels.h"
#include "pbf_mlp.h"
#include "pbf_mlp_dev.cuh"
#include "pbf_launch.cuh"
#include "pbf_packed.cuh"

#include <algorithm>
#include <type_traits>

namespace pbf {

// one truth value per component, and the components where it holds (+0 elsewhere)
struct bool2v {
    bool x, y;
};
__device__ __forceinline__ float keep_only(float a, bool k) { return k ? a : 0.0f; }
__device__ __forceinline__ float2 keep_only(float2 a, bool2v k) { return make_float2(k.x ? a.x : 0.0f, k.y ? a.y : 0.0f); }
// lo <= a <= hi
__device__ __forceinline__ bool within(float a, float lo, float hi) { return !(a < lo) && !(a > hi); }
__device__ __forceinline__ bool2v within(float2 a, float lo, float hi) { return {within(a.x, lo, hi), within(a.y, lo, hi)}; }
__device__ __forceinline__ bool below(float a, float s, bool valid) { return a < s && valid; }
__device__ __forceinline__ bool2v below(float2 a, float s, bool2v valid) { return {a.x < s && valid.x, a.y < s && valid.y}; }
// which components are entries of a list with `left` of them left
__device__ __forceinline__ bool entries_left(float, int left) { return left > 0; }
__device__ __forceinline__ bool2v entries_left(float2, int left) { return {left > 0, left > 1}; }
// which components are gathered particles, not the padding slot
__device__ __forceinline__ bool is_entry(const float4 (&a)[1]) { return a[0].x != PAD_POSITION; }
__device__ __forceinline__ bool2v is_entry(const float4 (&a)[2]) { return {a[0].x != PAD_POSITION, a[1].x != PAD_POSITION}; }
// the first butterfly step: the two lanes of a thread
__device__ __forceinline__ float fold(float a) { return a; }
__device__ __forceinline__ float fold(float2 a) { return a.x + a.y; }

// Negated pbf_rsqrt (pbf_device.cuh) on each component, without a negation:
// the steps y <- y fma(-x/2, y^2, 3/2) take -x/2 as the product (-0.5) x, and the
// last step multiplies by fma(x/2, y^2, -3/2) = -fma(-x/2, y^2, 3/2) (round to
// nearest is symmetric in sign), which yields exactly -pbf_rsqrt(x).
__device__ __forceinline__ unsigned rsqrt_seed(float x) { return 0x5f3759df - (__float_as_int(x) >> 1); }
__device__ __forceinline__ float rsqrt_seed_v(float x) { return __int_as_float(rsqrt_seed(x)); }
__device__ __forceinline__ float2 rsqrt_seed_v(float2 x) {
    return make_float2(__int_as_float(rsqrt_seed(x.x)), __int_as_float(rsqrt_seed(x.y)));
}
template <typename T> __device__ __forceinline__ T vrsqrt_neg(T x) {
    const T hx = vmul(bc<T>(0.5f), x);
    const T nhx = vmul(bc<T>(-0.5f), x);
    T y = rsqrt_seed_v(x);
#pragma unroll
    for (int i = 0; i < 2; ++i) y = vmul(y, vfma(nhx, vmul(y, y), bc<T>(1.5f)));
    return vmul(y, vfma(hx, vmul(y, y), bc<T>(-1.5f)));
}

template <typename T> struct T3 {
    T x, y, z;
};
template <typename T> __device__ __forceinline__ T3<T> add3(const T3<T>& a, const T3<T>& b) {
    return {vadd(a.x, b.x), vadd(a.y, b.y), vadd(a.z, b.z)};
}
template <typename T> __device__ __forceinline__ T3<T> zero3() { return {bc<T>(0.0f), bc<T>(0.0f), bc<T>(0.0f)}; }
__device__ __forceinline__ f3 fold3(const T3<float>& a) { return {a.x, a.y, a.z}; }
__device__ __forceinline__ f3 fold3(const T3<float2>& a) { return {fold(a.x), fold(a.y), fold(a.z)}; }
// The curl's cross product, one fused multiply-add per component:
// (fma(a_y, b_z, -(a_z b_y)), fma(a_z, b_x, -(a_x b_z)), fma(a_x, b_y, -(a_y b_x))).
// (A packed multiply whose only use is an add may be fused by the code generator,
// so every product that meets an addition in these passes is an explicit fma.)
// -(a b) is taken as (a b) (-1), which is the same value, signed zeros included.
template <typename T> __device__ __forceinline__ T3<T> cross3v(const T3<T>& a, const T3<T>& b) {
    const T m1 = bc<T>(-1.0f);
    return {vfma(a.y, b.z, vmul(vmul(a.z, b.y), m1)), vfma(a.z, b.x, vmul(vmul(a.x, b.z), m1)),
            vfma(a.x, b.y, vmul(vmul(a.y, b.x), m1))};
}

// .w of V gathered float4s as one packet
__device__ __forceinline__ float packw(const float4 (&a)[1]) { return a[0].w; }
__device__ __forceinline__ float2 packw(const float4 (&a)[2]) { return make_float2(a[0].w, a[1].w); }

// a - b_v for the xyz of V gathered float4s: one scalar subtraction per component,
// which leaves the V results side by side (packing the gathered registers first
// takes more instructions than it saves)
__device__ __forceinline__ T3<float> diff3(const f3& a, const float4 (&b)[1]) {
    return {a.x - b[0].x, a.y - b[0].y, a.z - b[0].z};
}
__device__ __forceinline__ T3<float2> diff3(const f3& a, const float4 (&b)[2]) {
    return {make_float2(a.x - b[0].x, a.x - b[1].x), make_float2(a.y - b[0].y, a.y - b[1].y),
            make_float2(a.z - b[0].z, a.z - b[1].z)};
}
// b_v - a
__device__ __forceinline__ T3<float> rdiff3(const float4 (&b)[1], const f3& a) {
    return {b[0].x - a.x, b[0].y - a.y, b[0].z - a.z};
}
__device__ __forceinline__ T3<float2> rdiff3(const float4 (&b)[2], const f3& a) {
    return {make_float2(b[0].x - a.x, b[1].x - a.x), make_float2(b[0].y - a.y, b[1].y - a.y),
            make_float2(b[0].z - a.z, b[1].z - a.z)};
}
// a + w_v
__device__ __forceinline__ float addw(float a, const float4 (&b)[1]) { return a + b[0].w; }
__device__ __forceinline__ float2 addw(float a, const float4 (&b)[2]) {
    return make_float2(a + b[0].w, a + b[1].w);
}

template <int V> using vec_t = typename std::conditional<V == 1, float, float2>::type;

// r = x_k - x_j, |r|^2 = fma(z, z, fma(y, y, x*x)), Wpoly6 (when NEED_W) and the
// spiky gradient of V pairs, exactly as w_poly6 / grad_spiky (pbf_device.cuh)
// evaluate one pair.
// Every difference a - b is fma(b, -1, a), which rounds the same exact value
// once (signed zeros included), and the rsqrt comes negated (ny = -y), so no
// operand needs a negation of its own: h - |r| = fma(|r|^2, ny, h), |r| > h is
// |r|^2 ny < -h, and ((c d) d) y = ((-c d) d) ny. The poly6 cutoff |r|^2 > h^2
// is max(h^2 - |r|^2, +0) (the difference is negative exactly when the same
// rounded |r|^2 exceeds h^2, and c (+0)^3 = +0). A padding entry is the padding
// slot, far from every particle: its weight is c (+0)^3 and the cutoff drops its
// gradient, so it gives w = +0 and g = +0 or -0.
template <typename T, bool NEED_W, int V>
__device__ __forceinline__ void pair_terms(const KParams& p, const f3& xk, const float4 (&xj)[V], T3<T>& r, T& w,
                                           T3<T>& g) {
    const T m1 = bc<T>(-1.0f);
    r = diff3(xk, xj);
    const T r2 = vfma(r.z, r.z, vfma(r.y, r.y, vmul(r.x, r.x)));
    if (NEED_W) {
        const T t = vmax(vfma(r2, m1, bc<T>(p.h2)), 0.0f);
        // c t^3 as fma(c, t^3, +0), the same value (c t^3 is never -0): the density
        // sum adds w, and a packed product whose only use is an addition may be fused
        // into it by the code generator
        w = vfma(bc<T>(p.poly6_c), vmul(vmul(t, t), t), bc<T>(0.0f));
    }
    const T ny = vrsqrt_neg(vmax(r2, 1e-30f));
    const T nrl = vmul(r2, ny);               // -|r| for the cutoff
    const T d = vfma(r2, ny, bc<T>(p.h));      // h - |r|
    const T s = vmul(vmul(vmul(bc<T>(-p.spiky_c), d), d), ny);
    // the mask on the magnitude: a dropped pair gives a gradient of +0 or -0,
    // which leaves every sum it enters unchanged (no accumulator is ever -0)
    const T sk = keep_only(s, within(nrl, -p.h, -p.rmin));
    g = {vmul(sk, r.x), vmul(sk, r.y), vmul(sk, r.z)};
}

// The dp pair weight (lambda_i + lambda_j) + s_corr (cu:193-195, Scorr cuh:142-144)
// as fma(-k (W / W(dq))^n, scorr_scale, lambda_i + lambda_j).
__device__ __forceinline__ float vpow(float q, const KParams& p) { return powf(q, p.n_exp); }
__device__ __forceinline__ float2 vpow(float2 q, const KParams& p) {
    return make_float2(powf(q.x, p.n_exp), powf(q.y, p.n_exp));
}
// N4: the usual n = 4, ((q q) q) q, as a constant, so that the pair loop has no
// branch and the pairs of a batch overlap.
template <bool N4, typename T> __device__ __forceinline__ T dp_weight(const KParams& p, T lij, T w) {
    const T q = vmul(w, bc<T>(p.inv_wdq));
    T pw;
    if (N4) {
        pw = vmul(vmul(vmul(q, q), q), q);
    } else if (p.n_int > 0) {
        pw = q;
        for (int i = 1; i < p.n_int; ++i) pw = vmul(pw, q);
    } else {
        pw = vpow(q, p);
    }
    return vfma(vmul(bc<T>(p.nk), pw), bc<T>(p.scorr_scale), lij);
}

// ---- teams -------------------------------------------------------------------
template <int L> struct Team {
    int k;          // particle slot
    int t;          // thread within the team
    unsigned mask;  // the team's lanes within the warp
};

// blockDim.x is a multiple of 32, so a team never straddles a warp. vb is the
// virtual block: blockIdx.x for one block per tile of slots, or one of the tiles
// a persistent block strides over.
template <int L> __device__ __forceinline__ Team<L> team_of(int vb) {
    Team<L> m;
    const long long g = (long long)vb * blockDim.x + threadIdx.x;
    m.k = (int)(g / L);
    m.t = (int)(threadIdx.x & (L - 1));
    const int lane = threadIdx.x & 31;
    m.mask = L >= 32 ? 0xffffffffu : (((1u << L) - 1u) << (lane & ~(L - 1)));
    return m;
}

// the butterfly across the team (distances 1, 2 between threads)
template <int L> __device__ __forceinline__ float team_sum(float v, unsigned mask) {
#pragma unroll
    for (int o = 1; o < L; o <<= 1) v += __shfl_xor_sync(mask, v, o);
    return v;
}
template <int L> __device__ __forceinline__ f3 team_sum3(f3 v, unsigned mask) {
    return {team_sum<L>(v.x, mask), team_sum<L>(v.y, mask), team_sum<L>(v.z, mask)};
}

// Entries q0 + u P + v (u < B, v < V) of slot k's (padded) list. All index loads of
// a batch are issued before the gathers that depend on them.
template <int V, int P, int B>
__device__ __forceinline__ void load_idx(const KParams& p, const int* __restrict__ nbr, int k, int q0,
                                         int (&jj)[B][V]) {
#pragma unroll
    for (int u = 0; u < B; ++u)
#pragma unroll
        for (int v = 0; v < V; ++v) jj[u][v] = nbr[(size_t)(q0 + u * P + v) * p.stride + k];
}

// How a pass's inner loop is laid out. A batch of E entries per thread has its
// gathers issued together and no branch inside, so the pairs of a batch overlap (a
// test per entry for the end of the list kept them apart: a step then took the whole latency of its arithmetic;
// 1 M particles, lambda: 81.6 us with the test, 68.9 without; 32,768 particles: 8.1
// and 6.2).
//   full device: four entries in the one-array passes, two in the two-array ones,
//     which then keep their next indices in registers at four blocks per SM (1 M
//     particles: curl 107 -> 102 us, vorticity 129 -> 118); the correction fits
//     five blocks (84.8 -> 71.6), lambda is faster at four (69 against 71.5);
//   ROOMY, all blocks resident at three per SM: four entries everywhere and
//     registers for it (32,768 particles: lambda 6.0 -> 5.9 us, correction 6.6 ->
//     5.8, curl 10.4 -> 6.7, vorticity 11 -> 8.3).
constexpr int ROOMY_BLOCKS = 3;

// body(xj, vj) for the neighbours of slot k that thread t of its team
// takes, gathered from NA arrays through the list of slots, E entries per batch; the
// next batch's indices load while a batch computes.
template <int L, int V, int E, int NA, typename F>
__device__ __forceinline__ void for_list(const KParams& p, const int* __restrict__ nbr, int k, int t, int cnt,
                                         const float4* __restrict__ a, const float4* __restrict__ b, F&& body) {
    constexpr int P = L * V, B = E / V;
    int jj[B][V];
    if (cnt > 0) load_idx<V, P, B>(p, nbr, k, V * t, jj);
    // (every thread of a team runs the same batches: the lists are padded for it)
    for (int q0 = 0; q0 < cnt; q0 += P * B) {
        float4 xj[B][V], vj[B][V];
#pragma unroll
        for (int u = 0; u < B; ++u)
#pragma unroll
            for (int c = 0; c < V; ++c) {
                xj[u][c] = a[jj[u][c]];
                if (NA == 2) vj[u][c] = b[jj[u][c]];
            }
        if (q0 + P * B < cnt) load_idx<V, P, B>(p, nbr, k, q0 + P * B + V * t, jj);
#pragma unroll
        for (int u = 0; u < B; ++u) body(xj[u], vj[u]);
    }
}

// Block-wide max and sum of a per-thread error, folded into one slot with a
// single pair of atomics per block (max as ordered double bits, value >= 0).
__device__ __forceinline__ void block_error_reduce(float e, double esum, unsigned long long* max_bits, double* sum) {
    __shared__ float s_max[32];
    __shared__ double s_sum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float m = e;
    double s = esum;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        s += __shfl_xor_sync(0xffffffffu, s, o);
    }
    if (lane == 0) { s_max[warp] = m; s_sum[warp] = s; }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        double dsum = 0.0;
        for (int w = 0; w < nw; ++w) { m = fmaxf(m, s_max[w]); dsum += s_sum[w]; }
        atomicMax(max_bits, (unsigned long long)__double_as_longlong((double)m));
        atomicAdd(sum, dsum);
    }
    __syncthreads();  // a persistent block's next tile writes s_max / s_sum again
}

// ---------------------------------------------------------------------------
// a9: density, constraint and lambda (calculateLambda cu:156-180), with the
// one-sided density error of the positions it sees
// ---------------------------------------------------------------------------
// Lambda of slot k from its combined fluid density and gradient sums: the wall
// term, the constraint and the denominator. rhos gains the wall term; err is
// the one-sided error of the fluid density alone.
__device__ __forceinline__ float lambda_tail(const KParams& p, int k, const f3& xk, float& rhos, float gms, f3 g3,
                                             float& err) {
    err = fmaxf(__fdiv_rn(rhos, p.rho0) - 1.0f, 0.0f);
    if (p.flags & FLAG_WALL_DENSITY) {
        f3 gw;
        rhos = rhos + wall_term(p, scene_of(p, k), xk, gw);
        g3 = {g3.x + gw.x, g3.y + gw.y, g3.z + gw.z};
    }
    float C = __fdiv_rn(rhos, p.rho0) - 1.0f;
    if (p.flags & FLAG_CLAMP_C) C = fmaxf(C, 0.0f);
    gms = __fmaf_rn(g3.x, g3.x, gms);
    gms = __fmaf_rn(g3.y, g3.y, gms);
    gms = __fmaf_rn(g3.z, g3.z, gms);
    gms = __fdiv_rn(gms, p.rho0sq);
    return __fdiv_rn(-C, gms + p.eps);
}

// The sums of one pair of the lambda pass.
template <typename T> struct LambdaSums {
    T rho, gm;
    T3<T> gs;
};
template <typename T> __device__ __forceinline__ LambdaSums<T> lambda_zero() {
    return {bc<T>(0.0f), bc<T>(0.0f), zero3<T>()};
}
template <typename T, int V>
__device__ __forceinline__ void lambda_pair(const KParams& p, const f3& xk, const float4 (&xj)[V],
                                            LambdaSums<T>& s) {
    T3<T> r, g;
    T w;
    pair_terms<T, true>(p, xk, xj, r, w, g);
    s.rho = vadd(s.rho, w);
    s.gs = add3(s.gs, g);
    s.gm = vfma(g.x, g.x, s.gm);
    s.gm = vfma(g.y, g.y, s.gm);
    s.gm = vfma(g.z, g.z, s.gm);
}
// The team's sums combined and slot k's lambda written; returns the density
// error on the team's first thread, 0 on the others.
template <bool DEBUG, int L, int V>
__device__ __forceinline__ float lambda_store(const KParams& p, const Team<L>& tm, const f3& xk,
                                              const LambdaSums<vec_t<V>>& s, float4* __restrict__ xl,
                                              float* __restrict__ rho_out, const IterCtl& ctl) {
    float rhos = team_sum<L>(fold(s.rho), tm.mask);
    const float gms = team_sum<L>(fold(s.gm), tm.mask);
    const f3 g3 = team_sum3<L>(fold3(s.gs), tm.mask);
    float err = 0.0f;
    if (tm.t == 0) {
        const int k = tm.k;
        const float lam = lambda_tail(p, k, xk, rhos, gms, g3, err);
        xl[k] = make_float4(xk.x, xk.y, xk.z, lam);
        if (ctl.lam_acc) ctl.lam_acc[k] += lam;
        if (DEBUG) rho_out[k] = rhos;
    }
    return err;
}
template <bool DEBUG, int L, int V>
__device__ __forceinline__ float lambda_list(const KParams& p, const Team<L>& tm, const float4* __restrict__ x,
                                             const int* __restrict__ nbr, const int* __restrict__ ncnt,
                                             float4* __restrict__ xl, float* __restrict__ rho_out,
                                             const IterCtl& ctl) {
    using T = vec_t<V>;
    const f3 xk = make3(x[tm.k]);
    LambdaSums<T> s = lambda_zero<T>();
    for_list<L, V, 4, 1>(p, nbr, tm.k, tm.t, ncnt[tm.k], x, x,
                            [&](const float4(&xj)[V], const float4(&)[V]) {
                                lambda_pair<T, V>(p, xk, xj, s);
                            });
    return lambda_store<DEBUG, L, V>(p, tm, xk, s, xl, rho_out, ctl);
}

// Adaptive loop: true when it has ended. In the device-side loop it also hands the
// delta-p pass its counter.
__device__ __forceinline__ bool lambda_skip(const IterCtl& ctl) {
    if (ctl.loop_next && blockIdx.x == 0 && threadIdx.x == 0) *ctl.loop_next = *ctl.loop_k + ctl.loop_add;
    return ctl.done && (*ctl.done || ctl.past_end());
}

// nvb tiles of blockDim.x slots' teams; the grid strides over them (a grid of
// nvb blocks is the ordinary one-block-per-tile launch)
template <bool DEBUG, bool ROOMY, int L, int V>
__global__ void __launch_bounds__(256, ROOMY ? ROOMY_BLOCKS : 4) k_lambda(KParams p, int nvb, const float4* __restrict__ x,
                                                                const int* __restrict__ nbr,
                                                                const int* __restrict__ ncnt, float4* __restrict__ xl,
                                                                float* __restrict__ rho_out, IterCtl ctl) {
    pdl_wait();
    if (lambda_skip(ctl)) return;
    for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x) {
        const Team<L> tm = team_of<L>(vb);
        float err = 0.0f;
        if (tm.k < p.n) err = lambda_list<DEBUG, L, V>(p, tm, x, nbr, ncnt, xl, rho_out, ctl);
        if (ctl.max_bits) {
            const int sl = ctl.cur_slot();
            block_error_reduce(err, err, ctl.max_bits + sl, ctl.sum + sl);
        }
    }
}

// ---------------------------------------------------------------------------
// a17: warm-start features (no reference counterpart), computed in the first
// lambda pass of a substep together with that pass's lambda (the same
// arithmetic as k_lambda, so recording features changes no result):
//   0 neighbour count / cap          1 fluid density / rho0
//   2 previous substep's total lambda
//   3 sum |grad C|^2 (the lambda denominator without eps)
//   4 velocity divergence sum (v_j - v_i) . grad W / rho0 (predicted velocities)
//   5-7 distance to the nearer wall per axis / h, clamped to [0, 4]
//   8 neighbours closer than h/2, / cap
//   9 |sum of (x_i - x_j)| / (h max(count, 1))  (offset of the neighbourhood)
//   10 |sum grad W| h / rho0
//   11 sum |v_j - v_i|^2 (dt / h)^2 / max(count, 1)
// None depends on the grid's cell size. lam_acc starts the substep's total lambda
// at this pass's lambda.
// ---------------------------------------------------------------------------
// One team's particle: writes xl[k] = (x, plain lambda), lam_acc[k] = lambda
// and, when feat is not null, the 12 features; returns true on the team's first
// thread (with the features in f and the plain lambda in lam) when k < n.
template <int L, int V>
__device__ __forceinline__ bool features_one(const KParams& p, const Team<L>& tm, const float4* __restrict__ x,
                                             const float4* __restrict__ v, const int* __restrict__ nbr,
                                             const int* __restrict__ ncnt, const float* __restrict__ lam_prev,
                                             float4* __restrict__ xl, float* __restrict__ feat,
                                             float* __restrict__ lam_acc, float (&f)[12], float& lam) {
    using T = vec_t<V>;
    constexpr int P = L * V, B = 2 / V;
    const int k = tm.k;
    if (k >= p.n) return false;  // uniform over the team
    const f3 xk = make3(x[k]);
    const f3 vk = make3(v[k]);
    const int cnt = ncnt[k];
    T rho = bc<T>(0.0f), gm = bc<T>(0.0f), div = bc<T>(0.0f), close = bc<T>(0.0f), dv2 = bc<T>(0.0f);
    T3<T> gs = zero3<T>(), rs = zero3<T>();
    const float q2 = 0.25f * p.h2;
    int jj[B][V];
    if (cnt > 0) load_idx<V, P, B>(p, nbr, k, V * tm.t, jj);
    for (int q0 = 0; q0 < cnt; q0 += P * B) {
        float4 xj[B][V], vj[B][V];
#pragma unroll
        for (int u = 0; u < B; ++u)
#pragma unroll
            for (int c = 0; c < V; ++c) {
                xj[u][c] = x[jj[u][c]];
                vj[u][c] = v[jj[u][c]];
            }
        // the next batch's indices load while this batch computes
        if (q0 + P * B < cnt) load_idx<V, P, B>(p, nbr, k, q0 + P * B + V * tm.t, jj);
#pragma unroll
        for (int u = 0; u < B; ++u) {
            const auto valid = entries_left(T{}, cnt - (q0 + u * P + V * tm.t));
            T3<T> r, g;
            T w;
            pair_terms<T, true>(p, xk, xj[u], r, w, g);
            rho = vadd(rho, w);
            gs = add3(gs, g);
            gm = vfma(g.x, g.x, gm);
            gm = vfma(g.y, g.y, gm);
            gm = vfma(g.z, g.z, gm);
            const T3<T> vji = rdiff3(vj[u], vk);
            div = vfma(vji.x, g.x, div);
            div = vfma(vji.y, g.y, div);
            div = vfma(vji.z, g.z, div);
            const T r2 = vfma(r.z, r.z, vfma(r.y, r.y, vmul(r.x, r.x)));
            close = vadd(close, keep_only(bc<T>(1.0f), below(r2, q2, valid)));
            rs = add3(rs, T3<T>{keep_only(r.x, valid), keep_only(r.y, valid), keep_only(r.z, valid)});
            dv2 = vadd(dv2, keep_only(vfma(vji.z, vji.z, vfma(vji.y, vji.y, vmul(vji.x, vji.x))), valid));
        }
    }
    float rhos = team_sum<L>(fold(rho), tm.mask);
    float gms = team_sum<L>(fold(gm), tm.mask);
    f3 g3 = team_sum3<L>(fold3(gs), tm.mask);
    const float divs = team_sum<L>(fold(div), tm.mask);
    const float closes = team_sum<L>(fold(close), tm.mask);
    const f3 r3 = team_sum3<L>(fold3(rs), tm.mask);
    const float dv2s = team_sum<L>(fold(dv2), tm.mask);
    if (tm.t != 0) return false;
    const SceneView sc = scene_of(p, k);
    const float rho_fluid = rhos;
    const float gsl = __fsqrt_rn(dot_fma(g3, g3));
    if (p.flags & FLAG_WALL_DENSITY) {
        f3 gw;
        rhos = rhos + wall_term(p, sc, xk, gw);
        g3 = {g3.x + gw.x, g3.y + gw.y, g3.z + gw.z};
    }
    float C = __fdiv_rn(rhos, p.rho0) - 1.0f;
    if (p.flags & FLAG_CLAMP_C) C = fmaxf(C, 0.0f);
    gms = __fmaf_rn(g3.x, g3.x, gms);
    gms = __fmaf_rn(g3.y, g3.y, gms);
    gms = __fmaf_rn(g3.z, g3.z, gms);
    gms = __fdiv_rn(gms, p.rho0sq);
    lam = __fdiv_rn(-C, gms + p.eps);
    xl[k] = make_float4(xk.x, xk.y, xk.z, lam);
    lam_acc[k] = lam;

    const float inv_cnt = 1.0f / (float)max(cnt, 1);
    f[0] = (float)cnt / (float)p.max_nbr;
    f[1] = rho_fluid / p.rho0;
    f[2] = lam_prev[k];
    f[3] = gms;
    f[4] = divs / p.rho0;
    const float qa[3] = {xk.x, xk.y, xk.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float dw = fminf(qa[a] - sc.bmin[a], sc.bmax[a] - qa[a]) * p.inv_h;
        f[5 + a] = fminf(fmaxf(dw, 0.0f), 4.0f);
    }
    f[8] = closes / (float)p.max_nbr;
    f[9] = __fsqrt_rn(dot_fma(r3, r3)) * p.inv_h * inv_cnt;
    f[10] = gsl * p.h / p.rho0;
    const float dth = p.dt * p.inv_h;
    f[11] = dv2s * (dth * dth) * inv_cnt;
    if (feat) {
#pragma unroll
        for (int i = 0; i < 12; ++i) feat[(size_t)k * 12 + i] = f[i];
    }
    return true;
}

// The network's input row of a particle: its normalised features as BF16, padded
// from 12 to 16 with zeros. norm: the network's biases and constants.
__device__ __forceinline__ void pack_row(const float (&f)[12], const float* norm, uint32_t (&pk)[8]) {
    float xf[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) xf[i] = 0.0f;
#pragma unroll
    for (int i = 0; i < MLP_IN; ++i) xf[i] = (f[i] - norm[FMEAN_OFF + i]) * norm[FISTD_OFF + i];
#pragma unroll
    for (int i = 0; i < 8; ++i)
        pk[i] = (uint32_t)bf16_bits(xf[2 * i]) | ((uint32_t)bf16_bits(xf[2 * i + 1]) << 16);
}

// ROWS: also writes the particle's network input, entries 0-7 to row_lo and 8-15
// to row_hi, for k_warm_rows. Two
// entries per batch and four blocks per SM, as the two-array passes: 34.7 us at
// 262,144 particles; two entries without the bound 42.6, four entries 36.2 at three
// blocks and 45.0 without a bound.
template <bool ROWS, int L, int V>
__global__ void __launch_bounds__(256, 4) k_features(KParams p, int nvb, const float4* __restrict__ x,
                                                  const float4* __restrict__ v, const int* __restrict__ nbr,
                                                  const int* __restrict__ ncnt, const float* __restrict__ lam_prev,
                                                  float4* __restrict__ xl, float* __restrict__ feat,
                                                  float* __restrict__ lam_acc, const float* __restrict__ norm,
                                                  uint4* __restrict__ row_lo, uint4* __restrict__ row_hi) {
    pdl_wait();
    for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x) {
        const Team<L> tm = team_of<L>(vb);
        float f[12], lam;
        const bool have = features_one<L, V>(p, tm, x, v, nbr, ncnt, lam_prev, xl, feat, lam_acc, f, lam);
        if (ROWS && have) {
            uint32_t pk[8];
            pack_row(f, norm, pk);
            row_lo[tm.k] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            row_hi[tm.k] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
    }
}

// ---------------------------------------------------------------------------
// a17, fused: the first lambda pass of a warm-started substep with the network
// in the same kernel. Each block computes its particles' features and plain
// lambda as k_features does; the team leaders write their normalised features
// as BF16 straight into the tensor core's A tile in shared memory (K-major,
// never to HBM), and the block evaluates 12 -> 64 -> 64 -> 64 on the tensor
// cores (one 128-row MMA per tile of rows and layer, issued by one thread,
// accumulated in TMEM, 64 columns per tile) with the GELU epilogues on the CUDA
// cores, then the output layer and the trust region. Thread t runs the
// epilogue of row t: a warp reads its quarter of the TMEM lanes, and the warps
// of the second half of a 256-thread block the second tile's columns. While
// one block waits on its MMAs the SM runs the other resident blocks' gathers.
// The arithmetic is k_mlp_fwd's (same operands, MMA shapes and epilogue), so
// lambda0 is the unfused path's bit for bit. The blocks' shared memory leaves the
// gathers 70 KB of L1: large scenes run the same two halves as k_features and
// k_warm_rows instead.
// ---------------------------------------------------------------------------
struct WarmIO {
    const uint16_t* w;  // BF16 weights (W1 [64][16], W2, W3 [64][64], w4 [64])
    const float* b;     // biases and constants (normalisation, output scale)
    float* lam0;        // lambda0 per slot
    float clamp;        // trust region around the plain lambda (0: none)
    int floor;          // 1: lambda0 at least as strong as the plain lambda
    int* err;           // PBF_DEVERR_MLP_TIMEOUT on an expired tensor-core wait
};

constexpr int FW_SW1 = 0;                     // W1 [64 x 16]  2 KB
constexpr int FW_SW2 = FW_SW1 + 64 * 16 * 2;  // W2 [64 x 64]  8 KB
constexpr int FW_SW3 = FW_SW2 + 64 * 64 * 2;  // W3 [64 x 64]  8 KB
constexpr int FW_SX = FW_SW3 + 64 * 64 * 2;   // X: per tile [128 x 16] BF16, 4 KB; then H: per tile [128 x 64], 16 KB
constexpr int FW_X_TILE = 128 * 16 * 2;
constexpr int FW_H_TILE = 128 * 64 * 2;
__host__ __device__ constexpr int warm_smem_bytes(int tiles) { return FW_SX + tiles * (FW_X_TILE + FW_H_TILE); }

// Stages the weights, biases and the barrier, allocates `cols` TMEM columns and
// returns their base. Called by every thread of the block.
__device__ __forceinline__ uint32_t warm_setup(const WarmIO& io, uint8_t* smem, uint64_t* mbar, uint32_t* tmem_slot,
                                               float* sb, float* sw4, uint32_t cols) {
    const int t = threadIdx.x;
    if (t < 32) tmem_alloc(tmem_slot, cols);
    if (t == 0) mbar_init(mbar, 1);
    stage_weight(smem + FW_SW1, io.w + W1_OFF, 64, 16);
    stage_weight(smem + FW_SW2, io.w + W2_OFF, 64, 64);
    stage_weight(smem + FW_SW3, io.w + W3_OFF, 64, 64);
    for (int i = t; i < MLP_NUM_BIASES; i += blockDim.x) sb[i] = io.b[i];
    if (t < 64) sw4[t] = bf16_val(io.w[W4_OFF + t]);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    return *tmem_slot;
}

// The three hidden layers and the read-out for the rows of `tiles` 128-row tiles:
// layer l reads X (l = 0, tile j at sX + j x_stride) or H and writes H (l < 2).
// Thread t has row t of the block and returns its output in y. synced() runs after
// the barrier that makes the block's X visible. False on an expired wait.
template <typename F>
__device__ __forceinline__ bool warm_layers(const WarmIO& io, const uint8_t* smem, const uint8_t* sX, int x_stride,
                                            uint8_t* sH, int tiles, uint32_t tbase, uint64_t* mbar, uint32_t& phase,
                                            const float* sb, const float* sw4, float& y, F&& synced) {
    const int t = threadIdx.x, warp = t >> 5;
    const bool ep_warp = (warp >> 2) < tiles;  // this warp's TMEM quarter holds rows of a tile
    const uint32_t lane_base = tmem_addr(tbase, 32 * (warp & 3), 64 * (warp >> 2));
    uint8_t* my_h = sH + (warp >> 2) * FW_H_TILE;
    y = sb[B4_OFF];
#pragma unroll 1
    for (int l = 0; l < 3; ++l) {
        sync_for_mma();
        if (l == 0) synced();
        if (t == 0) {
            for (int j = 0; j < tiles; ++j) {
                if (l == 0) gemm_issue(tbase + 64 * j, sX + j * x_stride, smem + FW_SW1, 64, 16, 0);
                else gemm_issue(tbase + 64 * j, sH + j * FW_H_TILE, smem + (l == 1 ? FW_SW2 : FW_SW3), 64, 64, 0);
            }
            commit(mbar);
        }
        if (!wait_mma(mbar, phase, io.err)) return false;
        if (ep_warp) {
            const float* bias = sb + (l == 0 ? B1_OFF : l == 1 ? B2_OFF : B3_OFF);
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                float vv[16];
                tmem_ld16(lane_base + 16 * c, vv);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const float4 bi = *reinterpret_cast<const float4*>(bias + 16 * c + i);
                    const float2 h0 = gelu2(vadd(make_float2(vv[i], vv[i + 1]), make_float2(bi.x, bi.y)));
                    const float2 h1 = gelu2(vadd(make_float2(vv[i + 2], vv[i + 3]), make_float2(bi.z, bi.w)));
                    vv[i] = h0.x;
                    vv[i + 1] = h0.y;
                    vv[i + 2] = h1.x;
                    vv[i + 3] = h1.y;
                }
                if (l < 2) {
                    put_row64(my_h, t & 127, vv, 16 * c);
                } else {
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const float4 w = *reinterpret_cast<const float4*>(sw4 + 16 * c + i);
                        y = __fmaf_rn(vv[i], w.x, y);
                        y = __fmaf_rn(vv[i + 1], w.y, y);
                        y = __fmaf_rn(vv[i + 2], w.z, y);
                        y = __fmaf_rn(vv[i + 3], w.w, y);
                    }
                }
            }
        }
    }
    return true;
}

// Slot k's lambda0 from the network's output y: the trust region around the plain
// lambda of this pass has its sign and at most clamp times its magnitude.
__device__ __forceinline__ void warm_store(const WarmIO& io, const float* sb, int k, float y, float lam_plain,
                                           float4* __restrict__ xl, float* __restrict__ lam_acc) {
    float l0 = y * sb[OSCALE_OFF];
    if (io.clamp > 0.0f) {
        const float a = io.clamp * lam_plain;
        const float f0 = io.floor ? lam_plain : 0.0f;  // the weak end of the interval
        l0 = fminf(fmaxf(l0, fminf(a, f0)), fmaxf(a, f0));
    }
    reinterpret_cast<float*>(xl)[4 * (size_t)k + 3] = l0;
    lam_acc[k] = l0;
    io.lam0[k] = l0;
}

template <int L, int V>
__global__ void __launch_bounds__(256, 3) k_features_warm(KParams p, int nvb, const float4* __restrict__ x,
                                                          const float4* __restrict__ v, const int* __restrict__ nbr,
                                                          const int* __restrict__ ncnt,
                                                          const float* __restrict__ lam_prev,
                                                          float4* __restrict__ xl, float* __restrict__ feat,
                                                          float* __restrict__ lam_acc, WarmIO io) {
    pdl_wait();
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(16) float sb[MLP_NUM_BIASES];
    __shared__ __align__(16) float sw4[64];
    __shared__ float s_lam[256];
    const int t = threadIdx.x;
    const int R = blockDim.x / L;            // particles per tile of slots: rows
    const int tiles = (R + 127) >> 7;        // 128-row MMA tiles
    const uint32_t cols = tiles > 1 ? 128u : 64u;
    uint8_t* sX = smem + FW_SX;
    uint8_t* sH = sX + tiles * FW_X_TILE;
    // rows of the last tile past R stay zero
    for (int i = t; i < tiles * FW_X_TILE / 16; i += blockDim.x)
        reinterpret_cast<uint4*>(sX)[i] = make_uint4(0u, 0u, 0u, 0u);
    const uint32_t tbase = warm_setup(io, smem, &mbar, &tmem_slot, sb, sw4, cols);
    uint32_t phase = 0;
    bool alive = true;
    for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x) {
        const Team<L> tm = team_of<L>(vb);
        float f[12], lam = 0.0f;
        const bool have = features_one<L, V>(p, tm, x, v, nbr, ncnt, lam_prev, xl, feat, lam_acc, f, lam);
        if (tm.t == 0) {
            const int row = t / L;
            uint32_t pk[8] = {};
            if (have) pack_row(f, sb, pk);
            uint8_t* xt = sX + (row >> 7) * FW_X_TILE;
            *reinterpret_cast<uint4*>(xt + kmajor_offset(row & 127, 0, 128)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            *reinterpret_cast<uint4*>(xt + kmajor_offset(row & 127, 8, 128)) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
            s_lam[row] = lam;
        }
        if (!alive) continue;  // an expired wait: no more tensor-core work (the error bit is set)
        // row t's plain lambda is read after the first barrier (its team leader
        // wrote it) and before the second (after which that leader may write
        // the next tile's)
        float y, lam_plain = 0.0f;
        alive = warm_layers(io, smem, sX, FW_X_TILE, sH, tiles, tbase, &mbar, phase, sb, sw4, y, [&] {
            if (t < R) lam_plain = s_lam[t];
        });
        if (!alive) continue;
        const int k = vb * R + t;
        if (t < R && k < p.n) warm_store(io, sb, k, y, lam_plain, xl, lam_acc);
    }
    fence_before_sync();
    __syncthreads();
    if (t < 32) tmem_dealloc(tbase, cols);
}

// The network over rows that k_features wrote: 256 rows (two tiles) per step, X in
// the first 4 KB of each tile's H (layer 0 has read it before its epilogue writes
// there), the next step's rows loaded during this one's layers. 50 KB and 128 TMEM
// columns: four blocks per SM. Bound by the GELU epilogues' instructions (2,000 per
// row; 56 % of the issue slots, 44 % of the MUFU's): 262,144 rows take 27.2 us, 28.6
// with one bias per shared load and no early loads, 29.3 in blocks of one tile.
constexpr int WR_SMEM = FW_SX + 2 * FW_H_TILE;
constexpr int WR_BLOCKS = 4;
__global__ void __launch_bounds__(256, WR_BLOCKS) k_warm_rows(int n, const uint4* __restrict__ row_lo,
                                                              const uint4* __restrict__ row_hi,
                                                              float4* __restrict__ xl, float* __restrict__ lam_acc,
                                                              WarmIO io) {
    pdl_wait();
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(16) float sb[MLP_NUM_BIASES];
    __shared__ __align__(16) float sw4[64];
    const int t = threadIdx.x;
    uint8_t* sH = smem + FW_SX;
    uint8_t* xt = sH + (t >> 7) * FW_H_TILE;
    const uint32_t tbase = warm_setup(io, smem, &mbar, &tmem_slot, sb, sw4, 128u);
    uint32_t phase = 0;
    uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
    float next_plain = 0.0f;
    const auto load = [&](int k) {
        if (k < n) {
            lo = row_lo[k];
            hi = row_hi[k];
            next_plain = lam_acc[k];
        }
    };
    load(blockIdx.x * 256 + t);
    for (int k = blockIdx.x * 256 + t; k - t < n; k += gridDim.x * 256) {
        const float lam_plain = next_plain;
        *reinterpret_cast<uint4*>(xt + kmajor_offset(t & 127, 0, 128)) = lo;
        *reinterpret_cast<uint4*>(xt + kmajor_offset(t & 127, 8, 128)) = hi;
        load(k + (int)gridDim.x * 256);
        float y;
        if (!warm_layers(io, smem, sH, FW_H_TILE, sH, 2, tbase, &mbar, phase, sb, sw4, y, [] {})) break;
        if (k < n) warm_store(io, sb, k, y, lam_plain, xl, lam_acc);
    }
    fence_before_sync();
    __syncthreads();
    if (t < 32) tmem_dealloc(tbase, 128u);
}

// ---------------------------------------------------------------------------
// a10 + a11: position correction with tensile s_corr, then x += dp, wall clamp,
// and on the last iteration v = (x - x_old) / dt
// (calculateOffset cu:182-199, updatePosition cu:15-22)
// ---------------------------------------------------------------------------
template <bool N4, typename T, int V>
__device__ __forceinline__ void dp_pair(const KParams& p, const f3& xk, float lk, const float4 (&xj)[V],
                                        T3<T>& a) {
    T3<T> r, g;
    T w;
    pair_terms<T, true>(p, xk, xj, r, w, g);
    T s = dp_weight<N4>(p, addw(lk, xj), w);
    // (a padding entry's weight is finite for whole exponents: 0^n = 0)
    if (!N4 && p.n_int == 0) s = keep_only(s, is_entry(xj));
    a = {vfma(s, g.x, a.x), vfma(s, g.y, a.y), vfma(s, g.z, a.z)};
}
struct DpOut {
    const float4* xold;
    float4 *xout, *vout, *dp_out;
};
// Particle k moved by its summed correction.
template <bool DEBUG>
__device__ __forceinline__ void dp_apply(const KParams& p, int k, const f3& xk, float lk, f3 as, const DpOut& o) {
    if (p.flags & FLAG_WALL_DENSITY) {
        f3 gw;
        wall_term(p, scene_of(p, k), xk, gw);
        as.x = __fmaf_rn(lk, gw.x, as.x);
        as.y = __fmaf_rn(lk, gw.y, as.y);
        as.z = __fmaf_rn(lk, gw.z, as.z);
    }
    const f3 dp = {__fdiv_rn(as.x, p.rho0), __fdiv_rn(as.y, p.rho0), __fdiv_rn(as.z, p.rho0)};
    f3 xn = {xk.x + dp.x, xk.y + dp.y, xk.z + dp.z};
    bound_particle(p, scene_of(p, k), xn);
    o.xout[k] = make_float4(xn.x, xn.y, xn.z, 0.0f);
    if (o.vout) {
        const float4 xo = o.xold[k];
        o.vout[k] = make_float4(__fdiv_rn(xn.x - xo.x, p.dt), __fdiv_rn(xn.y - xo.y, p.dt),
                                __fdiv_rn(xn.z - xo.z, p.dt), 0.0f);
    }
    if (DEBUG) o.dp_out[k] = make_float4(dp.x, dp.y, dp.z, 0.0f);
}
template <bool DEBUG, int L, int V>
__device__ __forceinline__ void dp_store(const KParams& p, const Team<L>& tm, const f3& xk, float lk,
                                         const T3<vec_t<V>>& a, const DpOut& o) {
    const f3 as = team_sum3<L>(fold3(a), tm.mask);
    if (tm.t == 0) dp_apply<DEBUG>(p, tm.k, xk, lk, as, o);
}
template <bool DEBUG, bool N4, int L, int V>
__device__ __forceinline__ void dp_list(const KParams& p, const Team<L>& tm, const float4* __restrict__ xl,
                                        const int* __restrict__ nbr, const int* __restrict__ ncnt, const DpOut& o) {
    using T = vec_t<V>;
    const float4 xk4 = xl[tm.k];
    const f3 xk = make3(xk4);
    T3<T> a = zero3<T>();
    for_list<L, V, 4, 1>(p, nbr, tm.k, tm.t, ncnt[tm.k], xl, xl,
                              [&](const float4(&xj)[V], const float4(&)[V]) {
                                  dp_pair<N4, T, V>(p, xk, xk4.w, xj, a);
                              });
    dp_store<DEBUG, L, V>(p, tm, xk, xk4.w, a, o);
}

// Adaptive loop: true when this correction is not to be applied (the loop ended
// before, or ends here because the positions it would correct are within
// tolerance). LOOP: in the device-side loop. The other kernels hold no call that sets a
// graph's condition: the profiler refuses graph nodes of kernels that do.
template <bool LOOP> __device__ __forceinline__ bool dp_skip(const IterCtl& ctl) {
    if (!ctl.done) return false;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    // the lambda pass just measured the positions this pass would correct;
    // when they are within tolerance the loop ends here
    const int sl = ctl.cur_slot();
    const bool over = *ctl.done != 0 || ctl.past_end();
    const bool met = !over && sl >= ctl.min_slot && __longlong_as_double((long long)ctl.max_bits[sl]) <= ctl.tol;
    if (lead) {
        if (met) {
            *ctl.done = 1;
            *ctl.conv_slot = sl;
        }
        if (!over && !met) atomicAdd(ctl.iters, 1);
        if constexpr (LOOP) {
            *ctl.loop_next = *ctl.loop_k + ctl.loop_add;
            cudaGraphSetConditional(ctl.handle, !over && !met && sl + 1 < ctl.max_slot ? 1u : 0u);
        }
    }
    return over || met;
}

template <bool DEBUG, bool N4, bool ROOMY, bool LOOP, int L, int V>
__global__ void __launch_bounds__(256, ROOMY ? ROOMY_BLOCKS : L == 1 && (N4 || V == 1) ? 5 : 4) k_dp(KParams p, int nvb, const float4* __restrict__ xl,
                                                            const int* __restrict__ nbr, const int* __restrict__ ncnt,
                                                            DpOut o, IterCtl ctl) {
    pdl_wait();
    if (dp_skip<LOOP>(ctl)) return;
    for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x) {
        const Team<L> tm = team_of<L>(vb);
        if (tm.k < p.n) dp_list<DEBUG, N4, L, V>(p, tm, xl, nbr, ncnt, o);  // uniform over the team
    }
}

// ---------------------------------------------------------------------------
// a12: vorticity (calculateCurl cu:201-215): w_i = sum (v_j - v_i) x gradW(x_i - x_j);
// writes (w_i, |w_i|) and (v_i, |w_i|): the vorticity pass then gathers two
// float4s per neighbour (x_j and v_j with |w_j|) instead of three
// ---------------------------------------------------------------------------
template <typename T, int V>
__device__ __forceinline__ void curl_pair(const KParams& p, const f3& xk, const f3& vk, const float4 (&xj)[V],
                                          const float4 (&vj)[V], T3<T>& wsum) {
    T3<T> r, g;
    T w;
    pair_terms<T, false>(p, xk, xj, r, w, g);
    const T3<T> vji = rdiff3(vj, vk);
    wsum = add3(wsum, cross3v(vji, g));
}
__device__ __forceinline__ void curl_apply(int k, const f3& vk, const f3& w3, float4* __restrict__ omega,
                                           float4* __restrict__ vw) {
    const float wl = __fsqrt_rn(dot_fma(w3, w3));
    omega[k] = make_float4(w3.x, w3.y, w3.z, wl);
    vw[k] = make_float4(vk.x, vk.y, vk.z, wl);
}
template <int L, int V>
__device__ __forceinline__ void curl_store(const Team<L>& tm, const f3& vk, const T3<vec_t<V>>& wsum,
                                           float4* __restrict__ omega, float4* __restrict__ vw) {
    const f3 w3 = team_sum3<L>(fold3(wsum), tm.mask);
    if (tm.t == 0) curl_apply(tm.k, vk, w3, omega, vw);
}
template <bool ROOMY, int L, int V>
__device__ __forceinline__ void curl_list(const KParams& p, const Team<L>& tm, const float4* __restrict__ x,
                                          const float4* __restrict__ v, const int* __restrict__ nbr,
                                          const int* __restrict__ ncnt, float4* __restrict__ omega,
                                          float4* __restrict__ vw) {
    using T = vec_t<V>;
    const f3 xk = make3(x[tm.k]), vk = make3(v[tm.k]);
    T3<T> wsum = zero3<T>();
    for_list<L, V, ROOMY ? 4 : 2, 2>(p, nbr, tm.k, tm.t, ncnt[tm.k], x, v,
                            [&](const float4(&xj)[V], const float4(&vj)[V]) {
                                curl_pair<T, V>(p, xk, vk, xj, vj, wsum);
                            });
    curl_store<L, V>(tm, vk, wsum, omega, vw);
}

template <bool ROOMY, int L, int V>
__global__ void __launch_bounds__(256, ROOMY ? ROOMY_BLOCKS : 4) k_curl(KParams p, int nvb, const float4* __restrict__ x,
                                              const float4* __restrict__ v, const int* __restrict__ nbr,
                                              const int* __restrict__ ncnt, float4* __restrict__ omega,
                                              float4* __restrict__ vw) {
    pdl_wait();
    for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x) {
        const Team<L> tm = team_of<L>(vb);
        if (tm.k < p.n) curl_list<ROOMY, L, V>(p, tm, x, v, nbr, ncnt, omega, vw);  // uniform over the team
    }
}

// ---------------------------------------------------------------------------
// a13: vorticity confinement and XSPH, applied to v
// (calculateVorticityAndViscosity cu:217-239, applyVorticityAndViscosity cu:24-29);
// also writes the substep's final state (x, v, perm) for the next substep, and
// with the final x and v in registers does the next substep's grid hash (a1 +
// a2: prediction, wall clamp, cell key and its histogram), which therefore needs
// no pass of its own.
// ---------------------------------------------------------------------------
struct VortIO {
    const float4* omega;
    float4 *xout, *vout;
    const int* perm_in;
    int* perm_out;
    float4 *vort_out, *visc_out;
    int *cell, *ticket, *hist, *err;
};
template <typename T> struct VortSums {
    T3<T> pv, eta;
};
template <typename T, int V>
__device__ __forceinline__ void vort_pair(const KParams& p, const f3& xk, const f3& vk, const float4 (&xj)[V],
                                          const float4 (&vj)[V], VortSums<T>& s) {
    T3<T> r, g;
    T w;
    pair_terms<T, true>(p, xk, xj, r, w, g);
    const T3<T> vji = rdiff3(vj, vk);
    s.pv = {vfma(vji.x, w, s.pv.x), vfma(vji.y, w, s.pv.y), vfma(vji.z, w, s.pv.z)};
    const T wl = packw(vj);  // |w_j| (k_curl)
    s.eta = {vfma(wl, g.x, s.eta.x), vfma(wl, g.y, s.eta.y), vfma(wl, g.z, s.eta.z)};
}
// Particle k from its sums; returns its next cell key.
template <bool DEBUG>
__device__ __forceinline__ int vort_apply(const KParams& p, int k, const f3& xk, const f3& vk, const f3& pvs, f3 etas,
                                          const VortIO& o) {
    const float el = __fsqrt_rn(dot_fma(etas, etas));
    if ((double)el > 1e-3) etas = {__fdiv_rn(etas.x, el), __fdiv_rn(etas.y, el), __fdiv_rn(etas.z, el)};
    const f3 cr = cross3(etas, make3(o.omega[k]));
    const f3 fv = {p.vort_eps * cr.x, p.vort_eps * cr.y, p.vort_eps * cr.z};
    const f3 vs = {p.visc_c * pvs.x, p.visc_c * pvs.y, p.visc_c * pvs.z};
    const f3 t = {p.dt * fv.x + vs.x, p.dt * fv.y + vs.y, p.dt * fv.z + vs.z};
    f3 vn = {vk.x + t.x, vk.y + t.y, vk.z + t.z};
    o.xout[k] = make_float4(xk.x, xk.y, xk.z, 0.0f);
    o.vout[k] = make_float4(vn.x, vn.y, vn.z, 0.0f);
    o.perm_out[k] = o.perm_in[k];
    if (DEBUG) {
        o.vort_out[k] = make_float4(fv.x, fv.y, fv.z, 0.0f);
        o.visc_out[k] = make_float4(vs.x, vs.y, vs.z, 0.0f);
    }
    // the next substep's prediction and cell key (as k_hash computes them from
    // the state just written)
    const SceneView sc = scene_of(p, k);
    f3 xq = xk;
    predict(p, sc, xq, vn);
    if (!(isfinite(xq.x) && isfinite(xq.y) && isfinite(xq.z))) atomicOr(o.err, DEVERR_NONFINITE);
    return cell_key(p, sc, xq);
}
// the same from the team's sums: the key on its first thread, -1 on the others
template <bool DEBUG, int L, int V>
__device__ __forceinline__ int vort_store(const KParams& p, const Team<L>& tm, const f3& xk, const f3& vk,
                                          const VortSums<vec_t<V>>& s, const VortIO& o) {
    const f3 pvs = team_sum3<L>(fold3(s.pv), tm.mask);
    const f3 etas = team_sum3<L>(fold3(s.eta), tm.mask);
    return tm.t == 0 ? vort_apply<DEBUG>(p, tm.k, xk, vk, pvs, etas, o) : -1;
}
// the next substep's histogram (every lane of the warp takes part)
__device__ __forceinline__ void vort_hash(int k, int key, const VortIO& o) {
    const int tk = warp_histogram(key, o.hist);
    if (key >= 0) {
        o.cell[k] = key;
        o.ticket[k] = tk;
    }
}
template <bool DEBUG, bool ROOMY, int L, int V>
__device__ __forceinline__ int vort_list(const KParams& p, const Team<L>& tm, const float4* __restrict__ x,
                                         const float4* __restrict__ vw, const int* __restrict__ nbr,
                                         const int* __restrict__ ncnt, const VortIO& o) {
    using T = vec_t<V>;
    const f3 xk = make3(x[tm.k]), vk = make3(vw[tm.k]);
    VortSums<T> s = {zero3<T>(), zero3<T>()};
    for_list<L, V, ROOMY ? 4 : 2, 2>(p, nbr, tm.k, tm.t, ncnt[tm.k], x, vw,
                             [&](const float4(&xj)[V], const float4(&vj)[V]) {
                                 vort_pair<T, V>(p, xk, vk, xj, vj, s);
                             });
    return vort_store<DEBUG, L, V>(p, tm, xk, vk, s, o);
}

template <bool DEBUG, bool ROOMY, int L, int V>
__global__ void __launch_bounds__(256, ROOMY ? ROOMY_BLOCKS : 4) k_vort(KParams p, int nvb, const float4* __restrict__ x,
                                                 const float4* __restrict__ vw, const int* __restrict__ nbr,
                                                 const int* __restrict__ ncnt, VortIO o) {
    pdl_wait();
    for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x) {
        const Team<L> tm = team_of<L>(vb);
        int key = -1;
        if (tm.k < p.n) key = vort_list<DEBUG, ROOMY, L, V>(p, tm, x, vw, nbr, ncnt, o);  // uniform over the team
        vort_hash(tm.k, key, o);
    }
}

// ---------------------------------------------------------------------------
// Small scenes. A thread per particle evaluates its 33 pairs one step after the
// other, and a pass over a few thousand particles takes that chain whatever their
// number. Here WIDE = 8 threads share a particle whatever the pair lanes: each takes
// every eighth entry and leaves what its pairs contribute in shared memory; the
// sums, whose order the pair lanes define, are then run one chain per thread (lane p
// of quantity q adds entries p, p + P, ...), the lanes combined as by the butterfly.
// The values are those of the other kernels bit for bit. 4,096 particles: lambda
// 5.4 us -> 4.7, correction 5.4 -> 4.6, curl 6.0 -> 3.9, vorticity 8.6 -> 6.1 (four
// threads per particle were slower than either: 5.9, 5.9, 5.9, 7.9).
// ---------------------------------------------------------------------------
constexpr int WIDE = 8;            // threads per particle
constexpr int WIDE_THREADS = 128;  // per block: 16 particles
constexpr int WIDE_ENTRIES = 5;    // per thread in flight (a list holds about 33)

// A team of WIDE threads: its particle and its slice of the block's shared memory:
// `rows` entries of NV float4, padded so that teams of a warp start on different
// banks.
struct WideTeam {
    int k, t;      // slot, thread of the team
    float4* s;     // the entries' values
    float* out;    // lane sums, [quantity][8]
    float* out0;   // those of the block's first team
};
template <int NV> __host__ __device__ constexpr int wide_stride(int rows) { return rows * NV + 2; }  // in float4
__host__ __device__ inline int wide_rows(int max_nbr) { return (max_nbr + 7) & ~7; }
template <int NV> static int wide_smem(int max_nbr) {
    return WIDE_THREADS / WIDE * (wide_stride<NV>(wide_rows(max_nbr)) * 16 + 64 * 4);
}

template <int NV> __device__ __forceinline__ WideTeam wide_team(int max_nbr) {
    extern __shared__ float4 s_wide[];
    constexpr int TEAMS = WIDE_THREADS / WIDE;
    const int team = threadIdx.x / WIDE, stride = wide_stride<NV>(wide_rows(max_nbr));
    WideTeam w;
    w.k = blockIdx.x * TEAMS + team;
    w.t = threadIdx.x & (WIDE - 1);
    w.s = s_wide + team * stride;
    w.out0 = reinterpret_cast<float*>(s_wide + TEAMS * stride);
    w.out = w.out0 + team * 64;
    return w;
}

// eval(xj, vj, dst) for every entry of the team's list that this thread takes: dst
// receives the entry's NV float4.
template <int NV, int NA, typename F>
__device__ __forceinline__ void wide_pairs(const KParams& p, const WideTeam& w, int cnt, const int* __restrict__ nbr,
                                           const float4* __restrict__ a, const float4* __restrict__ b, F&& eval) {
    constexpr int U = WIDE_ENTRIES;
    for (int q0 = w.t; q0 < cnt; q0 += WIDE * U) {
        int j[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int q = q0 + WIDE * u;
            j[u] = q < cnt ? nbr[(size_t)q * p.stride + w.k] : -1;
        }
        float4 xj[U][1], vj[U][1];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (j[u] >= 0) {
                xj[u][0] = a[j[u]];
                if (NA == 2) vj[u][0] = b[j[u]];
            }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (j[u] >= 0) eval(xj[u], vj[u], w.s + (q0 + WIDE * u) * NV);
    }
    __syncwarp();
}

// Quantity q of pair lane `lane` summed by add(q, acc, values of the entry), chains
// dealt to the team's threads; NQ quantities. Ends with a block barrier: the
// particles' epilogues then run on the block's first threads, one each, instead of
// on one thread of every team.
template <int NV, int NQ, typename F>
__device__ __forceinline__ void wide_sums(const WideTeam& w, int cnt, int P, F&& add) {
    for (int c = w.t; c < NQ * P; c += WIDE) {
        const int q = c / P, lane = c - q * P;
        float acc = 0.0f;
        const float4* e = w.s + lane * NV;
#pragma unroll 4
        for (int i = lane; i < cnt; i += P, e += P * NV) acc = add(q, acc, reinterpret_cast<const float*>(e));
        w.out[q * 8 + lane] = acc;
    }
    __syncthreads();
}
// the butterfly over P lane sums
__device__ __forceinline__ float wide_total(const float* s, int P) {
    float v = s[0];
    if (P >= 2) v = s[0] + s[1];
    if (P >= 4) v = v + (s[2] + s[3]);
    if (P >= 8) v = v + ((s[4] + s[5]) + (s[6] + s[7]));
    return v;
}
__device__ __forceinline__ f3 wide_total3(const float* s, int P) {
    return {wide_total(s, P), wide_total(s + 8, P), wide_total(s + 16, P)};
}
// the particle whose epilogue this thread runs, -1 for none, and its sums
__device__ __forceinline__ int wide_mine(const KParams& p, const WideTeam& w, const float*& sums) {
    constexpr int TEAMS = WIDE_THREADS / WIDE;
    const int k = blockIdx.x * TEAMS + threadIdx.x;
    sums = w.out0 + threadIdx.x * 64;
    return threadIdx.x < TEAMS && k < p.n ? k : -1;
}

template <bool DEBUG>
__global__ void __launch_bounds__(WIDE_THREADS) k_lambda_wide(KParams p, const float4* __restrict__ x,
                                                              const int* __restrict__ nbr,
                                                              const int* __restrict__ ncnt, float4* __restrict__ xl,
                                                              float* __restrict__ rho_out, IterCtl ctl) {
    pdl_wait();
    if (lambda_skip(ctl)) return;
    const WideTeam w = wide_team<1>(p.max_nbr);
    const bool on = w.k < p.n;
    const int cnt = on ? ncnt[w.k] : 0;
    const f3 xk = on ? make3(x[w.k]) : f3{0.0f, 0.0f, 0.0f};
    wide_pairs<1, 1>(p, w, cnt, nbr, x, x, [&](const float4(&xj)[1], const float4(&)[1], float4* dst) {
        T3<float> r, g;
        float wt;
        pair_terms<float, true>(p, xk, xj, r, wt, g);
        *dst = make_float4(g.x, g.y, g.z, wt);
    });
    // gradient sums, density, sum of squared gradients
    wide_sums<1, 5>(w, cnt, p.lanes, [&](int q, float acc, const float* v) {
        if (q < 4) return acc + v[q];
        acc = __fmaf_rn(v[0], v[0], acc);
        acc = __fmaf_rn(v[1], v[1], acc);
        return __fmaf_rn(v[2], v[2], acc);
    });
    float err = 0.0f;
    const float* s;
    const int k = wide_mine(p, w, s);
    if (k >= 0) {
        const f3 q = make3(x[k]);
        float rhos = wide_total(s + 24, p.lanes);
        const float lam = lambda_tail(p, k, q, rhos, wide_total(s + 32, p.lanes), wide_total3(s, p.lanes), err);
        xl[k] = make_float4(q.x, q.y, q.z, lam);
        if (ctl.lam_acc) ctl.lam_acc[k] += lam;
        if (DEBUG) rho_out[k] = rhos;
    }
    if (ctl.max_bits) {
        const int sl = ctl.cur_slot();
        block_error_reduce(err, err, ctl.max_bits + sl, ctl.sum + sl);
    }
}

template <bool DEBUG, bool N4, bool LOOP>
__global__ void __launch_bounds__(WIDE_THREADS) k_dp_wide(KParams p, const float4* __restrict__ xl,
                                                          const int* __restrict__ nbr, const int* __restrict__ ncnt,
                                                          DpOut o, IterCtl ctl) {
    pdl_wait();
    if (dp_skip<LOOP>(ctl)) return;
    const WideTeam w = wide_team<1>(p.max_nbr);
    const bool on = w.k < p.n;
    const int cnt = on ? ncnt[w.k] : 0;
    const float4 xk4 = on ? xl[w.k] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const f3 xk = make3(xk4);
    wide_pairs<1, 1>(p, w, cnt, nbr, xl, xl, [&](const float4(&xj)[1], const float4(&)[1], float4* dst) {
        T3<float> r, g;
        float wt;
        pair_terms<float, true>(p, xk, xj, r, wt, g);
        *dst = make_float4(g.x, g.y, g.z, dp_weight<N4>(p, addw(xk4.w, xj), wt));
    });
    wide_sums<1, 3>(w, cnt, p.lanes, [&](int q, float acc, const float* v) { return __fmaf_rn(v[3], v[q], acc); });
    const float* s;
    const int k = wide_mine(p, w, s);
    if (k >= 0) {
        const float4 q = xl[k];
        dp_apply<DEBUG>(p, k, make3(q), q.w, wide_total3(s, p.lanes), o);
    }
}

__global__ void __launch_bounds__(WIDE_THREADS) k_curl_wide(KParams p, const float4* __restrict__ x,
                                                            const float4* __restrict__ v, const int* __restrict__ nbr,
                                                            const int* __restrict__ ncnt, float4* __restrict__ omega,
                                                            float4* __restrict__ vw) {
    pdl_wait();
    const WideTeam w = wide_team<1>(p.max_nbr);
    const bool on = w.k < p.n;
    const int cnt = on ? ncnt[w.k] : 0;
    const f3 xk = on ? make3(x[w.k]) : f3{0.0f, 0.0f, 0.0f}, vk = on ? make3(v[w.k]) : f3{0.0f, 0.0f, 0.0f};
    wide_pairs<1, 2>(p, w, cnt, nbr, x, v, [&](const float4(&xj)[1], const float4(&vj)[1], float4* dst) {
        T3<float> r, g;
        float wt;
        pair_terms<float, false>(p, xk, xj, r, wt, g);
        const T3<float> c = cross3v(rdiff3(vj, vk), g);
        *dst = make_float4(c.x, c.y, c.z, 0.0f);
    });
    wide_sums<1, 3>(w, cnt, p.lanes, [&](int q, float acc, const float* s) { return acc + s[q]; });
    const float* s;
    const int k = wide_mine(p, w, s);
    if (k >= 0) curl_apply(k, make3(v[k]), wide_total3(s, p.lanes), omega, vw);
}

template <bool DEBUG>
__global__ void __launch_bounds__(WIDE_THREADS) k_vort_wide(KParams p, const float4* __restrict__ x,
                                                            const float4* __restrict__ vw,
                                                            const int* __restrict__ nbr, const int* __restrict__ ncnt,
                                                            VortIO o) {
    pdl_wait();
    const WideTeam w = wide_team<2>(p.max_nbr);
    const bool on = w.k < p.n;
    const int cnt = on ? ncnt[w.k] : 0;
    const f3 xk = on ? make3(x[w.k]) : f3{0.0f, 0.0f, 0.0f}, vk = on ? make3(vw[w.k]) : f3{0.0f, 0.0f, 0.0f};
    wide_pairs<2, 2>(p, w, cnt, nbr, x, vw, [&](const float4(&xj)[1], const float4(&vj)[1], float4* dst) {
        T3<float> r, g;
        float wt;
        pair_terms<float, true>(p, xk, xj, r, wt, g);
        const T3<float> d = rdiff3(vj, vk);
        dst[0] = make_float4(d.x, d.y, d.z, wt);
        dst[1] = make_float4(g.x, g.y, g.z, packw(vj));
    });
    // sum of (v_j - v_i) W, then of |w_j| grad W
    wide_sums<2, 6>(w, cnt, p.lanes, [&](int q, float acc, const float* s) {
        return q < 3 ? __fmaf_rn(s[q], s[3], acc) : __fmaf_rn(s[7], s[q + 1], acc);
    });
    if (threadIdx.x < 32) {  // the 16 particles: all on the first warp
        const float* s;
        const int k = wide_mine(p, w, s);
        int key = -1;
        if (k >= 0)
            key = vort_apply<DEBUG>(p, k, make3(x[k]), make3(vw[k]), wide_total3(s, p.lanes),
                                    wide_total3(s + 24, p.lanes), o);
        vort_hash(k, key, o);
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
// blocks for n particles with L threads each
static inline int team_blocks(int n, int L, int bs) { return (int)(((long long)n * L + bs - 1) / bs); }

static int sm_count() {
    static int sms = 0;
    if (!sms) {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        sms = v > 0 ? v : 1;
    }
    return sms;
}
// Grid of a neighbour pass over nvb tiles: nvb blocks, or with p.persistent the
// blocks that are resident at once (SMs x blocks per SM at this block size), each
// striding over the tiles.
template <typename K> static int pass_grid(const KParams& p, K kernel, int nvb) {
    if (!p.persistent) return nvb;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, p.block, 0) != cudaSuccess || per_sm <= 0)
        per_sm = 1;
    const long long g = (long long)per_sm * sm_count();
    return (int)(g < nvb ? g : nvb);
}
// All blocks of a pass with L threads per particle resident at ROOMY_BLOCKS x 256
// threads per SM.
static bool roomy(const KParams& p, int L) { return (long long)p.n * L <= (long long)sm_count() * ROOMY_BLOCKS * 256; }

using Yes = std::true_type;
using No = std::false_type;
// Calls f with the flags as compile-time constants.
template <typename F> static void with_flag(bool a, F&& f) {
    if (a) f(Yes{});
    else f(No{});
}
template <typename F> static void with_flags(bool a, bool b, F&& f) {
    with_flag(a, [&](auto x) { with_flag(b, [&](auto y) { f(x, y); }); });
}

// Calls f with (L, V) of pair_lanes as compile-time constants.
template <int A, int B> struct LV {
    static constexpr int L = A, V = B;
};
template <typename F> void with_lanes(int lanes, F&& f) {
    switch (lanes) {
        case 1: f(LV<1, 1>{}); break;
        case 4: f(LV<2, 2>{}); break;
        case 8: f(LV<4, 2>{}); break;
        default: f(LV<1, 2>{}); break;
    }
}

// The wide kernels run scenes of up to four of their blocks per SM, with one or two
// pair lanes: substeps of 4,096 particles take 69 us with them and 78 without, of
// 13,824 the same, and beyond that the flat kernels fill the device with less work
// (four and eight lanes already spread a particle over two and four threads).
static bool wide(const KParams& p) {
    return !p.persistent && p.lanes <= 2 && p.n <= sm_count() * 4 * (WIDE_THREADS / WIDE);
}
template <int NV, typename K, typename... A>
static void launch_wide(const KParams& p, K kernel, cudaStream_t st, A... args) {
    const int smem = wide_smem<NV>(p.max_nbr);  // at most 69 KB (127 entries of two float4)
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
        return;  // (the runtime's last error: the capture fails)
    const int per = WIDE_THREADS / WIDE;
    launch(p.pdl, kernel, (p.n + per - 1) / per, WIDE_THREADS, smem, st, p, args...);
}

void launch_lambda(const KParams& p, bool debug, const float4* x, const int* nbr, const int* ncnt, float4* xl,
                  float* rho, const IterCtl& ctl, cudaStream_t st) {
    if (wide(p)) {
        with_flag(debug, [&](auto d) {
            launch_wide<1>(p, k_lambda_wide<decltype(d)::value>, st, x, nbr, ncnt, xl, rho, ctl);
        });
        return;
    }
    with_lanes(p.lanes, [&](auto c) {
        constexpr int L = decltype(c)::L, V = decltype(c)::V;
        const int b = team_blocks(p.n, L, p.block);
        with_flags(debug, roomy(p, L), [&](auto d, auto r) {
            auto* k = k_lambda<decltype(d)::value, decltype(r)::value, L, V>;
            launch(p.pdl, k, pass_grid(p, k, b), p.block, 0, st, p, b, x, nbr, ncnt, xl, rho, ctl);
        });
    });
}

void launch_dp(const KParams& p, bool debug, const float4* xl, const int* nbr, const int* ncnt, const float4* xold,
               float4* xout, float4* vout, float4* dp, const IterCtl& ctl, cudaStream_t st) {
    const DpOut o{xold, xout, vout, dp};
    if (wide(p)) {
        with_flags(debug, p.n_int == 4, [&](auto d, auto n4) {
            with_flag(ctl.loop_next != nullptr, [&](auto lp) {
                auto* k = k_dp_wide<decltype(d)::value, decltype(n4)::value, decltype(lp)::value>;
                launch_wide<1>(p, k, st, xl, nbr, ncnt, o, ctl);
            });
        });
        return;
    }
    with_lanes(p.lanes, [&](auto c) {
        constexpr int L = decltype(c)::L, V = decltype(c)::V;
        const int b = team_blocks(p.n, L, p.block);
        with_flags(debug, p.n_int == 4, [&](auto d, auto n4) {
            with_flags(roomy(p, L), ctl.loop_next != nullptr, [&](auto r, auto lp) {
                auto* k = k_dp<decltype(d)::value, decltype(n4)::value, decltype(r)::value, decltype(lp)::value, L, V>;
                launch(p.pdl, k, pass_grid(p, k, b), p.block, 0, st, p, b, xl, nbr, ncnt, o, ctl);
            });
        });
    });
}

void launch_features(const KParams& p, const float4* x, const float4* v, const int* nbr, const int* ncnt,
                     const float* lam_prev, float4* xl, float* feat, float* lam_acc, cudaStream_t st) {
    with_lanes(p.lanes, [&](auto c) {
        constexpr int L = decltype(c)::L, V = decltype(c)::V;
        const int b = team_blocks(p.n, L, p.block);
        const auto k = k_features<false, L, V>;
        launch(p.pdl, k, pass_grid(p, k, b), p.block, 0, st, p, b, x, v, nbr, ncnt, lam_prev, xl, feat, lam_acc,
               (const float*)nullptr, (uint4*)nullptr, (uint4*)nullptr);
    });
}

int launch_features_warm(const KParams& p, const float4* x, const float4* v, const int* nbr, const int* ncnt,
                         const float* lam_prev, float4* xl, float* feat, float* lam_acc, const uint16_t* w,
                         const float* b, float* lam0, float clamp, int floor, uint4* row_lo, uint4* row_hi, int* err,
                         cudaStream_t st) {
    int rc = 0;
    const WarmIO io{w, b, lam0, clamp, floor, err};
    // In two launches above two blocks of 256 particles per SM: the gathers then have
    // the L1 and the warps that the fused pass gives to the network's tiles (262,144
    // particles: 34.7 + 27.2 us against 75.6; frames at 64,000 / 85,184 / 884,736
    // particles: 219 / 258 / 1,593 us against 216 / 261 / 1,635). Below, one launch
    // less is worth more (4,096: 128 us fused against 133).
    if (p.n > 2 * 256 * sm_count()) {
        if (cudaFuncSetAttribute(k_warm_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, WR_SMEM) != cudaSuccess)
            return -1;
        with_lanes(p.lanes, [&](auto c) {
            constexpr int L = decltype(c)::L, V = decltype(c)::V;
            const int nvb = team_blocks(p.n, L, p.block);
            const auto k = k_features<true, L, V>;
            launch(p.pdl, k, pass_grid(p, k, nvb), p.block, 0, st, p, nvb, x, v, nbr, ncnt, lam_prev, xl, feat, lam_acc,
                   b, row_lo, row_hi);
        });
        const int steps = (p.n + 255) / 256;
        return launch(p.pdl, k_warm_rows, std::min(steps, WR_BLOCKS * sm_count()), 256, WR_SMEM, st, p.n,
                      (const uint4*)row_lo, (const uint4*)row_hi, xl, lam_acc, io);
    }
    with_lanes(p.lanes, [&](auto c) {
        constexpr int L = decltype(c)::L, V = decltype(c)::V;
        const int rows = p.block / L;
        const int smem = warm_smem_bytes((rows + 127) / 128);
        if (cudaFuncSetAttribute(k_features_warm<L, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
            cudaSuccess) {
            rc = -1;
            return;
        }
        const int nvb = team_blocks(p.n, L, p.block);
        int grid = nvb;
        if (p.persistent) {
            int dev = 0, sms = 1, per_sm = 0;
            cudaGetDevice(&dev);
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_features_warm<L, V>, p.block, smem) !=
                    cudaSuccess || per_sm <= 0)
                per_sm = 1;
            grid = (int)std::min<long long>((long long)per_sm * sms, nvb);
        }
        launch(p.pdl, k_features_warm<L, V>, grid, p.block, smem, st, p, nvb, x, v, nbr, ncnt, lam_prev, xl, feat, lam_acc, io);
    });
    return rc;
}

void launch_curl(const KParams& p, const float4* x, const float4* v, const int* nbr, const int* ncnt, float4* omega,
                float4* vw, cudaStream_t st) {
    if (wide(p)) {
        launch_wide<1>(p, k_curl_wide, st, x, v, nbr, ncnt, omega, vw);
        return;
    }
    with_lanes(p.lanes, [&](auto c) {
        constexpr int L = decltype(c)::L, V = decltype(c)::V;
        const int b = team_blocks(p.n, L, p.block);
        with_flag(roomy(p, L), [&](auto r) {
            auto* k = k_curl<decltype(r)::value, L, V>;
            launch(p.pdl, k, pass_grid(p, k, b), p.block, 0, st, p, b, x, v, nbr, ncnt, omega, vw);
        });
    });
}

void launch_vort(const KParams& p, bool debug, const float4* x, const float4* vw, const float4* omega, const int* nbr,
                const int* ncnt, float4* xout, float4* vout, const int* perm_in, int* perm_out, float4* vort,
                float4* visc, int* cell, int* ticket, int* hist, int* err, cudaStream_t st) {
    const VortIO o{omega, xout, vout, perm_in, perm_out, vort, visc, cell, ticket, hist, err};
    if (wide(p)) {
        with_flag(debug, [&](auto d) { launch_wide<2>(p, k_vort_wide<decltype(d)::value>, st, x, vw, nbr, ncnt, o); });
        return;
    }
    with_lanes(p.lanes, [&](auto c) {
        constexpr int L = decltype(c)::L, V = decltype(c)::V;
        const int b = team_blocks(p.n, L, p.block);
        with_flags(debug, roomy(p, L), [&](auto d, auto r) {
            auto* k = k_vort<decltype(d)::value, decltype(r)::value, L, V>;
            launch(p.pdl, k, pass_grid(p, k, b), p.block, 0, st, p, b, x, vw, nbr, ncnt, o);
        });
    });
}

}  // namespace pbf
