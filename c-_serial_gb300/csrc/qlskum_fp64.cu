// FP64 kernels: the drop-in form of the q-LSKUM primal iteration.
//
// Every formula is the reference's, with FMA contraction on (GB300 runs FP64
// at 1/64 of the FP32 rate, and a fused multiply-add is one FP64 instruction
// instead of two), and the edge ends in the forms of qlskum_fast64.cuh, which
// need few FP64 instructions for the same value to a few ulps.  The
// directional solves are folded into per-edge weights once per cloud.  The
// results differ from the serial reference by those roundings: 1e-10 relative
// after 1000 iterations (the parity tests).
//
// Four lanes per point (one per component) in the gradient kernels, several
// threads per point in the flux kernels (flux_shape), one elsewhere; a point's
// edges are summed in the reference's neighbour order, read from the
// sliced-ELL edge arrays (coalesced across the warp); neighbour state is
// gathered through L1/L2 (points are Morton ordered, so most neighbours of a
// block's points are cache-resident).  All geometry that
// does not change between iterations (edge vectors, least-squares moments,
// 1/det, limiter epsilon) is precomputed on the host in the reference's
// operation order, which on this chip trades a few bytes per edge for FP64
// instructions, its scarce resource.
#include "qlskum_math.cuh"
#include "qlskum_fast64.cuh"
#include <type_traits>

namespace qlskum {
namespace fp64 {

static inline int grid_for(long long n, int block) { return (int)((n + block - 1) / block); }

// ----------------------------------------------------------------- q, c

// q_variables_mod.h:9-34
__global__ void k_q_variables(int n, const double4_32a *__restrict__ prim, double4_32a *__restrict__ q)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double P[4], Q[4];
    ld4(prim[i], P);
    fast64::q_of(P, Q);
    q[i] = mk4(Q);
}

// q and the wave speed of the current state (both read by the next stage's
// gradient kernel).
__global__ void k_derived(int n, const double4_32a *__restrict__ prim, double4_32a *__restrict__ q, double *__restrict__ cs)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double P[4], Q[4];
    ld4(prim[i], P);
    fast64::q_of(P, Q);
    q[i] = mk4(Q);
    cs[i] = fast64::wave_speed(P);
}

// ----------------------------------------------------------- gradients

// The gradient and inner-step kernels take four lanes per point, one per
// component: a lane walks all edges in the reference's neighbour order, the
// four lanes gather the 32 bytes of a neighbour's q (or of each half of its
// gradient) in one sector, and a small cloud fills four times the warps.

// The local time step of point i (state_update_mod.h:448-496), its edges over
// the point's four lanes.
__device__ __forceinline__ void point_dt(const DevCloud &c, int i, int r, long long base, int nb,
                                         const double *__restrict__ cs, double *__restrict__ delta, double cfl)
{
    double m = 1.0;
    for (int j = r; j < nb; j += 4) {
        const long long e = base + 32LL * j;
        const double dt = fast64::edge_dt(c.e_dist[e], cs[c.e_nbr[e]], cfl);
        if (m > dt) m = dt;
    }
    const unsigned mask = 0xfu << (threadIdx.x & 28u);
#pragma unroll
    for (int s = 1; s < 4; s <<= 1) {
        const double x = __shfl_xor_sync(mask, m, s);
        if (m > x) m = x;
    }
    if (r == 0) delta[i] = m;
}

// q_variables_mod.h:36-118 (+ state_update_mod.h:448-496 when delta != null):
// qm = neighbour max/min, dq = the least-squares gradient through its folded
// per-edge weights.  960 / 204,800 points: 29 / 113 us per launch with one
// thread per point, the moments' solve per point and comparisons on the FP64
// pipe, 12 / 62 us in this form.
template <bool DT>
__global__ void k_q_derivatives(DevCloud c, const double *__restrict__ q, double *__restrict__ dq,
                                double *__restrict__ qm, const double *__restrict__ cs, double *__restrict__ delta,
                                double cfl)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = t >> 2, r = t & 3;
    if (i >= c.n) return;
    const double qi = q[4 * (size_t)i + r];
    long long kmax = fast64::order_key(__double_as_longlong(qi)), kmin = kmax;
    double dx = 0.0, dy = 0.0;
    const int nb = c.nbhs[i];
    const long long base = c.slice_base[i >> 5] + (i & 31);
#pragma unroll 2
    for (int j = 0; j < nb; j++) {
        const long long e = base + 32LL * j;
        const double2 gw = c.e_gw64[e];
        const double qk = q[4 * (size_t)c.e_nbr[e] + r];
        const long long key = fast64::order_key(__double_as_longlong(qk));
        kmax = key > kmax ? key : kmax;
        kmin = key < kmin ? key : kmin;
        const double d = qk - qi;
        dx = fma(gw.x, d, dx);
        dy = fma(gw.y, d, dy);
    }
    const size_t o = 8 * (size_t)i + r;
    dq[o] = dx;
    dq[o + 4] = dy;
    qm[o] = __longlong_as_double(fast64::order_key(kmax));
    qm[o + 4] = __longlong_as_double(fast64::order_key(kmin));
    if (DT) point_dt(c, i, r, base, nb, cs, delta, cfl);
}

// q_variables_mod.h:120-213: the reference's sums over w d (t_k - t_i),
// t = q - d.dq / 2, by linearity: the solve of the sum over w d (q_k - q_i) is
// the first-order gradient dq0, the solve of the sum over w d (d.dq_i) is dq_i,
// so dq_out = dq0 + (dq_i - sum_e g_e (d_e.dq_k)) / 2 with the folded weights
// g_e: one gather and 4 FP64 instructions per edge and component instead of
// two and 9.  FIRST: dq0 is not at hand (a call of the inner step alone) and
// is formed here, with k_q_derivatives' sum.  204,800 points: 167 us per
// launch before, 73 us now.
template <bool FIRST>
__global__ void k_q_inner(DevCloud c, const double *__restrict__ q, const double *__restrict__ dq0,
                          const double *__restrict__ dq_in, double *__restrict__ dq_out)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = t >> 2, r = t & 3;
    if (i >= c.n) return;
    double ax = 0.0, ay = 0.0, d0x = 0.0, d0y = 0.0;
    const double qi = FIRST ? q[4 * (size_t)i + r] : 0.0;
    const int nb = c.nbhs[i];
    const long long base = c.slice_base[i >> 5] + (i & 31);
#pragma unroll 2
    for (int j = 0; j < nb; j++) {
        const long long e = base + 32LL * j;
        const double2 gw = c.e_gw64[e];
        const double2 d = *reinterpret_cast<const double2 *>(c.e_geo + e);  // delx, dely
        const size_t k = (size_t)c.e_nbr[e];
        const double u = fma(d.x, dq_in[8 * k + r], __dmul_rn(d.y, dq_in[8 * k + 4 + r]));
        ax = fma(gw.x, u, ax);
        ay = fma(gw.y, u, ay);
        if (FIRST) {
            const double dk = q[4 * k + r] - qi;
            d0x = fma(gw.x, dk, d0x);
            d0y = fma(gw.y, dk, d0y);
        }
    }
    const size_t o = 8 * (size_t)i + r;
    if (!FIRST) {
        d0x = dq0[o];
        d0y = dq0[o + 4];
    }
    dq_out[o] = fma(0.5, dq_in[o] - ax, d0x);
    dq_out[o + 4] = fma(0.5, dq_in[o + 4] - ay, d0y);
}

// state_update_mod.h:448-496 from the points' wave speeds.  51,200 points: 44 us
// with the neighbour's wave speed evaluated at every edge, 12 us with
// k_wave_speeds (5 us) before it.
__global__ void k_func_delta(DevCloud c, const double *__restrict__ cs, double *__restrict__ delta, double cfl)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = t >> 2;
    if (i < c.n) point_dt(c, i, t & 3, c.slice_base[i >> 5] + (i & 31), c.nbhs[i], cs, delta, cfl);
}

__global__ void k_wave_speeds(int n, const double4_32a *__restrict__ prim, double *__restrict__ cs)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double P[4];
    ld4(prim[i], P);
    cs[i] = fast64::wave_speed(P);
}

// ------------------------------------------------------------- flux

// Once per cloud: per edge half of {weight of its x half-range (xpos if it lies there,
// else xneg), weight of its y half-range (ypos, else yneg)}, and the gradient's
// 2x2 solve (q_variables_mod.h:112-116) times the edge's weights.
__global__ void k_fold_weights(DevCloud c, double2 *__restrict__ e_w64, double2 *__restrict__ e_gw64)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const int f = c.flag[i];
    const double4_32a m = c.ggeo[i];  // sxx, syy, sxy, 1/det
    const long long base = c.slice_base[i >> 5] + (i & 31);
    for (int j = 0; j < c.nbhs[i]; j++) {
        const long long e = base + 32LL * j;
        const unsigned dir = c.e_dir[e];
        const double2 sn = c.e_sn[e];
        const double4_32a g = c.e_geo[e];
        e_w64[e] = make_double2(0.5 * fast64::flux_weight(c, i, f, (dir & kXpos) ? 0 : 1, sn),
                                0.5 * fast64::flux_weight(c, i, f, (dir & kYpos) ? 2 : 3, sn));
        e_gw64[e] = make_double2(m.w * fast64::diff_of_products(m.y, g.z, m.z, g.w), m.w * fast64::diff_of_products(m.x, g.w, m.z, g.z));
    }
}

// The owner's data of the edge walk: q, its gradient, qmax - q, qmin - q and
// the limiter's eps^2.
struct Owner {
    double q[4], dx[4], dy[4], mx[4], mn[4], e2;
};

__device__ __forceinline__ void load_owner(const DevCloud &c, int i, const double4_32a *__restrict__ q,
                                           const double4_32a *__restrict__ dq, const double4_32a *__restrict__ qm,
                                           Owner &o)
{
    ld4(q[i], o.q);
    ld4(dq[2 * i], o.dx);
    ld4(dq[2 * i + 1], o.dy);
    ld4(qm[2 * i], o.mx);
    ld4(qm[2 * i + 1], o.mn);
#pragma unroll
    for (int r = 0; r < 4; r++) {
        o.mx[r] -= o.q[r];
        o.mn[r] -= o.q[r];
    }
    o.e2 = c.eps2[i];
}

// The weighted flux differences of edge e of point i, all half-ranges, in v
// (component 3 twice): both ends' limited reconstruction and moments once,
// the edge's x and y half-range by a sign per lane, so that the lanes of a
// warp do not diverge on their edges' sub-stencils.  An edge with dels == 0
// (deln == 0) lies in both half-ranges and takes a second, rare pass.
// ends (or NULL): see flux_residual.
__device__ __forceinline__ void edge_flux(const DevCloud &c, int i, int f, double nx, double ny, const Owner &o,
                                          long long e, const double4_32a *__restrict__ q,
                                          const double4_32a *__restrict__ dq, const double4_32a *__restrict__ qm,
                                          double v[4], double *__restrict__ ends, long long ns)
{
    const int k = c.e_nbr[e];
    const double4_32a g = c.e_geo[e];
    const double hx = -0.5 * g.x, hy = -0.5 * g.y;
    fast64::End si, sk;
    double t[4];
    {
        double qk[4], dxk[4], dyk[4], mxk[4], mnk[4];
        ld4(q[k], qk);
        ld4(dq[2 * k], dxk);
        ld4(dq[2 * k + 1], dyk);
        ld4(qm[2 * k], mxk);
        ld4(qm[2 * k + 1], mnk);
        const double e2k = c.eps2[k];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const double dn = fma(hx, dxk[r], __dmul_rn(hy, dyk[r]));
            t[r] = fast64::limited(qk[r], dn, (__double2hiint(dn) >= 0 ? mxk[r] : mnk[r]) - qk[r], e2k);
        }
        fast64::end(c, f, nx, ny, t, sk);
        if (ends) fast64::keep_end(ends + 6 * ns + e, ns, sk);
    }
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const double dn = fma(hx, o.dx[r], __dmul_rn(hy, o.dy[r]));
        t[r] = fast64::limited(o.q[r], dn, __double2hiint(dn) >= 0 ? o.mx[r] : o.mn[r], o.e2);
    }
    fast64::end(c, f, nx, ny, t, si);
    if (ends) fast64::keep_end(ends + e, ns, si);

    const unsigned dir = c.e_dir[e];
    const double2 w = c.e_w64[e];
    const unsigned neg = 0x80000000u;
    const unsigned sx = (dir & kXpos) ? 0u : neg, sy = (dir & kYpos) ? 0u : neg;
    const bool inner = f == kInterior;
    const unsigned s2 = f == kOuter ? 0u : neg;  // the n half range of the quadrant flux
#pragma unroll
    for (int r = 0; r < 4; r++) v[r] = 0.0;
    const double wx = inner ? w.x : 0.0;
    fast64::split_pair(si, sx, sy, -wx, -w.y, v);
    fast64::split_pair(sk, sx, sy, wx, w.y, v);
    if (!inner) {
        fast64::quad_x(si, sx, s2, -w.x, v);
        fast64::quad_x(sk, sx, s2, w.x, v);
    }
    if ((dir & (kXpos | kXneg)) == (kXpos | kXneg)) {
        const double w2 = 0.5 * fast64::flux_weight(c, i, f, 1, c.e_sn[e]);
        if (inner) {
            fast64::split_pair(si, neg, 0u, -w2, 0.0, v);
            fast64::split_pair(sk, neg, 0u, w2, 0.0, v);
        } else {
            fast64::quad_x(si, neg, s2, -w2, v);
            fast64::quad_x(sk, neg, s2, w2, v);
        }
    }
    if ((dir & (kYpos | kYneg)) == (kYpos | kYneg)) {
        const double w2 = 0.5 * fast64::flux_weight(c, i, f, 3, c.e_sn[e]);
        fast64::split_pair(si, 0u, neg, 0.0, -w2, v);
        fast64::split_pair(sk, 0u, neg, 0.0, w2, v);
    }
}

// The flux residual of the block's P points (flux_residual_mod.h:18-87):
// delta times the sum of a point's edge contributions.  Thread t takes point
// t % P and every T / P-th of its edges from t / P on; the contributions meet
// in shared memory and are added in the reference's neighbour order, so the
// result does not depend on P.  Returns true to the threads that hold their
// point's F (threads below `holders` with a point).
constexpr int kFluxThreads = 128;

template <int P>
__device__ __forceinline__ bool block_flux(const DevCloud &c, const double4_32a *__restrict__ q,
                                           const double4_32a *__restrict__ dq, const double4_32a *__restrict__ qm,
                                           const double *__restrict__ delta, double F[4], double *__restrict__ ends,
                                           long long ns, int holders = P)
{
    constexpr int T = kFluxThreads;
    __shared__ double sv[4 * P * kMaxNbhs];
    const int p = threadIdx.x % P, i = blockIdx.x * P + p;
    const bool has = i < c.n;
    const int nb = has ? c.nbhs[i] : 0;
    if (has) {
        const int f = c.flag[i];
        const double2 nn = c.nrm[i];
        const long long base = c.slice_base[i >> 5] + (i & 31);
        Owner o;
        load_owner(c, i, q, dq, qm, o);
        for (int j = threadIdx.x / P; j < nb; j += T / P) {
            double v[4];
            edge_flux(c, i, f, nn.x, nn.y, o, base + 32LL * j, q, dq, qm, v, ends, ns);
#pragma unroll
            for (int r = 0; r < 4; r++) sv[(4 * j + r) * P + p] = v[r];
        }
    }
    // component r = t / P of point t % P; its sum replaces edge 0's contribution
    __syncthreads();
    for (int r = threadIdx.x / P; r < 4; r += T / P) {
        double a = 0.0;
        for (int j = 0; j < nb; j++) a += sv[(4 * j + r) * P + p];
        sv[r * P + p] = a;
    }
    __syncthreads();
    if ((int)threadIdx.x >= holders || !has) return false;
    const double dl = delta[i];
#pragma unroll
    for (int r = 0; r < 4; r++) F[r] = (r == 3 ? 0.5 * dl : dl) * sv[r * P + p];
    return true;
}

// The same for the module path and for the adjoint, with the ends recorded (79%
// of the FP64 pipe).  It keeps k_flux_update's cap of 128 registers and spills 148 B;
// three blocks without the spills were not measured.
template <int P>
__global__ void __launch_bounds__(kFluxThreads, 4) k_flux_residual(DevCloud c, const double4_32a *__restrict__ q,
                                                     const double4_32a *__restrict__ dq, const double4_32a *__restrict__ qm,
                                                     const double *__restrict__ delta, double4_32a *__restrict__ flux_res,
                                                     double *__restrict__ ends, long long ns)
{
    double F[4];
    if (block_flux<P>(c, q, dq, qm, delta, F, ends, ns)) flux_res[blockIdx.x * P + threadIdx.x] = mk4(F);
}

// Sum and maximum of res_sqr over each 8 consecutive points (lanes of one
// aligned group of 8, all of them calling), the partials the residual norm is
// reduced from: the same grouping under every launch shape.
__device__ __forceinline__ void partial8(double v, int i, int n, double *__restrict__ psum, double *__restrict__ pmax)
{
    const unsigned mask = 0xffu << (threadIdx.x & 24u);
    double m = v;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        v += __shfl_down_sync(mask, v, o, 8);
        const double t = __shfl_down_sync(mask, m, o, 8);
        m = t > m ? t : m;
    }
    if ((i & 7) == 0 && i < n) {
        psum[i >> 3] = v;
        pmax[i >> 3] = m;
    }
}

// state_update_mod.h:92-283 over all points, with the residual's partial sums
// (prim_next may be prim).
__global__ void __launch_bounds__(kPointBlock) k_state_update(DevCloud c, CaseConst K, const double4_32a *prim,
                                                      const double4_32a *__restrict__ prim_old,
                                                      const double4_32a *__restrict__ flux_res,
                                                      double4_32a *prim_next, int rk, double *__restrict__ psum,
                                                      double *__restrict__ pmax)
{
    const int i = blockIdx.x * kPointBlock + threadIdx.x;
    double r2 = 0.0;
    if (i < c.n) {
        const double2 nn = c.nrm[i];
        double P[4], F[4];
        ld4(prim[i], P);
        ld4(flux_res[i], F);
        r2 = fast64::stage(K, c.gauss_tab, c.flag[i], nn.x, nn.y, P, prim_old + i, F, rk);
        prim_next[i] = mk4(P);
    }
    partial8(r2, i, c.n, psum, pmax);
}

// Fused stage: flux residual + SSPRK update of the block's points, then q and
// (after the last stage) the wave speed of the new state for the next stage's
// kernels.  Bound by the FP64 pipe, about 200 FP64 instructions per edge and
// 110 per point.  Measured on 204,800 points (2.05 M edges, inner 3): 2908 us
// per launch with CUDA's exp / erf / rsqrt, all four half-range fluxes at every
// edge and 32 directional sums (about 630 per edge), 1066 us in this form with
// a thread per point, 951 us with the edges spread (flux_shape), 898 us with
// the quotient, the reciprocals and the half weights in their present forms
// (220 -> 200 per edge, FP64 pipe 87% active).  Four blocks of 128 registers a
// thread per SM, which spill 32 B: 5% over three blocks at 146.
template <int P>
__global__ void __launch_bounds__(kFluxThreads, 4) k_flux_update(DevCloud c, CaseConst K, const double4_32a *__restrict__ q,
                                                   const double4_32a *__restrict__ dq,
                                                   const double4_32a *__restrict__ qm,
                                                   const double *__restrict__ delta,
                                                   const double4_32a *__restrict__ prim,
                                                   const double4_32a *__restrict__ prim_old,
                                                   double4_32a *__restrict__ prim_next, double4_32a *__restrict__ q_next,
                                                   double *__restrict__ cs_next, int rk,
                                                   double *__restrict__ psum, double *__restrict__ pmax)
{
    // Below 32 points the first warp has lanes to spare: lanes P to 2 P work on the
    // same points as the first P and take the logarithm of beta beside that of rho
    // (one instruction stream instead of two: 333 -> 326.5 us per iteration at 9,600
    // points, 155.5 -> 152 at 960; two warps would pay twice for the rest at P = 32).
    constexpr int H = P < 32 ? 2 * P : P;
    double F[4], S[4], r2 = 0.0, lg = 0.0;
    const int i = blockIdx.x * P + threadIdx.x % P;
    const bool has = block_flux<P>(c, q, dq, qm, delta, F, nullptr, 0, H);
    if (has) {
        const double2 nn = c.nrm[i];
        ld4(prim[i], S);
        r2 = fast64::stage(K, c.gauss_tab, c.flag[i], nn.x, nn.y, S, prim_old + i, F, rk);
        if (H > P) lg = log(threadIdx.x < P ? S[0] : fast64::beta_of(S));
    }
    if (threadIdx.x >= H) return;
    double lb = 0.0;
    if (H > P) lb = __shfl_down_sync(H == 32 ? 0xffffffffu : (1u << H) - 1u, lg, P);
    if (threadIdx.x >= P) return;
    if (has) {
        double Q[4];
        if (H > P) fast64::q_of(S, lg, lb, Q);
        else fast64::q_of(S, Q);
        prim_next[i] = mk4(S);
        q_next[i] = mk4(Q);
        if (cs_next) cs_next[i] = fast64::wave_speed(S);
    }
    if (psum) partial8(r2, i, c.n, psum, pmax);
}

// fpi_solver_mod.h:138-147: res_new = sqrt(sum)/n, residue against res_old
// latched at iterations 1 and 2; one block, fixed summation order.
// One block of RB threads: each thread sums a strided share of the block
// partials with four independent accumulators (its loads in flight together
// instead of one dependent chain), then a tree over the block; the order is
// fixed, so the result is the same on every run.  Every iteration waits for this
// one block, so sums of zeros are left out (accumulators and tree levels that no
// partial reaches: 32 warps of them are 512 FP64 cycles each) and the last
// levels are shuffles: iteration of 9,600 points, mixed 65.2 -> 63.2 us, of 960
// points, FP64 151.6 -> 149.4.
constexpr int RB = 1024;
__global__ void __launch_bounds__(RB) k_reduce_residual(int nblocks, const double *__restrict__ psum,
                                                       const double *__restrict__ pmax, int n, int it_arg,
                                                       double *hist, int capacity, double *res_old, int *iter,
                                                       int *status, int latch)
{
    __shared__ double ss[RB], sm[RB];
    begin_dependent();
    double v[4] = {0.0, 0.0, 0.0, 0.0}, mm[4] = {0.0, 0.0, 0.0, 0.0};
    int b = threadIdx.x;
    for (; b + 3 * RB < nblocks; b += 4 * RB) {
#pragma unroll
        for (int u = 0; u < 4; u++) {
            v[u] += psum[b + u * RB];
            const double x = pmax[b + u * RB];
            mm[u] = x > mm[u] ? x : mm[u];
        }
    }
    for (; b < nblocks; b += RB) {
        v[0] += psum[b];
        mm[0] = pmax[b] > mm[0] ? pmax[b] : mm[0];
    }
    double x = v[0], m = mm[0];
    if (nblocks > 3 * RB) {  // the other accumulators are zero below
        x = (v[0] + v[1]) + (v[2] + v[3]);
        for (int u = 1; u < 4; u++) m = mm[u] > m ? mm[u] : m;
    }
    ss[threadIdx.x] = x;
    sm[threadIdx.x] = m;
    // levels whose upper half holds no partial would add zeros
    int s = RB / 2;
    while (s >= nblocks && s > 16) s >>= 1;
    __syncthreads();
    for (; s > 16; s >>= 1) {
        if (threadIdx.x < s) {
            ss[threadIdx.x] += ss[threadIdx.x + s];
            sm[threadIdx.x] = sm[threadIdx.x + s] > sm[threadIdx.x] ? sm[threadIdx.x + s] : sm[threadIdx.x];
        }
        __syncthreads();
    }
    if (threadIdx.x >= 32) return;
    x = ss[threadIdx.x];
    m = sm[threadIdx.x];
    for (s = 16; s > 0; s >>= 1) {
        x += __shfl_down_sync(0xffffffffu, x, s);
        const double t = __shfl_down_sync(0xffffffffu, m, s);
        m = t > m ? t : m;
    }
    if (threadIdx.x == 0) {
        int it = it_arg > 0 ? it_arg : *iter + 1;
        double res_new = sqrt(x) / n;
        double residue;
        if (it <= 2 && latch) {
            *res_old = res_new;
            residue = 0;
        } else {
            residue = log10(res_new / *res_old);
        }
        if (it - 1 < capacity && it >= 1) {
            hist[3 * (it - 1)] = res_new;
            hist[3 * (it - 1) + 1] = residue;
            hist[3 * (it - 1) + 2] = m;
        }
        *iter = it;
        if (!isfinite(res_new)) *status = 1;
    }
}

__global__ void k_copy(int n, const double4_32a *__restrict__ src, double4_32a *__restrict__ dst)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[i];
}

// Point states between the cloud's order and the handle's (Morton / class)
// order: dst[perm[i]] = src[i] (in) or dst[i] = src[perm[i]] (out).
__global__ void k_permute_in(int n, const int *__restrict__ perm, const double4_32a *__restrict__ src,
                             double4_32a *__restrict__ dst)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[perm[i]] = src[i];
}

__global__ void k_permute_out(int n, const int *__restrict__ perm, const double4_32a *__restrict__ src,
                              double4_32a *__restrict__ dst)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[perm[i]];
}

__global__ void k_add(int n, const double4_32a *__restrict__ src, double4_32a *__restrict__ dst)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const double4_32a a = src[i], b = dst[i];
        dst[i] = make_double4_32a(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
    }
}

// compute_force_coeffs_mod.h:37-72 per shape point and compute_entropy_mod.h:
// 17-21 per point; each block writes its partial sums of H, V, pitching
// moment and entropy, k_objective_finish adds the partials in a fixed order.
// wall_geo per shape point: x = ds, y = mx - 0.25, z = my.
__global__ void __launch_bounds__(256) k_objective(DevCloud c, const double4_32a *__restrict__ prim,
                                                   const int *__restrict__ wall_perm,
                                                   const double4_32a *__restrict__ wall_geo, int n_wall,
                                                   double cp_scale, double pr_inf, double gamma,
                                                   double *__restrict__ entropy, double *__restrict__ partial)
{
    __shared__ double sh[4][256];
    const int t = blockIdx.x * 256 + threadIdx.x;
    double H = 0, V = 0, Mo = 0, E = 0;
    if (t < n_wall) {
        const int m = wall_perm[t];
        const double4_32a w = wall_geo[t];
        const double2 nn = c.nrm[m];
        double cp = prim[m].w - pr_inf;
        cp = -cp / cp_scale;
        H = cp * nn.x * w.x;
        V = cp * nn.y * w.x;
        Mo = (-cp * nn.y * w.x * w.y + cp * nn.x * w.x * w.z);
    }
    if (entropy && t < c.n) {
        const double4_32a P = prim[t];
        double temp1 = pow(P.x, gamma);
        temp1 = P.w / temp1;
        temp1 = log(temp1);
        const double s = fabs(temp1 - log(pr_inf));
        entropy[t] = s;
        E = s;
    }
    sh[0][threadIdx.x] = H;
    sh[1][threadIdx.x] = V;
    sh[2][threadIdx.x] = Mo;
    sh[3][threadIdx.x] = E;
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
        if (threadIdx.x < st)
            for (int q = 0; q < 4; q++) sh[q][threadIdx.x] += sh[q][threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x < 4) partial[4 * blockIdx.x + threadIdx.x] = sh[threadIdx.x][0];
}

__global__ void k_objective_finish(int nblocks, const double *__restrict__ partial, double *__restrict__ out4)
{
    __shared__ double sh[4][256];
    double v[4] = {0, 0, 0, 0};
    for (int b = threadIdx.x; b < nblocks; b += 256)
        for (int q = 0; q < 4; q++) v[q] += partial[4 * b + q];
    for (int q = 0; q < 4; q++) sh[q][threadIdx.x] = v[q];
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
        if (threadIdx.x < st)
            for (int q = 0; q < 4; q++) sh[q][threadIdx.x] += sh[q][threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x < 4) out4[threadIdx.x] = sh[threadIdx.x][0];
}

// ------------------------------------------------------------ diagnostics

// compute_enstrophy_mod.h:5-75: vorticity du2/dx - du1/dy by least squares
// over the full stencil (the gradient's weights and moments), its square, and
// per-block partial sums of the squares.
__global__ void __launch_bounds__(256) k_enstrophy(DevCloud c, const double4_32a *__restrict__ prim,
                                                   double *__restrict__ vort, double *__restrict__ partial)
{
    __shared__ double sh[256];
    const int i = blockIdx.x * 256 + threadIdx.x;
    double v2 = 0.0;
    if (i < c.n) {
        const double4_32a Pi = prim[i];
        double sx1 = 0., sx2 = 0., sy1 = 0., sy2 = 0.;
        const int nb = c.nbhs[i];
        const long long base = c.slice_base[i >> 5] + (i & 31);
        for (int j = 0; j < nb; j++) {
            const long long e = base + 32LL * j;
            const int k = c.e_nbr[e];
            const double4_32a g = c.e_geo[e];       // delx, dely, w delx, w dely
            const double4_32a Pk = prim[k];
            sx1 = sx1 + g.z * (Pk.y - Pi.y);
            sx2 = sx2 + g.z * (Pk.z - Pi.z);
            sy1 = sy1 + g.w * (Pk.y - Pi.y);
            sy2 = sy2 + g.w * (Pk.z - Pi.z);
        }
        const double4_32a m = c.ggeo[i];           // sxx, syy, sxy, 1/det
        const double du2_dx = (sx2 * m.y - sy2 * m.z) * m.w;
        const double du1_dy = (sy1 * m.x - sx1 * m.z) * m.w;
        const double t = du2_dx - du1_dy;
        vort[i] = t;
        v2 = t * t;
    }
    sh[threadIdx.x] = v2;
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
        if (threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

// Stagnation pressure p0 = p (1 + (gamma - 1)/2 M^2)^(gamma / (gamma - 1)) per
// point (stagnation_values_mod.h:9-48): per block the minimum and maximum
// (first index on ties), the sum of (p0_inf - p0)^2 (:51-80) and of p0.
// partial [blocks][6]: min, argmin, max, argmax, sum of squares, sum.
__global__ void __launch_bounds__(256) k_stagnation(int n, const double4_32a *__restrict__ prim, double gamma,
                                                    double p0_inf, double *__restrict__ partial)
{
    __shared__ double smin[256], smax[256], ssum[256], sp0[256];
    __shared__ int imin[256], imax[256];
    const int i = blockIdx.x * 256 + threadIdx.x;
    double p0 = 0.0, sq = 0.0;
    const double gp = gamma / (gamma - 1);
    if (i < n) {
        const double4_32a P = prim[i];
        const double angle = sqrt(gamma * P.w / P.x);
        const double mach_t = sqrt(pow(P.y, 2) + pow(P.z, 2)) / angle;
        p0 = P.w * pow(1 + ((gamma - 1) / 2) * mach_t * mach_t, gp);
        sq = pow(p0_inf - p0, 2);
    }
    const bool ok = i < n;
    smin[threadIdx.x] = ok ? p0 : INFINITY;
    smax[threadIdx.x] = ok ? p0 : -INFINITY;
    imin[threadIdx.x] = imax[threadIdx.x] = ok ? i : 0x7fffffff;
    ssum[threadIdx.x] = sq;
    sp0[threadIdx.x] = p0;
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
        const int t = threadIdx.x;
        if (t < st) {
            const int u = t + st;
            if (smin[u] < smin[t] || (smin[u] == smin[t] && imin[u] < imin[t])) { smin[t] = smin[u]; imin[t] = imin[u]; }
            if (smax[u] > smax[t] || (smax[u] == smax[t] && imax[u] < imax[t])) { smax[t] = smax[u]; imax[t] = imax[u]; }
            ssum[t] += ssum[u];
            sp0[t] += sp0[u];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        double *o = partial + 6 * (size_t)blockIdx.x;
        o[0] = smin[0];
        o[1] = (double)imin[0];
        o[2] = smax[0];
        o[3] = (double)imax[0];
        o[4] = ssum[0];
        o[5] = sp0[0];
    }
}

// ------------------------------------------------------------- launchers

// Points per block (of 128 threads) of the flux kernels by the number of
// points; the result is the same under each.  The kernels are bound by the FP64
// pipe, so what counts is that all SMs have work and end together: with one
// thread walking a point's edges, a small cloud keeps few SMs busy for the 10
// to 20 edges of its longest lists; with fewer points per block the last edges
// and the update leave lanes idle, which costs where every SM is full anyway.
// Measured per launch (us, inner 0):
//   points                       960  9,600  30,720  51,200  102,400  204,800
//   a thread per point           228    217     281     329      649     1061
//   8 per block, 128 threads      32     75     193     305      596     1163
//   16                            42     79     169     261      493      946
//   32                            64     85     196     262      479      898
// (the first row before the shorter quotient and reciprocals, 6% on the others).
template <typename F> void flux_shape(int n, F &&launch)
{
    using std::integral_constant;
    if (n <= 12288) launch(integral_constant<int, 8>{});
    else if (n <= 65536) launch(integral_constant<int, 16>{});
    else launch(integral_constant<int, 32>{});
}

#define QLSKUM_LAUNCHED(L) \
    do { if ((L).launches) ++*(L).launches; } while (0)

void fold_weights(const Launch &L, const DevCloud &c, double2 *e_w64, double2 *e_gw64)
{
    k_fold_weights<<<grid_for(c.n, 128), 128, 0, L.stream>>>(c, e_w64, e_gw64);
    QLSKUM_LAUNCHED(L);
}

void q_variables(const Launch &L, const DevCloud &c, const double4_32a *prim, double4_32a *q)
{
    k_q_variables<<<grid_for(c.n, kPointBlock), kPointBlock, 0, L.stream>>>(c.n, prim, q);
    QLSKUM_LAUNCHED(L);
}

void derived(const Launch &L, const DevCloud &c, const double4_32a *prim, double4_32a *q, double *cspeed)
{
    k_derived<<<grid_for(c.n, kPointBlock), kPointBlock, 0, L.stream>>>(c.n, prim, q, cspeed);
    QLSKUM_LAUNCHED(L);
}

void q_derivatives(const Launch &L, const DevCloud &c, const double4_32a *q, double4_32a *dq, double4_32a *qm,
                   const double *cspeed, double *delta, double cfl)
{
    const double *q1 = reinterpret_cast<const double *>(q);
    double *dq1 = reinterpret_cast<double *>(dq), *qm1 = reinterpret_cast<double *>(qm);
    const int g = grid_for(4 * (long long)c.n, L.block);
    if (delta) k_q_derivatives<true><<<g, L.block, 0, L.stream>>>(c, q1, dq1, qm1, cspeed, delta, cfl);
    else k_q_derivatives<false><<<g, L.block, 0, L.stream>>>(c, q1, dq1, qm1, nullptr, nullptr, cfl);
    QLSKUM_LAUNCHED(L);
}

void q_inner(const Launch &L, const DevCloud &c, const double4_32a *q, const double4_32a *dq0, const double4_32a *dq_in,
             double4_32a *dq_out)
{
    const double *q1 = reinterpret_cast<const double *>(q), *d0 = reinterpret_cast<const double *>(dq0),
                 *in = reinterpret_cast<const double *>(dq_in);
    double *out = reinterpret_cast<double *>(dq_out);
    const int g = grid_for(4 * (long long)c.n, L.block);
    if (dq0) k_q_inner<false><<<g, L.block, 0, L.stream>>>(c, nullptr, d0, in, out);
    else k_q_inner<true><<<g, L.block, 0, L.stream>>>(c, q1, nullptr, in, out);
    QLSKUM_LAUNCHED(L);
}

void wave_speeds(const Launch &L, int n, const double4_32a *prim, double *cs)
{
    k_wave_speeds<<<grid_for(n, kPointBlock), kPointBlock, 0, L.stream>>>(n, prim, cs);
    QLSKUM_LAUNCHED(L);
}

void func_delta(const Launch &L, const DevCloud &c, const double4_32a *prim, double *cs, double *delta, double cfl)
{
    wave_speeds(L, c.n, prim, cs);
    k_func_delta<<<grid_for(4 * (long long)c.n, L.block), L.block, 0, L.stream>>>(c, cs, delta, cfl);
    QLSKUM_LAUNCHED(L);
}

void flux_residual(const Launch &L, const DevCloud &c, const double4_32a *q, const double4_32a *dq, const double4_32a *qm,
                   const double *delta, double4_32a *flux_res, double *ends, long long ns)
{
    flux_shape(c.n, [&](auto p) {
        constexpr int P = decltype(p)::value;
        k_flux_residual<P><<<grid_for(c.n, P), kFluxThreads, 0, L.stream>>>(c, q, dq, qm, delta, flux_res, ends, ns);
    });
    QLSKUM_LAUNCHED(L);
}

void state_update(const Launch &L, const DevCloud &c, const CaseConst &k, const double4_32a *prim,
                  const double4_32a *prim_old, const double4_32a *flux_res, double4_32a *prim_next, int rk,
                  const Reduce &R)
{
    k_state_update<<<grid_for(c.n, kPointBlock), kPointBlock, 0, L.stream>>>(c, k, prim, prim_old, flux_res, prim_next, rk,
                                                             R.partial_sum, R.partial_max);
    QLSKUM_LAUNCHED(L);
}

void flux_update(const Launch &L, const DevCloud &c, const CaseConst &k, const double4_32a *q, const double4_32a *dq,
                 const double4_32a *qm, const double *delta, const double4_32a *prim, const double4_32a *prim_old,
                 double4_32a *prim_next, double4_32a *q_next, double *cspeed_next, int rk, const Reduce &R)
{
    flux_shape(c.n, [&](auto p) {
        constexpr int P = decltype(p)::value;
        k_flux_update<P><<<grid_for(c.n, P), kFluxThreads, 0, L.stream>>>(c, k, q, dq, qm, delta, prim, prim_old,
                                                                          prim_next, q_next, cspeed_next, rk,
                                                                          R.partial_sum, R.partial_max);
    });
    QLSKUM_LAUNCHED(L);
}

void reduce_residual(const Launch &L, const Reduce &R, int n, int it)
{
    launch_after(L, k_reduce_residual, 1, RB, 0, R.blocks, R.partial_sum, R.partial_max, n, it, R.hist, R.capacity,
                 R.res_old, R.iter, R.status, R.latch);
    QLSKUM_LAUNCHED(L);
}

void copy_prim(const Launch &L, int n, const double4_32a *src, double4_32a *dst)
{
    k_copy<<<grid_for(n, 256), 256, 0, L.stream>>>(n, src, dst);
    QLSKUM_LAUNCHED(L);
}

// out[0] = max over the n points and components of |a - b|, out[1] of |a|,
// as the bit patterns of non-negative doubles (which order like the values),
// per-warp maxima then one atomicMax per warp; out zeroed by the caller.
__global__ void k_max_change(int n, const double4_32a *__restrict__ a, const double4_32a *__restrict__ b,
                             unsigned long long *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double d = 0.0, m = 0.0;
    if (i < n) {
        const double4_32a x = a[i], y = b[i];
        d = fmax(fmax(fabs(x.x - y.x), fabs(x.y - y.y)), fmax(fabs(x.z - y.z), fabs(x.w - y.w)));
        m = fmax(fmax(fabs(x.x), fabs(x.y)), fmax(fabs(x.z), fabs(x.w)));
    }
    for (int o = 16; o > 0; o >>= 1) {
        d = fmax(d, __shfl_down_sync(0xffffffffu, d, o));
        m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(out, (unsigned long long)__double_as_longlong(d));
        atomicMax(out + 1, (unsigned long long)__double_as_longlong(m));
    }
}

void max_change(const Launch &L, int n, const double4_32a *a, const double4_32a *b, unsigned long long *out)
{
    k_max_change<<<grid_for(n, 256), 256, 0, L.stream>>>(n, a, b, out);
    QLSKUM_LAUNCHED(L);
}

__global__ void k_set_int(int *p, int v) { *p = v; }

void set_counter(const Launch &L, int *p, int v)
{
    k_set_int<<<1, 1, 0, L.stream>>>(p, v);
    QLSKUM_LAUNCHED(L);
}

// dst[i] = v for the n points.
__global__ void k_fill(int n, double4_32a v, double4_32a *__restrict__ dst)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = v;
}

void fill_prim(const Launch &L, int n, double4_32a v, double4_32a *dst)
{
    k_fill<<<grid_for(n, 256), 256, 0, L.stream>>>(n, v, dst);
    QLSKUM_LAUNCHED(L);
}

// out[0] += sum of src.y, out[1] += sum of src.z over the n points (warp
// sums, one atomic per warp).
__global__ void k_sum_yz(int n, const double4_32a *__restrict__ src, double *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double a = 0.0, b = 0.0;
    if (i < n) {
        const double4_32a v = src[i];
        a = v.y;
        b = v.z;
    }
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(out, a);
        atomicAdd(out + 1, b);
    }
}

void sum_yz(const Launch &L, int n, const double4_32a *src, double *out)
{
    k_sum_yz<<<grid_for(n, 256), 256, 0, L.stream>>>(n, src, out);
    QLSKUM_LAUNCHED(L);
}

void permute_in(const Launch &L, int n, const int *perm, const double4_32a *src, double4_32a *dst)
{
    k_permute_in<<<grid_for(n, 256), 256, 0, L.stream>>>(n, perm, src, dst);
    QLSKUM_LAUNCHED(L);
}

void permute_out(const Launch &L, int n, const int *perm, const double4_32a *src, double4_32a *dst)
{
    k_permute_out<<<grid_for(n, 256), 256, 0, L.stream>>>(n, perm, src, dst);
    QLSKUM_LAUNCHED(L);
}

void add_prim(const Launch &L, int n, const double4_32a *src, double4_32a *dst)
{
    k_add<<<grid_for(n, 256), 256, 0, L.stream>>>(n, src, dst);
    QLSKUM_LAUNCHED(L);
}

void enstrophy(const Launch &L, const DevCloud &c, const double4_32a *prim, double *vort, double *partial)
{
    k_enstrophy<<<grid_for(c.n, 256), 256, 0, L.stream>>>(c, prim, vort, partial);
    QLSKUM_LAUNCHED(L);
}

void stagnation(const Launch &L, int n, const double4_32a *prim, double gamma, double p0_inf, double *partial)
{
    k_stagnation<<<grid_for(n, 256), 256, 0, L.stream>>>(n, prim, gamma, p0_inf, partial);
    QLSKUM_LAUNCHED(L);
}

void objective(const Launch &L, const DevCloud &c, const double4_32a *prim, const int *wall_perm,
               const double4_32a *wall_geo, int n_wall, double cp_scale, double pr_inf, double gamma, double *entropy,
               double *out4, double *scratch)
{
    // entropy NULL: the force coefficients only (the wall points)
    const int items = (entropy && c.n > n_wall) ? c.n : n_wall;
    const int blocks = grid_for(items, 256);
    k_objective<<<blocks, 256, 0, L.stream>>>(c, prim, wall_perm, wall_geo, n_wall, cp_scale, pr_inf, gamma, entropy,
                                              scratch);
    k_objective_finish<<<1, 256, 0, L.stream>>>(blocks, scratch, out4);
    if (L.launches) *L.launches += 2;
}

}  // namespace fp64

namespace halo {

// One thread per (ghost, 16-byte word) of the element.
__global__ void k_pull16(int n, int w, const int *__restrict__ idx, const float4 *__restrict__ src,
                         float4 *__restrict__ dst)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)n * w) return;
    const int g = (int)(t / w), j = (int)(t - (long long)g * w);
    dst[t] = src[(long long)idx[g] * w + j];
}

template <typename T>
__global__ void k_pull(int n, const int *__restrict__ idx, const T *__restrict__ src, T *__restrict__ dst)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < n) dst[g] = src[idx[g]];
}

void pull(const Launch &L, int n, const int *idx, const void *src, void *dst, int bytes)
{
    if (n <= 0) return;
    if (bytes == 4) {
        k_pull<float><<<fp64::grid_for(n, 256), 256, 0, L.stream>>>(n, idx, static_cast<const float *>(src),
                                                             static_cast<float *>(dst));
    } else if (bytes == 8) {
        k_pull<double><<<fp64::grid_for(n, 256), 256, 0, L.stream>>>(n, idx, static_cast<const double *>(src),
                                                              static_cast<double *>(dst));
    } else {
        const int w = bytes / 16;
        const long long items = (long long)n * w;
        k_pull16<<<(int)((items + 255) / 256), 256, 0, L.stream>>>(n, w, idx, static_cast<const float4 *>(src),
                                                                    static_cast<float4 *>(dst));
    }
    if (L.launches) ++*L.launches;
}

}  // namespace halo
}  // namespace qlskum
