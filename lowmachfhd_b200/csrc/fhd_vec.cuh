// fhd_vec.cuh -- Stokes-vector kernels: the fused saddle-point operator,
// preconditioner glue, deterministic reductions and the Gram-Schmidt steps
// of GMRES.
#pragma once
#include "fhd_kernels.cuh"

namespace fhd {

// A Stokes vector (u_0 .. u_{dim-1}, p): component pointers, p at [dim].
template <typename T>
struct SVec {
    T* c[4];
};
template <typename T>
struct CSVec {
    const T* c[4];
};

// ---------------------------------------------------------------------
// deterministic reductions: grid-stride partial sums, a warp-shuffle tree
// per block, one partial per block, and the last block to finish adds the
// partials in block order.  The result lands in device memory so that
// following kernels can consume it without a host round trip.
// ---------------------------------------------------------------------
constexpr int RED_THREADS = 256;
constexpr int RED_MAX_BLOCKS = 1184;  // 8 blocks per SM on 148 SMs

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ double block_sum(double v, double* sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    v = warp_sum(v);
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    const int nw = blockDim.x >> 5;
    v = (threadIdx.x < nw) ? sh[threadIdx.x] : 0.0;
    if (wid == 0) v = warp_sum(v);
    __syncthreads();
    return v;  // valid in thread 0
}

struct RedSlot {
    double* partials;    // RED_MAX_BLOCKS entries
    unsigned* counter;   // zero between uses
    double* out;
};

__device__ __forceinline__ void red_finish(double v, RedSlot rs) {
    __shared__ double sh[32];
    __shared__ bool last;
    v = block_sum(v, sh);
    if (threadIdx.x == 0) {
        rs.partials[blockIdx.x] = v;
        __threadfence();
        const unsigned t = atomicAdd(rs.counter, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double s = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) s += ((volatile double*)rs.partials)[b];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) {
        *rs.out = s;
        *rs.counter = 0u;
    }
}

// ---------------------------------------------------------------------
// Orthogonalisation of a new Krylov vector w against i others
// (gmres.f90:352-389), two passes over the vectors, GS_MAXV at a time, instead of
// one per vector.  Modified Gram-Schmidt takes h_k = <w - sum_{j<k} h_j v_j, v_k>,
// that is h_k = <w, v_k> - sum_{j<k} h_j <v_j, v_k>: all products <w, v_k> and
// the new row of <v_j, v_k> come from one pass (k_gs_dots, whose last block
// solves for h), and w - sum h_k v_k with its norm from a second
// (k_gs_update).  The loss of orthogonality stays that of modified
// Gram-Schmidt, whose coefficients these are.
//
// The vectors are kept as computed (u_k, with n2_k = |u_k|^2) rather than
// scaled to length one: v_k = u_k / |u_k| enters through its coefficients,
// and the operator scales its result (k_stokes_apply's inv).  So a step of
// i <= GS_MAXV moves 2 i + 3 vectors where one pass per vector and the scaling
// moved 4 i + 3; every further GS_MAXV vectors read w, u_{i-1} and the partly
// updated vector again and write it, 4 more.
//
// Bound: DRAM (192^3, five vectors: dots 279 us, update 281 us for 1.6 GB,
// 5.6 TB/s).  Seven steps of the 192^3 solve with their norms: 5.2 ms one
// vector at a time with the scaling, 2.7 ms now.  Four resident blocks per SM
// and all components of an element loaded together keep enough bytes in
// flight (|w|^2 at 192^3: 97 us with one component after the other, 42 now).
// ---------------------------------------------------------------------
constexpr int GS_MAXV = 6;      // vectors per launch
constexpr int GS_BLOCKS = 592;  // 4 blocks of 256 threads per SM
constexpr int GS_MAXM = 64;

// device scalars of the orthogonalisation, vector index 0-based
struct GSData {
    double* h;        // h_1.. of the current column, at [1 + k]
    double* n2;       // |u_k|^2
    double* inv;      // 1 / |u_k|
    double* coef;     // h_k / |u_k|
    double* d;        // <w, u_k>
    double* g;        // <u_{i-1}, u_k>
    double* gram;     // <v_j, v_k> at [k * GS_MAXM + j], j < k
    double* partials; // GS_BLOCKS x 2 GS_MAXV
    unsigned* counter;
};

// block sums of N values per thread, then over the blocks in block order by
// the last block; true there, with the sums in out[0 .. N)
template <int N>
__device__ __forceinline__ bool red_many(const double (&v)[N], double* partials, unsigned* counter, double* out) {
    __shared__ double sh[N][RED_THREADS / 32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = RED_THREADS / 32;
#pragma unroll
    for (int q = 0; q < N; q++) {
        const double s = warp_sum(v[q]);
        if (lane == 0) sh[q][wid] = s;
    }
    __syncthreads();
    if (threadIdx.x < N) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < nw; k++) s += sh[threadIdx.x][k];
        partials[(size_t)threadIdx.x * GS_BLOCKS + blockIdx.x] = s;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = (atomicAdd(counter, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!last) return false;
    __threadfence();
    for (int q = wid; q < N; q += nw) {
        double s = 0.0;
        for (int b = lane; b < (int)gridDim.x; b += 32) s += __ldcg(partials + (size_t)q * GS_BLOCKS + b);
        s = warp_sum(s);
        if (lane == 0) out[q] = s;
    }
    if (threadIdx.x == 0) *counter = 0u;
    __syncthreads();
    return true;
}

// weighted |a|^2 (weight 1 for the velocity, wp2 for the pressure); with its
// inverse root where inv is not null
template <int NC>
static __global__ void __launch_bounds__(RED_THREADS, 4) k_norm2(i64 n, CSVec<double> a, double wp2, double* out,
                                                                 double* inv, double* partials, unsigned* counter) {
    __shared__ double tot[1];
    double s[1] = {0.0};
    for (i64 f = blockIdx.x * (i64)blockDim.x + threadIdx.x; f < n; f += (i64)gridDim.x * blockDim.x) {
        double x[NC];
#pragma unroll
        for (int c = 0; c < NC; c++) x[c] = a.c[c][f];
        double su = 0.0;
#pragma unroll
        for (int c = 0; c < NC - 1; c++) su += x[c] * x[c];
        su += wp2 * (x[NC - 1] * x[NC - 1]);
        s[0] += su;
    }
    if (!red_many<1>(s, partials, counter, tot) || threadIdx.x) return;
    *out = tot[0];
    if (inv) *inv = 1.0 / sqrt(tot[0]);
}

// sums of the N fields of a into out[0 .. N), in one pass (one launch for the
// null space of the preconditioner: a 64^2 field's sum costs its launch, 3.3 us
// each one by one)
template <int N>
static __global__ void __launch_bounds__(RED_THREADS, 4) k_sums(i64 n, CSVec<double> a, double* out, double* partials,
                                                                unsigned* counter) {
    double s[N];
#pragma unroll
    for (int c = 0; c < N; c++) s[c] = 0.0;
    for (i64 f = blockIdx.x * (i64)blockDim.x + threadIdx.x; f < n; f += (i64)gridDim.x * blockDim.x)
#pragma unroll
        for (int c = 0; c < N; c++) s[c] += a.c[c][f];
    __shared__ double tot[N];
    if (!red_many<N>(s, partials, counter, tot)) return;
    if (threadIdx.x < N) out[threadIdx.x] = tot[threadIdx.x];
}

// the fields less their means sum[c] / count
template <int N>
static __global__ void __launch_bounds__(256) k_sub_means(i64 n, SVec<double> a, const double* sum, double count) {
    double m[N];
#pragma unroll
    for (int c = 0; c < N; c++) m[c] = sum[c] / count;
    for (i64 f = blockIdx.x * (i64)blockDim.x + threadIdx.x; f < n; f += (i64)gridDim.x * blockDim.x)
#pragma unroll
        for (int c = 0; c < N; c++) a.c[c][f] = a.c[c][f] - m[c];
}

// <w, u_k> and <u_{i-1}, u_k> for k = k0 .. k0 + NV - 1; the last block of the
// launch that reaches k = i - 1 solves for h_k
template <int NC, int NV>
static __global__ void __launch_bounds__(RED_THREADS, 4) k_gs_dots(i64 n, CSVec<double> w, const double* __restrict__ V,
                                                                   i64 vstride, int k0, int i, double wp2, GSData G) {
    __shared__ double tot[2 * NV];
    double s[2 * NV];
#pragma unroll
    for (int q = 0; q < 2 * NV; q++) s[q] = 0.0;
    const double* __restrict__ ul = V + (i64)(i - 1) * vstride;
    const double* __restrict__ uk = V + (i64)k0 * vstride;
    for (i64 f = blockIdx.x * (i64)blockDim.x + threadIdx.x; f < n; f += (i64)gridDim.x * blockDim.x) {
        double x[NC], l[NC];
#pragma unroll
        for (int c = 0; c < NC; c++) {
            x[c] = w.c[c][f];
            l[c] = ul[(i64)c * n + f];
        }
        x[NC - 1] *= wp2;
        l[NC - 1] *= wp2;
#pragma unroll
        for (int v = 0; v < NV; v++) {
            double a = 0.0, b = 0.0;
#pragma unroll
            for (int c = 0; c < NC; c++) {
                const double u = uk[v * vstride + (i64)c * n + f];
                a += x[c] * u;
                b += l[c] * u;
            }
            s[v] += a;
            s[NV + v] += b;
        }
    }
    if (!red_many<2 * NV>(s, G.partials, G.counter, tot)) return;
    const int t = threadIdx.x;
    if (t < NV) {
        G.d[k0 + t] = tot[t];
        G.g[k0 + t] = tot[NV + t];
    }
    if (k0 + NV < i) return;
    __syncthreads();
    // h = (I + L)^-1 <w, v>, L the strictly lower triangle of <v_j, v_k>
    double* row = G.gram + (size_t)(i - 1) * GS_MAXM;
    for (int k = t; k < i - 1; k += blockDim.x) row[k] = G.g[k] * G.inv[i - 1] * G.inv[k];
    __syncthreads();
    if (t != 0) return;
    for (int k = 0; k < i; k++) {
        double h = G.d[k] * G.inv[k];
        const double* Lk = G.gram + (size_t)k * GS_MAXM;
        for (int j = 0; j < k; j++) h -= Lk[j] * G.h[1 + j];
        G.h[1 + k] = h;
        G.coef[k] = h * G.inv[k];
    }
}

// out = w - sum_k coef_k u_k for k = k0 .. k0 + NV - 1, in that order; norm:
// its |.|^2 and inverse root as those of u_i
template <int NC, int NV>
static __global__ void __launch_bounds__(RED_THREADS, 4) k_gs_update(i64 n, CSVec<double> w, SVec<double> out,
                                                                     const double* __restrict__ V, i64 vstride, int k0,
                                                                     int i, int norm, double wp2, GSData G) {
    __shared__ double tot[1];
    double s[1] = {0.0};
    double co[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) co[v] = G.coef[k0 + v];
    const double* __restrict__ uk = V + (i64)k0 * vstride;
    for (i64 f = blockIdx.x * (i64)blockDim.x + threadIdx.x; f < n; f += (i64)gridDim.x * blockDim.x) {
        double x[NC];
#pragma unroll
        for (int c = 0; c < NC; c++) x[c] = w.c[c][f];
#pragma unroll
        for (int v = 0; v < NV; v++)
#pragma unroll
            for (int c = 0; c < NC; c++) x[c] = x[c] - uk[v * vstride + (i64)c * n + f] * co[v];
        double su = 0.0;
#pragma unroll
        for (int c = 0; c < NC; c++) {
            out.c[c][f] = x[c];
            su += (c == NC - 1) ? wp2 * (x[c] * x[c]) : x[c] * x[c];
        }
        s[0] += su;
    }
    if (!norm || !red_many<1>(s, G.partials, G.counter, tot) || threadIdx.x) return;
    G.n2[i] = tot[0];
    G.inv[i] = 1.0 / sqrt(tot[0]);
}

// x += sum_{it < m} y[it] v_it (update_sol, gmres.f90:495-529; same order)
static __global__ void __launch_bounds__(256) k_update_sol(i64 n, int ncomp, SVec<double> x, const double* __restrict__ V,
                                                    i64 vstride, const double* y, int m) {
    for (i64 f = blockIdx.x * (i64)blockDim.x + threadIdx.x; f < n; f += (i64)gridDim.x * blockDim.x) {
        // all components advance together (each in the order of update_sol),
        // so the loads of every component are in flight at once
        double acc[4];
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (c < ncomp) acc[c] = x.c[c][f];
        for (int it = 0; it < m; it++) {
            const double yi = y[it];
#pragma unroll
            for (int c = 0; c < 4; c++)
                if (c < ncomp) acc[c] = acc[c] + V[it * vstride + (i64)c * n + f] * yi;
        }
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (c < ncomp) x.c[c][f] = acc[c];
    }
}

// N fields converted in one launch (the velocity between GMRES and the FP32
// multigrid)
template <typename TO, typename TI, int N>
static __global__ void __launch_bounds__(256) k_convs(i64 n, SVec<TO> o, CSVec<TI> in) {
    for (i64 f = blockIdx.x * (i64)blockDim.x + threadIdx.x; f < n; f += (i64)gridDim.x * blockDim.x) {
        TI v[N];
#pragma unroll
        for (int c = 0; c < N; c++) v[c] = in.c[c][f];
#pragma unroll
        for (int c = 0; c < N; c++) o.c[c][f] = (TO)v[c];
    }
}

template <typename TO, typename TI>
static __global__ void __launch_bounds__(256) k_copy_conv(i64 n, TO* __restrict__ o, const TI* __restrict__ in, double s) {
    // four grid strides per pass: four loads in flight per thread
    const i64 st = (i64)gridDim.x * blockDim.x;
    i64 f = blockIdx.x * (i64)blockDim.x + threadIdx.x;
    for (; f + 3 * st < n; f += 4 * st) {
        TI a[4];
#pragma unroll
        for (int u = 0; u < 4; u++) a[u] = in[f + u * st];
#pragma unroll
        for (int u = 0; u < 4; u++) o[f + u * st] = (TO)((double)a[u] * s);
    }
    for (; f < n; f += st) o[f] = (TO)((double)in[f] * s);
}

template <typename T>
static __global__ void __launch_bounds__(256) k_fill(i64 n, T* a, T v) {
    for (i64 f = blockIdx.x * (i64)blockDim.x + threadIdx.x; f < n; f += (i64)gridDim.x * blockDim.x) a[f] = v;
}

template <typename T>
static __global__ void __launch_bounds__(256) k_recip(i64 n, T* o, const double* a) {
    for (i64 f = blockIdx.x * (i64)blockDim.x + threadIdx.x; f < n; f += (i64)gridDim.x * blockDim.x)
        o[f] = (T)(1.0 / a[f]);
}

// ---------------------------------------------------------------------
// saddle-point operator, one pass (apply_matrix.f90:117-147):
//   b_u = (alpha_scale*alpha - L) x_u + G x_p ;  b_p = -D x_u
// mode 1 returns rhs - A x instead (the GMRES residual, gmres.f90:205-213);
// inv (device scalar, not null in mode 0 only) multiplies A x.
// ---------------------------------------------------------------------
template <int DIM, int VISC>
static __global__ void __launch_bounds__(256) k_stokes_apply(Grid g, StagOp<double> A, CSVec<double> x, CSVec<double> rhs,
                                                      SVec<double> out, int mode, double dxinv, const double* inv) {
    CellF P;
    if (!cellf_of_thread(g, P)) return;
    const double* phi[3] = {x.c[0], x.c[1], DIM == 3 ? x.c[2] : nullptr};
    const double* p = x.c[DIM];
    const i64 f = P.id(0, 0, 0);
    const double pc = ld(p, f);
    double div = 0.0;
#pragma unroll
    for (int c = 0; c < DIM; c++) {
        const int dx_ = (c == 0), dy_ = (c == 1), dz_ = (c == 2);
        double dg;
        double L = stag_lface_c<double, DIM, VISC>(c, A, phi, P, dg);
        const double gp = (pc - ld(p, P.id(-dx_, -dy_, -dz_))) * dxinv;
        L = L + gp;
        out.c[c][f] = mode ? ld(rhs.c[c], f) - L : inv ? L * *inv : L;
        div += (ld(phi[c], P.id(dx_, dy_, dz_)) - ld(phi[c], f)) * dxinv;
    }
    const double bp = div * -1.0;
    out.c[DIM][f] = mode ? ld(rhs.c[DIM], f) - bp : inv ? bp * *inv : bp;
}

// the same with gmres_spatial_order = 4 (apply_matrix.f90:124-135): the
// visc_type 1 operator of stag_applyop_4o_2d/_3d (stag_applyop.f90:1262-1510,
// per direction +16 phi(+-1) - phi(+-2) over 12 dx^2, diagonal 30 dim over
// 12 dx^2) and the gradient of compute_grad_4o (div_and_grad.f90:804-880,
// (-p(+1) + 15 p - 15 p(-1) + p(-2)) / 12 dx); the divergence stays second
// order.  Terms summed in the order of those loops.  The constant viscosity
// is the first cell's (stag_applyop.f90:1306); t2 = 1/(12 dx^2),
// t1 = 1/(12 dx).
template <int DIM>
static __global__ void __launch_bounds__(256) k_stokes_apply4(Grid g, StagOp<double> A, CSVec<double> x,
                                                              CSVec<double> rhs, SVec<double> out, int mode,
                                                              double dxinv, double t1, double t2, const double* inv) {
    Cell P;
    if (!cell_of_thread(g, P)) return;
    const double b = ld(A.beta, 0);
    const double* p = x.c[DIM];
    const i64 f = P.id(0, 0, 0);
    const double cdiag = DIM == 2 ? 60.0 : 90.0;
    double div = 0.0;
#pragma unroll
    for (int c = 0; c < DIM; c++) {
        const double* u = x.c[c];
        double s = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; d++) {
            const int e0 = d == 0, e1 = d == 1, e2 = d == 2;
            const double t = 16.0 * ld(u, P.id(e0, e1, e2));
            s = d == 0 ? t : s + t;
            s = s + 16.0 * ld(u, P.id(-e0, -e1, -e2));
            s = s - 1.0 * ld(u, P.id(2 * e0, 2 * e1, 2 * e2));
            s = s - 1.0 * ld(u, P.id(-2 * e0, -2 * e1, -2 * e2));
        }
        const double a = A.alpha_scale * ld(A.alpha[c], f);
        double L = (a + cdiag * b * t2) * ld(u, f) - s * b * t2;
        const int e0 = c == 0, e1 = c == 1, e2 = c == 2;
        const double gp = (-ld(p, P.id(e0, e1, e2)) + 15.0 * ld(p, f) - 15.0 * ld(p, P.id(-e0, -e1, -e2)) +
                           ld(p, P.id(-2 * e0, -2 * e1, -2 * e2))) *
                          t1;
        L = L + gp;
        out.c[c][f] = mode ? ld(rhs.c[c], f) - L : inv ? L * *inv : L;
        div += (ld(u, P.id(e0, e1, e2)) - ld(u, f)) * dxinv;
    }
    const double bp = div * -1.0;
    out.c[DIM][f] = mode ? ld(rhs.c[DIM], f) - bp : inv ? bp * *inv : bp;
}

// mac_rhs = D x_u + b_p  (apply_precon.f90:118-123)
template <typename T, int DIM>
static __global__ void __launch_bounds__(256) k_div_plus(Grid g, const T* u0, const T* u1, const T* u2, const double* bp,
                                                  T* out, T dxinv) {
    Cell P;
    if (!cell_of_thread(g, P)) return;
    const i64 f = P.id(0, 0, 0);
    T s = (ld(u0, P.id(1, 0, 0)) - ld(u0, f)) * dxinv + (ld(u1, P.id(0, 1, 0)) - ld(u1, f)) * dxinv;
    if constexpr (DIM == 3) s += (ld(u2, P.id(0, 0, 1)) - ld(u2, f)) * dxinv;
    out[f] = bp ? s + (T)bp[f] : s;
}

// mu^-1 = 1 / diagonal of the viscous operator on the faces
// (inverse_diag_lap.f90:17-330), evaluated in FP64 in the summation order of
// its 2D and 3D loops; visc_type 1 / 2 take the first cell's beta
template <typename T, int DIM>
static __global__ void __launch_bounds__(256) k_inv_diag_lap(Grid g, int visc, const double* beta, const double* be0,
                                                      const double* be1, const double* be2, T* o0, T* o1, T* o2) {
    Cell P;
    if (!cell_of_thread(g, P)) return;
    const i64 f = P.id(0, 0, 0);
    T* out[3] = {o0, o1, o2};
    if (visc == 1 || visc == 2) {
        const double m = (DIM == 2 ? (visc == 1 ? 4.0 : 6.0) : (visc == 1 ? 6.0 : 8.0)) * beta[0];
#pragma unroll
        for (int c = 0; c < DIM; c++) out[c][f] = (T)(1.0 / m);
        return;
    }
    const double cb = visc == -2 ? 2.0 : 1.0;
    const double* be[3] = {be0, be1, be2};
#pragma unroll
    for (int c = 0; c < DIM; c++) {
        double s = cb * beta[f] + cb * beta[P.id(-(c == 0), -(c == 1), -(c == 2))];
        if constexpr (DIM == 2) {
            // x face: node (i, j+1) then (i, j); y face: (i+1, j) then (i, j)
            s = s + be0[c == 0 ? P.id(0, 1, 0) : P.id(1, 0, 0)];
            s = s + be0[f];
        } else {
#pragma unroll
            for (int d = 0; d < 3; d++) {
                if (d == c) continue;
                const int e = (c + d == 1) ? 0 : (c + d == 2) ? 1 : 2;  // xy, xz, yz
                s = s + be[e][f];
                s = s + be[e][P.id(d == 0, d == 1, d == 2)];
            }
        }
        out[c][f] = (T)(1.0 / s);
    }
}

// out_d = (G Phi)_d * w_d on the faces (compute_grad, div_and_grad.f90:
// 417-703, then the face product of visc_schur_complement)
template <typename T, int DIM>
static __global__ void __launch_bounds__(256) k_grad_mul(Grid g, const T* Phi, const T* w0, const T* w1, const T* w2,
                                                  T* o0, T* o1, T* o2, T dxinv) {
    Cell P;
    if (!cell_of_thread(g, P)) return;
    const i64 f = P.id(0, 0, 0);
    const T* w[3] = {w0, w1, w2};
    T* out[3] = {o0, o1, o2};
#pragma unroll
    for (int d = 0; d < DIM; d++) {
        const T gp = (Phi[f] - Phi[P.id(-(d == 0), -(d == 1), -(d == 2))]) * dxinv;
        out[d][f] = gp * w[d][f];
    }
}

// a_c *= w_c on the faces
template <typename T>
static __global__ void __launch_bounds__(256) k_mul_faces(i64 n, int ncomp, T* a0, T* a1, T* a2, const T* w0,
                                                   const T* w1, const T* w2) {
    T* a[3] = {a0, a1, a2};
    const T* w[3] = {w0, w1, w2};
    for (i64 f = blockIdx.x * (i64)blockDim.x + threadIdx.x; f < n; f += (i64)gridDim.x * blockDim.x)
        for (int c = 0; c < ncomp; c++) a[c][f] = a[c][f] * w[c][f];
}

// x_p = Phi_mu (+ theta Phi when add), negated on request
// (visc_schur_complement's output, apply_precon.f90:664-683)
template <typename T>
static __global__ void __launch_bounds__(256) k_bfbt_out(i64 n, double* xp, const T* phimu, const T* phi,
                                                  double theta, int add, int negate) {
    for (i64 f = blockIdx.x * (i64)blockDim.x + threadIdx.x; f < n; f += (i64)gridDim.x * blockDim.x) {
        double v = (double)phimu[f];
        if (add) v = v + (double)phi[f] * theta;
        xp[f] = negate ? v * -1.0 : v;
    }
}

// x_u = phi - w * G Phi (subtract_weighted_gradp, macproject.f90:318-362),
// written to FP64 output (w = alphainv or 1 when null)
template <typename T, int DIM>
static __global__ void __launch_bounds__(256) k_sub_wgrad(Grid g, const T* phi0, const T* phi1, const T* phi2,
                                                   const T* w0, const T* w1, const T* w2, const T* Phi, double* o0,
                                                   double* o1, double* o2, T dxinv) {
    Cell P;
    if (!cell_of_thread(g, P)) return;
    const i64 f = P.id(0, 0, 0);
    const T pc = ld(Phi, f);
    const T* ph[3] = {phi0, phi1, phi2};
    const T* w[3] = {w0, w1, w2};
    double* o[3] = {o0, o1, o2};
#pragma unroll
    for (int c = 0; c < DIM; c++) {
        const int dx_ = (c == 0), dy_ = (c == 1), dz_ = (c == 2);
        T gp = (pc - ld(Phi, P.id(-dx_, -dy_, -dz_))) * dxinv;
        if (w[c]) gp = gp * ld(w[c], f);
        o[c][f] = (double)(ld(ph[c], f) + T(-1) * gp);
    }
}

// T-precision variant writing into T arrays (b_u - G x_p for precon 3/5)
template <typename T, int DIM>
static __global__ void __launch_bounds__(256) k_sub_grad_T(Grid g, const double* b0, const double* b1, const double* b2,
                                                    const double* xp, T* o0, T* o1, T* o2, double dxinv) {
    Cell P;
    if (!cell_of_thread(g, P)) return;
    const i64 f = P.id(0, 0, 0);
    const double pc = xp[f];
    const double* b[3] = {b0, b1, b2};
    T* o[3] = {o0, o1, o2};
#pragma unroll
    for (int c = 0; c < DIM; c++) {
        const int dx_ = (c == 0), dy_ = (c == 1), dz_ = (c == 2);
        const double gp = (pc - xp[P.id(-dx_, -dy_, -dz_)]) * dxinv;
        o[c][f] = (T)(b[c][f] + (-1.0) * gp);
    }
}

// Schur-complement pressure update (apply_precon.f90:140-195 and
// simple_schur_complement 479-534) into FP64 x_p.
//   kind 0: x_p = c*beta*(-mac_rhs) [+ gamma part] + theta*Phi
//   kind 1: precon_type = -1: -L_alpha Phi in place of -mac_rhs
// negate: multiply by -1 at the end (precon_type -2/-5)
template <typename T, int DIM>
static __global__ void __launch_bounds__(256) k_schur(Grid g, CCOp<T> A, const T* mac_rhs, const T* Phi, const double* beta,
                                               const double* gamma, double theta, int av, int kind, int add_phi,
                                               int negate, double* xp) {
    Cell P;
    if (!cell_of_thread(g, P)) return;
    const i64 f = P.id(0, 0, 0);
    double v;
    if (kind == 1) {
        T dg;
        v = -(double)cc_lap<T, DIM>(A, Phi, P, dg);
    } else {
        v = (double)mac_rhs[f] * -1.0;
    }
    if (av == 1 || av == 2) {
        v = v * beta[f];
        if (av == 2) v = v * 2.0;
    } else {
        const double m = v * gamma[f];
        v = v * beta[f];
        v = v * (4.0 / 3.0);
        v = v + m;
    }
    if (add_phi) v = v + (double)Phi[f] * theta;
    if (negate) v = v * -1.0;
    xp[f] = v;
}

// block-diagonal pressure update (apply_precon.f90:378-416)
static __global__ void __launch_bounds__(256) k_schur_blockdiag(i64 n, const double* bp, const double* beta,
                                                         const double* gamma, const double* Phi, double theta,
                                                         int use_phi, int av, int pt, double* xp) {
    for (i64 f = blockIdx.x * (i64)blockDim.x + threadIdx.x; f < n; f += (i64)gridDim.x * blockDim.x) {
        double ph = use_phi ? Phi[f] * theta : 0.0;
        double v = bp[f] * beta[f];
        v = v - ph;
        if (av == 1 && pt == 4) v = v * -1.0;
        else if (av == 2 && pt == 4) v = v * -2.0;
        else if (av == 2 && pt == -4) v = v * 2.0;
        else if (av == 3 && pt == 4) { v = v * (-4.0 / 3.0); v = v + (bp[f] * gamma[f]) * -1.0; }
        else if (av == 3 && pt == -4) { v = v * (4.0 / 3.0); v = v + bp[f] * gamma[f]; }
        xp[f] = v;
    }
}

}  // namespace fhd
