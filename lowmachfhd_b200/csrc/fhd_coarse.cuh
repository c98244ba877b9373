// fhd_coarse.cuh -- the coarse end of both multigrid V-cycles in ONE
// thread block.
//
// Below a few thousand cells a multigrid level is pure latency: every
// smoother colour, residual, restriction and prolongation of the
// stag_mg_solver V-cycle (stag_mg_solver.f90:301-599) and of the pressure
// V-cycle behind macproject (macproject.f90:294-298) is a dependent launch
// that moves a few kilobytes.  These kernels run every level from the first
// one whose arrays fit in shared memory (up to the cell limits of the host's
// coarse_first) down to the bottom inside one CTA of 512 threads: the unknowns,
// right-hand sides and residuals of all those levels live in shared memory, and
// a __syncthreads() replaces each launch boundary.
//
// Arithmetic is the same as the per-level kernels: the operator, smoother
// update, restriction and prolongation are the shared expressions of
// fhd_kernels.cuh (stag_lface_acc, cc_lap_acc, stag_restrict_expr,
// stag_prolong_expr) on the same operands in the same order, so in FP64 the
// result equals the multi-launch V-cycle bit for bit.
//
// What bounds it is one SM's issue rate on the largest level and the chain of
// sweeps (one per colour) below it:
//   * a level whose extents are all even keeps its two colours apart (red
//     values first, then black, one of each per x-pair of cells), the
//     components of a cell side by side: every shared-memory access of a
//     sweep is free of conflicts, and a thread works out the indices of its
//     pairs once per level and shares them among the components;
//   * components that do not couple (visc_type 1) are swept together: two
//     steps per smooth instead of four (2D) or six (3D);
//   * only as many warps as a level has pairs take part in its sweeps, down
//     to one warp and no block barrier;
//   * coefficients come from shared memory: the staggered diagonal of
//     visc_type 1 lies in the scratch array between two residuals, the pressure
//     coefficients beside the unknowns on every level that has room (a large
//     bottom may have none); the other viscosity types read theirs through the
//     L1 by non-coherent loads;
//   * transfers run one thread per coarse cell, whose coarse values and
//     indices serve all its children;
//   * an odd level (the colours meet across the wrap) is swept from one
//     buffer into the other, one step per colour.
// The other viscosity types and the Jacobi smoother keep components apart
// and cells in index order; an odd level takes them two passes per colour.
//
// One call before (1024 threads, a step per component and colour) and now:
// staggered FP32 16^3 down 133 -> 52 us, 10^3 down 81 -> 21, FP64 32^2 down
// 81 -> 40; pressure FP32 20^3 down 61 -> 49, FP64 64^2 down 59 -> 50 (14 issue
// slots per update and dimension now, no longer memory latency).
#pragma once
#include <type_traits>

#include "fhd_walls.cuh"

namespace fhd {

constexpr int CS_MAXL = 12;      // levels handled by one coarse kernel
// 512 threads: room for the registers of three components at a time (1024
// spilled), and fewer warps to feed through the small levels (pressure,
// 20^3 down: 49 us against 52 with 1024)
constexpr int CS_THREADS = 512;

__device__ __forceinline__ bool cs_all_even(const Grid& g) {
    return !(g.n[0] & 1) && !(g.n[1] & 1) && (g.dim == 2 || !(g.n[2] & 1));
}

// q / n and q % n for 0 <= q < 2^20, 0 < n < 2^20 (exact: (q + 0.5) / n is at
// least 0.5 / n away from an integer, the approximate quotient within
// 2^-22 q / n)
__device__ __forceinline__ void cs_divmod(int q, int n, int& d, int& r) {
    d = (int)__fdividef((float)q + 0.5f, (float)n);
    r = q - d * n;
}

// linear cell index -> (i, j, k)
__device__ __forceinline__ void cs_ijk(const Grid& g, int f, int& i, int& j, int& k) {
    int r;
    cs_divmod(f, g.n[0], r, i);
    cs_divmod(r, g.n[1], k, j);
}

// h-th cell of parity par on a level with even n[0]: the half-row index
// of the colour kernels (k_stag_gs, k_cc_gsrb)
__device__ __forceinline__ void cs_ijk_half(const Grid& g, int h, int par, int& i, int& j, int& k) {
    int r, ih;
    cs_divmod(h, g.n[0] >> 1, r, ih);
    cs_divmod(r, g.n[1], k, j);
    i = 2 * ih + ((j + k + par) & 1);
}

// Where a level keeps its cells: cell (i, j, k) is element x(i) + row(j, k),
// plus co if split and black.  Split: the red cells first and then the
// black ones, by x-pair; else index order.
struct CSIdx {
    int nx, ny, nz, rs, co;
    bool split;
    __device__ __forceinline__ void set(const Grid& g, bool sp) {
        nx = g.n[0]; ny = g.n[1]; nz = g.n[2];
        split = sp;
        rs = sp ? nx >> 1 : nx;
        co = sp ? (int)g.nc >> 1 : 0;
    }
    __device__ __forceinline__ int x(int i) const {
        i = wrapc(i, nx);
        return split ? i >> 1 : i;
    }
    __device__ __forceinline__ int row(int j, int k) const { return rs * (wrapc(j, ny) + ny * wrapc(k, nz)); }
    __device__ __forceinline__ int at(int i, int j, int k) const {
        return x(i) + row(j, k) + (((i + j + k) & 1) ? co : 0);
    }
};

// element of every cell at offsets -1, 0, 1 from one cell (even: the cell's
// parity, red 0)
template <int DIM>
struct CSNear {
    int xi[3], ro[3][3], co[2];
    __device__ __forceinline__ void set(const CSIdx& X, int i, int j, int k) {
#pragma unroll
        for (int d = 0; d < 3; d++) xi[d] = X.x(i + d - 1);
#pragma unroll
        for (int e = 0; e < 3; e++)
#pragma unroll
            for (int d = 0; d < 3; d++) ro[e][d] = (DIM == 3 || e == 1) ? X.row(j + d - 1, DIM == 3 ? k + e - 1 : 0) : 0;
        const int par = (i + j + k) & 1;
        co[0] = par ? X.co : 0;
        co[1] = par ? 0 : X.co;
    }
    __device__ __forceinline__ int at(int dx, int dy, int dz) const {
        return xi[dx + 1] + ro[dz + 1][dy + 1] + co[(dx + dy + dz) & 1];
    }
    // offset o along component c, pa and pb across
    __device__ __forceinline__ int comp(int c, int o, int pa, int pb) const {
        int off[3] = {0, 0, 0};
        off[c] += o;
        off[c == 0 ? 1 : 0] += pa;
        if (DIM == 3) off[c == 2 ? 1 : 2] += pb;
        return at(off[0], off[1], off[2]);
    }
};

// The x-pairs of a split level, dealt to its first nt threads: thread t takes
// pair t % np of every RP-th row.  Worked out once per level.  With walls
// (WALL, set_walls) a neighbour behind a wall is -1.
template <bool WALL = false>
struct CSPairs {
    int np, ny, nz, nh, nt;
    bool wx = false, wy = false, wz = false;
    int h0, j0, k0, dj, dk, RP;
    bool on;
    __device__ __forceinline__ void set(const Grid& g) {
        np = g.n[0] >> 1; ny = g.n[1]; nz = g.n[2];
        nh = (int)g.nc >> 1;
        nt = nh >= (int)blockDim.x ? (int)blockDim.x : (nh + 31) & ~31;
        RP = nt / np;
        int r;
        cs_divmod(threadIdx.x, np, r, h0);
        on = r < RP;
        cs_divmod(r, ny, k0, j0);
        cs_divmod(RP, ny, dk, dj);
    }
    __device__ __forceinline__ void set_walls(const Walls& W) {
        wx = W.lo[0] != 0;
        wy = W.lo[1] != 0;
        wz = W.lo[2] != 0;
    }
    // f(pair, its row's parity and first pair, those of the rows below and
    // above in y and z)
    template <class F>
    __device__ __forceinline__ void row(int h, int j, int k, F&& f) const {
        const int nl = np * ny, b = np * j + nl * k;
        const bool y_ = WALL && wy, z_ = WALL && wz;
        f(h, j + k, b, j == 0 ? (y_ ? -1 : b + nl - np) : b - np, j == ny - 1 ? (y_ ? -1 : b - nl + np) : b + np,
          k == 0 ? (z_ ? -1 : b + nl * (nz - 1)) : b - nl, k == nz - 1 ? (z_ ? -1 : b - nl * (nz - 1)) : b + nl);
    }
    template <class F>
    __device__ __forceinline__ void each(F&& f) const {
        if (RP > 0) {
            if (!on) return;
            int j = j0, k = k0;
            while (k < nz) {
                row(h0, j, k, f);
                j += dj;
                k += dk;
                if (j >= ny) {
                    j -= ny;
                    k++;
                }
            }
        } else {  // rows longer than the block
            for (int r = 0; r < ny * nz; r++)
                for (int h = threadIdx.x; h < np; h += nt) row(h, r % ny, r / ny, f);
        }
    }
    // the x neighbour in the next pair of the row's cell of colour col: to
    // the left of an even cell, to the right of an odd one
    __device__ __forceinline__ int across(int h, int s, int col) const {
        const bool x_ = WALL && wx;
        if ((s ^ col) & 1) return h + 1 == np ? (x_ ? -1 : 0) : h + 1;
        return h == 0 ? (x_ ? -1 : np - 1) : h - 1;
    }
};

// barrier of the first nt threads of the block (nt a multiple of 32)
__device__ __forceinline__ void cs_bar(int nt) {
    if (nt == 32) __syncwarp();
    else asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory");
}

// ---------------------------------------------------------------------
// staggered multigrid
// ---------------------------------------------------------------------
template <typename T>
struct StagCoarseArgs {
    int nlev;      // levels of this kernel; level 0 = the first coarse level
    int load_phi;  // level-0 unknowns from phi (else zero, the V-cycle's start)
    int n_down, n_up, n_bottom;
    int jacobi;    // stag_mg_smoother == 0
    T omega;
    T* phi[3];          // level-0 unknowns in global memory (in/out)
    const T* rhs[3];    // level-0 right-hand side
    Walls walls;        // (WALL instantiations)
    Grid g[CS_MAXL];
    StagOp<T> A[CS_MAXL];
    int off[CS_MAXL];   // shared-memory element offset of each level
};

// shared-memory arrays of one level: phi, rhs and scratch, dim components
// each of nc elements, in that order from off
template <typename T>
struct CSStag {
    T* ph[3];
    T* rh[3];
    T* tm[3];
    __device__ __forceinline__ void set(T* S, int off, int dim, int nc) {
        for (int c = 0; c < 3; c++) {
            const int cc = c < dim ? c : 0;
            ph[c] = S + off + cc * nc;
            rh[c] = S + off + (dim + cc) * nc;
            tm[c] = S + off + (2 * dim + cc) * nc;
        }
    }
};

// (alpha - L) phi of component C at cell P on shared-memory unknowns, and
// the diagonal
template <typename T, int DIM, int VISC, int C>
__device__ __forceinline__ T cs_lface(const StagOp<T>& A, const CSStag<T>& V, const CellF& P, T& dg) {
    const T* pc = V.ph[C];
    const i64 f = P.base;
    return stag_lface_acc<T, DIM, VISC, C>(
        A, P, [&](int a, int b, int c) { return pc[P.id(a, b, c)]; },
        [&](int d, int a, int b, int c) { return V.ph[d][P.id(a, b, c)]; },
        [&]() { return ld(A.alpha[C], f); }, dg);
}

// new value of the face of component C at (i, j, k): the update of
// k_stag_gs / k_stag_color_update
template <typename T, int DIM, int VISC, int C>
__device__ __forceinline__ T cs_stag_new(const Grid& g, const StagOp<T>& A, const CSStag<T>& V, int i, int j, int k,
                                         T omega, i64& f) {
    CellF P;
    P.set(g, i, j, k);
    f = P.base;
    T dg;
    const T L = cs_lface<T, DIM, VISC, C>(A, V, P, dg);
    return V.ph[C][f] + sm_quot(omega * (V.rh[C][f] - L), dg);
}

// one colour of component C (1-based colour of stag_mg_smoother 1)
template <typename T, int DIM, int VISC, int C>
__device__ void cs_stag_colour(const Grid& g, const StagOp<T>& A, const CSStag<T>& V, int par, T omega) {
    const int nc = (int)g.nc;
    if (cs_all_even(g)) {
        for (int h = threadIdx.x; h < (nc >> 1); h += blockDim.x) {
            int i, j, k;
            cs_ijk_half(g, h, par, i, j, k);
            i64 f;
            const T v = cs_stag_new<T, DIM, VISC, C>(g, A, V, i, j, k, omega, f);
            V.ph[C][f] = v;
        }
        __syncthreads();
    } else {
        for (int f0 = threadIdx.x; f0 < nc; f0 += blockDim.x) {
            int i, j, k;
            cs_ijk(g, f0, i, j, k);
            if (((i + j + k) & 1) != par) continue;
            i64 f;
            const T v = cs_stag_new<T, DIM, VISC, C>(g, A, V, i, j, k, omega, f);
            V.tm[C][f] = v;
        }
        __syncthreads();
        for (int f0 = threadIdx.x; f0 < nc; f0 += blockDim.x) {
            int i, j, k;
            cs_ijk(g, f0, i, j, k);
            if (((i + j + k) & 1) == par) V.ph[C][f0] = V.tm[C][f0];
        }
        __syncthreads();
    }
}

// count smooths of one level (stag_mg_smooth: colours 1..2*dim, or the
// Jacobi sweep)
template <typename T, int DIM, int VISC>
__device__ void cs_stag_smooths(const Grid& g, const StagOp<T>& A, const CSStag<T>& V, int count, int jacobi,
                                T omega) {
    const int nc = (int)g.nc;
    for (int s = 0; s < count; s++) {
        if (jacobi) {
            for (int f0 = threadIdx.x; f0 < nc; f0 += blockDim.x) {
                int i, j, k;
                cs_ijk(g, f0, i, j, k);
                i64 f;
                V.tm[0][f0] = cs_stag_new<T, DIM, VISC, 0>(g, A, V, i, j, k, omega, f);
                V.tm[1][f0] = cs_stag_new<T, DIM, VISC, 1>(g, A, V, i, j, k, omega, f);
                if constexpr (DIM == 3) V.tm[2][f0] = cs_stag_new<T, DIM, VISC, (DIM == 3 ? 2 : 1)>(g, A, V, i, j, k, omega, f);
            }
            __syncthreads();
            for (int f0 = threadIdx.x; f0 < nc; f0 += blockDim.x)
                for (int c = 0; c < DIM; c++) V.ph[c][f0] = V.tm[c][f0];
            __syncthreads();
            continue;
        }
        if constexpr (VISC == -1) {
            if (cs_all_even(g)) {  // the components do not couple
                for (int par = 0; par < 2; par++) {
                    for (int h = threadIdx.x; h < (nc >> 1); h += blockDim.x) {
                        int i, j, k;
                        cs_ijk_half(g, h, par, i, j, k);
                        i64 f;
                        T nv[3];
                        nv[0] = cs_stag_new<T, DIM, VISC, 0>(g, A, V, i, j, k, omega, f);
                        nv[1] = cs_stag_new<T, DIM, VISC, 1>(g, A, V, i, j, k, omega, f);
                        if constexpr (DIM == 3) nv[2] = cs_stag_new<T, DIM, VISC, (DIM == 3 ? 2 : 1)>(g, A, V, i, j, k, omega, f);
#pragma unroll
                        for (int c = 0; c < DIM; c++) V.ph[c][f] = nv[c];
                    }
                    __syncthreads();
                }
                continue;
            }
        }
        // colour 2c + 1 is component c at parity 0, colour 2c + 2 the same
        // component at parity 1
        cs_stag_colour<T, DIM, VISC, 0>(g, A, V, 0, omega);
        cs_stag_colour<T, DIM, VISC, 0>(g, A, V, 1, omega);
        cs_stag_colour<T, DIM, VISC, 1>(g, A, V, 0, omega);
        cs_stag_colour<T, DIM, VISC, 1>(g, A, V, 1, omega);
        if constexpr (DIM == 3) {
            cs_stag_colour<T, DIM, VISC, (DIM == 3 ? 2 : 1)>(g, A, V, 0, omega);
            cs_stag_colour<T, DIM, VISC, (DIM == 3 ? 2 : 1)>(g, A, V, 1, omega);
        }
    }
}

// residual rhs - L phi of every component into the scratch arrays
template <typename T, int DIM, int VISC>
__device__ void cs_stag_residual(const Grid& g, const StagOp<T>& A, const CSStag<T>& V) {
    const int nc = (int)g.nc;
    for (int f0 = threadIdx.x; f0 < nc; f0 += blockDim.x) {
        int i, j, k;
        cs_ijk(g, f0, i, j, k);
        CellF P;
        P.set(g, i, j, k);
        T dg;
        V.tm[0][f0] = V.rh[0][f0] - cs_lface<T, DIM, VISC, 0>(A, V, P, dg);
        V.tm[1][f0] = V.rh[1][f0] - cs_lface<T, DIM, VISC, 1>(A, V, P, dg);
        if constexpr (DIM == 3) V.tm[2][f0] = V.rh[2][f0] - cs_lface<T, DIM, VISC, (DIM == 3 ? 2 : 1)>(A, V, P, dg);
    }
    __syncthreads();
}

// visc_type 1 on neighbour pair sums: the expressions of stag_lface_acc
template <typename T, int DIM>
struct CSVisc1 {
    T b, q, bq, bd, as, omega;
    __device__ __forceinline__ void set(const StagOp<T>& A, T om) {
        b = A.beta0_set ? A.beta0 : A.beta[0];
        q = A.q;
        bq = b * q;
        bd = T(2 * DIM) * b * q;
        as = A.alpha_scale;
        omega = om;
    }
    // rhs - L phi of component c
    __device__ __forceinline__ T resid(int c, T v, T xs, T ys, T zs, T rh, T dg) const {
        const T own = c == 0 ? xs : (c == 1 ? ys : zs);
        T oth = c == 0 ? ys : xs;
        if (sizeof(T) == 8) oth = T(0) + oth;
        if (DIM == 3) oth = oth + (c == 2 ? ys : zs);
        const T L = sizeof(T) == 4 ? v * dg - (own + oth) * bq : v * dg - (own + oth) * b * q;
        return rh - L;
    }
    __device__ __forceinline__ T update(int c, T v, T xs, T ys, T zs, T rh, T dg) const {
        return v + sm_quot(omega * resid(c, v, xs, ys, zs, rh, dg), dg);
    }
};

// one level of the visc_type 1 staggered multigrid: unknowns, right-hand
// sides and scratch, the DIM components of a cell side by side
template <typename T>
struct CSLev {
    T *ph, *rh, *tm;
    __device__ __forceinline__ void set(T* S, int off, int n) {
        ph = S + off;
        rh = ph + n;
        tm = rh + n;
    }
};

// the diagonals of a split level into its scratch
template <typename T, int DIM, class Pairs>
__device__ __forceinline__ void cs_split_diag(const Pairs& Q, const CSVisc1<T, DIM>& U, const StagOp<T>& A,
                                              const CSLev<T>& V) {
    Q.each([&](int h, int s, int b, int, int, int, int) {
        const int p = b + h, r = s & 1;
#pragma unroll
        for (int c = 0; c < DIM; c++) {
            V.tm[p * DIM + c] = U.as * ld(A.alpha[c], 2 * p + r) + U.bd;
            V.tm[(Q.nh + p) * DIM + c] = U.as * ld(A.alpha[c], 2 * p + 1 - r) + U.bd;
        }
    });
}

// value of component c behind a wall of direction d and sign sg: zero normal
// to it, the face's own value v or its negative along it (wall_vel)
template <typename T>
__device__ __forceinline__ T cs_behind(int c, int d, int sg, T v) {
    return c == d ? T(0) : (sg < 0 ? -v : v);
}

// f(element, neighbour pair sums by component, components on a wall face) of
// the cells of colour col
template <typename T, int DIM, bool WALL, class F>
__device__ __forceinline__ void cs_split_cells(const CSPairs<WALL>& Q, const Walls& W, const T* ph, int col, F&& f) {
    const int own = (col ? Q.nh : 0) * DIM;
    const T* O = ph + (col ? 0 : Q.nh) * DIM;
    Q.each([&](int h, int s, int b, int ym, int yp, int zm, int zp) {
        const int hx = Q.across(h, s, col), e = own + (b + h) * DIM;
        T xs[DIM], ys[DIM], zs[DIM];
        if constexpr (WALL) {
            const bool odd = (s ^ col) & 1;
            const int ax = hx < 0 ? -1 : b + hx, ap = yp < 0 ? -1 : yp + h, am = ym < 0 ? -1 : ym + h,
                      aq = zp < 0 ? -1 : zp + h, an = zm < 0 ? -1 : zm + h;
            const int on = (Q.wx && !odd && h == 0 ? 1 : 0) | (ym < 0 ? 2 : 0) | (zm < 0 ? 4 : 0);
#pragma unroll
            for (int c = 0; c < DIM; c++) {
                const T v = ph[e + c];
                auto at = [&](int a, int d, int sg) { return a < 0 ? cs_behind(c, d, sg, v) : O[a * DIM + c]; };
                xs[c] = O[(b + h) * DIM + c] + at(ax, 0, odd ? W.hi[0] : W.lo[0]);
                ys[c] = at(ap, 1, W.hi[1]) + at(am, 1, W.lo[1]);
                zs[c] = DIM == 3 ? at(aq, 2, W.hi[2]) + at(an, 2, W.lo[2]) : T(0);
            }
            f(e, xs, ys, zs, on);
        } else {
            const T *o = O + (b + h) * DIM, *ox = O + (b + hx) * DIM, *op = O + (yp + h) * DIM,
                    *om = O + (ym + h) * DIM, *oq = O + (zp + h) * DIM, *on = O + (zm + h) * DIM;
#pragma unroll
            for (int c = 0; c < DIM; c++) {
                xs[c] = o[c] + ox[c];
                ys[c] = op[c] + om[c];
                zs[c] = DIM == 3 ? oq[c] + on[c] : T(0);
            }
            f(e, xs, ys, zs, 0);
        }
    });
}

// count smooths of a split level, its diagonals in the scratch
template <typename T, int DIM, bool WALL>
__device__ __forceinline__ void cs_split_smooths(const CSPairs<WALL>& Q, const Walls& W, const CSVisc1<T, DIM>& U,
                                                 const CSLev<T>& V, int count) {
    for (int m = 0; m < 2 * count; m++) {
        cs_split_cells<T, DIM, WALL>(Q, W, V.ph, m & 1, [&](int e, const T* xs, const T* ys, const T* zs, int on) {
            T nv[DIM];
#pragma unroll
            for (int c = 0; c < DIM; c++)
                nv[c] = U.update(c, V.ph[e + c], xs[c], ys[c], zs[c], V.rh[e + c], V.tm[e + c]);
#pragma unroll
            for (int c = 0; c < DIM; c++)
                if (!(on >> c & 1)) V.ph[e + c] = nv[c];
        });
        cs_bar(Q.nt);
    }
}

// residual of a split level over its diagonals, zero on wall faces
template <typename T, int DIM, bool WALL>
__device__ __forceinline__ void cs_split_residual(const CSPairs<WALL>& Q, const Walls& W, const CSVisc1<T, DIM>& U,
                                                  const CSLev<T>& V) {
    for (int col = 0; col < 2; col++)
        cs_split_cells<T, DIM, WALL>(Q, W, V.ph, col, [&](int e, const T* xs, const T* ys, const T* zs, int on) {
            T nv[DIM];
#pragma unroll
            for (int c = 0; c < DIM; c++)
                nv[c] = U.resid(c, V.ph[e + c], xs[c], ys[c], zs[c], V.rh[e + c], V.tm[e + c]);
#pragma unroll
            for (int c = 0; c < DIM; c++) V.tm[e + c] = (on >> c & 1) ? T(0) : nv[c];
        });
}

// smooths of an odd level: each colour of every component from one buffer
// into the other (an even number of times)
template <typename T, int DIM, bool WALL>
__device__ __forceinline__ void cs_odd_smooths(const Grid& g, const Walls& W, const CSVisc1<T, DIM>& U,
                                               const StagOp<T>& A, const CSLev<T>& V, int count, int nt) {
    const int nc = (int)g.nc;
    T *x = V.ph, *y = V.tm;
    for (int s = 0; s < 2 * count; s++) {
        for (int f0 = threadIdx.x; f0 < nc; f0 += nt) {
            int q[3];
            cs_ijk(g, f0, q[0], q[1], q[2]);
            T nv[DIM];
#pragma unroll
            for (int c = 0; c < DIM; c++) nv[c] = x[f0 * DIM + c];
            if (((q[0] + q[1] + q[2]) & 1) == (s & 1)) {
                CellF P;
                P.set(g, q[0], q[1], q[2]);
                const int xm = (int)P.id(-1, 0, 0), xp = (int)P.id(1, 0, 0), ym = (int)P.id(0, -1, 0),
                          yp = (int)P.id(0, 1, 0), zm = (int)P.id(0, 0, -1), zp = (int)P.id(0, 0, 1);
#pragma unroll
                for (int c = 0; c < DIM; c++) {
                    const T v = nv[c];
                    T xs, ys, zs = T(0);
                    if constexpr (WALL) {
                        if (W.lo[c] != 0 && q[c] == 0) continue;  // on the wall
                        auto pair = [&](int d, int lo, int hi) {
                            const bool w = W.lo[d] != 0;
                            return (w && q[d] == g.n[d] - 1 ? cs_behind(c, d, W.hi[d], v) : x[hi * DIM + c]) +
                                   (w && q[d] == 0 ? cs_behind(c, d, W.lo[d], v) : x[lo * DIM + c]);
                        };
                        xs = pair(0, xm, xp);
                        ys = pair(1, ym, yp);
                        if (DIM == 3) zs = pair(2, zm, zp);
                    } else {
                        xs = x[xp * DIM + c] + x[xm * DIM + c];
                        ys = x[yp * DIM + c] + x[ym * DIM + c];
                        if (DIM == 3) zs = x[zp * DIM + c] + x[zm * DIM + c];
                    }
                    nv[c] = U.update(c, v, xs, ys, zs, V.rh[f0 * DIM + c], U.as * ld(A.alpha[c], f0) + U.bd);
                }
            }
#pragma unroll
            for (int c = 0; c < DIM; c++) y[f0 * DIM + c] = nv[c];
        }
        cs_bar(nt);
        T* t = x;
        x = y;
        y = t;
    }
}

// the operator of level m with a constant viscosity (visc_type > 0) loaded
// into a register once, rather than after every block barrier
template <typename T, int VISC>
__device__ __forceinline__ StagOp<T> cs_op(const StagCoarseArgs<T>& a, int m) {
    StagOp<T> A = a.A[m];
    if constexpr (VISC > 0) {
        if (!A.beta0_set) {
            A.beta0 = A.beta[0];
            A.beta0_set = 1;
        }
    }
    return A;
}

// the coarse end of one staggered V-cycle in the calling CTA (shared memory
// from the dynamic allocation); also run per box by the batched solver
// (WALL: visc_type 1 with domain walls)
template <typename T, int DIM, int VISC, bool WALL = false>
__device__ __forceinline__ void stag_coarse_run(const StagCoarseArgs<T>& a) {
    static_assert(!WALL || VISC == 1, "walls: visc_type 1");
    const Walls& W = a.walls;
    extern __shared__ __align__(16) unsigned char cs_smem[];
    T* S = reinterpret_cast<T*>(cs_smem);
    const int nt = blockDim.x;
    // visc_type 1 keeps the components of a cell side by side and splits
    // the colours of even levels
    const bool aos = VISC == 1 && !a.jacobi;
    auto index = [&](int m) {
        CSIdx X;
        X.set(a.g[m], aos && cs_all_even(a.g[m]));
        return X;
    };
    const int es = aos ? DIM : 1;  // stride of elements; of components: cs(m)
    auto cs = [&](int m) { return aos ? 1 : (int)a.g[m].nc; };
    auto arr = [&](int m, int which) { return S + a.off[m] + which * DIM * (int)a.g[m].nc; };
    // smooths of level m; then, for the way down, its residual (res)
    auto smooths = [&](int m, int count, bool res) {
        const Grid& g = a.g[m];
        const StagOp<T> A = cs_op<T, VISC>(a, m);
        if constexpr (VISC == 1) {
            if (aos) {
                CSLev<T> V;
                V.set(S, a.off[m], DIM * (int)g.nc);
                CSVisc1<T, DIM> U;
                U.set(A, a.omega);
                if (cs_all_even(g)) {
                    CSPairs<WALL> Q;
                    Q.set(g);
                    if (WALL) Q.set_walls(W);
                    if ((int)threadIdx.x < Q.nt) {
                        cs_split_diag<T, DIM>(Q, U, A, V);  // (each thread reads the ones it wrote)
                        cs_split_smooths<T, DIM, WALL>(Q, W, U, V, count);
                        if (res) cs_split_residual<T, DIM, WALL>(Q, W, U, V);
                    }
                } else {
                    const int na = (int)g.nc >= nt ? nt : ((int)g.nc + 31) & ~31;
                    if ((int)threadIdx.x < na) cs_odd_smooths<T, DIM, WALL>(g, W, U, A, V, count, na);
                }
                __syncthreads();
                return;
            }
        }
        CSStag<T> V;
        V.set(S, a.off[m], DIM, (int)g.nc);
        cs_stag_smooths<T, DIM, VISC>(g, A, V, count, a.jacobi, a.omega);
        if (res) cs_stag_residual<T, DIM, VISC>(g, A, V);
    };
    {
        const CSIdx X = index(0);
        T *ph = arr(0, 0), *rh = arr(0, 1);
        for (int f = threadIdx.x; f < (int)a.g[0].nc; f += nt) {
            int i, j, k;
            cs_ijk(a.g[0], f, i, j, k);
            const int x = X.at(i, j, k) * es;
#pragma unroll
            for (int c = 0; c < DIM; c++) {
                ph[x + c * cs(0)] = a.load_phi ? a.phi[c][f] : T(0);
                rh[x + c * cs(0)] = a.rhs[c][f];
            }
        }
    }
    __syncthreads();
    // down: smooth, residual, restrict (stag_mg_solver.f90:301-380).  Every
    // level but the last is even (an odd extent does not coarsen).
    for (int m = 0; m + 1 < a.nlev; m++) {
        const Grid& gc = a.g[m + 1];
        smooths(m, a.n_down, true);
        const CSIdx X = index(m), Y = index(m + 1);
        const T* F = arr(m, 2);
        T *ph = arr(m + 1, 0), *rh = arr(m + 1, 1);
        const int cf = cs(m), cc = cs(m + 1);
        for (int q = threadIdx.x; q < (int)gc.nc; q += nt) {
            int qi, qj, qk;
            cs_ijk(gc, q, qi, qj, qk);
            const int y = Y.at(qi, qj, qk) * es;
            CSNear<DIM> N;
            N.set(X, 2 * qi, 2 * qj, DIM == 3 ? 2 * qk : 0);
#pragma unroll
            for (int c = 0; c < DIM; c++) {
                rh[y + c * cc] = stag_restrict_expr<T, DIM>(
                    0, [&](int o, int pa, int pb) { return F[N.comp(c, o, pa, pb) * es + c * cf]; });
                ph[y + c * cc] = T(0);
            }
        }
        __syncthreads();
    }
    smooths(a.nlev - 1, a.n_bottom, false);
    // up: prolong, smooth (stag_mg_solver.f90:380-420)
    for (int m = a.nlev - 2; m >= 0; m--) {
        const CSIdx X = index(m), Y = index(m + 1);
        T* F = arr(m, 0);
        const T* Cu = arr(m + 1, 0);
        const int cf = cs(m), cc = cs(m + 1);
        // the coarse value of component c at an offset, under the wall rules
        // (wall_vel)
        auto coarse = [&](const CSNear<DIM>& H, int qi, int qj, int qk, int c, int o, int pa, int pb) {
            if constexpr (WALL) {
                int off[3] = {0, 0, 0};
                off[c] += o;
                off[c == 0 ? 1 : 0] += pa;
                if (DIM == 3) off[c == 2 ? 1 : 2] += pb;
                T sg = T(1);
#pragma unroll
                for (int d = 0; d < DIM; d++) {
                    const int at = (d == 0 ? qi : d == 1 ? qj : qk) + off[d];
                    const bool lo = at < 0, hi = at >= a.g[m + 1].n[d];
                    if (W.lo[d] == 0 || (!lo && !hi)) continue;
                    off[d] = 0;
                    if (d == c) return T(0);
                    if ((lo ? W.lo[d] : W.hi[d]) < 0) sg = -sg;
                }
                return sg * Cu[H.at(off[0], off[1], off[2]) * es + c * cc];
            } else {
                return Cu[H.comp(c, o, pa, pb) * es + c * cc];
            }
        };
        for (int q = threadIdx.x; q < (int)a.g[m + 1].nc; q += nt) {
            int qi, qj, qk;
            cs_ijk(a.g[m + 1], q, qi, qj, qk);
            CSNear<DIM> H;
            H.set(Y, qi, qj, qk);
#pragma unroll
            for (int c = 0; c < DIM; c++) {
                T cv[2][3][3];
#pragma unroll
                for (int o = 0; o < 2; o++)
#pragma unroll
                    for (int pa = -1; pa <= 1; pa++)
#pragma unroll
                        for (int pb = -1; pb <= 1; pb++)
                            cv[o][pa + 1][pb + 1] = (DIM == 3 || pb == 0) ? coarse(H, qi, qj, qk, c, o, pa, pb) : T(0);
#pragma unroll
                for (int pz = 0; pz < (DIM == 3 ? 2 : 1); pz++)
#pragma unroll
                    for (int py = 0; py < 2; py++) {
                        const int r = X.row(2 * qj + py, DIM == 3 ? 2 * qk + pz : 0);
#pragma unroll
                        for (int px = 0; px < 2; px++) {
                            const int I[3] = {px, py, pz};
                            const int oa = I[c == 0 ? 1 : 0] ? 1 : -1;
                            const int ob = (DIM == 3) ? (I[c == 2 ? 1 : 2] ? 1 : -1) : 0;
                            T* v = F + (r + (X.split ? qi : 2 * qi + px) + (((px + py + pz) & 1) ? X.co : 0)) * es +
                                   c * cf;
                            const bool on = WALL && W.lo[c] != 0 && I[c] == 0 &&
                                            (c == 0 ? qi : c == 1 ? qj : qk) == 0;
                            if (!on)
                                *v = *v + stag_prolong_expr<T, DIM>(I[c] == 0, oa, ob, [&](int o, int pa, int pb) {
                                     return cv[o][pa + 1][pb + 1];
                                 });
                        }
                    }
            }
        }
        __syncthreads();
        smooths(m, a.n_up, false);
    }
    {
        const CSIdx X = index(0);
        const T* ph = arr(0, 0);
        for (int f = threadIdx.x; f < (int)a.g[0].nc; f += nt) {
            int i, j, k;
            cs_ijk(a.g[0], f, i, j, k);
            const int x = X.at(i, j, k) * es;
#pragma unroll
            for (int c = 0; c < DIM; c++) a.phi[c][f] = ph[x + c * cs(0)];
        }
    }
}

template <typename T, int DIM, int VISC, bool WALL = false, int NT = CS_THREADS>
__global__ void __launch_bounds__(NT) k_stag_coarse(const __grid_constant__ StagCoarseArgs<T> a) {
    stag_coarse_run<T, DIM, VISC, WALL>(a);
}

// ---------------------------------------------------------------------
// pressure multigrid
// ---------------------------------------------------------------------
// where a level's face coefficients come from
enum { CS_COEF_GLOBAL = 0, CS_COEF_SHARED = 1, CS_COEF_ONE = 2 };

template <typename T>
struct CCCoarseArgs {
    int nlev;
    int load_phi;
    int n_down, n_up, n_bottom;
    T* phi;          // level-0 unknowns in global memory (in/out)
    const T* rhs;
    Grid g[CS_MAXL];
    CCOp<T> A[CS_MAXL];
    int off[CS_MAXL];   // of each level: phi, rhs, odd levels scratch, and
    int coef[CS_MAXL];  // CS_COEF_SHARED: the dim coefficient arrays
};

// Shared-memory offsets of the levels (elements of T), their coefficients
// beside them from the coarsest up as long as cap bytes hold them (coefficients
// of the levels beyond are read from global memory by every sweep; one:
// they are all 1).  The total in bytes.
template <typename T>
inline size_t cc_coarse_layout(CCCoarseArgs<T>& a, int dim, bool one, size_t cap) {
    size_t tot = 0;
    bool even[CS_MAXL];
    for (int m = 0; m < a.nlev; m++) {
        const Grid& g = a.g[m];
        even[m] = !(g.n[0] & 1) && !(g.n[1] & 1) && (dim == 2 || !(g.n[2] & 1));
        tot += (even[m] ? 2 : 3) * (size_t)g.nc;
    }
    for (int m = a.nlev - 1; m >= 0; m--) {
        const size_t add = (size_t)dim * (size_t)a.g[m].nc;
        a.coef[m] = one ? CS_COEF_ONE : CS_COEF_GLOBAL;
        if (one || (tot + add) * sizeof(T) > cap) continue;
        tot += add;
        a.coef[m] = CS_COEF_SHARED;
    }
    size_t off = 0;
    for (int m = 0; m < a.nlev; m++) {
        a.off[m] = (int)off;
        off += ((even[m] ? 2 : 3) + (a.coef[m] == CS_COEF_SHARED ? dim : 0)) * (size_t)a.g[m].nc;
    }
    return tot * sizeof(T);
}

// shared-memory arrays of one level
template <typename T>
struct CSCC {
    T *ph, *rh, *tm, *a;
    int nc;
    __device__ __forceinline__ void set(T* S, int off, int nc_, bool even) {
        nc = nc_;
        ph = S + off;
        rh = ph + nc;
        tm = rh + nc;  // odd levels
        a = even ? rh + nc : tm + nc;
    }
};

// D a G phi and its diagonal at the cell of colour COL in pair h of a row
// (cc_lap_acc's expression; s: the parity of the row)
template <typename T, int DIM, int CF>
__device__ __forceinline__ T cs_cc_lap(const CSPairs<>& Q, const CCOp<T>& A, const CSCC<T>& V, int col, int h, int s,
                                       int b, int ym, int yp, int zm, int zp, T v, T& diag) {
    const bool odd = (s ^ col) & 1;  // the pair's cell of odd i
    const int hp = odd ? (h + 1 == Q.np ? 0 : h + 1) : h, hm = odd ? h : (h == 0 ? Q.np - 1 : h - 1);
    const int own = col ? Q.nh : 0, oth = col ? 0 : Q.nh;
    const T* O = V.ph + oth;
    const int nb[3][2] = {{b + hp, b + hm}, {yp + h, ym + h}, {zp + h, zm + h}};
    T sum = T(0), dg = T(0);
#pragma unroll
    for (int d = 0; d < DIM; d++) {
        T ahi = T(1), alo = T(1);
        if constexpr (CF == CS_COEF_SHARED) {
            ahi = V.a[d * V.nc + oth + nb[d][0]];
            alo = V.a[d * V.nc + own + b + h];
        } else if constexpr (CF == CS_COEF_GLOBAL) {
            // the neighbour above in x is the other cell of its pair
            ahi = ld(A.a[d], 2 * nb[d][0] + ((d == 0) != odd ? 1 : 0));
            alo = ld(A.a[d], 2 * (b + h) + (odd ? 1 : 0));
        }
        sum += ahi * (O[nb[d][0]] - v) - alo * (v - O[nb[d][1]]);
        dg += ahi + alo;
    }
    diag = -dg * A.q;
    return sum * A.q;
}

template <typename T, int DIM, int CF>
__device__ __forceinline__ void cs_cc_split_smooths(const CSPairs<>& Q, const CCOp<T>& A, const CSCC<T>& V, int count) {
    auto sweep = [&](auto Col) {
        constexpr int col = decltype(Col)::value;
        Q.each([&](int h, int s, int b, int ym, int yp, int zm, int zp) {
            const int me = (col ? Q.nh : 0) + b + h;
            const T v = V.ph[me];
            T dg;
            const T L = cs_cc_lap<T, DIM, CF>(Q, A, V, col, h, s, b, ym, yp, zm, zp, v, dg);
            V.ph[me] = v + sm_quot(V.rh[me] - L, dg);
        });
        cs_bar(Q.nt);
    };
    for (int c = 0; c < count; c++) {
        sweep(std::integral_constant<int, 0>());
        sweep(std::integral_constant<int, 1>());
    }
}

// residual of a split level averaged over the 2^dim children of each coarse
// cell (cc_resid_avg)
template <typename T, int DIM, int CF>
__device__ __forceinline__ void cs_cc_split_restrict(const CSPairs<>& Q, const CCOp<T>& A, const CSCC<T>& V,
                                                     const Grid& gc, const CSIdx& Y, const CSCC<T>& W) {
    for (int q = threadIdx.x; q < (int)gc.nc; q += blockDim.x) {
        int qi, qj, qk;
        cs_ijk(gc, q, qi, qj, qk);
        T acc = T(0);
#pragma unroll
        for (int dk = 0; dk < (DIM == 3 ? 2 : 1); dk++)
#pragma unroll
            for (int dj = 0; dj < 2; dj++)
                Q.row(qi, 2 * qj + dj, DIM == 3 ? 2 * qk + dk : 0,
                      [&](int h, int s, int b, int ym, int yp, int zm, int zp) {
#pragma unroll
                          for (int di = 0; di < 2; di++) {
                              const int col = (s + di) & 1;
                              const int me = (col ? Q.nh : 0) + b + h;
                              T dg;
                              const T L = cs_cc_lap<T, DIM, CF>(Q, A, V, col, h, s, b, ym, yp, zm, zp, V.ph[me], dg);
                              acc += V.rh[me] - L;
                          }
                      });
        const int y = Y.at(qi, qj, qk);
        W.rh[y] = acc * (DIM == 3 ? T(0.125) : T(0.25));
        W.ph[y] = T(0);
    }
    __syncthreads();
}

// smooths of an odd level, each colour from one buffer into the other
template <typename T, int DIM, int CF>
__device__ __forceinline__ void cs_cc_odd_smooths(const Grid& g, CCOp<T> A, const CSCC<T>& V, int count, int nt) {
    const int nc = (int)g.nc;
    T *x = V.ph, *y = V.tm;
    for (int s = 0; s < 2 * count; s++) {
        for (int f0 = threadIdx.x; f0 < nc; f0 += nt) {
            int i, j, k;
            cs_ijk(g, f0, i, j, k);
            T v = x[f0];
            if (((i + j + k) & 1) == (s & 1)) {
                CellF P;
                P.set(g, i, j, k);
                T sum = T(0), dg = T(0);
#pragma unroll
                for (int d = 0; d < DIM; d++) {
                    const int dx_ = (d == 0), dy_ = (d == 1), dz_ = (d == 2);
                    const int fp = (int)P.id(dx_, dy_, dz_), fm = (int)P.id(-dx_, -dy_, -dz_);
                    T ahi = T(1), alo = T(1);
                    if constexpr (CF == CS_COEF_SHARED) {
                        ahi = V.a[d * nc + fp];
                        alo = V.a[d * nc + f0];
                    } else if constexpr (CF == CS_COEF_GLOBAL) {
                        ahi = ld(A.a[d], fp);
                        alo = ld(A.a[d], f0);
                    }
                    sum += ahi * (x[fp] - v) - alo * (v - x[fm]);
                    dg += ahi + alo;
                }
                v = v + sm_quot(V.rh[f0] - sum * A.q, -dg * A.q);
            }
            y[f0] = v;
        }
        cs_bar(nt);
        T* t = x;
        x = y;
        y = t;
    }
}

// the coarse end of one pressure V-cycle in the calling CTA; also run per
// box by the batched solver (ONE: its coefficients are all 1)
template <typename T, int DIM, bool ONE>
__device__ __forceinline__ void cc_coarse_run(const CCCoarseArgs<T>& a) {
    extern __shared__ __align__(16) unsigned char cs_smem[];
    T* S = reinterpret_cast<T*>(cs_smem);
    const int nt = blockDim.x;
    auto level = [&](int m) {
        CSCC<T> V;
        V.set(S, a.off[m], (int)a.g[m].nc, cs_all_even(a.g[m]));
        return V;
    };
    auto idx = [&](int m) {
        CSIdx X;
        X.set(a.g[m], cs_all_even(a.g[m]));
        return X;
    };
    auto with_coef = [&](int m, auto&& f) {
        if constexpr (ONE) {
            f(std::integral_constant<int, CS_COEF_ONE>());
        } else {
            if (a.coef[m] == CS_COEF_SHARED) f(std::integral_constant<int, CS_COEF_SHARED>());
            else f(std::integral_constant<int, CS_COEF_GLOBAL>());
        }
    };
    auto smooths = [&](int m, int count) {
        const CSCC<T> V = level(m);
        const CCOp<T> A = a.A[m];
        with_coef(m, [&](auto Cf) {
            constexpr int CF = decltype(Cf)::value;
            if (cs_all_even(a.g[m])) {
                CSPairs<> Q;
                Q.set(a.g[m]);
                if ((int)threadIdx.x < Q.nt) cs_cc_split_smooths<T, DIM, CF>(Q, A, V, count);
            } else {
                const int na = V.nc >= nt ? nt : (V.nc + 31) & ~31;
                if ((int)threadIdx.x < na) cs_cc_odd_smooths<T, DIM, CF>(a.g[m], A, V, count, na);
            }
        });
        __syncthreads();
    };
    {
        const CSCC<T> V = level(0);
        const CSIdx X = idx(0);
        for (int f = threadIdx.x; f < V.nc; f += nt) {
            int i, j, k;
            cs_ijk(a.g[0], f, i, j, k);
            const int x = X.at(i, j, k);
            V.ph[x] = a.load_phi ? a.phi[f] : T(0);
            V.rh[x] = a.rhs[f];
        }
    }
    if constexpr (!ONE) {
        for (int m = 0; m < a.nlev; m++) {
            if (a.coef[m] != CS_COEF_SHARED) continue;
            const CSCC<T> V = level(m);
            const CSIdx X = idx(m);
            for (int f = threadIdx.x; f < V.nc; f += nt) {
                int i, j, k;
                cs_ijk(a.g[m], f, i, j, k);
                const int x = X.at(i, j, k);
#pragma unroll
                for (int d = 0; d < DIM; d++) V.a[d * V.nc + x] = ld(a.A[m].a[d], f);
            }
        }
    }
    __syncthreads();
    // every level but the last is even (an odd extent does not coarsen)
    for (int m = 0; m + 1 < a.nlev; m++) {
        smooths(m, a.n_down);
        with_coef(m, [&](auto Cf) {
            CSPairs<> Q;
            Q.set(a.g[m]);
            cs_cc_split_restrict<T, DIM, decltype(Cf)::value>(Q, a.A[m], level(m), a.g[m + 1], idx(m + 1),
                                                             level(m + 1));
        });
    }
    smooths(a.nlev - 1, a.n_bottom);
    for (int m = a.nlev - 2; m >= 0; m--) {
        const CSCC<T> V = level(m), W = level(m + 1);
        const CSIdx X = idx(m), Y = idx(m + 1);
        for (int q = threadIdx.x; q < W.nc; q += nt) {
            int i, j, k;
            cs_ijk(a.g[m + 1], q, i, j, k);
            const T w = W.ph[Y.at(i, j, k)];
#pragma unroll
            for (int dk = 0; dk < (DIM == 3 ? 2 : 1); dk++)
#pragma unroll
                for (int dj = 0; dj < 2; dj++) {
                    T* p = V.ph + X.row(2 * j + dj, DIM == 3 ? 2 * k + dk : 0) + i;  // (split: pair i of the row)
                    p[0] = p[0] + w;
                    p[X.co] = p[X.co] + w;
                }
        }
        __syncthreads();
        smooths(m, a.n_up);
    }
    {
        const CSCC<T> V = level(0);
        const CSIdx X = idx(0);
        for (int f = threadIdx.x; f < V.nc; f += nt) {
            int i, j, k;
            cs_ijk(a.g[0], f, i, j, k);
            a.phi[f] = V.ph[X.at(i, j, k)];
        }
    }
}

template <typename T, int DIM>
__global__ void __launch_bounds__(CS_THREADS) k_cc_coarse(const __grid_constant__ CCCoarseArgs<T> a) {
    cc_coarse_run<T, DIM, false>(a);
}

}  // namespace fhd
