// fhd_t2.cuh -- whole red-black smooths of the 2D multigrid levels, one or two
// per launch, on tiles in shared memory.
//
// A 2D level of any size in use fits the L2, and a colour launch on it costs
// its launch (1.7 us in a replayed graph at 512^2).  Here a warp owns rows of 32
// x-pairs of cells, one red and one black cell each; a block loads a tile and
// a ring of one cell per sweep, keeps right-hand sides and diagonals (or face
// coefficients) in registers and the values of each colour in shared memory,
// sweeps 2 NS colours with a barrier after each, and stores the tile (out of
// place, so blocks exchange nothing; what the ring computes past its use is
// never stored).  Every update evaluates the expression of the colour sweeps
// on the same operands in the same order: results agree bit for bit.
//
// Two smooths in a replayed graph, FP32 512^2: staggered 14.2 us as eight colour
// launches, 3.6 now; pressure 7.0 us as four, 3.7 now.
#pragma once
#include "fhd_coarse.cuh"

namespace fhd {

constexpr int T2_WARPS = 8;
constexpr int T2_ROWS = 3;  // rows per warp (w, w + 8, w + 16)
constexpr int T2_EY = T2_WARPS * T2_ROWS;
constexpr int T2_THREADS = 32 * T2_WARPS;
// interior of a tile with ns smooths per launch
__host__ __device__ constexpr int t2_tx(int ns) { return 64 - 4 * ns; }
__host__ __device__ constexpr int t2_ty(int ns) { return T2_EY - 4 * ns; }

// a pair of values, as one access where vec says that it is aligned
template <typename T>
__device__ __forceinline__ typename Pair2<T>::V t2_ld(const T* p, bool vec) {
    typedef typename Pair2<T>::V V2;
    if (vec) return *reinterpret_cast<const V2*>(p);
    V2 v = {p[0], p[1]};
    return v;
}
template <typename T>
__device__ __forceinline__ void t2_st(T* p, typename Pair2<T>::V v, bool vec) {
    if (vec) {
        *reinterpret_cast<typename Pair2<T>::V*>(p) = v;
    } else {
        p[0] = v.x;
        p[1] = v.y;
    }
}

// the thread's place in the tile at (x0, y0) of an nx x ny level (both even)
struct T2Place {
    int lane, row, e[T2_ROWS];      // e: linear index of its pair's first cell in each row
    bool inner[T2_ROWS], odd[T2_ROWS];  // stored here; red cell at odd x
    __device__ __forceinline__ void set(int nx, int ny, int x0, int y0, int H) {
        const int tid = threadIdx.x + blockDim.x * threadIdx.y;
        lane = tid & 31;
        row = tid >> 5;
        const int np = nx >> 1, h = (x0 - H) / 2 + lane;  // (x0 and H even; may be negative: exact division)
        int hw = h % np;
        hw = hw < 0 ? hw + np : hw;
#pragma unroll
        for (int r = 0; r < T2_ROWS; r++) {
            const int ry = row + T2_WARPS * r, j = y0 - H + ry;
            int jw = j % ny;
            jw = jw < 0 ? jw + ny : jw;
            e[r] = 2 * hw + nx * jw;
            odd[r] = jw & 1;
            inner[r] = lane >= H / 2 && lane < 32 - H / 2 && h < np && ry >= H && ry < T2_EY - H && j < ny;
        }
    }
    // shared-memory index of the pair at (lane, row of r), the rows below and
    // above it, and the pair to the left or right; at the tile's edge its own
    __device__ __forceinline__ int at(int r) const { return (row + T2_WARPS * r) * 32 + lane; }
    __device__ __forceinline__ int dn(int r) const { return row + T2_WARPS * r > 0 ? at(r) - 32 : at(r); }
    __device__ __forceinline__ int up(int r) const { return row + T2_WARPS * r < T2_EY - 1 ? at(r) + 32 : at(r); }
    __device__ __forceinline__ int side(int r, bool right) const {
        return right ? (lane < 31 ? at(r) + 1 : at(r)) : (lane > 0 ? at(r) - 1 : at(r));
    }
};

// NS smooths of both components of the visc_type 1 operator (ONE: alpha = 1);
// vec: every array is aligned to pairs; sm: 4 x T2_EY x 32
template <typename T, int NS, bool ONE>
__device__ __forceinline__ void t2_stag(int nx, int ny, int x0, int y0, const T* const (&src)[2], T* const (&dst)[2],
                                        const T* const (&rhs)[2], const T* const (&alpha)[2],
                                        const CSVisc1<T, 2>& U, int zero, bool vec, T* sm) {
    typedef typename Pair2<T>::V V2;
    constexpr int H = 2 * NS, PL = 32 * T2_EY;
    T2Place P;
    P.set(nx, ny, x0, y0, H);
    // by colour (0 red, 1 black), component and row
    T v[2][2][T2_ROWS], f[2][2][T2_ROWS], d[2][2][T2_ROWS];
#pragma unroll
    for (int r = 0; r < T2_ROWS; r++)
#pragma unroll
        for (int c = 0; c < 2; c++) {
            V2 u = {T(0), T(0)};
            if (!zero) u = t2_ld(src[c] + P.e[r], vec);
            const V2 b = t2_ld(rhs[c] + P.e[r], vec);
            V2 a = {T(1), T(1)};
            if (!ONE) a = t2_ld(alpha[c] + P.e[r], vec);
            const T d0 = U.as * a.x + U.bd, d1 = U.as * a.y + U.bd;
            const bool o = P.odd[r];
            v[0][c][r] = o ? u.y : u.x; v[1][c][r] = o ? u.x : u.y;
            f[0][c][r] = o ? b.y : b.x; f[1][c][r] = o ? b.x : b.y;
            d[0][c][r] = o ? d1 : d0;   d[1][c][r] = o ? d0 : d1;
            sm[(2 + c) * PL + P.at(r)] = v[1][c][r];
        }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < 2 * NS; s++) {
        const int col = s & 1, oth = col ^ 1;
#pragma unroll
        for (int r = 0; r < T2_ROWS; r++) {
            // the cell is at odd x if its row is odd (red) or even (black);
            // its x neighbour in the next pair is to the right then
            const int ix = P.side(r, P.odd[r] != (col == 1));
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const T* O = sm + (2 * oth + c) * PL;
                const T xs = v[oth][c][r] + O[ix], ys = O[P.up(r)] + O[P.dn(r)];
                v[col][c][r] = U.update(c, v[col][c][r], xs, ys, T(0), f[col][c][r], d[col][c][r]);
                if (s < 2 * NS - 1) sm[(2 * col + c) * PL + P.at(r)] = v[col][c][r];
            }
        }
        if (s < 2 * NS - 1) __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < T2_ROWS; r++)
        if (P.inner[r])
#pragma unroll
            for (int c = 0; c < 2; c++) {
                V2 o;
                o.x = P.odd[r] ? v[1][c][r] : v[0][c][r];
                o.y = P.odd[r] ? v[0][c][r] : v[1][c][r];
                t2_st(dst[c] + P.e[r], o, vec);
            }
}

// NS smooths of the pressure operator D a G (ONE: a = 1); sm: 2 x T2_EY x 32
template <typename T, int NS, bool ONE>
__device__ __forceinline__ void t2_cc(int nx, int ny, int x0, int y0, const T* src, T* dst, const T* rhs, const T* ax,
                                      const T* ay, T q, int zero, bool vec, T* sm) {
    typedef typename Pair2<T>::V V2;
    constexpr int H = 2 * NS, PL = 32 * T2_EY;
    T2Place P;
    P.set(nx, ny, x0, y0, H);
    T v[2][T2_ROWS], f[2][T2_ROWS];
    // x coefficients below the pair, inside it and above; y coefficients below
    // and above, by cell of the pair
    T cx[3][T2_ROWS], cl[2][T2_ROWS], ch[2][T2_ROWS];
#pragma unroll
    for (int r = 0; r < T2_ROWS; r++) {
        V2 u = {T(0), T(0)};
        if (!zero) u = t2_ld(src + P.e[r], vec);
        const V2 b = t2_ld(rhs + P.e[r], vec);
        if (!ONE) {
            const int i0 = P.e[r] % nx, row0 = P.e[r] - i0;
            const int en = i0 + 2 == nx ? row0 : P.e[r] + 2, eu = row0 + nx == nx * ny ? i0 : P.e[r] + nx;
            const V2 a = t2_ld(ax + P.e[r], vec), l = t2_ld(ay + P.e[r], vec), h = t2_ld(ay + eu, vec);
            cx[0][r] = a.x; cx[1][r] = a.y; cx[2][r] = ax[en];
            cl[0][r] = l.x; cl[1][r] = l.y; ch[0][r] = h.x; ch[1][r] = h.y;
        }
        const bool o = P.odd[r];
        v[0][r] = o ? u.y : u.x; v[1][r] = o ? u.x : u.y;
        f[0][r] = o ? b.y : b.x; f[1][r] = o ? b.x : b.y;
        sm[PL + P.at(r)] = v[1][r];
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < 2 * NS; s++) {
        const int col = s & 1, oth = col ^ 1;
#pragma unroll
        for (int r = 0; r < T2_ROWS; r++) {
            const bool odd = P.odd[r] != (col == 1);  // the cell at odd x of its pair
            const T* O = sm + oth * PL;
            const T w = v[col][r], in = v[oth][r], out = O[P.side(r, odd)];
            const T xh = odd ? out : in, xl = odd ? in : out;
            T ah = T(1), al = T(1), bh = T(1), bl = T(1);
            if (!ONE) {
                ah = odd ? cx[2][r] : cx[1][r];
                al = odd ? cx[1][r] : cx[0][r];
                bh = odd ? ch[1][r] : ch[0][r];
                bl = odd ? cl[1][r] : cl[0][r];
            }
            T sum = T(0), dg = T(0);  // cc_lap_acc
            sum += ah * (xh - w) - al * (w - xl);
            dg += ah + al;
            sum += bh * (O[P.up(r)] - w) - bl * (w - O[P.dn(r)]);
            dg += bh + bl;
            const T diag = -dg * q, L = sum * q;
            v[col][r] = w + sm_quot(f[col][r] - L, diag);
            if (s < 2 * NS - 1) sm[col * PL + P.at(r)] = v[col][r];
        }
        if (s < 2 * NS - 1) __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < T2_ROWS; r++)
        if (P.inner[r]) {
            V2 o;
            o.x = P.odd[r] ? v[1][r] : v[0][r];
            o.y = P.odd[r] ? v[0][r] : v[1][r];
            t2_st(dst + P.e[r], o, vec);
        }
}

template <typename T>
struct T2Args {
    const T* src[2];
    T* dst[2];
    const T* rhs[2];
};

template <typename T, int NS>
__global__ void __launch_bounds__(T2_THREADS) k_stag_t2(int nx, int ny, StagOp<T> A, T2Args<T> R, T omega, int zero) {
    __shared__ T sm[4 * 32 * T2_EY];
    CSVisc1<T, 2> U;
    U.set(A, omega);
    const T* const alpha[2] = {A.alpha[0], A.alpha[1]};
    t2_stag<T, NS, false>(nx, ny, blockIdx.x * t2_tx(NS), blockIdx.y * t2_ty(NS), R.src, R.dst, R.rhs, alpha, U, zero, true, sm);
}

template <typename T, int NS>
__global__ void __launch_bounds__(T2_THREADS) k_cc_t2(int nx, int ny, CCOp<T> A, const T* src, T* dst, const T* rhs,
                                                      int zero) {
    __shared__ T sm[2 * 32 * T2_EY];
    t2_cc<T, NS, false>(nx, ny, blockIdx.x * t2_tx(NS), blockIdx.y * t2_ty(NS), src, dst, rhs, A.a[0], A.a[1], A.q,
                        zero, true, sm);
}

inline dim3 t2_grid(const Grid& g, int ns) {
    return dim3((g.n[0] + t2_tx(ns) - 1) / t2_tx(ns), (g.n[1] + t2_ty(ns) - 1) / t2_ty(ns));
}

}  // namespace fhd
