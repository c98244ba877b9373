// fhd_zm.cuh -- whole red-black smooths of the 3D multigrid levels, one or
// two smooths per launch, marching in z with one pair of cells per thread.
//
// A thread owns the cells (2h, 2h+1) of one row: one red and one black cell
// in every plane, so no lane idles in a colour sweep.  Both sit in one
// vector access, and the values a cell needs above and below it are the
// thread's own registers of the neighbouring planes.  Only the x neighbour
// in the next pair and the two y neighbours pass through shared memory, one
// value per pair and colour.
//
// When plane P arrives, stage 0 updates the red cells of plane P-1, stage 1
// the black cells of P-2, and with two smooths per launch stages 2 and 3 the
// red cells of P-3 and the black cells of P-4; the finished plane leaves.
// The stages of a step touch different planes, so one block barrier per
// plane orders them.  A block owns a tile of rows and pairs plus a ring of
// one cell per stage, recomputed from the pre-smooth values it reads (out of
// place, src -> dst), so blocks exchange nothing; rows as long as the domain
// wrap inside the tile and need no ring in x.
//
// Bounds.  Two smooths per launch move the unknown, the right-hand side and
// alpha once instead of twice (256^3: 883 MB of DRAM traffic for two smooths);
// what limits it now is the chain of a step's four stages, which 20 to 28 warps
// an SM (15 in FP64) do not hide: 132 instructions per pair and plane step (FP64
// 172), a third of them the stencil's arithmetic, on 58 % of the issue slots (43
// %), DRAM at 33 % (28 %); of the 8.7 cycles between two issues of a warp 2.6 wait
// for shared memory and 1.6 for the pipeline (1.5 and 2.8).  Staging by
// asynchronous copies three planes ahead, each thread its own pair, took the
// 256^3 pair from 338 to 280 us over register prefetch; unrolling by four
// planes, so that no value is moved between registers, and dropping the
// per-stage bounds checks (what the ring computes past its use is never
// stored) took 454 to 338.
//
// Every update evaluates the expression of the colour sweeps
// (stag_lface_acc) on the same operands in the same order: results agree
// with them bit for bit in FP32 and FP64.
#pragma once
#include <type_traits>

#include "fhd_rb.cuh"

namespace fhd {

// geometry of a march: smooths per launch, the tile and its threads
struct ZMGeom {
    int ns;       // smooths per launch, 1 or 2 (2 ns stages)
    int np;       // pairs per row of the level
    int ip, tx;   // pairs per tile and tiles in x (tx = 1: the whole row, wrapped)
    int TY, ty;   // rows per tile and tiles in y
    int LX, RY;   // pairs and rows of the block, ring included
    int KZ, chunks;
    int threads;
    size_t smem;
};

// most threads of a block: 72 registers each in FP32, 128 in FP64 (twice the
// state); measured best of 640, 768, 896 (FP32, 256^3: 283, 283, 280 us a
// pair of smooths) and 416, 448, 512 (FP64, 128^3: 113, 113, 99 us)
template <typename T>
constexpr int zm_max_threads() { return sizeof(T) == 4 ? 896 : 512; }

constexpr int ZM_AHEAD = 3;  // planes in flight beyond the current one

// asynchronous copy of one pair to shared memory
__device__ __forceinline__ void zm_cp(float2* s, const float* g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g)
                 : "memory");
}
__device__ __forceinline__ void zm_cp(double2* s, const double* g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g)
                 : "memory");
}

template <typename T>
struct ZMArgs {
    const T* src[3];
    T* dst[3];
    const T* rhs[3];
};

// visc_type 1: the update of one cell given its neighbour pair sums
template <typename T, int C>
struct ZMVisc1 {
    T b, q, bq, omega;
    __device__ __forceinline__ T operator()(T v, T xs, T ys, T zs, T rhs, T dg) const {
        const T own = C == 0 ? xs : (C == 1 ? ys : zs);
        T L;
        if constexpr (sizeof(T) == 4) {
            const T oth = C == 0 ? ys + zs : (C == 1 ? xs + zs : xs + ys);
            L = v * dg - (own + oth) * bq;
        } else {
            T oth = T(0);
            oth += C == 0 ? ys : xs;
            oth += C == 2 ? ys : zs;
            L = v * dg - (own + oth) * b * q;
        }
        return v + sm_quot(omega * (rhs - L), dg);
    }
};

template <typename T, int NS, int C>
__device__ __forceinline__ void stag_zm_run(const Grid& g, const ZMGeom& G, const StagOp<T>& A, const ZMArgs<T>& R,
                                            T omega, int zero, T* sm) {
    typedef typename Pair2<T>::V V2;
    constexpr int S = 2 * NS;
    constexpr int PL = zm_max_threads<T>();  // shared-memory values of one plane and stream
    const int nx = g.n[0], ny = g.n[1], nz = g.n[2];
    const int nxy = nx * ny;
    const int tid = threadIdx.x;
    const int ly = tid / G.LX, lx = tid - ly * G.LX;
    const bool on = ly < G.RY;
    const bool wrapx = G.tx == 1;
    const int tile_y = blockIdx.x / G.tx, tile_x = blockIdx.x - tile_y * G.tx;
    int h = tile_x * G.ip - (wrapx ? 0 : NS) + lx, y = tile_y * G.TY - S + ly;
    // interior: the cells this block stores
    const bool inner = on && ly >= S && ly < S + G.TY && y < ny &&
                       (wrapx || (lx >= NS && lx < NS + G.ip && h < G.np));
    h = h < 0 ? h + G.np : h >= G.np ? h - G.np : h;
    y = y < 0 ? y + ny : y >= ny ? y - ny : y;
    const int k0 = blockIdx.y * G.KZ, k1 = k0 + G.KZ < nz ? k0 + G.KZ : nz;
    const i64 base = 2 * (i64)h + (i64)nx * y;
    const T* __restrict__ src = R.src[C] + base;
    const T* __restrict__ rhs = R.rhs[C] + base;
    const T* __restrict__ alp = A.alpha[C] + base;
    ZMVisc1<T, C> U;
    U.b = A.beta[0];
    U.q = A.q;
    U.bq = U.b * A.q;
    U.omega = omega;
    const T bd = T(6) * U.b * A.q;
    const T as = A.alpha_scale;
    // shared memory: stream s (the neighbour values stage s reads), the
    // planes of each parity apart.  A thread outside the staged tile, and
    // the neighbours across the tile's edge, point at the thread's own
    // value: what they give never reaches the interior.
    const int me = tid;
    const int up = on && ly + 1 < G.RY ? me + G.LX : me, dn = on && ly > 0 ? me - G.LX : me;
    const int xm = !on ? me : lx > 0 ? me - 1 : (wrapx ? me + G.LX - 1 : me);
    const int xp = !on ? me : lx + 1 < G.LX ? me + 1 : (wrapx ? me - (G.LX - 1) : me);
    const bool ucoef = on && ly >= 1 && ly < G.RY - 1, uphi = on && !zero;
    // position of the red cell in the pair on the planes of even and odd
    // step, and the pair that holds the x neighbour across the pair's edge
    // (the same for every stage of a step)
    const bool pr0 = (y + k0) & 1;
    const int ox0 = pr0 ? xm : xp, ox1 = pr0 ? xp : xm;
    // values by plane, four planes deep: slot = step % 4 of the plane's
    // arrival (constant indices in the unrolled steps)
    T r0[4], b0[4], r1[4], b1[4], r2[4];  // red / black as read, after smooth 1, red after smooth 2
    T fr[4], dr[4], fb[4], db[4];         // rhs and diagonal of the red and the black cell
    // the thread's own pairs of the planes in flight (the unknown, and the
    // coefficients one plane behind): four slots each, behind the streams
    V2* ring = reinterpret_cast<V2*>(sm + 4 * NS * PL) + me;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        r0[i] = b0[i] = r1[i] = b1[i] = r2[i] = fr[i] = fb[i] = T(0);
        dr[i] = db[i] = T(1);
    }
    const int Pend = k1 + S;  // one past the last plane
    // offsets of the next plane to fetch, wrapped periodically
    int Pf = k0 - S;
    int ou = (Pf < 0 ? Pf + nz : Pf) * nxy;
    auto fetch = [&](int slot) {
        const bool in = Pf < Pend;
        // the coefficients of plane Pf - 1, from the first one used on
        const int oc = ou == 0 ? (nz - 1) * nxy : ou - nxy;
        V2* q = ring + slot * PL;
        if (in && uphi) zm_cp(q, src + ou);
        if (in && ucoef && Pf > k0 - S + 1) {
            zm_cp(q + 4 * PL, rhs + oc);
            zm_cp(q + 8 * PL, alp + oc);
        }
        cp_async_commit();
        Pf++;
        ou += nxy;
        if (ou == nz * nxy) ou = 0;
    };
    {
        // zero unknowns; right-hand sides and alpha of one for the threads that
        // load none: an FP64 quotient of zero takes the division's long way,
        // and with one such thread its warp, for which the block's barrier waits
        // every plane (FP64, one V-cycle: 160^3 1199 -> 950 us, 320 x 320 x 128
        // 3102 -> 2356, 1024 x 512 x 32 4609 -> 3388)
        const V2 z2 = {T(0), T(0)}, o2 = {T(1), T(1)};
        for (int i = 0; i < 12; i++) ring[i * PL] = i < 4 ? z2 : o2;
    }
#pragma unroll
    for (int i = 0; i < ZM_AHEAD; i++) fetch(i);
    T* dst = R.dst[C] + base + (i64)(k0 - 2 * S) * nxy;  // plane P - S of the first step; stored from step 2 S on
    int t = 0;
    const int nst = k1 - k0 + 2 * S;
    auto step = [&](auto Pc) {
        constexpr int p = decltype(Pc)::value;               // step % 4
        constexpr int m1 = (p + 3) & 3, m2 = (p + 2) & 3, m3 = (p + 1) & 3;  // planes P-1, P-2, P-3 (and P-4 = p)
        constexpr int sl = p & 1;
        cp_async_wait<ZM_AHEAD - 1>();
        const V2 u = ring[p * PL], f = ring[(p + 4) * PL], a = ring[(p + 8) * PL];
        fetch((p + ZM_AHEAD) & 3);
        const bool pr = sl ? !pr0 : pr0;
        const int ox = sl ? ox1 : ox0;
        T* s0 = sm + sl * PL;        // the planes of P's parity
        T* s1 = sm + (sl ^ 1) * PL;  // the others
        // the black cell of plane P-4 is finished by this step, from the
        // values that slot p still holds
        const T b0_2 = b0[m2];
        // plane P arrives
        const T rP = pr ? u.y : u.x, bP = pr ? u.x : u.y;
        s0[me] = bP;
        // the coefficients of plane P-1 (its colours the other way round)
        const T d0 = as * a.x + bd, d1 = as * a.y + bd;
        fr[m1] = pr ? f.x : f.y;
        dr[m1] = pr ? d0 : d1;
        const T fbn = pr ? f.y : f.x, dbn = pr ? d1 : d0;
        // stage 0: red of plane P-1
        const T v0 = U(r0[m1], b0[m1] + s1[ox], s1[up] + s1[dn], bP + b0_2, fr[m1], dr[m1]);
        s1[2 * PL + me] = v0;
        // stage 1: black of plane P-2
        const T* q1 = s0 + 2 * PL;
        const T v1 = U(b0_2, r1[m2] + q1[ox], q1[up] + q1[dn], v0 + r1[m3], fb[m2], db[m2]);
        T vr, vb;  // the finished plane P - S
        if constexpr (NS == 2) {
            s0[4 * PL + me] = v1;
            // stage 2: red of plane P-3
            const T* q2 = s1 + 4 * PL;
            const T v2 = U(r1[m3], b1[m3] + q2[ox], q2[up] + q2[dn], v1 + b1[p], fr[m3], dr[m3]);
            s1[6 * PL + me] = v2;
            // stage 3: black of plane P-4
            const T* q3 = s0 + 6 * PL;
            vb = U(b1[p], r2[p] + q3[ox], q3[up] + q3[dn], v2 + r2[m1], fb[p], db[p]);
            vr = r2[p];
            b1[m2] = v1;
            r2[m3] = v2;
        } else {
            vr = r1[m2];
            vb = v1;
        }
        r0[p] = rP;
        b0[p] = bP;
        r1[m1] = v0;
        fb[m1] = fbn;
        db[m1] = dbn;
        if (inner && t >= 2 * S && t < nst) {
            V2 o;
            o.x = pr ? vb : vr;
            o.y = pr ? vr : vb;
            *reinterpret_cast<V2*>(dst) = o;
        }
        dst += nxy;
        t++;
        __syncthreads();
    };
    while (t < nst) {
        step(std::integral_constant<int, 0>());
        step(std::integral_constant<int, 1>());
        step(std::integral_constant<int, 2>());
        step(std::integral_constant<int, 3>());
    }
}

template <typename T, int NS>
__global__ void __launch_bounds__(zm_max_threads<T>(), 1) k_stag_zm(Grid g, ZMGeom G, StagOp<T> A, ZMArgs<T> R,
                                                                    T omega, int zero) {
    extern __shared__ __align__(16) unsigned char zm_raw[];
    T* sm = reinterpret_cast<T*>(zm_raw);
    if (blockIdx.z == 0) stag_zm_run<T, NS, 0>(g, G, A, R, omega, zero, sm);
    else if (blockIdx.z == 1) stag_zm_run<T, NS, 1>(g, G, A, R, omega, zero, sm);
    else stag_zm_run<T, NS, 2>(g, G, A, R, omega, zero, sm);
}

// geometry with ip pairs and TY rows per tile and z-runs of KZ planes; false
// when the level cannot take it (an odd extent, an extent below the ring, or
// a block above its limits)
// (maxt threads a block, per_thread bytes of shared memory each)
inline bool zm_geom(const Grid& g, int ns, int ip, int TY, int KZ, int maxt, int per_thread, ZMGeom& G) {
    const int S = 2 * ns;
    if (g.dim != 3 || g.nc >= (1ll << 31)) return false;
    for (int d = 0; d < 3; d++)
        if ((g.n[d] & 1) || g.n[d] < 4) return false;
    G.ns = ns;
    G.np = g.n[0] / 2;
    G.ip = ip < G.np ? ip : G.np;
    G.tx = (G.np + G.ip - 1) / G.ip;
    G.TY = TY < g.n[1] ? TY : g.n[1];
    G.ty = (g.n[1] + G.TY - 1) / G.TY;
    G.LX = G.tx == 1 ? G.np : G.ip + 2 * ns;
    G.RY = G.TY + 2 * S;
    G.KZ = KZ < g.n[2] ? KZ : g.n[2];
    if (G.ip < 1 || G.TY < 1 || G.KZ < 2 || (G.KZ & 1)) return false;
    G.chunks = (g.n[2] + G.KZ - 1) / G.KZ;
    // one periodic wrap brings every staged index into the domain
    if (G.tx > 1 && (G.tx * G.ip + ns > 2 * G.np || ns > G.np)) return false;
    if (G.ty * G.TY + S > 2 * g.n[1]) return false;
    G.threads = (G.LX * G.RY + 31) / 32 * 32;
    if (G.threads > maxt) return false;
    G.smem = (size_t)per_thread * maxt;
    return true;
}

// pairs that the blocks of a march work on, rings and run-in included, for each
// pair that they store
inline double zm_work(const Grid& g, const ZMGeom& G) {
    return (double)G.threads * G.tx * G.ty * G.chunks * (G.KZ + 4 * G.ns) / ((double)G.np * g.n[1] * g.n[2]);
}

// The tile and the z-runs of a level: the least of waves x plane steps x
// cycles per step.  One block is counted per SM at a time: FP64 blocks of two
// smooths fill its shared memory (128 KB), FP32 ones (112 KB) of more than 448
// threads its registers; smaller FP32 tiles may pair, which the model leaves out.
// A step takes as long as its warps need to issue (per_warp cycles each), or
// the chain of a step's stages when they are few (least).
inline bool zm_pick(const Grid& g, int ns, int sms, int ncomp, int maxt, int per_thread, double per_warp,
                    double least, ZMGeom& best) {
    double cost = -1.0;
    const int np = g.n[0] / 2;
    for (int tx = 1; tx <= 24; tx++) {
        const int ip = (np + tx - 1) / tx;
        if (tx > 1 && ip < 4) break;
        for (int ty = 1; ty <= g.n[1]; ty++) {
            const int TY = (g.n[1] + ty - 1) / ty;
            if (ty > 1 && TY < 4) break;
            if (TY > 32) continue;
            ZMGeom G;
            if (!zm_geom(g, ns, ip, TY, g.n[2] & ~1, maxt, per_thread, G)) continue;
            const double step = per_warp * (G.threads / 32) > least ? per_warp * (G.threads / 32) : least;
            // as many z-runs as fill one, two, .. waves; no split of a tile takes
            // less than its planes spread over the SMs
            const long tiles = (long)G.tx * G.ty * ncomp;
            if (cost >= 0.0 && (double)tiles * g.n[2] / sms * step >= cost) continue;
            int last = 0;
            for (long w = 1; w <= tiles / sms + 4; w++) {
                const long ch = w * sms / tiles;
                if (ch < 1) continue;
                int KZ = ((int)((g.n[2] + ch - 1) / ch) + 1) & ~1;
                if (KZ < 4) KZ = 4;
                if (KZ == last) break;
                last = KZ;
                const long blocks = tiles * ((g.n[2] + KZ - 1) / KZ);
                const double c = (double)((blocks + sms - 1) / sms) * (KZ + 4 * ns) * step;
                if (cost >= 0.0 && c >= cost) continue;
                if (!zm_geom(g, ns, ip, TY, KZ, maxt, per_thread, G)) continue;
                cost = c;
                best = G;
            }
        }
    }
    return cost >= 0.0;
}

// measured on a B200, two smooths per launch: FP32 52 cycles per warp (27
// warps 1430, 20 warps 1010) and no less than 800; FP64 112 and 1650.  The
// forms picked are within 6 % of the best of a sweep over all forms from
// 40^3 to 256^3.
template <typename T>
inline bool stag_zm_pick(const Grid& g, int ns, int sms, ZMGeom& G) {
    return zm_pick(g, ns, sms, 3, zm_max_threads<T>(), (int)sizeof(T) * (4 * ns + 24),
                   (sizeof(T) == 4 ? 26.0 : 56.0) * ns, (sizeof(T) == 4 ? 400.0 : 825.0) * ns, G);
}

}  // namespace fhd
