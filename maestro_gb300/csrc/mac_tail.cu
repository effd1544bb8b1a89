// Cluster "tail" of the V-cycle: every level from the first one small enough down to the bottom
// solve runs inside one kernel, on one thread-block cluster whose CTAs share the levels through
// distributed shared memory, so the small levels pay a cluster barrier instead of a kernel launch
// per half-sweep.  The levels' arithmetic is the multi-kernel V-cycle's, operation for operation
// (same fused-multiply-add order per cell, same child order in the restriction, same separable
// trilinear prolongation), so the result is bitwise that of the levels launched one by one with this
// kernel for the bottom alone (coarse_tail = 0).  The bottom solver has reductions and a stopping test
// of its own: it agrees with the one-CTA solver of larger bottoms (mac_kernels.cu) to its tolerance.
//
// What bounds it: latency.  On GB300 a cluster barrier takes ~380 cycles (256 threads a CTA), a
// dependent distributed-shared-memory load ~240, a block barrier 20-80, and an SM sub-partition
// issues one FP64 warp instruction per 64 cycles; a launch-chained half-sweep kernel takes 2-3 us.
// So
//  * a level's rows are spread over all CTAs; a thread owns a pair of x-neighbours (one cell of each
//    colour) for a whole visit of the level, their operator, right-hand side and neighbour addresses in
//    registers; only e and the defects are in (distributed) shared memory;
//  * levels of at most kReplCells<T> cells and the exactly solved bottom are computed by every CTA
//    alone: block barriers only.  Above that the FP64 rate, or the work, of one SM costs more than
//    the cluster barriers saved (whole calls against 512 / 128 cells: none 128^2 mixed +9%, 64^3 +5%;
//    2048 / 256 and 4096 / 512 96 x 112 x 96 mixed +16%);
//  * the first red half-sweep of a level starts from a zero correction, so it reads no neighbour.
// A V-cycle's tail of a 256^3 call (16^3, 8^3 and an exact 4^3 bottom) takes 19 us in FP32 (54 in the
// one-CTA tail it replaces) and 33 in FP64, of which the first execution of every instruction is the
// largest part; a bottom of 3360 cells about 380 us (1358 in one CTA).
#include "mac_internal.cuh"
#include "mac_bottom.cuh"
#include "mac_cluster.cuh"

namespace mac {
namespace {

constexpr int kInvThreads = 1024;
constexpr int kTailMaxThreads = 512;
constexpr int kOps = 17;                 // operator values of a pair in shared memory
template <typename T>
constexpr int kReplCells = sizeof(T) == 4 ? 512 : 128;

__device__ __forceinline__ double fmaT2(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fmaT2(float a, float b, float c) { return fmaf(a, b, c); }

__device__ __forceinline__ void sync_level(bool repl) {
    if (repl)
        __syncthreads();
    else
        cluster_sync();
}

// A level as this CTA sees it: its share of the rows (row = j + n1 k), or all of them (repl).
struct Geo {
    int n0, n1, n2, rz, hn0;
    int row0, rows, repl;
    unsigned cpc, mcpc, mn1, mhn0;
    unsigned ea, ra;   // shared addresses of e and r, index i + n0 (row - row0)
    int pairs;         // pairs per CTA: stride of the operator arrays
    int nops;          // byte offset of the operator arrays in the dynamic shared memory
};
template <typename T>
__device__ __forceinline__ Geo geo_of(const TailParams<T>& P, int l, unsigned rank, unsigned smem) {
    const TailGeo& q = P.geo[l];
    const Dims& D = P.lev[l];
    Geo g;
    g.n0 = D.n0;
    g.n1 = D.n1;
    g.n2 = D.n2;
    g.rz = D.rz;
    g.hn0 = D.n0 >> 1;
    g.repl = q.repl;
    const int R = D.n1 * D.n2;
    g.row0 = q.repl ? 0 : min(R, (int)rank * q.rpc);
    g.rows = min(R - g.row0, q.rpc);
    g.cpc = q.rpc * D.n0;
    g.mcpc = q.mcpc;
    g.mn1 = q.mn1;
    g.mhn0 = q.mhn0;
    g.ea = smem + q.off;
    g.ra = g.ea + g.cpc * (unsigned)sizeof(T);
    g.pairs = q.rpc * g.hn0;
    g.nops = q.off + 2 * (int)(g.cpc * sizeof(T));
    return g;
}

// Shared (cluster) address of entry lin of an array of the level (its local address: base).
template <typename T>
__device__ __forceinline__ unsigned addr_of(const Geo& g, unsigned base, unsigned lin) {
    if (g.repl) return base + lin * (unsigned)sizeof(T);
    const unsigned cta = fdiv(lin, g.mcpc);
    return mapa(base + (lin - cta * g.cpc) * (unsigned)sizeof(T), cta);
}

// A pair of x-neighbours of one row; index s: 0 the colour-0 cell, 1 the colour-1 cell.
template <typename T>
struct Pair {
    bool on;
    int p;              // position (0: cell 2h, 1: cell 2h + 1) of the colour-0 cell
    T c[2][6];          // low/high face coefficients: x-, x+, y-, y+, z-, z+
    T id[2], f[2], e[2];
    unsigned own, xm[2], xp[2];   // shared addresses: cell 2h of e; the x-neighbours outside ...
    unsigned row[4];    // cell 2h of the rows y-, y+, z-, z+ (cluster addresses)
};

// Operator arrays of a pair (stride g.pairs): bx of cells 2h, 2h+1, 2h+2, then by, by+, bz, bz+,
// 1/diag, diag, f of the two cells.
enum { kBx = 0, kBy = 3, kByp = 5, kBz = 7, kBzp = 9, kId = 11, kDg = 13, kF = 15 };

template <typename T, bool Z3>
__device__ __forceinline__ void load_pair(Pair<T>& q, const Geo& g, const T* ops, int t) {
    q.on = t < g.rows * g.hn0;
    if (!q.on) return;
    const int lr = fdiv(t, g.mhn0), h = t - lr * g.hn0;
    const int row = g.row0 + lr, k = fdiv(row, g.mn1), j = row - k * g.n1;
    const int p = (j + k) & 1;
    q.p = p;
    const int S = g.pairs;
    const T* o = ops + t;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const int a = s ? 1 - p : p;   // position of the colour-s cell
        q.c[s][0] = o[(kBx + a) * S];
        q.c[s][1] = o[(kBx + a + 1) * S];
        q.c[s][2] = o[(kBy + a) * S];
        q.c[s][3] = o[(kByp + a) * S];
        q.c[s][4] = o[(kBz + a) * S];
        q.c[s][5] = o[(kBzp + a) * S];
        q.id[s] = o[(kId + a) * S];
        q.f[s] = o[(kF + a) * S];
    }
    constexpr unsigned z = sizeof(T);
    const unsigned base = g.ea + (unsigned)(lr * g.n0) * z;
    q.own = base + 2 * h * z;
    const unsigned lo = base + (h == 0 ? g.n0 - 1 : 2 * h - 1) * z;          // left of cell 2h
    const unsigned hi = base + (h == g.hn0 - 1 ? 0 : 2 * h + 2) * z;         // right of cell 2h+1
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const int a = s ? 1 - p : p;
        q.xm[s] = a ? q.own : lo;
        q.xp[s] = a ? hi : q.own + z;
    }
    const int jm = j == 0 ? g.n1 - 1 : j - 1, jp = j == g.n1 - 1 ? 0 : j + 1;
    const int km = k == 0 ? g.n2 - 1 : k - 1, kp = k == g.n2 - 1 ? 0 : k + 1;
    q.row[0] = addr_of<T>(g, g.ea, 2 * h + g.n0 * (jm + g.n1 * k));
    q.row[1] = addr_of<T>(g, g.ea, 2 * h + g.n0 * (jp + g.n1 * k));
    if (Z3) {
        q.row[2] = addr_of<T>(g, g.ea, 2 * h + g.n0 * (j + g.n1 * km));
        q.row[3] = addr_of<T>(g, g.ea, 2 * h + g.n0 * (j + g.n1 * kp));
    }
}

// acc + the six arms (x-, x+, y-, y+, z-, z+) of the pair's colour-s cell; a 2-D level has no z arm
template <typename T, bool Z3>
__device__ __forceinline__ T arms(T acc, const Pair<T>& q, int s) {
    const unsigned o = (s ? 1 - q.p : q.p) * (unsigned)sizeof(T);
    const T u0 = ld_cluster(q.xm[s], T(0)), u1 = ld_cluster(q.xp[s], T(0));
    const T u2 = ld_cluster(q.row[0] + o, T(0)), u3 = ld_cluster(q.row[1] + o, T(0));
    T u4 = T(0), u5 = T(0);
    if (Z3) {
        u4 = ld_cluster(q.row[2] + o, T(0));
        u5 = ld_cluster(q.row[3] + o, T(0));
    }
    acc = fmaT2(q.c[s][0], u0, acc);
    acc = fmaT2(q.c[s][1], u1, acc);
    acc = fmaT2(q.c[s][2], u2, acc);
    acc = fmaT2(q.c[s][3], u3, acc);
    if (Z3) {
        acc = fmaT2(q.c[s][4], u4, acc);
        acc = fmaT2(q.c[s][5], u5, acc);
    }
    return acc;
}

template <typename T>
__device__ __forceinline__ void store_e(const Pair<T>& q, int s) {
    lds_store(q.own + (s ? 1 - q.p : q.p) * (unsigned)sizeof(T), q.e[s]);
}

// nu sweeps.  zero: from e = 0 -- the first colour-0 half-sweep has no arm that contributes.
// (A predicated-off FP64 instruction still takes its pipe's 64 cycles: the dimension is a template
// parameter, and FP64 levels are never over-relaxed.)
template <typename T, bool Z3>
__device__ __forceinline__ void sweeps(Pair<T>& q, const Geo& g, int nu, T omega, bool zero) {
    const bool sor = sizeof(T) == 4 && omega != T(1);
    if (zero) {
        q.e[0] = q.e[1] = T(0);
        if (nu == 0 && q.on) {
            store_e(q, 0);
            store_e(q, 1);
        }
        if (nu == 0) sync_level(g.repl);
    }
    for (int it = 0; it < nu; ++it) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            if (q.on) {
                T acc = q.f[s];
                if (!(zero && it == 0 && s == 0)) acc = arms<T, Z3>(acc, q, s);
                if (sor)
                    q.e[s] = fmaT2(omega, fmaT2(acc, q.id[s], -q.e[s]), q.e[s]);
                else
                    q.e[s] = acc * q.id[s];
                store_e(q, s);
            }
            sync_level(g.repl);
        }
    }
}

// One level down: sweeps from e = 0 and the defects (colour 0 only after a plain Gauss-Seidel
// black half-sweep) into r.
template <typename T, bool Z3>
__device__ __forceinline__ void visit_down(const TailParams<T>& P, int l, unsigned rank, unsigned char* sm,
                                        bool red_only) {
    const Geo g = geo_of<T>(P, l, rank, smem_u32(sm));
    const T* ops = reinterpret_cast<const T*>(sm + g.nops);
    Pair<T> q;
    load_pair<T, Z3>(q, g, ops, threadIdx.x);
    sweeps<T, Z3>(q, g, P.nu1, P.omega, true);
    const unsigned dr = g.ra - g.ea;
    if (q.on) {
        for (int s = 0; s < (red_only ? 1 : 2); ++s) {
            const int a = s ? 1 - q.p : q.p;
            const T dg = ops[(kDg + a) * g.pairs + threadIdx.x];
            const T e = s ? q.e[1] : q.e[0], f = s ? q.f[1] : q.f[0];
            const T r0 = fmaT2(-dg, e, f);
            const T r = s ? arms<T, Z3>(r0, q, 1) : arms<T, Z3>(r0, q, 0);
            lds_store(q.own + dr + a * (unsigned)sizeof(T), r);
        }
    }
    sync_level(g.repl);
}

// the restricted defect of coarse cell (I, J, K): the mean of its children's, in the order of the
// multi-kernel restriction
template <typename T, bool Z3>
__device__ __forceinline__ T restricted(const Geo& F, int I, int J, int K, bool red_only) {
    constexpr int rz = Z3 ? 2 : 1;
    T v[8];
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            if (b >= rz) continue;
            const int j = 2 * J + a, k = Z3 ? 2 * K + b : K, s = (j + k) & 1;
            const unsigned at = addr_of<T>(F, F.ra, 2 * I + F.n0 * (j + F.n1 * k));
            v[(b * 2 + a) * 2] = ld_cluster(at + s * (unsigned)sizeof(T), T(0));
            if (!red_only) v[(b * 2 + a) * 2 + 1] = ld_cluster(at + (1 - s) * (unsigned)sizeof(T), T(0));
        }
    T sum = T(0);
#pragma unroll
    for (int q = 0; q < 8; ++q)
        if ((q >> 2) < rz && !(red_only && (q & 1))) sum += v[q];
    return sum * (T)(1.0 / (4 * rz));
}

template <typename T>
__device__ __forceinline__ void nb_w(int q, int n, int blo, int bhi, int& qm, int& qp, T& wm, T& wp) {
    wm = T(0.25);
    wp = T(0.25);
    if (q > 0) qm = q - 1;
    else if (blo == MAC_BC_PER) qm = n - 1;
    else {
        qm = 0;
        if (blo == MAC_BC_DIR) wm = T(-0.25);
    }
    if (q < n - 1) qp = q + 1;
    else if (bhi == MAC_BC_PER) qp = 0;
    else {
        qp = n - 1;
        if (bhi == MAC_BC_DIR) wp = T(-0.25);
    }
}

// Where the coarse correction lies: level l + 1's e, or the bottom's (own CTA, or M cells a CTA).
template <typename T>
struct Coarse {
    Geo g;
    unsigned base;
    __device__ __forceinline__ T operator()(int c) const {
        return ld_cluster(addr_of<T>(g, base, (unsigned)c), T(0));
    }
};

// One level up: e += trilinear interpolation of the coarse correction, then the sweeps.
// black_only: colour-1 cells only (plain Gauss-Seidel post-smoothing follows; see k_prolong_add).
template <typename T, bool Z3>
__device__ __forceinline__ void visit_up(const TailParams<T>& P, int l, unsigned rank, unsigned char* sm,
                                      const Coarse<T>& ec, int cn1, int cn2, bool black_only) {
    const Geo g = geo_of<T>(P, l, rank, smem_u32(sm));
    const T* ops = reinterpret_cast<const T*>(sm + g.nops);
    const int cn0 = g.hn0;
    // a row's pairs lie in one warp: the neighbouring coarse columns come from its lanes
    const bool lanes = cn0 <= 32 && (cn0 & (cn0 - 1)) == 0;
    Pair<T> q;
    const int t = threadIdx.x;
    load_pair<T, Z3>(q, g, ops, t);
    const int tt = q.on ? t : 0;   // (idle lanes stay for the shuffles)
    const int lr = fdiv(tt, g.mhn0), I = tt - lr * g.hn0;
    const int row = min(g.row0 + lr, g.n1 * g.n2 - 1);   // (a CTA may own no row)
    const int k = fdiv(row, g.mn1), j = row - k * g.n1;
    const int J = j >> 1, Kc = Z3 ? k >> 1 : k;
    int xs[3], qq[2];
    T wx[2], w[2];
    xs[1] = I;
    nb_w<T>(I, cn0, P.bc.lo[0], P.bc.hi[0], xs[0], xs[2], wx[0], wx[1]);
    nb_w<T>(J, cn1, P.bc.lo[1], P.bc.hi[1], qq[0], qq[1], w[0], w[1]);
    const int Yn = j & 1 ? qq[1] : qq[0];
    const T wy = j & 1 ? w[1] : w[0];
    int Zn = Kc;
    T wz = T(0);
    if (Z3) {
        nb_w<T>(Kc, cn2, P.bc.lo[2], P.bc.hi[2], qq[0], qq[1], w[0], w[1]);
        Zn = k & 1 ? qq[1] : qq[0];
        wz = k & 1 ? w[1] : w[0];
    }
    const int r00 = cn0 * (J + cn1 * Kc), r10 = cn0 * (Yn + cn1 * Kc);
    const int r01 = cn0 * (J + cn1 * Zn), r11 = cn0 * (Yn + cn1 * Zn);
    // coarse column X interpolated in z, then y
    auto column = [&](int X) -> T {
        T zc = ec(X + r00), zn = ec(X + r10);
        if (Z3) {
            const T pc = ec(X + r01), pn = ec(X + r11);
            zc = fmaT2(wz, pc, T(0.75) * zc);
            zn = fmaT2(wz, pn, T(0.75) * zn);
        }
        return fmaT2(wy, zn, T(0.75) * zc);
    };
    T Y[3];
    Y[1] = column(I);
    if (lanes) {
        const int l0 = (threadIdx.x & 31) - I;
        Y[0] = __shfl_sync(0xffffffffu, Y[1], l0 + xs[0]);
        Y[2] = __shfl_sync(0xffffffffu, Y[1], l0 + xs[2]);
    } else {
        Y[0] = column(xs[0]);
        Y[2] = column(xs[2]);
    }
    if (q.on) {
        const T mid = T(0.75) * Y[1];
        const T d0 = fmaT2(wx[0], Y[0], mid), d1 = fmaT2(wx[1], Y[2], mid);   // cells 2I, 2I + 1
        const int p = q.p;
        const unsigned z = sizeof(T);
        const T e0 = ld_cluster(q.own + p * z, T(0)), e1 = ld_cluster(q.own + (1 - p) * z, T(0));
        q.e[0] = black_only ? e0 : e0 + (p ? d1 : d0);
        q.e[1] = e1 + (p ? d0 : d1);
        if (!black_only) store_e(q, 0);
        store_e(q, 1);
    }
    sync_level(g.repl);
    sweeps<T, Z3>(q, g, P.nu2, P.omega, false);
}

// Asynchronous 4/8-byte global -> shared copy (cp.async); completed by cp_async_wait().
template <typename T>
__device__ __forceinline__ void cp_async(T* dst, const T* src) {
    static_assert(sizeof(T) == 4 || sizeof(T) == 8, "4 or 8 bytes");
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src),
                 "n"(sizeof(T))
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.commit_group;\ncp.async.wait_all;" ::: "memory");
}

// ---- bottom: Gauss-Seidel sweeps and BiCGStab over the cluster -------------------------------
// The coarsest level's cells in linear order, M consecutive ones a CTA, one a thread: its operator
// row, its entries of every vector and its neighbours' addresses are registers; x and y, which
// neighbours read, are in distributed shared memory.  nub red/black sweeps, Jacobi-preconditioned
// BiCGStab reducing ||f - A x||_inf by eps, nub sweeps (FBoxLib's bottom, Docs/mg/mg.tex:221-249)
// with f_c / diag_c + sum_n gc_n x_n as the Gauss-Seidel update (gc_n = a_n / diag).  A warp's
// cells have one colour (odd rows excepted), so a half-sweep issues half the FP64 instructions.
// Up to kOneBottom cells belong to one CTA (ONE), four warps on its four FP64 units: spread out they
// issue no faster, and every step waits for the cluster's barrier and remote loads (whole FP64
// calls, 16 CTAs -> one: 40^3 with 125 cells 1701 -> 1270 us, 24 x 40 x 56 with 105 cells 4011 ->
// 2841).  Above that the units are shared by more warps: 26 x 22 with 143 cells takes 1457 us spread
// out and took 1784 in a tail of one CTA.
struct ClBottom {
    int N;
    bool on, odd;            // a cell here; a periodic extent is odd (same-colour neighbours)
    int colour;
    unsigned nb[6];          // cluster addresses of the neighbours' x
    unsigned xa, yoff;       // own x; byte distance from x to y
    double gc[6], dg, id;
};

// Cluster-wide sums v[0..NS) and the maximum of the key in a fixed order; fin(sums, key, out)
// forms the scalars that follow from them in one thread a CTA (an FP64 instruction costs a
// sub-partition 64 cycles for every warp that issues it).  Every thread gets R.out.  The slots
// alternate between calls, so one is rewritten only after a later cluster barrier.
struct ClReduce {
    double ws[4][kTailMaxThreads];
    unsigned long long wk[kTailMaxThreads];
    double slot[2][5][kClusterMax];
    double tot[5];
    double out[4];
};
// The CTAs' barrier, or that of the one CTA's first kOneBottom threads.
constexpr int kOneBottom = 128;
template <bool ONE>
__device__ __forceinline__ void bot_sync() {
    if (ONE)
        asm volatile("bar.sync 1, %0;" ::"n"(kOneBottom) : "memory");
    else
        cluster_sync();
}
template <bool ONE>
__device__ __forceinline__ void cta_sync() {
    if (ONE)
        bot_sync<true>();
    else
        __syncthreads();
}

template <bool ONE, int NS, class Fin>
__device__ __forceinline__ void cl_reduce(ClReduce& R, int& parity, const double (&v)[NS],
                                          unsigned long long key, int nw, Fin fin) {
    static_assert(NS <= 4 && kOneBottom >= 4 * 32, "four sums, a warp each");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (w < nw) {
#pragma unroll
        for (int s = 0; s < NS; ++s) R.ws[s][threadIdx.x] = v[s];
        R.wk[threadIdx.x] = key;
    }
    cta_sync<ONE>();
    const unsigned nc = cluster_size(), rank = cluster_rank();
    constexpr int kw = NS < 4 ? NS : 0;   // the warp that takes the key
    if (w < NS) {
        double s = R.ws[w][lane];
        for (int i = 1; i < nw; ++i) s += R.ws[w][32 * i + lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (ONE) {
            if (lane == 0) R.tot[w] = s;
        } else if (lane < (int)nc) {
            st_cluster(mapa(smem_u32(&R.slot[parity][w][rank]), lane), s);
        }
    }
    if (w == kw) {
        unsigned long long k = R.wk[lane];
        for (int i = 1; i < nw; ++i) {
            const unsigned long long q = R.wk[32 * i + lane];
            k = q > k ? q : k;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long q = __shfl_xor_sync(0xffffffffu, k, o);
            k = q > k ? q : k;
        }
        if (ONE) {
            if (lane == 0) R.tot[4] = __longlong_as_double((long long)k);
        } else if (lane < (int)nc) {
            st_cluster(mapa(smem_u32(&R.slot[parity][4][rank]), lane), __longlong_as_double((long long)k));
        }
    }
    bot_sync<ONE>();
    if (!ONE && w < NS) {
        double s = lane < (int)nc ? R.slot[parity][w][lane] : 0.0;
#pragma unroll
        for (int o = kClusterMax / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) R.tot[w] = s;
    }
    if (!ONE && w == kw) {
        unsigned long long k =
            lane < (int)nc ? (unsigned long long)__double_as_longlong(R.slot[parity][4][lane]) : 0ull;
#pragma unroll
        for (int o = kClusterMax / 2; o > 0; o >>= 1) {
            const unsigned long long q = __shfl_xor_sync(0xffffffffu, k, o);
            k = q > k ? q : k;
        }
        if (lane == 0) R.tot[4] = __longlong_as_double((long long)k);
    }
    if (!ONE) __syncthreads();
    if (threadIdx.x == 0) fin(R.tot, R.tot[4], R.out);
    cta_sync<ONE>();
    parity ^= 1;
}

__device__ __forceinline__ double cl_gsum(const ClBottom& B, unsigned off, double s, bool neg) {
    double u[6];
#pragma unroll
    for (int n = 0; n < 6; ++n) u[n] = ld_cluster(B.nb[n] + off, 0.0);
#pragma unroll
    for (int n = 0; n < 6; ++n) s = fma(neg ? -B.gc[n] : B.gc[n], u[n], s);
    return s;
}

// nu red/black sweeps on x (register x, published).  Where a periodic extent is odd, same-colour
// cells neighbour each other: they are updated from each other's old values.
template <bool ONE>
__device__ __forceinline__ double cl_gsrb(const ClBottom& B, double fi, double x, int nu) {
    for (int it = 0; it < 2 * nu; ++it) {
        const bool act = B.on && B.colour == (it & 1);
        if (act) x = cl_gsum(B, 0, fi, false);
        if (B.odd) bot_sync<ONE>();
        if (act) lds_store(B.xa, x);
        bot_sync<ONE>();
    }
    return x;
}

// Solves for x (in: zero, already published at B.xa by every owner: a bottom is a coarse correction,
// one-level contexts are refused); f's mean comes off when singular.  Every CTA of the cluster runs the same control flow (ONE: the first kOneBottom threads of
// the one CTA).
template <bool ONE>
__device__ __noinline__ double cl_solve(const ClBottom& bottom, ClReduce& R, double f, double x, int nw,
                                        int singular, int nub, double eps, int max_iter, int* iters) {
    const ClBottom B = bottom;   // (registers)
    int parity = 0;
    const unsigned ya = B.xa + B.yoff;
    {
        const double v[1] = {B.on ? f : 0.0};
        cl_reduce<ONE>(R, parity, v, 0ull, nw, [&](const double* t, double, double* o) {
            o[0] = singular ? t[0] / B.N : 0.0;
        });   // (its barrier also publishes x)
    }
    if (singular && B.on) f -= R.out[0];
    const double fi = B.on ? f * B.id : 0.0;
    x = cl_gsrb<ONE>(B, fi, x, nub);
    double r = 0.0, dx = 0.0;
    if (B.on) {
        r = f - B.dg * cl_gsum(B, 0, x, true);
        dx = B.dg * x;
    }
    const double rh = r;
    double p = 0.0, vv = 0.0, rho, beta, omega = 1.0, alpha = 1.0, tol, low;
    {
        const double v[2] = {B.on ? r * r : 0.0, B.on ? fma(f, f, dx * dx) : 0.0};
        // [0] rho = (rh, r) and the first beta (rho_old = alpha = omega = 1); [1] ||r||;  [2] the
        // rounding level of f - A x: a residual that small (the sweeps alone solved the bottom, or
        // a singular one's right-hand side keeps a rounded mean) cannot be reduced further, and
        // iterating on it only adds noise to x.  A 2-norm, so larger than the largest residual's level
        // by up to 10 sqrt(N): harmless from x = 0, decades under what a cycle needs of its bottom, but
        // it would stall a solver that called this again on its own result
        cl_reduce<ONE>(R, parity, v, abs_key(r), nw, [&](const double* t, double k, double* o) {
            o[0] = t[0];
            o[1] = k;
            o[2] = 2e-15 * sqrt(t[1]);
        });
        rho = beta = R.out[0];
        low = R.out[2];
        tol = fmax(eps * R.out[1], low);
    }
    int count = 0;
    if (R.out[1] > low) {
        for (int it = 0; it < max_iter && rho != 0.0; ++it) {
            ++count;
            double y = 0.0, s = 0.0, t = 0.0;
            if (B.on) {
                p = fma(beta, fma(-omega, vv, p), r);
                y = p * B.id;
                lds_store(ya, y);
            }
            bot_sync<ONE>();
            if (B.on) vv = B.dg * cl_gsum(B, B.yoff, y, true);
            // (rh, v); ||r|| of the step before: its test costs one operator application after
            // convergence instead of a reduction every iteration
            const double v1[1] = {B.on ? rh * vv : 0.0};
            cl_reduce<ONE>(R, parity, v1, abs_key(r), nw, [&](const double* q, double k, double* o) {
                o[0] = q[0] == 0.0 ? 0.0 : rho * recip_nr(q[0]);
                o[1] = k;
                o[2] = q[0];
            });
            if (R.out[1] <= tol || R.out[2] == 0.0) break;
            alpha = R.out[0];
            if (B.on) {
                s = fma(-alpha, vv, r);
                x = fma(alpha, y, x);
                y = s * B.id;
                lds_store(ya, y);
            }
            bot_sync<ONE>();
            if (B.on) t = B.dg * cl_gsum(B, B.yoff, y, true);
            double v4[4] = {0.0, 0.0, 0.0, 0.0};
            if (B.on) {
                v4[0] = t * s;
                v4[1] = t * t;
                v4[2] = rh * s;
                v4[3] = rh * t;
            }
            // omega = (t, s) / (t, t); (rh, r_new) = (rh, s) - omega (rh, t); the next beta
            cl_reduce<ONE>(R, parity, v4, abs_key(s), nw, [&](const double* q, double k, double* o) {
                const double w = q[1] > 0.0 ? q[0] * recip_nr(q[1]) : 0.0;
                const double rn = fma(-w, q[3], q[2]);
                o[0] = w;
                o[1] = k;
                o[2] = rn;
                o[3] = (rn * alpha) * recip_nr(rho * w);
            });
            if (R.out[1] <= tol) break;
            omega = R.out[0];
            rho = R.out[2];
            beta = R.out[3];
            if (B.on) {
                x = fma(omega, y, x);
                r = fma(-omega, t, s);
            }
            if (omega == 0.0) break;
        }
    }
    if (B.on) lds_store(B.xa, x);
    bot_sync<ONE>();
    *iters = count;
    return cl_gsrb<ONE>(B, fi, x, nub);
}

// bottom cells per CTA (even: pairs of cells) and the threads they take (colours in warps of
// their own)
__host__ __device__ __forceinline__ int bottom_cells(int N, int nc) {
    const int ctas = N <= kOneBottom ? 1 : nc;
    return 2 * ((N + 2 * ctas - 1) / (2 * ctas));
}
__host__ __device__ __forceinline__ int bottom_threads(int M) { return 2 * ((M / 2 + 31) / 32 * 32); }

}  // namespace

// ONE: a bottom of at most kOneBottom cells, solved by one CTA or by its inverse (an instantiation of its
// own: with both solvers in one kernel the spread one lost 1% of a 3360-cell call).
template <typename T, bool ONE>
__global__ void __launch_bounds__(kTailMaxThreads)
k_tail(const __grid_constant__ TailParams<T> P) {
    extern __shared__ __align__(16) unsigned char tail_smem[];
    __shared__ ClReduce R;
    __shared__ double smean;
    const int tid = threadIdx.x, nt = blockDim.x;
    const unsigned rank = cluster_rank(), nc = cluster_size();
    const bool z3 = P.bottom.n2 > 1 || (P.nlev > 0 && P.lev[0].n2 > 1);
    const int nl = P.nlev;   // non-bottom tail levels
    const Dims& BD = P.bottom;
    const int NB = BD.ncell;
    const bool exact = ONE && P.binv != nullptr;
    const unsigned sbase = smem_u32(tail_smem);
    cluster_arrive();   // (waited for below: every CTA runs before another touches its memory)
    // bottom's shared memory.  exact: the inverse, f, then the solution as T; else x, y (M cells
    // each), then the solution as T
    const int M = P.bottom_m;
    double* bsm = reinterpret_cast<double*>(tail_smem + P.bottom_off);
    double *binv = bsm, *fb = bsm + (size_t)NB * NB;
    T* eb = reinterpret_cast<T*>(exact ? fb + NB : bsm + 2 * M);
    // load the operators (split layout in global memory -> a pair's arrays in shared memory, read
    // back by the same thread).  They are built before the solve starts (and the host waits for
    // that), so their copies are issued before the wait on the preceding kernel and overlap its
    // last part; only the restricted defect f0 comes from that kernel.
    for (int l = 0; l < nl; ++l) {
        const Geo g = geo_of<T>(P, l, rank, sbase);
        const Dims& D = P.lev[l];
        T* ops = reinterpret_cast<T*>(tail_smem + g.nops);
        const T *gbx = P.bx[l], *gby = P.by[l], *gbz = P.bz[l], *gdg = P.dg[l], *gid = P.idg[l];
        const int S = g.pairs;
        for (int t = tid; t < g.rows * g.hn0; t += nt) {
            const int lr = fdiv(t, g.mhn0), h = t - lr * g.hn0;
            const int row = g.row0 + lr, k = fdiv(row, g.mn1), j = row - k * g.n1;
            const int rp = j == g.n1 - 1 ? row - j : row + 1;                      // row of j + 1
            const int rz = k == g.n2 - 1 ? j : row + g.n1;                         // row of k + 1
            // split index of (2h + a) in a row of colour parity c: half ((a + c) & 1), column h
            const int c = (j + k) & 1, cp = (rp - fdiv(rp, g.mn1) * g.n1 + k) & 1;
            const int cz = (j + (k == g.n2 - 1 ? 0 : k + 1)) & 1;
            const int i0 = row * D.hn0 + h, ip = rp * D.hn0 + h, iz = rz * D.hn0 + h;
            const int hn = h == g.hn0 - 1 ? 0 : h + 1;
            T* o = ops + t;
            cp_async(o + (kBx + 2) * S, gbx + c * D.half + row * D.hn0 + hn);
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                const int q = ((a + c) & 1) * D.half + i0;
                cp_async(o + (kBx + a) * S, gbx + q);
                cp_async(o + (kBy + a) * S, gby + q);
                cp_async(o + (kByp + a) * S, gby + ((a + cp) & 1) * D.half + ip);
                cp_async(o + (kBz + a) * S, gbz + q);
                cp_async(o + (kBzp + a) * S, gbz + ((a + cz) & 1) * D.half + iz);
                cp_async(o + (kId + a) * S, gid + q);
                cp_async(o + (kDg + a) * S, gdg + q);
            }
        }
    }
    ClBottom B;
    int bc = 0;   // the thread's bottom cell
    if (exact) {
        for (int q = tid; q < NB * NB; q += nt) cp_async(binv + q, P.binv + q);
    } else {
        // pair q of the CTA's cells: colour 0 to thread q, the other one to the upper half
        const int c0 = min(NB, (int)rank * M), m = min(NB - c0, M), half = bottom_threads(M) / 2;
        const int up = tid >= half, q = tid - (up ? half : 0);
        auto colour = [&](int c) {
            const int row = c / BD.n0;
            return (c - row * BD.n0 + row % BD.n1 + row / BD.n1) & 1;
        };
        int lm = 2 * q + up;
        if (2 * q + 1 < m && colour(c0 + 2 * q) == 1 && colour(c0 + 2 * q + 1) == 0) lm = 2 * q + 1 - up;
        B.N = NB;
        B.on = tid < 2 * half && lm < m;
        B.odd = (BD.n0 & 1 && P.bc.lo[0] == MAC_BC_PER) || (BD.n1 & 1 && P.bc.lo[1] == MAC_BC_PER) ||
                (BD.n2 > 1 && BD.n2 & 1 && P.bc.lo[2] == MAC_BC_PER);
        B.yoff = M * 8u;
        B.xa = smem_u32(bsm) + (B.on ? lm : 0) * 8u;
        B.colour = 0;
        if (B.on) {
            const int c = bc = c0 + lm;
            const int row = c / BD.n0, i = c - row * BD.n0, k = row / BD.n1, j = row - k * BD.n1;
            const int im = i == 0 ? BD.n0 - 1 : i - 1, ip = i == BD.n0 - 1 ? 0 : i + 1;
            const int jm = j == 0 ? BD.n1 - 1 : j - 1, jp = j == BD.n1 - 1 ? 0 : j + 1;
            const int km = k == 0 ? BD.n2 - 1 : k - 1, kp = k == BD.n2 - 1 ? 0 : k + 1;
            const int nb[6] = {im + BD.n0 * row, ip + BD.n0 * row, i + BD.n0 * (jm + BD.n1 * k),
                               i + BD.n0 * (jp + BD.n1 * k), i + BD.n0 * (j + BD.n1 * km),
                               i + BD.n0 * (j + BD.n1 * kp)};
            const double id = P.bidg[c];
            const double w[6] = {P.bbx[c], P.bbx[nb[1]], P.bby[c], P.bby[nb[3]], P.bbz[c], P.bbz[nb[5]]};
            B.colour = (i + j + k) & 1;
            B.id = id;
            B.dg = P.bdg[c];
#pragma unroll
            for (int n = 0; n < 6; ++n) {
                const unsigned cta = fdiv(nb[n], P.bottom_mm);
                B.gc[n] = w[n] * id;
                B.nb[n] = mapa(smem_u32(bsm) + (nb[n] - cta * M) * 8u, cta);
            }
        }
    }
    pdl_wait();
    pdl_trigger();
    double bf = 0.0, bx = 0.0;   // the bottom cell's right-hand side and solution
    if (nl > 0) {
        const Geo g = geo_of<T>(P, 0, rank, sbase);
        const Dims& D = P.lev[0];
        T* ops = reinterpret_cast<T*>(tail_smem + g.nops);
        for (int t = tid; t < g.rows * g.hn0; t += nt) {
            const int lr = fdiv(t, g.mhn0), h = t - lr * g.hn0;
            const int row = g.row0 + lr, k = fdiv(row, g.mn1), j = row - k * g.n1;
#pragma unroll
            for (int a = 0; a < 2; ++a)
                cp_async(ops + (kF + a) * g.pairs + t,
                         P.f0 + ((a + j + k) & 1) * D.half + row * D.hn0 + h);
        }
    } else if (exact) {
        for (int c = tid; c < NB; c += nt) fb[c] = (double)P.f0[c];
    } else if (B.on) {
        bf = (double)P.f0[bc];
        bx = (double)P.e0[bc];
    }
    cp_async_wait();
    __syncthreads();
    cluster_wait();
    // down the V.  red-only defect / black-only prolongation rest on plain Gauss-Seidel half-sweeps
    const bool gs = P.omega == T(1);
    const bool red = gs && P.nu1 > 0, black = gs && P.nu2 > 0;
    for (int l = 0; l < nl; ++l) {
        if (z3) {
            visit_down<T, true>(P, l, rank, tail_smem, red);
        } else {
            visit_down<T, false>(P, l, rank, tail_smem, red);
        }
        const Geo F = geo_of<T>(P, l, rank, sbase);
        auto coarse_f = [&](int I, int J, int K) -> T {
            return z3 ? restricted<T, true>(F, I, J, K, red) : restricted<T, false>(F, I, J, K, red);
        };
        if (l + 1 < nl || exact) {
            // the next level's right-hand side.  One held by every CTA below one that is spread
            // out: each CTA restricts its share and writes it to all of them (reading every
            // defect sixteen times took 8000 cycles for 8^3 cells, this 1500).
            const bool lev = l + 1 < nl;
            const Geo C = geo_of<T>(P, lev ? l + 1 : l, rank, sbase);
            const int n0 = lev ? C.n0 : BD.n0, n1 = lev ? C.n1 : BD.n1;
            const int all = lev ? C.rows * C.n0 : NB;
            const bool push = !F.repl && (!lev || C.repl);
            const int share = push ? (all + (int)nc - 1) / (int)nc : all;
            const int first = push ? (int)rank * share : 0, last = min(all, first + share);
            for (int t = first + tid; t < last; t += nt) {
                const int lrow = t / n0, i = t - lrow * n0;
                const int row = (lev ? C.row0 : 0) + lrow, K = row / n1, J = row - K * n1;
                const T v = coarse_f(i, J, K);
                const unsigned a = lev ? sbase + C.nops + ((kF + (i & 1)) * C.pairs + lrow * C.hn0 + (i >> 1)) * (unsigned)sizeof(T)
                                       : smem_u32(fb) + t * 8u;
                if (push) {
                    for (unsigned c = 0; c < nc; ++c) {
                        if (lev)
                            st_cluster(mapa(a, c), v);
                        else
                            st_cluster(mapa(a, c), (double)v);
                    }
                } else if (lev) {
                    lds_store(a, v);
                } else {
                    lds_store(a, (double)v);
                }
            }
            sync_level(!push);
        } else if (B.on) {
            const int row = bc / BD.n0, K = row / BD.n1;
            bf = (double)coarse_f(bc - row * BD.n0, row - K * BD.n1, K);
        }
    }
    // bottom, FP64 (input rhs rounded through T as in the multi-kernel path); its solution is
    // handed up as T
    int count = 0;
    Coarse<T> cb;
    cb.base = smem_u32(eb);
    cb.g.repl = exact;
    cb.g.cpc = M;
    cb.g.mcpc = P.bottom_mm;
    if (exact) {
        // exact solve by the precomputed (pseudo-)inverse: x = B^-1 (f - mean f) (the mean comes
        // off for a singular operator, whose constant mode B^-1 only scales), by every CTA
        if (P.singular) {
            if (tid < 32) {
                double s = 0.0;
                for (int c = tid; c < NB; c += 32) s += fb[c];
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (tid == 0) smean = s / NB;
            }
            __syncthreads();
            const double mean = smean;
            for (int c = tid; c < NB; c += nt) fb[c] -= mean;
            __syncthreads();
        }
        // row r of B^-1 by kDenseSeg lanes of one warp, the rows spread over the CTAs, each written
        // to all of them (one CTA's FP64 rate makes 64 rows 4000 cycles)
        const int sg = tid % kDenseSeg, share = (NB + (int)nc - 1) / (int)nc;
        const int first = (int)rank * share, last = min(NB, first + share);
        for (int r0 = first; r0 < last; r0 += nt / kDenseSeg) {
            const int r = r0 + tid / kDenseSeg;
            if (r0 + (tid & ~31) / kDenseSeg >= last) continue;   // (whole warps)
            double acc = 0.0;
            if (r < last)
                for (int c = sg; c < NB; c += kDenseSeg) acc = fma(binv[r * NB + c], fb[c], acc);
            for (int o = kDenseSeg / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (r < last && sg < (int)nc) st_cluster(mapa(smem_u32(eb + r), sg), (T)acc);
        }
        cluster_sync();
    } else {
        if (B.on) lds_store(B.xa, bx);
        if (!ONE || (rank == 0 && tid < kOneBottom))
            bx = cl_solve<ONE>(B, R, bf, bx, (ONE ? kOneBottom : bottom_threads(M)) / 32, P.singular, P.nub,
                               P.bottom_eps, P.bottom_max_iter, &count);
        if (B.on) eb[bc - (int)rank * M] = (T)bx;
        cluster_sync();
    }
    // up the V
    for (int l = nl - 1; l >= 0; --l) {
        int cn1 = BD.n1, cn2 = BD.n2;
        Coarse<T> ec = cb;
        if (l + 1 < nl) {
            ec.g = geo_of<T>(P, l + 1, rank, sbase);
            ec.base = ec.g.ea;
            cn1 = ec.g.n1;
            cn2 = ec.g.n2;
        }
        if (z3) {
            visit_up<T, true>(P, l, rank, tail_smem, ec, cn1, cn2, black);
        } else {
            visit_up<T, false>(P, l, rank, tail_smem, ec, cn1, cn2, black);
        }
    }
    // hand the correction back: of the first tail level (its split layout), or the bottom's
    if (nl > 0) {
        const Geo g = geo_of<T>(P, 0, rank, sbase);
        const Dims& D = P.lev[0];
        const T* e = reinterpret_cast<const T*>(tail_smem + P.geo[0].off);
        if (!g.repl || rank == 0)
            for (int t = tid; t < g.rows * g.n0; t += nt) {
                const int pr = t >> 1, a = t & 1;
                const int lr = fdiv(pr, g.mhn0), h = pr - lr * g.hn0;
                const int row = g.row0 + lr, k = fdiv(row, g.mn1), j = row - k * g.n1;
                P.e0[((a + j + k) & 1) * D.half + row * D.hn0 + h] = e[t];
            }
    } else if (exact) {
        if (rank == 0)
            for (int c = tid; c < NB; c += nt) P.e0[c] = eb[c];
    } else if (B.on) {
        P.e0[bc] = (T)bx;
    }
    if (tid == 0 && rank == 0 && P.iters) atomicAdd(P.iters, count);
    cluster_sync();   // no CTA leaves while another may read its shared memory
}

// (Pseudo-)inverse of the bottom operator for the exact bottom solve of the V-cycles: the
// dense N x N matrix of A x = diag x - sum_n a_n x_n (N <= kDenseBottomMax, natural layout; a
// periodic arm that wraps onto the same neighbour twice adds up), plus sigma 1 1^T with sigma =
// mean(diag) / N when A is singular (constant null space: B^-1 f = A^+ f for f of zero mean).
// B is symmetric positive definite, so it is inverted by the symmetric sweep operator (Gauss-
// Jordan elimination without pivoting that keeps the matrix symmetric; after sweeping every
// pivot the matrix holds -B^-1), updating only the upper triangle: N (N + 1) / 2 FMAs a pivot,
// each thread owning fixed elements of the packed triangle so that warps stay full (GB300 issues
// FP64 instructions per warp, whatever the number of active lanes).  FP64, shared memory, one
// CTA, once per solve (on a side stream, overlapping the right-hand-side setup).
constexpr int kInvPerThread = (kDenseBottomMax * (kDenseBottomMax + 1) / 2 + kInvThreads - 1) / kInvThreads;

__global__ void __launch_bounds__(kInvThreads)
k_bottom_inverse(Dims D, const double* __restrict__ bx, const double* __restrict__ by,
                 const double* __restrict__ bz, const double* __restrict__ dg, int singular,
                 double* __restrict__ out) {
    __shared__ double M[kDenseBottomMax * kDenseBottomMax];
    __shared__ double row[kDenseBottomMax], sk[kDenseBottomMax];
    __shared__ double sdiag, sip;
    const int N = D.ncell, tid = threadIdx.x, nt = blockDim.x;
    if (tid < 32) {
        double s = 0.0;
        for (int c = tid; c < N; c += 32) s += dg[c];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (tid == 0) sdiag = singular ? s / ((double)N * N) : 0.0;
    }
    __syncthreads();
    for (int q = tid; q < N * N; q += nt) M[q] = sdiag;
    __syncthreads();
    // row c by thread c (its six arms load in parallel with the other rows')
    if (tid < N) {
        const int c = tid;
        const int i = c % D.n0, rw = c / D.n0, j = rw % D.n1, k = rw / D.n1;
        const int im = i == 0 ? D.n0 - 1 : i - 1, ip = i == D.n0 - 1 ? 0 : i + 1;
        const int jm = j == 0 ? D.n1 - 1 : j - 1, jp = j == D.n1 - 1 ? 0 : j + 1;
        const int km = k == 0 ? D.n2 - 1 : k - 1, kp = k == D.n2 - 1 ? 0 : k + 1;
        const int nbr[6] = {im + D.n0 * (j + D.n1 * k), ip + D.n0 * (j + D.n1 * k),
                            i + D.n0 * (jm + D.n1 * k), i + D.n0 * (jp + D.n1 * k),
                            i + D.n0 * (j + D.n1 * km), i + D.n0 * (j + D.n1 * kp)};
        const double a[6] = {bx[c], bx[nbr[1]], by[c], by[nbr[3]], bz[c], bz[nbr[5]]};
        M[c * N + c] += dg[c];
        for (int n = 0; n < 6; ++n) M[c * N + nbr[n]] -= a[n];
    }
    // the upper-triangle elements (i <= j) this thread updates: packed indices tid + m nt
    int ei[kInvPerThread], ej[kInvPerThread];
    const int npk = N * (N + 1) / 2;
#pragma unroll
    for (int m = 0; m < kInvPerThread; ++m) {
        int p = tid + m * nt, i = 0;
        ei[m] = -1;
        ej[m] = 0;
        if (p < npk) {
            while (p >= N - i) {
                p -= N - i;
                ++i;
            }
            ei[m] = i;
            ej[m] = i + p;
        }
    }
    __syncthreads();
    for (int k = 0; k < N; ++k) {
        // row k of the symmetric matrix (upper-triangle storage) and the pivot's reciprocal
        if (tid < N) row[tid] = tid < k ? M[tid * N + k] : M[k * N + tid];
        if (tid == 0) sip = recip_nr(M[k * N + k]);
        __syncthreads();
        if (tid < N) sk[tid] = row[tid] * sip;
        __syncthreads();
#pragma unroll
        for (int m = 0; m < kInvPerThread; ++m) {
            const int i = ei[m], j = ej[m];
            if (i < 0) continue;
            double& v = M[i * N + j];
            if (i == k)
                v = j == k ? -sip : sk[j];
            else if (j == k)
                v = sk[i];
            else
                v = fma(-row[i], sk[j], v);
        }
        __syncthreads();
    }
    for (int q = tid; q < N * N; q += nt) {
        const int i = q / N, j = q - i * N;
        out[q] = -(i <= j ? M[i * N + j] : M[j * N + i]);
    }
}

void launch_bottom_inverse(const Dims& d, const double* bx, const double* by, const double* bz,
                           const double* dg, bool singular, double* out, cudaStream_t s) {
    k_bottom_inverse<<<1, kInvThreads, 0, s>>>(d, bx, by, bz, dg, singular ? 1 : 0, out);
}

// Fills P's plan (rows a CTA, shared-memory offsets) for a cluster of nc CTAs; returns the dynamic
// shared memory of a CTA, or 0 when the levels or the bottom do not fit.  *threads: of a CTA.
template <typename T>
static size_t plan_tail(TailParams<T>& P, int nc, int* threads) {
    size_t off = 0;
    int most = 0;   // pairs of the widest level
    for (int l = 0; l < P.nlev; ++l) {
        const Dims& D = P.lev[l];
        TailGeo& q = P.geo[l];
        const int R0 = D.n1 * D.n2;
        q.repl = D.ncell <= kReplCells<T>;
        q.rpc = q.repl ? R0 : (R0 + nc - 1) / nc;
        q.mcpc = div_magic(q.rpc * D.n0);
        q.mn1 = div_magic(D.n1);
        q.mhn0 = div_magic(D.n0 >> 1);
        q.off = (int)off;
        const int pairs = q.rpc * (D.n0 >> 1);
        most = pairs > most ? pairs : most;
        off += pad16((size_t)(2 * q.rpc * D.n0 + kOps * pairs) * sizeof(T));
        if (off > (size_t)kTailSmemMax || pairs > kTailMaxThreads) return 0;
    }
    const size_t N = P.bottom.ncell;
    P.bottom_off = (int)off;
    P.bottom_m = bottom_cells(P.bottom.ncell, nc);
    P.bottom_mm = div_magic(P.bottom_m);
    const bool exact = P.binv != nullptr;
    if (exact)
        off += (N * N + N) * sizeof(double) + N * sizeof(T);
    else
        off += P.bottom_m * (2 * sizeof(double) + sizeof(T));
    const int need = exact ? 256 : bottom_threads(P.bottom_m);
    if (off > (size_t)kTailSmemMax || need > kTailMaxThreads) return 0;
    // a pair a thread (a cluster barrier costs 380 cycles with 256 threads, 470 with 512)
    int t = 128;
    while (t < kTailMaxThreads && (t < most || t < need)) t *= 2;
    *threads = t;
    return off;
}

template <typename T>
bool tail_fits(const Dims* lev, int nl, const Dims& bottom, bool exact, int nc) {
    if (nl > kTailMaxLevels) return false;
    TailParams<T> P;
    P.nlev = nl;
    for (int l = 0; l < nl; ++l) P.lev[l] = lev[l];
    P.bottom = bottom;
    static const double some = 0.0;
    P.binv = exact ? &some : nullptr;
    int t;
    return plan_tail<T>(P, nc, &t) > 0;
}

template <typename T>
void launch_tail(TailParams<T>& P, int nc, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    int threads = 0;
    cfg.dynamicSmemBytes = plan_tail<T>(P, nc, &threads);
    cfg.gridDim = dim3(nc);
    cfg.blockDim = dim3(threads);
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = nc;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, P.bottom.ncell <= kOneBottom ? k_tail<T, true> : k_tail<T, false>, P);
}

// Opts the tail kernels into their shared memory and cluster size; *nc: the CTAs of a cluster.
int prepare_tail_kernels(int* nc) {
    *nc = kClusterMax;
    for (const void* k : {(const void*)k_tail<float, true>, (const void*)k_tail<float, false>,
                          (const void*)k_tail<double, true>, (const void*)k_tail<double, false>})
        if (!cluster_opt_in(k, kTailMaxThreads, kTailSmemMax, nc)) return MAC_ERR_CUDA;
    return MAC_OK;
}

template bool tail_fits<float>(const Dims*, int, const Dims&, bool, int);
template bool tail_fits<double>(const Dims*, int, const Dims&, bool, int);
template void launch_tail<float>(TailParams<float>&, int, cudaStream_t);
template void launch_tail<double>(TailParams<double>&, int, cudaStream_t);

}  // namespace mac
