// Cluster tail of the nodal V-cycle: the coarse levels of the dense 3-D hierarchy and the exact
// bottom in one kernel on one thread-block cluster.  A level's z-slabs are spread over the CTAs;
// phi, the right-hand side, the defect and the cell coefficients of a CTA's slabs are in its shared
// memory, phi also of the two slabs beside them.  The colours p_0 + 2 p_1 + 4 p_2 of one slab parity
// only read slabs of the other one across CTAs, so a sweep is, for each parity, four in-slab colours
// between block barriers, a cluster barrier and the copy of the neighbours' new slabs -- the update
// order of the slab and colour launches it replaces.
//
// What bounds it: latency, and in FP64 the issue rate of the SMs that hold a slab (64 cycles a warp
// instruction and sub-partition).  The launches it replaces (two a sweep and a level, 8-20 us each on
// 2 to 17 blocks, and four of 7-20 us for defect, restriction and prolongation) were a fifth of a
// 256^3 projection and a third of a 96x80x64 FP64 one.
#include "hg_tail.cuh"
#include "mac_cluster.cuh"

namespace mac {
namespace {

// A level as this CTA holds it.  Planes of nodes: row pitch px = nn0 + 1 (column nn0 and row nn1 hold
// zeros: the neighbours outside a non-periodic face); planes 0 .. ks + 1 are the slabs z0 - 1 .. z0 +
// ks.  Layers of cells: pitch n0 + 1, column n0 and row n1 zero; layers 0 .. ks are the cells z0 - 1
// .. z0 + ks - 1.
template <typename T>
struct Slabs {
    int n0, n1, n2;
    int per0, per1, per2;
    int z0, ks;            // own slabs z0 .. z0 + ks - 1
    int nzu, spc;          // slabs with unknowns, slabs a CTA
    int px, pl, cx, cl;    // node row pitch and plane, cell row pitch and layer
    int lx0, lx1, ly0, ly1, lz0, lz1;   // unknown nodes' ranges
    T *phi, *sig, *f, *r;
    unsigned pa, ra;       // shared addresses of phi and r
};

template <typename T>
__device__ __forceinline__ Slabs<T> slabs_of(const HgTailParams<T>& P, int l, int rank, unsigned char* sm) {
    const hg::LevT<T>& L = P.lev[l];
    Slabs<T> S;
    S.n0 = L.n[0];
    S.n1 = L.n[1];
    S.n2 = L.n[2];
    S.per0 = P.geo.per[0];
    S.per1 = P.geo.per[1];
    S.per2 = P.geo.per[2];
    S.spc = P.spc[l];
    S.nzu = S.n2 + (S.per2 ? 0 : 1);
    S.z0 = min(S.nzu, rank * S.spc);
    S.ks = min(S.nzu - S.z0, S.spc);
    S.px = L.nn[0] + 1;
    S.pl = S.px * (L.nn[1] + 1);
    S.cx = S.n0 + 1;
    S.cl = S.cx * (S.n1 + 1);
    S.lx0 = P.geo.dlo[0] ? 1 : 0;
    S.lx1 = S.n0 - (S.per0 || P.geo.dhi[0] ? 1 : 0);
    S.ly0 = P.geo.dlo[1] ? 1 : 0;
    S.ly1 = S.n1 - (S.per1 || P.geo.dhi[1] ? 1 : 0);
    S.lz0 = P.geo.dlo[2] ? 1 : 0;
    S.lz1 = S.n2 - (S.per2 || P.geo.dhi[2] ? 1 : 0);
    S.phi = reinterpret_cast<T*>(sm + P.off[l]);
    S.f = S.phi + (S.spc + 2) * S.pl;
    S.r = S.f + S.spc * S.pl;
    S.sig = S.r + S.spc * S.pl;
    S.pa = smem_u32(S.phi);
    S.ra = smem_u32(S.r);
    return S;
}

// Cluster address of node (x, y) of slab z in phi (its owner's own plane) or in r.
template <typename T>
__device__ __forceinline__ unsigned phi_addr(const Slabs<T>& S, int z, int q) {
    const int cta = z / S.spc;
    return mapa(S.pa + (unsigned)(((z - cta * S.spc + 1) * S.pl + q) * (int)sizeof(T)), cta);
}
template <typename T>
__device__ __forceinline__ unsigned r_addr(const Slabs<T>& S, int z, int q) {
    const int cta = z / S.spc;
    return mapa(S.ra + (unsigned)(((z - cta * S.spc) * S.pl + q) * (int)sizeof(T)), cta);
}

__device__ __forceinline__ float quot(float a, float b) { return a / b; }
__device__ __forceinline__ double quot(double a, double b) { return a * recip_nr(b); }

// The dense operator at node (x, y) of own slab k: node_op_dense3's sums by weight class, the missing
// neighbours and cells read as zeros.
template <typename T, bool ISO>
__device__ __forceinline__ void slab_op(const HgTailParams<T>& P, int l, const Slabs<T>& S, int k, int x, int y,
                                        T& dg, T& off) {
    const int xm = x > 0 ? x - 1 : (S.per0 ? S.n0 - 1 : S.n0 + 1);
    const int xp = S.per0 ? (x == S.n0 - 1 ? 0 : x + 1) : x + 1;       // (x = n0: the zero column)
    const int ym = y > 0 ? y - 1 : (S.per1 ? S.n1 - 1 : S.n1 + 1);
    const int yp = S.per1 ? (y == S.n1 - 1 ? 0 : y + 1) : y + 1;
    const int col[3] = {xm, x, xp}, row[3] = {ym * S.px, y * S.px, yp * S.px};
    const int ca = x > 0 ? x - 1 : (S.per0 ? S.n0 - 1 : S.n0), ra = y > 0 ? y - 1 : (S.per1 ? S.n1 - 1 : S.n1);
    const T* g = S.sig + k * S.cl;
    T s[2][2][2];
#pragma unroll
    for (int zz = 0; zz < 2; ++zz)
#pragma unroll
        for (int yy = 0; yy < 2; ++yy)
#pragma unroll
            for (int xx = 0; xx < 2; ++xx)
                s[zz][yy][xx] = g[zz * S.cl + (yy ? y : ra) * S.cx + (xx ? x : ca)];
    T sx[2][2][3];
#pragma unroll
    for (int zz = 0; zz < 2; ++zz)
#pragma unroll
        for (int yy = 0; yy < 2; ++yy) {
            sx[zz][yy][0] = s[zz][yy][0];
            sx[zz][yy][1] = s[zz][yy][0] + s[zz][yy][1];
            sx[zz][yy][2] = s[zz][yy][1];
        }
    T sxy[2][3][3];
#pragma unroll
    for (int zz = 0; zz < 2; ++zz)
#pragma unroll
        for (int ox = 0; ox < 3; ++ox) {
            sxy[zz][0][ox] = sx[zz][0][ox];
            sxy[zz][1][ox] = sx[zz][0][ox] + sx[zz][1][ox];
            sxy[zz][2][ox] = sx[zz][1][ox];
        }
    const T* ph = S.phi + k * S.pl;
    T am[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    T centre = 0;
#pragma unroll
    for (int oz = 0; oz < 3; ++oz)
#pragma unroll
        for (int oy = 0; oy < 3; ++oy)
#pragma unroll
            for (int ox = 0; ox < 3; ++ox) {
                const T w = oz == 0 ? sxy[0][oy][ox] : (oz == 2 ? sxy[1][oy][ox] : sxy[0][oy][ox] + sxy[1][oy][ox]);
                const int mask = (ox != 1 ? 1 : 0) | (oy != 1 ? 2 : 0) | (oz != 1 ? 4 : 0);
                if (mask == 0)
                    centre = w;
                else if (!(ISO && (mask == 1 || mask == 2 || mask == 4)))
                    am[mask] = fma(w, ph[oz * S.pl + row[oy] + col[ox]], am[mask]);
            }
    const hg::LevT<T>& L = P.lev[l];
    T acc = 0;
#pragma unroll
    for (int m = 1; m < 8; ++m)
        if (!(ISO && (m == 1 || m == 2 || m == 4))) acc = fma(L.kw[m], am[m], acc);
    dg = -L.kw[0] * centre;
    off = acc;
}

// Copies the neighbour slabs of parity sp (both: sp < 0) from their owners.
template <typename T>
__device__ __forceinline__ void refresh(const Slabs<T>& S, int sp) {
    if (S.ks <= 0) return;
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        int z = side ? S.z0 + S.ks : S.z0 - 1;
        if (z < 0 || z >= S.nzu) {
            if (!S.per2) continue;   // (stays zero)
            z += z < 0 ? S.nzu : -S.nzu;
        }
        if (sp >= 0 && (z & 1) != sp) continue;
        T* d = S.phi + (side ? S.ks + 1 : 0) * S.pl;
        const unsigned a = phi_addr(S, z, 0);
        for (int q = threadIdx.x; q < S.pl; q += blockDim.x) d[q] = ld_cluster(a + q * (unsigned)sizeof(T), T(0));
    }
}

template <typename T, bool ISO>
__device__ __forceinline__ void sweeps(const HgTailParams<T>& P, int l, const Slabs<T>& S, int nu) {
    for (int it = 0; it < nu; ++it)
        for (int sp = 0; sp < 2; ++sp) {
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                const int px = c & 1, py = c >> 1;
                const int mx = (S.n0 + 1 - px + 1) / 2, my = (S.n1 + 1 - py + 1) / 2;
                for (int k = (S.z0 + sp) & 1; k < S.ks; k += 2) {
                    const int z = S.z0 + k;
                    if (z < S.lz0 || z > S.lz1) continue;
                    for (int t = threadIdx.x; t < mx * my; t += blockDim.x) {
                        const int iy = fdiv(t, P.mag[l][px]), x = 2 * (t - iy * mx) + px, y = 2 * iy + py;
                        if (x < S.lx0 || x > S.lx1 || y < S.ly0 || y > S.ly1) continue;
                        T dg, off;
                        slab_op<T, ISO>(P, l, S, k, x, y, dg, off);
                        const int q = y * S.px + x;
                        S.phi[(k + 1) * S.pl + q] = quot(S.f[k * S.pl + q] + off, dg);
                    }
                }
                __syncthreads();
            }
            cluster_sync();
            refresh(S, sp);
            __syncthreads();
        }
}

template <typename T, bool ISO>
__device__ __forceinline__ void defects(const HgTailParams<T>& P, int l, const Slabs<T>& S) {
    for (int k = 0; k < S.ks; ++k) {
        const bool zin = S.z0 + k >= S.lz0 && S.z0 + k <= S.lz1;
        for (int q = threadIdx.x; q < S.pl; q += blockDim.x) {
            const int y = q / S.px, x = q - y * S.px;
            T v = 0;
            if (zin && x >= S.lx0 && x <= S.lx1 && y >= S.ly0 && y <= S.ly1) {
                T dg, off;
                slab_op<T, ISO>(P, l, S, k, x, y, dg, off);
                v = S.f[k * S.pl + q] - (dg * S.phi[(k + 1) * S.pl + q] - off);
            }
            S.r[k * S.pl + q] = v;
        }
    }
    cluster_sync();
}

// Full weighting of level F's defect at coarse node (X, Y, Z) (hg::restrict_node).
template <typename T>
__device__ __forceinline__ T restricted(const Slabs<T>& F, int X, int Y, int Z) {
    int qx[3], qy[3], qz[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int x = 2 * X + a - 1, y = 2 * Y + a - 1, z = 2 * Z + a - 1;
        qx[a] = F.per0 ? (x < 0 ? x + F.n0 : x >= F.n0 ? x - F.n0 : x) : (x > F.n0 ? -1 : x);
        qy[a] = F.per1 ? (y < 0 ? y + F.n1 : y >= F.n1 ? y - F.n1 : y) : (y > F.n1 ? -1 : y);
        qz[a] = F.per2 ? (z < 0 ? z + F.n2 : z >= F.n2 ? z - F.n2 : z) : (z > F.n2 ? -1 : z);
    }
    T s = 0;
#pragma unroll
    for (int a2 = 0; a2 < 3; ++a2) {
        const unsigned base = r_addr(F, max(qz[a2], 0), 0);
#pragma unroll
        for (int a1 = 0; a1 < 3; ++a1)
#pragma unroll
            for (int a0 = 0; a0 < 3; ++a0) {
                const bool in = qx[a0] >= 0 && qy[a1] >= 0 && qz[a2] >= 0;
                const T v = ld_cluster(base + (unsigned)((max(qy[a1], 0) * F.px + max(qx[a0], 0)) * (int)sizeof(T)), T(0));
                const T w = (a0 == 1 ? T(1) : T(0.5)) * (a1 == 1 ? T(1) : T(0.5)) * (a2 == 1 ? T(1) : T(0.5));
                s += in ? w * v : T(0);
            }
    }
    return s * T(0.125);
}

// phi += multilinear interpolation of the coarse correction, val(X, Y, Z) at folded coarse nodes
// (hg::prolong_node); then every CTA's neighbour slabs.
template <typename T, class Val>
__device__ __forceinline__ void prolong(const Slabs<T>& S, Val val) {
    const int c0 = S.n0 / 2, c1 = S.n1 / 2, c2 = S.n2 / 2;
    for (int k = 0; k < S.ks; ++k) {
        const int z = S.z0 + k;
        if (z < S.lz0 || z > S.lz1) continue;
        for (int q = threadIdx.x; q < S.pl; q += blockDim.x) {
            const int y = q / S.px, x = q - y * S.px;
            if (x < S.lx0 || x > S.lx1 || y < S.ly0 || y > S.ly1) continue;
            const int X[2] = {x >> 1, S.per0 && (x >> 1) + 1 == c0 ? 0 : (x >> 1) + 1};
            const int Y[2] = {y >> 1, S.per1 && (y >> 1) + 1 == c1 ? 0 : (y >> 1) + 1};
            const int Z[2] = {z >> 1, S.per2 && (z >> 1) + 1 == c2 ? 0 : (z >> 1) + 1};
            const int ox = x & 1, oy = y & 1, oz = z & 1;
            const T w = (ox ? T(0.5) : T(1)) * (oy ? T(0.5) : T(1)) * (oz ? T(0.5) : T(1));
            T s = 0;
#pragma unroll
            for (int a2 = 0; a2 < 2; ++a2)
#pragma unroll
                for (int a1 = 0; a1 < 2; ++a1)
#pragma unroll
                    for (int a0 = 0; a0 < 2; ++a0)
                        if (a2 <= oz && a1 <= oy && a0 <= ox) s += w * val(X[a0], Y[a1], Z[a2]);
            S.phi[(k + 1) * S.pl + q] += s;
        }
    }
    cluster_sync();
    refresh(S, -1);
    cluster_sync();   // (the next sweep rewrites slabs another CTA may still be copying)
}

// Mean of v[0 .. M) in one warp.
template <typename T>
__device__ __forceinline__ double warp_mean(const T* v, int M) {
    double s = 0.0;
    for (int q = threadIdx.x & 31; q < M; q += 32) s += (double)v[q];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s / M;
}

constexpr int kSeg = 16;             // lanes a row of its inverse

}  // namespace

template <typename T>
__global__ void __launch_bounds__(kHgTailThreads)
k_hg_tail(const __grid_constant__ HgTailParams<T> P) {
    extern __shared__ __align__(16) unsigned char hg_tail_smem[];
    __shared__ T fb[kHgTailBottom], eb[kHgTailBottom];
    __shared__ double smean;
    const int tid = threadIdx.x, nt = blockDim.x, M = P.M;
    const unsigned nc = cluster_size();
    const int rank = (int)cluster_rank();
    cluster_arrive();   // (waited for below: every CTA runs before another touches its memory)
    for (int l = 0; l < P.nlev; ++l) {
        const Slabs<T> S = slabs_of<T>(P, l, rank, hg_tail_smem);
        const hg::LevT<T>& L = P.lev[l];
        for (int q = tid; q < (S.spc + 2) * S.pl; q += nt) S.phi[q] = T(0);
        for (int k = 0; k <= S.ks && S.ks > 0; ++k) {
            int z = S.z0 - 1 + k;
            if (S.per2) z = z < 0 ? z + S.n2 : z >= S.n2 ? z - S.n2 : z;
            const bool zin = z >= 0 && z < S.n2;
            for (int q = tid; q < S.cl; q += nt) {
                const int y = q / S.cx, x = q - y * S.cx;
                S.sig[k * S.cl + q] = zin && x < S.n0 && y < S.n1
                                          ? L.sig[x + (long)S.n0 * (y + (long)S.n1 * z)] : T(0);
            }
        }
        if (l == 0) {
            for (int k = 0; k < S.ks; ++k)
                for (int q = tid; q < S.pl; q += nt) {
                    const int y = q / S.px, x = q - y * S.px;
                    S.f[k * S.pl + q] = x <= S.n0 && y <= S.n1
                                            ? P.f0[x + (long)(S.n0 + 1) * (y + (long)(S.n1 + 1) * (S.z0 + k))] : T(0);
                }
        }
    }
    int* bmap = reinterpret_cast<int*>(hg_tail_smem + P.boff);
    const int nb = P.bot.nn[0] * P.bot.nn[1] * P.bot.nn[2];
    for (int q = tid; q < nb; q += nt) bmap[q] = P.map[q];
    __syncthreads();
    cluster_wait();
    // down
    for (int l = 0; l < P.nlev; ++l) {
        const Slabs<T> S = slabs_of<T>(P, l, rank, hg_tail_smem);
        if (P.iso[l]) {
            sweeps<T, true>(P, l, S, P.nu1);
            defects<T, true>(P, l, S);
        } else {
            sweeps<T, false>(P, l, S, P.nu1);
            defects<T, false>(P, l, S);
        }
        if (l + 1 < P.nlev) {
            const Slabs<T> C = slabs_of<T>(P, l + 1, rank, hg_tail_smem);
            for (int k = 0; k < C.ks; ++k) {
                const int z = C.z0 + k;
                for (int q = tid; q < C.pl; q += nt) {
                    const int y = q / C.px, x = q - y * C.px;
                    const bool un = z >= C.lz0 && z <= C.lz1 && x >= C.lx0 && x <= C.lx1 && y >= C.ly0 && y <= C.ly1;
                    C.f[k * C.pl + q] = un ? restricted<T>(S, x, y, z) : T(0);
                }
            }
            __syncthreads();
        } else {
            // bottom: the unknown nodes' right-hand side to every CTA, then the rows of the inverse
            // spread over them, each row's value to every CTA
            const int share = (M + (int)nc - 1) / (int)nc, first = rank * share, last = min(M, first + share);
            for (int u = first + tid; u < last; u += nt) {
                int p[3];
                hg::node_coords(P.bot, P.node[u], p);
                const T v = restricted<T>(S, p[0], p[1], p[2]);
                for (unsigned c = 0; c < nc; ++c) st_cluster(mapa(smem_u32(fb + u), c), v);
            }
            cluster_sync();
            if (P.singular) {
                if (tid < 32) {
                    const double m = warp_mean(fb, M);
                    if (tid == 0) smean = m;
                }
                __syncthreads();
                const T m = (T)smean;
                for (int u = tid; u < M; u += nt) fb[u] -= m;
                __syncthreads();
            }
            for (int u0 = first; u0 < last; u0 += nt / kSeg) {
                const int u = u0 + tid / kSeg, sg = tid % kSeg;
                if (u0 + (tid & ~31) / kSeg >= last) continue;   // (whole warps)
                double x = 0.0;
                if (u < last)
                    for (int v = sg; v < M; v += kSeg) x = fma(__ldg(P.binv + (size_t)u * P.ldb + v), (double)fb[v], x);
                for (int o = kSeg / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                if (u < last && sg < (int)nc) st_cluster(mapa(smem_u32(eb + u), sg), (T)x);
            }
            cluster_sync();
            if (P.singular) {
                if (tid < 32) {
                    const double m = warp_mean(eb, M);
                    if (tid == 0) smean = m;
                }
                __syncthreads();
                const T m = (T)smean;
                for (int u = tid; u < M; u += nt) eb[u] -= m;
                __syncthreads();
            }
        }
    }
    // up
    for (int l = P.nlev - 1; l >= 0; --l) {
        const Slabs<T> S = slabs_of<T>(P, l, rank, hg_tail_smem);
        if (l + 1 < P.nlev) {
            const Slabs<T> C = slabs_of<T>(P, l + 1, rank, hg_tail_smem);
            prolong(S, [&](int X, int Y, int Z) { return ld_cluster(phi_addr(C, Z, Y * C.px + X), T(0)); });
        } else {
            const int m0 = P.bot.nn[0], m1 = P.bot.nn[1];
            prolong(S, [&](int X, int Y, int Z) {
                const int u = bmap[X + m0 * (Y + m1 * Z)];
                return u >= 0 ? eb[u] : T(0);
            });
        }
        if (P.iso[l])
            sweeps<T, true>(P, l, S, P.nu2);
        else
            sweeps<T, false>(P, l, S, P.nu2);
    }
    const Slabs<T> S = slabs_of<T>(P, 0, rank, hg_tail_smem);
    for (int k = 0; k < S.ks; ++k) {
        const int z = S.z0 + k;
        if (z < S.lz0 || z > S.lz1) continue;
        for (int q = tid; q < S.pl; q += nt) {
            const int y = q / S.px, x = q - y * S.px;
            if (x < S.lx0 || x > S.lx1 || y < S.ly0 || y > S.ly1) continue;
            P.e0[x + (long)(S.n0 + 1) * (y + (long)(S.n1 + 1) * z)] = S.phi[(k + 1) * S.pl + q];
        }
    }
    cluster_sync();   // no CTA leaves while another may read its shared memory
}

template <typename T>
size_t hg_tail_plan(HgTailParams<T>& P, int nc) {
    size_t off = 0;
    for (int l = 0; l < P.nlev; ++l) {
        const hg::LevT<T>& L = P.lev[l];
        const int nzu = L.n[2] + (P.geo.per[2] ? 0 : 1);
        P.spc[l] = (nzu + nc - 1) / nc;
        P.off[l] = (int)off;
        for (int px = 0; px < 2; ++px) P.mag[l][px] = div_magic((L.nn[0] - px + 1) / 2);
        const size_t pl = (size_t)(L.nn[0] + 1) * (L.nn[1] + 1), cl = (size_t)(L.n[0] + 1) * (L.n[1] + 1);
        off += pad16(sizeof(T) * ((3 * P.spc[l] + 2) * pl + (P.spc[l] + 1) * cl));
        if (off > (size_t)kHgTailSmem) return 0;
    }
    P.boff = (int)off;
    off += sizeof(int) * (size_t)P.bot.nn[0] * P.bot.nn[1] * P.bot.nn[2];
    return off <= (size_t)kHgTailSmem && P.M <= kHgTailBottom ? off : 0;
}

template <typename T>
void launch_hg_tail(const HgTailParams<T>& P, size_t smem, int nc, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nc);
    cfg.blockDim = dim3(kHgTailThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = nc;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_hg_tail<T>, P);
}

int prepare_hg_tail_kernels(int* nc) {
    *nc = kClusterMax;
    return cluster_opt_in((const void*)k_hg_tail<float>, kHgTailThreads, kHgTailSmem, nc) &&
                   cluster_opt_in((const void*)k_hg_tail<double>, kHgTailThreads, kHgTailSmem, nc)
               ? MAC_OK
               : MAC_ERR_CUDA;
}

template size_t hg_tail_plan<float>(HgTailParams<float>&, int);
template size_t hg_tail_plan<double>(HgTailParams<double>&, int);
template void launch_hg_tail<float>(const HgTailParams<float>&, size_t, int, cudaStream_t);
template void launch_hg_tail<double>(const HgTailParams<double>&, size_t, int, cudaStream_t);

}  // namespace mac
