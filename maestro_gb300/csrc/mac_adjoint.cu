// Adjoint (reverse-mode derivative) of the whole-domain MAC projection.  No counterpart in the
// reference; the forward map is the one of Source/macproject.f90:51-328 as implemented here.
//
// Forward (entries e of the face arrays; face 0 and face n of a periodic direction are separate
// entries of the same physical face):
//   h_f     = 2 / (rho_a + rho_b)                   (physical face f between cells a, b)
//   beta_f  = beta0_f^p h_f,   c_e = beta0_e^(p-1) h_f(e),   p = 1 (+1 with use_alt_energy_fix)
//   f       = P (macrhs - D(beta0 U))               (P removes the mean: singular problem)
//   L phi   = G^T B G phi = f                       (G: cells -> physical faces, 0 on walls)
//   U_proj  = U - c (G phi)
// Loss L = sum_e w_e U_proj,e.  Reverse sweep:
//   lambda  = dL/dphi = G^T-weighted sum of c_e w_e        (k_adj_rhs)
//   L mu    = lambda   -- the same V-cycle solves it (L is symmetric), nu = P mu
//   dL/dmacrhs = nu
//   dL/dU_e    = w_e + beta0_e (nu_hi - nu_lo)/dx   (zero outside the domain: D^T per entry)
//   dL/dbeta_f = -(G nu)_f (G phi)_f,   dL/dc_e = -w_e (G phi)_e
//   dL/dh_f    = beta0^p dL/dbeta_f + sum_{e on f} beta0_e^(p-1) dL/dc_e
//   dL/d(1/rho_a) = sum_{f of a} dL/dh_f * h_f^2 rho_a^2 / 2
//   dL/dbeta0_e   = -U_e (D^T nu)_e + p beta0^(p-1) h dL/dbeta_f + (p-1) beta0^(p-2) h dL/dc_e,
//   summed per layer, beta0_edge = cell_to_edge(beta0) chained on the host (1-D).
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "mac_internal.cuh"

namespace mac {
namespace {

constexpr int kB = 256;

struct AdjGeom {
    int n[3];
    int dm, p;      // p: beta0 exponent (0: no beta0)
    int per[3];
    double idx[3];
    Dims d0;
};

// All kernels below are bound by the FP64 pipe (one warp instruction per 16 cycles of an SM: an
// operation on every cell of 256^3 is 29 us, a pass over an array of 256^3 doubles 20 us), so they
// divide nowhere: the stored coefficient of the finest level is beta'_f = beta0^p h_f / dx^2, and the
// per-layer tables of the forward setup turn it into whatever multiple of h_f is wanted.

// lambda_a = sum over the face entries touching cell a of c_e w_e (+1/dx on the low entry,
// -1/dx on the high entry), walls excluded;  c_e / dx = beta'_f dx / beta0.  A thread marches
// kAdjPlanes planes up and hands the upper face's product to the next plane: 8 FP64 operations a
// cell (with a division for each of the six faces: 2399 us at 256^3; now 346).
constexpr int kAdjPlanes = 8;

template <int DM>
__global__ void __launch_bounds__(kB)
k_adj_rhs(AdjGeom G, const double* __restrict__ bx, const double* __restrict__ by,
          const double* __restrict__ bz, const double* __restrict__ tab,
          const double* __restrict__ wx, const double* __restrict__ wy,
          const double* __restrict__ wz, double* __restrict__ lam) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k0 = blockIdx.z * kAdjPlanes;
    const int n0 = G.n[0], n1 = G.n[1], n2 = G.n[2];
    if (i >= n0 || j >= n1) return;
    const Dims& d = G.d0;
    const int st = G.n[DM - 1] + 1;
    const double* K0 = tab + kTabK0 * st;
    const double* K1 = K0 + st;
    const double* K2 = K1 + st;
    const int plane = n0 * n1;
    double zl = 0.0;   // beta' dx/beta0 w of the cell's lower z face
    if (DM == 3) {
        const int q = i + n0 * j + plane * k0;
        double w = wz[q];
        if (k0 == 0) w = G.per[2] ? w + wz[q + plane * n2] : 0.0;
        zl = bz[level_index(d, i, j, k0)] * w * K2[k0];
    }
    for (int k = k0; k < min(k0 + kAdjPlanes, n2); ++k) {
        const int c = level_index(d, i, j, k);
        const int fx = i + (n0 + 1) * (j + n1 * k), fy = i + n0 * (j + (n1 + 1) * k);
        const int fz = i + n0 * j + plane * (k + 1);
        double xl = wx[fx], xh = wx[fx + 1], yl = wy[fy], yh = wy[fy + n0];
        double zw = DM == 3 ? wz[fz] : 0.0;
        const bool ex = i == 0 || i == n0 - 1, ey = j == 0 || j == n1 - 1;
        const bool ez = DM == 3 && k == n2 - 1;
        if (ex || ey || ez) {   // entries 0 and n of a periodic direction are one face; walls: none
            if (i == 0) xl = G.per[0] ? xl + wx[fx + n0] : 0.0;
            if (i == n0 - 1) xh = G.per[0] ? xh + wx[fx + 1 - n0] : 0.0;
            if (j == 0) yl = G.per[1] ? yl + wy[fy + n0 * n1] : 0.0;
            if (j == n1 - 1) yh = G.per[1] ? yh + wy[fy + n0 - n0 * n1] : 0.0;
            if (ez) zw = G.per[2] ? zw + wz[fz - plane * n2] : 0.0;
        }
        const double bxh = bx[level_index(d, i < n0 - 1 ? i + 1 : 0, j, k)];
        const double byh = by[level_index(d, i, j < n1 - 1 ? j + 1 : 0, k)];
        double s = fma(bxh, xh, -(bx[c] * xl)) * K0[DM == 3 ? k : j];
        if (DM == 3) {
            s = fma(fma(byh, yh, -(by[c] * yl)), K1[k], s);
            const double zh = bz[level_index(d, i, j, k < n2 - 1 ? k + 1 : 0)] * zw * K2[k + 1];
            s += zh - zl;
            zl = zh;
        } else {
            s = fma(byh * yh, K1[j + 1], s);
            s = fma(-(by[c] * yl), K1[j], s);
        }
        lam[i + n0 * (j + n1 * k)] = s;
    }
}

// Sum of a level-0 array for the mean of mu, in a fixed order: kMeanBlocks blocks, each thread
// four running sums (a shared-memory tree for every 256 elements took 247 us at 256^3; now 30).
constexpr int kMeanBlocks = 608;

__device__ __forceinline__ double block_sum(double v) {   // result in thread 0
    __shared__ double sm[32];
    const int t = threadIdx.x + blockDim.x * threadIdx.y;
    const int nw = (blockDim.x * blockDim.y) >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((t & 31) == 0) sm[t >> 5] = v;
    __syncthreads();
    if (t == 0)
        for (int w = 1; w < nw; ++w) v += sm[w];
    return v;
}

__global__ void __launch_bounds__(kB)
k_partial_sum(int n, const double* __restrict__ a, double* __restrict__ part) {
    const int step = kMeanBlocks * kB;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    long q = blockIdx.x * kB + threadIdx.x;
    for (; q + 3L * step < n; q += 4L * step) {
        s0 += a[q];
        s1 += a[q + step];
        s2 += a[q + 2L * step];
        s3 += a[q + 3L * step];
    }
    for (; q < n; q += step) s0 += a[q];
    const double s = block_sum((s0 + s1) + (s2 + s3));
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

__global__ void k_final_mean(int n, const double* __restrict__ part, double* __restrict__ out) {
    double s = 0.0;
    for (int b = threadIdx.x; b < kMeanBlocks; b += blockDim.x) s += part[b];
    s = block_sum(s);
    if (threadIdx.x == 0) out[0] = s / n;
}

// nu = mu - mean(mu) in the natural layout.
__global__ void __launch_bounds__(kB)
k_mu_to_nat(Dims d, const double* __restrict__ mu, const double* __restrict__ mean,
            double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    if (i >= d.n0 || j >= d.n1) return;
    out[i + d.n0 * (j + d.n1 * k)] = mu[level_index(d, i, j, k)] - mean[0];
}

struct FaceIo {
    const double* beta;   // beta' of this direction, level-0 layout
    const double* u;
    const double* w;
    const double* phi;    // natural
    const double* nu;     // natural
    double* du;           // dL/dU entries (natural face layout)
    double* g;            // -dL/dh_f h_f^2 / 2 shares per entry (null: not wanted)
    double* part;         // [layer][tile] sums of the dL/dbeta0_e shares (null: not wanted)
    int cols, tiles;      // tiles of a layer's plane: along x, in all
};

// Per face entry of direction D, all in one pass: dU, the share of dL/d(1/rho) and the layer sums
// of dL/dbeta0_e.  With t = beta' dphi, dmu = nu_hi - nu_lo (nu = 0 outside the domain), b = beta0:
//   dU = w + (b/dx) dmu,   g = -(1/2) h^2 dL/dh = beta' t (A dmu + C w),
//   dL/dbeta0_e = u dmu / dx - t (p/b dmu + (p-1) dx/b^2 w)
// with A and C constant on a layer, like every factor of the last line, which is therefore summed
// as three plain products.  A block covers blockDim.x columns and kFaceRows rows a thread of one
// layer's plane, so that its reduction costs about one FP64 operation an entry.  11 of them an entry:
// 256^3 took 1012 us a direction (division, general index arrays, an array of shares and 470 us to
// sum it), now 393 to 459.
constexpr int kFaceRows = 8;

template <int D, bool ALT>   // ALT: p = 2
__global__ void __launch_bounds__(kB)
k_adj_face(AdjGeom G, const double* __restrict__ tab, FaceIo io) {
    const int n0 = G.n[0], n1 = G.n[1];
    const int m0 = n0 + (D == 0), m1 = n1 + (D == 1);
    const bool v3 = G.dm == 3;
    const int r = blockIdx.x / io.tiles;      // vertical index: z in 3-D, y in 2-D
    const int tile = blockIdx.x - r * io.tiles;
    const int st = G.n[G.dm - 1] + 1;
    const int rows = v3 ? m1 : 1;             // rows of the layer's plane
    const int i = tile % io.cols * blockDim.x + threadIdx.x;
    const int row0 = tile / io.cols * blockDim.y * kFaceRows;
    const int row1 = min(rows, row0 + (int)blockDim.y * kFaceRows);
    const double gd = tab[(kTabG0 + D) * st + r], kd = tab[(kTabK0 + D) * st + r];
    const double A = -recip_nr(tab[(kTabFac0 + D) * st + r]), C = kd * A;
    const int sd = D == 0 ? 1 : (D == 1 ? n0 : n0 * n1);
    const int nd = G.n[D];
    const bool sums = io.part != nullptr;
    double a1 = 0.0, a2 = 0.0, a3 = 0.0;
    if (i < m0)
        for (int row = row0 + threadIdx.y; row < row1; row += blockDim.y) {
            const int j = v3 ? row : r, k = v3 ? r : 0;
            const int q = i + m0 * (j + m1 * k);
            const int c = i + n0 * (j + n1 * k);   // the cell above the face
            const int qd = D == 0 ? i : (D == 1 ? j : k);
            const double we = io.w[q];
            // dmu: over the entry, nu = 0 outside; dmf: over the physical face, which the solve uses
            // once (entry n of a periodic direction is the duplicate)
            double dmu, dmf = 0.0, dphi = 0.0, b = 0.0;
            if (qd > 0 && qd < nd) {
                dmu = io.nu[c] - io.nu[c - sd];
                dphi = io.phi[c] - io.phi[c - sd];
                b = io.beta[level_index(G.d0, i, j, k)];
                dmf = dmu;
            } else {
                dmu = qd == 0 ? io.nu[c] : -io.nu[c - sd];
                if (G.per[D]) {
                    const int lo = qd == 0 ? c + (nd - 1) * sd : c - sd;
                    const int hi = qd == 0 ? c : c - nd * sd;
                    dphi = io.phi[hi] - io.phi[lo];
                    b = io.beta[level_index(G.d0, D == 0 ? 0 : i, D == 1 ? 0 : j, D == 2 ? 0 : k)];
                    if (qd == 0) dmf = io.nu[hi] - io.nu[lo];
                }
            }
            const double ue = sums ? io.u[q] : 0.0;
            const double t = b * dphi;
            io.du[q] = fma(gd, dmu, we);
            if (io.g) io.g[q] = t * fma(A, dmf, C * we) * b;
            if (sums) {
                a1 = fma(ue, dmu, a1);
                a2 = fma(t, dmf, a2);
                if (ALT) a3 = fma(t, we, a3);
            }
        }
    if (!sums) return;
    const double ib = kd * G.idx[D];   // 1 / beta0
    double v = a1 * G.idx[D];
    v = fma(ALT ? -2.0 * ib : -ib, a2, v);
    if (ALT) v = fma(-ib * kd, a3, v);
    v = block_sum(v);
    if (threadIdx.x == 0 && threadIdx.y == 0)
        io.part[blockIdx.x] = v;
}

// dL/d(1/rho_a) = sum over the physical faces of a of dL/dh_f * h_f^2 rho_a^2 / 2: the faces'
// shares g carry the factors of dL/dh_f (zero on walls), so 7 FP64 operations a cell remain
// (2300 us at 256^3 with a division a face; now 246).
__global__ void __launch_bounds__(kB)
k_adj_sigma(AdjGeom G, const double* __restrict__ rho, const double* __restrict__ gx,
            const double* __restrict__ gy, const double* __restrict__ gz,
            double* __restrict__ ds) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    const int n0 = G.n[0], n1 = G.n[1], n2 = G.n[2];
    if (i >= n0 || j >= n1) return;
    const int q = i + n0 * (j + n1 * k);
    const double rc = rho[q];
    const int fx = i + (n0 + 1) * (j + n1 * k), fy = i + n0 * (j + (n1 + 1) * k);
    double s = (gx[fx] + gx[fx + 1]) + (gy[fy] + gy[fy + n0]);
    const int pl = n0 * n1;
    if (G.dm == 3) s += gz[q] + gz[q + pl];
    // periodic: the other entry of a boundary face (one branch, no predicated FP64 adds inside)
    const bool ex = i == 0 || i == n0 - 1, ey = j == 0 || j == n1 - 1;
    const bool ez = G.dm == 3 && (k == 0 || k == n2 - 1);
    if (ex || ey || ez) {
        if (ex) s += gx[i == 0 ? fx + n0 : fx + 1 - n0];
        if (ey) s += gy[j == 0 ? fy + n0 * n1 : fy + n0 - n0 * n1];
        if (ez) s += gz[k == 0 ? q + pl * n2 : q + pl - pl * n2];
    }
    ds[q] = s * (rc * rc);
}

// One warp per vertical index r: the block sums of the horizontal faces of layer r (r < nr) into
// sh[r], of the vertical faces of plane r (r <= nr) into sv[r].
__global__ void k_layer_sums(int dm, int nr, int t0, int t1, int t2, const double* __restrict__ p0,
                             const double* __restrict__ p1, const double* __restrict__ p2,
                             double* __restrict__ sh, double* __restrict__ sv) {
    const int r = blockIdx.x;
    const int nb[3] = {t0, t1, t2};
    const double* p[3] = {p0, p1, p2};
    double a = 0.0, v = 0.0;
    if (r < nr)
        for (int d = 0; d < dm - 1; ++d)
            for (int t = threadIdx.x; t < nb[d]; t += 32) a += p[d][(long)r * nb[d] + t];
    for (int t = threadIdx.x; t < nb[dm - 1]; t += 32) v += p[dm - 1][(long)r * nb[dm - 1] + t];
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        v += __shfl_down_sync(0xffffffffu, v, o);
    }
    if (threadIdx.x == 0) {
        if (r < nr) sh[r] = a;
        sv[r] = v;
    }
}

// Transpose of cell_to_edge (Source/cell_to_edge.f90:39-60) applied to the edge sensitivities sv:
// adds sum_r sv[r] d(edge_r)/d(cell_k) to g[k].  The limiter is taken in the branch the forward
// evaluation selects.
void cell_to_edge_vjp(int nr, const double* c, const double* sv, double* g) {
    for (int r = 0; r <= nr; ++r) {
        const double s = sv[r];
        if (r == 0) {
            g[0] += s;
        } else if (r == 1) {
            g[0] += 0.5 * s;
            if (nr > 1) g[1] += 0.5 * s;
        } else if (r == nr) {
            g[r - 1] += s;
        } else if (r == nr - 1) {
            g[r] += 0.5 * s;
            g[r - 1] += 0.5 * s;
        } else {
            const double tmp = 7.0 / 12.0 * (c[r] + c[r - 1]) - 1.0 / 12.0 * (c[r + 1] + c[r - 2]);
            const double lo = std::min(c[r], c[r - 1]), hi = std::max(c[r], c[r - 1]);
            if (tmp < lo) {
                g[c[r] <= c[r - 1] ? r : r - 1] += s;
            } else if (tmp > hi) {
                g[c[r] >= c[r - 1] ? r : r - 1] += s;
            } else {
                g[r] += 7.0 / 12.0 * s;
                g[r - 1] += 7.0 / 12.0 * s;
                g[r + 1] -= 1.0 / 12.0 * s;
                g[r - 2] -= 1.0 / 12.0 * s;
            }
        }
    }
}

// Block of k_adj_face: (32, 8) threads over a plane in 3-D, a single row in 2-D.
dim3 face_block(const mac_ctx* c) { return c->dm == 3 ? dim3(32, 8) : dim3(kB, 1); }

}  // namespace
}  // namespace mac

using namespace mac;

extern "C" int mac_macproject_adjoint_dense(mac_ctx* c, const double* ux, const double* uy,
                                            const double* uz, const double* rho,
                                            const double* macrhs, const double* beta0,
                                            const double* beta0_edge, const double* wx,
                                            const double* wy, const double* wz, double* dux,
                                            double* duy, double* duz, double* drinv,
                                            double* dbeta0, double* dmacrhs, double* phi_out,
                                            mac_stats* stats) {
    mac_stats local;
    mac_stats* st = stats ? stats : &local;
    std::memset(st, 0, sizeof(*st));
    if (!c || !ux || !uy || !rho || !wx || !wy || !dux || !duy) return st->status = MAC_ERR_INVALID;
    if (c->dm == 3 && (!uz || !wz || !duz)) return st->status = MAC_ERR_INVALID;
    if ((beta0 == nullptr) != (beta0_edge == nullptr)) return st->status = MAC_ERR_INVALID;
    if (dbeta0 && !beta0) return st->status = MAC_ERR_INVALID;
    // MAESTRO's vertical direction is never periodic (beta0 is a stratified profile); the
    // periodic-vertical face bookkeeping of beta0_edge is not differentiated
    if (beta0 && c->bc_lo[c->va] == MAC_BC_PER) return st->status = MAC_ERR_UNSUPPORTED;
    for (int d = 0; d < c->dm; ++d)
        if (c->bc_lo[d] == MAC_BC_DIR || c->bc_hi[d] == MAC_BC_DIR) return st->status = MAC_ERR_UNSUPPORTED;
    const auto t0 = std::chrono::steady_clock::now();
    begin_call_stats(c, st);
    const size_t N = (size_t)c->n[0] * c->n[1] * c->n[2];
    const int nr = c->n[c->va];
    // sums of this call: [mean, kMeanBlocks partials, sh[nr], sv[nr + 1], layer partials of each d];
    // everything of the size of a field uses solver arrays that are idle at the time
    size_t off[4] = {(size_t)(1 + kMeanBlocks + 2 * nr + 1), 0, 0, 0};
    const dim3 fb = face_block(c);
    int cols[3], tiles[3] = {0, 0, 0}, layers[3];
    for (int d = 0; d < c->dm; ++d) {
        cols[d] = ceil_div(c->n[0] + (d == 0), fb.x);
        tiles[d] = cols[d] * ceil_div(c->dm == 3 ? c->n[1] + (d == 1) : 1, fb.y * kFaceRows);
        layers[d] = nr + (d == c->va);
        off[d + 1] = off[d] + (size_t)tiles[d] * layers[d];
    }
    if (!c->adj_sums && alloc_device(c, (void**)&c->adj_sums, off[c->dm] * sizeof(double)))
        return st->status = MAC_ERR_ALLOC;
    double* mean = c->adj_sums;
    double* part = mean + 1;
    double* layer = part + kMeanBlocks;
    cudaStream_t s = c->stream;
    Level& F = c->lev[0];
    const double* uin[3] = {ux, uy, uz};
    const double* win[3] = {wx, wy, wz};
    double* dout[3] = {dux, duy, duz};
    // ---- forward: phi of the projection, in c->phin.  The velocities are read where they are and
    // not corrected (the gradient does not need the projected ones).
    double* saved_rho = c->rho;
    double* saved_u[3] = {c->u[0], c->u[1], c->u[2]};
    c->rho = const_cast<double*>(rho);
    for (int d = 0; d < c->dm; ++d) c->u[d] = const_cast<double*>(uin[d]);
    mac_stats fst;
    std::memset(&fst, 0, sizeof(fst));
    auto forward = [&]() -> int {
        MAC_CUDA_TRY(cudaMemsetAsync(c->phin, 0, N * sizeof(double), s));
        const int r = beta0 ? load_beta0(c, MAC_PTR_DEVICE, beta0, beta0_edge) : MAC_OK;
        return r ? r : forward_phi(c, macrhs, beta0 != nullptr, &fst);
    };
    int rc = forward();
    for (int d = 0; d < c->dm; ++d) c->u[d] = saved_u[d];
    if (rc != MAC_OK) {
        c->rho = saved_rho;
        return st->status = rc;
    }

    AdjGeom G;
    for (int d = 0; d < 3; ++d) {
        G.n[d] = c->n[d];
        G.per[d] = (d < c->dm && c->bc_lo[d] == MAC_BC_PER) ? 1 : 0;
        G.idx[d] = 1.0 / c->dx[d];
    }
    G.dm = c->dm;
    G.p = beta0 ? (c->o.use_alt_energy_fix ? 2 : 1) : 0;
    G.d0 = F.d;
    const Grid3 g = grid3(c->n[0], c->n[1], c->n[2]);

    // ---- adjoint right-hand side and solve with the same hierarchy
    auto adjoint_rhs = [&]() -> int {
        if (phi_out)
            MAC_CUDA_TRY(cudaMemcpyAsync(phi_out, c->phin, N * sizeof(double), cudaMemcpyDeviceToDevice, s));
        const dim3 rg(g.grid.x, g.grid.y, ceil_div(c->n[2], kAdjPlanes));
        auto kern = c->dm == 3 ? k_adj_rhs<3> : k_adj_rhs<2>;
        kern<<<rg, g.block, 0, s>>>(G, F.a64.bx, F.a64.by, F.a64.bz, c->b0tab, wx, wy,
                                    c->dm == 3 ? wz : wy, c->scratch);
        MAC_CUDA_TRY(cudaGetLastError());
        const int r = setup_rhs_from(c, c->scratch);
        if (r) return r;
        MAC_CUDA_TRY(cudaMemsetAsync(F.a64.phi, 0, N * sizeof(double), s));
        return MAC_OK;
    };
    rc = adjoint_rhs();
    if (rc) {
        c->rho = saved_rho;
        return st->status = rc;
    }
    const int solve_rc = run_solve(c, st);
    c->rho = saved_rho;
    if (solve_rc != MAC_OK && solve_rc != MAC_ERR_NOT_CONVERGED) return st->status = solve_rc;
    // nu = mu - mean(mu)
    double* nu = dmacrhs ? dmacrhs : c->scratch;
    k_partial_sum<<<kMeanBlocks, kB, 0, s>>>((int)N, F.a64.phi, part);
    k_final_mean<<<1, 1024, 0, s>>>((int)N, part, mean);
    k_mu_to_nat<<<g.grid, g.block, 0, s>>>(F.d, F.a64.phi, mean, nu);
    MAC_CUDA_TRY(cudaGetLastError());

    // ---- per-face gradients (the faces' shares of dL/d(1/rho) go to the solver's velocity arrays)
    const double* beta[3] = {F.a64.bx, F.a64.by, F.a64.bz};
    for (int d = 0; d < c->dm; ++d) {
        const FaceIo io{beta[d], uin[d], win[d], c->phin, nu, dout[d], drinv ? c->u[d] : nullptr,
                        dbeta0 ? c->adj_sums + off[d] : nullptr, cols[d], tiles[d]};
        auto kern = G.p == 2 ? (d == 0   ? k_adj_face<0, true>
                                : d == 1 ? k_adj_face<1, true>
                                         : k_adj_face<2, true>)
                             : (d == 0   ? k_adj_face<0, false>
                                : d == 1 ? k_adj_face<1, false>
                                         : k_adj_face<2, false>);
        kern<<<tiles[d] * layers[d], fb, 0, s>>>(G, c->b0tab, io);
        MAC_CUDA_TRY(cudaGetLastError());
    }
    if (drinv) {
        k_adj_sigma<<<g.grid, g.block, 0, s>>>(G, rho, c->u[0], c->u[1], c->u[2], drinv);
        MAC_CUDA_TRY(cudaGetLastError());
    }
    if (dbeta0) {
        k_layer_sums<<<nr + 1, 32, 0, s>>>(c->dm, nr, tiles[0], tiles[1], tiles[2],
                                           c->adj_sums + off[0], c->adj_sums + off[1],
                                           c->adj_sums + off[2], layer, layer + nr);
        MAC_CUDA_TRY(cudaGetLastError());
        std::vector<double> h(2 * nr + 1), cb(nr), gb(nr);
        MAC_CUDA_TRY(cudaMemcpyAsync(h.data(), layer, (2 * nr + 1) * sizeof(double), cudaMemcpyDeviceToHost, s));
        MAC_CUDA_TRY(cudaMemcpyAsync(cb.data(), beta0, nr * sizeof(double), cudaMemcpyDeviceToHost, s));
        MAC_CUDA_TRY(cudaStreamSynchronize(s));
        for (int k = 0; k < nr; ++k) gb[k] = h[k];
        cell_to_edge_vjp(nr, cb.data(), h.data() + nr, gb.data());
        MAC_CUDA_TRY(cudaMemcpyAsync(dbeta0, gb.data(), nr * sizeof(double), cudaMemcpyHostToDevice, s));
    }
    MAC_CUDA_TRY(cudaStreamSynchronize(s));
    st->vcycles += fst.vcycles;
    st->setup_ms += fst.setup_ms;
    st->solve_ms += fst.solve_ms;
    st->status = solve_rc;
    end_call_stats(c, st);
    st->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return solve_rc;
}
