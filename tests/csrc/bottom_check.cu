// Runs one bottom problem through the cluster's solver (mac_tail.cu) and through the one-CTA solver
// (mac_kernels.cu), two implementations of the same method with their own reductions, stopping tests
// and memory, from a zero guess; up to 64 cells also through the dense inverse.  Prints the largest
// residuals (over |f|) and the distance of the solutions (mean removed where the operator is singular).
// Arguments: n0 n1 n2 dm top(1: Dirichlet) per_vertical seed.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "mac_internal.cuh"

using namespace mac;

int main(int argc, char** argv) {
    if (argc != 8) return 2;
    const int n[3] = {atoi(argv[1]), atoi(argv[2]), atoi(argv[3])}, dm = atoi(argv[4]);
    const int top = atoi(argv[5]), per_v = atoi(argv[6]);
    std::mt19937_64 g((unsigned)atoi(argv[7]));
    std::uniform_real_distribution<double> coef(0.5, 2.0), val(-1.0, 1.0);
    const int N = n[0] * n[1] * n[2], va = dm - 1;
    BcDesc bc;
    for (int d = 0; d < 3; ++d) bc.lo[d] = bc.hi[d] = d < dm ? (d < va || per_v ? MAC_BC_PER : MAC_BC_NEU) : MAC_BC_NEU;
    if (top && !per_v) bc.hi[va] = MAC_BC_DIR;
    const bool singular = bc.hi[va] != MAC_BC_DIR;
    auto at = [&](int i, int j, int k) { return i + n[0] * (j + n[1] * k); };
    std::vector<double> b[3], dg(N, 0.0), id(N), f(N);
    std::vector<int> nb(6 * (size_t)N);
    for (int d = 0; d < 3; ++d) b[d].assign(N, 0.0);
    for (int k = 0; k < n[2]; ++k)
        for (int j = 0; j < n[1]; ++j)
            for (int i = 0; i < n[0]; ++i) {
                const int q[3] = {i, j, k}, c = at(i, j, k);
                f[c] = val(g);
                for (int d = 0; d < 3; ++d) {
                    int m[3] = {i, j, k}, p[3] = {i, j, k};
                    m[d] = (q[d] + n[d] - 1) % n[d];
                    p[d] = (q[d] + 1) % n[d];
                    nb[6 * (size_t)c + 2 * d] = at(m[0], m[1], m[2]);
                    nb[6 * (size_t)c + 2 * d + 1] = at(p[0], p[1], p[2]);
                    if (d < dm && (q[d] > 0 || bc.lo[d] == MAC_BC_PER)) b[d][c] = coef(g);
                    if (d == va && q[d] == n[d] - 1 && bc.hi[d] == MAC_BC_DIR) dg[c] += 2.0 * coef(g);
                }
            }
    auto arm = [&](int c, int s) { return s & 1 ? b[s / 2][nb[6 * (size_t)c + s]] : b[s / 2][c]; };
    double mean = 0.0;
    for (int c = 0; c < N; ++c) {
        for (int s = 0; s < 6; ++s) dg[c] += arm(c, s);
        id[c] = 1.0 / dg[c];
        mean += f[c] / N;
    }
    auto dev = [&](const std::vector<double>& v) {
        double* p = nullptr;
        cudaMalloc(&p, v.size() * sizeof(double));
        cudaMemcpy(p, v.data(), v.size() * sizeof(double), cudaMemcpyHostToDevice);
        return p;
    };
    LevelArrays<double> A;
    A.bx = dev(b[0]);
    A.by = dev(b[1]);
    A.bz = dev(b[2]);
    A.diag = dev(dg);
    A.invdiag = dev(id);
    double* df = dev(f);
    double* dx = dev(std::vector<double>(N, 0.0));
    double* scr = dev(std::vector<double>((size_t)(2 + kBotScrPerCell) * N, 0.0));
    double* inv = dev(std::vector<double>((size_t)kDenseBottomMax * kDenseBottomMax, 0.0));
    int* its = nullptr;
    cudaMalloc(&its, sizeof(int));
    Dims D{n[0], n[1], n[2], n[0] / 2, N / 2, N, 0, dm == 3 ? 2 : 1};
    int nc = 0;
    if (prepare_tail_kernels(&nc)) return 3;
    const double eps = 1e-10;
    std::vector<double> x[3];
    int count[3] = {0, 0, 0};
    for (int way = 0; way < (N <= kDenseBottomMax ? 3 : 2); ++way) {
        cudaMemset(dx, 0, N * sizeof(double));
        cudaMemset(its, 0, sizeof(int));
        if (way == 0) {
            launch_bottom<double>(D, A, dx, df, scr, singular, 10, eps, 1000, its, 0);
        } else {
            TailParams<double> P{};
            P.nlev = 0;
            P.bottom = D;
            P.bbx = A.bx;
            P.bby = A.by;
            P.bbz = A.bz;
            P.bdg = A.diag;
            P.bidg = A.invdiag;
            P.f0 = df;
            P.e0 = dx;
            P.bc = bc;
            P.nu1 = P.nu2 = 2;
            P.nub = 10;
            P.singular = singular ? 1 : 0;
            P.bottom_max_iter = 1000;
            P.bottom_eps = eps;
            P.iters = its;
            P.omega = 1.0;
            if (way == 2) {
                launch_bottom_inverse(D, A.bx, A.by, A.bz, A.diag, singular, inv, 0);
                P.binv = inv;
            }
            launch_tail<double>(P, nc, 0);
        }
        x[way].resize(N);
        if (cudaDeviceSynchronize() != cudaSuccess) return 4;
        cudaMemcpy(x[way].data(), dx, N * sizeof(double), cudaMemcpyDeviceToHost);
        cudaMemcpy(&count[way], its, sizeof(int), cudaMemcpyDeviceToHost);
    }
    double res[3] = {0, 0, 0}, dist[3] = {0, 0, 0}, fm = 0.0, xm = 0.0;
    for (int way = 0; way < 3 && !x[way].empty(); ++way) {
        double m = 0.0;
        for (int c = 0; c < N; ++c) m += x[way][c] / N;
        for (int c = 0; c < N; ++c) {
            double r = f[c] - (singular ? mean : 0.0) - dg[c] * x[way][c];
            for (int s = 0; s < 6; ++s) r += arm(c, s) * x[way][nb[6 * (size_t)c + s]];
            res[way] = std::max(res[way], std::fabs(r));
            fm = std::max(fm, std::fabs(f[c]));
        }
        if (singular)
            for (double& v : x[way]) v -= m;
        for (int c = 0; c < N; ++c) {
            xm = std::max(xm, std::fabs(x[0][c]));
            dist[way] = std::max(dist[way], std::fabs(x[way][c] - x[0][c]));
        }
    }
    const cudaError_t e = cudaGetLastError();
    printf("iters %d %d res %.3e %.3e %.3e dist %.3e %.3e status %s\n", count[0], count[1], res[0] / fm,
           res[1] / fm, res[2] / fm, dist[1] / xm, dist[2] / xm, cudaGetErrorString(e));
    return e == cudaSuccess ? 0 : 1;
}
