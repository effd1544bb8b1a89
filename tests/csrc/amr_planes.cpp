// Host execution of the index arithmetic and cell functions that the multi-level CUDA kernels run
// (TEST INFRASTRUCTURE ONLY): every thread of every plane and of the extra planes of listed cells, as
// the launches of mac_amr.cu form them, against the general functions over whole levels.
//
// Built by tests/test_amr_planes.py with g++ (no CUDA involved).
#include <random>

#include "amr_host.cpp"

namespace {

constexpr unsigned kBlock = 256;   // threads of a block of the launches

struct Check {
    double worst = 0.0;   // largest difference over the largest value, of any output
    long missed = 0;      // entries of an output that one side wrote and the other did not
    template <typename T>
    void operator()(const std::vector<T>& got, const std::vector<T>& want, double tol) {
        double top = 0.0, dif = 0.0;
        for (size_t i = 0; i < want.size(); ++i) {
            if ((got[i] != got[i]) != (want[i] != want[i])) {
                ++missed;
                continue;
            }
            if (want[i] != want[i]) continue;
            top = std::max(top, std::fabs((double)want[i]));
            dif = std::max(dif, std::fabs((double)got[i] - (double)want[i]));
        }
        if (top > 0.0) worst = std::max(worst, dif / top / tol);
    }
};

template <typename T>
std::vector<T> noise(long n, std::mt19937_64& g, double lo, double hi) {
    std::uniform_real_distribution<double> d(lo, hi);
    std::vector<T> v((size_t)n);
    for (T& x : v) x = (T)d(g);
    return v;
}

unsigned blocks(long cells) { return (unsigned)((cells + kBlock - 1) / kBlock); }

// f(t, k) for every thread t of `planes` planes of `cells` threads' blocks
template <class F>
void planes(long cells, unsigned count, F f) {
    for (unsigned k = 0; k < count; ++k)
        for (unsigned t = 0; t < blocks(cells) * kBlock; ++t) f(t, k);
}
// f(cell) for the listed cells, through the extra planes
template <class F>
void rest(long cells, const std::vector<int>& list, int n, F f) {
    const long slice = (long)blocks(cells) * kBlock;
    for (long t = 0; t < amr::rest_planes(n, slice) * slice; ++t) {
        const int q = amr::rest_entry(list.data(), n, (unsigned)t);
        if (q >= 0) f(q);
    }
}

// The cell kernels of one level and, for l > 0, its hand-over with the coarser one.
template <typename T>
void cells(const HostExec& E, const HostMl<T>& M, int l, std::mt19937_64& g, Check& check, double tol) {
    const amr::Geo& G = E.geo;
    amr::LevT<T> L = M.L[l];
    std::vector<std::vector<T>> b(3);
    for (int d = 0; d < G.dm; ++d) {
        b[d] = noise<T>(amr::nfaces(L, d), g, 0.5, 2.0);
        L.b[d] = b[d].data();
    }
    std::vector<unsigned char> mask(L.mask, L.mask + amr::ncells(L));
    int near = 0;
    const std::vector<int> list = amr::classify(G.dm, E.L[l], mask, &near);
    amr::LevT<T> K = L;   // as the kernels see the level: with the class bits
    K.mask = mask.data();
    const amr::LevT<T> C = l ? M.L[l - 1] : L;
    const long N = amr::ncells(L), plane = (long)L.ext[0] * L.ext[1];
    const std::vector<T> u = noise<T>(N, g, -1, 1), f = noise<T>(N, g, -1, 1), cu = noise<T>(amr::ncells(C), g, -1, 1);
    const T nan = std::numeric_limits<T>::quiet_NaN();
    const unsigned nz = 2 * ((L.ext[2] + 1) / 2);   // two planes a thread
    const amr::Plane P = amr::plane(L.ext[0], L.ext[1]);
    for (int coarse = 0; coarse <= (l ? 1 : 0); ++coarse) {
        const T* cp = coarse ? cu.data() : nullptr;
        std::vector<T> want((size_t)N, nan), got((size_t)N, nan);
        for (long i = 0; i < N; ++i) amr::defect_cell(G, L, C, i, u.data(), cp, f.data(), want.data());
        planes(plane, nz, [&](unsigned t, unsigned k) {
            amr::Cell c;
            if (!amr::plane_cell(K, P, t, k, c)) return;
            amr::Stencil<T> A;
            amr::load_stencil(G, K, c, u.data(), f.data(), A);
            amr::defect_near(G, K, A, c.q, coarse != 0, got.data());
        });
        rest(plane, list, coarse ? (int)list.size() : near,
             [&](int q) { amr::defect_cell(G, K, C, (long)q, u.data(), cp, f.data(), got.data()); });
        check(got, want, tol);
    }
    const int hw = (L.ext[0] + 1) / 2;
    for (int colour = 0; colour < 2; ++colour) {
        std::vector<T> want = u, got = u;
        for (long i = 0; i < N; ++i) amr::gsrb_cell(G, L, i, colour, want.data(), f.data());
        planes((long)hw * L.ext[1], nz, [&](unsigned t, unsigned k) {
            amr::Cell c;
            if (!amr::colour_plane_cell(K, amr::plane(hw, L.ext[1]), colour, t, k, c)) return;
            amr::Stencil<T> A;
            amr::load_stencil(G, K, c, got.data(), f.data(), A);
            amr::gsrb_near(G, K, A, c.q, got.data());
        });
        rest((long)hw * L.ext[1], list, near,
             [&](int q) { amr::gsrb_cell(G, K, (long)q, colour, got.data(), f.data()); });
        check(got, want, tol);
    }
    if (!l) return;
    std::vector<int> reflux;
    std::vector<amr::Child> cover;
    amr::coarse_lists(G, E.L[l], E.L[l - 1], E.mask[l - 1], reflux, cover);
    for (int coarse = 0; coarse < 2; ++coarse) {
        const T* cp = coarse ? cu.data() : nullptr;
        std::vector<T> want((size_t)amr::ncells(C), 0), got = want;
        amr::LevT<T> CC = C;
        std::vector<std::vector<T>> cb(3);
        for (int d = 0; d < G.dm; ++d) {
            cb[d] = noise<T>(amr::nfaces(C, d), g, 0.5, 2.0);
            CC.b[d] = cb[d].data();
        }
        for (long i = 0; i < amr::ncells(C); ++i) amr::reflux_cell(G, L, CC, i, u.data(), cp, want.data());
        for (int q : reflux) amr::reflux_cell(G, K, CC, (long)q, u.data(), cp, got.data());
        check(got, want, tol);
    }
    std::vector<T> want((size_t)amr::ncells(C), nan), got = want;
    for (long i = 0; i < amr::ncells(C); ++i) amr::restrict_cell(G, L, C, i, u.data(), want.data());
    for (const amr::Child& q : cover) amr::restrict_child(G, K, q, u.data(), got.data());
    check(got, want, tol);
    want.assign((size_t)N, nan);
    got = want;
    for (long i = 0; i < N; ++i) amr::prolong_cell(G, L, C, i, cu.data(), want.data());
    planes(plane, L.ext[2],
           [&](unsigned t, unsigned k) { amr::prolong_plane(G, K, C, P, t, k, cu.data(), got.data()); });
    check(got, want, tol);
}

// The face kernels of one level (FP64) and the copies from and to the level-domain arrays.
void faces(const HostExec& E, int l, std::mt19937_64& g, Check& check, double tol) {
    const amr::Geo& G = E.geo;
    const amr::Lev L = E.L[l], C = l ? E.L[l - 1] : L;
    const long N = amr::ncells(L), plane = (long)L.ext[0] * L.ext[1];
    const double nan = std::numeric_limits<double>::quiet_NaN();
    const std::vector<double> rho = noise<double>(N, g, 0.5, 2), phi = noise<double>(N, g, -1, 1),
                              cphi = noise<double>(amr::ncells(C), g, -1, 1),
                              b0 = noise<double>(L.n[G.va], g, 0.5, 2), b0e = noise<double>(L.n[G.va] + 1, g, 0.5, 2);
    std::vector<std::vector<double>> u(3);
    for (int d = 0; d < G.dm; ++d) {
        const amr::Plane P = amr::face_plane(L, d);
        const long nf = amr::nfaces(L, d), fp = (long)(L.ext[0] + (d == 0)) * (L.ext[1] + (d == 1));
        const unsigned np = L.ext[2] + (d == 2);
        u[d] = noise<double>(nf, g, -1, 1);
        for (int mult = 0; mult < 2; ++mult) {
            std::vector<double> want = u[d], got = u[d];
            for (long i = 0; i < nf; ++i) {
                int f[3];
                amr::face_coords(L, d, i, f);
                const double bb = amr::beta0_of_face(G, d, f, b0.data(), b0e.data());
                want[i] = mult ? want[i] * bb : want[i] / bb;
            }
            planes(fp, np, [&](unsigned t, unsigned k) {
                amr::scale_b0_plane(G, L, d, P, t, k, got.data(), b0.data(), b0e.data(), mult);
            });
            check(got, want, tol);
        }
        const std::vector<double> beta = noise<double>(nf, g, 0.5, 2);
        std::vector<double> want = u[d], got = u[d];
        for (long i = 0; i < nf; ++i)
            amr::correct_face(G, L, C, d, i, phi.data(), l ? cphi.data() : nullptr, beta.data(), want.data());
        planes(fp, np, [&](unsigned t, unsigned k) {
            amr::correct_plane(G, L, C, d, P, t, k, phi.data(), l ? cphi.data() : nullptr, beta.data(), got.data());
        });
        check(got, want, tol);
        want.assign((size_t)nf, nan);
        got = want;
        for (long i = 0; i < nf; ++i)
            amr::coeff_face(G, L, d, i, rho.data(), b0.data(), b0e.data(), 1, want.data());
        planes(fp, np, [&](unsigned t, unsigned k) {
            amr::coeff_plane(G, L, d, P, t, k, rho.data(), b0.data(), b0e.data(), 1, got.data());
        });
        check(got, want, tol);
        planes(fp, np, [&](unsigned t, unsigned k) {
            amr::Face c;
            if (!amr::plane_face(L, d, P, t, k, c)) return;
            int f[3];
            amr::face_coords(L, d, (long)c.q, f);
            if ((long)amr::full_face(L, d, c) != amr::full_face(L, d, (long)c.q) ||
                amr::face_used(G, L, d, c) != amr::face_in_level(G, L, d, f))
                ++check.missed;
        });
        if (!l) continue;
        const long cf = (long)(C.ext[0] + (d == 0)) * (C.ext[1] + (d == 1));
        want = noise<double>(amr::nfaces(C, d), g, -1, 1);
        got = want;
        for (long i = 0; i < amr::nfaces(C, d); ++i) amr::edge_restrict_face(G, L, C, d, i, want.data(), u[d].data());
        planes(cf, C.ext[2] + (d == 2), [&](unsigned t, unsigned k) {
            amr::edge_restrict_plane(G, L, C, d, amr::face_plane(C, d), t, k, got.data(), u[d].data());
        });
        check(got, want, tol);
    }
    const amr::Plane P = amr::plane(L.ext[0], L.ext[1]);
    std::vector<double> want((size_t)N, nan), got = want;
    const double* u2 = G.dm > 2 ? u[2].data() : nullptr;
    for (long i = 0; i < N; ++i) amr::divergence_cell(G, L, i, u[0].data(), u[1].data(), u2, rho.data(), want.data());
    planes(plane, L.ext[2], [&](unsigned t, unsigned k) {
        amr::divergence_plane(G, L, P, t, k, u[0].data(), u[1].data(), u2, rho.data(), got.data());
        amr::Cell c;
        if (amr::plane_cell(L, P, t, k, c) && (long)amr::full_cell(L, c) != amr::full_cell(L, (long)c.q)) ++check.missed;
    });
    check(got, want, tol);
}

}  // namespace

// out[0]: the worst difference over its tolerance (FP64 1e-13, FP32 1e-5 of the largest value);
// out[1]: entries written by one side only, wrong indices.
extern "C" void amrp_check(const orc_opts* o, int nlev, const int* nboxes, const int* boxes, int seed,
                           double* out) {
    HostExec E;
    build(E, o, nlev, nboxes, boxes);
    HostMl<float> M32;
    build_levels<float>(M32, E);
    std::mt19937_64 g(seed);
    Check check;
    for (int l = 0; l < nlev; ++l) {
        cells<double>(E, E, l, g, check, 1e-13);
        cells<float>(E, M32, l, g, check, 1e-5);
        faces(E, l, g, check, 1e-13);
    }
    out[0] = check.worst;
    out[1] = (double)check.missed;
}
