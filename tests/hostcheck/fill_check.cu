// CPU build of the ghost fills (csrc/boundary.cuh) for tests/test_fill_model.py:
// the one-pass fill against the passes it stands for, and whether what it reads
// is left alone by the pass itself. Host code of an nvcc build; no GPU needed.
#include <cstring>
#include <vector>

#include "../../dragon_b200/csrc/boundary.cuh"

using namespace dgpu;

namespace {

Geo geo(int dim, const int* n, int g) {
    Geo G{};
    G.dim = dim;
    G.g = g;
    for (int a = 0; a < 3; a++) {
        G.n[a] = a < dim ? n[a] : 1;
        G.ext[a] = a < dim ? n[a] + 2 * g : 1;
    }
    G.pitch = dim > 2 ? G.ext[2] : G.ext[1];
    G.pitch2 = dim > 2 ? (long long)G.ext[1] * G.pitch : 0;
    G.plane = (long long)G.ext[0] * (dim > 2 ? G.pitch2 : G.pitch);
    return G;
}

std::vector<double> noise(long long count, unsigned seed) {
    std::vector<double> v(count);
    unsigned long long s = seed * 2654435761ull + 12345;
    for (double& x : v) {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        x = (double)(s >> 11) * 0x1p-52 - 1.0;
    }
    return v;
}

// Every point outside [0, n) of a padded box with hi layers above.
template <class F>
void for_shell(const Geo& G, const int* n, int hi, bool backwards, F f) {
    const ShellBox b = shell_box(G, n, G.g, hi);
    for (unsigned t = 0; t < b.total; t++) {
        int c[3];
        shell_point(b, backwards ? b.total - 1 - t : t, c);
        f(c);
    }
}

template <bool MHD>
int check(int dim, const int* n, int g, int nent, const int* types, const int* faces, unsigned seed) {
    int nf[3] = {n[0] + 1, n[1] + 1, n[2] + 1};
    const Geo G = geo(dim, n, g), FG = geo(dim, nf, g);
    DirectList list{};
    list.n = nent;
    for (int e = 0; e < nent; e++) {
        list.e[e] = BCEntry{types[e], faces[e], 1, 0, {}};
        for (int f = 0; f < 8; f++) list.e[e].state[f] = 0.1 * (f + 1) + e;
    }
    if (!direct_fill_ok(G, list.e, 0, nent, MHD)) return -1;
    constexpr int NF = MHD ? 8 : 5;
    const std::vector<double> w0 = noise(NF * G.plane, seed), B0 = noise(3 * FG.plane, seed + 1);
    std::vector<double> w = w0, B = B0;
    for (int e = 0; e < nent; e++) {
        for (int a = 0; a < dim; a++) bc_cells_axis<MHD>(G, w.data(), list.e[e], a, 0, 1);
        if (MHD)
            for (int a = 0; a < dim; a++) bc_faces_axis(FG, G.n, B.data(), list.e[e], a, 0, 1);
    }
    // values read from the input (0), and in place in both orders (1, 2): the
    // threads of one launch may see either
    for (int k = 0; k < 3; k++) {
        std::vector<double> v = w0, b = B0;
        const double* src = k == 0 ? w0.data() : v.data();
        const double* bsrc = k == 0 ? B0.data() : b.data();
        for_shell(G, n, g, k == 2, [&](const int* c) {
            Prim<double> q;
            if (direct_cell<MHD>(G, src, list, c, q)) store_prim<MHD>(v.data(), G.plane, gidx(G, c), q);
        });
        if (std::memcmp(v.data(), w.data(), v.size() * 8)) return 1 + k;
        if (!MHD) continue;
        for_shell(FG, n, g + 1, k == 2, [&](const int* c) {
            for (int f = 0; f < 3; f++) {
                double x;
                if (direct_face(FG, bsrc, list, G.n, c, f, x)) b[f * FG.plane + gidx(FG, c)] = x;
            }
        });
        if (std::memcmp(b.data(), B.data(), b.size() * 8)) return 11 + k;
    }
    return 0;
}

}  // namespace

// 0: equal in every order; -1: the list does not take the one pass; else the
// first that differs (1-3 cells, 11-13 face B; read from the input, forwards, backwards).
extern "C" int fill_check(int dim, const int* n, int g, int mhd, int nent, const int* types, const int* faces,
                          unsigned seed) {
    return mhd ? check<true>(dim, n, g, nent, types, faces, seed) : check<false>(dim, n, g, nent, types, faces, seed);
}
