// Host-only check of the global face list (built by tests/test_face_pairs.py
// with g++ from the library's host sources): reads a deck directory, builds
// the flattened mesh and prints whether its faces are paired and the largest
// distance of a cell face's centre from the mean of its own vertices,
// relative to the face's own size.
#include <algorithm>
#include <cmath>
#include <cstdio>

#include "gbte_internal.h"

using namespace gbte;

int main(int argc, char **argv) {
    Deck D;
    if (argc < 2 || read_deck(argv[1], D).code) return 2;
    D.bands.kappa.assign(D.bands.nmat, 1.0);
    D.bands.capb.assign(D.bands.nmat, 1.0);
    FlatMesh m;
    if (build_flat_mesh(D.mesh, D.bcs, D.bands, m).code) return 2;
    double worst = 0;
    for (int k = 0; k < m.ncf(); k++) {
        double x = 0, y = 0, z = 0;
        for (int t = 0; t < m.dim; t++) {
            const int v = m.cf_v[3 * k + t];
            x += m.node_x[v] / m.dim, y += m.node_y[v] / m.dim, z += m.node_z[v] / m.dim;
        }
        const double size = m.dim == 2 ? m.cf_area[k] : std::sqrt(m.cf_area[k]);
        worst = std::max(worst, std::hypot(m.cf_fx[k] - x, std::hypot(m.cf_fy[k] - y, m.cf_fz[k] - z)) / size);
    }
    std::printf("paired %d centre_error %.3e faces %d\n", m.faces_paired ? 1 : 0, worst, m.nf());
    return 0;
}
