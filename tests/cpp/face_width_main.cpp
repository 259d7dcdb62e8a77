// Host-only: the block width of the face-value gradient on a deck's mesh, cells
// in the deck's order (built by tests/test_face_width.py with g++). Prints, for
// FP32 and FP64, the cells per block and its shared memory, then the shared
// memory of every width that may be taken (32 or 24 cells, and fewer in the
// rule's steps).
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
    for (size_t size : {4, 8}) {
        GradTiles t;
        if (build_face_path_tiles(m, size, t).code) return 2;
        std::printf("%d %zu", t.B, t.B ? face_tile_smem(t, m.dim, size) : 0);
        for (int B : {32, 28, 24, 20, 16, 8}) {
            GradTiles c;
            if (B <= (size == 4 ? 32 : 24) && build_grad_tiles(m, B, c).code == 0)
                std::printf(" %d %zu", B, face_tile_smem(c, m.dim, size));
        }
        std::printf("\n");
    }
    return 0;
}
