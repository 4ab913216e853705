// The tiles a handle starts with (default_tiles), for every component count and
// meshes of all sizes: zsme_set_launch takes them.  Prints what a few models get.
#include <cstdio>

#include "prepared_mesh.h"

int main() {
    long checked = 0, bad = 0;
    for (int nq = 1; nq <= 133; ++nq)   // 134 do not leave the face + gather kernel 64 faces either
        for (int faces = 10; faces < 100000000; faces = faces * 5 / 4 + 1) {
            zsme::LaunchConfig lc{128, 128, 128, 128};
            zsme::default_tiles(lc, nq, faces, 148);
            const bool ok = lc.tile_faces >= 64 && lc.tile_faces <= 1024 && lc.prep_lean >= 0 && lc.prep_lean <= 4 &&
                            (size_t)lc.tile_faces * 3 * nq * sizeof(double) <= zsme::kMaxTileSmem;
            if (!ok && !bad) printf("%d components, %d faces: %d\n", nq, faces, lc.tile_faces);
            bad += !ok;
            ++checked;
        }
    for (int nq : {3, 4, 6, 8, 12, 54})
        for (int faces : {1600, 77000, 174000, 3000000}) {
            zsme::LaunchConfig lc{128, 128, 128, 128};
            zsme::default_tiles(lc, nq, faces, 148);
            printf("%d %d %d %d %d\n", nq, faces, lc.tile_faces, lc.fuse_final, lc.prep_lean);
        }
    printf("checked %ld bad %ld\n", checked, bad);
    return bad != 0;
}
