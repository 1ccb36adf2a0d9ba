/* What the BLAS walks make of a caller's tree (sofren2_gb300/csrc/sftg_walk.h): reads node images
 * (256 B each) of a model of argv[2] meshlets from the file argv[1] and prints a line per node with the
 * child words of its 8 slots, then whether the tree may be expanded ahead of the sequential walk. */
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "sftg_walk.h"

static_assert(sizeof(sftg_bvh_node) == 256, "node image");

int main(int argc, char** argv) {
    if (argc != 3) return 2;
    FILE* f = fopen(argv[1], "rb");
    if (!f) return 3;
    std::vector<sftg_bvh_node> n;
    sftg_bvh_node t;
    while (fread(&t, sizeof(t), 1, f) == 1) n.push_back(t);
    fclose(f);
    for (const sftg_bvh_node& nd : n) {
        for (uint32_t c = 0; c < 8; c++) printf("%u ", sftg_walk_child(&nd, c, (uint32_t)n.size()));
        printf("\n");
    }
    printf("%u\n", sftg_blas_nested(n.data(), (uint32_t)n.size(), (uint32_t)atoi(argv[2])));
    return 0;
}
