/*
 * What the BLAS walks rely on in a tree, for the host and the device: a caller's tree is uploaded as
 * it is, and a node or meshlet index outside the model has to end the walk that meets it, not to be read.
 */
#ifndef SFTG_WALK_H
#define SFTG_WALK_H

#include "sftg_types.h"

#ifdef __CUDACC__
#define SFTG_WALK_HD __host__ __device__ __forceinline__
#else
#define SFTG_WALK_HD static inline
#endif

/* On the stack of k_ray_wide: a triangle's place, not a node.  Node ids stay below it. */
#define SFTG_WALK_TRI 0x80000000u

/* Child word of slot c as the walks' forms hold it: an inner node's child outside the `count` nodes
 * becomes an id that is outside them too (below 2^31) and never reads as a triangle's place. */
SFTG_WALK_HD uint32_t sftg_walk_child(const sftg_bvh_node* nd, uint32_t c, uint32_t count) {
    const uint32_t ch = nd->child[c];
    return nd->leaf || ch == SFTG_INVALID || ch < count ? ch : SFTG_WALK_TRI - 1u;
}

/* Whether every node's boxes lie inside the box its parent holds for it and every slot's child is a node
 * of the tree or a triangle of the model's `meshlets` (sftg_model.nested): true of a tree built from its
 * triangles, not checked by the loaders of caller-built ones.  Only such a tree is expanded ahead of the
 * sequential walk: of another, what that walk would have skipped may be nearer than its parent, or
 * end the walk. */
static inline uint32_t sftg_blas_nested(const sftg_bvh_node* nodes, uint32_t count, uint32_t meshlets) {
    for (uint32_t i = 0; i < count; i++) {
        for (uint32_t c = 0; c < nodes[i].count && c < 8; c++) {
            const uint32_t ch = nodes[i].child[c];
            if (ch == SFTG_INVALID) continue;
            if (nodes[i].leaf) {
                if ((ch & ~SFTG_WALK_TRI) >> 7 >= meshlets) return 0;
                continue;
            }
            if (ch >= count) return 0;
            for (uint32_t q = 0; q < nodes[ch].count && q < 8; q++)
                for (int a = 0; a < 3; a++)
                    if (!(nodes[ch].mn[a][q] >= nodes[i].mn[a][c] && nodes[ch].mx[a][q] <= nodes[i].mx[a][c])) return 0;
        }
    }
    return 1;
}

#endif
