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

#endif
