/* Both ray walks (sofren2_gb300/csrc/sftg_ray.cu, its device code in ray_body.inc) on the CPU
 * (warp_sim.h), on a caller's tree.  argv[1]: u32 nodes, root, meshlets, rays, whether the tree is nested
 * (2: as an upload finds); the node images; attr and inds of the meshlets; the rays.  Writes the records of the
 * walk of many rays, then those of a warp per ray, to argv[2].  Built with the address sanitizer: a read
 * outside the tree's arrays ends the program. */
#include "warp_sim.h"
#include <vector>
#include "sftg.h"
#include "sftg_types.h"
#include "sftg_walk.h"
#include "ray_body.inc"
#include "forms_body.inc"

template <class T> static std::vector<T> take(FILE* f, size_t n) {
    std::vector<T> v(n);
    if (fread(v.data(), sizeof(T), n, f) != n) exit(3);
    return v;
}

int main(int argc, char** argv) {
    if (argc != 3) return 2;
    FILE* f = fopen(argv[1], "rb");
    if (!f) return 3;
    const std::vector<uint32_t> hd = take<uint32_t>(f, 5);
    const uint32_t nn = hd[0], nm = hd[2], nr = hd[3];
    const auto nodes = take<sftg_bvh_node>(f, nn);
    const auto attr = take<float>(f, (size_t)nm * 640);
    const auto inds = take<uint8_t>(f, (size_t)nm * 512);
    auto rays = take<sftg_ray>(f, nr);
    fclose(f);
    std::vector<sftg_wslot> slots(nn * 8);
    std::vector<sftg_wtri> tris(nn * 8);
    blockDim.x = 1;
    threadIdx.x = 0;
    for (blockIdx.x = 0; blockIdx.x < nn * 8; blockIdx.x++) k_blas_walk_forms(nodes.data(), nn, attr.data(), inds.data(), nm, slots.data(), tris.data());
    sftg_model M;
    memset(&M, 0, sizeof(M));
    M.total_meshlets = nm; M.blas_count = nn; M.blas_root = hd[1]; M.nested = hd[4] == 2 ? sftg_blas_nested(nodes.data(), nn, nm) : hd[4];
    for (sftg_ray& r : rays) r.model = 0;
    std::vector<sftg_ray_hit> many(nr), few(nr);
    uint32_t next = 0;
    for (unsigned w = 0; w < 2; w++)
        if (const char* e = sim_warp(0, w, 50000000, [&] { k_ray_walks(rays.data(), nr, &M, 1, slots.data(), tris.data(), many.data(), &next); })) {
            printf("many rays, warp %u: %s\n", w, e);
            return 1;
        }
    blockDim.x = 1;
    threadIdx.x = 0;
    for (blockIdx.x = 0; blockIdx.x < nr; blockIdx.x++) k_ray_records(rays.data(), nr, &M, tris.data(), many.data());
    for (uint32_t k = 0; k < nr; k++)
        if (const char* e = sim_warp(k / RAY_WARPS, k % RAY_WARPS, 1000000, [&] { k_ray_wide(rays.data(), nr, &M, 1, slots.data(), tris.data(), few.data()); })) {
            printf("few rays, ray %u: %s\n", k, e);
            return 1;
        }
    f = fopen(argv[2], "wb");
    if (!f) return 3;
    fwrite(many.data(), sizeof(sftg_ray_hit), nr, f);
    fwrite(few.data(), sizeof(sftg_ray_hit), nr, f);
    fclose(f);
    return 0;
}
