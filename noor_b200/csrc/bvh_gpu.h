// GPU bottom-level BVH builder: the per-mesh trees of BVH::build
// (noor/source/bvh.cpp:88-258) built level by level on the device, with the
// same bytes as the host builder (scene_build.cpp).
#pragma once
#include <cstdint>
#include <memory>
#include <string>
#include <vector>

#include "host_array.h"

namespace nbg {

// The current device's default pool keeps up to 4 GiB that is given back to it,
// for the next build, and for the next context's first frame (1920x1080: 4.1 ms
// where its buffers come from the system, 1.06 from the pool)
void keep_pool();

// one source mesh: its slice of the triangle order, and the boxes of its
// triangles and of their centroids (Model::computeBBoxes)
struct GpuMesh {
    uint32_t start, count;
    float box[6];   // lo xyz, hi xyz
    float cbox[6];  // centroid box
};
struct GpuBvhParams {
    uint32_t num_bins, max_height, min_leaf, max_leaf;
    float Ci, Ct;
};
// one mesh's tree: its first node's index in the scene's node array
struct GpuTree {
    uint32_t first = 0, height = 0, num_inner = 0, num_leaf = 0, max_leaf_tris = 0;
};
// the scene's arrays on the host; they outlive the build
struct GpuInput {
    uint32_t n_tris;
    const uint32_t *vindices, *nindices, *uvindices;  // 3 per source triangle
    const float* vertices;                            // float4
    uint32_t n_vertices;
    const float* normals;  // float4
    uint32_t n_normals;
    const float* uvs;  // float2
    uint32_t n_uvs;
    const uint32_t* material_indices;  // per source triangle
};
struct GpuTailOut {
    nbh::HostArray<float> vertices, normals, uvs;
    nbh::HostArray<uint32_t> wald[3], attr;
};

// One payload's build, its steps in this order.  The scene's arrays go to the
// device once, the triangle boxes and the triangle order never leave it
// between the steps, and two more host threads carry what the steps do not
// wait for: the arrays that only tail() reads go up during boxes() and
// trees(), while the pages of tail()'s output are taken from the system; the
// nodes come down during tail().
class GpuPayload {
public:
    // out outlives the build; its wald and attr hold 4 words per triangle
    GpuPayload(const GpuInput& in, GpuTailOut& out);
    ~GpuPayload();
    GpuPayload(const GpuPayload&) = delete;
    GpuPayload& operator=(const GpuPayload&) = delete;
    // box and cbox of each mesh from its start and count
    int boxes(std::vector<GpuMesh>& meshes, std::string& err);
    // the trees of the meshes, right-child words counted from the scene's
    // first node; lead[i] nodes of other trees stand before tree i (and after
    // tree i - 1's), `others` in all
    int trees(const std::vector<GpuMesh>& meshes, const GpuBvhParams& p, const std::vector<uint32_t>& lead,
              uint32_t others, std::vector<GpuTree>& trees, double* device_ms, std::string& err);
    // starts the copy of the nodes (4 words of lo and 4 of hi each, the other trees' places left
    // undefined) and of the triangle order, done at finish(); after trees()
    // and before tail()
    void download(uint32_t* lo, uint32_t* hi, uint32_t* order);
    // The rest of Model::loadCudaPayload (model.cpp:333-458): vertex
    // de-duplication in BVH order (the first occurrence of a (vertex, normal,
    // uv) index triple gets the next index) and the Wald records and attribute
    // words of each triangle in BVH order.
    int tail(const std::vector<uint32_t>& material_types, double* device_ms, std::string& err);
    int finish(std::string& err);

private:
    struct Impl;
    std::unique_ptr<Impl> I;
};

}  // namespace nbg
