// aur_bvh.cuh — BVH layout shared by the device build and the traversal kernels.
//
// Replaces Embree's "bvh4.spatialsplit"/"triangle4" accelerator
// (Aurora/src/geometry/embreeAccelerator.cpp:19-35). Binary BVH, one 64-byte
// record per interior node holding BOTH children's boxes (so a node visit is
// four coalesced 128-bit loads and two slab tests):
//   a = (c0.lo.x, c0.hi.x, c0.lo.y, c0.hi.y)
//   b = (c1.lo.x, c1.hi.x, c1.lo.y, c1.hi.y)
//   c = (c0.lo.z, c0.hi.z, c1.lo.z, c1.hi.z)
//   d = (ref0, ref1, count0, count1)   ref >= 0: interior node index;
//        ref < 0: leaf; ~ref = start << 5 | count, triangles [start, start+count)
//        (so a leaf holds at most 31 triangles and a BVH at most 2^26 triangles)
// Triangles are stored in leaf order, 48 bytes each, as the exact inputs of the
// Moller-Trumbore test: (p1, prim id bits), (e1 = p2-p1, 0), (e2 = p3-p1, 0).
// Child boxes are padded outward by 2^-19 of their magnitude so that FP32
// rounding in the slab test can never cull a triangle the exact test accepts.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace aur {

struct BvhNode { float4 a, b, c, d; };
struct BvhTri { float4 p1, e1, e2; };

// 4-wide node (128 bytes, one cache line) collapsed from the binary tree: the
// four children's boxes as structure of arrays (lox = the four children's lo.x,
// ...) and their refs in the binary tree's encoding (>= 0: 4-wide node index;
// < 0: leaf ~(start << 5 | count)). The boxes are the binary tree's padded child
// boxes, bit for bit. Unused slots have +inf boxes (never entered) and ref ~0 (an
// empty leaf).
struct BvhNode4 { float4 lox, hix, loy, hiy, loz, hiz; int4 ref; int4 pad; };

// The 4-wide node with quantised boxes (64 bytes): the four children's planes as one byte each
// on the node's own grid, rounded outward. Byte q of an axis is the plane p + s (1 + q 2^-15): p
// lies one s below the grid's origin and s is 2^15 cells, so that the byte placed in a float's
// mantissa (1 + q 2^-15) decodes with a single FMA. Same children and refs as the full-precision
// node, at the same index; unused slots have an inverted box (255, 0) and ref ~0.
// Its boxes contain the full-precision ones, so the traversals find the same hits; only the
// visiting order differs, which decides a hit's identity where two triangles lie at exactly the
// same distance. Such ties are detected and traced again over the full-precision nodes. (Any form's order
// also decides for a ray that grazes an edge so flatly that a triangle's computed distance is off by more
// than the boxes' slack: found first, the other triangle hides it. Of 524,288 rays towards a bumpy sheet, a
// quarter of them at its vertices and half grazing, 3 to 30 differ between the forms of the ray queries.)
// The padding covers origins within some sixteen scene magnitudes in both forms' terms but one: the
// distance to the grid's origin is rounded once more here, which leaves about eleven. Of 13 million
// such rays from half to 128 magnitudes away none lost a hit to the quantised boxes (any hit gains some that the
// tighter boxes lose); from 1,024 on both forms lose hits, and not the same.
struct __align__(64) BvhNode4Q {
    float p[3], s[3];
    uint32_t lox, hix, loy, hiy, loz, hiz;
    int ref[4];
};

struct DeviceBvh {
    BvhNode* nodes = nullptr;     // num_nodes records, root at 0
    BvhTri* tris = nullptr;       // num_tris records in leaf order
    int num_nodes = 0;
    int num_tris = 0;
    int depth = 0;                // longest root-to-leaf path (interior levels + 1)
    float lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};   // scene bounds
    BvhNode4* nodes4 = nullptr;   // the 4-wide form, root at 0 (same triangles)
    BvhNode4Q* nodes4q = nullptr; // the same with quantised boxes
    int num_nodes4 = 0;
    int depth4 = 0;               // 4-wide levels on the longest path
};

// From this many 4-wide nodes on, closest-hit and any-hit rays traverse the quantised nodes; below
// it the full-precision ones, which then sit in the L1, where their requests are cheap and the
// byte decoding is not. Measured on the 512 x 512, 64 sample sphere frame with 644 / 5,444 /
// 20,804 / 82,244 triangles (about a third as many nodes), closest hit full vs quantised: 2.34
// vs 2.60, 3.35 vs 3.57, 3.89 vs 4.05, 4.55 vs 4.56 ms; on the 3.4 M triangle terrain 106.8 vs
// 95.9. Any hit: 1.67 vs 1.62, 2.23 vs 2.10, 2.57 vs 2.38, 3.04 vs 2.75 ms; terrain 54.8 vs 44.2;
// 344 triangles 1.38 vs 1.37; a batch of 36-triangle boxes 5.65 vs 5.81 ms.
constexpr int kQuantMinNodes4 = 1 << 15;
constexpr int kQuantMinNodes4Any = 1 << 7;

struct BvhBuildOptions {
    int max_leaf = 4;             // triangles per leaf at most (<= 31)
    float cost_traverse = 1.0f;   // SAH node-visit cost
    float cost_intersect = 1.0f;  // SAH triangle-test cost
    int ploc_radius = 16;         // PLOC nearest-neighbour search radius
};

// Builds into freshly allocated device buffers (cudaMallocAsync on `stream`), the 4-wide forms
// included (left null where the tree is too deep for any of their stacks). verts: device
// float3[nvert]; idx: device uint32[3*ntri]. Returns cudaSuccess or the first CUDA error; what was
// allocated until then is the caller's to free. *in_range = false, and nothing is built, when an
// index is not below nvert. ntri must be >= 1. Synchronises the stream.
cudaError_t bvh_build_device(const float* verts, const uint32_t* idx, int ntri, uint32_t nvert, const BvhBuildOptions& opt,
                             DeviceBvh* out, bool* in_range, cudaStream_t stream);
void bvh_free_device(DeviceBvh* bvh, cudaStream_t stream);

}  // namespace aur
