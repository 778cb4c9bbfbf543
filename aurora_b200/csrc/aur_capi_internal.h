// aur_capi_internal.h — handle layouts and helpers shared by the C-ABI sources.
#pragma once
#include "aurora_b200.h"
#include "aur_kernels.h"
#include <array>
#include <atomic>
#include <map>
#include <mutex>
#include <string>
#include <vector>

struct aur_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    float* kelemen = nullptr;                  // 21 tables x 2048 floats
    bool kel_ready[aur::kAlbedoRefl] = {};
    cudaStream_t work_stream = nullptr;        // non-blocking stream for captured work (wavefront graphs)
    cudaEvent_t ev_order = nullptr;            // orders work_stream after `stream`
    std::map<uint64_t, std::array<int, 3>> wf_batch_tuned;   // autotuned batch configs (pool, block, sort)
    std::map<uint64_t, std::array<int, 3>> wf_scene_tuned;   // autotuned configs by scene signature
    uint32_t* trace_cursors = nullptr;         // kTraceSlots of kCursorWords, for launch_trace_*
    std::atomic<uint64_t> trace_slots{0};      // slots in use, by bit
    std::atomic<int> live{0};                  // BVHs and scenes created on this context and not destroyed
    std::mutex kelemen_mutex;                  // kelemen, kel_ready
    std::mutex wf_mutex;                       // the wavefront engines, work_stream, ev_order and the tuned configurations
};

struct aur_bvh {
    aur_ctx* ctx = nullptr;
    aur::DeviceBvh bvh;
    int* tri_attr = nullptr;                   // device, per original triangle id
    bool owns_attr = false;
    bool owned_by_scene = false;
    // corner normals and uvs per triangle for aur_bvh_intersect: the scene's records for a scene's
    // BVH, else made by aur_bvh_set_shading (owned)
    aur::TriShade* tri = nullptr;
    bool owns_shading = false;
};

struct aur_scene {
    aur_ctx* ctx = nullptr;
    aur_bvh bvh;                               // owned_by_scene = true
    // device buffers
    aur::TriShade* tri = nullptr;
    uint8_t* tri_type = nullptr;
    bool has_uv = false;
    aur::Attr* attrs = nullptr;
    aur::Material* mats = nullptr;
    aur::Light* lights = nullptr;
    aur::Texture* texs = nullptr;
    float* texels = nullptr;
    float* attr_c2o = nullptr;                 // 16 floats per attribute
    // host copies
    std::vector<aur::Material> h_mats;
    std::vector<aur::Light> h_lights;
    std::vector<aur::Texture> h_texs;
    uint32_t ntri = 0, nattr = 0, ntexel_floats = 0;
    aur::Camera cam{};
    bool wf_tuned = false;                     // autotuned wavefront configuration
    int wf_pool = 0, wf_block = 0, wf_sort = 0;
    aur::DevScene dev() const;
};

#define CUDA_TRY(x, where) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) return aur::cuda_fail(e_, where); } while (0)

namespace aur {

aur_status fail(aur_status s, const std::string& msg);
aur_status cuda_fail(cudaError_t e, const char* where);
bool is_device_ptr(const void* p);
// Checks on the device that v[0, n) < bound (device pointer v); synchronises the stream.
cudaError_t indices_below(const uint32_t* v, size_t n, uint32_t bound, bool* ok, cudaStream_t s);
cudaError_t ctx_kelemen_ensure(aur_ctx* ctx, int refl_index);
int kelemen_index(float reflectance);
aur_status bvh_options(const aur_bvh_opts* o, BvhBuildOptions* out);
aur_status render_options(const aur_scene* sc, const aur_render_opts* o, PathParams* p);
aur_status render_wavefront(aur_scene* sc, const aur_render_opts* o, float* film, aur_render_stats* stats);
void wf_release_context(aur_ctx* ctx);   // frees the wavefront engines cached for a context
// Record pass of the adjoint's wavefront form; a vertex record is `stride` float4s:
//   0  radiance collected up to and including the vertex, material (int bits)
//   1  T dD/dtheta of the next-event estimate, 0
//   2  radiance before the vertex's next-event estimate, d ln P(lobe) / d roughness
//   3  (dw/dtheta) / w of the continuation weight, parameter: kind | index << 2 (kind 0: none; the
//      rest of the record is then not written; 1 diffuse colour of material `index`, 2 texel
//      `index`, 3 roughness of material `index`)
//   4, 5 (stride 6) the texels and weights of kind 2
constexpr int kVertexRec = 4;
aur_status wf_record_pass(aur_scene* sc, const PathParams& p, int s0, int nsamples, float4* rec, int stride,
                          float4* lo_raw, uint64_t* launches, unsigned long long* rays);

// Packs the triangles' shading records from device arrays (corner uvs and attributes may be null: 0)
// into a new buffer of the stream's pool.
cudaError_t pack_tri_shade(const float* corner_n, const float* corner_uv, const int* tri_attr, size_t ntri, TriShade** out,
                           cudaStream_t s);
// The material type of every triangle, into a new buffer.
cudaError_t make_tri_type(const int* tri_attr, const Attr* attrs, const Material* mats, uint32_t nmat, size_t ntri,
                          uint8_t** out, cudaStream_t s);

struct DeviceGuard {
    explicit DeviceGuard(int dev);
    ~DeviceGuard();
    int prev_ = 0;
};

// Device memory of one call, from the stream's pool and given back to it in stream order: calls on one
// context from several host threads interleave on its stream and must not share any.
struct DevBuf {
    void* ptr = nullptr;
    cudaStream_t stream = nullptr;
    cudaError_t init(size_t bytes, cudaStream_t s) {
        stream = s;
        const cudaError_t e = cudaMallocAsync(&ptr, bytes ? bytes : 1, s);
        if (e != cudaSuccess) ptr = nullptr;
        return e;
    }
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { if (ptr) cudaFreeAsync(ptr, stream); }
};

// A ray query's place among the context's cursors (ptr null: all are taken). done() gives it back, once the
// query's work is finished and has left it zero; a query that failed keeps it.
constexpr int kTraceSlots = 64;
struct TraceSlot {
    aur_ctx* ctx;
    int slot = -1;
    uint32_t* ptr = nullptr;
    explicit TraceSlot(aur_ctx* c) : ctx(c) {
        uint64_t used = c->trace_slots.load();
        while (~used) {
            const int k = __builtin_ctzll(~used);
            if (c->trace_slots.compare_exchange_weak(used, used | 1ull << k)) {
                slot = k;
                ptr = c->trace_cursors + aur::kCursorWords * k;
                return;
            }
        }
    }
    void done() { if (slot >= 0) ctx->trace_slots.fetch_and(~(1ull << slot)); }
};

struct DevIn {
    const void* ptr = nullptr;
    void* owned = nullptr;
    cudaStream_t stream = nullptr;
    cudaError_t init(const void* p, size_t bytes, size_t align, cudaStream_t s);
    ~DevIn();
};

struct DevOut {
    void* ptr = nullptr;
    void* owned = nullptr;
    void* user = nullptr;
    size_t size = 0;
    bool host = false;
    cudaStream_t stream = nullptr;
    cudaError_t init(void* p, size_t bytes, size_t align, cudaStream_t s);
    cudaError_t finish();
    ~DevOut();
};

}  // namespace aur
