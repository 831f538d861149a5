// gbpt_kernels.h -- device data views and launch wrappers of the sm_103a
// kernels (gbpt_kernels.cu).  Host code only sees plain pointers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "gbpt_math.h"

namespace gb {

// Resident scene (device pointers).
struct DevScene {
    const float4* nodes;     // 5 float4 per 8-wide node
    const float4* tris;      // 3 float4 per triangle (v0|id, e1, e2), leaf order
    const float4* shade;     // 6 float4 per canonical triangle: a|mat, b, c, na, nb, nc
    const float* mats;       // kMaterialFloats per material
    const LightRec* lights;
    int n_lights;
    float overall_power;
    int n_nodes, n_tris;
    // records the BRDF values and light emission are evaluated with: the same
    // as mats / lights, except in a frozen-sampling replay (directions,
    // lobes, pdfs and light picks still come from mats / lights)
    const float* mats_eval;
    const LightRec* lights_eval;
    SkyRec sky;  // the scene's sky light (sky.light = -1 when it has none)
    // textures: 6 texture coordinates per canonical triangle (null when the
    // scene has none; then no ray differentials are kept either)
    const float* texcoord;
    const TexRec* tex;
    int n_tex;
};

// The six 32-bit component words of a curandStateMRG32k3a (s1[3], s2[3]):
// all a uniform draw reads and writes, stored in 24 bytes instead of 48.
struct MrgState {
    uint32_t s1[3], s2[3];
};

// Status bits written by the kernels (never a trap).
enum { ST_STACK_OVERFLOW = 1u, ST_ITER_LIMIT = 2u };

// One scene of a frame (single renders are a frame of one scene; batches
// have many): geometry, camera, shading parameters and its pixel range.
struct SceneRec {
    DevScene S;
    CameraRec cam;
    ShadeParams sp;
    int w, h, n;        // resolution, pixels
    int spp, L, rng_mode;
    uint32_t pixel_base;  // first global pixel of the scene
    uint32_t seed;
    MrgPowers jump;       // MRG32k3a jumps by the 3 L draws of a path
    int n_mats;
    uint32_t grad_base;   // first record-gradient float of the scene (adjoint)
};

// Render modes of a chunk.
enum { MODE_FORWARD = 0, MODE_FROZEN = 1, MODE_ADJOINT = 2 };
constexpr int kAdjPlanes = 5;        // float4s of one adjoint vertex record (adj_sector, adj_tail)
constexpr int kMaxAdjBounces = 16;   // bounces the adjoint records per path
constexpr int kAdjMaxSlots = 1 << 22;  // slots of an adjoint chunk (vertex records: 80 B x bounces each)

constexpr int kMaxRounds = 64;  // path samples per chunk

// Per-slot state of the wavefront: arrays of 32-byte sectors, one entry per
// path slot, each moved by one 256-bit access.  A sector holds what a stage
// reads or writes together, so that no access moves part of a sector (a
// partly written sector costs DRAM a read-modify-write when it leaves the
// L2), and queue order stays close to slot order (paths restart on their own
// slot, queues are filled block by block), so that neighbouring lanes touch
// neighbouring sectors.
//   ray    origin 3, direction 3, path index << 10 | bounce, global pixel
//   path   throughput 3, col_accum 3, pending light sample x, y
//   strm   light/path stream of the path (MrgState), pending z, 0
//   shray  shadow ray: origin 3, direction 3, max_t, scene
// The pending light sample is the contribution of the last vertex's light
// sample; it is added once its shadow ray is known to be free.  `hit` (16
// bytes: beta, gamma, triangle id) and `occl` (1 byte) are what a traced
// extension / shadow ray returns.
struct alignas(32) Sector { uint32_t w[8]; };
constexpr size_t kSlotBytes = 4 * sizeof(Sector) + 16 + 1 + 6 * 4;  // sectors, hit, occl, six queue entries
constexpr size_t kSlotAlign = 256;  // slot counts of an allocation are multiples of this

// Loads and stores of the per-iteration state stream (slot records, samples,
// jitter pool, stream cursors) carry the cache-streaming hint (ld.cs /
// st.cs: lines allocated evict-first in L1 and L2), so that the state
// streaming through every iteration -- several times the L2 -- is evicted
// before the scene's nodes and triangles.  GB_REC_EVICT_FIRST=0 makes them
// plain accesses.
#ifndef GB_REC_EVICT_FIRST
#define GB_REC_EVICT_FIRST 1
#endif
#ifdef __CUDACC__
template <class T>
__device__ __forceinline__ T rec_ld(const T* p) {
#if GB_REC_EVICT_FIRST
    return __ldcs(p);
#else
    return *p;
#endif
}
template <class T>
__device__ __forceinline__ void rec_st(T* p, const T& v) {
#if GB_REC_EVICT_FIRST
    __stcs(p, v);
#else
    *p = v;
#endif
}
#endif

#ifdef __CUDACC__
__device__ __forceinline__ Sector rec_ld(const Sector* p) {
    Sector r;
#if GB_REC_EVICT_FIRST
    asm volatile("ld.global.cs.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
#else
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
#endif
                 : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]), "=r"(r.w[6]),
                   "=r"(r.w[7])
                 : "l"(__cvta_generic_to_global(p))
                 : "memory");
    return r;
}
__device__ __forceinline__ void rec_st(Sector* p, const Sector& r) {
#if GB_REC_EVICT_FIRST
    asm volatile("st.global.cs.v8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
#else
    asm volatile("st.global.v8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
#endif
                 :
                 : "r"(r.w[0]), "r"(r.w[1]), "r"(r.w[2]), "r"(r.w[3]), "r"(r.w[4]), "r"(r.w[5]), "r"(r.w[6]),
                   "r"(r.w[7]), "l"(__cvta_generic_to_global(p))
                 : "memory");
}
#endif

// Wavefront state: per path slot (sectors above) and per global pixel.
struct Frame {
    int ntot;          // pixels of all scenes
    int nslots;        // path slots in flight
    const SceneRec* scenes;  // device array
    int nscenes;
    // per slot (bind_slots): the sectors, what traced rays return, and the queues
    Sector *ray, *path, *strm, *shray;
    float4* hit;         // beta, gamma, triangle id bits (0xffffffff: miss), 0
    uint8_t* occl;       // 1 = the slot's shadow ray was blocked
    uint32_t* q[6];      // extension rays (0 / 1, by iteration), shadow rays (2), ended paths whose light sample
                         // is still pending (3 / 4), finished paths of the adjoint (5)
    float4* rdiff;       // ray differentials of textured frames: 3 planes of nslots
    // per global pixel
    float4* out;       // output_color (moving average)
    MrgState* pristine;  // stream after curand_init(seed, pixel, 0)
    MrgState* cursor;    // light/path stream at the pixel's next chunk
    MrgState* jcursor;   // camera-jitter stream at the pixel's next chunk
    uint32_t* pscene;  // scene of each pixel
    float2* halton;    // Halton light draw of each pixel (null when no scene of the frame uses it)
    float4* samples;   // sample of path l of the chunk (l = round_start[r] + pixel)
    float4* jpool;     // camera jitter of path l of the chunk (rounds from RenderParams::pool_round on)
    MrgState* spool;   // light/path stream state at the start of path l of the chunk (the same rounds)
    // control
    uint32_t* ctr;     // 3 sets of 8 (by iteration % 3), see CTR_*
    uint32_t* path_ctr;  // next path of the chunk to start
    int* iter;         // iteration index of the chunk's slot-pool loop: [0] as k_rays reads it (k_shade moves it
                       // on), [1] as the kernels after it read it (k_rays copies it there); [2] 1 = the loop has stopped
                       // for k_finish
    unsigned long long* stats;  // 0 camera, 1 ext, 2 shadow rays; 3/4 closest, 5/6 shadow node visits / tri tests;
                                // 7 iterations; 8 closest hits (light samples); 16 words
    uint32_t* status;
    // frozen-sampling replay: throughput of the path under the sampling records
    float4* tp0;
    // adjoint: vertex records [bounce][plane][slot], per-pixel loss gradient
    // (already divided by spp), per-block gradient replicas of the record fields
    float4* adj;
    float4* dimg;
    float* grad;
    int grad_stride;   // floats per replica
    int grad_replicas;
};

// Counter set of an iteration: extension rays, shadow rays and pending ended
// paths queued for it, head of its ray queue, finished paths of the adjoint,
// paths started.
enum { CTR_EXT = 0, CTR_SHADOW = 1, CTR_ENDED = 2, CTR_HEAD = 3, CTR_DONE = 4, CTR_STARTED = 5 };

// Points the per-slot arrays of F at `base` (kSlotBytes * cap bytes, cap a
// multiple of kSlotAlign).
inline void bind_slots(Frame& F, unsigned char* base, size_t cap) {
    F.ray = (Sector*)base;
    F.path = F.ray + cap;
    F.strm = F.path + cap;
    F.shray = F.strm + cap;
    F.hit = (float4*)(F.shray + cap);
    for (int k = 0; k < 6; ++k) F.q[k] = (uint32_t*)(F.hit + cap) + (size_t)k * cap;
    F.occl = (uint8_t*)(F.q[5] + cap);
}

// Launch-wide parameters of one chunk.
struct RenderParams {
    int refill;        // refill a warp's lanes once this many are idle (1..32)
    int tri_mode;      // 0: a warp step is a node visit or a triangle test; 1/2: triangle postponing, one / all triangles;
                       // 3: warp-cooperative triangle tests, then a node
    int blocks_per_sm; // resident blocks per SM of the traversal kernels (0 = occupancy limit)
    int sampling_terms; // adjoint: add the derivatives of the sampling decisions (sampling_scores)
    int trav_variant;  // traversal kernels of the default triangle policy: stack entries / threads per
                       // block 0: 32 / 128, 1: 24 / 128, 2: 32 / 64, 3: 24 / 64
    int mode;          // MODE_*
    int textured;      // some scene of the frame has textures (k_shade's texture variant, Frame::rdiff)
    int p0, rounds;    // path samples p0 .. p0+rounds-1
    int pool_round;    // first round of the chunk that k_start does not start whole (rounds: none)
    int more;          // chunks of the frame follow: the pixels' stream cursors move on
    int pad_;          // no hidden padding before the pointers: the words are a graph's key
    int max_iters;     // iteration bound of the chunk's loop
    int finish_max;    // the loop leaves the chunk's last paths to k_finish once at most this many are alive (0: never)
    const float4* nodes;  // the tree of a frame of one scene (null: every lane has its own scene's)
    const float4* tris;
    // L2 window of the traversal launches (GB_NODE_L2_PERSIST, frames of one
    // scene): the scene's node array, accessed as persisting
    const void* l2_nodes;
    unsigned long long l2_nodes_bytes;
    float l2_hit_ratio;  // fraction of the window's accesses that persist
    uint32_t chunk_paths;  // paths of the chunk
    uint32_t round_start[kMaxRounds + 1];  // first path index of each round (prefix sums of N_p)
};

cudaError_t k_launch_trace(const DevScene& S, int n, const float* orig, const float* dir, const float* tmax,
                           float4* hits, uint8_t* occluded, bool any, uint32_t* head, uint32_t* status,
                           cudaStream_t st);
cudaError_t k_launch_frame_init(const Frame& F, bool rng, cudaStream_t st);
cudaError_t k_launch_start(const Frame& F, const RenderParams& P, int nstart, cudaStream_t st);
cudaError_t k_launch_rays(const Frame& F, const RenderParams& P, bool instrument, unsigned long long cond,
                          bool has_cond, cudaStream_t st);
cudaError_t k_launch_shade(const Frame& F, const RenderParams& P, cudaStream_t st);
cudaError_t k_launch_paths(const Frame& F, const RenderParams& P, cudaStream_t st);
cudaError_t k_launch_finish(const Frame& F, const RenderParams& P, cudaStream_t st);
cudaError_t k_launch_regen(const Frame& F, const RenderParams& P, cudaStream_t st);
cudaError_t k_launch_jitter_pool(const Frame& F, const RenderParams& P, cudaStream_t st);
cudaError_t k_launch_combine(const Frame& F, const RenderParams& P, cudaStream_t st);
cudaError_t k_launch_pack_rgb(const float4* src, int n, float* dst, cudaStream_t st);
cudaError_t k_launch_adjoint(const Frame& F, const RenderParams& P, cudaStream_t st);
cudaError_t k_launch_direct(const DevScene& S, const CameraRec& cam, int w, int h, int samples, uint32_t seed,
                            float shadow_offset, v3 background, float* out, uint32_t* status, cudaStream_t st);
cudaError_t k_launch_direct_hybrid(const DevScene& S, const CameraRec& cam, int w, int h, int cam_samples,
                                   int light_samples, uint32_t seed, float shadow_offset, v3 background, float* out,
                                   uint32_t* status, cudaStream_t st);
int k_adjoint_grid();  // blocks of the adjoint, as many as gradient copies
cudaError_t k_launch_dimg_pack(const float* src, int n, float scale, float4* dst, cudaStream_t st);
cudaError_t k_launch_grad_reduce(const float* grad, int replicas, int stride, double* out, cudaStream_t st);
// One scene of a fitting step's loss: its pixels are base .. base + n - 1 of the
// frame (n <= 2^28, at most 1024 scenes).
struct FitLossItem {
    const float* target;
    float* image;  // null: not wanted
    uint32_t base;
    int n;
    float scale;
};
constexpr int kLossBlock = 256, kLossBlocks = 64;  // blocks per scene; partial: kLossBlocks doubles per scene
cudaError_t k_launch_l2_loss(const FitLossItem* items, int n, const float4* img, float4* dimg, double* partial,
                             double* loss, cudaStream_t st);
// Kernel launches of one slot-pool iteration in a render mode.
int k_launches_per_iteration(int mode);
cudaError_t k_launch_mrg_states(uint32_t seed, const uint32_t* sub, int n, int method, uint32_t* out,
                                cudaStream_t st);
cudaError_t k_launch_mrg_pool(int pixel0, int npix, uint32_t seed, int first_update, int num_updates, float* out,
                              cudaStream_t st);
cudaError_t k_launch_nee_stage(const DevScene& S, int n, float shadow_offset, const float* rnd, const float4* hits,
                               float* ray_orig, float* ray_dir, float* max_t, float* psc, cudaStream_t st);
cudaError_t k_launch_shade_stage(const DevScene& S, int n, const ShadeParams& sp, float* ray_orig, float* ray_dir,
                                 float* max_t, const float4* hits, const uint8_t* occl, const float* rnd,
                                 float* tp, float* accum, const float* to_light, const float* psc, int path,
                                 int bounce, cudaStream_t st);

}  // namespace gb
