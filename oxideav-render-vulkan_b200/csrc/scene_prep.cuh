// Scene preparation on the device (scene_prep.cu, bvh_build.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "../../include/oxpt.h"

namespace oxd {

// Scratch memory of a scene build: pieces of one block, handed out in order
// and given back all at once. A build used to make some 35 allocations, each
// of which can cost a page-table update (a 4800-triangle sync took 4 to 24 ms,
// most of it there). A request beyond the block is allocated by itself.
// Everything handed out is used on the build's stream, or on the atlas stream
// that the build waits for, before release().
class Arena {
  public:
    // Blocks up to this size stay for the next build of the same owner.
    static constexpr size_t KEEP = 64u << 20;
    ~Arena() { drop(); }
    // Starts a build that needs about `bytes`.
    cudaError_t begin(size_t bytes) {
        release();
        if (bytes <= cap_) return cudaSuccess;
        drop();
        cudaError_t e = cudaMalloc((void**)&base_, bytes);
        if (e != cudaSuccess) base_ = nullptr;
        else cap_ = bytes;
        return e;
    }
    template <class T>
    cudaError_t get(T** p, size_t bytes) {
        const size_t at = (used_ + 255) & ~(size_t)255;
        if (at + bytes <= cap_) {
            *p = reinterpret_cast<T*>(base_ + at);
            used_ = at + bytes;
            return cudaSuccess;
        }
        void* own = nullptr;
        cudaError_t e = cudaMalloc(&own, bytes ? bytes : 1);
        *p = static_cast<T*>(own);
        if (e == cudaSuccess) more_.push_back(own);
        return e;
    }
    // The block's pieces are free again (pieces outside it stay until release).
    void rewind() { used_ = 0; }
    void release() {
        used_ = 0;
        for (void* p : more_) cudaFree(p);
        more_.clear();
    }
    // The end of a build.
    void end() {
        release();
        if (cap_ > KEEP) drop();
    }
    void drop() {
        release();
        if (base_) cudaFree(base_);
        base_ = nullptr;
        cap_ = 0;
    }
    size_t bytes() const { return cap_; }
    Arena() = default;
    Arena(const Arena&) = delete;
    Arena& operator=(const Arena&) = delete;

  private:
    char* base_ = nullptr;
    size_t cap_ = 0, used_ = 0;
    std::vector<void*> more_;
};
namespace bvhb {

// Binned-SAH BVH over n triangles whose positions (9 floats each) are in
// device memory, built on stream st. On success *words (nodes x 8 words)
// and *slots (leaf slot -> triangle, n entries) are pieces of `mem`, as all
// scratch is (scratch_bytes(n) in all). False with *err when an allocation
// or launch fails.
size_t scratch_bytes(uint32_t n);
bool build_on_device(const float* pos, uint32_t n, cudaStream_t st, Arena* mem, uint32_t** words, uint32_t** slots,
                     uint32_t* nodes, uint32_t* depth, uint32_t* launches, std::string* err);

}  // namespace bvhb

// Four-wide any-hit tree collapsed on the device from binary node words in
// device memory (bvh4_build.cu): the host collapse's words (host/bvh4.cpp),
// node for node. BUILT: *out holds n4 x 32 words (the caller's buffer of
// *out_cap bytes when large enough, else a new cudaMalloc that replaces
// it; untouched when the root is a leaf; with room for more_per_node bytes a
// node and `more` behind the nodes), *root_ref and *need are set. REFUSED: the host collapse
// refuses the tree too (keep the binary walk). UNSUPPORTED: deeper than
// 64 four-wide levels (collapse on the host). FAILED: a CUDA error. Scratch
// comes from `mem`, or is stream-ordered (cudaMallocAsync) without it.
enum class Collapse { BUILT, REFUSED, UNSUPPORTED, FAILED };
Collapse collapse4_device(const uint32_t* words, uint32_t nodes, cudaStream_t st, uint32_t** out, size_t* out_cap,
                          uint32_t* n4,
                          uint32_t* root_ref, uint32_t* need, std::string* err, size_t more_per_node = 0,
                          size_t more = 0, Arena* mem = nullptr);
// Levels of the binary tree (65 when deeper than 64 or malformed), as the
// host's depth walk counts them.
bool binary_depth_device(const uint32_t* words, uint32_t nodes, cudaStream_t st, uint32_t* depth, std::string* err);
// The four-wide nodes with 8-bit child boxes, 16 words each: lower corner and
// step per axis, a byte per child and plane, the child references. `words`:
// the binary nodes.
cudaError_t launch_wide_nodes(const uint32_t* words, const uint4* bvh4, uint32_t n4, uint32_t* out, cudaStream_t st);
// map[slot] = the binary leaf node that holds the slot, for every slot below
// `slots` (0 for a slot in no leaf).
cudaError_t launch_leaf_map(const uint32_t* words, uint32_t nodes, uint32_t* map, uint32_t slots, cudaStream_t st);
// *outside = 1 when some leaf's triangle has a vertex outside the leaf's box,
// else 0; `count`: words of the nodes and the triangles behind them.
cudaError_t launch_leaf_contents(const uint32_t* words, uint32_t nodes, uint64_t count, uint32_t* outside,
                                 cudaStream_t st);

namespace prep {

// Device buffers of one prepared scene, owned by the caller before and
// afterwards: a build writes into those it is given when they are large
// enough (and not more than twice too large) and replaces the others.
struct DeviceScene {
    float4* geom = nullptr;   // nodes, then triangles in leaf-slot order
    size_t geom_vec4 = 0, geom_cap = 0;
    float4* attrs = nullptr;  // 12 float4 per slot
    size_t slot_count = 0, attrs_cap = 0;
    uint2* atlas = nullptr;   // side x side x layers RGBA16F texels
    size_t atlas_cap = 0;
    uint32_t node_count = 0, depth = 0;

    // Device time of the phases (CUDA events): source upload, BVH, slot
    // flattening, atlas (texel upload + mip chains, on its own stream).
    float phase_ms[4] = {0, 0, 0, 0};
    uint32_t launches = 0;  // kernels this build launched
};

// Builds every buffer of `src` on st (oxpt_build_scene), with scratch from
// `mem`. Nothing may still read the buffers given in *out. On failure *out
// holds whatever buffers exist, without a scene in them, and *err says why.
oxpt_status build_scene(const oxpt_scene_src& src, cudaStream_t st, Arena* mem, DeviceScene* out,
                        uint32_t* light_slots, std::string* err);

}  // namespace prep
}  // namespace oxd
