// coul_internal.h -- state and helpers shared by the translation units behind the C ABI.
#pragma once

#include <cuda_runtime.h>

#include <functional>
#include <memory>
#include <string>
#include <vector>

#include "coul_forward.cuh"
#include "coulktt.h"

struct coul_batch;

constexpr int kHostSlabs = 16;  // slabs of a host-buffer call (at most)

namespace coul {

struct CaptureBuffer;

// A buffer of coul_workspace.cu's.
struct Workspace {
    void* mem = nullptr;
    size_t bytes = 0;
    cudaEvent_t used = nullptr;  // the end of its last use
    bool recorded = false;       // `used` has been recorded since the memory was had
    // The balanced form's counters (at the start of the memory, one per CTA) are known to be zero for
    // this many CTAs (0: unknown).  Its kernel leaves them at zero when it completes, so a following
    // launch of the same grid needs no reset; the queue form's use of the memory, a reallocation or
    // a kernel that failed or timed out clears this.
    int64_t clean = 0;
};

enum WorkspaceKind { kWorkspaceAdjoint, kWorkspaceSplit, kWorkspacePairs, kWorkspaceKinds };

}  // namespace coul

struct coul_ctx {
    int device = 0;
    void* user_context = nullptr;  // the caller's CUcontext (coul_ctx_create_on), else the primary context
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;  // the stream every call of this context is enqueued on
    cudaEvent_t ev_start = nullptr; // bracket the most recent timed call
    cudaEvent_t ev_stop = nullptr;
    cudaEvent_t last_stop = nullptr;  // the last call's end: ev_stop or its workspace's event
    bool have_timing = false;
    bool timing_held = false;       // a call of several launches records the events itself
    // host-buffer calls in slabs (created by the first): every other slab's stream, the copies' stream, the
    // slabs' ends
    cudaStream_t second_stream = nullptr;
    cudaStream_t copy_stream = nullptr;
    cudaEvent_t slab_events[kHostSlabs] = {};
    int* d_status = nullptr;  // device status word written by kernels whose bounded waits expire
    float* d_atoms_cache = nullptr;  // buffers of the host-pointer convenience calls
    size_t atoms_cap = 0;
    float* d_out_cache = nullptr;
    size_t out_cap = 0;
    int sm_count = 0;
    int cc_major = 0;
    int cc_minor = 0;
    std::vector<std::function<void()>> cleanups;  // frees buffers owned by other units (run at destroy)
    coul::Workspace workspaces[coul::kWorkspaceKinds];  // coul_workspace.cu
    coul::Workspace* open_workspace = nullptr;          // that of the call in progress
    std::vector<std::shared_ptr<coul::CaptureBuffer>> capture_buffers;  // of captured calls
    std::vector<coul_batch*> batches;             // live batches (their device resources go with the context)
    struct Occupancy {
        const void* kernel;
        int threads;
        size_t smem;
        int blocks_per_sm;
    };
    std::vector<Occupancy> occupancy_cache;       // persistent forms' resident blocks (coul_capi.cu)
};

namespace coul {

int set_error(int status, const std::string& msg);
int cuda_error(cudaError_t e, const char* what);
int ctx_activate(coul_ctx* ctx);
int ctx_begin_timing(coul_ctx* ctx);
int ctx_end_timing(coul_ctx* ctx);
// `need` bytes for the call in progress, ordered after their last use (coul_workspace.cu).  *own: the call is
// captured and the memory is its graph's alone (nothing is known of its contents).  ctx_end_timing ends the use; a
// call that fails after this returns through workspace_fail.
int workspace_begin(coul_ctx* ctx, WorkspaceKind kind, size_t need, const char* what, void** mem, bool* own);
int workspace_fail(coul_ctx* ctx, int rc);
void release_workspaces(coul_ctx* ctx);
bool aligned16(const void* p);
int validate_tune(const coul_tune* t, int mode, int soa, const VariantEntry** out);
int validate_grid(const coul_grid* g);
// nz: planes of the whole grid, by which a small 3D map's atoms are split over more CTAs (prm.z_base and
// prm.nz bound the slab); 0: one warp runs through all atoms of a tile, as in the batched kernel.
int launch_forward(coul_ctx* ctx, const VariantEntry* v, const FwdParams& prm, int mode, const coul_tune* t, int nz);
// The plain 3D kernel on planes [f.z_base, f.nz) of a map of nz planes, `soft` of 16 reciprocal square roots on
// the FMA pipe (coul_plain.cu).
int launch_plain_3d(coul_ctx* ctx, const FwdParams& f, int nz, int soft);
int queue_split_setup(coul_ctx* ctx, const VariantEntry* v, FwdLaunch& L, const coul_tune* t);
int balanced_split_setup(coul_ctx* ctx, const VariantEntry* v, FwdLaunch& L, const coul_tune* t);
// Releases the device resources of the context's live batches and detaches them (coul_batched.cu);
// their handles stay valid for coul_batch_destroy.  Called by coul_ctx_destroy, context current.
void orphan_batches(coul_ctx* ctx);

}  // namespace coul
