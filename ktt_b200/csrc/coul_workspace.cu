// coul_workspace.cu -- device memory in which one kernel of a call leaves sums for another: the adjoint's FP64
// partials, the partial blocks and counters of the queue and balanced atom splits, the N-body pair form's
// accelerations.
//
// A context keeps one buffer for each of the three and grows it on demand.  The calls of a context may come on
// different streams (the PyTorch binding binds the current one each time), so every use waits for the end of
// the one before it, by an event that the use before it left: the stream's handle would not tell, since a destroyed
// stream's can come back and cudaStreamPerThread is one handle for many.  The event is also the call's end for
// coul_elapsed_ms, so the order costs no second record.  A buffer that grows is given back only after that event.
//
// A call under stream capture gets a buffer of its own: a graph keeps the pointer, so the buffer must neither be
// freed while the graph can be launched nor be written by calls beside it.  The graph holds a user object whose
// end marks the buffer free for a later capture; captured calls that follow one another on one stream share it.
#include <cuda_runtime.h>

#include <atomic>

#include "coul_internal.h"

namespace coul {

struct CaptureBuffer {
    void* mem = nullptr;
    size_t bytes = 0;
    unsigned long long capture = 0;
    cudaStream_t stream = nullptr;         // of the capture, while it lasts
    std::atomic<bool> held{false};         // by a graph
};

namespace {

// While it lives, this thread may allocate and synchronise although another thread is capturing a stream.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

int no_memory(cudaError_t e, const char* what)
{
    cudaGetLastError();
    return set_error(COUL_ERR_OUT_OF_MEMORY, std::string(what) + " workspace: " + cudaGetErrorString(e));
}

int capture_buffer(coul_ctx* ctx, unsigned long long capture, cudaGraph_t graph, size_t need, const char* what, void** mem)
{
    for (const auto& b : ctx->capture_buffers)
        if (b->held && b->capture == capture && b->stream == ctx->stream && b->bytes >= need) {
            *mem = b->mem;
            return COUL_OK;
        }
    std::shared_ptr<CaptureBuffer> buffer;
    for (const auto& b : ctx->capture_buffers)
        if (!b->held && b->bytes >= need && (!buffer || b->bytes < buffer->bytes))
            buffer = b;
    cudaError_t e;
    if (!buffer) {
        const RelaxedCapture relaxed;
        auto& all = ctx->capture_buffers;
        for (size_t i = all.size(); i-- > 0;)
            if (!all[i]->held) {  // too small
                cudaFree(all[i]->mem);
                all.erase(all.begin() + static_cast<std::ptrdiff_t>(i));
            }
        buffer = std::make_shared<CaptureBuffer>();
        if ((e = cudaMalloc(&buffer->mem, need)) != cudaSuccess)
            return no_memory(e, what);
        buffer->bytes = need;
        all.push_back(buffer);
    }
    // the graph's reference; it ends on a thread of the runtime's, without CUDA calls
    auto* reference = new std::shared_ptr<CaptureBuffer>(buffer);
    cudaUserObject_t object = nullptr;
    e = cudaUserObjectCreate(&object, reference, [](void* r) {
        auto* last = static_cast<std::shared_ptr<CaptureBuffer>*>(r);
        (*last)->held = false;
        delete last;
    }, 1, cudaUserObjectNoDestructorSync);
    if (e != cudaSuccess) {
        delete reference;
        return cuda_error(e, "workspace of a captured call");
    }
    buffer->held = true;
    buffer->capture = capture;
    buffer->stream = ctx->stream;
    if ((e = cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove)) != cudaSuccess) {
        cudaUserObjectRelease(object, 1);
        return cuda_error(e, "workspace of a captured call");
    }
    *mem = buffer->mem;
    return COUL_OK;
}

}  // namespace

int workspace_begin(coul_ctx* ctx, WorkspaceKind kind, size_t need, const char* what, void** mem, bool* own)
{
    *own = false;
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long capture = 0;
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamGetCaptureInfo(ctx->stream, &status, &capture, &graph);
    if (e != cudaSuccess)
        return cuda_error(e, "cudaStreamGetCaptureInfo");
    if (status == cudaStreamCaptureStatusActive) {
        *own = true;
        return capture_buffer(ctx, capture, graph, need, what, mem);
    }
    Workspace& ws = ctx->workspaces[kind];
    if (ws.used == nullptr && (e = cudaEventCreate(&ws.used)) != cudaSuccess)
        return cuda_error(e, "workspace event");
    if (need > ws.bytes) {
        const RelaxedCapture relaxed;
        if (ws.recorded && (e = cudaEventSynchronize(ws.used)) != cudaSuccess)
            return cuda_error(e, "workspace's last use");
        ws.recorded = false;
        ws.clean = 0;
        if (ws.mem)
            cudaFree(ws.mem);
        ws.mem = nullptr;
        ws.bytes = 0;
        if ((e = cudaMalloc(&ws.mem, need)) != cudaSuccess)
            return no_memory(e, what);
        ws.bytes = need;
    }
    if (ws.recorded && (e = cudaStreamWaitEvent(ctx->stream, ws.used, 0)) != cudaSuccess)
        return cuda_error(e, "workspace order");
    ctx->open_workspace = &ws;
    *mem = ws.mem;
    return COUL_OK;
}

int workspace_fail(coul_ctx* ctx, int rc)
{
    if (Workspace* ws = ctx->open_workspace) {  // some of the call may be running
        ctx->open_workspace = nullptr;
        ws->clean = 0;
        ws->recorded = cudaEventRecord(ws->used, ctx->stream) == cudaSuccess || ws->recorded;
    }
    return rc;
}

void release_workspaces(coul_ctx* ctx)
{
    for (Workspace& ws : ctx->workspaces) {
        if (ws.recorded)
            cudaEventSynchronize(ws.used);
        if (ws.mem)
            cudaFree(ws.mem);
        if (ws.used)
            cudaEventDestroy(ws.used);
    }
    for (const auto& b : ctx->capture_buffers)
        cudaFree(b->mem);
}

}  // namespace coul
