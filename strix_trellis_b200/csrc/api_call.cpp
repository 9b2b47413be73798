// strix_b200_linear_call: strix_gemv / strix_gemm from plain arguments (strix_trellis_b200.h).
//
// The immediate call of a small layer is bound by the host: 30 us per call from Python for a kernel of
// 5 us, spent on two descriptors, a workspace query, a workspace allocation and an extra launch that
// marks its planes empty.  The descriptors are filled in here, and a GEMV without a workspace takes
// a scratch area that the context keeps per stream: launches leave it empty, so none has to reset it.
#include "api_internal.h"

using namespace sapi;

namespace {

// The calling stream's scratch area; null when all are taken.  Areas belong to streams, not to their
// handles: cudaStreamPerThread is another stream in every thread, and the handle of a destroyed
// stream may come back for a new one while the old one's work still runs.  They are there, and empty,
// since the context is: an allocation here would fail, and end the capture, while another thread
// captures in global mode.  The caller holds scratch_lock, and holds it until its launch is enqueued:
// strix_b200_device_status empties the areas between two launches.
cudaError_t stream_scratch(strix_context c, cudaStream_t stream, void** out) {
    *out = nullptr;
    unsigned long long id = 0;
    const cudaError_t found = cudaStreamGetId(stream, &id);
    if (found != cudaSuccess) return found;
    size_t at = 0;
    while (at < c->scratch_used && c->scratch_streams[at] != id) ++at;
    if (at == kScratchStreams) return cudaSuccess;
    if (at == c->scratch_used) c->scratch_streams[c->scratch_used++] = id;
    *out = c->scratch + at * scratch_area_bytes(c);
    return cudaSuccess;
}

void fill_tensor(strix_tensor_desc& t, const strix_b200_tensor& v) {
    t.struct_size = sizeof(t);
    t.abi_version = STRIX_TRELLIS_ABI_VERSION;
    t.data = v.data;
    t.dtype = static_cast<decltype(t.dtype)>(v.dtype);
    t.rank = v.rank;
    const uint64_t size = v.dtype == STRIX_DTYPE_F32 ? 4 : 2, rows = v.rank == 1 ? 1 : v.rows;
    if (v.rank == 1) {
        t.shape[0] = v.width;
        t.strides[0] = v.column_stride;
    } else {
        t.shape[0] = v.rows;
        t.shape[1] = v.width;
        t.strides[0] = v.row_stride;
        t.strides[1] = v.column_stride;
    }
    t.buffer_bytes = rows && v.data ? ((rows - 1) * v.row_stride + v.width) * size : 0;
}

}  // namespace

extern "C" strix_status strix_b200_linear_call(strix_context c, strix_weights w, uint32_t operation, const strix_b200_tensor* x,
                                               const strix_b200_tensor* y, float alpha, float beta, void* workspace,
                                               uint64_t workspace_bytes, void* stream) {
    if (!w || !x || !y || (operation != STRIX_OPERATION_GEMV && operation != STRIX_OPERATION_GEMM)) return STRIX_ERROR_INVALID_ARGUMENT;
    strix_matmul_desc d;
    strix_matmul_desc_init(&d);
    d.weights = w;
    d.alpha = alpha;
    d.beta = beta;
    d.workspace = workspace;
    d.workspace_bytes = workspace_bytes;
    fill_tensor(d.input, *x);
    fill_tensor(d.output, *y);
    strix_stream sd{};
    sd.struct_size = sizeof(sd);
    sd.abi_version = STRIX_TRELLIS_ABI_VERSION;
    sd.hip_stream = stream;
    const bool gemv = operation == STRIX_OPERATION_GEMV;
    if (workspace || workspace_bytes) return submit(c, &d, &sd, gemv);

    strix_status s = context_check(c);
    if (s != STRIX_SUCCESS) return s;
    cudaStream_t cs{};
    s = stream_check(c, &sd, cs);
    if (s != STRIX_SUCCESS) return s;
    View v{};
    s = view_check(c, &d, true, v);
    if (s != STRIX_SUCCESS) return s;
    if ((gemv && v.rows > 8) || (!gemv && d.input.rank != 2)) return STRIX_ERROR_UNSUPPORTED_FORMAT;
    s = storage_check(c, d, v, 0, nullptr, 0);
    if (s != STRIX_SUCCESS || !v.rows) return s;
    if (v.rows > 8) return STRIX_ERROR_INSUFFICIENT_BUFFER;
    // A captured launch replays on whatever stream the graph is launched on: it brings its own scratch.
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(cs, &capturing);
    if (e != cudaSuccess) return cuda_status(e);
    void* scratch = nullptr;
    std::lock_guard<std::mutex> hold(c->scratch_lock);
    if (capturing == cudaStreamCaptureStatusNone) e = stream_scratch(c, cs, &scratch);
    if (e != cudaSuccess) return cuda_status(e);
    if (!scratch) return STRIX_ERROR_INSUFFICIENT_BUFFER;
    return cuda_status(st::launch_gemv(make_call(c, d, v), st::plan_gemv(w->device, v.rows, c->sm_count), scratch,
                                       c->programmatic_launch, cs));
}
