// m3_scan_forward_noalloc: the forward scan for callers that must not allocate.
//
// Some hosts of this library cannot ask the driver for device memory while they run:
// a serving process that handed the whole GPU to its own arena at start-up and treats
// any later driver allocation as a fault; a latency-bound decode loop for which the
// implicit synchronisation of an allocation is unacceptable; code running inside a
// region where allocation calls are simply not permitted.  m3_scan_forward takes its
// scratch (head-major copies, chunk states) from the stream-ordered pool, which such a
// caller cannot afford.  This entry point runs the same kernels on a fixed block of
// device memory that is part of the library image instead.
//
// The price: every GPU that loads the library holds M3_NOALLOC_SCRATCH_BYTES until the
// process exits, requests needing more are refused, and all calls share the block: those of
// different streams are put one behind the other.
#include <mutex>

#include "m3_internal.h"
#include "m3_rows.cuh"
#include "m3_tc.h"

namespace {

// The scratch itself.  In host code this name is only a handle for the runtime's symbol
// table, never a device address: the address is looked up once per device below.
static __device__ __align__(256) unsigned char g_noalloc_scratch[M3_NOALLOC_SCRATCH_BYTES];

// Device code may name the array directly.  This kernel is never launched; it exists so
// that the array is referenced from device code and stays in the image.
__global__ void k_noalloc_anchor(unsigned char* out) { out[0] = g_noalloc_scratch[0]; }

constexpr int kMaxDevices = 64;
std::mutex g_mu;
char* g_scratch_addr[kMaxDevices] = {nullptr};

// Device address of the scratch on `device`, which must be the current device.
cudaError_t scratch_address(int device, char** out) {
  std::lock_guard<std::mutex> lock(g_mu);
  if (!g_scratch_addr[device]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    g_scratch_addr[device] = static_cast<char*>(p);
  }
  *out = g_scratch_addr[device];
  return cudaSuccess;
}

// Every kernel that a call with this element type may launch, loaded once per device (which must be current): which of
// them a call takes depends on its shape, and a caller warms up with one shape only.
cudaError_t load_kernels_once(int device, int dtype) {
  static bool loaded[kMaxDevices][2] = {};
  std::lock_guard<std::mutex> lock(g_mu);
  bool& done = loaded[device][dtype == M3_BF16 ? 1 : 0];
  if (done) return cudaSuccess;
  cudaError_t e = m3::generic_load(dtype);
  if (e == cudaSuccess) e = m3::rows_load(dtype);
  if (e == cudaSuccess && dtype == M3_BF16) e = m3::tc_load();
  done = e == cudaSuccess;
  return e;
}

// Calls that use the block wait on the device for the one before them: a tensor-core call of one stream must not
// write what a call of another is reading.  Held from before the first launch until the event behind the last one is
// recorded, so that calls of several threads enter one at a time.
struct BlockOrder {
  std::mutex mu;
  cudaEvent_t behind[kMaxDevices] = {};   // the last call's end
};
BlockOrder& block_order() {
  static BlockOrder* o = new BlockOrder;   // (never destroyed: a stream may outlive the statics)
  return *o;
}
class BlockUse {
 public:
  explicit BlockUse(m3_ctx* ctx) : ctx_(ctx), lock_(block_order().mu) {
    cudaEvent_t& ev = block_order().behind[ctx->device];
    if (ev) status = cudaStreamWaitEvent(ctx->stream, ev, 0);
    else status = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
  }
  ~BlockUse() {
    if (status == cudaSuccess) cudaEventRecord(block_order().behind[ctx_->device], ctx_->stream);
  }
  cudaError_t status;

 private:
  m3_ctx* ctx_;
  std::lock_guard<std::mutex> lock_;
};

bool capturing(cudaStream_t st) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cs) == cudaSuccess) return cs != cudaStreamCaptureStatusNone;
  cudaGetLastError();
  return true;
}

// Whether m3_scan_forward will run the tensor-core family (or, asked for it by name, refuse): with a y that is not 16-byte
// aligned it would take another family, and that one's scratch from the pool.
bool tensor_core(const m3_scan_desc& s, const m3_scan_out& out, const m3::Dims& d) {
  return m3::tc_supported(s) && !d.raw && s.path != M3_PATH_GENERIC && (s.path == M3_PATH_TENSOR || m3::tc_aligned(out.y));
}

// One call, with the block's address in `base`; NULL: the block may not be used.
int forward_on(m3_ctx* ctx, const m3_scan_desc* desc, const m3_scan_out* out, m3::Dims d, char* base) {
  // Shapes the tensor-core family serves need no scratch at all when nothing is kept for a backward
  // pass - or, for few long stripes, states at segment boundaries, which go to the block while they fit.
  if (tensor_core(*desc, *out, d)) {
    ctx->fixed_scratch = base;
    ctx->fixed_bytes = base ? M3_NOALLOC_SCRATCH_BYTES : 0;
    ctx->no_scratch = true;
    const int rc = m3_scan_forward(ctx, desc, out, nullptr);
    ctx->no_scratch = false;
    return rc;
  }
  const bool rows = m3::rows_supported(*desc, out->y);
  if (rows) d = m3::rows_dims(d);
  const size_t need = rows ? m3::rows_ws_layout(d, nullptr, nullptr) : m3::generic_ws_layout(d, nullptr, nullptr);
  if (need > (size_t)M3_NOALLOC_SCRATCH_BYTES)
    return m3::fail(ctx, M3_ERR_UNSUPPORTED,
                    "this scan needs %zu bytes of scratch; the built-in block holds %zu - use m3_scan_forward",
                    need, (size_t)M3_NOALLOC_SCRATCH_BYTES);
  // Every scratch region is written in full before it is read (padded rows are stored
  // as zeros, every chunk-state slot is produced by the chunk kernels), so nothing left
  // behind by the previous call needs clearing.
  cudaError_t e;
  if (rows) {
    m3::rows::RowsWs ws;
    m3::rows_ws_layout(d, &ws, base);
    e = m3::rows_forward(ctx->stream, d, *desc, *out, ws, &ctx->launches);
  } else {
    m3::GenericWs ws;
    m3::generic_ws_layout(d, &ws, base);
    e = m3::generic_forward(ctx->stream, d, *desc, *out, ws, &ctx->launches);
  }
  if (e != cudaSuccess) return m3::cuda_fail(ctx, e, "forward on built-in scratch");
  return M3_OK;
}

}  // namespace

extern "C" int m3_scan_forward_noalloc(m3_ctx* ctx, const m3_scan_desc* desc, const m3_scan_out* out) {
  if (!ctx) return M3_ERR_NULL;
  if (!desc || !out) return m3::fail(ctx, M3_ERR_NULL, "descriptor and outputs are required");
  m3::Dims d;
  int rc = m3::make_dims(ctx, *desc, &d);
  if (rc != M3_OK) return rc;
  if (d.T == 0) return m3_scan_forward(ctx, desc, out, nullptr);  // that branch only copies the state
  if (!out->y) return m3::fail(ctx, M3_ERR_NULL, "y is required");
  if (ctx->device < 0 || ctx->device >= kMaxDevices)
    return m3::fail(ctx, M3_ERR_UNSUPPORTED, "device ordinal %d outside the table of %d", ctx->device, kMaxDevices);
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return m3::cuda_fail(ctx, e, "cudaSetDevice");
  char* base = nullptr;
  e = scratch_address(ctx->device, &base);
  if (e != cudaSuccess) return m3::cuda_fail(ctx, e, "cudaGetSymbolAddress");
  e = load_kernels_once(ctx->device, desc->dtype);
  if (e != cudaSuccess) return m3::cuda_fail(ctx, e, "loading kernels");
  if (capturing(ctx->stream)) {
    // A graph's launches cannot be put behind other streams' here.  The tensor-core family runs whole stripes then, which
    // need no scratch; the other families' calls have always shared the block.
    return forward_on(ctx, desc, out, d, tensor_core(*desc, *out, d) ? nullptr : base);
  }
  const BlockUse use(ctx);
  if (use.status != cudaSuccess) return m3::cuda_fail(ctx, use.status, "order of the calls on the built-in scratch");
  return forward_on(ctx, desc, out, d, base);
}
