// b200fft_c2c_noalloc: a batched C2C transform that allocates no memory.
//
// Who needs it: some callers cannot call cudaMalloc at the point where they
// transform. Typical cases are a host application that hands out all device
// memory itself from a pool fixed at start-up (so an extra library allocation
// can fail or break its accounting), and latency-critical loops that must not
// stall other streams: cudaMalloc and cudaFree may synchronize the device.
// A b200fft handle allocates a stream and a twiddle table, so those callers
// use this entry point instead.
//
// How: the one piece of memory the transform needs besides its input and
// output, the twiddle table, lives in fixed arrays in the library's own device
// image (8191 entries per precision, 192 KiB, held on every device that loads
// the library until the process exits). They hold the table pyramid of 4096
// points, whose levels are the tables of every shorter power of two: one fill
// per device and precision serves all lengths, and a call is one kernel. (A
// fill before every transform made each call two dependent kernels: forward and
// backward of 512 columns of 128 FP32 points 20.5 us; 13.5 us without it.)
//
// Limits and rules for callers:
//  * lengths are powers of two from 2 to 4096 (the arrays' capacity); other
//    lengths are rejected with B200FFT_ERR_UNSUPPORTED before any GPU work;
//  * the first call on a device looks up the arrays' device addresses with
//    cudaGetSymbolAddress (once per device, with that device current), and the
//    first call of a precision fills its table on the caller's stream; make
//    these before any stream capture begins: a captured call is then one kernel
//    (and a wait for the fill where that has not finished). A capture that comes
//    first fills the table inside the captured work, at every replay;
//  * the addresses are kept for the life of the process: calls after
//    cudaDeviceReset on that device are not supported (the module, and with
//    it the arrays, may move);
//  * the transform runs the kernel an Estimate plan of the same shape takes (few
//    FP64 columns of 128, 256 or 1024 points the full tile);
//  * calls on different streams need no ordering among themselves: until the
//    fill has finished, calls on other streams wait for it (on the device).
#include <cuda_runtime.h>

#include <mutex>
#include <string>

#include "../../include/b200fft.h"
#include "fft_common.hpp"
#include "launch.hpp"

namespace b200fft {
void set_error_text(const std::string &msg); // api.cu: text of b200fft_last_error()
}

#define NOALLOC_MAX_LENGTH 4096

// The table pyramids of NOALLOC_MAX_LENGTH points, FP64 and FP32. Host code
// must not pass these names to a kernel: on the host they only stand for the
// symbols. The device addresses come from cudaGetSymbolAddress (device_table
// below).
static __device__ __align__(256) unsigned char g_noalloc_table64[2 * NOALLOC_MAX_LENGTH * 16];
static __device__ __align__(256) unsigned char g_noalloc_table32[2 * NOALLOC_MAX_LENGTH * 8];

namespace {

constexpr int kNoAllocMaxLength = NOALLOC_MAX_LENGTH;
constexpr int kMaxDevices = 64;

// One precision's table on one device.
struct Table {
  void *addr = nullptr;
  bool filled = false;         // the fill has finished on the device
  cudaEvent_t fill = nullptr;  // recorded after the fill until then
  bool in_graph = false;       // a captured graph waits for that event
};
std::mutex g_mu;
Table g_tables[kMaxDevices][2];

int fail(int code, const std::string &msg) {
  b200fft::set_error_text(msg);
  return code;
}

// While another stream of the process captures in global mode (the default),
// event queries are not permitted to threads of the default capture mode and
// would invalidate that capture. The queries below touch no captured work.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// The current device's table of one precision, ready for work that `st` runs
// from now on. *waits: `st` was made to wait for a fill in flight elsewhere.
int device_table(bool f64, cudaStream_t st, bool capturing, void **out, bool *waits) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    return fail(B200FFT_ERR_NO_DEVICE,
                std::string("b200fft_c2c_noalloc: no usable current device: ") +
                    cudaGetErrorString(e));
  std::lock_guard<std::mutex> lk(g_mu);
  Table &t = g_tables[dev][f64 ? 1 : 0];
  if (t.addr == nullptr) {
    void *p = nullptr;
    e = f64 ? cudaGetSymbolAddress(&p, g_noalloc_table64)
            : cudaGetSymbolAddress(&p, g_noalloc_table32);
    if (e != cudaSuccess || p == nullptr)
      return fail(B200FFT_ERR_CUDA,
                  std::string("b200fft_c2c_noalloc: cudaGetSymbolAddress failed: ") +
                      cudaGetErrorString(e));
    t.addr = p;
  }
  *out = t.addr;
  if (t.filled)
    return B200FFT_SUCCESS;
  const RelaxedCapture relaxed;
  if (t.fill != nullptr) { // by an earlier call, perhaps not finished yet
    if (cudaEventQuery(t.fill) == cudaSuccess) {
      t.filled = true;
      if (!t.in_graph)
        cudaEventDestroy(t.fill);
      t.fill = nullptr;
      return B200FFT_SUCCESS;
    }
    cudaGetLastError(); // not ready yet
    // a capture takes the wait as a node of its own, which keeps the event
    e = cudaStreamWaitEvent(st, t.fill, capturing ? cudaEventWaitExternal : cudaEventWaitDefault);
    t.in_graph = t.in_graph || capturing;
    *waits = true;
  } else {
    cudaEvent_t fill = nullptr;
    if (!capturing)
      e = cudaEventCreateWithFlags(&fill, cudaEventDisableTiming);
    if (e == cudaSuccess)
      e = f64 ? b200fft::launch_twiddle_table(static_cast<double2 *>(t.addr), nullptr,
                                              kNoAllocMaxLength, st)
              : b200fft::launch_twiddle_table(nullptr, static_cast<float2 *>(t.addr),
                                              kNoAllocMaxLength, st);
    if (e == cudaSuccess && !capturing)
      e = cudaEventRecord(fill, st);
    if (e == cudaSuccess)
      t.fill = fill; // null in a capture: its replays fill, calls outside do too
    else if (fill != nullptr)
      cudaEventDestroy(fill);
  }
  if (e != cudaSuccess) {
    cudaGetLastError(); // reported here
    return fail(B200FFT_ERR_CUDA,
                std::string("b200fft_c2c_noalloc: twiddle table: ") + cudaGetErrorString(e));
  }
  return B200FFT_SUCCESS;
}

} // namespace

extern "C" int b200fft_c2c_noalloc(int precision, int direction, int length, size_t batch,
                                   ptrdiff_t stride, ptrdiff_t dist, const void *in,
                                   void *out, void *cuda_stream) {
  using namespace b200fft;
  if (precision != B200FFT_F32 && precision != B200FFT_F64)
    return fail(B200FFT_ERR_INVALID_ARG,
                "b200fft_c2c_noalloc: precision must be B200FFT_F32 or B200FFT_F64");
  if (direction != B200FFT_FORWARD && direction != B200FFT_BACKWARD)
    return fail(B200FFT_ERR_INVALID_ARG,
                "b200fft_c2c_noalloc: direction must be B200FFT_FORWARD or B200FFT_BACKWARD");
  if (in == nullptr || out == nullptr || batch < 1 || stride < 1 || dist < 1)
    return fail(B200FFT_ERR_INVALID_ARG,
                "b200fft_c2c_noalloc: null data pointer or batch/stride/dist below 1");
  if (length > kNoAllocMaxLength || !static_pow2_ok(length))
    return fail(B200FFT_ERR_UNSUPPORTED,
                "b200fft_c2c_noalloc: length " + std::to_string(length) +
                    " is not a power of two in [2, " + std::to_string(kNoAllocMaxLength) +
                    "] (the size of its fixed twiddle array)");
  if (batch > (1ull << 40) || stride > (1ll << 44) || dist > (1ll << 44))
    return fail(B200FFT_ERR_RANGE,
                "b200fft_c2c_noalloc: batch/stride/dist exceed the supported range");
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  const bool f64 = precision == B200FFT_F64;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) {
    cudaGetLastError(); // the legacy stream while another stream captures
    cap = cudaStreamCaptureStatusActive;
  }
  const bool capturing = cap != cudaStreamCaptureStatusNone;
  void *table = nullptr;
  bool waits = false;
  const int rc = device_table(f64, st, capturing, &table, &waits);
  if (rc != B200FFT_SUCCESS)
    return rc;
  // level `length` of the pyramid: its table and those of the shorter lengths
  const size_t level = static_cast<size_t>(2 * kNoAllocMaxLength - 2 * length);
  PassArgs a{};
  a.in = in;
  a.out = out;
  a.tw = static_cast<const char *>(table) + level * (f64 ? sizeof(double2) : sizeof(float2));
  a.total = static_cast<long long>(batch);
  a.batch = static_cast<long long>(batch);
  a.idist = a.odist = dist;
  a.istride = a.ostride = stride;
  a.islab = a.oslab = 0;
  a.chained = !capturing && !waits && // as a handle's passes
              2 * a.total * length * (f64 ? 16 : 8) <= kChainedBytes;
  const cudaError_t e = launch_default_c2c(f64, length, dist < stride,
                                           direction == B200FFT_FORWARD, a, st);
  if (e != cudaSuccess)
    return fail(B200FFT_ERR_CUDA,
                std::string("b200fft_c2c_noalloc: transform kernel: ") + cudaGetErrorString(e));
  return B200FFT_SUCCESS;
}
