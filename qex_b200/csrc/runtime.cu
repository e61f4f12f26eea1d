// runtime.cu -- error reporting, device selection, stream and the reduction
// scratch of the kernels that end in a grid-wide sum.
#include <atomic>
#include <cstdio>
#include <mutex>
#include <new>
#include <string>

#include "internal.cuh"

namespace qs {

void noalloc_forget(int dev);  // noalloc.cu

namespace {
thread_local std::string g_last_error = "no error";
thread_local cudaStream_t g_stream = nullptr;
thread_local long long g_launches = 0;

// One thread's scratch on one device.  A sum may be left in it by one kernel for
// the next, and its pinned half carries states to and from the device, so two
// threads that solve at the same time, on one stream or on two, need one each.
struct Scratch {
  double *partials = nullptr;
  double *results = nullptr;  // kNumResults doubles
  unsigned *tickets = nullptr;
  double *host_results = nullptr;  // pinned, kNumResults doubles
};
// 264 KB for each thread, allocated one by one: they share the allocator's 2 MB
// block with the small buffers of handles (with four or eight at a time the
// links of an 8^3 x 16 lattice took 2.15 ms to make, now 1.80 as before)
constexpr size_t kScratchDoubles = (size_t)kMaxRedBlocks * 8 + kNumResults + kNumTickets;

struct DeviceRuntime {
  bool ready = false;
  int sms = 148;
  std::atomic<unsigned> epoch{0};  // qexstag_finalize calls: older scratch is gone
  std::vector<Scratch> all, idle;
};
constexpr int kMaxDevices = 64;
// never destroyed: a thread may end after the process's static objects
DeviceRuntime *const g_dev = new DeviceRuntime[kMaxDevices];
std::mutex &g_mutex = *new std::mutex;

// what this thread holds, given back when it ends
struct Held {
  struct One {
    Scratch s;
    unsigned epoch = 0;
    bool have = false;
  } of[kMaxDevices];
  ~Held() {
    std::lock_guard<std::mutex> lock(g_mutex);
    for (int d = 0; d < kMaxDevices; d++)
      if (of[d].have && of[d].epoch == g_dev[d].epoch) g_dev[d].idle.push_back(of[d].s);
  }
};
thread_local Held g_held;

int current_device() {
  int d = 0;
  cudaGetDevice(&d);
  return d;
}

// scratch for one more thread on the current device, tickets zero
int add_scratch(DeviceRuntime &r) {
  Scratch c;
  cudaStream_t s = nullptr;
  cudaError_t e = device_malloc(&c.partials, sizeof(double) * kScratchDoubles);
  if (e == cudaSuccess) e = cudaHostAlloc(&c.host_results, sizeof(double) * kNumResults, cudaHostAllocDefault);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMemsetAsync(c.partials, 0, sizeof(double) * kScratchDoubles, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (s) cudaStreamDestroy(s);
  if (e != cudaSuccess) {
    cudaGetLastError();
    if (c.host_results) cudaFreeHost(c.host_results);
    if (c.partials) cudaFree(c.partials);
    if (e == cudaErrorMemoryAllocation) return fail(QEXSTAG_ERR_ALLOC, "reduction scratch: allocation failed");
    return cuda_fail(e, "reduction scratch");
  }
  c.results = c.partials + (size_t)kMaxRedBlocks * 8;
  c.tickets = (unsigned *)(c.results + kNumResults);
  r.all.push_back(c);
  r.idle.reserve(r.all.size());
  r.idle.push_back(c);
  return QEXSTAG_OK;
}

// this thread's scratch on device d, which is current
int scratch_of(int d, Scratch **out) {
  if (d < 0 || d >= kMaxDevices) return fail(QEXSTAG_ERR_ARG, "device index out of range");
  Held::One &h = g_held.of[d];
  DeviceRuntime &r = g_dev[d];
  *out = &h.s;
  if (h.have && h.epoch == r.epoch) return QEXSTAG_OK;
  std::lock_guard<std::mutex> lock(g_mutex);
  if (!r.ready) {
    cudaDeviceProp prop;
    QS_CUDA(cudaGetDeviceProperties(&prop, d));
    r.sms = prop.multiProcessorCount;
  }
  if (r.idle.empty()) {
    // the thread may be capturing a graph on its stream: the allocation is no part of it
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    const int rc = add_scratch(r);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (rc) return rc;
  }
  h.s = r.idle.back();
  r.idle.pop_back();
  h.epoch = r.epoch;
  h.have = true;
  r.ready = true;
  return QEXSTAG_OK;
}

// (entry points have called runtime_ready, so the scratch is there)
Scratch scratch() {
  Scratch *s;
  return scratch_of(current_device(), &s) == QEXSTAG_OK ? *s : Scratch();
}
}  // namespace

void set_error(const std::string &msg) { g_last_error = msg; }
void note_launch(int n) { g_launches += n; }
long long launch_count() { return g_launches; }

int fail(int code, const std::string &msg) {
  g_last_error = msg;
  return code;
}

int cuda_fail(cudaError_t e, const char *what) {
  g_last_error = std::string("CUDA error in ") + what + ": " + cudaGetErrorString(e);
  return QEXSTAG_ERR_CUDA;
}

cudaStream_t stream() { return g_stream; }

int num_sms() { return g_dev[current_device()].sms; }

double *red_partials() { return scratch().partials; }
unsigned *red_tickets() { return scratch().tickets; }
double *red_results() { return scratch().results; }
double *host_results() { return scratch().host_results; }

int runtime_ready() {
  Scratch *s;
  return scratch_of(current_device(), &s);
}

}  // namespace qs

extern "C" {

int qexstag_init(int device) {
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess) return qs::cuda_fail(e, "cudaGetDeviceCount");
  if (device < 0 || device >= n) return qs::fail(QEXSTAG_ERR_ARG, "qexstag_init: no such device");
  e = cudaSetDevice(device);
  if (e != cudaSuccess) return qs::cuda_fail(e, "cudaSetDevice");
  return qs::runtime_ready();
}

int qexstag_finalize(void) {
  int d = qs::current_device();
  qs::noalloc_forget(d);
  std::lock_guard<std::mutex> lock(qs::g_mutex);
  qs::DeviceRuntime &r = qs::g_dev[d];
  if (!r.ready) return QEXSTAG_OK;
  cudaDeviceSynchronize();
  for (const qs::Scratch &c : r.all) {
    cudaFree(c.partials);
    cudaFreeHost(c.host_results);
  }
  r.all.clear();
  r.idle.clear();
  r.epoch++;
  r.ready = false;
  return QEXSTAG_OK;
}

int qexstag_set_stream(void *s) {
  qs::g_stream = (cudaStream_t)s;
  return QEXSTAG_OK;
}

const char *qexstag_last_error(void) { return qs::g_last_error.c_str(); }

int qexstag_synchronize(void) {
  QS_CUDA(cudaStreamSynchronize(qs::g_stream));
  return QEXSTAG_OK;
}

}  // extern "C"
