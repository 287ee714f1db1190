// Library runtime shared by every kernel unit: thread-local error message, device query, programmatic-dependent-launch
// switches, version string.  Kept apart from the dispatchers so that a library linked from a subset of the units loads.
#include <stdarg.h>
#include <stdlib.h>

#include <atomic>
#include <mutex>

#include "common.cuh"
#include "tc_ptx.cuh"

namespace b200p {

static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

int cuda_fail(cudaError_t e, const char* what) {
  set_error("%s: %s", what, cudaGetErrorString(e));
  return B200P_ERR_CUDA;
}

// 0 off, 1 every kernel, 2 the GEMMs and the classes of g_pdl_mask (B200P_PDL overrides the default at load time)
static int g_pdl = [] { const char* e = getenv("B200P_PDL"); return e ? atoi(e) : 2; }();
static int g_sm_count = -1;
static int g_cc_major = -1;

static int query_device() {
  if (g_cc_major >= 0) return B200P_OK;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  cudaDeviceProp p;
  e = cudaGetDeviceProperties(&p, dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDeviceProperties");
  g_cc_major = p.major;
  g_sm_count = p.multiProcessorCount;
  return B200P_OK;
}

// per-class PDL mask for the non-GEMM kernels (see common.cuh).  Attention by default: its launch and set-up hide behind rope and append, and its
// reduction behind it (us, off / on: decode steps 16 x 8192 77.3 / 75.0, prompts 4 x 777 61.9 / 59.4, decode step of one sequence 257.5 / 252.7);
// rope as well gives nothing more in captured steps (255.1).  Which sizes of decode attention are launched plainly all the same: attn_decode.cu.
static int g_pdl_mask = [] { const char* e = getenv("B200P_PDL_MASK"); return e ? atoi(e) : 8; }();
static thread_local int g_pdl_class = 0;
void pdl_set_class(int cls) { g_pdl_class = cls; }
bool pdl_enabled() { return g_pdl == 1 || (g_pdl != 0 && (g_pdl_mask & g_pdl_class) != 0); }
bool pdl_enabled_gemm() { return g_pdl != 0; }
bool pdl_chained() { return g_pdl != 0 && g_pdl_class == 128; }

int sm_count() {
  query_device();
  return g_sm_count > 0 ? g_sm_count : 148;
}

static std::atomic<int*> g_wait_words{nullptr};      // [WAIT_KINDS], kept until the process exits: captured graphs hold the address
static std::mutex g_wait_mutex;

static int wait_words(int** words) {
  if ((*words = g_wait_words.load(std::memory_order_acquire))) return B200P_OK;
  std::lock_guard<std::mutex> lk(g_wait_mutex);
  if (!g_wait_words.load(std::memory_order_relaxed)) {
    // the first launch may be part of a stream capture, which this allocation has nothing to do with
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    void* p = nullptr;
    cudaError_t e = cudaHostAlloc(&p, WAIT_KINDS * sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) return cuda_fail(e, "cudaHostAlloc(wait words)");
    memset(p, 0, WAIT_KINDS * sizeof(int));
    g_wait_words.store((int*)p, std::memory_order_release);
  }
  *words = g_wait_words.load(std::memory_order_relaxed);
  return B200P_OK;
}

static int wait_pending(const int* words) {
  for (int k = 0; k < WAIT_KINDS; ++k) {
    const int v = reinterpret_cast<const volatile int*>(words)[k];
    if (v) return 256 * (k + 1) + v;
  }
  return 0;
}

int wait_word(WaitKind kind, int** word) {
  int* words;
  const int rc = wait_words(&words);
  if (rc) return rc;
  const int v = wait_pending(words);
  B200P_REQUIRE(v == 0, B200P_ERR_TIMEOUT, "a bounded wait of an earlier launch gave up (kernel %d, role %d): outputs since then are incomplete",
                v / 256, v % 256);
  *word = words + kind;
  return B200P_OK;
}

int wait_take(WaitKind kind) {
  if (cudaDeviceSynchronize() != cudaSuccess) return -1;
  int* words = g_wait_words.load(std::memory_order_acquire);
  if (!words) return 0;
  volatile int* w = words + kind;
  const int v = *w;
  *w = 0;
  return v;
}

// One warp waits for an arrival that nothing makes; TMA, TMEM and copies have no part in it.
__global__ void wait_probe_kernel(int* word, long long cycles) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar), 1);
    fence_barrier_init();
  }
  __syncwarp();
  mbar_wait_warp(smem_u32(&bar), 0, nullptr, word, 0, cycles);
}

}  // namespace b200p

using namespace b200p;

extern "C" int b200p_wait_fault(void) {
  const int* words = g_wait_words.load(std::memory_order_acquire);
  return words ? wait_pending(words) : 0;
}

extern "C" int b200p_wait_probe(void* stream) {
  int* words;
  const int rc = wait_words(&words);
  if (rc) return rc;
  wait_probe_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(words + WAIT_QMV_RING, 1000000ll);
  B200P_LAUNCH_CHECK("wait_probe_kernel");
  return B200P_OK;
}

// 0.3: dense GEMM, ragged batches, gated delta rule and latent attention entry points added to the 0.2 ABI
extern "C" const char* b200p_version(void) { return "b200parallm 0.3 (sm_100a)"; }
extern "C" const char* b200p_last_error(void) { return g_err; }

extern "C" int b200p_arch_check(void) {
  int rc = query_device();
  if (rc) return rc;
  B200P_REQUIRE(g_cc_major == 10, B200P_ERR_ARCH, "device compute capability %d.x is not sm_100", g_cc_major);
  return B200P_OK;
}

extern "C" int b200p_sm_count(void) {
  int rc = query_device();
  if (rc) return rc;
  return g_sm_count;
}

extern "C" int b200p_set_pdl(int enabled) {
  g_pdl = enabled;
  return B200P_OK;
}

