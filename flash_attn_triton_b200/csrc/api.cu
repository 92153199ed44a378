// C ABI: argument validation, kernel-family dispatch, error strings.  See include/fa_b200.h.
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <type_traits>
#ifdef FA_SKEW
#include <vector>
#endif

#include "common.cuh"
#include "queue_slots.h"

namespace fa {

static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("%s: launch failed: %s", what, cudaGetErrorString(e));
    return FA_ERR_LAUNCH;
  }
  return FA_OK;
}

int ensure_device(int device) {
  int cur = -1;
  cudaError_t e = cudaGetDevice(&cur);
  if (e == cudaSuccess && cur == device) return FA_OK;
  e = cudaSetDevice(device);
  if (e != cudaSuccess) {
    set_error("cudaSetDevice(%d): %s", device, cudaGetErrorString(e));
    return FA_ERR_LAUNCH;
  }
  return FA_OK;
}

int sm_count(int device) {
  static int cached[64] = {0};
  const bool slot = device >= 0 && device < 64;
  if (slot && cached[device] > 0) return cached[device];
  int n = 0;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n <= 0) n = 148;
  if (slot) cached[device] = n;
  return n;
}

// One word per device ordinal, in a page of its own that is registered (pinned and mapped) on
// first use: no allocation, the kernels write it through the mapping, the host just reads it.
alignas(4096) static volatile int g_host_wait[1024];
static std::mutex g_host_wait_mu;
static int g_host_wait_registered = 0;   // 0 not tried, 1 mapped, -1 unavailable

int* host_wait_word(int device) {
  if (device < 0 || device >= 1024) return nullptr;
  std::lock_guard<std::mutex> lock(g_host_wait_mu);
  if (g_host_wait_registered == 0) {
    cudaError_t e = cudaHostRegister(const_cast<int*>(g_host_wait), sizeof(g_host_wait),
                                     cudaHostRegisterPortable | cudaHostRegisterMapped);
    g_host_wait_registered = (e == cudaSuccess) ? 1 : -1;
    if (e != cudaSuccess) cudaGetLastError();
  }
  if (g_host_wait_registered != 1) return nullptr;
  int* dptr = nullptr;
  if (cudaHostGetDevicePointer(&dptr, const_cast<int*>(&g_host_wait[device]), 0) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return dptr;
}

int host_wait_status(int device) { return (device >= 0 && device < 1024) ? g_host_wait[device] : 0; }

// Per device: 1024 streams, and 15 k launches in graphs.
using WorkQueues = QueueSlots<1024, 15 * 1024>;
static __device__ unsigned int g_work_queues[WorkQueues::kPairs][2];
constexpr int kQueueDevices = 64;

static WorkQueues g_queue_slots[kQueueDevices];      // (of which the devices in use are in memory)
static_assert(std::is_trivially_destructible<WorkQueues>::value, "the last graphs may go when the process ends");
// A graph that a launch was captured into is gone, with all that was made of it.  Called on a thread of the driver: no CUDA call here, and
// none under the lock that this takes.
static void give_work_queue(void* where) {
  const uintptr_t w = reinterpret_cast<uintptr_t>(where);
  g_queue_slots[w % kQueueDevices].give((int)(w / kQueueDevices));
}
#ifdef FA_SKEW
static int g_debug_no_queues = 0;
#endif
static int work_queue_of(int device, cudaStream_t st) {
  constexpr int kNone = WorkQueues::kNone;
#ifdef FA_SKEW
  if (g_debug_no_queues) return kNone;
#endif
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  cudaGraph_t graph = nullptr;
  if (cudaStreamGetCaptureInfo_v2(st, &status, nullptr, &graph, nullptr, nullptr) != cudaSuccess) return kNone;
  if (status == cudaStreamCaptureStatusNone) return cudaStreamGetId(st, &id) == cudaSuccess ? g_queue_slots[device].of_stream(id) : kNone;
  if (status != cudaStreamCaptureStatusActive) return kNone;
  const int i = g_queue_slots[device].take();
  if (i == kNone) return kNone;
  cudaUserObject_t owner = nullptr;
  void* const where = reinterpret_cast<void*>((uintptr_t)i * kQueueDevices + device);
  if (cudaUserObjectCreate(&owner, where, give_work_queue, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
    g_queue_slots[device].give(i);
    return kNone;
  }
  if (cudaGraphRetainUserObject(graph, owner, 1, cudaGraphUserObjectMove) != cudaSuccess) {
    cudaUserObjectRelease(owner, 1);                 // gives the pair back
    return kNone;
  }
  return i;
}

int queue_grid(int device, cudaStream_t st, int ncand, int ctas, unsigned int** queue) {
  *queue = nullptr;
  if (ncand <= ctas || device < 0 || device >= kQueueDevices) return ncand;
  static std::atomic<unsigned int*> base[kQueueDevices];
  unsigned int* p = base[device].load(std::memory_order_acquire);
  int i = WorkQueues::kNone;
  if (p == nullptr) {
    void* at = nullptr;
    if (cudaGetSymbolAddress(&at, g_work_queues) == cudaSuccess) p = static_cast<unsigned int*>(at);
    base[device].store(p, std::memory_order_release);
  }
  if (p != nullptr) i = work_queue_of(device, st);
  if (i == WorkQueues::kNone) {
    cudaGetLastError();
    return ncand;
  }
  *queue = p + 2 * (int64_t)i;
  return ctas;
}

// kernel families (defined in the other translation units)
int fwd_mma(const fa_attn_args&, const ScoreCfg&, cudaStream_t);
int attn_probs(const fa_attn_args&, const ScoreCfg&, float*, const int64_t*, float*, int64_t, cudaStream_t);
int bwd_preprocess(const fa_attn_args&, cudaStream_t);
int bwd_dq_mma(const fa_attn_args&, const ScoreCfg&, cudaStream_t);
int bwd_dkdv_mma(const fa_attn_args&, const ScoreCfg&, cudaStream_t);
bool fwd_sm100_supported(const fa_attn_args&);
int fwd_sm100(const fa_attn_args&, const ScoreCfg&, cudaStream_t);
bool bwd_sm100_supported(const fa_attn_args&);
int bwd_dq_sm100(const fa_attn_args&, const ScoreCfg&, cudaStream_t);
int bwd_dkdv_sm100(const fa_attn_args&, const ScoreCfg&, cudaStream_t);
int fwd_alt_sm100(const fa_attn_args&, const ScoreCfg&, cudaStream_t);
int fwd_alt_sm100_status();
int fwd_duo_sm100_status();
int64_t dropout_bits_words(int, int);
int dropout_bits(const fa_attn_args&, const ScoreCfg&, uint32_t*, cudaStream_t);
int fwd_alt_sm100_clear_status();
int fwd_duo_sm100_clear_status();
int decode_paged(const fa_decode_args&, cudaStream_t);
int decode_paged_checked(const fa_decode_args&, uint32_t*, cudaStream_t);
int varlen_check(const int32_t*, const int32_t*, int, int64_t, int64_t, bool, int64_t, int64_t, int, int32_t*, cudaStream_t);
int check_result(int32_t, uint32_t*, cudaStream_t);
int decode_num_counters(const fa_decode_args&);
size_t decode_workspace_bytes(const fa_decode_args&);
size_t decode_checked_workspace_bytes(const fa_decode_args&);
int decode_paged_static(const fa_decode_args&, cudaStream_t);
size_t decode_static_scratch_bytes();
int quantize_k(const void*, int8_t*, float*, int64_t, int, cudaStream_t);
int fwd_int8_mma(const fa_int8_args&, cudaStream_t);
bool fwd_int8_sm100_supported(const fa_int8_args&);
int fwd_int8_sm100(const fa_int8_args&, cudaStream_t);
bool int8_codes16_supported(const fa_int8_args&);
int quantize_codes16(const void*, void*, float*, int64_t, bool, cudaStream_t);
int fwd_int8_codes16(const fa_int8_args&, const void*, const void*, cudaStream_t);
int rotary(const fa_rotary_args&, cudaStream_t);
int gather_rows(const void*, void*, const int64_t*, int64_t, int64_t, int64_t, int, cudaStream_t);
int scatter_rows(const void*, void*, const int64_t*, int64_t, int64_t, int64_t, int, int, cudaStream_t);
int fwd_sm100_status();
int bwd_sm100_status();
void fwd_sm100_clear_status();
void bwd_sm100_clear_status();
int wait_probe(int device, long long clocks, cudaStream_t st);
#ifdef FA_SKEW
int skew_mode_bwd(int), skew_mode_duo(int);
#endif
int mma_peak_probe(int device, int kind, int iters, cudaStream_t st);

static bool mult8(const int64_t* s, int n) {
  for (int i = 0; i < n; ++i)
    if (s[i] % 8 != 0) return false;
  return true;
}
static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

static int validate_common(const fa_attn_args* a, bool need_cu) {
  FA_REQUIRE(a != nullptr, "args is NULL");
  FA_REQUIRE(a->dtype == FA_F16 || a->dtype == FA_BF16, "dtype must be FA_F16 or FA_BF16");
  FA_REQUIRE(a->batch >= 0 && a->seqlen_q >= 0 && a->seqlen_k >= 0, "negative size");
  FA_REQUIRE(a->heads_q > 0 && a->heads_kv > 0 && a->heads_q % a->heads_kv == 0,
             "heads_q (%d) must be a positive multiple of heads_kv (%d)", a->heads_q, a->heads_kv);
  FA_REQUIRE(a->head_dim == 16 || a->head_dim == 32 || a->head_dim == 64 || a->head_dim == 128 ||
                 a->head_dim == 256,
             "head dimension must be one of 16, 32, 64, 128, or 256 (got %d)", a->head_dim);
  FA_REQUIRE(a->softcap >= 0.f, "softcap must be non-negative");
  FA_REQUIRE(a->dropout_p >= 0.f && a->dropout_p < 1.f, "dropout_p must be in the range [0, 1)");
  FA_REQUIRE(a->dropout_p == 0.f || a->dropout_row_stride > 0, "dropout needs dropout_row_stride > 0");
  FA_REQUIRE(a->attn_bias == nullptr || a->cu_seqlens_q == nullptr, "attn_bias is for the dense layout only");
  FA_REQUIRE((a->seqused_q == nullptr && a->seqused_k == nullptr) || a->cu_seqlens_q != nullptr,
             "seqused_q/seqused_k need the packed layout");
  FA_REQUIRE((a->cu_seqlens_q == nullptr) == (a->cu_seqlens_k == nullptr),
             "cu_seqlens_q and cu_seqlens_k must be given together");
  if (need_cu) FA_REQUIRE(a->cu_seqlens_q != nullptr, "packed layout needs cu_seqlens_q/k");
  if (a->cu_seqlens_q) {
    FA_REQUIRE(a->q_pos_offset == 0, "q_pos_offset is dense-only");
    FA_REQUIRE(a->total_q >= 0 && a->total_k >= 0, "total_q/total_k must be the packed row counts");
  }
  const bool empty = a->batch == 0 || a->seqlen_q == 0;
  if (!empty) {
    FA_REQUIRE(a->q && a->o, "q/o is NULL");
    FA_REQUIRE(a->seqlen_k == 0 || (a->k && a->v), "k/v is NULL");
    FA_REQUIRE(aligned16(a->q) && aligned16(a->k) && aligned16(a->v) && aligned16(a->o),
               "q/k/v/o must be 16-byte aligned");
    FA_REQUIRE(mult8(a->q_stride, 3) && mult8(a->k_stride, 3) && mult8(a->v_stride, 3) &&
                   mult8(a->o_stride, 3),
               "strides must be multiples of 8 elements (16-byte rows)");
  }
  return FA_OK;
}

static int validate_bwd(const fa_attn_args* a) {
  if (a->batch == 0 || a->seqlen_q == 0) return FA_OK;
  FA_REQUIRE(a->dout && a->lse2 && a->delta, "backward needs dout, lse2 and delta");
  FA_REQUIRE(aligned16(a->dout) && mult8(a->do_stride, 3), "dout alignment/stride");
  return FA_OK;
}

static ScoreCfg cfg_of(const fa_attn_args* a) {
  ScoreCfg c = make_score_cfg(a->softmax_scale, a->softcap, a->causal, a->window_left, a->window_right,
                              a->alibi_slopes != nullptr);
  c.bias = a->attn_bias;
  for (int i = 0; i < 4; ++i) c.bias_stride[i] = a->bias_stride[i];
  if (a->dropout_p > 0.f) {
    c.dropout_p = a->dropout_p;
    c.dropout_scale = 1.f / (1.f - a->dropout_p);
    c.seed_lo = (uint32_t)(a->dropout_seed & 0xffffffffull);
    c.seed_hi = (uint32_t)(a->dropout_seed >> 32);
    c.drop_stride = (uint32_t)a->dropout_row_stride;
  }
  return c;
}

// Bias and dropout drawn per score are features of the mma.sync kernels (dropout as bits: fa_fwd_dropout and its
// companions).
static bool needs_mma(const fa_attn_args* a) { return a->attn_bias != nullptr || a->dropout_p > 0.f; }

// Calls whose dropout mask the tcgen05 kernels read as bits: the plain dense variants of both kernels.
// 64 MiB for the two copies is a square problem of 16384; longer ones draw per score.
constexpr int64_t kDropoutBitsLimit = 64ll << 20;
static int64_t dropout_bits_bytes(const fa_attn_args* a, bool backward) {
  if (a == nullptr || !(a->dropout_p > 0.f) || a->impl != FA_IMPL_AUTO || a->cu_seqlens_q != nullptr || a->attn_bias != nullptr ||
      a->alibi_slopes != nullptr || a->softcap > 0.f)
    return 0;
  if (a->head_dim != 64 && a->head_dim != 128) return 0;
  if (!(a->softmax_scale * FA_LOG2E > 2e-5f)) return 0;     // see launch_dkdv in bwd_sm100.cu
  if (!(backward ? bwd_sm100_supported(*a) : fwd_sm100_supported(*a))) return 0;
  const int64_t bytes = 2 * 4 * dropout_bits_words(a->seqlen_q, a->seqlen_k);
  return bytes <= kDropoutBitsLimit ? bytes : 0;
}

// A bounded wait that ran out earlier on this device (host mirror of the status word): the tcgen05
// kernels would return at their first wait, so the call is refused before anything is launched.
static int refuse_after_timeout(int device, const char* what) {
  if (const int c = host_wait_status(device)) {
    set_error("%s: a bounded device-side wait ran out earlier on device %d (code %d); the tcgen05 kernels stay "
              "off until fa_device_wait_clear()", what, device, c);
    return FA_ERR_DEVICE_WAIT;
  }
  return FA_OK;
}

static int fwd_impl(const fa_attn_args* a, void* stream, bool need_cu) {
  if (int r = validate_common(a, need_cu)) return r;
  if (a->impl != FA_IMPL_MMA && fwd_sm100_supported(*a) && !needs_mma(a))
    if (int r = refuse_after_timeout(a->device, "fa_fwd")) return r;
  if (int r = ensure_device(a->device)) return r;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const ScoreCfg cfg = cfg_of(a);
  if (a->impl == FA_IMPL_TCGEN05) {
    if (!fwd_sm100_supported(*a) || needs_mma(a)) {
      set_error("no tcgen05 forward kernel for this shape/feature set");
      return FA_ERR_UNSUPPORTED;
    }
    return fwd_sm100(*a, cfg, st);
  }
  if (a->impl == FA_IMPL_AUTO && fwd_sm100_supported(*a) && !needs_mma(a)) return fwd_sm100(*a, cfg, st);
  return fwd_mma(*a, cfg, st);
}

static int dq_impl(const fa_attn_args* a, void* stream, bool need_cu) {
  if (int r = validate_common(a, need_cu)) return r;
  if (int r = validate_bwd(a)) return r;
  if (a->batch && a->seqlen_q) {
    FA_REQUIRE(a->dq && aligned16(a->dq) && mult8(a->dq_stride, 3), "dq pointer/alignment/stride");
  }
  if (a->impl != FA_IMPL_MMA && bwd_sm100_supported(*a) && !needs_mma(a))
    if (int r = refuse_after_timeout(a->device, "fa_bwd_dq")) return r;
  if (int r = ensure_device(a->device)) return r;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const ScoreCfg cfg = cfg_of(a);
  if (a->impl == FA_IMPL_TCGEN05) {
    if (!bwd_sm100_supported(*a) || needs_mma(a)) {
      set_error("no tcgen05 backward kernel for this shape/feature set");
      return FA_ERR_UNSUPPORTED;
    }
    return bwd_dq_sm100(*a, cfg, st);
  }
  if (a->impl == FA_IMPL_AUTO && bwd_sm100_supported(*a) && !needs_mma(a)) return bwd_dq_sm100(*a, cfg, st);
  return bwd_dq_mma(*a, cfg, st);
}

static int dkdv_impl(const fa_attn_args* a, void* stream, bool need_cu) {
  if (int r = validate_common(a, need_cu)) return r;
  if (int r = validate_bwd(a)) return r;
  if (a->batch && a->seqlen_k) {
    FA_REQUIRE(a->dk && a->dv && aligned16(a->dk) && aligned16(a->dv) && mult8(a->dk_stride, 3) &&
                   mult8(a->dv_stride, 3),
               "dk/dv pointer/alignment/stride");
  }
  if (a->impl != FA_IMPL_MMA && bwd_sm100_supported(*a) && !needs_mma(a))
    if (int r = refuse_after_timeout(a->device, "fa_bwd_dkdv")) return r;
  if (int r = ensure_device(a->device)) return r;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const ScoreCfg cfg = cfg_of(a);
  if (a->impl == FA_IMPL_TCGEN05) {
    if (!bwd_sm100_supported(*a) || needs_mma(a)) {
      set_error("no tcgen05 backward kernel for this shape/feature set");
      return FA_ERR_UNSUPPORTED;
    }
    return bwd_dkdv_sm100(*a, cfg, st);
  }
  if (a->impl == FA_IMPL_AUTO && bwd_sm100_supported(*a) && !needs_mma(a)) return bwd_dkdv_sm100(*a, cfg, st);
  return bwd_dkdv_mma(*a, cfg, st);
}

enum DropoutOp { kDropFwd, kDropDq, kDropDkdv };

static int dropout_impl(const fa_attn_args* a, const void* bits, void* stream, DropoutOp op) {
  if (int r = validate_common(a, false)) return r;
  FA_REQUIRE(dropout_bits_bytes(a, op != kDropFwd) > 0, "the call does not take its dropout mask as bits");
  FA_REQUIRE(bits != nullptr && aligned16(bits), "dropout bits must be a 16-byte aligned buffer");
  if (op != kDropFwd)
    if (int r = validate_bwd(a)) return r;
  if (op == kDropDq) FA_REQUIRE(a->dq && aligned16(a->dq) && mult8(a->dq_stride, 3), "dq pointer/alignment/stride");
  if (op == kDropDkdv)
    FA_REQUIRE(a->dk && a->dv && aligned16(a->dk) && aligned16(a->dv) && mult8(a->dk_stride, 3) && mult8(a->dv_stride, 3),
               "dk/dv pointer/alignment/stride");
  if (int r = refuse_after_timeout(a->device, op == kDropFwd ? "fa_fwd_dropout" : "fa_bwd_dropout")) return r;
  if (int r = ensure_device(a->device)) return r;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  ScoreCfg cfg = cfg_of(a);
  const int64_t tiles_q = (a->seqlen_q + 127) / 128, tiles_k = (a->seqlen_k + 127) / 128;
  const uint32_t* words = static_cast<const uint32_t*>(bits);
  cfg.drop_log2 = log2f(cfg.dropout_scale);
  cfg.keep = op == kDropDkdv ? words + dropout_bits_words(a->seqlen_q, a->seqlen_k) : words;
  cfg.keep_words = 4 * (op == kDropDkdv ? tiles_q : tiles_k);
  return op == kDropFwd ? fwd_sm100(*a, cfg, st) : op == kDropDq ? bwd_dq_sm100(*a, cfg, st) : bwd_dkdv_sm100(*a, cfg, st);
}

}  // namespace fa

using namespace fa;

extern "C" {

int fa_fwd(const fa_attn_args* a, void* stream) { return fwd_impl(a, stream, false); }
int fa_varlen_fwd(const fa_attn_args* a, void* stream) { return fwd_impl(a, stream, true); }

int fa_attn_probs(const fa_attn_args* a, float* probs, const int64_t* probs_stride, float* lse_nat,
                  int64_t lse_nat_stride, void* stream) {
  if (int r = validate_common(a, false)) return r;
  if (a->batch == 0 || a->seqlen_q == 0 || a->seqlen_k == 0) return FA_OK;
  FA_REQUIRE(probs != nullptr && probs_stride != nullptr && a->lse2 != nullptr, "probs, probs_stride and lse2 are required");
  if (int r = ensure_device(a->device)) return r;
  return attn_probs(*a, cfg_of(a), probs, probs_stride, lse_nat, lse_nat_stride, reinterpret_cast<cudaStream_t>(stream));
}

int fa_bwd_preprocess(const fa_attn_args* a, void* stream) {
  if (int r = validate_common(a, false)) return r;
  if (int r = validate_bwd(a)) return r;
  if (int r = ensure_device(a->device)) return r;
  return bwd_preprocess(*a, reinterpret_cast<cudaStream_t>(stream));
}

int fa_bwd_dq(const fa_attn_args* a, void* stream) { return dq_impl(a, stream, false); }
int fa_varlen_bwd_dq(const fa_attn_args* a, void* stream) { return dq_impl(a, stream, true); }
int fa_bwd_dkdv(const fa_attn_args* a, void* stream) { return dkdv_impl(a, stream, false); }
int fa_varlen_bwd_dkdv(const fa_attn_args* a, void* stream) { return dkdv_impl(a, stream, true); }

size_t fa_dropout_bits_bytes(const fa_attn_args* a, int32_t backward) { return (size_t)dropout_bits_bytes(a, backward != 0); }
int fa_dropout_bits(const fa_attn_args* a, void* bits, void* stream) {
  if (int r = validate_common(a, false)) return r;
  FA_REQUIRE(dropout_bits_bytes(a, false) > 0 || dropout_bits_bytes(a, true) > 0,
             "the call does not take its dropout mask as bits");
  FA_REQUIRE(bits != nullptr && aligned16(bits), "dropout bits must be a 16-byte aligned buffer");
  if (int r = ensure_device(a->device)) return r;
  return dropout_bits(*a, cfg_of(a), static_cast<uint32_t*>(bits), reinterpret_cast<cudaStream_t>(stream));
}
int fa_fwd_dropout(const fa_attn_args* a, const void* bits, void* stream) { return dropout_impl(a, bits, stream, kDropFwd); }
int fa_bwd_dq_dropout(const fa_attn_args* a, const void* bits, void* stream) { return dropout_impl(a, bits, stream, kDropDq); }
int fa_bwd_dkdv_dropout(const fa_attn_args* a, const void* bits, void* stream) { return dropout_impl(a, bits, stream, kDropDkdv); }

static int validate_decode(const fa_decode_args* a) {
  FA_REQUIRE(a != nullptr, "args is NULL");
  FA_REQUIRE(a->dtype == FA_F16 || a->dtype == FA_BF16, "dtype must be FA_F16 or FA_BF16");
  FA_REQUIRE(a->batch >= 0 && a->seqlen_q >= 0, "negative size");
  FA_REQUIRE(a->heads_q > 0 && a->heads_kv > 0 && a->heads_q % a->heads_kv == 0,
             "heads_q must be a positive multiple of heads_kv");
  FA_REQUIRE(a->head_dim == 16 || a->head_dim == 32 || a->head_dim == 64 || a->head_dim == 128 ||
                 a->head_dim == 256,
             "head dimension must be one of 16, 32, 64, 128, or 256 (got %d)", a->head_dim);
  if (a->batch == 0 || a->seqlen_q == 0) return FA_OK;
  FA_REQUIRE(a->q && a->o && a->k_cache && a->v_cache && a->cache_seqlens,
             "q, o, k_cache, v_cache and cache_seqlens are required");
  FA_REQUIRE(a->page_size > 0, "page_size must be positive");
  FA_REQUIRE(aligned16(a->k_cache) && aligned16(a->v_cache) && mult8(a->kc_stride, 3) &&
                 mult8(a->vc_stride, 3),
             "cache rows must be 16-byte aligned");
  FA_REQUIRE(aligned16(a->q) && aligned16(a->o), "q and o must be 16-byte aligned");
  FA_REQUIRE(mult8(a->q_stride, 3) && mult8(a->o_stride, 3), "q/o strides must be multiples of 8 elements");
  FA_REQUIRE(a->workspace == nullptr || aligned16(a->workspace), "workspace must be 16-byte aligned");
  FA_REQUIRE(a->num_splits >= 0, "num_splits must be non-negative");
  FA_REQUIRE(a->block_table == nullptr || a->block_table_stride > 0,
             "block_table_stride must be positive when a block table is given");
  FA_REQUIRE(!(a->block_table && a->cache_batch_idx), "cache_batch_idx cannot be combined with paged KV caches");
  FA_REQUIRE(!(a->block_table && a->cache_leftpad), "cache_leftpad cannot be combined with paged KV caches");
  FA_REQUIRE((a->k_new == nullptr) == (a->v_new == nullptr), "k and v must be supplied together");
  FA_REQUIRE((a->rotary_cos == nullptr) == (a->rotary_sin == nullptr),
             "rotary_cos and rotary_sin must be supplied together");
  if (a->rotary_cos) {
    FA_REQUIRE(a->rotary_dim > 0 && a->rotary_dim % 2 == 0 && a->rotary_dim <= a->head_dim,
               "rotary tables exceed the head dimension");
    FA_REQUIRE(a->rotary_seqlen > 0, "rotary_seqlen must be the number of rows of the rotary tables");
  }
  if (a->k_new) {
    FA_REQUIRE(a->seqlen_new > 0, "seqlen_new must be positive when k/v are given");
    FA_REQUIRE(aligned16(a->k_new) && aligned16(a->v_new) && mult8(a->kn_stride, 3) && mult8(a->vn_stride, 3),
               "new k/v rows must be 16-byte aligned");
  }
  return FA_OK;
}

int fa_decode_paged(const fa_decode_args* a, void* stream) {
  if (int r = validate_decode(a)) return r;
  if (int r = ensure_device(a->device)) return r;
  return decode_paged(*a, reinterpret_cast<cudaStream_t>(stream));
}

int fa_decode_paged_checked(const fa_decode_args* a, uint32_t* failed, void* stream) {
  if (int r = validate_decode(a)) return r;
  FA_REQUIRE(failed != nullptr, "failed is NULL");
  if (int r = ensure_device(a->device)) return r;
  return decode_paged_checked(*a, failed, reinterpret_cast<cudaStream_t>(stream));
}

int fa_varlen_check(const int32_t* cu_q, const int32_t* cu_k, int32_t batch, int64_t total_q, int64_t total_k, int32_t k_at_most,
                    int64_t max_q, int64_t max_k, int32_t device, int32_t* ticket, void* stream) {
  FA_REQUIRE(cu_q != nullptr && cu_k != nullptr && ticket != nullptr && batch >= 0, "cu_seqlens and ticket are required");
  if (int r = ensure_device(device)) return r;
  return varlen_check(cu_q, cu_k, batch, total_q, total_k, k_at_most != 0, max_q, max_k, device, ticket,
                      reinterpret_cast<cudaStream_t>(stream));
}

int fa_check_result(int32_t ticket, uint32_t* failed, void* stream) {
  FA_REQUIRE(failed != nullptr, "failed is NULL");
  return check_result(ticket, failed, reinterpret_cast<cudaStream_t>(stream));
}

int32_t fa_decode_counters(const fa_decode_args* a) {
  if (a == nullptr || a->heads_kv <= 0 || a->heads_q <= 0 || a->batch <= 0 || a->seqlen_q <= 0) return 0;
  return decode_num_counters(*a);
}

int fa_decode_paged_static(const fa_decode_args* a, void* stream) {
  if (int r = validate_decode(a)) return r;
  if (int r = ensure_device(a->device)) return r;
  return decode_paged_static(*a, reinterpret_cast<cudaStream_t>(stream));
}

size_t fa_decode_static_scratch_bytes(void) { return decode_static_scratch_bytes(); }

size_t fa_decode_checked_workspace_bytes(const fa_decode_args* a) {
  if (a == nullptr || a->heads_kv <= 0 || a->heads_q <= 0 || a->page_size <= 0) return 0;
  return decode_checked_workspace_bytes(*a);
}
size_t fa_decode_workspace_bytes(const fa_decode_args* a) {
  if (a == nullptr || a->heads_kv <= 0 || a->heads_q <= 0 || a->page_size <= 0) return 0;
  return decode_workspace_bytes(*a);
}

int fa_quantize_k_int8(const void* k, int8_t* k8, float* s_k, int64_t rows, int32_t head_dim,
                       int32_t device, void* stream) {
  FA_REQUIRE(rows >= 0, "negative rows");
  if (rows == 0) return FA_OK;
  FA_REQUIRE(k && k8 && s_k, "NULL pointer");
  FA_REQUIRE(aligned16(k) && (reinterpret_cast<uintptr_t>(k8) & 7) == 0, "k must be 16-byte, k8 8-byte aligned");
  FA_REQUIRE(head_dim >= 32 && (head_dim & (head_dim - 1)) == 0,
             "The INT8 kernel requires a power-of-two head dim of at least 32");
  if (int r = ensure_device(device)) return r;
  return quantize_k(k, k8, s_k, rows, head_dim, reinterpret_cast<cudaStream_t>(stream));
}

int fa_fwd_int8(const fa_int8_args* a, void* stream) {
  FA_REQUIRE(a != nullptr, "args is NULL");
  FA_REQUIRE(a->batch >= 0 && a->heads >= 0 && a->seqlen >= 0, "negative size");
  FA_REQUIRE(a->head_dim >= 32 && (a->head_dim & (a->head_dim - 1)) == 0,
             "The INT8 kernel requires a power-of-two head dim of at least 32");
  if (a->batch * a->heads == 0 || a->seqlen == 0) return FA_OK;
  FA_REQUIRE(a->q && a->k8 && a->s_k && a->v && a->o, "NULL pointer");
  FA_REQUIRE(a->seqlen_k_valid >= 0 && a->seqlen_k_valid <= a->seqlen, "seqlen_k_valid must lie in [0, seqlen]");
  FA_REQUIRE(aligned16(a->q) && aligned16(a->k8) && aligned16(a->v) && aligned16(a->o), "16-byte alignment");
  if (a->impl != FA_IMPL_MMA && fwd_int8_sm100_supported(*a))
    if (int r = refuse_after_timeout(a->device, "fa_fwd_int8")) return r;
  if (int r = ensure_device(a->device)) return r;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (a->impl == FA_IMPL_TCGEN05) {
    if (!fwd_int8_sm100_supported(*a)) {
      set_error("no tcgen05 INT8 kernel for this shape");
      return FA_ERR_UNSUPPORTED;
    }
    return fwd_int8_sm100(*a, st);
  }
  if (a->impl == FA_IMPL_AUTO && fwd_int8_sm100_supported(*a)) return fwd_int8_sm100(*a, st);
  return fwd_int8_mma(*a, st);
}

size_t fa_int8_codes16_bytes(const fa_int8_args* a) {
  if (a == nullptr || a->batch <= 0 || a->heads <= 0 || a->seqlen <= 0 || !int8_codes16_supported(*a)) return 0;
  return (size_t)a->batch * a->heads * a->seqlen * a->head_dim * 4;
}

int fa_fwd_int8_codes16(const fa_int8_args* a, const void* k, float* s_k, void* codes, void* stream) {
  FA_REQUIRE(a != nullptr, "args is NULL");
  FA_REQUIRE(fa_int8_codes16_bytes(a) > 0, "the call does not take its codes as 16-bit floats");
  FA_REQUIRE(a->q && k && s_k && a->v && a->o && a->sq_scratch && codes, "NULL pointer");
  FA_REQUIRE(a->seqlen_k_valid >= 0 && a->seqlen_k_valid <= a->seqlen, "seqlen_k_valid must lie in [0, seqlen]");
  FA_REQUIRE(aligned16(a->q) && aligned16(k) && aligned16(a->v) && aligned16(a->o) && aligned16(codes), "16-byte alignment");
  if (int r = refuse_after_timeout(a->device, "fa_fwd_int8_codes16")) return r;
  if (int r = ensure_device(a->device)) return r;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int64_t rows = (int64_t)a->batch * a->heads * a->seqlen;
  void* k16 = static_cast<char*>(codes) + rows * a->head_dim * 2;
  if (int r = quantize_codes16(a->q, codes, a->sq_scratch, rows, true, st)) return r;
  if (int r = quantize_codes16(k, k16, s_k, rows, false, st)) return r;
  fa_int8_args p = *a;
  p.s_k = s_k;
  return fwd_int8_codes16(p, codes, k16, st);
}

int fa_rotary(const fa_rotary_args* a, void* stream) {
  FA_REQUIRE(a != nullptr, "args is NULL");
  FA_REQUIRE(a->dtype == FA_F16 || a->dtype == FA_BF16 || a->dtype == FA_F32, "dtype must be FA_F16, FA_BF16 or FA_F32");
  FA_REQUIRE(a->batch >= 0 && a->seqlen >= 0 && a->heads >= 0 && a->head_dim > 0, "negative size");
  FA_REQUIRE(a->head_dim <= 256, "Only support headdim <= 256");
  FA_REQUIRE(a->rotary_dim >= 0 && a->rotary_dim % 2 == 0 && a->rotary_dim <= a->head_dim,
             "rotary_dim must be even and <= headdim");
  FA_REQUIRE(a->rotary_seqlen >= 0, "negative rotary table length");
  if (a->batch == 0 || a->seqlen == 0 || a->heads == 0) return FA_OK;
  FA_REQUIRE(a->x && a->out, "x/out is NULL");
  FA_REQUIRE(a->rotary_dim == 0 || (a->cos && a->sin), "cos/sin is NULL");
  if (int r = ensure_device(a->device)) return r;
  return rotary(*a, reinterpret_cast<cudaStream_t>(stream));
}

static int validate_rows(const void* src, void* dst, const int64_t* idx, int64_t n_idx, int64_t row_bytes,
                         int64_t rows) {
  FA_REQUIRE(n_idx >= 0 && row_bytes >= 0 && rows >= 0, "negative size");
  if (n_idx == 0 || row_bytes == 0) return FA_OK;
  FA_REQUIRE(src && dst && idx, "NULL pointer");
  FA_REQUIRE(row_bytes % 16 == 0 && aligned16(src) && aligned16(dst), "rows must be 16-byte multiples, 16-byte aligned");
  FA_REQUIRE(row_bytes / 16 <= 0x7fffffff, "row too long");
  return FA_OK;
}

int fa_gather_rows(const void* src, void* dst, const int64_t* idx, int64_t n_idx, int64_t row_bytes,
                   int64_t src_rows, int32_t device, void* stream) {
  if (int r = validate_rows(src, dst, idx, n_idx, row_bytes, src_rows)) return r;
  if (n_idx == 0 || row_bytes == 0) return FA_OK;
  if (int r = ensure_device(device)) return r;
  return gather_rows(src, dst, idx, n_idx, row_bytes, src_rows, device, reinterpret_cast<cudaStream_t>(stream));
}

int fa_scatter_rows(const void* src, void* dst, const int64_t* idx, int64_t n_idx, int64_t row_bytes,
                    int64_t dst_rows, int32_t add_dtype, int32_t device, void* stream) {
  if (int r = validate_rows(src, dst, idx, n_idx, row_bytes, dst_rows)) return r;
  FA_REQUIRE(add_dtype >= -1 && add_dtype <= FA_F32, "add_dtype must be -1 or an fa_dtype");
  if (n_idx == 0 || row_bytes == 0) return FA_OK;
  if (int r = ensure_device(device)) return r;
  return scatter_rows(src, dst, idx, n_idx, row_bytes, dst_rows, add_dtype, device,
                      reinterpret_cast<cudaStream_t>(stream));
}

const char* fa_version(void) { return "fa_b200 0.1 (sm_100a)"; }
const char* fa_last_error(void) { return g_err; }
int fa_fwd_uses_tcgen05(const fa_attn_args* a) {
  return a != nullptr && a->impl != FA_IMPL_MMA && fwd_sm100_supported(*a) ? 1 : 0;
}

int fa_device_wait_status(int device) {
  if (int r = ensure_device(device)) return r;
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    set_error("cudaDeviceSynchronize: %s", cudaGetErrorString(e));
    return FA_ERR_LAUNCH;
  }
  int s = fwd_sm100_status();
  if (s == 0) s = bwd_sm100_status();
  if (s == 0) s = fwd_alt_sm100_status();
  if (s == 0) s = fwd_duo_sm100_status();
  if (s == 0) s = host_wait_status(device);
  if (s != 0 && device >= 0 && device < 1024) g_host_wait[device] = s;   // remembered for the launchers
  return s;
}

int fa_device_wait_clear(int device) {
  if (int r = ensure_device(device)) return r;
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    set_error("cudaDeviceSynchronize: %s", cudaGetErrorString(e));
    return FA_ERR_LAUNCH;
  }
  fwd_sm100_clear_status();
  bwd_sm100_clear_status();
  fwd_alt_sm100_clear_status();
  fwd_duo_sm100_clear_status();
  // a launch whose CTAs gave up has not put its pair of counters back to zero; the next one to get the pair would skip items
  void* queues = nullptr;
  e = cudaGetSymbolAddress(&queues, g_work_queues);
  if (e == cudaSuccess) e = cudaMemset(queues, 0, sizeof(g_work_queues));
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    set_error("clearing the work queues: %s", cudaGetErrorString(e));
    return FA_ERR_LAUNCH;
  }
  if (device >= 0 && device < 1024) g_host_wait[device] = 0;
  return FA_OK;
}

int fa_wait_probe(int32_t device, int64_t clocks, void* stream) {
  FA_REQUIRE(clocks > 0 && clocks <= 2000000000LL, "clocks must be in (0, 2e9]");
  if (int r = ensure_device(device)) return r;
  return wait_probe(device, clocks, reinterpret_cast<cudaStream_t>(stream));
}

int fa_mma_peak_probe(int32_t device, int32_t kind, int32_t iters, void* stream) {
  FA_REQUIRE(kind == 0 || kind == 1, "kind: 0 = fp16 operands, 1 = int8 operands");
  FA_REQUIRE(iters > 0 && iters <= (1 << 24), "iters must be in (0, 2^24]");
  if (int r = ensure_device(device)) return r;
  return mma_peak_probe(device, kind, iters, reinterpret_cast<cudaStream_t>(stream));
}

#ifdef FA_SKEW
// Side build of the tests: the counters as launches whose CTAs gave up on a wait may leave them; launches as where no pair is left; pairs
// that captured launches have.
int fa_debug_dirty_queues(unsigned int value) {
  const std::vector<unsigned int> pairs(2 * WorkQueues::kPairs, value);
  return (int)cudaMemcpyToSymbol(g_work_queues, pairs.data(), sizeof(g_work_queues));
}
int fa_debug_no_queues(int on) {
  g_debug_no_queues = on;
  return 0;
}
// The warps that are late (skew.cuh).
int fa_debug_skew(int mode) {
  const int e = skew_mode_bwd(mode);
  return e != 0 ? e : skew_mode_duo(mode);
}
int fa_debug_captured_queues(int device) { return g_queue_slots[device].taken(); }
#endif

int fa_debug_set_wait_status(int32_t device, int32_t code) {
  FA_REQUIRE(device >= 0 && device < 1024, "device ordinal out of range");
  g_host_wait[device] = code;
  return FA_OK;
}

size_t fa_sizeof_args(int which) {
  switch (which) {
    case 0: return sizeof(fa_attn_args);
    case 1: return sizeof(fa_decode_args);
    case 2: return sizeof(fa_int8_args);
    case 3: return sizeof(fa_rotary_args);
  }
  return 0;
}

}  // extern "C"
