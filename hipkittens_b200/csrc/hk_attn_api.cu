// Host side of libhk_attn: argument validation, TMA descriptors, launches. C ABI in include/hk_attn.h.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "../../include/hk_attn.h"
#include "attn_bwd_sm100.cuh"
#include "attn_fwd_sm100.cuh"
#include "dependent_launch.cuh"
#include "key_padding_sm100.cuh"
#include "paged_decode_sm100.cuh"
#include "paged_kv_append_sm100.cuh"
#include "rotary_sm100.cuh"

namespace {

constexpr int kMaxDevices = 64;

thread_local char g_cuda_err[256] = "";
std::atomic<unsigned long long> g_launches{0};

int cuda_fail(cudaError_t e, const char* what) {
  cudaGetLastError();  // reported here, and not once more by the caller's next check
  snprintf(g_cuda_err, sizeof(g_cuda_err), "%s: %s", what, cudaGetErrorString(e));
  return HK_ECUDA;
}
#define HK_CUDA(call)                                   \
  do {                                                  \
    cudaError_t e__ = (call);                           \
    if (e__ != cudaSuccess) return cuda_fail(e__, #call); \
  } while (0)

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                   CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                   CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess) p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// Per-device state: SM count, the device status word, one-time kernel attribute set-up.
struct DeviceState {
  std::mutex mu;
  bool ready = false;     // set once init_device succeeded; a failed attempt is retried by the next call
  int sm_count = 0;
  int cc_major = 0;
  hk::DecodeLimits decode;
  int bwd_clusters[hk::kMaxDkdvSplit + 1] = {};  // clusters of so many dK/dV CTAs that the device holds at once
  int* status = nullptr;       // the status word, device address (kernels write it only when something went wrong)
  int* status_host = nullptr;  // ... and host address: mapped memory, so that reading it needs no copy
};
DeviceState g_dev[kMaxDevices];

template <int D, bool CAUSAL, bool DEP>
int prepare_fwd_kernel() {
  auto* fn = hk::attn_fwd_kernel<D, CAUSAL, DEP>;
  HK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, hk::FwdSmem<D, CAUSAL>::kDynBytes));
  cudaFuncAttributes attr;
  HK_CUDA(cudaFuncGetAttributes(&attr, fn));
  // The kernel re-balances registers between warpgroups (208 per softmax thread, 88 per producer thread);
  // that only adds up if it was compiled to exactly kFwdRegsAtLaunch registers per thread at launch.
  // Refuse to launch otherwise: a register pool that is too small would block the re-allocation forever.
  if (attr.numRegs != hk::kFwdRegsAtLaunch) {
    snprintf(g_cuda_err, sizeof(g_cuda_err), "attn_fwd_kernel<%d,%d,%d> compiled to %d registers, expected %d", D,
             int(CAUSAL), int(DEP), attr.numRegs, hk::kFwdRegsAtLaunch);
    return HK_EUNSUPPORTED;
  }
  return HK_OK;
}

template <int D, bool CAUSAL>
int prepare_fwd_kernels() {
  const int rc = prepare_fwd_kernel<D, CAUSAL, true>();
  if (rc != HK_OK) return rc;
  return prepare_fwd_kernel<D, CAUSAL, hk::kLongFwdDependent<D, CAUSAL>>();
}

template <typename Kernel>
int prepare_bwd_kernel(Kernel* fn, int dyn_bytes, const char* name) {
  HK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn_bytes));
  cudaFuncAttributes attr;
  HK_CUDA(cudaFuncGetAttributes(&attr, fn));
  // the count at launch has to be exact, as for the forward kernel: refuse to launch a build it would not add up in
  if (attr.numRegs != hk::kBwdRegsAtLaunch) {
    snprintf(g_cuda_err, sizeof(g_cuda_err), "%s compiled to %d registers, expected %d", name, attr.numRegs,
             hk::kBwdRegsAtLaunch);
    return HK_EUNSUPPORTED;
  }
  if (attr.sharedSizeBytes != 0) {  // the kernels assume their dynamic shared memory starts the CTA's window
    snprintf(g_cuda_err, sizeof(g_cuda_err), "%s has %zu bytes of static shared memory, expected none", name,
             attr.sharedSizeBytes);
    return HK_EUNSUPPORTED;
  }
  return HK_OK;
}

template <int D, bool CAUSAL>
int prepare_bwd_kernels() {
  int rc = HK_OK;
  for (auto* fn : {hk::attn_bwd_dkdv_kernel<D, CAUSAL, false>, hk::attn_bwd_dkdv_kernel<D, CAUSAL, true>})
    if ((rc = prepare_bwd_kernel(fn, hk::BwdSmem<D>::kDynBytes, "attn_bwd_dkdv_kernel")) != HK_OK) return rc;
  return prepare_bwd_kernel(hk::attn_bwd_dq_kernel<D, CAUSAL>, hk::BwdSmem<D>::kDynBytes, "attn_bwd_dq_kernel");
}

int init_device(int device) {
  DeviceState& st = g_dev[device];
  cudaDeviceProp prop;
  HK_CUDA(cudaGetDeviceProperties(&prop, device));
  st.sm_count = prop.multiProcessorCount;
  st.cc_major = prop.major;
  if (prop.major != 10) {
    snprintf(g_cuda_err, sizeof(g_cuda_err), "device %d is sm_%d%d; this library needs sm_100", device, prop.major,
             prop.minor);
    return HK_EUNSUPPORTED;
  }
  int rc;
  if ((rc = prepare_fwd_kernels<128, false>()) != HK_OK) return rc;
  if ((rc = prepare_fwd_kernels<128, true>()) != HK_OK) return rc;
  if ((rc = prepare_fwd_kernels<64, false>()) != HK_OK) return rc;
  if ((rc = prepare_fwd_kernels<64, true>()) != HK_OK) return rc;
  if ((rc = hk::prepare_decode_kernels(g_cuda_err, sizeof(g_cuda_err), st.sm_count, &st.decode)) != HK_OK) return rc;
  if ((rc = prepare_bwd_kernels<128, false>()) != HK_OK) return rc;
  if ((rc = prepare_bwd_kernels<128, true>()) != HK_OK) return rc;
  if ((rc = prepare_bwd_kernels<64, false>()) != HK_OK) return rc;
  if ((rc = prepare_bwd_kernels<64, true>()) != HK_OK) return rc;
  for (int n = 2; n <= hk::kMaxDkdvSplit; ++n)
    st.bwd_clusters[n] = hk::clusters_held(hk::attn_bwd_dkdv_kernel<128, true, true>, hk::kBwdThreads, hk::BwdSmem<128>::kDynBytes, n);
  // the one allocation this library makes: the status word (last, so that a failure above leaves nothing behind). It
  // lies in mapped host memory: a blocking call reads it after its synchronisation, and a 4-byte copy from device
  // memory to a pageable variable took 18 us of every one of them.
  void* word = nullptr;
  HK_CUDA(cudaHostAlloc(&word, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable));
  *static_cast<volatile int*>(word) = 0;
  void* dev_word = nullptr;
  cudaError_t e = cudaHostGetDevicePointer(&dev_word, word, 0);
  if (e != cudaSuccess) {
    cudaFreeHost(word);
    return cuda_fail(e, "cudaHostGetDevicePointer(status word)");
  }
  st.status_host = static_cast<int*>(word);
  st.status = static_cast<int*>(dev_word);
  return HK_OK;
}

// Makes a device current for the duration of one entry point and puts the caller's current device back when the
// entry point returns (the reference launcher never touches the current device; a torch program whose current
// device is another GPU must not find it changed).
class DeviceScope {
 public:
  DeviceScope() = default;
  DeviceScope(const DeviceScope&) = delete;
  DeviceScope& operator=(const DeviceScope&) = delete;
  ~DeviceScope() {
    if (prev_ >= 0 && prev_ != cur_) cudaSetDevice(prev_);
  }
  // Switches to `device` (< 0: stay on the current one) and reports the index in use through *resolved.
  int enter_raw(int device, int* resolved) {
    HK_CUDA(cudaGetDevice(&prev_));
    if (device < 0) device = prev_;
    if (device >= kMaxDevices) return HK_EINVAL;
    if (device != prev_) HK_CUDA(cudaSetDevice(device));
    cur_ = device;
    *resolved = device;
    return HK_OK;
  }
  // enter_raw plus the device's state, initialised on first use. A failed initialisation is not remembered: the
  // next call tries again (the failing thread finds the reason in hk_last_cuda_error()).
  int enter(int device, DeviceState** out) {
    int rc = enter_raw(device, &device);
    if (rc != HK_OK) return rc;
    DeviceState& st = g_dev[device];
    {
      std::lock_guard<std::mutex> lock(st.mu);
      if (!st.ready) {
        rc = init_device(device);
        if (rc != HK_OK) return rc;
        st.ready = true;
      }
    }
    *out = &st;
    return HK_OK;
  }

 private:
  int prev_ = -1, cur_ = -1;
};

#ifdef HK_TRACE
long long* g_trace_buf = nullptr;
int g_trace_bwd_kernel = 0;  // which backward kernel stamps: 0 = dK/dV, 1 = dQ
#endif

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int unsupported_decode_shape(int S, int H_KV, int max_pages) {
  snprintf(g_cuda_err, sizeof(g_cuda_err),
           "paged decode supports S <= 65535, H_KV <= 65535 and max_pages_per_seq <= %d (got S=%d, H_KV=%d, "
           "max_pages_per_seq=%d)", hk::kMaxCombineSplits * hk::kChunkPagesMin, S, H_KV, max_pages);
  return HK_EUNSUPPORTED;
}

// Device status word -> HK_* code.
int status_to_code(int word) {
  switch (word) {
    case hk::kStatusOk: return HK_OK;
    case hk::kStatusSmemAlign: return HK_EUNSUPPORTED;
    case hk::kStatusBadPage: return HK_EBADPAGE;
    case hk::kStatusBadLen: return HK_EBADLEN;
    default: return HK_ETIMEOUT;
  }
}

// 4-D map over a contiguous bf16 [B, N, heads, D] tensor, box = 64 columns x 1 head x 128 rows,
// 128-byte swizzle (rows of the box are 128 B, the layout tcgen05 descriptors expect).
// `st` = element strides of the batch, sequence and head dimensions (the D dimension is contiguous); every
// stride must be a multiple of 8 elements (16 bytes), which TMA requires.
int make_bnhd_map(CUtensorMap* map, const void* base, int B, int N, int heads, int D, const long long* st,
                  int box_rows = hk::kBlockM) {
  EncodeTiledFn enc = get_encode();
  if (!enc) {
    snprintf(g_cuda_err, sizeof(g_cuda_err), "cuTensorMapEncodeTiled not available from the driver");
    return HK_ECUDA;
  }
  cuuint64_t dims[4] = {cuuint64_t(D), cuuint64_t(heads), cuuint64_t(N), cuuint64_t(B)};
  cuuint64_t strides[3] = {cuuint64_t(st[2]) * 2, cuuint64_t(st[1]) * 2, cuuint64_t(st[0]) * 2};
  cuuint32_t box[4] = {64, 1, cuuint32_t(box_rows), 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  auto encode = [&] {
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = encode();
  if (r == CUDA_ERROR_INVALID_CONTEXT) {
    // a thread that has made no runtime call yet (autograd's) has no current context: let the runtime bind the
    // device's own and try again. cudaSetDevice does that and, unlike cudaFree(nullptr), leaves a graph alone that
    // some thread is capturing at the time.
    int device = 0;
    HK_CUDA(cudaGetDevice(&device));
    HK_CUDA(cudaSetDevice(device));
    r = encode();
  }
  if (r != CUDA_SUCCESS) {
    snprintf(g_cuda_err, sizeof(g_cuda_err), "cuTensorMapEncodeTiled failed with CUresult %d", int(r));
    return HK_ECUDA;
  }
  return HK_OK;
}

__global__ void bounded_wait_selftest_kernel(int* status, unsigned long long limit_ns) {
  __shared__ uint64_t bar;
  __shared__ uint32_t abort_flag;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    hk::ptx::mbar_init(&bar, 1);
    hk::ptx::fence_mbar_init();
  }
  __syncthreads();
  // the limit is given in nanoseconds; 2 cycles per nanosecond is the SM's maximum clock, rounded up
  const bool ok = hk::ptx::mbar_wait(&bar, 0, &abort_flag, limit_ns * 2);  // nobody ever arrives
  if (!ok && threadIdx.x == 0) atomicCAS(status, hk::kStatusOk, hk::kStatusTimeout);
}

// Whether an attention kernel is launched so that it may start under the tail of the one before it: up to 100 tiles per CTA
// (two heads x 128 x 128 in the forward, one in the backward), where a launch and a prologue are a visible share of it.
// The tiles are counted as if nothing were masked. A causal call has about half of them, and a paged one those of its
// contexts, which the host does not know, and not of its block table's width: such calls are launched the ordinary way
// from half the time on, or earlier.
// us per call in a loop, dependent / ordinary, at 28, 62, 111, 221 and 443 tiles per CTA (H32/8 D128, B1 N2048, N3072, N4096,
// B2 and B4 N4096): non-causal 65.8 / 67.9, 134.8 / 136.8, 232.0 / 233.7, 415.7 / 417.0, 830.7 / 830.1; causal
// 39.0 / 40.3, 77.2 / 79.4, 117.7 / 120.4, 230.7 / 229.8, 456.6 / 452.8. Append and paged chunk, 8 x 512 tokens on contexts
// of 4096 (221 tiles): 487.8 / 479.2, and so the line is no higher.
bool short_kernel(long long tiles, int grid) { return tiles <= 100ll * grid; }

// Units of a causal sweep group that has fewer items (`per_unit` each) than the GPU has SMs: the fewest of what fills one to
// four rounds, or all units, that need the fewest rounds. Larger groups stay as they are.
int group_for_fewest_rounds(long long u, long long units, long long per_unit, long long sms) {
  u = std::max(1ll, std::min(u, units));
  if (u == units || u * per_unit >= sms) return int(u);
  auto rounds = [&](long long n) {
    return units / n * ((n * per_unit + sms - 1) / sms) + (units % n * per_unit + sms - 1) / sms;
  };
  for (long long k = 1; k <= 5; ++k) {
    const long long n = k == 5 ? units : std::min(units, k * sms / per_unit);
    if (n > u && rounds(n) < rounds(u)) u = n;
  }
  return int(u);
}

template <int D, bool CAUSAL>
int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to,
               const hk::FwdParams& p, int grid, cudaStream_t stream) {
  const int nk_tiles = (p.NK + hk::kBlockN - 1) / hk::kBlockN;
  const bool early = short_kernel(1ll * p.n_items * nk_tiles, grid);
  auto* fn = early ? hk::attn_fwd_kernel<D, CAUSAL, true> : hk::attn_fwd_kernel<D, CAUSAL, hk::kLongFwdDependent<D, CAUSAL>>;
  HK_CUDA(hk::launch_dependent(early, fn, grid, hk::kFwdThreads, hk::FwdSmem<D, CAUSAL>::kDynBytes, stream, tq, tk, tv, to, p));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return HK_OK;
}

// Sets the fields that say how a kernel's `n_items` work items are dealt to `grid` CTAs - one group (everything)
// unless causal, where a group is `group_units` units of `per_unit` items each - and the divisors of the item
// decode: `per_unit` items per (batch, kv-head) unit, `per_pos` of them per key block or query tile (1 in the dK/dV
// kernel, G in the dQ kernel), `inner` the dQ kernel's second divisor.
void set_bwd_decode(hk::BwdParams& p, int per_unit, int per_pos, int inner, int grid, bool causal) {
  p.group_items = causal ? p.group_units * per_unit : p.n_items;
  const int n_groups = (p.n_items + p.group_items - 1) / p.group_items;
  p.rounds_per_group = (p.group_items + grid - 1) / grid;
  p.total_rounds = p.rounds_per_group * n_groups;
  const int units = p.B * p.H_KV;
  p.G = p.H / p.H_KV;
  p.last_group = (units - 1) / p.group_units;
  p.fd_rounds = hk::FastDiv(p.rounds_per_group);
  p.fd_hkv = hk::FastDiv(p.H_KV);
  p.fd_unit = hk::FastDiv(per_unit);
  p.fd_inner = hk::FastDiv(inner);
  p.fd_group = hk::FastDiv(p.group_units * per_unit);
  p.fd_in_grp = hk::FastDiv(p.group_units * per_pos);
  p.fd_in_grp_last = hk::FastDiv((units - p.last_group * p.group_units) * per_pos);
}

// Whether the causal dK/dV kernel takes its key blocks in pairs (j, nbk - 1 - j), which all cost the same, or singly, the
// longest of all units first, which leaves no round badly filled whatever their number.
// Pairs lose the idle part of their last round, and about half of what the missing partner of a middle block (odd
// counts) leaves idle; the other half is made up by CTAs that drift apart. Single blocks run through many units at a
// time, so a unit's Q and dO, which its blocks share, come from HBM once the units in flight hold more than L2 keeps.
// The line is where the two losses meet, fitted to 581 measured shapes (D 64 and 128, 4 to 314 units, 2 to 68 blocks,
// groups of 1 to 8, pairs 0.61 to 1.00 full): in dK/dV and dQ together a shape takes 0.1 % longer than with the better
// dealing on average, 2.7 % at worst; always pairs would be 25 % off at worst, always single blocks 10 %. At most 5 %
// idle stay in pairs, where single blocks gain 2.6 % at best.
// us, pairs / single: 12 blocks (B2 N384 H8/2 D128) 34.6 / 25.1 and B4 N4096 H32/8 D128 (pairs 0.865 full, 256 MB of Q
// and dO) 920 / 859, dK/dV alone; with dQ, D128 H16/4: B48 N2048 (0.943 full, 768 MB) 2467 / 2680, B24 N2048 (0.865,
// 384 MB) 1280 / 1310, B24 N512 (0.649, 96 MB) 152 / 130.
bool deal_in_pairs(int units, int G, int N, int nbk, int D, int sm_count) {
  const long long pairs = 1ll * units * ((nbk + 1) / 2), rounds = (pairs + sm_count - 1) / sm_count;
  const double slots = double(rounds * sm_count);
  const double idle = 1.0 - 0.5 * (double(pairs) + 0.5 * units * nbk) / slots;
  constexpr double kKept = 70.0 * (1 << 20);                              // what of the 126 MB of L2 serves Q and dO
  const int in_flight = units < sm_count ? units : sm_count;
  const double bytes = 4.0 * in_flight * G * N * D;                       // their Q and dO
  const double missed = bytes > kKept ? 1.0 - kKept / bytes : 0.0;        // share of the reads that go to HBM
  const double unshared = std::sqrt(double(in_flight) / double(sm_count));  // few units: their blocks run side by side
  const double lost = (D == 128 ? 0.22 : 0.13) * missed * unshared;       // a D = 64 tile has half the bytes
  return idle <= (lost > 0.05 ? lost : 0.05);
}

// How many CTAs share a key block of the dK/dV kernel: with few K/V heads there are few blocks, each with all query tiles of
// the group's heads, and most SMs would have none. Estimated in (query tile, key block) pairs (about 2 us each): a CTA
// costs its pairs and 2 more, one of a cluster of n 5 + 0.75 n more (launch, first loads, the merge); a call ends when its
// longest CTA does, when the clusters that the device holds at once are through, or when all SMs have done dK/dV and dQ
// (half the time per pair), whichever is last. Fitted to 61 shapes of 1 to 300 blocks: the estimate's choice takes 1.5 %
// longer than the best on average, never to split 20 %. us per backward, 1 / chosen: B1 N1024 H8/1 D128 causal 108 / 33 (8),
// B1 N4096 H8/1 D128 488 / 214 (4), B1 N8192 H8/1 D128 causal 936 / 423 (3), B1 N2048 H8/1 D64 causal 164 / 38 (8),
// B2 N384 H8/2 D128 causal 28 / 21 (4), B2 N1024 H16/4 D128 87 / 71 (2).
// A block's sums are split in other places than those of a call that does not split it, so a batch element's dK and dV are not
// those of the same element in a batch, or a shard, of another size to the last bit. Two limits keep that to the calls that
// gain most, and cost the others what they would gain: causal calls take no pairs of CTAs, and clusters of several waves have
// to take half the time. us per backward in a loop, 1 / 2 / 3 / 4 CTAs per block: causal B1 N2048 H16/4 D128 131 / 90 / 81 /
// 84, B1 N2944 H16/4 D64 149 / 101 / 107 / 108, B1 N1536 H24/8 D128 87 / 68 / 90 / 93, B2 N2048 H16/4 D128 163 / 126 / 152 /
// 163, B1 N3000 H32/8 D64 193 / 185 / 214 / 222 (all stay whole). Without a causal mask they cost nothing: B1 N2944 H16/4 D128
// 244 / 257 / 244 / 235, B2 N2048 H16/4 D128 204 / 220 / 240 / 252, B1 N4096 H32/4 D128 825 / 844 / 856 / 873.
int dkdv_split(int units, int G, int N, int NK, bool causal, int sm_count, const int* clusters) {
  const int nbq = (N + hk::kBlockM - 1) / hk::kBlockM, nbk = (NK + hk::kBlockN - 1) / hk::kBlockN;
  if (1ll * units * nbk > 2ll * sm_count) return 1;
  const int items = units * nbk;
  double longest = 0, pairs = 0;  // of one unit, as if no keys were padding
  for (int j = 0; j < nbk; ++j) {
    const long long first = causal ? 1ll * j * hk::kBlockN - (NK - N) : 0;  // the first query that sees the block
    const long long tiles = nbq - (first > 0 ? first / hk::kBlockM : 0);
    const double n = tiles > 0 ? double(G) * tiles : 0;
    longest = n > longest ? n : longest;
    pairs += n;
  }
  const double dq_work = 0.5 * units * pairs + 1.0 * units * G * nbq;
  auto estimate = [&](int n, int held) {
    const double more = n == 1 ? 2.0 : 5.0 + 0.75 * n;
    const double top = std::ceil(longest / n) + more, mean = pairs / nbk / n + more;
    double span;
    if (causal) span = std::max(top, items * mean / held + (items > held ? 0.5 * mean : 0.0));
    else span = std::ceil(double(items) / held) * top;
    return std::max(span, (items * n * mean + dq_work) / sm_count);
  };
  const double alone = estimate(1, sm_count);
  int best = 1;
  double best_time = alone;
  for (int n = causal ? 3 : 2; n <= hk::kMaxDkdvSplit; ++n) {
    if (clusters[n] == 0) continue;
    const double t = estimate(n, clusters[n]);
    if (t < best_time && t < (items <= clusters[n] ? 0.95 : 0.5) * alone) {
      best = n;
      best_time = t;
    }
  }
  return best;
}

// Deals the key blocks to CTAs (dkdv_item_for_round); returns the grid.
template <int D, bool CAUSAL>
int deal_dkdv(hk::BwdParams& p, int nbk, int sm_count, const int* clusters) {
  const int units = p.B * p.H_KV;
  p.n_items = units * nbk;
  p.split = dkdv_split(units, p.H / p.H_KV, p.N, p.NK, CAUSAL, sm_count, clusters);
  if (p.split > 1) {  // one cluster per item, the longest first
    p.fd_split = hk::FastDiv(p.split);
    set_bwd_decode(p, nbk, 1, 1, p.n_items, false);
    p.n_pairs = 0;
    p.fd_pairs = hk::FastDiv(units);
    p.total_rounds = 1;
    return p.n_items * p.split;
  }
  int grid = p.n_items < sm_count ? p.n_items : sm_count;
  set_bwd_decode(p, nbk, 1, 1, grid, false);
  p.n_pairs = 0;
  if (CAUSAL) {
    if (deal_in_pairs(units, p.H / p.H_KV, p.N, nbk, D, sm_count)) {
      const int per_unit = (nbk + 1) / 2;
      p.n_pairs = units * per_unit;
      p.fd_pairs = hk::FastDiv(per_unit);
      grid = p.n_pairs < sm_count ? p.n_pairs : sm_count;
      p.total_rounds = 2 * ((p.n_pairs + grid - 1) / grid);
    } else {
      p.fd_pairs = hk::FastDiv(units);
      p.total_rounds = (p.n_items + grid - 1) / grid;
    }
  }
  return grid;
}

// The dQ kernel may run on the SMs that the dK/dV kernel (of `grid` CTAs) leaves, or behind it. Returns its CTAs, negative if
// they wait for the dK/dV kernel.
//  * With a CTA for every SM those that find an SM early do their share and the others start when the dK/dV kernel has
//    ended. That fills gaps (us behind / beside, in a loop: B1 N512 H8/8 D128 23.6 / 15.3, B4 N1024 H12 D64 85 / 70, B6 N567
//    H4 D128 causal 29.3 / 23.8, B1 N2560 H8 D64 causal 56.4 / 42.7), but two kernels at a time also cost the key blocks that
//    are still running: longer calls are better off one after the other (D128 B2 N4096 H4 193 / 203, B13 N505 H32/8 203 /
//    215; B1 N4096 H32/8 causal 392 / 408; D64 B6 N7554 H6/2 1 981 / 2 067). So are those whose key blocks all run long, and
//    as long, while dQ comes to them: groups of heads on blocks for 5/8 of a round of the SMs and more (B5 N1408 H8/2 D64 101
//    / 118, B4 N940 H16/8 D64 89 / 105, B3 N1405 H16/4 D64 116 / 129) or with a last round more than a quarter full (B6
//    N1129 H16/4 D64 164 / 189), single heads with one more than 0.6 full (B8 N2176 H4 D64 166 / 182; 0.4 full: B9 N1100 H8
//    D128 180 / 167) and no key lengths, which leave rounds that are not known here (B16 N512 H16 D64 97 / 86 when padded);
//    of causal blocks, whose lengths differ, groups of 3 heads and more on 3/4 to 1.4 rounds (B5 N300 H32/8 53 / 61, B7
//    N457 H32/4 104 / 117, B2 N1280 H64/8 D128 233 / 259, B3 N2073 H16/4 D64 151 / 162) unless there are 24 lengths of them
//    (B5 N4218 H4/1 D64 254 / 241); either with groups of 8 from 3/8 of a round on (B4 N295 H64/8 D64 68 / 81, B10 N256
//    H32/4 D64 causal 49 / 55); and pairs (B9 N2857 H8/4 D64 348 / 360; 0.98 to 1.11 of the time behind). Of 2465 shapes of
//    20 to 600 us, 5 take more than 2.5 % longer than behind in a loop, 5 % at most (121 and 21 % without these lines);
//    what the lines give up of calls waited for one by one is 0.1 % on average.
//  * When the last round of key blocks leaves many SMs free, these are dealt all of dQ, if that is estimated to end sooner: in
//    the pairs of dkdv_split, a dQ item costs 1 and 0.45 per pair alone, 1.5 and 0.65 beside dK/dV. us behind / all SMs /
//    the free ones (D128 unless said), calls waited for one by one: B5 N512 H32/8 108 / 101 / 78, B1 N2500 H32/8 420 / 383 / 285,
//    B11 N1000 H16/2 D64 263 / 281 / 217, B6 N900 H12/4 141 / 149 / 130, B4 N293 H16 D64 32 / 30 / 25. In a loop the next call
//    fills such SMs too, and less or nothing is left of it: B2 N1511 H24/8 D64 158 / 160 / 139 one by one, 152 / 160 / 156 in a
//    loop, B1 N1408 H24/8 D128 101 / 100 / 88, 97 / 99 / 103.
template <int D, bool CAUSAL>
int dq_ctas(const hk::BwdParams& p, int nbq, int nbk, int grid, int sm_count) {
  const long long items = 1ll * p.B * p.H * nbq;
  const int all = items < sm_count ? int(items) : sm_count;
  double round = 0, pairs = nbk;    // of a round of dK/dV, of an item of dQ
  long long rounds = 1, last = -1;  // last: CTAs busy in the last round; -1: blocks of every length, in no rounds
  if (p.split > 1) {
    if (!CAUSAL) {
      round = std::ceil(double(p.G) * nbq / p.split) + 5.0 + 0.75 * p.split;
      last = grid;
    }
  } else if (!CAUSAL || p.n_pairs > 0) {
    const long long units = CAUSAL ? p.n_pairs : p.n_items;
    round = CAUSAL ? p.G * (nbq + 1.0) + 4.0 : double(p.G) * nbq + 2.0;
    if (CAUSAL) pairs = 0.5 * (nbk + 1);
    rounds = (units + grid - 1) / grid;
    last = units - (rounds - 1) * grid;
  }
  const long long free = sm_count - last;
  if (last >= 0 && free > 0) {
    if (items <= free) return all;
    const double behind = rounds * round + std::ceil(double(items) / sm_count) * (1.0 + 0.45 * pairs);
    const double beside = (rounds - 1) * round + std::ceil(double(items) / double(free)) * (1.5 + 0.65 * pairs);
    if (std::max(rounds * round, beside) < 0.97 * behind) return int(free);
  }
  const long long tiles = 1ll * p.B * p.H * nbq * nbk;
  const bool long_call = tiles > (D == 64 ? 300ll : CAUSAL ? 120ll : 40ll) * grid;
  bool held_up = p.n_pairs > 0;  // the key blocks, by dQ beside them
  if (p.split == 1 && p.n_pairs == 0) {
    const double full = double(p.n_items) / sm_count, from = p.G >= 8 ? 3.0 / 8 : CAUSAL ? 3.0 / 4 : 5.0 / 8;
    if (CAUSAL) held_up = p.G >= 3 && full > from && full <= 1.4 && nbk < 24;
    else if (rounds == 1) held_up = p.G >= 2 && full > from;
    else held_up = p.G == 1 ? !p.kv_lens && last > 0.6 * sm_count : last > 0.25 * sm_count;
  }
  return long_call || held_up ? -all : all;
}

template <int D, bool CAUSAL>
int launch_bwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
               hk::BwdParams p, int B, int N, int NK, int H, int H_KV, bool dq_beside, int sm_count,
               const int* clusters, cudaStream_t stream) {
  const int nbq = (N + hk::kBlockM - 1) / hk::kBlockM;   // query tiles
  const int nbk = (NK + hk::kBlockN - 1) / hk::kBlockN;  // key blocks
  if (static_cast<long long>(B) * H * nbq > 0x3fffffffll || static_cast<long long>(B) * H_KV * nbk > 0x3fffffffll)
    return HK_EINVAL;  // work items are indexed with int
  int grid = deal_dkdv<D, CAUSAL>(p, nbk, sm_count, clusters);
#ifdef HK_TRACE
  long long* const trace_buf = p.trace;
  p.trace = g_trace_bwd_kernel == 0 ? trace_buf : nullptr;
#endif
  const long long tiles = 1ll * B * H * nbq * nbk;
  const auto dkdv = p.split > 1 ? hk::attn_bwd_dkdv_kernel<D, CAUSAL, true> : hk::attn_bwd_dkdv_kernel<D, CAUSAL, false>;
  HK_CUDA(hk::launch_dependent(short_kernel(tiles, grid), dkdv, grid, hk::kBwdThreads, hk::BwdSmem<D>::kDynBytes, stream,
                               hk::ClusterX{unsigned(p.split)}, tq, tk, tv, tdo, p));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  const int ctas = dq_ctas<D, CAUSAL>(p, nbq, nbk, grid, sm_count);
  p.dq_waits = !dq_beside || ctas < 0;
  p.n_items = B * H * nbq;
  grid = !p.dq_waits ? ctas : (p.n_items < sm_count ? p.n_items : sm_count);
  set_bwd_decode(p, (H / H_KV) * nbq, H / H_KV, CAUSAL ? H / H_KV : nbq, grid, CAUSAL);
#ifdef HK_TRACE
  p.trace = g_trace_bwd_kernel == 1 ? trace_buf : nullptr;
#endif
  HK_CUDA(hk::launch_dependent(!p.dq_waits || short_kernel(tiles, grid), hk::attn_bwd_dq_kernel<D, CAUSAL>, grid, hk::kBwdThreads,
                               hk::BwdSmem<D>::kDynBytes, stream, tq, tk, tv, tdo, p));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return HK_OK;
}

}  // namespace

extern "C" {

#ifdef HK_TRACE
void hk_debug_set_trace(long long* buf) { g_trace_buf = buf; }
void hk_debug_set_trace_bwd_kernel(int which) { g_trace_bwd_kernel = which; }
#endif

int hk_attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B, int N, int H, int H_KV,
                int D, int causal, float softmax_scale, int device, void* cuda_stream) {
  const long long qs[3] = {(long long)N * H * D, (long long)H * D, D};
  const long long ks[3] = {(long long)N * H_KV * D, (long long)H_KV * D, D};
  return hk_attn_fwd_strided(q, k, v, o, lse, B, N, H, H_KV, D, qs, ks, ks, causal, softmax_scale, device, cuda_stream);
}

int hk_attn_fwd_strided(const void* q, const void* k, const void* v, void* o, float* lse, int B, int N, int H,
                        int H_KV, int D, const long long* q_strides, const long long* k_strides,
                        const long long* v_strides, int causal, float softmax_scale, int device,
                        void* cuda_stream) {
  return hk_attn_fwd_varlen(q, k, v, o, lse, B, N, H, H_KV, D, q_strides, k_strides, v_strides, nullptr, causal,
                            softmax_scale, device, cuda_stream);
}

int hk_attn_fwd_varlen(const void* q, const void* k, const void* v, void* o, float* lse, int B, int N, int H,
                       int H_KV, int D, const long long* q_strides, const long long* k_strides,
                       const long long* v_strides, const int32_t* kv_lens, int causal, float softmax_scale,
                       int device, void* cuda_stream) {
  return hk_attn_fwd_cross(q, k, v, o, lse, B, N, N, H, H_KV, D, q_strides, k_strides, v_strides, kv_lens, causal,
                           softmax_scale, device, cuda_stream);
}

// Shared tail of the forward entries. Contiguous K/V: k, v are [B, NK, H_KV, D] with strides; paged K/V
// (block_table != null): k, v are the page pools [num_pages, 16, H_KV, D] and NK = max_pages * 16.
static int fwd_launch(const void* q, const void* k, const void* v, void* o, float* lse, int B, int N, int NK, int H,
                      int H_KV, int D, const long long* q_strides, const long long* k_strides,
                      const long long* v_strides, const int32_t* kv_lens, const int32_t* block_table, int max_pages,
                      int num_pages, int causal, float softmax_scale, int device, void* cuda_stream) {
  DeviceState* st = nullptr;
  DeviceScope scope;
  int rc = scope.enter(device, &st);
  if (rc != HK_OK) return rc;

  CUtensorMap tq, tk, tv, to;
  if ((rc = make_bnhd_map(&tq, q, B, N, H, D, q_strides)) != HK_OK) return rc;
  {
    // O is written by TMA from a swizzled staging tile, a [128 rows x 64 columns] box at a time
    const long long os[3] = {(long long)N * H * D, (long long)H * D, D};
    if ((rc = make_bnhd_map(&to, o, B, N, H, D, os)) != HK_OK) return rc;
  }
  if (block_table) {
    // the pools as [num_pages * 16 rows, H_KV, D], fetched one page (16 rows) at a time
    const long long ps[3] = {(long long)num_pages * 16 * H_KV * D, (long long)H_KV * D, D};
    if ((rc = make_bnhd_map(&tk, k, 1, num_pages * 16, H_KV, D, ps, 16)) != HK_OK) return rc;
    if ((rc = make_bnhd_map(&tv, v, 1, num_pages * 16, H_KV, D, ps, 16)) != HK_OK) return rc;
  } else {
    if ((rc = make_bnhd_map(&tk, k, B, NK, H_KV, D, k_strides)) != HK_OK) return rc;
    if ((rc = make_bnhd_map(&tv, v, B, NK, H_KV, D, v_strides)) != HK_OK) return rc;
  }

  const int G = H / H_KV;
  const int nqb = (N + hk::kBlockM - 1) / hk::kBlockM;
  hk::FwdParams p;
  p.o = static_cast<__nv_bfloat16*>(o);
  p.lse = lse;
  p.B = B;
  p.N = N;
  p.NK = NK;
  p.H = H;
  p.H_KV = H_KV;
  p.pair_heads = (G % 2 == 0) ? 1 : 0;
  {
    // causal sweep groups: as many (batch, kv-head) units as keep K and V of the group within HK_GROUP_MB (the
    // whole tensor at once re-reads K/V 2.6 times at N = 8192)
    const long long kv_bytes = 4ll * NK * D;  // K and V of one unit, bf16
#ifndef HK_GROUP_MB
#define HK_GROUP_MB 32
#endif
    long long u = (static_cast<long long>(HK_GROUP_MB) << 20) / kv_bytes;
    // A group is dealt in rounds of its own, so one with fewer items than the GPU has SMs leaves the others idle: few
    // queries on many keys, or on a block table that is wide for its contexts (which the host does not know).
    // us, before / now, H64/8 D128 paged: 1 x 64 queries on 1000 keys, table of 8192 pages 71 / 23; 4 x 512 on 8192, 8192
    // pages 1831 / 514; 16 x 512 on 2048, 2048 pages 994 / 482; H32/8 2 x 128 on 16000, 1000 pages 471 / 251. Contiguous, causal:
    // 64 queries on 65536 keys 3449 / 890.
    const long long per_unit = p.pair_heads ? 1ll * (G / 2) * nqb : 1ll * G * ((nqb + 1) / 2);
    p.group_units = group_for_fewest_rounds(u, 1ll * B * H_KV, per_unit, st->sm_count);
  }
  if (static_cast<long long>(B) * H * nqb > 0x3fffffffll) return HK_EINVAL;  // work items are indexed with int
  p.n_items = p.pair_heads ? B * H_KV * (G / 2) * nqb : B * H_KV * G * ((nqb + 1) / 2);
  p.scale = softmax_scale > 0.f ? softmax_scale : 1.0f / std::sqrt(float(D));
  p.scale_log2 = p.scale * 1.4426950408889634f;
  p.kv_lens = kv_lens;
  p.block_table = block_table;
  p.max_pages = max_pages;
  p.num_pages = num_pages;
  p.status = st->status;
#ifdef HK_TRACE
  p.trace = g_trace_buf;
#endif
  const int grid = p.n_items < st->sm_count ? p.n_items : st->sm_count;
  {
    // rounds in which the items are dealt to the CTAs: one group (everything) unless causal
    const int per_unit = p.n_items / (B * H_KV);
    p.group_items = causal ? p.group_units * per_unit : p.n_items;
    const int n_groups = (p.n_items + p.group_items - 1) / p.group_items;
    p.rounds_per_group = (p.group_items + grid - 1) / grid;
    p.total_rounds = p.rounds_per_group * n_groups;
  }
  hk::set_item_decode(p);
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  if (D == 128) return causal ? launch_fwd<128, true>(tq, tk, tv, to, p, grid, stream)
                              : launch_fwd<128, false>(tq, tk, tv, to, p, grid, stream);
  return causal ? launch_fwd<64, true>(tq, tk, tv, to, p, grid, stream)
                : launch_fwd<64, false>(tq, tk, tv, to, p, grid, stream);
}

int hk_attn_fwd_cross(const void* q, const void* k, const void* v, void* o, float* lse, int B, int N, int NK, int H,
                      int H_KV, int D, const long long* q_strides, const long long* k_strides,
                      const long long* v_strides, const int32_t* kv_lens, int causal, float softmax_scale,
                      int device, void* cuda_stream) {
  if (!q || !k || !v || !o || !lse || !q_strides || !k_strides || !v_strides) return HK_EINVAL;
  if (B <= 0 || N <= 0 || NK <= 0 || H <= 0 || H_KV <= 0) return HK_EINVAL;
  if (D != 64 && D != 128) return HK_EUNSUPPORTED;
  if (H % H_KV != 0) return HK_EINVAL;
  for (int i = 0; i < 3; ++i) {
    const long long s3[3] = {q_strides[i], k_strides[i], v_strides[i]};
    for (long long st_i : s3)
      if (st_i <= 0 || st_i % 8 != 0 || st_i >= (1ll << 39)) return HK_EINVAL;
  }
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o) || (reinterpret_cast<uintptr_t>(lse) & 3))
    return HK_EINVAL;
  return fwd_launch(q, k, v, o, lse, B, N, NK, H, H_KV, D, q_strides, k_strides, v_strides, kv_lens, nullptr, 0, 0,
                    causal, softmax_scale, device, cuda_stream);
}

int hk_attn_fwd_paged(const void* q, const void* k_pages, const void* v_pages, const int32_t* block_table,
                      const int32_t* ctx_lens, void* o, float* lse, int S, int T, int H, int H_KV, int D,
                      int page_size, int max_pages_per_seq, int num_pages, int causal, float softmax_scale,
                      int device, void* cuda_stream) {
  if (!q || !k_pages || !v_pages || !block_table || !ctx_lens || !o || !lse) return HK_EINVAL;
  if (S <= 0 || T <= 0 || H <= 0 || H_KV <= 0 || max_pages_per_seq <= 0 || num_pages <= 0) return HK_EINVAL;
  if ((D != 64 && D != 128) || page_size != 16) return HK_EUNSUPPORTED;
  if (H % H_KV != 0) return HK_EINVAL;
  if (static_cast<long long>(num_pages) * 16 > 0x7fffffffll || static_cast<long long>(max_pages_per_seq) * 16 > 0x3fffffffll)
    return HK_EINVAL;
  if (!aligned16(q) || !aligned16(k_pages) || !aligned16(v_pages) || !aligned16(o) ||
      (reinterpret_cast<uintptr_t>(lse) & 3))
    return HK_EINVAL;
  const long long qs[3] = {(long long)T * H * D, (long long)H * D, D};
  return fwd_launch(q, k_pages, v_pages, o, lse, S, T, max_pages_per_seq * 16, H, H_KV, D, qs, qs, qs, ctx_lens,
                    block_table, max_pages_per_seq, num_pages, causal, softmax_scale, device, cuda_stream);
}

static int prep_launch(const void* o, const void* d_o, float* delta, int B, int N, int H, int D, cudaStream_t stream) {
  const long long rows = static_cast<long long>(B) * N * H;
  if (rows > 0x7fffffffll) return HK_EINVAL;  // rows are indexed with int
  const int rows_per_block = hk::row_pass_rows(D / 8);
  const unsigned blocks = unsigned((rows + rows_per_block - 1) / rows_per_block);
  const auto* po = static_cast<const __nv_bfloat16*>(o);
  const auto* pd = static_cast<const __nv_bfloat16*>(d_o);
  auto* fn = D == 128 ? hk::attn_bwd_prep_kernel<128> : hk::attn_bwd_prep_kernel<64>;
  HK_CUDA(hk::launch_dependent(true, fn, blocks, 256, 0, stream, po, pd, delta, int(rows), N, H, hk::FastDiv(H), hk::FastDiv(N)));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return HK_OK;
}

int hk_attn_bwd_prep(const void* o, const void* d_o, float* delta, int B, int N, int H, int D, int device,
                     void* cuda_stream) {
  if (!o || !d_o || !delta) return HK_EINVAL;
  if (B <= 0 || N <= 0 || H <= 0) return HK_EINVAL;
  if (D != 64 && D != 128) return HK_EUNSUPPORTED;
  if (!aligned16(o) || !aligned16(d_o) || (reinterpret_cast<uintptr_t>(delta) & 3)) return HK_EINVAL;
  DeviceState* st = nullptr;
  DeviceScope scope;
  int rc = scope.enter(device, &st);
  if (rc != HK_OK) return rc;
  return prep_launch(o, d_o, delta, B, N, H, D, static_cast<cudaStream_t>(cuda_stream));
}

int hk_attn_bwd(const void* q, const void* k, const void* v, const void* d_o, const float* lse, const float* delta,
                void* dq, void* dk, void* dv, int B, int N, int H, int H_KV, int D, int causal, float softmax_scale,
                int dq_layout, int device, void* cuda_stream) {
  return hk_attn_bwd_varlen(q, k, v, d_o, lse, delta, dq, dk, dv, B, N, H, H_KV, D, nullptr, causal, softmax_scale,
                            dq_layout, device, cuda_stream);
}

int hk_attn_bwd_varlen(const void* q, const void* k, const void* v, const void* d_o, const float* lse,
                       const float* delta, void* dq, void* dk, void* dv, int B, int N, int H, int H_KV, int D,
                       const int32_t* kv_lens, int causal, float softmax_scale, int dq_layout, int device,
                       void* cuda_stream) {
  return hk_attn_bwd_cross(q, k, v, d_o, lse, delta, dq, dk, dv, B, N, N, H, H_KV, D, kv_lens, causal, softmax_scale,
                           dq_layout, device, cuda_stream);
}

// Element strides of the batch, sequence and head dimensions of the tensors of one backward call.
struct BwdStrides {
  const long long *q, *k, *v, *dq, *dk, *dv;
};

// The addresses from the first byte of an input or output to behind its last, and whether two of them may share memory.
struct Span {
  uintptr_t begin, end;
  Span(const void* p, long long bytes) : begin(reinterpret_cast<uintptr_t>(p)), end(begin + uintptr_t(bytes)) {}
  // of a [B, N, H, D] tensor of 16-bit elements with these strides
  Span(const void* p, const long long* strides, int B, int N, int H, int D)
      : Span(p, 2 * ((B - 1) * strides[0] + (N - 1) * strides[1] + (H - 1) * strides[2] + D)) {}
  bool meets(const Span& o) const { return begin < o.end && o.begin < end; }
};

// Shared tail of the backward entries. o != null: delta is computed here first.
static int bwd_launch(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse,
                      float* delta, void* dq, void* dk, void* dv, int B, int N, int NK, int H, int H_KV, int D,
                      const BwdStrides& s, const int32_t* kv_lens, int causal, float softmax_scale, int device,
                      void* cuda_stream) {
  if (!q || !k || !v || !d_o || !lse || !delta || !dq || !dk || !dv) return HK_EINVAL;
  if (B <= 0 || N <= 0 || NK <= 0 || H <= 0 || H_KV <= 0) return HK_EINVAL;
  if (D != 64 && D != 128) return HK_EUNSUPPORTED;
  if (H % H_KV != 0) return HK_EINVAL;
  for (const long long* s3 : {s.q, s.k, s.v, s.dq, s.dk, s.dv})
    for (int i = 0; i < 3; ++i)
      if (s3[i] <= 0 || s3[i] % 8 != 0 || s3[i] >= (1ll << 39)) return HK_EINVAL;
  if ((o && !aligned16(o)) || !aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(d_o) || !aligned16(dq) || !aligned16(dk) ||
      !aligned16(dv) || (reinterpret_cast<uintptr_t>(lse) & 3) || (reinterpret_cast<uintptr_t>(delta) & 3))
    return HK_EINVAL;
  DeviceState* st = nullptr;
  DeviceScope scope;
  int rc = scope.enter(device, &st);
  if (rc != HK_OK) return rc;

  const long long dos[3] = {(long long)N * H * D, (long long)H * D, D};
  CUtensorMap tq, tk, tv, tdo;
  if ((rc = make_bnhd_map(&tq, q, B, N, H, D, s.q)) != HK_OK) return rc;
  if ((rc = make_bnhd_map(&tk, k, B, NK, H_KV, D, s.k)) != HK_OK) return rc;
  if ((rc = make_bnhd_map(&tv, v, B, NK, H_KV, D, s.v)) != HK_OK) return rc;
  if ((rc = make_bnhd_map(&tdo, d_o, B, N, H, D, dos)) != HK_OK) return rc;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  if (o && (rc = prep_launch(o, d_o, delta, B, N, H, D, stream)) != HK_OK) return rc;

  hk::BwdParams p;
  p.lse = lse;
  p.delta = delta;
  p.dq = static_cast<__nv_bfloat16*>(dq);
  p.dk = static_cast<__nv_bfloat16*>(dk);
  p.dv = static_cast<__nv_bfloat16*>(dv);
  p.dq_stride_b = s.dq[0], p.dq_stride_n = s.dq[1], p.dq_stride_h = s.dq[2];
  p.dk_stride_b = s.dk[0], p.dk_stride_n = s.dk[1], p.dk_stride_h = s.dk[2];
  p.dv_stride_b = s.dv[0], p.dv_stride_n = s.dv[1], p.dv_stride_h = s.dv[2];
  p.B = B;
  p.N = N;
  p.NK = NK;
  p.H = H;
  p.H_KV = H_KV;
  p.n_items = 0;
  {
    // causal sweep groups of the dQ kernel: units whose Q, dO, K and V together stay within ~64 MB of L2, in groups that
    // need the fewest rounds (us per backward, before / now: B1 64 queries on 32768 keys H64/8 D128 894 / 555, B4 200 on 16384
    // H16 D64 587 / 356, B2 512 on 16384 H8 D128 499 / 351)
    const int G = H / H_KV;
    const long long unit_bytes = 4ll * G * N * D + 4ll * NK * D;
    p.group_units = group_for_fewest_rounds((64ll << 20) / unit_bytes, 1ll * B * H_KV,
                                            1ll * G * ((N + hk::kBlockM - 1) / hk::kBlockM), st->sm_count);
  }
  p.scale = softmax_scale > 0.f ? softmax_scale : 1.0f / std::sqrt(float(D));
  p.scale_log2 = p.scale * 1.4426950408889634f;
  p.kv_lens = kv_lens;
  p.status = st->status;
#ifdef HK_TRACE
  p.trace = g_trace_buf;
#endif
  // The dQ kernel starts while the dK/dV kernel is still reading, unless it would write over what that reads: dQ in the place
  // of an input whose rows are read by the CTA that writes there, and before it does (Q and dO; K and V with one tile of
  // each and as many K/V heads as heads), is as good as anywhere else when one kernel follows the other.
  const Span out(dq, s.dq, B, N, H, D);
  const long long stats = 4ll * B * H * N;
  const bool dq_beside = !out.meets({q, s.q, B, N, H, D}) && !out.meets({d_o, dos, B, N, H, D}) &&
                         !out.meets({k, s.k, B, NK, H_KV, D}) && !out.meets({v, s.v, B, NK, H_KV, D}) &&
                         !out.meets({lse, stats}) && !out.meets({delta, stats}) &&
                         !(kv_lens && out.meets({kv_lens, 4ll * B}));
  if (D == 128) return causal ? launch_bwd<128, true>(tq, tk, tv, tdo, p, B, N, NK, H, H_KV, dq_beside, st->sm_count, st->bwd_clusters, stream)
                              : launch_bwd<128, false>(tq, tk, tv, tdo, p, B, N, NK, H, H_KV, dq_beside, st->sm_count, st->bwd_clusters, stream);
  return causal ? launch_bwd<64, true>(tq, tk, tv, tdo, p, B, N, NK, H, H_KV, dq_beside, st->sm_count, st->bwd_clusters, stream)
                : launch_bwd<64, false>(tq, tk, tv, tdo, p, B, N, NK, H, H_KV, dq_beside, st->sm_count, st->bwd_clusters, stream);
}

int hk_attn_bwd_cross(const void* q, const void* k, const void* v, const void* d_o, const float* lse,
                      const float* delta, void* dq, void* dk, void* dv, int B, int N, int NK, int H, int H_KV, int D,
                      const int32_t* kv_lens, int causal, float softmax_scale, int dq_layout, int device,
                      void* cuda_stream) {
  // in the order in which a call that is wrong in several ways is answered
  if (!q || !k || !v || !d_o || !lse || !delta || !dq || !dk || !dv) return HK_EINVAL;
  if (B <= 0 || N <= 0 || NK <= 0 || H <= 0 || H_KV <= 0) return HK_EINVAL;
  if (D != 64 && D != 128) return HK_EUNSUPPORTED;
  if (dq_layout != HK_DQ_BNHD && dq_layout != HK_DQ_BHND) return HK_EINVAL;
  const long long qs[3] = {(long long)N * H * D, (long long)H * D, D};
  const long long ks[3] = {(long long)NK * H_KV * D, (long long)H_KV * D, D};
  const long long dqs[3] = {(long long)N * H * D, D, (long long)N * D};  // [B, H, N, D]
  const BwdStrides s{qs, ks, ks, dq_layout == HK_DQ_BNHD ? qs : dqs, ks, ks};
  return bwd_launch(q, k, v, nullptr, d_o, lse, const_cast<float*>(delta), dq, dk, dv, B, N, NK, H, H_KV, D, s, kv_lens,
                    causal, softmax_scale, device, cuda_stream);
}

int hk_attn_bwd_strided(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse,
                        float* delta, void* dq, void* dk, void* dv, int B, int N, int NK, int H, int H_KV, int D,
                        const long long* q_strides, const long long* k_strides, const long long* v_strides,
                        const long long* dq_strides, const long long* dk_strides, const long long* dv_strides,
                        const int32_t* kv_lens, int causal, float softmax_scale, int device, void* cuda_stream) {
  if (!q_strides || !k_strides || !v_strides || !dq_strides || !dk_strides || !dv_strides) return HK_EINVAL;
  const BwdStrides s{q_strides, k_strides, v_strides, dq_strides, dk_strides, dv_strides};
  return bwd_launch(q, k, v, o, d_o, lse, delta, dq, dk, dv, B, N, NK, H, H_KV, D, s, kv_lens, causal, softmax_scale,
                    device, cuda_stream);
}

int hk_key_padding_lens(const unsigned char* mask, int32_t* lens, int32_t* bad, int B, int N, int device,
                        void* cuda_stream) {
  if (!mask || !lens || !bad || B <= 0 || N <= 0) return HK_EINVAL;
  if ((reinterpret_cast<uintptr_t>(lens) & 3) || (reinterpret_cast<uintptr_t>(bad) & 3)) return HK_EINVAL;
  DeviceState* st = nullptr;
  DeviceScope scope;
  int rc = scope.enter(device, &st);
  if (rc != HK_OK) return rc;
  HK_CUDA(hk::launch_dependent(true, hk::key_padding_lens_kernel, B, 256, 0, static_cast<cudaStream_t>(cuda_stream), mask, lens,
                               bad, N));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return HK_OK;
}

int hk_attn_dq_shuffle(const void* dq_bhnd, void* dq_bnhd, int B, int N, int H, int D, int device,
                       void* cuda_stream) {
  if (!dq_bhnd || !dq_bnhd || dq_bhnd == dq_bnhd) return HK_EINVAL;
  if (B <= 0 || N <= 0 || H <= 0 || D <= 0 || D % 8 != 0) return HK_EINVAL;
  if (!aligned16(dq_bhnd) || !aligned16(dq_bnhd)) return HK_EINVAL;
  DeviceState* st = nullptr;
  DeviceScope scope;
  int rc = scope.enter(device, &st);
  if (rc != HK_OK) return rc;
  const int vec = D / 8;
  const long long rows = static_cast<long long>(B) * N * H, total = rows * vec;
  const long long blocks = (total + 256 * hk::kRowPassUnroll - 1) / (256 * hk::kRowPassUnroll);
  if (blocks > 0x7fffffffll) return HK_EINVAL;
  if ((vec == 8 || vec == 16) && rows > 0x7fffffffll) return HK_EINVAL;  // these index rows with int
  auto* fn = vec == 16 ? hk::attn_dq_shuffle_kernel<16>
                       : (vec == 8 ? hk::attn_dq_shuffle_kernel<8> : hk::attn_dq_shuffle_kernel<0>);
  HK_CUDA(hk::launch_dependent(true, fn, unsigned(blocks), 256, 0, static_cast<cudaStream_t>(cuda_stream),
                               static_cast<const uint4*>(dq_bhnd), static_cast<uint4*>(dq_bnhd), total, N, H, vec,
                               hk::FastDiv(H), hk::FastDiv(N)));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return HK_OK;
}

static int rotary_launch(const void* x, void* o, const void* sin, const void* cos, long long rows, int N, int D,
                         int rotary_dim, int n_div, int pos0, int device, void* cuda_stream) {
  if (!x || !o || !sin || !cos) return HK_EINVAL;
  if (rows <= 0 || N <= 0 || D <= 0 || pos0 < 0) return HK_EINVAL;
  if (rotary_dim <= 0) rotary_dim = D;
  if (D % 8 != 0 || rotary_dim % 16 != 0 || rotary_dim > D) return HK_EUNSUPPORTED;
  if (!aligned16(x) || !aligned16(o) || !aligned16(sin) || !aligned16(cos)) return HK_EINVAL;
  DeviceState* st = nullptr;
  DeviceScope scope;
  int rc = scope.enter(device, &st);
  if (rc != HK_OK) return rc;
  hk::RotaryParams p;
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.o = static_cast<__nv_bfloat16*>(o);
  p.cos = static_cast<const __nv_bfloat16*>(cos);
  p.sin = static_cast<const __nv_bfloat16*>(sin);
  p.rows = rows;
  p.N = N;
  p.D = D;
  p.R = rotary_dim;
  p.n_div = n_div;
  p.pos0 = pos0;
  const long long units = p.rows * (rotary_dim / 16 + (D - rotary_dim) / 8);
  const long long blocks = (units + 255) / 256;
  if (blocks > 0x7fffffffll) return HK_EINVAL;
  HK_CUDA(hk::launch_dependent(true, hk::rotary_kernel, unsigned(blocks), 256, 0, static_cast<cudaStream_t>(cuda_stream), p));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return HK_OK;
}

int hk_rotary(const void* x, void* o, const void* sin, const void* cos, int B, int H, int N, int D, int rotary_dim,
              int device, void* cuda_stream) {
  if (B <= 0 || H <= 0) return HK_EINVAL;
  return rotary_launch(x, o, sin, cos, static_cast<long long>(B) * H * N, N, D, rotary_dim, 1, 0, device, cuda_stream);
}

int hk_rotary_bnhd(const void* x, void* o, const void* sin, const void* cos, int B, int N, int H, int D,
                   int rotary_dim, int pos_offset, int device, void* cuda_stream) {
  if (B <= 0 || H <= 0) return HK_EINVAL;
  return rotary_launch(x, o, sin, cos, static_cast<long long>(B) * N * H, N, D, rotary_dim, H, pos_offset, device,
                       cuda_stream);
}

size_t hk_attn_paged_decode_workspace_bytes(int S, int H, int D, int max_pages_per_seq, int page_size) {
  return hk::decode_workspace_bytes(S, H, D, max_pages_per_seq, page_size);
}

int hk_attn_paged_decode(const void* q, const void* k_pages, const void* v_pages, const int32_t* block_table,
                         const int32_t* ctx_lens, void* o, float* lse, int S, int H, int H_KV, int D,
                         int page_size, int max_pages_per_seq, int num_pages, float softmax_scale,
                         void* workspace, size_t workspace_bytes, int device, void* cuda_stream) {
  if (!q || !k_pages || !v_pages || !block_table || !ctx_lens || !o || !lse) return HK_EINVAL;
  if (S <= 0 || H <= 0 || H_KV <= 0 || max_pages_per_seq <= 0 || num_pages <= 0) return HK_EINVAL;
  if (D != 128 || page_size != 16) return HK_EUNSUPPORTED;
  if (H % H_KV != 0) return HK_EINVAL;
  const int G = H / H_KV;
  if (G < 1 || G > 8) return HK_EUNSUPPORTED;  // the heads of a group sit in the 8 usable rows of one MMA tile
  if (!aligned16(q) || !aligned16(k_pages) || !aligned16(v_pages) || !aligned16(o)) return HK_EINVAL;
  if (!hk::decode_shape_supported(S, H_KV, max_pages_per_seq)) return unsupported_decode_shape(S, H_KV, max_pages_per_seq);
  const size_t need = hk::decode_workspace_bytes(S, H, D, max_pages_per_seq, page_size);
  if (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255)) return HK_EWORKSPACE;
  DeviceState* st = nullptr;
  DeviceScope scope;
  int rc = scope.enter(device, &st);
  if (rc != HK_OK) return rc;
  hk::DecodeParams p;
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.k_pages = static_cast<const __nv_bfloat16*>(k_pages);
  p.v_pages = static_cast<const __nv_bfloat16*>(v_pages);
  p.block_table = block_table;
  p.ctx_lens = ctx_lens;
  p.o = static_cast<__nv_bfloat16*>(o);
  p.lse = lse;
  p.S = S;
  p.H = H;
  p.H_KV = H_KV;
  p.max_pages = max_pages_per_seq;
  p.num_pages = num_pages;
  p.scale = softmax_scale > 0.f ? softmax_scale : 1.0f / std::sqrt(float(D));
  p.scale_log2 = p.scale * 1.4426950408889634f;
  p.workspace = workspace;
  p.status = st->status;
  int launched = 0;
  cudaError_t e = hk::launch_paged_decode(p, st->decode, static_cast<cudaStream_t>(cuda_stream), &launched);
  g_launches.fetch_add(launched, std::memory_order_relaxed);
  if (e != cudaSuccess) return cuda_fail(e, "paged decode launch");
  return HK_OK;
}

int hk_paged_kv_append(const void* k_new, const void* v_new, void* k_pages, void* v_pages,
                       const int32_t* block_table, const int32_t* start_pos, int S, int T, int H_KV, int D,
                       int page_size, int max_pages_per_seq, int num_pages, int device, void* cuda_stream) {
  if (!k_new || !v_new || !k_pages || !v_pages || !block_table || !start_pos) return HK_EINVAL;
  if (S <= 0 || T <= 0 || H_KV <= 0 || D <= 0 || max_pages_per_seq <= 0 || num_pages <= 0) return HK_EINVAL;
  if (page_size != hk::kPageTokens) return HK_EUNSUPPORTED;
  if ((H_KV * D) % 8 != 0 || T > 65535 || S > 65535) return HK_EINVAL;
  if (!aligned16(k_new) || !aligned16(v_new) || !aligned16(k_pages) || !aligned16(v_pages)) return HK_EINVAL;
  DeviceState* st = nullptr;
  DeviceScope scope;
  int rc = scope.enter(device, &st);
  if (rc != HK_OK) return rc;
  hk::AppendParams p;
  p.k_new = static_cast<const __nv_bfloat16*>(k_new);
  p.v_new = static_cast<const __nv_bfloat16*>(v_new);
  p.k_pages = static_cast<__nv_bfloat16*>(k_pages);
  p.v_pages = static_cast<__nv_bfloat16*>(v_pages);
  p.block_table = block_table;
  p.start_pos = start_pos;
  p.S = S;
  p.T = T;
  p.row_vec16 = H_KV * D * 2 / 16;
  p.max_pages = max_pages_per_seq;
  p.num_pages = num_pages;
  p.status = st->status;
  const long long groups = (static_cast<long long>(S) * T + hk::kAppendUnroll - 1) / hk::kAppendUnroll;
  const long long max_blocks = static_cast<long long>(st->sm_count) * 16;  // 16 x 128 threads fill an SM
  const unsigned blocks = static_cast<unsigned>(groups < max_blocks ? groups : max_blocks);
  HK_CUDA(hk::launch_dependent(true, hk::paged_kv_append_kernel, blocks, 128, 0, static_cast<cudaStream_t>(cuda_stream), p));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return HK_OK;
}

int hk_paged_kv_append_rotary(const void* k_new, const void* v_new, void* k_pages, void* v_pages,
                              const int32_t* block_table, const int32_t* start_pos, const void* sin, const void* cos,
                              int S, int T, int H_KV, int D, int rotary_dim, int cos_rows, int page_size,
                              int max_pages_per_seq, int num_pages, int device, void* cuda_stream) {
  if (!k_new || !v_new || !k_pages || !v_pages || !block_table || !start_pos || !sin || !cos) return HK_EINVAL;
  if (S <= 0 || T <= 0 || H_KV <= 0 || D <= 0 || max_pages_per_seq <= 0 || num_pages <= 0 || cos_rows <= 0)
    return HK_EINVAL;
  if (page_size != hk::kPageTokens) return HK_EUNSUPPORTED;
  if (rotary_dim <= 0) rotary_dim = D;
  if (D % 8 != 0 || rotary_dim % 16 != 0 || rotary_dim > D) return HK_EUNSUPPORTED;
  if (T > 65535 || S > 65535) return HK_EINVAL;
  if (!aligned16(k_new) || !aligned16(v_new) || !aligned16(k_pages) || !aligned16(v_pages) || !aligned16(sin) ||
      !aligned16(cos))
    return HK_EINVAL;
  DeviceState* st = nullptr;
  DeviceScope scope;
  int rc = scope.enter(device, &st);
  if (rc != HK_OK) return rc;
  hk::AppendRotaryParams q;
  q.a.k_new = static_cast<const __nv_bfloat16*>(k_new);
  q.a.v_new = static_cast<const __nv_bfloat16*>(v_new);
  q.a.k_pages = static_cast<__nv_bfloat16*>(k_pages);
  q.a.v_pages = static_cast<__nv_bfloat16*>(v_pages);
  q.a.block_table = block_table;
  q.a.start_pos = start_pos;
  q.a.S = S;
  q.a.T = T;
  q.a.row_vec16 = H_KV * D * 2 / 16;
  q.a.max_pages = max_pages_per_seq;
  q.a.num_pages = num_pages;
  q.a.status = st->status;
  q.cos = static_cast<const __nv_bfloat16*>(cos);
  q.sin = static_cast<const __nv_bfloat16*>(sin);
  q.cos_rows = cos_rows;
  q.H_KV = H_KV;
  q.D = D;
  q.R = rotary_dim;
  const long long tokens = static_cast<long long>(S) * T;
  const long long max_blocks = static_cast<long long>(st->sm_count) * 16;  // 16 x 128 threads fill an SM
  const unsigned blocks = static_cast<unsigned>(tokens < max_blocks ? tokens : max_blocks);
  HK_CUDA(hk::launch_dependent(true, hk::paged_kv_append_rotary_kernel, blocks, 128, 0, static_cast<cudaStream_t>(cuda_stream), q));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return HK_OK;
}

int hk_last_device_status(int device) {
  DeviceState* st = nullptr;
  DeviceScope scope;
  int rc = scope.enter(device, &st);
  if (rc != HK_OK) return rc;
  HK_CUDA(cudaDeviceSynchronize());
  volatile int* const host = st->status_host;
  const int word = *host;
  if (word != 0) *host = 0;
  return status_to_code(word);
}

int hk_selftest_dkdv_in_pairs(int B, int Nq, int Nk, int H, int H_KV, int D, int sm_count) {
  if (B <= 0 || Nq <= 0 || Nk <= 0 || H <= 0 || H_KV <= 0 || H % H_KV != 0 || sm_count <= 0) return HK_EINVAL;
  if (D != 64 && D != 128) return HK_EUNSUPPORTED;
  const int nbk = (Nk + hk::kBlockN - 1) / hk::kBlockN;
  if (static_cast<long long>(B) * H_KV * nbk > 0x3fffffffll) return HK_EINVAL;
  return deal_in_pairs(B * H_KV, H / H_KV, Nq, nbk, D, sm_count) ? 1 : 0;
}

int hk_selftest_bwd_dealing(int B, int Nq, int Nk, int H, int H_KV, int D, int causal, int sm_count, const int* clusters,
                            int* dq_ctas_out) {
  if (B <= 0 || Nq <= 0 || Nk <= 0 || H <= 0 || H_KV <= 0 || H % H_KV != 0 || sm_count <= 0 || !clusters || !dq_ctas_out)
    return HK_EINVAL;
  if (D != 64 && D != 128) return HK_EUNSUPPORTED;
  const int nbq = (Nq + hk::kBlockM - 1) / hk::kBlockM, nbk = (Nk + hk::kBlockN - 1) / hk::kBlockN;
  if (static_cast<long long>(B) * H * nbq > 0x3fffffffll || static_cast<long long>(B) * H_KV * nbk > 0x3fffffffll)
    return HK_EINVAL;
  hk::BwdParams p = {};
  p.B = B, p.N = Nq, p.NK = Nk, p.H = H, p.H_KV = H_KV, p.G = H / H_KV;
  p.group_units = 1;
  auto deal = [&](auto dkdv, auto dq) {
    const int grid = dkdv(p, nbk, sm_count, clusters);
    *dq_ctas_out = dq(p, nbq, nbk, grid, sm_count);
    return p.split;
  };
  if (D == 128) return causal ? deal(deal_dkdv<128, true>, dq_ctas<128, true>) : deal(deal_dkdv<128, false>, dq_ctas<128, false>);
  return causal ? deal(deal_dkdv<64, true>, dq_ctas<64, true>) : deal(deal_dkdv<64, false>, dq_ctas<64, false>);
}

int hk_selftest_decode_shape(int S, int H_KV, int max_pages, int sm_count, const int* clusters, int clusters8, int* warps) {
  if (!hk::decode_shape_supported(S, H_KV, max_pages) || sm_count <= 0 || !clusters || !warps) return HK_EINVAL;
  hk::DecodeLimits lim;
  lim.sm_count = sm_count;
  for (int n = 2; n <= hk::kMaxCluster; ++n) lim.clusters4[n] = clusters[n];
  lim.clusters8 = clusters8;
  const hk::DecodeShape shape = hk::decode_pick_shape(S, H_KV, max_pages, lim);
  *warps = shape.warps;
  return shape.cluster;
}

int hk_selftest_fastdiv(void) {
  // host only: the multiply-and-shift division of the item decode against the division it replaces, for every
  // divisor up to 4096, divisors around every power of two, and dividends at the edges of [0, 2^31)
  auto check = [](int d) {
    const hk::FastDiv fd(d);
    const long long top = 0x7fffffffll;
    const long long probes[] = {0, 1, d - 1ll, d, d + 1ll, 2ll * d - 1, 2ll * d, 1000003ll * d + d - 1, top - d, top - 1, top,
                                0x3fffffffll, 123456789ll, 2000000011ll};
    for (long long n : probes) {
      if (n < 0 || n > top) continue;
      if (fd.div_host(int(n)) != int(n / d)) return false;
    }
    return true;
  };
  for (int d = 1; d <= 4096; ++d)
    if (!check(d)) return HK_EINVAL;
  for (int k = 1; k < 31; ++k)
    for (int e = -1; e <= 1; ++e) {
      const long long d = (1ll << k) + e;
      if (d >= 1 && d <= 0x7fffffffll && !check(int(d))) return HK_EINVAL;
    }
  return HK_OK;
}

int hk_selftest_bounded_wait(int device, unsigned limit_us) {
  DeviceState* st = nullptr;
  DeviceScope scope;
  int rc = scope.enter(device, &st);
  if (rc != HK_OK) return rc;
  if (limit_us == 0 || limit_us > 1000000u) return HK_EINVAL;
  bounded_wait_selftest_kernel<<<1, 32>>>(st->status, static_cast<unsigned long long>(limit_us) * 1000ull);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  HK_CUDA(cudaGetLastError());
  return hk_last_device_status(device);
}

unsigned long long hk_kernel_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

const char* hk_strerror(int code) {
  switch (code) {
    case HK_OK: return "ok";
    case HK_EINVAL: return "invalid argument (shape, null or misaligned pointer)";
    case HK_EUNSUPPORTED: return "unsupported configuration or device";
    case HK_ECUDA: return "CUDA call failed";
    case HK_ETIMEOUT: return "bounded device-side wait expired";
    case HK_EWORKSPACE: return "workspace missing, misaligned or too small";
    case HK_EBADPAGE: return "block-table entry outside the page pool";
    case HK_EBADLEN: return "context length beyond the block table's capacity (clamped)";
    default: return "unknown error code";
  }
}

const char* hk_last_cuda_error(void) { return g_cuda_err; }

}  // extern "C"

// ---------------------------------------------------------------------------------------------------
// Allocation-free paged decode: scratch and status live in the library image instead of in memory the
// caller or this library would have to allocate (see hk_attn_paged_decode_static in hk_attn.h).
// In host code `g_decode_static_scratch` is only a handle for the runtime, not a device address; the
// address each device gave the array is looked up once per device with cudaGetSymbolAddress.
static __device__ __align__(256) unsigned char g_decode_static_scratch[HK_DECODE_STATIC_SCRATCH_BYTES];
static __device__ int g_decode_static_status;

namespace {

struct StaticDecodeState {
  std::mutex mu;
  bool ready = false;       // a failed set-up is retried by the next call
  int sm_count = 0;
  hk::DecodeLimits decode;
  void* scratch = nullptr;  // device address of g_decode_static_scratch on this device
  int* status = nullptr;    // device address of g_decode_static_status on this device
};
StaticDecodeState g_static_dev[kMaxDevices];

// Runs once per device, with that device current. Nothing in here allocates.
int init_static_decode(int device) {
  StaticDecodeState& st = g_static_dev[device];
  cudaDeviceProp prop;
  HK_CUDA(cudaGetDeviceProperties(&prop, device));
  if (prop.major != 10) {
    snprintf(g_cuda_err, sizeof(g_cuda_err), "device %d is sm_%d%d; this library needs sm_100", device, prop.major,
             prop.minor);
    return HK_EUNSUPPORTED;
  }
  st.sm_count = prop.multiProcessorCount;
  HK_CUDA(cudaGetSymbolAddress(&st.scratch, g_decode_static_scratch));
  HK_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&st.status), g_decode_static_status));
  if (!st.scratch || !st.status || (reinterpret_cast<uintptr_t>(st.scratch) & 255)) {
    snprintf(g_cuda_err, sizeof(g_cuda_err), "static decode scratch has no usable device address");
    return HK_ECUDA;
  }
  return hk::prepare_decode_kernels(g_cuda_err, sizeof(g_cuda_err), st.sm_count, &st.decode);
}

}  // namespace

extern "C" int hk_attn_paged_decode_static(const void* q, const void* k_pages, const void* v_pages,
                                           const int32_t* block_table, const int32_t* ctx_lens, void* o, float* lse,
                                           int S, int H, int H_KV, int D, int page_size, int max_pages_per_seq,
                                           int num_pages, float softmax_scale, int device, void* cuda_stream,
                                           int* status_out) {
  if (!q || !k_pages || !v_pages || !block_table || !ctx_lens || !o || !lse) return HK_EINVAL;
  if (S <= 0 || H <= 0 || H_KV <= 0 || max_pages_per_seq <= 0 || num_pages <= 0) return HK_EINVAL;
  if (D != 128 || page_size != 16) return HK_EUNSUPPORTED;
  if (H % H_KV != 0) return HK_EINVAL;
  const int G = H / H_KV;
  if (G < 1 || G > 8) return HK_EUNSUPPORTED;  // the heads of a group sit in the 8 usable rows of one MMA tile
  if (!aligned16(q) || !aligned16(k_pages) || !aligned16(v_pages) || !aligned16(o)) return HK_EINVAL;
  if (!hk::decode_shape_supported(S, H_KV, max_pages_per_seq)) return unsupported_decode_shape(S, H_KV, max_pages_per_seq);
  const size_t need = hk::decode_workspace_bytes(S, H, D, max_pages_per_seq, page_size);
  if (need == 0 || need > HK_DECODE_STATIC_SCRATCH_BYTES) {
    snprintf(g_cuda_err, sizeof(g_cuda_err),
             "problem needs %zu bytes of scratch, the built-in array holds %u: use hk_attn_paged_decode", need,
             unsigned(HK_DECODE_STATIC_SCRATCH_BYTES));
    return HK_EWORKSPACE;
  }
  DeviceScope scope;  // the caller's current device is put back on return
  {
    const int rc = scope.enter_raw(device, &device);
    if (rc != HK_OK) return rc;
  }
  StaticDecodeState& st = g_static_dev[device];
  {
    std::lock_guard<std::mutex> lock(st.mu);
    if (!st.ready) {
      const int rc = init_static_decode(device);
      if (rc != HK_OK) return rc;
      st.ready = true;
    }
  }

  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  // the status word is shared by all calls and keeps the last call's value: start this call from zero
  HK_CUDA(cudaMemsetAsync(st.status, 0, sizeof(int), stream));
  hk::DecodeParams p;
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.k_pages = static_cast<const __nv_bfloat16*>(k_pages);
  p.v_pages = static_cast<const __nv_bfloat16*>(v_pages);
  p.block_table = block_table;
  p.ctx_lens = ctx_lens;
  p.o = static_cast<__nv_bfloat16*>(o);
  p.lse = lse;
  p.S = S;
  p.H = H;
  p.H_KV = H_KV;
  p.max_pages = max_pages_per_seq;
  p.num_pages = num_pages;
  p.scale = softmax_scale > 0.f ? softmax_scale : 1.0f / std::sqrt(float(D));
  p.scale_log2 = p.scale * 1.4426950408889634f;
  p.workspace = st.scratch;  // the looked-up device address, never the host-side symbol
  p.status = st.status;
  int launched = 0;
  cudaError_t e = hk::launch_paged_decode(p, st.decode, stream, &launched);
  g_launches.fetch_add(launched, std::memory_order_relaxed);
  if (e != cudaSuccess) return cuda_fail(e, "paged decode launch");
  if (status_out) {
    int word = 0;
    HK_CUDA(cudaMemcpyAsync(&word, st.status, sizeof(int), cudaMemcpyDeviceToHost, stream));
    HK_CUDA(cudaStreamSynchronize(stream));
    *status_out = status_to_code(word);
  }
  return HK_OK;
}

