// Library-internal plumbing: the device context behind an apg_ctx handle,
// status propagation and scratch memory.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/apogee_gpu.h"
#include "curve.cuh"

namespace apg {

// A failure carrying the C ABI status it maps to. Every entry point catches
// it at the boundary; nothing escapes into the caller's process as a throw.
struct Error : std::runtime_error {
  int status;
  Error(int s, const std::string& m) : std::runtime_error(m), status(s) {}
};

#define APG_CUDA(call)                                                                                      \
  do {                                                                                                      \
    cudaError_t e_ = (call);                                                                                \
    if (e_ != cudaSuccess)                                                                                  \
      throw ::apg::Error(e_ == cudaErrorMemoryAllocation ? APG_ERR_OUT_OF_MEMORY : APG_ERR_CUDA,          \
                         std::string(#call) + ": " + cudaGetErrorString(e_));                              \
  } while (0)

#define APG_LAUNCH_CHECK() APG_CUDA(cudaGetLastError())

// Device-side error flags a kernel may raise; read back after a sync.
enum DeviceFlag : uint32_t {
  DEV_NONCANONICAL = 1u,   // an input coordinate or scalar was >= its modulus
  DEV_OFF_CURVE = 2u,      // an input point failed y^2 = x^3 + 3
  DEV_TRANSCRIPT = 4u,     // a transcript invariant was broken
  DEV_DEGENERATE = 8u,     // Mercury's {z, 1/z, alpha} had a repeat
  DEV_NONZERO_REM = 16u,   // a division that must be exact left a remainder
  DEV_INVERSE = kFlagInverse,  // a field inversion did not converge (field.cuh)
};

// A grow-only device buffer.
struct DevBuf {
  void* p = nullptr;
  size_t cap = 0;
  void* get(size_t bytes) {
    if (bytes > cap) {
      if (p) cudaFree(p);
      p = nullptr;
      cap = 0;
      size_t want = bytes + bytes / 8 + 256;
      APG_CUDA(cudaMalloc(&p, want));
      cap = want;
    }
    return p;
  }
  template <class T>
  T* as(size_t count) {
    return reinterpret_cast<T*>(get(count * sizeof(T)));
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
  }
};

// The precomputed window table of the resident SRS for one window width:
// tab[w * n + i] = 2^(c*w) * P_i, affine Montgomery. Contexts and lanes that read the
// same table hold its memory together: it is freed with the last of them, each of
// which has its stream idle when it lets go.
struct SrsTable {
  int c = 0, windows = 0;
  size_t n = 0;
  Affine* tab = nullptr;
  std::shared_ptr<void> mem;
  bool owned = true;  // false: borrowed from another context (apg_srs_share), counted there
};

enum ScratchSlot {
  S_ENTRIES, S_SORTED, S_SCANBLK, S_BUCKETS, S_HEAD, S_TAIL, S_FLAGS, S_LEVEL_A,
  S_LEVEL_B, S_LEVEL_T, S_TSUM, S_RESULT, S_BASES, S_SCALARS, S_TMP0, S_TMP1, S_TMP2, S_TMP3, S_TMP4,
  S_TMP5, S_TMP6, S_TMP7, S_ROUND, S_PAIR_A, S_PAIR_B, S_PAIR_PP, S_PAIR_CNT, S_PAIR_TERMS,
  S_SPLIT_BASES, S_SPLIT_SCALARS, S_COUNT
};

// Per-kernel CUDA-event timers (ids are public: APG_TIMER_* in the header).
struct Timers {
  static constexpr int N = 8;
  bool on = false;
  bool kernels = false;  // also bracket every launch (APG_TIMER_KERNELS)
  std::vector<cudaEvent_t> pool;
  std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> pending;
  double ms[N] = {0};
  uint64_t count[N] = {0};
  cudaEvent_t get() {
    if (pool.empty()) {
      cudaEvent_t e;
      APG_CUDA(cudaEventCreate(&e));
      return e;
    }
    cudaEvent_t e = pool.back();
    pool.pop_back();
    return e;
  }
  void flush() {
    for (auto& p : pending) {
      APG_CUDA(cudaEventSynchronize(p.second.second));
      float t = 0;
      APG_CUDA(cudaEventElapsedTime(&t, p.second.first, p.second.second));
      ms[p.first] += t;
      count[p.first] += 1;
      pool.push_back(p.second.first);
      pool.push_back(p.second.second);
    }
    pending.clear();
  }
};

struct Ctx {
  int device = 0;
  int sm_count = 0;
  cudaStream_t stream = nullptr;
  std::mutex mu;
  std::string last_error;
  Affine* srs = nullptr;
  size_t srs_n = 0;
  bool srs_owned = true;  // false: borrowed from another context (apg_srs_share)
  std::vector<SrsTable> tables;
  // Window width chosen by apg_msm_autotune per size class (index: ceil of
  // log2 of the point count); 0 = the default rule of srs_table_for.
  int tuned_c[64] = {0};
  DevBuf scratch[S_COUNT];
  DevBuf fft_tw[16];  // twiddles of the one-block transforms, by log2 of the size (mercury.cu)
  uint32_t* d_flags = nullptr;  // device error flags (DeviceFlag bits)
  uint64_t launches = 0;        // kernels launched on this context
  Timers timers;
  // A second stream with its own scratch that borrows this context's SRS:
  // batches of commits alternate between the two so that one MSM's
  // latency-bound tail (and the next column's copy) overlaps another's
  // bucket accumulation.
  std::unique_ptr<Ctx> lane;
  // Host-to-device copies of batch commits' host columns.
  cudaStream_t copy_stream = nullptr;

  // Pinned host memory that kernels write their results into: a flag word the
  // host waits for, a round's sums (at kPinnedSums) and tables or final values
  // (from kPinnedTables). The host reads a kernel's result as soon as its last
  // block has stored the flag, with no copy and no stream synchronisation
  // between (they took 28 us a sumcheck round).
  static constexpr size_t kPinnedBytes = 128 << 10, kPinnedSums = 128, kPinnedTables = 4096;
  void* pinned = nullptr;
  uint32_t flag_seq = 0;  // the value the latest flagged kernel stores
  uint8_t* host_pinned() {
    if (!pinned) {
      APG_CUDA(cudaMallocHost(&pinned, kPinnedBytes));
      memset(pinned, 0, kPinnedSums);
    }
    return static_cast<uint8_t*>(pinned);
  }
  // Wait until the stream's latest flagged kernel has stored flag_seq.
  void wait_flag() {
    const volatile uint32_t* f = reinterpret_cast<const volatile uint32_t*>(host_pinned());
    for (uint64_t spin = 1; *f != flag_seq; ++spin)
      if ((spin & 0x3fff) == 0) {  // a failed launch would leave the flag unset
        const cudaError_t e = cudaStreamQuery(stream);
        if (e == cudaSuccess && *f != flag_seq) throw Error(APG_ERR_INTERNAL, "a kernel ended without its flag");
        if (e != cudaSuccess && e != cudaErrorNotReady) APG_CUDA(e);
      }
    std::atomic_thread_fence(std::memory_order_acquire);
  }

  // What goes on the stream beside kernels. A kernel launched as the end of a
  // chain (launch_chained) waits for the kernel before it; what stands before it
  // has to be a kernel of this call, so everything else is noted here: copies,
  // memsets, event waits, allocations in stream order (which may wait for another
  // stream's release), and a call's beginning (the caller may have queued any of
  // them on the context's stream).
  bool after_kernel = false;
  void copy(void* to, const void* from, size_t bytes, cudaMemcpyKind kind) {
    after_kernel = false;
    APG_CUDA(cudaMemcpyAsync(to, from, bytes, kind, stream));
  }
  void fill(void* p, int value, size_t bytes) {
    after_kernel = false;
    APG_CUDA(cudaMemsetAsync(p, value, bytes, stream));
  }
  void wait_event(cudaEvent_t e) {
    after_kernel = false;
    APG_CUDA(cudaStreamWaitEvent(stream, e, 0));
  }
  template <class T>
  void alloc(T** p, size_t bytes) {  // (freed by cudaFreeAsync on the stream)
    after_kernel = false;
    APG_CUDA(cudaMallocAsync(reinterpret_cast<void**>(p), bytes, stream));
  }

  // Bracket work on the stream with a timer's events (no-op unless enabled).
  cudaEvent_t timer_begin() {
    if (!timers.on) return nullptr;
    cudaEvent_t e = timers.get();
    APG_CUDA(cudaEventRecord(e, stream));
    return e;
  }
  void timer_end(int id, cudaEvent_t begin) {
    if (!timers.on || !begin) return;
    cudaEvent_t e = timers.get();
    APG_CUDA(cudaEventRecord(e, stream));
    timers.pending.push_back({id, {begin, e}});
  }

  void check_flags() {
    uint32_t f = 0;
    copy(&f, d_flags, 4, cudaMemcpyDeviceToHost);
    APG_CUDA(cudaStreamSynchronize(stream));
    if (f) {
      fill(d_flags, 0, 4);
      if (f & DEV_NONCANONICAL) throw Error(APG_ERR_NONCANONICAL, "an input value is not below its modulus");
      if (f & DEV_OFF_CURVE) throw Error(APG_ERR_INVALID_POINT, "an input point is not on the curve");
      if (f & DEV_DEGENERATE) throw Error(APG_ERR_DEGENERATE_CHALLENGE, "degenerate Mercury challenge set");
      if (f & DEV_NONZERO_REM) throw Error(APG_ERR_INTERNAL, "an exact division left a remainder");
      if (f & DEV_INVERSE) throw Error(APG_ERR_INTERNAL, "a field inversion did not converge");
      throw Error(APG_ERR_INTERNAL, "device invariant failed");
    }
  }
};

// Launch a kernel on the context's stream, check the launch and count it.
// With kernel timing on, every launch is bracketed by a pair of events, so
// the sum of kernel durations (the device's busy time on this stream) can be
// set against the wall clock.
template <class... KArgs, class... Args>
inline void launch(Ctx& c, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, Args... args) {
  cudaEvent_t e0 = nullptr;
  if (c.timers.on && c.timers.kernels) {
    if (c.timers.pending.size() > 4096) c.timers.flush();
    e0 = c.timers.get();
    APG_CUDA(cudaEventRecord(e0, c.stream));
  }
  kernel<<<grid, block, smem, c.stream>>>(args...);
  APG_CUDA(cudaGetLastError());
  c.after_kernel = true;
  ++c.launches;
  if (e0) {
    cudaEvent_t e1 = c.timers.get();
    APG_CUDA(cudaEventRecord(e1, c.stream));
    c.timers.pending.push_back({APG_TIMER_KERNELS, {e0, e1}});
  }
}

// The same for a kernel that begins with chain_begin(): where it follows another
// kernel on the stream, its blocks may be set up while that one's last blocks still run
// (programmatic stream serialization), and wait there for it to end. Every kernel of a
// chain waits, so each sees all that stands before it. The wait is specified for
// kernels: what follows anything else (Ctx::after_kernel) is launched plainly, in
// order with all of it. Measured on a GB300, the chains of an MSM and an
// opening launched so: commitments of four 2^8-point columns 178 -> 160 us, a stacked
// 2^16-variable opening (93 launches) 2359 -> 2176.
template <class... KArgs, class... Args>
inline void launch_chained(Ctx& c, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, Args... args) {
  if (c.timers.on || !c.after_kernel) return launch(c, kernel, grid, block, smem, args...);
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c.stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  APG_CUDA(cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...));
  ++c.launches;
}

#ifdef __CUDACC__
// The first thing that a kernel of launch_chained does, before it reads or writes
// memory: wait for the kernel before it, then let the one after it be set up.
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

// ---------------------------------------------------------------------------
// Entry points implemented in the .cu files.
// ---------------------------------------------------------------------------

// Canonical Fr -> Montgomery in place, raising DEV_NONCANONICAL for values >= p.
__global__ void k_fr_to_mont(Fr* v, size_t n, uint32_t* flags);

// `bytes` of a result on the stream to the host, the error flags checked: a
// kernel stores both in pinned memory and the host waits for its flag (instead of
// two copies and a synchronisation: about 15 us less a result on a GB300).
void fetch_checked(Ctx& c, const void* d_src, size_t bytes, void* host);
// The same in two halves: publish on the stream (work may follow), collect before
// anything else is published.
uint32_t publish_checked(Ctx& c, const void* d_src, size_t bytes);
void collect_checked(Ctx& c, uint32_t seq, size_t bytes, void* host);
// Canonical 64-byte points (host) -> device affine Montgomery, validated.
void upload_points(Ctx& c, const uint8_t* host, size_t n, Affine* dst);
// The same without waiting: the flags are the caller's to check.
void upload_points_async(Ctx& c, const uint8_t* host, size_t n, Affine* dst);
// Device affine Montgomery -> canonical 64-byte points (host).
void download_points(Ctx& c, const Affine* src, size_t n, uint8_t* host);
// SRS [tau^i]G for i < n, generated on the device.
void generate_srs(Ctx& c, const uint8_t tau_canonical[32], size_t n, Affine* dst);
// n seeded benchmark Fr (canonical, 8 LE words each) from the ChaCha20 keystream:
// kind 0 trace-like (bits, register words, uniform Fr), kind 1 uniform Fr.
void synth_column(Ctx& c, uint64_t seed, int kind, size_t n, void* d_out);

struct MsmPlan {
  int c;         // window width
  int windows;   // signed-digit windows
  bool precomp;  // read bases from an SRS window table
  uint32_t buckets;  // a space: 2^(c-1), or fewer when no digit can reach them
};
// `bits`: the width of small scalars.
MsmPlan msm_plan(size_t n, bool small_scalars, const SrsTable* table, int bits, int full_bits = 254);
// k MSMs over the same bases (lens[j] scalars each, device pointers); result
// j is written to d_out + 64 * j. Columns are processed in groups that share
// one sort, one accumulation and one bucket reduction.
struct MsmBatchOpts {
  const size_t* offs = nullptr;  // first base of each column (nullable: all 0)
  bool stack = false;            // one result: the sum of every column's MSM
  int bits = 32;                 // width of small scalars: 32, 16, 8 or 1 (bit-packed u64)
  bool uniform = false;          // field elements without structure (nearly every digit nonzero)
  int full_bits = 254;           // width of the other scalars
};
void msm_multi(Ctx& c, const Affine* bases, const SrsTable* table, const void* const* scalars, const size_t* lens,
               size_t k, bool small_scalars, bool scalars_canonical, uint8_t* d_out,
               const MsmBatchOpts& o = MsmBatchOpts());
// Pippenger over device inputs; the result (canonical affine bytes, 64) is
// written to device memory `out64` when non-null and returned to `host_out`
// when non-null.
void msm_device(Ctx& c, const Affine* bases, const SrsTable* table, const void* scalars, bool small_scalars,
                bool scalars_canonical, size_t n, uint8_t* out64_device, uint8_t* host_out,
                const MsmBatchOpts& o = MsmBatchOpts());
const SrsTable* srs_table(Ctx& c, int cbits, size_t need);
// The table that `cols` MSMs over the first n SRS powers read together: 6-bit
// windows up to 2^8 points and 7-bit ones up to 2^12 (a short bucket reduction),
// 17-bit windows from kWideTableMin, and between them 15-bit windows for one or two
// columns and 13-bit ones for more, which pay the reduction of each column's buckets.
// 15 and 17 divide the 255 bits of a signed scalar (17 and 15 windows: 16 and 18 bits
// take as many digits over twice the buckets). Measured on a GB300, us: four 2^8-point
// columns 138 at 6 bits, 146 at 7, 156 at 8 (uniform 165, 172, 168); four of 2^10 167,
// 161, 166 (205, 188, 193); one of 2^12 169, 158, 166 and 223 at 13 (uniform 205, 184,
// 191, 248); 2^16 alone 395 at 13, 401 at 15
// (uniform 578, 532), sixteen 1509, 1711 (uniform 3420, 3496); sixteen of 2^14
// 930, 1140; sixteen of 2^18 3654 at 13, 4114 at 17, uniform 12024, 10675; 2^20
// alone 1394 at 17, 1402 at 16, 1881 at 20 (uniform 3142, 3254, 3453); 2^22 3264
// at 17, 3433 at 16, 3626 at 20 (uniform 10124, 10811, 10108).
// `tuned`: use the width apg_msm_autotune chose for the size class, if any
// (commits of the caller's columns); openings commit uniformly random
// quotient polynomials, for which the default rule is the uniform-scalar one.
constexpr size_t kNarrowTableMax = (size_t)1 << 12;
constexpr size_t kNarrowWindowMax = (size_t)1 << 16;  // points that widths below 12 are timed over
constexpr int narrow_window(size_t n) { return n <= ((size_t)1 << 8) ? 6 : 7; }
constexpr size_t kWideTableMin = (size_t)1 << 18;
const SrsTable* srs_table_for(Ctx& c, size_t n, size_t cols, bool tuned = true);
constexpr int default_table_window(size_t n, size_t cols) {
  return n <= kNarrowTableMax ? narrow_window(n) : n >= kWideTableMin ? 17 : cols <= 2 ? 15 : 13;
}
// The scratch that msm_multi holds for `cols` columns of n field elements over an
// SRS table of `window` bits (at most: the pair rounds' lists at their bounds).
size_t msm_scratch_bytes(size_t n, size_t cols, int window, bool uniform);
// Time SRS commits of the first 2^k sample scalars for k in [kmin, kmax] with
// each candidate width and record the fastest in c.tuned_c (see
// apg_msm_autotune).
void msm_autotune(Ctx& c, const void* d_sample, size_t sample_len, int kmin, int kmax, const int* cands,
                  size_t ncands, int* chosen);
double probe_fq_mul_rate(Ctx& c, double target_ms);
// The group side of pcs::discharge (weights null) or check_pairings (one
// weight a check): see apg_discharge_msms / apg_pairing_msms.
int accumulator_msms(Ctx& c, const uint8_t* sides, const uint8_t* scalars, const uint8_t* points, size_t n,
                     const size_t* checks, size_t nchecks, const uint8_t* weights, uint8_t* a_out, uint8_t* b_out,
                     uint8_t* nu_out);

}  // namespace apg
