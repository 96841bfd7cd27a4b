// The sumcheck prover on the device: one fused kernel per round folds every
// table with the previous round's challenge and sums the summand over the
// hypercube at the nodes the round needs; the host rebuilds the round's cubic
// and draws the next challenge.
//
// Restates crates/sumcheck/src/lib.rs (prove_zerocheck :359-408,
// round_evaluations :324-349) and crates/gkr/src/lib.rs (prove_sumcheck
// :792-899): per pair (2i, 2i+1) of every table the line lo + X*(hi - lo),
// the summand at X = 0..3 weighted by eq, SUMCHECK_ROUND then
// SUMCHECK_CHALLENGE, and the bind f'(i) = f(2i) + r*(f(2i+1) - f(2i))
// (crates/poly/src/lib.rs:156-185). The cubic factors as eq_r(X) q(X) with q
// quadratic, so the device sums q at X = 0 and 2 (and 1 in the first round)
// and the host derives the rest (run_sumcheck). Round r's kernel reads the
// level-(r-1) tables once, writes the level-r tables once and never re-reads
// them.
#include <algorithm>
#include <chrono>
#include <queue>
#include <tuple>

#include "sumcheck.cuh"

namespace apg {

namespace {

constexpr int kRoundThreads = 128;
constexpr int kWarpModeGates = 16;  // weighted gates from which an interpreted list goes one pair per warp

struct RoundArgs {
  int nd;                    // data tables (eq is separate)
  int nv;                    // virtual tables
  uint8_t vkinds[8];
  const Fr* const* src;      // round-0 tables (nd data, then eq), device pointers
  const Fr* in_base;         // previous level (when !in_is_src): table k at in_base + k * in_len
  size_t in_len;
  int in_is_src;
  int bind;                  // fold the previous level with c first
  Fr c;
  Fr* out_base;              // this level (when bind): table k at out_base + k * (in_len / 2)
  size_t npairs;
  int slots_step0;           // first step slot
  int n_val_slots;           // nd + nv
  unsigned* done;            // blocks finished this round (zero between rounds)
  Fr* out;                   // the round's sums at nodes 0..2 (pinned host memory), by the last block
  uint32_t* flag;            // set to seq (pinned host memory) once they are there
  uint32_t seq;
  int to_host;               // out_base is host memory
  int xsplit;                // one thread per (pair, node X) instead of per pair
  const uint8_t* src_bits;   // stored width of each src table (null: all Fr)
  int nodes;                 // bit X set: evaluate the summand at node X (0..2)
};

__device__ __forceinline__ const Fr* table_in(const RoundArgs& A, int k) {
  return A.in_is_src ? A.src[k] : A.in_base + (size_t)k * A.in_len;
}

// Pair i of table k: (lo, hi) = entries (2i, 2i + 1) of this round's level,
// folded from the previous level with c first when the round binds (the
// folded pair is stored when `store` is set). OUTLINE: the fold's two
// products are one call of the shared out-of-line rmul2 instead of two
// inlined multiplies, for the kernels of small rounds, where a launch runs its
// code once and fetching inlined copies of the multiply costs more than the
// call.
template <bool OUTLINE = false>
__device__ __forceinline__ void load_line(const RoundArgs& A, int k, size_t i, Fr& lo, Fr& hi, bool store = true) {
  const Fr* t = table_in(A, k);
  const int bits = A.in_is_src && A.src_bits ? A.src_bits[k] : 0;
  if (!A.bind) {
    lo = bits ? narrow_entry(t, bits, 2 * i) : ld_fe(&t[2 * i]);
    hi = bits ? narrow_entry(t, bits, 2 * i + 1) : ld_fe(&t[2 * i + 1]);
    return;
  }
  Fr a0, a1, a2, a3;
  if (bits) {
    a0 = narrow_entry(t, bits, 4 * i);
    a1 = narrow_entry(t, bits, 4 * i + 1);
    a2 = narrow_entry(t, bits, 4 * i + 2);
    a3 = narrow_entry(t, bits, 4 * i + 3);
  } else {
    a0 = ld_fe(&t[4 * i]);
    a1 = ld_fe(&t[4 * i + 1]);
    a2 = ld_fe(&t[4 * i + 2]);
    a3 = ld_fe(&t[4 * i + 3]);
  }
  if (OUTLINE) {
    const FrPair f = rmul2(A.c, fe_sub(a1, a0), A.c, fe_sub(a3, a2));
    lo = fe_add(a0, f.a);
    hi = fe_add(a2, f.b);
  } else {
    lo = fe_add(a0, fe_mul(A.c, fe_sub(a1, a0)));
    hi = fe_add(a2, fe_mul(A.c, fe_sub(a3, a2)));
  }
  if (!store) return;
  Fr* o = A.out_base + (size_t)k * (A.in_len / 2);
  st_fe(&o[2 * i], lo);
  st_fe(&o[2 * i + 1], hi);
}

// lo + x * (hi - lo) for a node x in 0..2.
__device__ __forceinline__ Fr at_node(const Fr& lo, const Fr& step, int x) {
  Fr v = lo;
  for (int j = 0; j < x; ++j) v = fe_add(v, step);
  return v;
}

// The sum of a value over the warp's (or the narrower block's) lanes, in every lane.
__device__ __forceinline__ Fr warp_sum(Fr a, int width, unsigned mask) {
#pragma unroll 1
  for (int off = width >> 1; off > 0; off >>= 1) {
    Fr o;
#pragma unroll
    for (int w = 0; w < 8; ++w) o.v[w] = __shfl_xor_sync(mask, a.v[w], off);
    a = fe_add(a, o);
  }
  return a;
}

// The end of a round kernel: warp w's sums at the round's nodes stand in
// ws[3 w + x]. One thread a node adds them up; with several blocks they go to
// `partials`, and the last block to finish (it takes the last ticket) adds every
// block's, a warp a node. The sums land in pinned host memory, then the flag the
// host spins on; a level of tables that the host is to read is visible with it. Only
// then does every thread fence its stores to the system: otherwise one thread's fence
// after the block's barrier covers the few words that others read before the kernel
// ends (a GKR proof of 10 columns of 2^21 rows 18.5 -> 18.2 ms, a zerocheck of 2^21 rows
// 1741 -> 1685 us).
__device__ __forceinline__ void round_finish(const RoundArgs& A, const Fr* ws, int nwarps, Fr* partials) {
  __shared__ bool last;
  const int x = threadIdx.x;
  if (A.to_host) __threadfence_system();  // (the level that the block stored)
  __syncthreads();
  if (x < 3) {
    Fr a = ws[x];
    for (int w = 1; w < nwarps; ++w) a = fe_add(a, ws[3 * w + x]);
    st_fe(gridDim.x == 1 ? &A.out[x] : &partials[(size_t)blockIdx.x * 4 + x], a);
  }
  // (One thread's fence after the barrier orders the block's stores, here and below.)
  __syncthreads();
  if (x == 0) {
    last = gridDim.x == 1;
    if (!last) {
      __threadfence();
      last = atomicAdd(A.done, 1u) == gridDim.x - 1;
      __threadfence();
    }
  }
  __syncthreads();
  if (!last) return;
  if (gridDim.x > 1) {
    const int width = min(32, (int)blockDim.x), lane = threadIdx.x & 31;
    const unsigned mask = width == 32 ? 0xffffffffu : (1u << width) - 1;
    for (int node = threadIdx.x >> 5; node < 3; node += max(1, (int)blockDim.x >> 5)) {
      Fr a = fe_zero<FrConsts>();
      for (unsigned b = lane; b < gridDim.x; b += width) {
        const uint4* q = reinterpret_cast<const uint4*>(&partials[(size_t)b * 4 + node]);
        const uint4 u0 = __ldcg(q), u1 = __ldcg(q + 1);
        Fr v;
        v.v[0] = u0.x, v.v[1] = u0.y, v.v[2] = u0.z, v.v[3] = u0.w;
        v.v[4] = u1.x, v.v[5] = u1.y, v.v[6] = u1.z, v.v[7] = u1.w;
        a = fe_add(a, v);
      }
      a = warp_sum(a, width, mask);
      if (lane == 0) st_fe(&A.out[node], a);
    }
    __syncthreads();
  }
  if (x == 0) {
    *A.done = 0;
    __threadfence_system();
    *reinterpret_cast<volatile uint32_t*>(A.flag) = A.seq;
  }
}

// Every thread's sums at the three nodes, reduced a warp at a time.
__device__ __forceinline__ void round_finish_threads(const RoundArgs& A, const Fr acc[3], Fr* ws, Fr* partials) {
  const int width = min(32, (int)blockDim.x);
  const unsigned mask = width == 32 ? 0xffffffffu : (1u << width) - 1;
#pragma unroll 1
  for (int x = 0; x < 3; ++x) {
    const Fr a = warp_sum(acc[x], width, mask);
    if ((threadIdx.x & 31) == 0) ws[3 * (threadIdx.x >> 5) + x] = a;
  }
  round_finish(A, ws, max(1, (int)blockDim.x >> 5), partials);
}

// Resident blocks a SM k_round is compiled for (1: the compiler's choice).
#ifndef APG_ROUND_MIN_BLOCKS
#define APG_ROUND_MIN_BLOCKS 1
#endif
__global__ void __launch_bounds__(kRoundThreads, APG_ROUND_MIN_BLOCKS)
    k_round(RoundArgs A, DevProgram P, VirtualRound V, Fr* partials) {
  extern __shared__ uint32_t sm_raw[];
  const Slots sm = thread_slots(sm_raw);
  __shared__ Fr ws[3 * kRoundThreads / 32];
  Fr acc[3];
#pragma unroll
  for (int x = 0; x < 3; ++x) acc[x] = fe_zero<FrConsts>();
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  if (A.xsplit) {
    // Small rounds: thread t evaluates pair t / 4 at node X = t % 4 alone
    // (X = 3 and, after the first round, X = 1 stay idle), so the evaluations
    // of a pair run side by side (latency, not work, is what bounds a round
    // with few pairs). Threads 4j..4j+3 of a block share a pair; the X = 0
    // thread stores the folded level.
    const int x = threadIdx.x & 3;
    // The X = 0 thread also stores the folded level, so it always runs.
    const bool on = x == 0 || ((A.nodes >> x) & 1);
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; on && t / 4 < A.npairs; t += stride) {
      const size_t i = t / 4;
      Fr lo, hi;
      for (int k = 0; k < A.nd; ++k) {
        load_line(A, k, i, lo, hi, x == 0);
        sm_st(sm, k, at_node(lo, fe_sub(hi, lo), x));
      }
      for (int v = 0; v < A.nv; ++v) {
        virtual_line_dev(V, A.vkinds[v], i, lo, hi);  // hi is the step here
        sm_st(sm, A.nd + v, at_node(lo, hi, x));
      }
      Fr e_lo, e_hi;
      load_line(A, A.nd, i, e_lo, e_hi, x == 0);
      acc[0] = fe_add(acc[0], fe_mul(fe_add(e_lo, e_hi), eval_summand(P, sm)));
    }
    if (x == 1 || x == 2) {
      acc[x == 1 ? 1 : 2] = acc[0];
      acc[0] = fe_zero<FrConsts>();
    }
  } else {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < A.npairs; i += stride) {
    Fr lo, hi;
    for (int k = 0; k < A.nd; ++k) {
      load_line(A, k, i, lo, hi);
      sm_st(sm, k, lo);
      sm_st(sm, A.slots_step0 + k, fe_sub(hi, lo));
    }
    Fr e_lo, e_hi;
    load_line(A, A.nd, i, e_lo, e_hi);
    const Fr w = fe_add(e_lo, e_hi);  // the pair's eq weight without the current variable's factor
    for (int v = 0; v < A.nv; ++v) {
      virtual_line_dev(V, A.vkinds[v], i, lo, hi);
      sm_st(sm, A.nd + v, lo);
      sm_st(sm, A.slots_step0 + A.nd + v, hi);
    }
    for (int x = 0; x < 3; ++x) {
      if ((A.nodes >> x) & 1) {
        Fr s = eval_summand(P, sm);
        acc[x] = fe_add(acc[x], fe_mul(w, s));
      }
      if (x == 0 && !((A.nodes >> 1) & 1)) {  // straight to node 2: lo + 2 step
        for (int k = 0; k < A.n_val_slots; ++k) {
          const Fr st = sm_ld(sm, A.slots_step0 + k);
          sm_st(sm, k, fe_add(sm_ld(sm, k), fe_add(st, st)));
        }
        ++x;
      } else if (x < 2) {
        for (int k = 0; k < A.n_val_slots; ++k) sm_st(sm, k, fe_add(sm_ld(sm, k), sm_ld(sm, A.slots_step0 + k)));
      }
    }
  }
  }
  round_finish_threads(A, acc, ws, partials);
}

// A summand as a factored quadratic form in its tables,
//   S = sum_g T_{a_g} (d_g + sum_t B_gt T_{b_gt}),
// a group's factor or its constant possibly absent (kNoTable: 1; kNoConst: 0).
// What most summands are: a halving list's products, a zerocheck's gate, a
// family circuit's 131 gates merged (QuadForm, below).
constexpr uint16_t kNoTable = 0xffff;
constexpr uint32_t kNoConst = 0xffffffffu;
enum TermKind : uint16_t { TERM_MUL = 0, TERM_PLUS = 1, TERM_MINUS = 2 };  // B, 1, -1

struct FormGroup {
  uint16_t a, n;
  uint32_t off, d;  // first term (and its coefficient); the constant's coefficient
};
struct FormTerm {
  uint16_t b, kind;
};
struct DevForm {
  const FormGroup* groups;
  const FormTerm* terms;
  const Fr* coeffs;
  int ng;
};

// A round of a factored quadratic form, staged through shared memory. A block
// takes 2^log_pp pairs at a time, nshare warps a tile of them: they fold the tile's
// lines of every table with the previous challenge (a line a thread) and leave each
// line's values at the round's nodes in shared memory; then each takes every
// nshare-th group of terms, so its lanes run the same terms and read the same
// coefficients. Both the inner sums and the sum over the groups stay
// unreduced (wide_mac): 64 products a term instead of 136. A tile is 16 pairs at
// two nodes; at three nodes 32 pairs in three passes (two of 16 pairs at nodes 0
// and 2, one of 32 at node 1) or, where so many pairs' values are too much shared
// memory, 8 pairs at three nodes and a quarter of the lanes idle. The small
// rounds' chain is two folds, a share of the groups and the pair's weight; a
// value's 16-byte halves lie apart so that lanes of consecutive pairs read
// consecutive 16 bytes. Measured on a GB300: the first rounds of a shard circuit's
// row-wise list over 2^21 rows 2791 and 1287 us with the interpreter, 1669 and
// 721 so; of add_sub's list 0 (131 gates, 69 columns) over 2^16 992 us a pair a
// warp, 396 so; small rounds of such lists 42-83 -> 18-45 us.
constexpr int kFormMaxWarps = 16;

__device__ __forceinline__ Fr form_ld(const uint4* val, int at, int pp) {
  const uint4 u = val[at], v = val[at + pp];
  Fr r;
  r.v[0] = u.x, r.v[1] = u.y, r.v[2] = u.z, r.v[3] = u.w;
  r.v[4] = v.x, r.v[5] = v.y, r.v[6] = v.z, r.v[7] = v.w;
  return r;
}

__device__ __forceinline__ void form_st(uint4* val, int at, int pp, const Fr& a) {
  val[at] = make_uint4(a.v[0], a.v[1], a.v[2], a.v[3]);
  val[at + pp] = make_uint4(a.v[4], a.v[5], a.v[6], a.v[7]);
}

// WARPS: the most a block has. At 8 the registers (128, no spills; three
// blocks of 80 spill and are 7 % slower) leave two blocks of 256 threads an SM, at
// 16 (small rounds, where a block's shares count) one of 512.
template <int WARPS, int BLOCKS, bool SUB>
__global__ void __launch_bounds__(32 * WARPS, BLOCKS)
    k_round_form(RoundArgs A, DevForm F, VirtualRound V, int nshare, int log_pp, int passes, Fr* partials) {
  chain_begin();
  extern __shared__ uint4 val[];  // node xi of table k, pair i, half q: ((k nn + xi) 2 + q) pp + i
  __shared__ Fr ws[3 * WARPS];
  const int three = (A.nodes >> 1) & 1, nn = 2 + three, pp = 1 << log_pp;
  const int ns = A.nd + A.nv;  // slots; eq's weights stand in slot ns, node 0
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  // Lanes of a pass: 2^log_l pairs a node, the nodes from lane slot 0 on (the
  // idle quarter of the 8-pair tile repeats the last node). SUB: the tile has fewer
  // pairs, and the lanes beyond them take shares of the groups too.
  const int log_l = three && passes == 1 ? 3 : 4, slot = lane >> log_l;
  const int log_t = passes == 3 ? 5 : log_l, log_tp = min(log_pp, log_t);
  const int share = warp % nshare, group = warp / nshare, tile = group << log_t;
  const int log_sub = SUB ? log_l - log_tp : 0, step_g = nshare << log_sub;
  const int first_g = SUB ? share + nshare * ((lane & ((1 << log_l) - 1)) >> log_tp) : share;
  // The warps of a tile are a group: they fold its lines and wait for one another only.
  auto group_sync = [&]() {
    if (nshare == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(32 * nshare) : "memory");
  };
  Fr acc = fe_zero<FrConsts>(), acc1 = fe_zero<FrConsts>();  // (acc1: node 1 of the third pass)
  for (size_t p0 = (size_t)blockIdx.x << log_pp; p0 < A.npairs; p0 += (size_t)gridDim.x << log_pp) {
    for (int t = 32 * share + lane; t < (ns + 1) << log_tp; t += 32 * nshare) {
      const int k = t >> log_tp, at = tile + (t & ((1 << log_tp) - 1));
      const size_t pair = p0 + at;
      if (pair >= A.npairs) continue;
      Fr lo, hi;
      if (k < A.nd || k == ns) {
        load_line<true>(A, k == ns ? A.nd : k, pair, lo, hi);
      } else {
        virtual_line_dev(V, A.vkinds[k - A.nd], pair, lo, hi);
        hi = fe_add(lo, hi);
      }
      uint4* o = val + (size_t)(k * nn) * 2 * pp;
      if (k == ns) {
        form_st(o, at, pp, fe_add(lo, hi));  // the pair's weight without the current variable's factor
        continue;
      }
      form_st(o, at, pp, lo);
      if (three) form_st(o, 2 * pp + at, pp, hi);
      form_st(o, (nn - 1) * 2 * pp + at, pp, fe_sub(fe_add(hi, hi), lo));
    }
    group_sync();
    for (int pass = 0; pass < passes; ++pass) {
      const int i = tile + (pass == 2 ? lane : (pass << 4) + (lane & ((1 << (log_l - log_sub)) - 1)));
      const int xi = pass == 2 ? 1 : passes == 3 ? 2 * slot : min(slot, nn - 1);
      if (i >= pp || p0 + i >= A.npairs) continue;
      const uint4* mine = val + xi * 2 * pp + i;
      const int step = nn * 2 * pp;  // between tables
      Fr s = fe_zero<FrConsts>();
      FeWide<FrConsts> outer = wide_zero<FrConsts>();
      int no = 0;
      for (int g = first_g; g < F.ng; g += step_g) {
        const FormGroup G = F.groups[g];
        Fr in = G.d == kNoConst ? fe_zero<FrConsts>() : ld_fe(&F.coeffs[G.d]);
        FeWide<FrConsts> sum = wide_zero<FrConsts>();
        int ni = 0;
        for (uint32_t t = G.off; t < G.off + G.n; ++t) {
          const FormTerm T = F.terms[t];
          const Fr v = form_ld(mine, T.b * step, pp);
          if (T.kind == TERM_PLUS) in = fe_add(in, v);
          else if (T.kind == TERM_MINUS) in = fe_sub(in, v);
          else {
            wide_mac(sum, ld_fe(&F.coeffs[t]), v);
            ++ni;
          }
          if (ni == kWideProducts || (ni > 0 && t + 1 == G.off + G.n)) {
            in = fe_add(in, fe_from_wide(sum));
            sum = wide_zero<FrConsts>();
            ni = 0;
          }
        }
        if (G.a == kNoTable) {
          s = fe_add(s, in);
        } else {
          wide_mac(outer, form_ld(mine, G.a * step, pp), in);
          ++no;
        }
        if (no == kWideProducts || (no > 0 && g + step_g >= F.ng)) {
          s = fe_add(s, fe_from_wide(outer));
          outer = wide_zero<FrConsts>();
          no = 0;
        }
      }
      s = rmul(form_ld(val + i, ns * step, pp), s);
      if (pass == 2) acc1 = fe_add(acc1, s);
      else if (slot < nn) acc = fe_add(acc, s);
    }
    group_sync();
  }
  // The warp's sum a node, from the slot's first lane.
#pragma unroll 1
  for (int off = 1; off < 1 << log_l; off <<= 1) {
    Fr o;
#pragma unroll
    for (int w = 0; w < 8; ++w) o.v[w] = __shfl_xor_sync(0xffffffffu, acc.v[w], off);
    acc = fe_add(acc, o);
  }
  if (passes == 3) acc1 = warp_sum(acc1, 32, 0xffffffffu);
  const int node = three && passes == 1 ? slot : 2 * slot;
  if (lane == 0 && !(three && passes == 1)) ws[3 * warp + 1] = acc1;  // (zero at two nodes)
  if ((lane & ((1 << log_l) - 1)) == 0 && slot < nn) ws[3 * warp + node] = acc;
  round_finish(A, ws, nwarps, partials);
}

typedef void (*FormKernel)(RoundArgs, DevForm, VirtualRound, int, int, int, Fr*);
inline FormKernel form_kernel(unsigned threads, bool sub) {
  if (threads <= 256) return sub ? k_round_form<8, 2, true> : k_round_form<8, 2, false>;
  return sub ? k_round_form<kFormMaxWarps, 1, true> : k_round_form<kFormMaxWarps, 1, false>;
}

// Wide gate lists (many gates, many tables): one warp per pair. The pair's
// tables sit once in the warp's shared slots (values, then cached entries,
// then steps, then eq's value and step), written lane-parallel; at each node
// the lanes split the gates and the warp adds their weighted values.
// Five resident blocks a SM (96 registers, no spills) measured about 1 %
// faster than the unconstrained allocation (128 registers, four blocks).
#ifndef APG_ROUND_WARP_MIN_BLOCKS
#define APG_ROUND_WARP_MIN_BLOCKS 5
#endif
template <bool OUTLINE>
__global__ void __launch_bounds__(kRoundThreads, APG_ROUND_WARP_MIN_BLOCKS) k_round_warp(RoundArgs A, DevProgram P, VirtualRound V,
                                                              Fr* partials) {
  extern __shared__ uint32_t sm_raw[];
  __shared__ Fr ws[3 * kRoundThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int per_warp = A.slots_step0 + A.n_val_slots + 2;
  const Slots S = warp_slots(sm_raw + (size_t)warp * per_warp * 8, per_warp);
  const int eq_slot = per_warp - 2;
  Fr acc[3];
#pragma unroll
  for (int x = 0; x < 3; ++x) acc[x] = fe_zero<FrConsts>();
  const size_t wstride = (size_t)gridDim.x * nwarps;
  for (size_t i = (size_t)blockIdx.x * nwarps + warp; i < A.npairs; i += wstride) {
    Fr lo, hi;
    for (int k = lane; k <= A.nd; k += 32) {
      load_line<OUTLINE>(A, k, i, lo, hi);
      if (k < A.nd) {
        sm_st(S, k, lo);
        sm_st(S, A.slots_step0 + k, fe_sub(hi, lo));
      } else {
        sm_st(S, eq_slot, fe_add(lo, hi));  // the pair's eq weight without the current variable's factor
      }
    }
    for (int v = lane; v < A.nv; v += 32) {
      virtual_line_dev(V, A.vkinds[v], i, lo, hi);  // hi is the step here
      sm_st(S, A.nd + v, lo);
      sm_st(S, A.slots_step0 + A.nd + v, hi);
    }
    __syncwarp();
    for (int x = 0; x < 3; ++x) {
      if ((A.nodes >> x) & 1) {  // uniform across the warp
        if (lane == 0)
          for (int g = 0; g < P.n_cached; ++g) sm_st(S, P.cached_slot0 + g, eval_gate_dev(P, g, S));
        __syncwarp();
        Fr part = fe_zero<FrConsts>();
        for (int j = lane; j < P.n_weighted; j += 32)
          part = fe_add(part, weigh(P, j, eval_gate_dev(P, P.n_cached + j, S)));
        for (int off = 16; off > 0; off >>= 1) {
          Fr o;
#pragma unroll
          for (int w = 0; w < 8; ++w) o.v[w] = __shfl_xor_sync(0xffffffffu, part.v[w], off);
          part = fe_add(part, o);
        }
        if (lane == 0) acc[x] = fe_add(acc[x], OUTLINE ? rmul(sm_ld(S, eq_slot), part) : fe_mul(sm_ld(S, eq_slot), part));
      }
      __syncwarp();
      if (x == 0 && !((A.nodes >> 1) & 1)) {  // straight to node 2: lo + 2 step
        for (int k = lane; k < A.n_val_slots; k += 32) {
          const Fr st = sm_ld(S, A.slots_step0 + k);
          sm_st(S, k, fe_add(sm_ld(S, k), fe_add(st, st)));
        }
        ++x;
      } else if (x < 2) {
        for (int k = lane; k < A.n_val_slots; k += 32) sm_st(S, k, fe_add(sm_ld(S, k), sm_ld(S, A.slots_step0 + k)));
      }
      __syncwarp();
    }
  }
  if (lane == 0)
#pragma unroll
    for (int x = 0; x < 3; ++x) ws[3 * warp + x] = acc[x];
  round_finish(A, ws, nwarps, partials);
}

// Tables of length 2 -> their bound value (the last round's fold).
// With no rounds at all (a one-entry table) c is ignored and the entry itself
// is the value.
// One block; the values and then the flag go to pinned host memory.
__global__ void k_final_bind(const Fr* const* src, const uint8_t* src_bits, const Fr* in_base, size_t in_len,
                             int in_is_src, int nt, Fr c, int no_rounds, Fr* out, uint32_t* flag, uint32_t seq) {
  chain_begin();
  for (int k = threadIdx.x; k < nt; k += blockDim.x) {
    const Fr* t = in_is_src ? src[k] : in_base + (size_t)k * in_len;
    const int bits = in_is_src && src_bits ? src_bits[k] : 0;
    const Fr a0 = bits ? narrow_entry(t, bits, 0) : ld_fe(&t[0]);
    if (no_rounds) {
      st_fe(&out[k], a0);
      continue;
    }
    const Fr a1 = bits ? narrow_entry(t, bits, 1) : ld_fe(&t[1]);
    st_fe(&out[k], fe_add(a0, rmul(c, fe_sub(a1, a0))));
  }
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) *reinterpret_cast<volatile uint32_t*>(flag) = seq;
}

// The source tables' entries, table after table, into pinned host memory, then
// the flag (one block: the few entries the host takes over).
__global__ void k_gather(const Fr* const* src, const uint8_t* src_bits, int nt, size_t len, Fr* out, uint32_t* flag,
                         uint32_t seq) {
  chain_begin();
  for (size_t t = threadIdx.x; t < nt * len; t += blockDim.x) {
    const int k = (int)(t / len);
    const int bits = src_bits ? src_bits[k] : 0;
    st_fe(&out[t], bits ? narrow_entry(src[k], bits, t - k * len) : ld_fe(&src[k][t - k * len]));
  }
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) *reinterpret_cast<volatile uint32_t*>(flag) = seq;
}

__global__ void k_lift(const void* p, int bits, size_t n, Fr* out) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) st_fe(&out[i], narrow_entry(p, bits, i));
}

// eq(r, y) = prod_j (y_j ? r_j : 1 - r_j) for every y < 2^n, a block 1024
// consecutive y: the low ten variables as the product of two tables of five, the
// others one factor for the block, folded into the first table. About eleven
// products after one another whatever n, and one an entry (chains of n products
// with their factors in device memory, three launches above 2^12: 345 us over the
// 22 lists of a 10-column 2^21-row proof on a GB300, now 226).
struct EqPoint {
  Fr r[40];
};
constexpr int kEqLow = 10;

__device__ __forceinline__ Fr eq_factor(const Fr& r, bool bit) { return bit ? r : fe_sub(fe_one<FrConsts>(), r); }

__global__ void __launch_bounds__(256) k_eq_table(const __grid_constant__ EqPoint P, int n, Fr* out) {
  chain_begin();
  __shared__ Fr tab[2][1 << (kEqLow / 2)], high;
  const int nl = min(n, kEqLow), na = nl / 2, t = threadIdx.x, lane = t & 31;
  if (t < 64) {
    const int h = t >> 5, first = h ? na : 0, bits = h ? nl - na : na;
    if (lane < 1 << bits) {
      Fr a = fe_one<FrConsts>();
      for (int j = 0; j < bits; ++j) a = rmul(a, eq_factor(P.r[first + j], (lane >> j) & 1));
      tab[h][lane] = a;
    }
  } else if (t < 96) {
    Fr a = nl + lane < n ? eq_factor(P.r[nl + lane], (blockIdx.x >> lane) & 1) : fe_one<FrConsts>();
    for (int off = 1; off < n - nl; off <<= 1) {
      Fr o;
#pragma unroll
      for (int w = 0; w < 8; ++w) o.v[w] = __shfl_down_sync(0xffffffffu, a.v[w], off);
      if (lane + off < 32) a = rmul(a, o);
    }
    if (lane == 0) high = a;
  }
  __syncthreads();
  if (n > nl && t < 1 << na) tab[0][t] = rmul(tab[0][t], high);
  __syncthreads();
  for (int e = t; e < 1 << nl; e += 256)
    st_fe(&out[((size_t)blockIdx.x << nl) + e], rmul(tab[0][e & ((1 << na) - 1)], tab[1][e >> na]));
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

using host::F;

static Fr to_dev(const F& a) {
  Fr r;
  memcpy(r.v, a.w, 32);
  return r;
}

void lift_column(Ctx& c, const void* p, int bits, size_t n, Fr* out) {
  if (n) launch(c, k_lift, (unsigned)((n + 255) / 256), 256, 0, p, bits, n, out);
}

void build_eq_table(Ctx& c, const std::vector<F>& r, Fr* out) {
  const int n = (int)r.size();
  EqPoint p;
  if (n > (int)(sizeof(p.r) / sizeof(Fr))) throw Error(APG_ERR_INVALID_ARGUMENT, "an eq table of more than 40 variables");
  memset(&p, 0, sizeof(p));
  if (n) memcpy(p.r, r.data(), 32 * (size_t)n);
  launch_chained(c, k_eq_table, 1u << std::max(0, n - kEqLow), 256, 0, p, n, out);
}

static VirtualRound virtual_round(const std::vector<F>& point, int nvars) {
  using namespace host;
  VirtualRound V;
  memset(&V, 0, sizeof(V));
  const int b = (int)point.size();
  V.bound = b;
  V.nvars = nvars;
  F row = fzero(), r19 = fzero(), r16 = fzero(), q = fone(), pw = fone();
  for (int j = 0; j < b; ++j) {
    F t = fmul(point[j], pw);
    row = fadd(row, t);
    if (j < 19) r19 = fadd(r19, t);
    if (j < 16) r16 = fadd(r16, t);
    if (j >= 14) q = fmul(q, fsub(fone(), point[j]));
    if (j < 16) V.r16[j] = to_dev(point[j]);
    pw = fadd(pw, pw);
  }
  V.row_prefix = to_dev(row);
  V.range19_prefix = to_dev(r19);
  V.range16_prefix = to_dev(r16);
  V.ram_q = to_dev(q);
  V.pow2_b = to_dev(pw);
  return V;
}

// The host's side of a factored quadratic form (k_round_form).
struct HostForm {
  std::vector<FormGroup> groups;  // by falling cost
  std::vector<FormTerm> terms;
  std::vector<F> coeffs;  // one a term, then the groups' constants
  size_t cost = 0;        // wide products a node
  size_t muls = 0;        // products a node
};
bool quadratic_form(const HostProgram& hp, int slots, int n, HostForm& out);

// How many of a short form's last rounds run on the host. Both sides
// pay the transcript's permutations (6 us each: three a round on the device's
// way, which hides one, four on the host's); a device round adds its launch, a
// kernel of about 10 us and the flag, a host round its products at 20 ns: two a
// table to bind and up to two a term and node. So the host takes the rounds of
// up to kHostTailProducts products; its tables then fit the pinned buffer.
// Measured on a GB300 at 0, 200, 600 and 1500: a 2^8-row zerocheck of a*b 396,
// 352, 356, 381 us, 2^16 rows 807, 754, 743, 774, the GKR proof of a 7-column
// 2^12-row shard 4528, 4290, 4343, 4496.
constexpr size_t kHostTailProducts = 200;
static int host_tail_rounds(int n, int nd, const HostForm& f) {
  const size_t nt = (size_t)nd + 1, per_pair = 2 * nt + 2 * f.muls + 2;
  int k = 0;
  while (k < n && (per_pair << k) <= kHostTailProducts) ++k;
  if (n == k + 1) ++k;  // round 0 binds nothing: a list this short is gathered whole
  while (k > 0 && (nt << (k + 1)) * 32 > Ctx::kPinnedBytes - Ctx::kPinnedTables) --k;
  return n == k + 1 ? 0 : k;
}

// k_round_form's block: `share` warps split the groups of each tile of pairs.
struct FormShape {
  int share, log_pp, passes;
  unsigned threads, blocks;
  size_t smem;
  bool sub;
};
constexpr size_t kFormSmemMax = 200 * 1024;
constexpr size_t kFormSmem = 48 * 1024;       // (20, 28, 36, 72, 100 KB: within 1 % or up to 6 % slower)
constexpr size_t kFormSmemThree = 40 * 1024;  // (three passes: zerochecks 5 % faster, 21-table lists 1 % slower)
constexpr size_t kFormShareCost = 2000;       // (500, 1000: a 10-column 2^21-row GKR proof 17 %, 5 % slower)
static FormShape form_shape(const HostForm& f, size_t npairs, int slots, bool three, int sm_count) {
  const size_t line = (size_t)(slots + 1) * (three ? 3 : 2) * sizeof(Fr);  // a pair's values
  FormShape s;
  s.sub = false;
  s.passes = three && line * 32 <= kFormSmemThree ? 3 : 1;
  const int log_p = s.passes == 3 ? 5 : three ? 3 : 4;  // a tile
  s.log_pp = log_p;
  if (npairs <= ((size_t)sm_count * 2 << 4)) {
    // About a tile a block: every warp a share of its own, and few enough lines
    // a block that a thread folds one or two.
    s.share = f.groups.size() > 16 ? kFormMaxWarps : 8;
    s.threads = 32 * s.share;
    while (s.log_pp > 0 && ((size_t)1 << (s.log_pp - 1)) >= npairs) --s.log_pp;
    while (s.log_pp > 0 && ((size_t)(slots + 1) << s.log_pp) > 2 * s.threads && (npairs >> (s.log_pp - 1)) <= (size_t)sm_count)
      --s.log_pp;
    // More groups than warps: the lanes without a pair take some, and a block fewer
    // pairs while a lane still has several (a zerocheck of 560 products over 40 columns
    // of 2^8 rows 1233 us with a warp's groups after one another, 1040 so). A form of
    // its own, because the other lists' small rounds lose 1.5 us to it.
    s.sub = s.passes == 1 && f.groups.size() > (size_t)s.share;
    while (s.sub && s.log_pp > 0 && f.groups.size() > (size_t)s.share << (log_p - s.log_pp) &&
           (npairs >> (s.log_pp - 1)) <= (size_t)sm_count)
      --s.log_pp;
    s.sub = s.sub && s.log_pp < log_p;
  } else {
    // As many tiles as the shared memory of four blocks an SM takes, and a
    // share for every two thousand wide products (a share costs its own weight
    // and reduction, 270). Blocks of four warps, four to an SM, where the values
    // fit: their folds, which wait for memory, run beside others' products
    // (zerochecks of 2^21 rows 1485 and 1783 us with two blocks of eight, 1445 and
    // 1711 so).
    int tiles = 1, share = 1;
    const int warps = (line << log_p) * 4 <= kFormSmemMax ? 4 : 8;
    while (tiles < warps && line * ((size_t)2 * tiles << log_p) <= kFormSmem) tiles *= 2;
    while (share * tiles < warps && ((size_t)share * 2 * kFormShareCost <= f.cost || share * tiles < 4)) share *= 2;
    s.share = share;
    s.threads = 32 * share * tiles;
    for (int t = tiles; t > 1; t /= 2) ++s.log_pp;
  }
  while (s.log_pp > 0 && (line << s.log_pp) > kFormSmemMax) {
    --s.log_pp;
    if (s.log_pp >= log_p) s.threads /= 2;
  }
  s.smem = line << s.log_pp;
  s.blocks = (unsigned)std::min<size_t>((npairs + ((size_t)1 << s.log_pp) - 1) >> s.log_pp, (size_t)sm_count * 8);
  return s;
}

void run_sumcheck(Ctx& c, const HostProgram& hp, int nd, const std::vector<uint8_t>& vkinds,
                  const std::vector<const Fr*>& src, const std::vector<F>& eq_point, host::Transcript& tr,
                  std::vector<std::array<F, 4>>& rounds, std::vector<F>& point, std::vector<F>& finals,
                  const std::vector<uint8_t>& src_bits) {
  const int n = (int)eq_point.size();
  const int nt = nd + 1;  // with eq
  if (vkinds.size() > 8) throw Error(APG_ERR_BAD_CIRCUIT, "more than 8 virtual tables");
  rounds.clear();
  point.clear();
  finals.assign(nd, host::fzero());
  const size_t len0 = (size_t)1 << n;
  Fr* eq = c.scratch[S_TMP3].as<Fr>(len0);
  build_eq_table(c, eq_point, eq);

  const int n_val = nd + (int)vkinds.size(), n_cached = hp.n_cached;
  HostForm form;
  const bool use_form = (size_t)(n_val + 1) * 3 * sizeof(Fr) <= kFormSmemMax && quadratic_form(hp, n_val, n, form);
  const int host_rounds = use_form && vkinds.empty() ? host_tail_rounds(n, nd, form) : 0;

  // One upload: the counter of finished blocks (zero), the round-0 sources (the
  // data tables, then eq), their stored widths when any is narrow (eq is Fr)
  // and the form or the program. `up` lives until the copy from it has surely run (the rounds).
  bool narrow = false;
  for (uint8_t b : src_bits) narrow |= b != 0;
  if (narrow && (int)src_bits.size() != nd) throw Error(APG_ERR_INTERNAL, "one width per data table");
  std::vector<const Fr*> srcs(src);
  srcs.push_back(eq);
  std::vector<uint8_t> bits(narrow ? src_bits : std::vector<uint8_t>());
  if (narrow) bits.push_back(0);
  Packer up;
  const uint32_t zero[8] = {0};
  up.put(zero, sizeof(zero));
  const size_t at_src = up.put(srcs.data(), sizeof(Fr*) * nt), at_bits = up.put(bits.data(), bits.size()),
               at_g = up.put(form.groups.data(), form.groups.size() * sizeof(FormGroup)),
               at_t = up.put(form.terms.data(), form.terms.size() * sizeof(FormTerm)),
               at_c = up.put(form.coeffs.data(), form.coeffs.size() * 32);
  PackedProgram packed{};
  if (!use_form) packed = pack_program(hp, up);
  uint8_t* d_up = c.scratch[S_PAIR_TERMS].as<uint8_t>(up.bytes.size());
  c.copy(d_up, up.bytes.data(), up.bytes.size(), cudaMemcpyHostToDevice);
  unsigned* done = reinterpret_cast<unsigned*>(d_up);
  const Fr** d_src = reinterpret_cast<const Fr**>(d_up + at_src);
  const uint8_t* d_bits = narrow ? d_up + at_bits : nullptr;
  DevForm DF;
  DF.groups = reinterpret_cast<const FormGroup*>(d_up + at_g);
  DF.terms = reinterpret_cast<const FormTerm*>(d_up + at_t);
  DF.coeffs = reinterpret_cast<const Fr*>(d_up + at_c);
  DF.ng = (int)form.groups.size();

  // Level buffers: level r (r >= 1) holds nt tables of 2^(n-r) entries.
  Fr* lvl[2] = {nullptr, nullptr};
  if (n >= 2) {
    lvl[1] = c.scratch[S_LEVEL_A].as<Fr>((size_t)nt * (len0 / 2));
    lvl[0] = c.scratch[S_LEVEL_B].as<Fr>((size_t)nt * (len0 / 4 > 0 ? len0 / 4 : 1));
  }
  // The interpreter's shapes (gate lists that are no quadratic form).
  // Wide gate lists get narrower blocks (a power of two, for the reduction
  // tree) so that every thread's slots still fit in shared memory.
  // (Down to 8 threads a block for the widest lists, e.g. 130-column ones.)
  const int slots = 2 * n_val + n_cached;
  int threads = kRoundThreads;
  while (threads > 8 && (size_t)std::max(slots, 1) * 32 * threads > 200 * 1024) threads /= 2;
  const size_t smem = (size_t)std::max(slots, 1) * 32 * threads;
  // Lists of many gates go one pair per warp (k_round_warp): the pair's
  // tables are stored once for the warp instead of once per thread.
  const bool warp_mode = hp.n_weighted >= kWarpModeGates;
  const int max_blocks = c.sm_count * 8 * (kRoundThreads / threads);  // the same thread count in smaller blocks
  const int warp_slots = n_val + n_cached + n_val + 2;
  const size_t warp_smem = (size_t)(kRoundThreads / 32) * warp_slots * 32;
  // Rounds with few enough pairs for one warp each in a single wave run one
  // pair per warp whatever the list's width: the lanes fold the tables and
  // evaluate the gates side by side, so a round's latency is a fold and a gate,
  // not one thread's chain through every fold and gate.
  const bool small_warp_ok = warp_smem <= 200 * 1024;
  const int warp_max_blocks = c.sm_count * 16;
  DevProgram P;
  memset(&P, 0, sizeof(P));
  if (use_form) {
    for (auto k : {form_kernel(256, false), form_kernel(256, true), form_kernel(512, false), form_kernel(512, true)})
      APG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFormSmemMax));
  } else {
    if ((warp_mode ? warp_smem : smem) > 200 * 1024)
      throw Error(APG_ERR_BAD_CIRCUIT, "gate list too wide for one thread block");
    P = packed.on_device(d_up);
    P.cached_slot0 = n_val;
    APG_CUDA(cudaFuncSetAttribute(k_round, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    APG_CUDA(cudaFuncSetAttribute(k_round_warp<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    APG_CUDA(cudaFuncSetAttribute(k_round_warp<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  }
  Fr* partials = c.scratch[S_TMP6].as<Fr>((size_t)std::max(max_blocks, warp_max_blocks) * 4);
  uint8_t* pinned = c.host_pinned();
  const F* sums = reinterpret_cast<const F*>(pinned + Ctx::kPinnedSums);
  Fr* host_tables = reinterpret_cast<Fr*>(pinned + Ctx::kPinnedTables);

  // 1/r_j for every nonzero eq coordinate, from one inversion (Montgomery's
  // batch trick): the rounds divide by their coordinate. Found while the device
  // works on round 0, which needs none.
  std::vector<F> inv_r(n, host::fzero());
  auto invert_coordinates = [&]() {
    std::vector<F> pre(n + 1, host::fone());
    for (int j = 0; j < n; ++j) pre[j + 1] = eq_point[j].zero() ? pre[j] : host::fmul(pre[j], eq_point[j]);
    F inv = host::finv(pre[n]);
    for (int j = n; j-- > 0;) {
      if (eq_point[j].zero()) continue;
      inv_r[j] = host::fmul(inv, pre[j]);
      inv = host::fmul(inv, eq_point[j]);
    }
  };
  F chal = host::fzero();
  // The round polynomial factors as s(X) = eq_r(X) q(X): eq's factor for this
  // variable, eq_r(X) = (1 - r_r)(1 - X) + r_r X, is common to every pair, and
  // the rest of a pair's eq weight is e(2i) + e(2i + 1). q has degree 2 and is
  // summed at nodes 0 and 2; from the second round on q(1) follows from s(0) +
  // s(1) = s_{r-1}(c_{r-1}), which holds for any tables because the bound tables
  // are the lines at c. Round 0, and a round whose eq coordinate is 0, sum at
  // node 1 as well.
  auto needs_one = [&](int r) { return r == 0 || eq_point[r].zero(); };
  // A round from its sums q(0), q(1) (when needed) and q(2): the cubic onto the
  // transcript (whose tag and length have been absorbed), the next challenge.
  auto close_round = [&](int r, F q[4]) {
    const F rr = eq_point[r], one_m_r = host::fsub(host::fone(), rr);
    if (!needs_one(r)) {
      const auto& gp = rounds.back();  // s_{r-1}(X), ascending coefficients
      const F claim = host::fadd(
          gp[0], host::fmul(chal, host::fadd(gp[1], host::fmul(chal, host::fadd(gp[2], host::fmul(chal, gp[3]))))));
      q[1] = host::fmul(host::fsub(claim, host::fmul(one_m_r, q[0])), inv_r[r]);
    }
    // q(3) = q(0) - 3 q(1) + 3 q(2); s(X) = eq_r(X) q(X) with eq_r(X) = 1 - r - X + 2 r X.
    const F three = host::from_u64(3);
    q[3] = host::fadd(q[0], host::fmul(three, host::fsub(q[2], q[1])));
    F sv[4];
    F eqx = one_m_r;                          // eq_r(0)
    const F step = host::fsub(host::fadd(rr, rr), host::fone());  // eq_r(X + 1) - eq_r(X) = 2r - 1
    for (int x = 0; x < 4; ++x) {
      sv[x] = host::fmul(eqx, q[x]);
      eqx = host::fadd(eqx, step);
    }
    auto g = host::cubic_through(sv);
    for (const F& v : g) tr.observe(v);
    chal = tr.challenge(host::T_SUMCHECK_CHALLENGE);
    rounds.push_back(g);
    point.push_back(chal);
  };
  typedef std::chrono::steady_clock Clock;
  auto count_host = [&](Clock::time_point t0) {
    if (!c.timers.on) return;  // the host's share of a round: interpolation and the transcript step
    c.timers.ms[APG_TIMER_HOST_ROUND] += std::chrono::duration<double, std::milli>(Clock::now() - t0).count();
    c.timers.count[APG_TIMER_HOST_ROUND] += 1;
  };
  const int dev_rounds = n - host_rounds;
  for (int r = 0; r < dev_rounds; ++r) {
    RoundArgs A;
    memset(&A, 0, sizeof(A));
    A.nd = nd;
    A.nv = (int)vkinds.size();
    for (size_t v = 0; v < vkinds.size(); ++v) A.vkinds[v] = vkinds[v];
    A.src = d_src;
    A.bind = r > 0;
    A.c = to_dev(chal);
    A.in_is_src = r <= 1;
    A.in_len = (size_t)1 << (n - r + (r > 0 ? 1 : 0));
    A.in_base = r >= 2 ? lvl[(r - 1) & 1] : nullptr;
    // (the last level before the host's rounds lands where the host reads it)
    A.out_base = r < 1 ? nullptr : host_rounds && r == dev_rounds - 1 ? host_tables : lvl[r & 1];
    A.to_host = A.out_base == host_tables;
    A.npairs = (size_t)1 << (n - r - 1);
    A.slots_step0 = n_val + n_cached;
    A.n_val_slots = n_val;
    A.done = done;
    A.out = reinterpret_cast<Fr*>(pinned + Ctx::kPinnedSums);
    A.flag = reinterpret_cast<uint32_t*>(pinned);
    A.seq = ++c.flag_seq;
    VirtualRound V = virtual_round(point, n);
    // Rounds too small to fill the device evaluate the nodes of a pair on
    // threads of their own.
    A.xsplit = A.npairs * 4 <= (size_t)threads * max_blocks ? 1 : 0;
    A.src_bits = d_bits;
    A.nodes = needs_one(r) ? 7 : 5;
    const size_t work = A.xsplit ? A.npairs * 4 : A.npairs;
    const int blocks = warp_mode
                           ? (int)std::min<size_t>((A.npairs + kRoundThreads / 32 - 1) / (kRoundThreads / 32),
                                                   (size_t)warp_max_blocks)
                           : (int)std::min<size_t>((work + threads - 1) / threads, (size_t)max_blocks);
    cudaEvent_t t0 = c.timer_begin();
    if (use_form) {
      const FormShape f = form_shape(form, A.npairs, n_val, needs_one(r), c.sm_count);
      launch_chained(c, form_kernel(f.threads, f.sub), f.blocks, f.threads, f.smem, A, DF, V, f.share, f.log_pp, f.passes, partials);
    }
    else if (small_warp_ok && A.npairs * 32 <= (size_t)kRoundThreads * c.sm_count * 4)
      launch(c, k_round_warp<true>, (int)((A.npairs + kRoundThreads / 32 - 1) / (kRoundThreads / 32)), kRoundThreads,
             warp_smem, A, P, V, partials);
    else if (warp_mode) launch(c, k_round_warp<false>, blocks, kRoundThreads, warp_smem, A, P, V, partials);
    else launch(c, k_round, blocks, threads, smem, A, P, V, partials);
    c.timer_end(APG_TIMER_SUMCHECK_ROUND, t0);
    // While the device works: the message's tag and length need no sums.
    tr.open(host::T_SUMCHECK_ROUND, 4);
    if (r == 0 && n > 1) invert_coordinates();
    c.wait_flag();
    const auto host0 = Clock::now();
    F q[4] = {sums[0], sums[1], sums[2], host::fzero()};
    close_round(r, q);
    count_host(host0);
  }
  if (host_rounds > 0) {
    if (dev_rounds == 0) {
      launch_chained(c, k_gather, 1, 256, 0, (const Fr* const*)d_src, d_bits, nt, len0, host_tables,
             reinterpret_cast<uint32_t*>(pinned), ++c.flag_seq);
      if (n > 1) invert_coordinates();
      c.wait_flag();
    }
    // Level dev_rounds - 1 (or the source tables), still to be bound with the last challenge.
    const F* t0 = reinterpret_cast<const F*>(host_tables);
    size_t len = (size_t)1 << (host_rounds + (dev_rounds > 0 ? 1 : 0));
    std::vector<F> tab(t0, t0 + nt * len);
    auto bind = [&]() {
      for (size_t k = 0; k < (size_t)nt; ++k)
        for (size_t i = 0; i < len / 2; ++i) {
          const F lo = tab[k * len + 2 * i], hi = tab[k * len + 2 * i + 1];
          tab[k * (len / 2) + i] = host::fadd(lo, host::fmul(chal, host::fsub(hi, lo)));
        }
      len /= 2;
    };
    if (dev_rounds > 0) bind();
    for (int r = dev_rounds; r < n; ++r) {
      const auto host0 = Clock::now();
      F q[4] = {host::fzero(), host::fzero(), host::fzero(), host::fzero()};
      for (size_t i = 0; i < len / 2; ++i) {
        const F* e = tab.data() + nd * len + 2 * i;
        const F w = host::fadd(e[0], e[1]);
        for (int x = 0; x < 3; ++x) {
          if (x == 1 && !needs_one(r)) continue;
          auto at = [&](uint16_t k) {
            const F* t = tab.data() + k * len + 2 * i;
            return x == 0 ? t[0] : x == 1 ? t[1] : host::fsub(host::fadd(t[1], t[1]), t[0]);
          };
          F s = host::fzero();
          for (const FormGroup& G : form.groups) {
            F in = G.d == kNoConst ? host::fzero() : form.coeffs[G.d];
            for (uint32_t t = G.off; t < G.off + G.n; ++t) {
              const F v = at(form.terms[t].b);
              const uint16_t kind = form.terms[t].kind;
              in = kind == TERM_MINUS ? host::fsub(in, v)
                                      : host::fadd(in, kind == TERM_PLUS ? v : host::fmul(form.coeffs[t], v));
            }
            s = host::fadd(s, G.a == kNoTable ? in : host::fmul(at(G.a), in));
          }
          q[x] = host::fadd(q[x], host::fmul(w, s));
        }
      }
      tr.open(host::T_SUMCHECK_ROUND, 4);
      close_round(r, q);
      bind();
      count_host(host0);
    }
    for (int k = 0; k < nd; ++k) finals[k] = tab[k];
    return;
  }
  // The last fold: every table bound to the full point.
  if (nd > 0) {
    const Fr* base = n >= 2 ? lvl[(n - 1) & 1] : nullptr;
    const bool in_pinned = (size_t)nd * 32 <= Ctx::kPinnedBytes - Ctx::kPinnedTables;
    Fr* d_fin = in_pinned ? host_tables : c.scratch[S_TMP7].as<Fr>(nt);
    launch_chained(c, k_final_bind, 1, 256, 0, (const Fr* const*)d_src, d_bits, base, (size_t)2, n <= 1 ? 1 : 0, nd,
           to_dev(chal), n == 0 ? 1 : 0, d_fin, reinterpret_cast<uint32_t*>(pinned), ++c.flag_seq);
    if (!in_pinned)
      c.copy(finals.data(), d_fin, 32 * (size_t)nd, cudaMemcpyDeviceToHost);
    c.wait_flag();
    if (in_pinned) memcpy(finals.data(), host_tables, 32 * (size_t)nd);
    else APG_CUDA(cudaStreamSynchronize(c.stream));
  } else {
    APG_CUDA(cudaStreamSynchronize(c.stream));
  }
}

// A device copy of a resolved gate list.
namespace {

// A polynomial of degree two at most in the slots: terms keyed by their two slots,
// the lower one high, kNoTable for an absent second one. Terms are appended as they
// come and merged once (a tree of them took 46 us more of a call with 560 terms).
struct QuadPoly {
  struct Term {
    uint32_t key;
    F v;
    uint16_t a() const { return (uint16_t)(key >> 16); }
    uint16_t b() const { return (uint16_t)key; }
  };
  F c = host::fzero();
  std::vector<Term> m;
  void add(uint16_t a, uint16_t b, const F& v) { m.push_back({a < b ? (uint32_t)a << 16 | b : (uint32_t)b << 16 | a, v}); }
  // Equal monomials added up, in the keys' order.
  void merge() {
    std::vector<uint64_t> order(m.size());
    for (size_t i = 0; i < m.size(); ++i) order[i] = (uint64_t)m[i].key << 32 | i;
    std::sort(order.begin(), order.end());
    std::vector<Term> out;
    out.reserve(m.size());
    for (uint64_t o : order) {
      const Term& t = m[(uint32_t)o];
      if (!out.empty() && out.back().key == t.key) out.back().v = host::fadd(out.back().v, t.v);
      else out.push_back(t);
    }
    m.swap(out);
  }
};

// Adds w times the gate's value to `out`, over the operands as they stand (a cached
// entry counts as a slot of its own).
void add_gate(const HostProgram& hp, const DevGate& g, const F& w, QuadPoly& out) {
  const F* c = hp.coeffs.data() + g.cf_off;
  const uint16_t* o = hp.ops.data() + g.op_off;
  const bool unit = w == host::fone();
  auto weighed = [&](const F& v) { return unit ? v : host::fmul(w, v); };
  const int t = g.p1, u = g.p2;
  switch (g.kind) {
    case G_LINEAR:
      for (int i = 0; i < t; ++i) out.add(o[i], kNoTable, weighed(c[i]));
      out.c = host::fadd(out.c, weighed(c[t]));
      break;
    case G_PRODUCT:
      out.add(o[0], o[1], weighed(c[0]));
      break;
    case G_MASK:  // x m + 1 - m
      out.add(o[0], o[1], w);
      out.add(o[1], kNoTable, host::fneg(w));
      out.c = host::fadd(out.c, w);
      break;
    case G_AFFINE: {  // (sum l_i x_i + l_t)(sum r_k y_k + r_u)
      const F lt = weighed(c[t]), ru = c[t + 1 + u];
      for (int i = 0; i < t; ++i) {
        const F li = weighed(c[i]);
        for (int k = 0; k < u; ++k) out.add(o[i], o[t + k], host::fmul(li, c[t + 1 + k]));
        out.add(o[i], kNoTable, host::fmul(li, ru));
      }
      for (int k = 0; k < u; ++k) out.add(o[t + k], kNoTable, host::fmul(lt, c[t + 1 + k]));
      out.c = host::fadd(out.c, host::fmul(lt, ru));
      break;
    }
    case G_TREE_PRODUCT:
      out.add(o[0], o[1], w);
      break;
    case G_TREE_CROSS:
      out.add(o[0], o[3], w);
      out.add(o[1], o[2], w);
      break;
    case G_QUADRATIC:
      out.c = host::fadd(out.c, weighed(c[0]));
      for (int i = 0; i < t; ++i) out.add(o[i], kNoTable, weighed(c[1 + i]));
      for (int k = 0; k < u; ++k) out.add(o[t + 2 * k], o[t + 2 * k + 1], weighed(c[1 + t + k]));
      break;
  }
}

// p, merged, with its cached slots (from `slots` on) replaced by their polynomials:
// p = q + sum_i C_i L_i, L_i what stands beside the entry C_i (or an earlier one than
// it). L_i is added up first, so each entry is multiplied out once, however many
// products it is in. False when the degree passes two, or before multiplying where that
// takes more than `limit` terms or leaves monomials of more than `most` wide products.
bool substitute(QuadPoly& p, int slots, const std::vector<QuadPoly>& cached, size_t limit, size_t most) {
  p.merge();
  std::vector<QuadPoly> beside(cached.size());
  QuadPoly out;
  out.c = p.c;
  bool any = false;
  for (const auto& t : p.m) {
    const uint16_t a = t.a(), b = t.b();
    const uint16_t top = b == kNoTable ? a : b;  // (a <= b)
    if (top < slots) {
      out.m.push_back(t);
      continue;
    }
    any = true;
    QuadPoly& L = beside[top - slots];
    if (b == kNoTable) {
      L.c = host::fadd(L.c, t.v);
    } else if (a < slots) {
      L.add(a, kNoTable, t.v);
    } else {
      const QuadPoly& C = cached[a - slots];
      L.c = host::fadd(L.c, host::fmul(t.v, C.c));
      for (const auto& u : C.m) L.add(u.a(), u.b(), host::fmul(t.v, u.v));
    }
  }
  if (!any) return true;
  auto linear = [](const QuadPoly& q) {
    for (const auto& t : q.m)
      if (t.b() != kNoTable) return false;
    return true;
  };
  const F one = host::fone(), minus_one = host::fneg(one);
  size_t terms = 0;
  for (size_t i = 0; i < cached.size(); ++i) {
    QuadPoly& L = beside[i];
    L.merge();
    if (!L.m.empty() && !(linear(L) && linear(cached[i]))) return false;
    // Two linear forms have at least this many monomials, at 72 wide products each
    // unless their coefficients come out as 1 or -1.
    const size_t nc = cached[i].m.size(), nl = L.m.size(), both = std::min(nc, nl);
    const size_t left = nc * nl - (both > 0 ? both * (both - 1) / 2 : 0);
    size_t each = 72;
    for (const auto& t : L.m)
      if (t.v == one || t.v == minus_one) each = 8;
    if ((terms += (nc + 1) * (nl + 1)) > limit || left * each > most) return false;
  }
  for (size_t i = 0; i < cached.size(); ++i) {
    const QuadPoly &C = cached[i], &L = beside[i];
    if (L.m.empty() && L.c.zero()) continue;
    out.c = host::fadd(out.c, host::fmul(C.c, L.c));
    if (!C.c.zero())
      for (const auto& u : L.m) out.add(u.a(), kNoTable, host::fmul(C.c, u.v));
    for (const auto& t : C.m) {
      if (!L.c.zero()) out.add(t.a(), t.b(), host::fmul(t.v, L.c));
      for (const auto& u : L.m) out.add(t.a(), u.a(), host::fmul(t.v, u.v));
    }
  }
  out.merge();
  p = std::move(out);
  return true;
}

// The products a node takes gate by gate.
size_t gate_products(const HostProgram& hp, const DevGate& g) {
  const F one = host::fone(), minus_one = host::fneg(one), zero = host::fzero();
  const size_t t = g.p1, u = g.p2;
  const size_t ncoef = g.kind == G_LINEAR ? t : g.kind == G_PRODUCT ? 1 : g.kind == G_AFFINE ? t + u + 1 : g.kind == G_QUADRATIC ? 1 + t + u : 0;
  size_t products = g.kind == G_LINEAR ? 0 : g.kind == G_QUADRATIC ? u : g.kind == G_TREE_CROSS ? 2 : 1;
  for (size_t i = 0; i < ncoef; ++i) {
    const F& v = hp.coeffs[g.cf_off + i];
    products += v == one || v == minus_one || v == zero ? 0 : 1;
  }
  return products;
}

// The terms that add_gate adds for it.
size_t gate_terms(const DevGate& g) {
  const size_t t = g.p1, u = g.p2;
  return g.kind == G_AFFINE ? (t + 1) * (u + 1) : 1 + t + u;
}

}  // namespace

// The summed gate list as one factored quadratic form: every gate expanded with
// its weight and its cached operands' polynomials, equal monomials merged
// (exact arithmetic: the sum is the same at every node), then grouped greedily
// by the slot that the most remaining products share, whose linear term becomes
// its group's constant. False when the degree passes two, when the gates as
// they stand take fewer products than the form, or when finding the form costs the
// host more than the interpreter would cost the device. A term is 30 to 50 ns on the
// host; a list's product is half a microsecond or more a round in the interpreter and
// 1.3 ns a row (forty products of eight cached forms over 32 columns: 1.15 ms at 2^2
// rows, 6.2 at 2^12, 31 at 2^16, where the form takes 3.4), so a list may have ten terms
// a product and round, and one a product and 32 rows.
bool quadratic_form(const HostProgram& hp, int slots, int n, HostForm& out) {
  out = HostForm();
  if (!hp.summed || slots + hp.n_cached >= kNoTable) return false;
  const F one = host::fone(), minus_one = host::fneg(one);
  size_t products = 0, terms = 0;
  for (const DevGate& g : hp.gates) {
    products += gate_products(hp, g);
    terms += gate_terms(g);
  }
  for (const F& w : hp.weights) products += w == one ? 0 : 1;
  const size_t worth = 4 * products + products * (10 * n + (((size_t)1 << std::min(n, 30)) >> 5));
  const size_t cap = (size_t)1 << 22;  // (of 40 bytes)
  if (terms > std::min(20000 + worth, cap)) return false;
  const size_t limit = std::min(1000 + worth, cap), most = 136 * products + 1000;
  std::vector<QuadPoly> cached;
  for (int j = 0; j < hp.n_cached; ++j) {
    QuadPoly c;
    add_gate(hp, hp.gates[j], one, c);
    if (!substitute(c, slots, cached, limit, most) || c.m.size() > limit) return false;
    cached.push_back(std::move(c));
  }
  QuadPoly s;
  s.m.reserve(terms);
  for (int j = 0; j < hp.n_weighted; ++j) {
    const F w = j < (int)hp.weights.size() ? hp.weights[j] : one;
    add_gate(hp, hp.gates[hp.n_cached + j], w, s);
  }
  if (!substitute(s, slots, cached, limit, most)) return false;
  // The products by slot; the linear terms apart.
  struct Edge {
    uint16_t a, b;
    F v;
    bool used;
  };
  std::vector<Edge> edges;
  std::vector<std::vector<int>> at(slots);
  std::vector<F> lin(slots, host::fzero());
  for (auto& t : s.m) {
    if (t.v.zero()) continue;
    const uint16_t a = t.a(), b = t.b();
    if (b == kNoTable) {
      lin[a] = t.v;
      continue;
    }
    at[a].push_back((int)edges.size());
    if (b != a) at[b].push_back((int)edges.size());
    edges.push_back({a, b, t.v, false});
  }
  struct Group {
    uint16_t a;
    F d;
    std::vector<std::pair<uint16_t, F>> terms;
    size_t cost;
  };
  std::vector<Group> groups;
  auto weigh = [&](Group& g) {
    size_t mul = 0;
    for (auto& t : g.terms) mul += t.second == one || t.second == minus_one ? 0 : 1;
    out.muls += mul + (g.a == kNoTable ? 0 : 1);
    g.cost = 8 + 8 * g.terms.size() + 64 * mul + (mul ? 72 : 0) + (g.a == kNoTable ? 0 : 64);
    out.cost += g.cost;
  };
  std::priority_queue<std::pair<int, int>> open;  // (remaining products, -slot), the latest entry of a slot counts
  std::vector<int> left(slots);
  for (int k = 0; k < slots; ++k)
    if ((left[k] = (int)at[k].size()) > 0) open.push({left[k], -k});
  while (!open.empty()) {
    const int a = -open.top().second;
    const bool stale = open.top().first != left[a];
    open.pop();
    if (stale) continue;
    Group g{(uint16_t)a, lin[a], {}, 0};
    lin[a] = host::fzero();
    for (int e : at[a]) {
      Edge& E = edges[e];
      if (E.used) continue;
      E.used = true;
      const uint16_t b = E.a == a ? E.b : E.a;
      g.terms.push_back({b, E.v});
      if (b != a && --left[b] > 0) open.push({left[b], -b});
    }
    left[a] = 0;
    weigh(g);
    groups.push_back(std::move(g));
  }
  Group rest{kNoTable, s.c, {}, 0};
  for (int k = 0; k < slots; ++k)
    if (!lin[k].zero()) rest.terms.push_back({(uint16_t)k, lin[k]});
  if (!rest.terms.empty() || !rest.d.zero()) {
    weigh(rest);
    groups.push_back(std::move(rest));
  }
  if (out.cost > most) {
    out = HostForm();
    return false;
  }
  std::stable_sort(groups.begin(), groups.end(), [](const Group& x, const Group& y) { return x.cost > y.cost; });
  for (const Group& g : groups) {
    out.groups.push_back({g.a, (uint16_t)g.terms.size(), (uint32_t)out.terms.size(), kNoConst});
    for (auto& t : g.terms) {
      out.terms.push_back({t.first, (uint16_t)(t.second == one ? TERM_PLUS : t.second == minus_one ? TERM_MINUS : TERM_MUL)});
      out.coeffs.push_back(t.second);
    }
  }
  for (size_t k = 0; k < groups.size(); ++k)
    if (!groups[k].d.zero()) {
      out.groups[k].d = (uint32_t)out.coeffs.size();
      out.coeffs.push_back(groups[k].d);
    }
  return true;
}

PackedProgram pack_program(const HostProgram& hp, Packer& out) {
  std::vector<DevGate> gates = hp.gates;
  const std::vector<F>& coeffs = hp.coeffs;
  std::vector<F> weights = hp.weights;
  // Weights equal to 1 (lambda^0, a zerocheck's gate) skip their product.
  // Folding the other weights into the gates' coefficients was measured and
  // was slower: it turns coefficients of 1 and -1, which cost nothing, into
  // products.
  for (auto& g : gates) g.flags = 0;
  for (size_t j = 0; j < weights.size() && hp.n_cached + j < gates.size(); ++j)
    if (weights[j] == host::fone()) gates[hp.n_cached + j].flags |= kGateUnitWeight;
  // Mark unit coefficients so the device skips their products.
  const host::F one = host::fone(), minus_one = host::fneg(host::fone()), zero = host::fzero();
  for (auto& g : gates) {
    g.ones = g.negs = g.zeros = 0;
    for (uint32_t i = 0; i < 32 && g.cf_off + i < coeffs.size(); ++i) {
      const host::F& v = coeffs[g.cf_off + i];
      if (v == one) g.ones |= 1u << i;
      else if (v == minus_one) g.negs |= 1u << i;
      else if (v == zero) g.zeros |= 1u << i;
    }
  }
  // The weighted sum does not depend on the order of its gates: group gates
  // of one shape together (with their weights), so the lanes of a warp that
  // evaluate consecutive gates take the same code path (measured: the add_sub
  // circuit's proof 17 % faster; sorting on the 0/1/-1 coefficient patterns
  // as well gained nothing more).
  if (hp.summed) {
    const int n0 = hp.n_cached, nw = hp.n_weighted;
    std::vector<int> perm(nw);
    for (int j = 0; j < nw; ++j) perm[j] = j;
    auto key = [&](int j) {
      const DevGate& g = gates[n0 + j];
      return std::make_tuple(g.kind, g.flags, g.p1, g.p2, g.nops);
    };
    std::stable_sort(perm.begin(), perm.end(), [&](int a, int b) { return key(a) < key(b); });
    std::vector<DevGate> wg(nw);
    std::vector<F> ww(nw);
    for (int j = 0; j < nw; ++j) {
      wg[j] = gates[n0 + perm[j]];
      ww[j] = perm[j] < (int)weights.size() ? weights[perm[j]] : host::fone();
    }
    for (int j = 0; j < nw; ++j) gates[n0 + j] = wg[j];
    weights = ww;
  }
  PackedProgram P;
  P.gates = out.put(gates.data(), gates.size() * sizeof(DevGate));
  P.ops = out.put(hp.ops.data(), hp.ops.size() * sizeof(uint16_t));
  P.coeffs = out.put(coeffs.data(), coeffs.size() * 32);
  P.weights = out.put(weights.data(), weights.size() * 32);
  P.n_cached = hp.n_cached;
  P.n_weighted = hp.n_weighted;
  return P;
}

DevProgram PackedProgram::on_device(const uint8_t* base) const {
  DevProgram P;
  P.gates = reinterpret_cast<const DevGate*>(base + gates);
  P.ops = reinterpret_cast<const uint16_t*>(base + ops);
  P.coeffs = reinterpret_cast<const Fr*>(base + coeffs);
  P.weights = reinterpret_cast<const Fr*>(base + weights);
  P.n_cached = n_cached;
  P.n_weighted = n_weighted;
  P.cached_slot0 = 0;
  return P;
}

}  // namespace apg
