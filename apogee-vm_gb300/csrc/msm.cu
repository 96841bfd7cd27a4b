// Pippenger MSM on sm_103a (replaces crates/curve/src/msm.rs:48-311).
//
// Pipeline for a group of columns over the same bases, all on the context's
// stream (msm_group):
//  0. k_split       without an SRS table: scalars as two halves over P and phi(P).
//  1. k_digits      Montgomery -> canonical, signed c-bit digits in
//                   [-2^(c-1), 2^(c-1)] (the reference's recoding rule,
//                   msm.rs:180-198), counted by bucket: up to 8192 buckets a
//                   column in shared memory (k_digits_few), else by atomics on
//                   the buckets' counters.
//  2. scan          exclusive scan of the counts (bucket starts).
//  3. k_digits      the same digits again, each placed as a 4-byte reference
//                   at its bucket's cursor: a counting sort without an
//                   intermediate entry list.
//  4. k_bucket_acc  persistent, load-balanced bucket accumulation: one wave of
//                   threads, each folding an equal slice of the sorted list
//                   run by run into XYZZ accumulators with mixed adds; runs cut
//                   by a slice edge are stitched by k_fold_edges.
//  5. k_reduce      bucket reduction sum_k k*B_k, every column's bucket range
//                   at once, four lanes a point.
//  6. k_finish      per column, combine windows (Horner) or, with a
//                   precomputed SRS window table, nothing: there every window
//                   shares one bucket set because the table already holds
//                   2^(c*w) * P_i; then the canonical affine encoding.
// The allocation-free variant at the end of this file keeps the first
// single-MSM form of the sort and the accumulation (k_recode, k_scatter,
// k_accumulate).
#include "common.cuh"
#include "curve_quad.cuh"

namespace apg {

namespace {

__device__ __forceinline__ void raise_flag(uint32_t* flags, uint32_t f) { atomicOr(flags, f); }

__device__ __forceinline__ Fq fq_const_u32(uint32_t v) {
  Fq a = fe_zero<FqConsts>();
  a.v[0] = v;
  return fe_to_mont(a);
}

__device__ __forceinline__ Affine generator_affine() {
  Affine g;
  g.x = fe_one<FqConsts>();
  g.y = fq_const_u32(2);
  return g;
}

__device__ __forceinline__ bool on_curve(const Affine& p) {
  Fq rhs = fe_add(fe_mul(fe_sqr(p.x), p.x), fq_const_u32(3));
  return fe_eq(fe_sqr(p.y), rhs);
}

// ---- point conversion -------------------------------------------------------

__global__ void k_points_in(const uint4* raw, size_t n, Affine* dst, uint32_t* flags) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint4 q0 = raw[4 * i], q1 = raw[4 * i + 1], q2 = raw[4 * i + 2], q3 = raw[4 * i + 3];
  uint32_t w[16] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w,
                    q2.x, q2.y, q2.z, q2.w, q3.x, q3.y, q3.z, q3.w};
  uint32_t any = 0;
#pragma unroll
  for (int k = 0; k < 16; ++k) any |= w[k];
  Affine a;
  if (any == 0) {
    a.x = fe_zero<FqConsts>();
    a.y = fe_zero<FqConsts>();
  } else {
    if (!fe_lt_mod<FqConsts>(w) || !fe_lt_mod<FqConsts>(w + 8)) raise_flag(flags, DEV_NONCANONICAL);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      a.x.v[k] = w[k];
      a.y.v[k] = w[8 + k];
    }
    a.x = fe_to_mont(a.x);
    a.y = fe_to_mont(a.y);
    if (!on_curve(a)) raise_flag(flags, DEV_OFF_CURVE);
  }
  st_fe(&dst[i].x, a.x);
  st_fe(&dst[i].y, a.y);
}

__global__ void k_points_out(const Affine* src, size_t n, uint4* raw) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  Affine a = ld_affine(&src[i]);
  Fq x = fe_from_mont(a.x), y = fe_from_mont(a.y);
  raw[4 * i] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
  raw[4 * i + 1] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
  raw[4 * i + 2] = make_uint4(y.v[0], y.v[1], y.v[2], y.v[3]);
  raw[4 * i + 3] = make_uint4(y.v[4], y.v[5], y.v[6], y.v[7]);
}

// A result (16-byte pieces) and the error flags into pinned host memory, then the
// flag the host waits for.
__global__ void __launch_bounds__(512) k_publish(const uint4* src, uint32_t n, const uint32_t* err, uint4* dst,
                                                 uint32_t* head, uint32_t seq) {
  chain_begin();
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
  if (threadIdx.x == 0) head[1] = *err;
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) *reinterpret_cast<volatile uint32_t*>(head) = seq;
}

}  // namespace

// Canonical Fr -> Montgomery in place, flagging values >= p.
__global__ void k_fr_to_mont(Fr* v, size_t n, uint32_t* flags) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  Fr a = ld_fe(&v[i]);
  if (!fe_lt_mod<FrConsts>(a.v)) atomicOr(flags, (uint32_t)DEV_NONCANONICAL);
  st_fe(&v[i], fe_to_mont(a));
}

namespace {

// [tau^i] G by double-and-add over the canonical bits of tau^i.
__global__ void k_srs_powers(Fr tau, size_t n, Affine* dst, uint32_t* flags) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  Fr s = fe_one<FrConsts>(), base = tau;
  for (size_t e = i; e; e >>= 1) {
    if (e & 1) s = fe_mul(s, base);
    base = fe_sqr(base);
  }
  Fr sc = fe_from_mont(s);
  const Affine g = generator_affine();
  Xyzz acc = xyzz_inf();
  for (int bit = 253; bit >= 0; --bit) {
    acc = xyzz_dbl(acc);
    if ((sc.v[bit >> 5] >> (bit & 31)) & 1) acc = xyzz_add_affine(acc, g);
  }
  Affine a = xyzz_to_affine(acc, flags);
  st_fe(&dst[i].x, a.x);
  st_fe(&dst[i].y, a.y);
}

// tab[w*n + i] = 2^(c*w) * base[i].
__global__ void k_window_table(const Affine* base, size_t n, int c, int windows, Affine* tab, uint32_t* flags) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  Affine cur = ld_affine(&base[i]);
  st_fe(&tab[i].x, cur.x);
  st_fe(&tab[i].y, cur.y);
  for (int w = 1; w < windows; ++w) {
    if (!aff_is_inf(cur)) {
      Xyzz acc = xyzz_from_affine(cur);
      for (int j = 0; j < c; ++j) acc = xyzz_dbl(acc);
      cur = xyzz_to_affine(acc, flags);
    }
    st_fe(&tab[(size_t)w * n + i].x, cur.x);
    st_fe(&tab[(size_t)w * n + i].y, cur.y);
  }
}

// ---- recode + histogram -------------------------------------------------------

// Entry layout: bits 63..32 bucket (space*K + |d|-1), bit 31 negate, bits 30..0
// base index. A zero digit writes kSkip and is not counted.
constexpr uint64_t kSkip = ~0ull;

template <bool SMALL>
__global__ void k_recode(const void* scalars, size_t n, int c, int windows, int precomp, size_t tab_n,
                         int canonical_in, uint64_t* entries, uint32_t* counts, uint32_t* flags) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t limbs[8];
  if (SMALL) {
    limbs[0] = reinterpret_cast<const uint32_t*>(scalars)[i];
#pragma unroll
    for (int k = 1; k < 8; ++k) limbs[k] = 0;
  } else {
    Fr s = ld_fe(reinterpret_cast<const Fr*>(scalars) + i);
    if (!fe_lt_mod<FrConsts>(s.v)) raise_flag(flags, DEV_NONCANONICAL);
    if (!canonical_in) s = fe_from_mont(s);
#pragma unroll
    for (int k = 0; k < 8; ++k) limbs[k] = s.v[k];
  }
  const uint32_t K = 1u << (c - 1);
  const uint32_t mask = (1u << c) - 1;
  uint32_t carry = 0;
  for (int w = 0; w < windows; ++w) {
    int off = w * c;
    uint32_t raw = 0;
    if (off < 256) {
      int limb = off >> 5, sh = off & 31;
      uint64_t v = limbs[limb] >> sh;
      if (limb + 1 < 8) v |= (uint64_t)limbs[limb + 1] << (32 - sh);
      raw = (uint32_t)v & mask;
    }
    uint32_t coef = raw + carry;
    uint32_t mag;
    uint32_t neg = 0;
    if (w == windows - 1 || coef < K) {
      mag = coef;
      carry = 0;
    } else {
      mag = (1u << c) - coef;  // digit coef - 2^c < 0
      neg = 1;
      carry = 1;
    }
    uint64_t e = kSkip;
    if (mag) {
      uint32_t space = precomp ? 0u : (uint32_t)w;
      uint32_t bucket = space * K + (mag - 1);
      uint64_t pidx = precomp ? (uint64_t)w * tab_n + i : i;
      e = ((uint64_t)bucket << 32) | ((uint64_t)neg << 31) | pidx;
      atomicAdd(&counts[bucket], 1u);
    }
    entries[(size_t)w * n + i] = e;
  }
}

// ---- exclusive scan (u32), two passes ------------------------------------

constexpr int kScanBlock = 1024;
constexpr int kScanItems = 4;  // per thread

__global__ void k_scan_local(uint32_t* data, size_t n, uint32_t* block_sums) {
  chain_begin();
  __shared__ uint32_t sh[kScanBlock];
  size_t base = (size_t)blockIdx.x * kScanBlock * kScanItems + (size_t)threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t sum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = (base + k < n) ? data[base + k] : 0;
    sum += v[k];
  }
  sh[threadIdx.x] = sum;
  __syncthreads();
  for (int off = 1; off < kScanBlock; off <<= 1) {
    uint32_t t = threadIdx.x >= (unsigned)off ? sh[threadIdx.x - off] : 0;
    __syncthreads();
    sh[threadIdx.x] += t;
    __syncthreads();
  }
  uint32_t run = sh[threadIdx.x] - sum;  // exclusive prefix of this thread
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) data[base + k] = run;
    run += v[k];
  }
  if (threadIdx.x == kScanBlock - 1) block_sums[blockIdx.x] = sh[threadIdx.x];
}

// Adds to each k_scan_local block's entries the sums of the blocks before it,
// which every block adds up for itself (kScanBlock of them at most); the total
// goes to *total_out. One block's scan (its total already in block_sums[0])
// needs no such launch.
__global__ void __launch_bounds__(256) k_scan_add(uint32_t* data, size_t n, const uint32_t* block_sums,
                                                  uint32_t* total_out) {
  chain_begin();
  __shared__ uint32_t part[8];
  uint32_t before = 0;
  for (unsigned b = threadIdx.x; b < blockIdx.x; b += 256) before += block_sums[b];
  for (int off = 16; off > 0; off >>= 1) before += __shfl_xor_sync(0xffffffffu, before, off);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = before;
  __syncthreads();
  before = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) before += part[w];
  const size_t base = (size_t)blockIdx.x * kScanBlock * kScanItems;
#pragma unroll
  for (int k = 0; k < kScanBlock * kScanItems / 256; ++k) {
    const size_t i = base + k * 256 + threadIdx.x;
    if (i < n) data[i] += before;
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total_out = before + block_sums[blockIdx.x];
}

__global__ void k_scatter(const uint64_t* entries, size_t e_count, uint32_t* cursor, uint64_t* sorted) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= e_count) return;
  uint64_t e = entries[i];
  if (e == kSkip) return;
  uint32_t pos = atomicAdd(&cursor[e >> 32], 1u);
  sorted[pos] = e;
}

// ---- accumulation -----------------------------------------------------------

__device__ __forceinline__ Affine load_base(const Affine* bases, uint64_t e) {
  Affine a = ld_affine(&bases[e & 0x7fffffffu]);
  if ((e >> 31) & 1) a.y = fe_neg(a.y);
  return a;
}

// Runs of equal buckets are folded by fixed-length segments; a run that
// touches a segment edge is only partial and leaves the segment as an item
// (key, point, present) in slot 2s (the run the segment started inside) or
// 2s+1 (the run it ends inside). Absent slots carry the neighbouring key and
// the identity, so the item list stays sorted and gap-free; the next level
// folds it the same way until one segment holds everything. A run that
// starts and ends inside a segment is a whole bucket and is written directly,
// so every bucket is written exactly once however skewed the digits are.
constexpr uint32_t kNoKey = 0xffffffffu;

__device__ __forceinline__ void put_item(uint32_t* keys, Xyzz* pts, uint8_t* present, size_t slot, uint32_t key,
                                         const Xyzz* p) {
  keys[slot] = key;
  present[slot] = p ? 1 : 0;
  if (p) st_xyzz(&pts[slot], *p);
}

__global__ void __launch_bounds__(128) k_accumulate(const uint64_t* sorted, const uint32_t* total, int seg_len,
                                                    size_t nseg, const Affine* bases, Xyzz* buckets,
                                                    uint32_t* okeys, Xyzz* opts, uint8_t* opres) {
  size_t s = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  const size_t E = *total;
  const size_t lo = s * (size_t)seg_len;
  if (lo >= E) {
    put_item(okeys, opts, opres, 2 * s, kNoKey, nullptr);
    put_item(okeys, opts, opres, 2 * s + 1, kNoKey, nullptr);
    return;
  }
  const size_t hi = min(lo + (size_t)seg_len, E);
  const uint32_t first = (uint32_t)(sorted[lo] >> 32);
  uint32_t cur = first;
  const bool starts_before = lo > 0 && (uint32_t)(sorted[lo - 1] >> 32) == cur;
  const bool continues = hi < E && (uint32_t)(sorted[hi] >> 32) == (uint32_t)(sorted[hi - 1] >> 32);
  bool first_run = true, head_written = false;
  Xyzz acc = xyzz_inf();
  for (size_t i = lo; i < hi; ++i) {
    uint64_t e = sorted[i];
    uint32_t b = (uint32_t)(e >> 32);
    if (b != cur) {
      if (first_run && starts_before) {
        put_item(okeys, opts, opres, 2 * s, cur, &acc);
        head_written = true;
      } else {
        st_xyzz(&buckets[cur], acc);
      }
      first_run = false;
      cur = b;
      acc = xyzz_inf();
    }
    Affine p = load_base(bases, e);
    if (!aff_is_inf(p)) acc = xyzz_add_affine(acc, p);
  }
  if (first_run && starts_before) {
    put_item(okeys, opts, opres, 2 * s, cur, &acc);
    head_written = true;
    put_item(okeys, opts, opres, 2 * s + 1, cur, nullptr);
  } else {
    if (continues) put_item(okeys, opts, opres, 2 * s + 1, cur, &acc);
    else {
      st_xyzz(&buckets[cur], acc);
      put_item(okeys, opts, opres, 2 * s + 1, cur, nullptr);
    }
  }
  if (!head_written) put_item(okeys, opts, opres, 2 * s, first, nullptr);
}

// One level of the edge-run folding over items (see k_accumulate), a quad of
// lanes a point (curve_quad.cuh). A block takes 63 quads' worth of
// consecutive items: each quad folds `per` of them in turn, then quad i holds
// what crosses its left edge (the tail of quad i - 1 plus its own head; quad
// 63 only closes the block's right edge), and a segmented scan by doubling
// distances adds up the runs. So a level's chain is per + log2(run) additions
// and leaves two items a block, where one thread folding eight items in turn
// leaves a quarter of them. 64 quads are two warps a scheduler, as many as a
// scheduler's multiply pipe feeds without slowing a chain (128 quads: 4.0 us an
// addition against 2.3). Measured on a GB300, all levels together: 251 -> 90 us
// for a 2^16-point commit (155,000 items), 153 -> 38 for a 2^8-point one.
constexpr int kFoldQuads = 64;
constexpr int kFoldLastPer = 8;  // items a quad at most in a level of one block

template <int BLOCKS>
__global__ void __launch_bounds__(4 * kFoldQuads, BLOCKS) k_fold_edges(const uint32_t* keys, const Xyzz* pts,
                                                               const uint8_t* pres, size_t len, int per,
                                                               Xyzz* buckets, uint32_t* okeys, Xyzz* opts,
                                                               uint8_t* opres) {
  chain_begin();
  __shared__ __align__(16) Fq sv[4 * kFoldQuads];  // (read and written 16 bytes at a time)
  __shared__ uint32_t skey[kFoldQuads];
  __shared__ uint8_t slive[kFoldQuads], spres[kFoldQuads];
  const int l = threadIdx.x & 3, i = threadIdx.x >> 2;
  const size_t base = blockIdx.x * (size_t)(kFoldQuads - 1) * per;
  const size_t end = min(base + (size_t)(kFoldQuads - 1) * per, len);
  const size_t lo = min(base + (size_t)i * per, end), hi = min(lo + per, end);
  // The boundary at lo: live when the run of item lo - 1 goes on past it. Of
  // the quads that start at the block's end only the first one's counts.
  const bool mine = i == 0 || lo < end || base + (size_t)(i - 1) * per < end;
  const bool live = mine && lo > 0 && lo < len && keys[lo - 1] == keys[lo];
  const bool cont = hi > lo && hi < len && keys[hi - 1] == keys[hi];
  Fq acc = fe_zero<FqConsts>(), head = acc;
  bool any = false, head_any = false, first = true;
  uint32_t cur = lo < hi ? keys[lo] : kNoKey;
  for (int t = 0; t < per; ++t) {
    const size_t at = lo + t;
    const bool in = at < hi;
    const uint32_t k = in ? keys[at] : cur;
    const bool pr = in && pres[at];
    const Fq pt = pr ? quad_ld(&pts[at], l) : fe_zero<FqConsts>();
    if (k != cur) {
      if (first && live) {
        head = acc;
        head_any = any;
      } else if (any && cur != kNoKey) {
        quad_st(&buckets[cur], l, acc);
      }
      first = false;
      cur = k;
      any = false;
    }
    const bool both = pr && any;
    if (__any_sync(0xffffffffu, both)) {
      const Fq sum = quad_add(acc, pt);
      if (both) acc = sum;
    }
    if (pr && !any) acc = pt;
    any |= pr;
  }
  bool tail = false;
  if (lo < hi) {
    if (first && live) {
      head = acc;
      head_any = any;
    } else if (cont) {
      tail = any;
    } else if (any && cur != kNoKey) {
      quad_st(&buckets[cur], l, acc);
    }
  }
  st_fe(&sv[threadIdx.x], acc);
  if (l == 0) {
    spres[i] = tail;
    slive[i] = live;
    skey[i] = live ? keys[lo] : kNoKey;
  }
  __syncthreads();
  // What crosses the boundary at lo: the previous quad's tail, this one's head.
  const bool tp = live && i > 0 && spres[i - 1], hp = live && head_any;
  Fq v = tp ? ld_fe(&sv[threadIdx.x - 4]) : head;
  bool have = tp || hp;
  if (__any_sync(0xffffffffu, tp && hp)) {
    const Fq sum = quad_add(v, head);
    if (tp && hp) v = sum;
  }
  const uint32_t key = skey[i];
  __syncthreads();
  for (int off = 1; off < kFoldQuads; off <<= 1) {
    st_fe(&sv[threadIdx.x], v);
    if (l == 0) spres[i] = have;
    const int j = i + off;
    const bool match = live && j < kFoldQuads && slive[j] && skey[j] == key;
    if (!__syncthreads_or(match)) break;  // no run reaches this far
    const bool take = match && spres[j];
    const Fq o = take ? ld_fe(&sv[threadIdx.x + 4 * off]) : fe_zero<FqConsts>();
    if (__any_sync(0xffffffffu, take && have)) {
      const Fq sum = quad_add(v, o);
      if (take && have) v = sum;
    }
    if (take && !have) v = o;
    have |= take;
    __syncthreads();
  }
  // The runs' first boundaries hold their sums.
  const int ne = (int)((end - base + per - 1) / per);  // the boundary at the block's end
  const bool end_live = slive[ne] != 0, through = end_live && slive[0] && skey[0] == skey[ne];
  const bool lead = live && (i == 0 || !slive[i - 1] || skey[i - 1] != key);
  const size_t out = 2 * (size_t)blockIdx.x;
  if (lead) {
    const bool left = i == 0, right = !left && end_live && skey[ne] == key;
    if (left || right) {
      const size_t slot = out + (left ? 0 : 1);
      if (have) quad_st(&opts[slot], l, v);
      if (l == 0) {
        okeys[slot] = key;
        opres[slot] = have;
      }
    } else if (have && key != kNoKey) {
      quad_st(&buckets[key], l, v);
    }
  }
  if (threadIdx.x == 0) {
    if (!slive[0]) {
      okeys[out] = keys[base];
      opres[out] = 0;
    }
    if (!end_live || through) {
      okeys[out + 1] = keys[end - 1];
      opres[out + 1] = 0;
    }
  }
}

// ---- bucket reduction -------------------------------------------------------
//
// sum_k (k + 1) B_k over a space's K buckets, a quad of lanes a point. A block
// of Q quads takes Q * 2^lf consecutive entries, each (R_k, T_k) with weight
// 2^scale k + 1 within the block: quad q folds its 2^lf entries into their sum
// and their weighted sum W_q = sum_j j R_j, a suffix scan over the quads gives
// S_q = sum_{q' >= q} R_q', and
//   R' = S_0,   T' = sum_q (T_q + 2^scale (W_q + [q > 0] 2^lf S_q))
// is the block's own entry for the next level, whose scale grows by the
// block's length. The first level reads buckets (T_k = 0, scale 0); the last
// (`last`) is one block a space and adds R' in, the + 1 of every weight. A
// block's chain is 2^(lf+1) + 2 log2 Q additions and scale + lf doublings.
// Measured on a GB300 against eight buckets a thread and level with block sums
// of each level: 2^15 buckets 697 -> 135 us, 128 buckets 101 -> 48, four sets
// of 2^19 (bound by the products) 1.9 -> 1.65 ms.
constexpr int kReduceQuads = 64;  // a block at most: two warps a scheduler (see kFoldQuads)

template <int BLOCKS>
__global__ void __launch_bounds__(4 * kReduceQuads, BLOCKS) k_reduce(const Xyzz* R, const Xyzz* T, int M, int lf, int scale,
                                                             int last, Xyzz* outT, Xyzz* outR) {
  chain_begin();
  extern __shared__ uint4 sm_points[];
  Fq* sh = reinterpret_cast<Fq*>(sm_points);
  const int l = threadIdx.x & 3, q = threadIdx.x >> 2, Q = blockDim.x >> 2, sp = blockIdx.y;
  const size_t base = (size_t)sp * M;
  const int f = 1 << lf, k0 = (blockIdx.x * Q + q) << lf;
  Fq run = fe_zero<FqConsts>(), W = run, Ts = run;
  for (int j = f - 1; j >= 0; --j) {
    const int k = k0 + j;
    const Fq r = k < M ? quad_ld(&R[base + k], l) : fe_zero<FqConsts>();
    run = j == f - 1 ? r : quad_add(run, r);
    if (j > 0) W = j == f - 1 ? run : quad_add(W, run);
    if (T) {
      const Fq t = k < M ? quad_ld(&T[base + k], l) : fe_zero<FqConsts>();
      Ts = j == f - 1 ? t : quad_add(Ts, t);
    }
  }
  for (int off = 1; off < Q; off <<= 1) {
    st_fe(&sh[threadIdx.x], run);
    __syncthreads();
    const bool has = q + off < Q;
    const Fq o = has ? ld_fe(&sh[threadIdx.x + 4 * off]) : fe_zero<FqConsts>();
    if (__any_sync(0xffffffffu, has)) run = quad_add(run, o);
    __syncthreads();
  }
  Fq V = q > 0 ? run : fe_zero<FqConsts>();
  for (int d = 0; d < lf; ++d) V = quad_dbl(V);
  if (lf > 0) V = quad_add(V, W);
  for (int d = 0; d < scale; ++d) V = quad_dbl(V);
  if (T) V = quad_add(V, Ts);
  for (int off = Q >> 1; off > 0; off >>= 1) {
    st_fe(&sh[threadIdx.x], V);
    __syncthreads();
    const bool has = q < off;
    const Fq o = has ? ld_fe(&sh[threadIdx.x + 4 * off]) : fe_zero<FqConsts>();
    if (__any_sync(0xffffffffu, has)) V = quad_add(V, o);
    __syncthreads();
  }
  if (threadIdx.x >= 32) return;
  if (last) V = quad_add(V, run);
  if (q != 0) return;
  const size_t o = (size_t)sp * gridDim.x + blockIdx.x;
  quad_st(&outT[o], l, V);
  if (!last) quad_st(&outR[o], l, run);
}

// One warp per result: Horner over the result's spaces (windows, in 2^c),
// then the canonical affine bytes. Every quad runs the same chain. With one
// space a result (an SRS window table) there is no Horner; an MSM over the caller's
// bases has sixteen windows of 8 bits (its scalars in halves), 120 doublings after
// one another, 1.7 us each over a quad (2,484 points: 265 us of the call's 483).
__global__ void __launch_bounds__(32) k_finish(const Xyzz* tsum, int spaces, int c, uint32_t* out64,
                                               uint32_t* flags) {
  chain_begin();
  const int lane = threadIdx.x & 31, l = lane & 3;
  const Xyzz* in = tsum + (size_t)blockIdx.x * spaces;
  Fq total = quad_ld(&in[spaces - 1], l);
  for (int w = spaces - 2; w >= 0; --w) {
    for (int j = 0; j < c; ++j) total = quad_dbl(total);
    total = quad_add(total, quad_ld(&in[w], l));
  }
  // (X / ZZ, Y / ZZZ) with 1 / (ZZ ZZZ) from one inversion, x and y in lanes 0 and 1.
  const Xyzz t = quad_gather(total, lane);
  const Fq inv = fe_inverse(cmul(t.zz, t.zzz), flags);  // (0 at infinity: the result is (0, 0))
  const Fq r = fe_from_mont(cmul(l == 1 ? t.y : t.x, cmul(inv, l == 1 ? t.zz : t.zzz)));
  if (lane >= 2) return;
  uint32_t* o = out64 + 16 * (size_t)blockIdx.x + 8 * lane;
#pragma unroll
  for (int k = 0; k < 8; ++k) o[k] = r.v[k];
}

// ---- the grouped pipeline -----------------------------------------------------
//
// A group is up to kMaxCols scalar columns against one set of bases (an SRS
// window table or generic bases). Bucket keys are (col * spaces + space) * K +
// |d| - 1, with spaces = 1 over a window table and one space per window
// otherwise, so every column owns a key range and one counting sort, one
// accumulation and one bucket reduction serve the whole group: the
// latency-bound reduction is paid once per group instead of once per column.
// The sorted list holds 4-byte references (bit 31 negate, bits 30..0 base
// index); after the scatter the cursor array holds every bucket's end, which
// is all the accumulation needs to find its runs.

constexpr int kMaxCols = 32;

struct MsmCols {
  const void* s[kMaxCols];
  uint32_t len[kMaxCols];
  uint32_t off[kMaxCols];  // first base of the column (a stack's slot j starts at j * 2^n)
  int shared;              // 1: every column feeds one bucket set (one result, the sum)
  int bits;                // small scalars: 32, 16, 8 or 1 (bit-packed in u64 limbs)
};

// Scalar i of a small-scalar column of the given width.
__device__ __forceinline__ uint32_t small_scalar(const void* col, uint32_t i, int bits) {
  switch (bits) {
    case 1:
      return (uint32_t)((reinterpret_cast<const uint64_t*>(col)[i >> 6] >> (i & 63)) & 1u);
    case 8:
      return reinterpret_cast<const uint8_t*>(col)[i];
    case 16:
      return reinterpret_cast<const uint16_t*>(col)[i];
    default:
      return reinterpret_cast<const uint32_t*>(col)[i];
  }
}

// ---- scalars in two halves ----------------------------------------------------
//
// BN254 has the endomorphism phi(x, y) = (beta x, y) = lambda (x, y), with beta and
// lambda cube roots of one in Fq and Fr (Gallant, Lambert and Vanstone, "Faster point
// multiplication on elliptic curves with efficient endomorphisms", 2001): a scalar
// splits as k = k1 + lambda k2 with |k1|, |k2| < 2^127, so n products become 2n of half
// the length and the windows' Horner chain half as deep. (a1, -b1), (a2, b2) is the
// short basis of {(x, y): x + lambda y = 0 mod r} that the extended Euclidean algorithm
// gives, and g1, g2 are round(2^256 b2 / r), round(2^256 b1 / r).
__device__ constexpr uint32_t kSplitA1[2] = {0x94d213e3u, 0x89d32568u};  // (b2 is the same)
__device__ constexpr uint32_t kSplitA2[4] = {0x1221250bu, 0x0be4e154u, 0xeeb859fdu, 0x6f4d8248u};
__device__ constexpr uint32_t kSplitB1[4] = {0x7d4f1128u, 0x8211bbebu, 0xeeb859fcu, 0x6f4d8248u};
__device__ constexpr uint32_t kSplitG1[3] = {0xc7e0b3d7u, 0xd91d232eu, 0x00000002u};
__device__ constexpr uint32_t kSplitG2[5] = {0x391eb18eu, 0x7a7bd9d4u, 0xa773d2cfu, 0x4ccef014u, 0x00000002u};
__device__ constexpr uint32_t kSplitBeta[8] = {0xd782e155u, 0x71930c11u, 0xffbe3323u, 0xa6bb947cu, 0xd4741444u, 0xaa303344u, 0x26594943u, 0x2c3b3f0du};  // Montgomery form

// The NO words of a * b from word LO on.
template <int NA, int NB, int LO, int NO>
__device__ __forceinline__ void product_words(const uint32_t* a, const uint32_t* b, uint32_t* out) {
  uint32_t t[NA + NB];
#pragma unroll
  for (int i = 0; i < NA + NB; ++i) t[i] = 0;
#pragma unroll
  for (int i = 0; i < NA; ++i) {
    uint64_t carry = 0;
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      carry += (uint64_t)a[i] * b[j] + t[i + j];
      t[i + j] = (uint32_t)carry;
      carry >>= 32;
    }
    t[i + NB] = (uint32_t)carry;
  }
#pragma unroll
  for (int i = 0; i < NO; ++i) out[i] = i + LO < NA + NB ? t[i + LO] : 0u;
}

// out = a - b over five words, modulo 2^160.
__device__ __forceinline__ void sub160(const uint32_t* a, const uint32_t* b, uint32_t* out) {
  uint64_t borrow = 0;
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const uint64_t d = (uint64_t)a[i] - b[i] - borrow;
    out[i] = (uint32_t)d;
    borrow = d >> 63;
  }
}

// Scalar i of column j leaves |k1| at 2 off + i and |k2| len further on, over P and
// phi(P) with the halves' signs folded into the points: columns of twice the length
// for the ordinary kernels (`at` holds the columns' first places).
struct SplitCols {
  MsmCols in;
  uint32_t at[kMaxCols];
};
__global__ void __launch_bounds__(128) k_split(const __grid_constant__ SplitCols S, const Affine* bases,
                                               int canonical_in, Affine* out_bases, Fr* out_scalars,
                                               uint32_t* flags) {
  const uint32_t col = blockIdx.y, n = S.in.len[col], i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  Fr k = ld_fe(reinterpret_cast<const Fr*>(S.in.s[col]) + i);
  if (!fe_lt_mod<FrConsts>(k.v)) raise_flag(flags, DEV_NONCANONICAL);
  if (!canonical_in) k = fe_from_mont(k);
  uint32_t c1[2], c2[4], x[5], y[5], k1[5], k2[5];
  product_words<8, 3, 8, 2>(k.v, kSplitG1, c1);
  product_words<8, 5, 8, 4>(k.v, kSplitG2, c2);
  product_words<2, 2, 0, 5>(c1, kSplitA1, x);
  sub160(k.v, x, k1);
  product_words<4, 4, 0, 5>(c2, kSplitA2, y);
  sub160(k1, y, k1);
  product_words<2, 4, 0, 5>(c1, kSplitB1, x);
  product_words<4, 2, 0, 5>(c2, kSplitA1, y);
  sub160(x, y, k2);
  const Affine p = ld_affine(&bases[S.in.off[col] + i]);
  Fq beta;
#pragma unroll
  for (int w = 0; w < 8; ++w) beta.v[w] = kSplitBeta[w];
  const uint32_t zero[5] = {0, 0, 0, 0, 0};
  Fr half;
#pragma unroll
  for (int w = 0; w < 8; ++w) half.v[w] = 0;
  const size_t o = (size_t)S.at[col] + i;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t* v = h ? k2 : k1;
    const bool neg = v[4] >> 31;
    if (neg) sub160(zero, v, v);
#pragma unroll
    for (int w = 0; w < 4; ++w) half.v[w] = v[w];
    const size_t to = o + (h ? n : 0);
    st_fe(&out_scalars[to], half);
    st_fe(&out_bases[to].x, h ? fe_mul(p.x, beta) : p.x);
    st_fe(&out_bases[to].y, neg ? fe_neg(p.y) : p.y);
  }
}

// Digits of one scalar, counted (SCATTER = false) or placed (SCATTER = true).
//
// A block takes 256 scalars. Its threads first run the windows of a scalar's low 32
// bits; scalars with anything above those go to shared memory, close together, and
// the block's warps run their other windows, so that a column of mostly narrow values
// doesn't walk whole warps through every window for the few wide ones. Lanes of a warp
// that hit the same bucket share one atomic where that is common: those of digit 1
// ({0,1} columns, carries of 32-bit values) and, when the first other lane's bucket is
// shared, all lanes' (columns of few distinct values). Matching every lane with every
// other one at every window takes longer than the atomics it saves and kept both
// passes at it (the shuffle queue full nine cycles in ten); now a uniform column is
// bound by its scattered accesses in L2, about 170 G a second. A placed digit is
// stored one window later, when its cursor's atomic has come back. Measured on a
// GB300, counted and placed: four mixed columns of 2^20 196 + 297 -> 134 + 212 us, four
// uniform ones 461 + 929 -> 383 + 776.
constexpr int kDigitThreads = 256;

struct DigitOut {
  uint32_t* cursor;
  uint32_t* sorted;
  uint32_t* flags;
  uint32_t stride;
};

template <bool SCATTER>
struct DigitStep {
  uint32_t base = 0, ref = 0;  // the digit placed last: its group's first place (in the leader), its reference
  unsigned peers = 0;          // its group; 0: none

  __device__ __forceinline__ void flush(const DigitOut& o, unsigned lane) {
    if (!SCATTER) return;
    const uint32_t b = __shfl_sync(0xffffffffu, base, peers ? __ffs(peers) - 1 : 0);
    if (peers) o.sorted[b + (uint32_t)__popc(peers & ((1u << lane) - 1u))] = ref;
    peers = 0;
  }

  // One window of the warp's scalars: digit mag (0: none) of bucket range key0.
  __device__ __forceinline__ void put(const DigitOut& o, unsigned lane, uint32_t mag, uint32_t key0, uint32_t r) {
    if (mag > o.stride) {  // unreachable for values below r; never index past the bucket range
      if (!SCATTER) raise_flag(o.flags, DEV_NONCANONICAL);
      mag = 0;
    }
    const unsigned some = __ballot_sync(0xffffffffu, mag != 0);
    if (!some) return;
    const uint32_t key = key0 + mag - 1;
    const unsigned ones = __ballot_sync(0xffffffffu, mag == 1), left = some & ~ones;
    unsigned group = mag == 1 ? ones : mag ? 1u << lane : 0u;
    if (left) {
      const uint32_t k = __shfl_sync(0xffffffffu, mag, __ffs(left) - 1);
      const unsigned same = __ballot_sync(0xffffffffu, mag == k);
      if (mag == k) group = same;
      if ((same & (same - 1)) && left != same) {
        const unsigned peers = __match_any_sync(0xffffffffu, mag);
        if (mag) group = peers;
      }
    }
    const bool lead = group && (int)lane == __ffs(group) - 1;
    uint32_t b = 0;
    if (lead) {
      if (SCATTER) b = atomicAdd(&o.cursor[key], (uint32_t)__popc(group));
      else atomicAdd(&o.cursor[key], (uint32_t)__popc(group));
    }
    if (SCATTER) {
      flush(o, lane);
      base = b;
      peers = group;
      ref = r;
    }
  }
};

// The signed digit of a window's c bits and the carry into it: its size, the sign and
// the next carry in neg.
__device__ __forceinline__ uint32_t signed_digit(uint32_t coef, uint32_t K, bool top, uint32_t& neg) {
  neg = !top && coef >= K;
  return neg ? 2 * K - coef : coef;  // coef - 2^c < 0
}

template <bool SMALL, bool SCATTER>
__global__ void __launch_bounds__(kDigitThreads) k_digits(MsmCols cols, int c, int windows, int precomp,
                                                          uint32_t stride, uint32_t tab_n, int canonical_in,
                                                          uint32_t* cursor, uint32_t* sorted, uint32_t* flags) {
  chain_begin();
  __shared__ uint32_t wide[SMALL ? 1 : 9][kDigitThreads];  // limbs, then the place in the block and the carry
  __shared__ uint32_t nwide;
  const uint32_t col = blockIdx.y;
  const uint32_t n = cols.len[col];
  const uint32_t i0 = blockIdx.x * kDigitThreads, i = i0 + threadIdx.x;
  const uint32_t lane = threadIdx.x & 31u;
  if (i0 >= n) return;  // the whole block lies past the column's end
  const bool live = i < n;
  uint32_t limbs[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) limbs[k] = 0;
  if (live) {
    if (SMALL) {
      limbs[0] = small_scalar(cols.s[col], i, cols.bits);
    } else {
      Fr s = ld_fe(reinterpret_cast<const Fr*>(cols.s[col]) + i);
      if (!SCATTER && !fe_lt_mod<FrConsts>(s.v)) raise_flag(flags, DEV_NONCANONICAL);
      if (!canonical_in) s = fe_from_mont(s);
#pragma unroll
      for (int k = 0; k < 8; ++k) limbs[k] = s.v[k];
    }
  }
  const uint32_t K = 1u << (c - 1), mask = (1u << c) - 1;
  const uint32_t spaces = precomp ? 1u : (uint32_t)windows;
  const uint32_t key0 = cols.shared ? 0u : col * spaces * stride;
  const uint32_t key_step = precomp ? 0u : stride, ref_step = precomp ? tab_n : 0u;
  const DigitOut out = {cursor, sorted, flags, stride};
  DigitStep<SCATTER> st;
  const int low = min(windows, (32 + c) / c);  // 33 bits: a 32-bit value and its carry
  uint32_t carry = 0, ref = cols.off[col] + i, key = key0;
  uint64_t v = limbs[0] | (uint64_t)limbs[1] << 32;
  for (int w = 0; w < low; ++w) {
    uint32_t neg;
    const uint32_t mag = signed_digit(((uint32_t)v & mask) + carry, K, w == windows - 1, neg);
    st.put(out, lane, live ? mag : 0u, key, (neg << 31) | ref);
    v >>= c;
    carry = neg;
    key += key_step;
    ref += ref_step;
  }
  if (!SMALL && low < windows) {
    if (threadIdx.x == 0) nwide = 0;
    __syncthreads();
    uint32_t above = carry | (uint32_t)v | (uint32_t)(v >> 32);
#pragma unroll
    for (int k = 2; k < 8; ++k) above |= limbs[k];
    const unsigned some = __ballot_sync(0xffffffffu, above != 0);
    uint32_t at = 0;
    if (lane == 0 && some) at = atomicAdd(&nwide, (uint32_t)__popc(some));
    at = __shfl_sync(0xffffffffu, at, 0) + (uint32_t)__popc(some & ((1u << lane) - 1u));
    if (above) {
#pragma unroll
      for (int k = 0; k < 8; ++k) wide[k][at] = limbs[k];
      wide[8][at] = threadIdx.x | carry << 31;
    }
    __syncthreads();
    if (threadIdx.x - lane < nwide) {
      const bool on = threadIdx.x < nwide;
      const uint32_t who = on ? wide[8][threadIdx.x] : 0u;
      carry = who >> 31;
      ref = cols.off[col] + i0 + (who & 0x7fffffffu) + (uint32_t)low * ref_step;
      for (int w = low; w < windows; ++w) {
        const int off = w * c, limb = off >> 5;
        uint32_t raw = 0;
        if (on && limb < 8) {
          const uint32_t a = wide[limb][threadIdx.x], b = limb < 7 ? wide[limb + 1][threadIdx.x] : 0u;
          raw = __funnelshift_r(a, b, off & 31) & mask;
        }
        uint32_t neg;
        const uint32_t mag = signed_digit(raw + carry, K, w == windows - 1, neg);
        st.put(out, lane, mag, key, (neg << 31) | ref);
        carry = neg;
        key += key_step;
        ref += ref_step;
      }
    }
  }
  st.flush(out, lane);
}

// The same digits when a column has few buckets (kFewBins at most: 8-bit
// windows, a generic-base MSM, a narrow column): a block counts its tile of
// scalars into a histogram in shared memory and touches each bucket's global
// counter once, to add its count or, when it places, to reserve that many
// slots and hand them out from shared memory. The warp-wide form above matches
// lanes and waits for a global atomic at every window, and with few buckets all
// warps wait for the same counters (2^20 one-byte scalars: 215 -> 12 us a
// pass; 2^8 scalars of 32 windows: 12.7 and 18.5 -> 6.5 and 8 us).
constexpr uint32_t kFewBins = 8192;  // 32 KB of counters

//
// Here the digits are independent of one another: with K = 2^(c-1) added at every
// window but the top one (DigitBias), window w of the sum is digit w plus K. A thread
// walks a scalar's windows, or, in tiles of less than 256 scalars, takes (scalar,
// window) pairs of scalars that lie in shared memory, so that small calls spread over
// more blocks and all their threads (a commitment of four 2^8-point columns 144 -> 133
// us, of one 158 -> 149 at 2^12).
struct DigitBias {
  uint32_t w[8];
};
constexpr uint32_t kFewChunk = 256;

template <bool SMALL, bool SCATTER>
__global__ void __launch_bounds__(256) k_digits_few(MsmCols cols, int c, int windows, int precomp, uint32_t stride,
                                                    uint32_t tab_n, int canonical_in, uint32_t tile,
                                                    const __grid_constant__ DigitBias bias, uint32_t* cursor,
                                                    uint32_t* sorted, uint32_t* flags) {
  chain_begin();
  extern __shared__ uint32_t bins[];
  const uint32_t col = blockIdx.y;
  const uint32_t n = cols.len[col];
  const uint32_t lo = blockIdx.x * tile, hi = min(lo + tile, n);
  if (lo >= n) return;
  const uint32_t spaces = precomp ? 1u : (uint32_t)windows;
  const uint32_t nb = spaces * stride, key0 = cols.shared ? 0u : col * nb;
  const uint32_t K = 1u << (c - 1), mask = (1u << c) - 1;
  constexpr int kLimbs = SMALL ? 2 : 8;
  // Scalar i plus the bias.
  auto load = [&](uint32_t i, uint32_t* v) {
#pragma unroll
    for (int k = 0; k < kLimbs; ++k) v[k] = 0;
    if (SMALL) {
      v[0] = small_scalar(cols.s[col], i, cols.bits);
    } else {
      Fr s = ld_fe(reinterpret_cast<const Fr*>(cols.s[col]) + i);
      if (!SCATTER && !fe_lt_mod<FrConsts>(s.v)) raise_flag(flags, DEV_NONCANONICAL);
      if (!canonical_in) s = fe_from_mont(s);
#pragma unroll
      for (int k = 0; k < kLimbs; ++k) v[k] = s.v[k];
    }
    uint64_t carry = 0;
#pragma unroll
    for (int k = 0; k < kLimbs; ++k) {
      carry += (uint64_t)v[k] + bias.w[k];
      v[k] = (uint32_t)carry;
      carry >>= 32;
    }
  };
  // Window w, its bits of the sum and the base it multiplies.
  auto put = [&](int pass, int w, uint32_t raw, uint32_t idx) {
    const bool top = w == windows - 1, neg = !top && raw < K;
    uint32_t mag = top ? raw : neg ? K - raw : raw - K;
    if (mag > stride) {  // unreachable for values below r; never index past the bucket range
      if (!SCATTER) raise_flag(flags, DEV_NONCANONICAL);
      mag = 0;
    }
    if (!mag) return;
    uint32_t* bin = &bins[(precomp ? 0u : (uint32_t)w * stride) + mag - 1];
    if (pass == 0) atomicAdd(bin, 1u);
    else sorted[atomicAdd(bin, 1u)] = ((uint32_t)neg << 31) | idx;
  };
  uint32_t* limbs = bins + nb;  // (tile < 256, a power of two) limb k of the tile's scalar i at k tile + i
  for (uint32_t b = threadIdx.x; b < nb; b += blockDim.x) bins[b] = 0;
  if (tile < kFewChunk && lo + threadIdx.x < hi) {
    uint32_t v[kLimbs];
    load(lo + threadIdx.x, v);
#pragma unroll
    for (int k = 0; k < kLimbs; ++k) limbs[k * tile + threadIdx.x] = v[k];
  }
  __syncthreads();
  for (int pass = 0; pass < (SCATTER ? 2 : 1); ++pass) {
    if (tile < kFewChunk) {
      const uint32_t i = threadIdx.x & (tile - 1);
      for (int w = lo + i < hi ? threadIdx.x / tile : windows; w < windows; w += blockDim.x / tile) {
        const int off = w * c, limb = off >> 5;
        uint32_t raw = 0;
        if (limb < kLimbs) {
          const uint32_t x = limbs[limb * tile + i], y = limb + 1 < kLimbs ? limbs[(limb + 1) * tile + i] : 0u;
          raw = __funnelshift_r(x, y, off & 31) & mask;
        }
        put(pass, w, raw, cols.off[col] + lo + i + (precomp ? (uint32_t)w * tab_n : 0u));
      }
    } else {
      for (uint32_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        uint32_t v[kLimbs], idx = cols.off[col] + i;
        load(i, v);
        for (int w = 0; w < windows; ++w) {
          const uint32_t raw = v[0] & mask;
#pragma unroll
          for (int k = 0; k < kLimbs; ++k) v[k] = __funnelshift_r(v[k], k + 1 < kLimbs ? v[k + 1] : 0u, c);
          put(pass, w, raw, idx);
          if (precomp) idx += tab_n;
        }
      }
    }
    __syncthreads();
    if (pass == 0)
      for (uint32_t b = threadIdx.x; b < nb; b += blockDim.x) {
        const uint32_t m = bins[b];
        if (m) bins[b] = atomicAdd(&cursor[key0 + b], m);
      }
    __syncthreads();
  }
}

// Persistent bucket accumulation: the grid is one wave of resident threads
// and thread s folds the s-th of nseg equal slices of the sorted list, so the
// work is balanced however the digits are distributed. Runs are found from
// the bucket ends; a run cut by a slice edge leaves as an item for
// k_fold_edges exactly as in k_accumulate.
// Four resident blocks per SM (128 registers a thread): measured 2-3 % faster
// than the three that the unconstrained allocation (144) leaves room for.
#ifndef APG_ACC_MIN_BLOCKS
#define APG_ACC_MIN_BLOCKS 4
#endif
// After affine pair rounds (`mode` non-null and *mode == 0) the input is the
// last round's explicit point list, position i holding point i, with its own
// bucket ends and total; otherwise references into `bases`.
__global__ void __launch_bounds__(128, APG_ACC_MIN_BLOCKS) k_bucket_acc(const uint32_t* sorted, const uint32_t* ends, uint32_t nbins,
                                                    const uint32_t* total, size_t nseg, const Affine* bases,
                                                    Xyzz* buckets, uint32_t* okeys, Xyzz* opts, uint8_t* opres,
                                                    const uint32_t* mode, const uint32_t* pair_ends,
                                                    const Affine* pair_pts) {
  chain_begin();
  const size_t s = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  const bool direct = mode && *mode == 0;
  if (direct) {
    ends = pair_ends;
    total = pair_ends + nbins - 1;
    bases = pair_pts;
  }
  const size_t E = *total;
  const size_t seg = (E + nseg - 1) / nseg;
  const size_t lo = s * seg;
  if (lo >= E) {
    put_item(okeys, opts, opres, 2 * s, kNoKey, nullptr);
    put_item(okeys, opts, opres, 2 * s + 1, kNoKey, nullptr);
    return;
  }
  const size_t hi = min(lo + seg, E);
  // The bucket holding position lo: the first key whose end lies past it.
  uint32_t a = 0, b = nbins - 1;
  while (a < b) {
    const uint32_t m = (a + b) >> 1;
    if (ends[m] > lo) b = m;
    else a = m + 1;
  }
  uint32_t cur = a;
  size_t run_end = ends[cur];
  const bool starts_before = lo > (cur ? (size_t)ends[cur - 1] : 0);
  const uint32_t first = cur;
  bool first_run = true, head_written = false;
  Xyzz acc = xyzz_inf();
  for (size_t i = lo; i < hi; ++i) {
    if (i == run_end) {
      if (first_run && starts_before) {
        put_item(okeys, opts, opres, 2 * s, cur, &acc);
        head_written = true;
      } else {
        st_xyzz(&buckets[cur], acc);
      }
      first_run = false;
      do {
        run_end = ends[++cur];
      } while (run_end <= i);
      acc = xyzz_inf();
    }
    const uint32_t e = direct ? (uint32_t)i : sorted[i];
    Affine p = ld_affine(&bases[e & 0x7fffffffu]);
    if (!direct && (e >> 31)) p.y = fe_neg(p.y);
    if (!aff_is_inf(p)) acc = xyzz_add_affine(acc, p);
  }
  const bool continues = hi < run_end;
  if (first_run && starts_before) {
    put_item(okeys, opts, opres, 2 * s, cur, &acc);
    head_written = true;
    put_item(okeys, opts, opres, 2 * s + 1, cur, nullptr);
  } else {
    if (continues) {
      put_item(okeys, opts, opres, 2 * s + 1, cur, &acc);
    } else {
      st_xyzz(&buckets[cur], acc);
      put_item(okeys, opts, opres, 2 * s + 1, cur, nullptr);
    }
  }
  if (!head_written) put_item(okeys, opts, opres, 2 * s, first, nullptr);
}

// ---- affine pair rounds ------------------------------------------------------
//
// Before the XYZZ accumulation, a few rounds halve every bucket's run by adding
// its points in adjacent pairs in affine coordinates. All the pairs one thread
// owns share one field inversion (Montgomery's batch trick: the running product
// of the denominators going forward, one inversion, then each pair's inverse at
// two products going backward), so a pair sum costs 5M + 1S plus a share of one
// inversion, against 8M + 2S for each mixed XYZZ addition it replaces. Equal x
// (a doubling, or P + (-P)) and infinity are classified per pair, so no zero
// ever enters the product.
//
// Round r reads a list with bucket ends `ends_in` and writes the list of
// ceil(len/2) points per bucket at the exclusive-scan offsets `start_out`
// (nbins + 1 entries, the total last). Round 0 reads sorted references into
// the bases; later rounds read the previous round's points. A round 0 whose
// output would not fit the scratch sets *mode = 1 and every later step takes
// the references instead.

// Four rounds (a bucket's run cut to a sixteenth before the XYZZ tail):
// measured 1.2 % faster on the 2^22 commit than three; the fourth round's
// lists are short, but its pair sums still replace XYZZ additions.
#ifndef APG_PAIR_ROUNDS
#define APG_PAIR_ROUNDS 4
#endif
constexpr int kPairRounds = APG_PAIR_ROUNDS;
// Groups of fewer digits are left to the XYZZ kernel alone: the rounds' fixed
// cost (four inversions and 24 launches, about 450 us) exceeds what they save.
// Both sides cost the same at about 2^23 digits that are there; the host knows
// only how many there could be, and a trace column has a quarter of them (bits
// and 32-bit words), so columns of unknown values take the rounds from twice
// that. Measured on a GB300 with and without the rounds: one 2^20-point mixed
// column (16 M possible digits, 4 M real) 1400 and 1160 us, uniform 3133 and
// 3373; four of 2^18 mixed 1617 and 1366, uniform 3284 and 3597.
#ifndef APG_PAIR_MIN_ENTRIES
#define APG_PAIR_MIN_ENTRIES ((size_t)1 << 23)
#endif
constexpr size_t kPairMinEntries = APG_PAIR_MIN_ENTRIES;
// Round 0's output list is held to this many points (64 bytes each).
constexpr size_t kPairMaxPoints = (size_t)48 << 20;

__global__ void k_halve_counts(const uint32_t* ends_in, uint32_t nbins, uint32_t* cnt) {
  const size_t b = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (b > nbins) return;
  if (b == nbins) {
    cnt[b] = 0;
    return;
  }
  const uint32_t len = ends_in[b] - (b ? ends_in[b - 1] : 0u);
  cnt[b] = (len + 1) / 2;
}

template <bool REFS>
__device__ __forceinline__ Affine pair_point(const uint32_t* refs, const Affine* src, uint32_t i) {
  if (REFS) {
    const uint32_t e = refs[i];
    Affine p = ld_affine(&src[e & 0x7fffffffu]);
    if (e >> 31) p.y = fe_neg(p.y);
    return p;
  }
  return ld_affine(&src[i]);
}

enum : int { kPairFirst = 0, kPairSecond = 1, kPairInf = 2, kPairAdd = 3, kPairDbl = 4 };

// The pair rounds' products are inlined (unlike the XYZZ formulas, whose ten
// inlined products a step overflowed the instruction cache): the compiler
// interleaves the independent ones, measured 2 % faster than calls.
// APG_PAIR_CALLS=1 makes them out-of-line calls instead (a build knob for
// measurement).
#ifndef APG_PAIR_CALLS
#define APG_PAIR_CALLS 0
#endif
__device__ __forceinline__ Fq pmul(const Fq& a, const Fq& b) { return APG_PAIR_CALLS ? cmul(a, b) : fe_mul(a, b); }
__device__ __forceinline__ Fq psqr(const Fq& a) { return APG_PAIR_CALLS ? csqr(a) : fe_sqr(a); }
__device__ __forceinline__ Fq2 pmul2(const Fq& a, const Fq& b, const Fq& c, const Fq& d) {
  if (APG_PAIR_CALLS) return cmul2(a, b, c, d);
  Fq2 r;
  r.a = fe_mul(a, b);
  r.b = fe_mul(c, d);
  return r;
}

// What the pair (p0, p1) sums to: p0 or p1 when the other is infinity, the
// point at infinity for P + (-P), else an addition or a doubling.
__device__ __forceinline__ int pair_kind(const Affine& p0, const Affine& p1) {
  if (aff_is_inf(p1)) return kPairFirst;
  if (aff_is_inf(p0)) return kPairSecond;
  if (!fe_eq(p0.x, p1.x)) return kPairAdd;
  return fe_eq(p0.y, p1.y) ? kPairDbl : kPairInf;
}

// The forward pass needs only the x coordinates (and y where x decides nothing).
template <bool REFS>
__device__ __forceinline__ bool pair_denominator(const uint32_t* refs, const Affine* src, uint32_t i0, Fq& d) {
  uint32_t j0 = i0, j1 = i0 + 1;
  bool n0 = false, n1 = false;
  if (REFS) {
    const uint32_t e0 = refs[i0], e1 = refs[i0 + 1];
    j0 = e0 & 0x7fffffffu;
    j1 = e1 & 0x7fffffffu;
    n0 = e0 >> 31;
    n1 = e1 >> 31;
  }
  const Fq x0 = ld_fe(&src[j0].x), x1 = ld_fe(&src[j1].x);
  if (!fe_eq(x0, x1)) {
    if (fe_is_zero(x0) && fe_is_zero(ld_fe(&src[j0].y))) return false;
    if (fe_is_zero(x1) && fe_is_zero(ld_fe(&src[j1].y))) return false;
    d = fe_sub(x1, x0);
    return true;
  }
  Fq y0 = ld_fe(&src[j0].y), y1 = ld_fe(&src[j1].y);
  if (n0) y0 = fe_neg(y0);
  if (n1) y1 = fe_neg(y1);
  if (fe_is_zero(x0) && (fe_is_zero(y0) || fe_is_zero(y1))) return false;  // an infinity
  if (!fe_eq(y0, y1)) return false;                                        // P + (-P)
  d = fe_add(y0, y0);
  return true;
}

// Field element shuffles across a full warp.
__device__ __forceinline__ Fq shfl_up_fq(const Fq& a, int off) {
  Fq r;
#pragma unroll
  for (int w = 0; w < 8; ++w) r.v[w] = __shfl_up_sync(0xffffffffu, a.v[w], off);
  return r;
}
__device__ __forceinline__ Fq shfl_down_fq(const Fq& a, int off) {
  Fq r;
#pragma unroll
  for (int w = 0; w < 8; ++w) r.v[w] = __shfl_down_sync(0xffffffffu, a.v[w], off);
  return r;
}

// Each thread's 1/v (v != 0) from one inversion a block of kPairThreads:
// per warp the inclusive prefix and suffix products across the lanes give
// the warp's total and each lane's product of the others; warp 0 inverts the
// product of the warps' totals (the binary Euclid costs as many instructions
// as a lane's work in a late pair round, so one a block instead of one a warp
// is a quarter of that) and hands each warp the inverse of its total; then
// 1/v_i = (1/total_w) * (lanes before i) * (lanes after i). All threads of the
// block must call it.
constexpr int kPairThreads = 128;
constexpr int kPairWarps = kPairThreads / 32;

__device__ __forceinline__ Fq block_inverse(const Fq& v, uint32_t* flags) {
  __shared__ Fq tot[kPairWarps], tinv[kPairWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  Fq pre = v, suf = v;
#pragma unroll 1
  for (int off = 1; off < 32; off <<= 1) {
    const Fq a = shfl_up_fq(pre, off), b = shfl_down_fq(suf, off);
    const Fq2 q = cmul2(pre, a, suf, b);
    if (lane >= off) pre = q.a;
    if (lane + off < 32) suf = q.b;
  }
  if (lane == 31) tot[w] = pre;
  Fq ex = shfl_up_fq(pre, 1), sx = shfl_down_fq(suf, 1);
  if (lane == 0) ex = fe_one<FqConsts>();
  if (lane == 31) sx = fe_one<FqConsts>();
  const Fq others = cmul(ex, sx);
  __syncthreads();
  if (w == 0) {
    Fq all = tot[0];
#pragma unroll 1
    for (int i = 1; i < kPairWarps; ++i) all = cmul(all, tot[i]);
    Fq o = fe_inverse(all, flags);  // every lane of warp 0 inverts the same value
#pragma unroll 1
    for (int i = 0; i < kPairWarps; ++i)
      if (i != lane) o = cmul(o, tot[i]);
    if (lane < kPairWarps) tinv[lane] = o;
  }
  __syncthreads();
  return cmul(tinv[w], others);
}

// The first bucket whose output reaches past slot o (o below the total).
__device__ __forceinline__ uint32_t pair_bucket(const uint32_t* start_out, uint32_t nbins, size_t o) {
  uint32_t a = 0, b = nbins - 1;
  while (a < b) {
    const uint32_t mid = (a + b) >> 1;
    if (start_out[mid + 1] > o) b = mid;
    else a = mid + 1;
  }
  return a;
}

// The bucket holding output slot o, from the bucket b of an earlier (seek_up)
// or later (seek_down) slot of the same lane. A lane's slots are 32 apart, so
// where most buckets are empty (a short column grouped with a long one) the
// cursor may pass many buckets in one step: it gallops (1, 2, 4, ... buckets)
// and then bisects, one comparison where buckets are dense.
__device__ __forceinline__ uint32_t pair_seek_up(const uint32_t* start_out, uint32_t nbins, uint32_t b, size_t o) {
  if (start_out[b + 1] > o) return b;
  uint32_t lo = b + 1, hi, step = 1;  // start_out[lo] <= o: the bucket is at or past lo
  for (;;) {
    hi = lo + step;
    if (hi >= nbins - 1 || start_out[hi + 1] > o) break;
    lo = hi + 1;
    step <<= 1;
  }
  hi = min(hi, nbins - 1);
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (start_out[mid + 1] > o) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

__device__ __forceinline__ uint32_t pair_seek_down(const uint32_t* start_out, uint32_t b, size_t o) {
  if (start_out[b] <= o) return b;
  uint32_t hi = b - 1, lo, step = 1;  // the bucket is at or before hi
  for (;;) {
    if (hi < step) {
      lo = 0;
      break;
    }
    lo = hi - step;
    if (start_out[lo] <= o) break;
    hi = lo - 1;
    step <<= 1;
  }
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (start_out[mid] <= o) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Slot o of bucket b reads input i0 and, when `two`, i0 + 1.
__device__ __forceinline__ uint32_t pair_input(const uint32_t* ends_in, const uint32_t* start_out, uint32_t b,
                                               size_t o, bool& two) {
  const uint32_t i0 = (b ? ends_in[b - 1] : 0u) + 2u * (uint32_t)(o - start_out[b]);
  two = i0 + 1 < ends_in[b];
  return i0;
}

// One output slot of the backward pass: what it needs of its inputs (x0, y0,
// x1), its kind, and the denominator and numerator of the slope when it has
// one (1 and 0 otherwise, which leave the running inverse unchanged).
struct PairSlot {
  Fq x0, y0, x1, d, num;
  uint32_t i0;
  int kind;
};

template <bool REFS>
__device__ __forceinline__ void pair_load(const uint32_t* refs, const Affine* src, uint32_t i0, bool two,
                                          PairSlot& t) {
  const Affine p0 = pair_point<REFS>(refs, src, i0);
  Affine p1 = p0;
  t.i0 = i0;
  t.kind = kPairFirst;
  if (two) {
    p1 = pair_point<REFS>(refs, src, i0 + 1);
    t.kind = pair_kind(p0, p1);
  }
  t.x0 = p0.x;
  t.y0 = p0.y;
  t.x1 = p1.x;
  t.d = fe_one<FqConsts>();
  t.num = fe_zero<FqConsts>();
  if (t.kind == kPairAdd) {
    t.d = fe_sub(p1.x, p0.x);
    t.num = fe_sub(p1.y, p0.y);
  } else if (t.kind == kPairDbl) {
    t.d = fe_add(p0.y, p0.y);
    const Fq q = psqr(p0.x);
    t.num = fe_add(q, fe_add(q, q));
  }
}

// The slot's sum, given the slope lam when it has one.
template <bool REFS>
__device__ __forceinline__ void pair_store(const uint32_t* refs, const Affine* src, const PairSlot& t,
                                           const Fq& lam, const Fq& l2, Affine* dst) {
  Fq x = t.x0, y = t.y0;
  if (t.kind == kPairSecond) {
    const Affine p1 = pair_point<REFS>(refs, src, t.i0 + 1);
    x = p1.x;
    y = p1.y;
  } else if (t.kind == kPairInf) {
    x = fe_zero<FqConsts>();
    y = fe_zero<FqConsts>();
  } else if (t.kind != kPairFirst) {
    x = fe_sub(fe_sub(l2, t.x0), t.x1);
    y = fe_sub(pmul(lam, fe_sub(t.x0, x)), t.y0);
  }
  st_fe(&dst->x, x);
  st_fe(&dst->y, y);
}

// Resident blocks a SM for the backward half of a round (it holds a slot's two
// points, its running inverse and the slope): six blocks cap it at 80
// registers with a few bytes spilled, measured 1 % faster on the headline
// step than five at 92 registers; seven (72 registers) spilled more and was
// slower.
#ifndef APG_PAIR_MIN_BLOCKS
#define APG_PAIR_MIN_BLOCKS 6
#endif
// The slots of a pair round. A warp owns 32 * m consecutive output slots and
// lane l takes slots base + 32 j + l, so the lanes' references, explicit input
// points, running products and outputs move in coalesced rows. Both halves of
// a round derive the same assignment from (E, T).
struct PairLane {
  size_t o0, steps;
};

__device__ __forceinline__ PairLane pair_lane(size_t s, size_t E, size_t T) {
  PairLane l;
  const size_t m = (E + T - 1) / T;
  l.o0 = (s / 32) * 32 * m + (s & 31);
  l.steps = l.o0 < E ? min(m, (E - l.o0 + 31) / 32) : 0;
  return l;
}

// Forward half: lane s multiplies up the slope denominators of its slots,
// leaving the running product before slot j in pp[j * T + s] and the lane's
// total in tot[s]. No barrier: the lanes of a block finish independently.
// A round 0 whose output would not fit the scratch (E > cap) sets *mode = 1,
// and every later step takes the references instead.
// Slot inputs handed from the forward to the backward half (`idx`, one word a
// slot in the same j * T + s layout as the running products): the first
// input's position, and bit 31 when the slot has a second input. With it the
// backward half neither searches the bucket offsets nor waits on them, and
// issues a slot's reference loads one slot ahead and its word loads two
// ahead (k_pair_bwd_pf). APG_PAIR_PF=0 keeps the searching k_pair_bwd (a
// build knob for measurement). Measured on a GB300 (uniform 2^22
// accumulation / mixed 16 x 2^22 commit): searching 11.86 / 56.6 ms; words
// and references ahead 11.36 / 54.8 ms at five blocks an SM (11.23 / 56.1 at
// four); also the points and running product one slot ahead (128 registers,
// three or four blocks) 11.8-12.0 / 56.7-59.0; the x coordinates one slot
// ahead with the slope's inverse started on x alone 11.35 / 56.0 at four
// blocks, 12.1 / 57.7 at five.
#ifndef APG_PAIR_PF
#define APG_PAIR_PF 1
#endif
constexpr uint32_t kPairTwo = 0x80000000u;
// APG_PAIR_FWD_AHEAD: the forward half also loads the next slot's word and
// references while the current slot's x coordinates are in flight.
#ifndef APG_PAIR_FWD_AHEAD
#define APG_PAIR_FWD_AHEAD 1
#endif

// A slot word's references: table references in round 0, list positions
// after it (a one-input slot repeats its first).
template <bool REFS>
__device__ __forceinline__ void pair_refs(const uint32_t* refs, uint32_t w, uint32_t& e0, uint32_t& e1) {
  const uint32_t i0 = w & ~kPairTwo;
  const bool two = (w & kPairTwo) != 0;
  if (REFS) {
    e0 = refs[i0];
    e1 = two ? refs[i0 + 1] : e0;
  } else {
    e0 = i0;
    e1 = two ? i0 + 1 : i0;
  }
}

// pair_denominator with the two x coordinates already loaded.
template <bool REFS>
__device__ __forceinline__ bool pair_denominator_x(const Affine* src, uint32_t e0, uint32_t e1, const Fq& x0,
                                                   const Fq& x1, Fq& d) {
  const uint32_t j0 = REFS ? (e0 & 0x7fffffffu) : e0, j1 = REFS ? (e1 & 0x7fffffffu) : e1;
  if (!fe_eq(x0, x1)) {
    if (fe_is_zero(x0) && fe_is_zero(ld_fe(&src[j0].y))) return false;
    if (fe_is_zero(x1) && fe_is_zero(ld_fe(&src[j1].y))) return false;
    d = fe_sub(x1, x0);
    return true;
  }
  Fq y0 = ld_fe(&src[j0].y), y1 = ld_fe(&src[j1].y);
  if (REFS && (e0 >> 31)) y0 = fe_neg(y0);
  if (REFS && (e1 >> 31)) y1 = fe_neg(y1);
  if (fe_is_zero(x0) && (fe_is_zero(y0) || fe_is_zero(y1))) return false;  // an infinity
  if (!fe_eq(y0, y1)) return false;                                        // P + (-P)
  d = fe_add(y0, y0);
  return true;
}

template <bool REFS>
__global__ void __launch_bounds__(kPairThreads)
    k_pair_fwd(const uint32_t* refs, const Affine* src, const uint32_t* ends_in, const uint32_t* start_out,
               uint32_t nbins, size_t cap, uint32_t* mode, size_t T, Fq* pp, Fq* tot, uint32_t* idx) {
  const size_t s = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (s >= T || *mode) return;
  const size_t E = start_out[nbins];
  if (E > cap) {
    if (s == 0) *mode = 1;
    return;
  }
  const PairLane L = pair_lane(s, E, T);
  uint32_t b = L.steps ? pair_bucket(start_out, nbins, L.o0) : 0u;
  Fq acc = fe_one<FqConsts>();
  if (APG_PAIR_PF && APG_PAIR_FWD_AHEAD) {
    // The next slot's bucket search, word and references are issued while
    // this slot's x coordinates are in flight.
    uint32_t wa = 0, ea0 = 0, ea1 = 0;
    if (L.steps) {
      bool two;
      wa = pair_input(ends_in, start_out, b, L.o0, two);
      wa |= two ? kPairTwo : 0u;
      pair_refs<REFS>(refs, wa, ea0, ea1);
    }
    for (size_t j = 0; j < L.steps; ++j) {
      const Fq x0 = ld_fe(&src[REFS ? (ea0 & 0x7fffffffu) : ea0].x);
      const Fq x1 = ld_fe(&src[REFS ? (ea1 & 0x7fffffffu) : ea1].x);
      uint32_t wb = 0, eb0 = 0, eb1 = 0;
      if (j + 1 < L.steps) {
        const size_t o = L.o0 + 32 * (j + 1);
        b = pair_seek_up(start_out, nbins, b, o);
        bool two;
        wb = pair_input(ends_in, start_out, b, o, two);
        wb |= two ? kPairTwo : 0u;
        pair_refs<REFS>(refs, wb, eb0, eb1);
      }
      idx[j * T + s] = wa;
      Fq d;
      if ((wa & kPairTwo) && pair_denominator_x<REFS>(src, ea0, ea1, x0, x1, d)) {
        st_fe(&pp[j * T + s], acc);
        acc = fe_mul(acc, d);
      }
      wa = wb;
      ea0 = eb0;
      ea1 = eb1;
    }
    st_fe(&tot[s], acc);
    return;
  }
  for (size_t j = 0; j < L.steps; ++j) {
    const size_t o = L.o0 + 32 * j;
    b = pair_seek_up(start_out, nbins, b, o);
    bool two;
    const uint32_t i0 = pair_input(ends_in, start_out, b, o, two);
    if (APG_PAIR_PF) idx[j * T + s] = i0 | (two ? kPairTwo : 0u);
    Fq d;
    if (!two || !pair_denominator<REFS>(refs, src, i0, d)) continue;
    st_fe(&pp[j * T + s], acc);
    acc = fe_mul(acc, d);
  }
  st_fe(&tot[s], acc);
}

// Backward half: the block shares one inversion of its lanes' totals (every
// lane reaches it first, before any slot), then each slot takes its inverse
// at two products from the running inverse and writes its sum.
template <bool REFS>
__global__ void __launch_bounds__(kPairThreads, APG_PAIR_MIN_BLOCKS)
    k_pair_bwd(const uint32_t* refs, const Affine* src, const uint32_t* ends_in, const uint32_t* start_out,
               uint32_t nbins, const uint32_t* mode, size_t T, const Fq* pp, const Fq* tot, Affine* out,
               uint32_t* flags) {
  const size_t s = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (*mode) return;  // uniform across the grid: set before this launch
  const size_t E = start_out[nbins];
  const PairLane L = pair_lane(s, E, T);
  Fq inv = block_inverse(s < T ? ld_fe(&tot[s]) : fe_one<FqConsts>(), flags);  // every thread of the block
  if (s >= T || !L.steps) return;
  uint32_t b = pair_bucket(start_out, nbins, L.o0 + 32 * (L.steps - 1));
  for (size_t j = L.steps; j-- > 0;) {
    const size_t o = L.o0 + 32 * j;
    b = pair_seek_down(start_out, b, o);
    bool two;
    PairSlot t;
    pair_load<REFS>(refs, src, pair_input(ends_in, start_out, b, o, two), two, t);
    if (t.kind < kPairAdd) {
      pair_store<REFS>(refs, src, t, t.num, t.num, &out[o]);
      continue;
    }
    const Fq2 di = pmul2(inv, ld_fe(&pp[j * T + s]), inv, t.d);  // 1/d, and the running inverse one back
    inv = di.b;
    const Fq lam = pmul(t.num, di.a);
    pair_store<REFS>(refs, src, t, lam, psqr(lam), &out[o]);
  }
}

// The backward half over the forward half's slot words (see `idx` above). A
// slot's chain of dependent loads (its word, then its references, then its
// points) is spread over consecutive iterations: the word and the
// references are loaded while the two slots before it are summed, so only
// the point gather itself waits at the slot's start.
template <bool REFS>
__device__ __forceinline__ Affine pair_fetch(const Affine* src, uint32_t e) {
  return ld_affine(&src[REFS ? (e & 0x7fffffffu) : e]);
}

template <bool REFS>
__device__ __forceinline__ void pair_sign(Affine& p, uint32_t e) {
  if (REFS && (e >> 31)) p.y = fe_neg(p.y);
}

// One slot from its loaded inputs: the same kinds, running inverse and sum
// as pair_load/pair_store.
__device__ __forceinline__ void pair_finish(const Affine& p0, const Affine& p1, bool two, const Fq& ppj, Fq& inv,
                                            Affine* dst) {
  const int kind = two ? pair_kind(p0, p1) : (int)kPairFirst;
  if (kind < kPairAdd) {
    Fq x = p0.x, y = p0.y;
    if (kind == kPairSecond) {
      x = p1.x;
      y = p1.y;
    } else if (kind == kPairInf) {
      x = fe_zero<FqConsts>();
      y = fe_zero<FqConsts>();
    }
    st_fe(&dst->x, x);
    st_fe(&dst->y, y);
    return;
  }
  Fq d, num;
  if (kind == kPairAdd) {
    d = fe_sub(p1.x, p0.x);
    num = fe_sub(p1.y, p0.y);
  } else {
    d = fe_add(p0.y, p0.y);
    const Fq q = psqr(p0.x);
    num = fe_add(q, fe_add(q, q));
  }
  const Fq2 di = pmul2(inv, ppj, inv, d);  // 1/d, and the running inverse one back
  inv = di.b;
  const Fq lam = pmul(num, di.a);
  const Fq x = fe_sub(fe_sub(psqr(lam), p0.x), p1.x);
  st_fe(&dst->x, x);
  st_fe(&dst->y, fe_sub(pmul(lam, fe_sub(p0.x, x)), p0.y));
}

#ifndef APG_PAIR_PF_MIN_BLOCKS
#define APG_PAIR_PF_MIN_BLOCKS 5
#endif

template <bool REFS>
__global__ void __launch_bounds__(kPairThreads, APG_PAIR_PF_MIN_BLOCKS)
    k_pair_bwd_pf(const uint32_t* refs, const Affine* src, const uint32_t* idx, const uint32_t* start_out,
                  uint32_t nbins, const uint32_t* mode, size_t T, const Fq* pp, const Fq* tot, Affine* out,
                  uint32_t* flags) {
  const size_t s = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (*mode) return;  // uniform across the grid: set before this launch
  const size_t E = start_out[nbins];
  const PairLane L = pair_lane(s, E, T);
  Fq inv = block_inverse(s < T ? ld_fe(&tot[s]) : fe_one<FqConsts>(), flags);  // every thread of the block
  if (s >= T || !L.steps) return;
  // Entering the loop for slot j: slot j's word and references, slot j - 1's
  // word. Each pass issues slot j's point and running-product loads, slot
  // j - 1's reference loads and slot j - 2's word load together, then sums
  // slot j.
  size_t j = L.steps - 1;
  uint32_t wa = idx[j * T + s], ea0, ea1;
  pair_refs<REFS>(refs, wa, ea0, ea1);
  uint32_t wb = j >= 1 ? idx[(j - 1) * T + s] : 0u;
  for (;;) {
    Affine p0 = pair_fetch<REFS>(src, ea0), p1 = pair_fetch<REFS>(src, ea1);
    const Fq ppj = ld_fe(&pp[j * T + s]);
    uint32_t nb0 = 0, nb1 = 0, nw = 0;
    if (j >= 1) pair_refs<REFS>(refs, wb, nb0, nb1);
    if (j >= 2) nw = idx[(j - 2) * T + s];
    pair_sign<REFS>(p0, ea0);
    pair_sign<REFS>(p1, ea1);
    pair_finish(p0, p1, (wa & kPairTwo) != 0, ppj, inv, &out[L.o0 + 32 * j]);
    if (j == 0) break;
    --j;
    wa = wb;
    ea0 = nb0;
    ea1 = nb1;
    wb = nw;
  }
}

// out64 = the sum of m canonical affine points in64[0..m) (a stack whose
// columns took more than one group).
__global__ void k_add_points(const uint32_t* in64, int m, uint32_t* out64, uint32_t* flags) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  Xyzz acc = xyzz_inf();
  for (int j = 0; j < m; ++j) {
    Affine a;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      a.x.v[k] = in64[16 * j + k];
      a.y.v[k] = in64[16 * j + 8 + k];
    }
    if (aff_is_inf(a)) continue;
    a.x = fe_to_mont(a.x);
    a.y = fe_to_mont(a.y);
    acc = xyzz_add(acc, xyzz_from_affine(a));
  }
  const Affine r = xyzz_to_affine(acc, flags);
  const Fq x = fe_from_mont(r.x), y = fe_from_mont(r.y);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    out64[k] = x.v[k];
    out64[8 + k] = y.v[k];
  }
}

struct FoldLevel {
  unsigned blocks;
  int per;
};
// A level of k_fold_edges over len items: one block while its quads take at
// most kFoldLastPer each, else two items a quad, or four where that saves a
// level.
inline FoldLevel fold_level(size_t len) {
  const size_t q = kFoldQuads - 1;
  if (len <= q * kFoldLastPer) return {1u, (int)((len + q - 1) / q)};
  const size_t per = len <= q * q * kFoldLastPer ? 2 : 4;  // (two items leave len / 63 <= 504)
  return {(unsigned)((len + q * per - 1) / (q * per)), (int)per};
}

// k_reduce's levels over S spaces of K buckets (a power of two): one block a
// space for up to 256 buckets; above that a first level of blocks of 64 quads, 2^lf
// buckets a quad, and then one block a space over the blocks' results. lf weighs a
// block's chain, 2^(lf + 1) additions for its runs and 12 for the scan and the tree,
// against how many blocks an SM has after one another: an addition takes 2.3 us in a
// block that has its SM to itself and 2.0 for each block where there are more (at
// 2^16 buckets: 64 against 80 us for one space at three and two bits, for four spaces
// 175, 176 and 224 at five, four and three, for seven 264 at four and 304 at five;
// four a quad while that fitted four blocks an SM: one 2^18-point column 517 -> 489
// us, four 1249 -> 1192, one of 2^14 264 -> 258, one-byte pairs of 2^20 517 -> 489).
constexpr uint32_t kReduceOneBlock = 256;
struct ReducePlan {
  unsigned blocks = 1;  // a space, in the first level (last_scale 0: no such level)
  int lf = 0;
  int last_quads, last_m, last_lf = 0, last_scale = 0;
};
inline ReducePlan reduce_plan(uint32_t K, int S, int sm_count) {
  ReducePlan p;
  p.last_m = (int)K;
  if (K > kReduceOneBlock) {
    auto blocks = [&](int lf) { return K / ((uint32_t)kReduceQuads << lf); };
    size_t best = 0;
    for (int lf = 1; blocks(lf) >= 1; ++lf) {
      const size_t all = (size_t)S * blocks(lf), turns = (all + sm_count - 1) / sm_count;
      const size_t last = std::max<size_t>(1, blocks(lf) / kReduceQuads);  // entries a quad at the end
      const size_t cost = (((size_t)2 << lf) + 12) * (turns == 1 ? 23 : 20 * turns) + 3 * (last - 1) * 23;
      if (blocks(lf) <= 1024u && (best == 0 || cost < best)) {
        best = cost;
        p.lf = lf;
      }
    }
    p.blocks = blocks(p.lf);
    p.last_m = (int)p.blocks;
    for (uint32_t len = (uint32_t)kReduceQuads << p.lf; len > 1; len >>= 1) ++p.last_scale;
  }
  while ((p.last_m >> p.last_lf) > kReduceQuads) ++p.last_lf;
  p.last_quads = std::max(8, p.last_m >> p.last_lf);  // whole warps
  return p;
}
// The tails' kernels hold about 170 registers, one block an SM; where there are more
// blocks than SMs, a form of 128 (some spilled) lets two share one: four 2^12-point
// columns 285 -> 264 us, 2^20 one-byte scalars 470 -> 451, but 2^8 points 176 -> 178.
template <class K>
inline K tail_kernel(K one, K two, size_t blocks, int sm_count) {
  return blocks > (size_t)sm_count ? two : one;
}
inline size_t reduce_smem(int quads) { return (size_t)quads * sizeof(Xyzz); }

template <class T>
inline unsigned blocks_for(size_t n, int threads) {
  return (unsigned)((n + threads - 1) / threads);
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

uint32_t publish_checked(Ctx& c, const void* d_src, size_t bytes) {
  uint8_t* pinned = c.host_pinned();
  if (bytes > Ctx::kPinnedBytes - Ctx::kPinnedTables || bytes % 16) throw Error(APG_ERR_INTERNAL, "an odd result");
  launch_chained(c, k_publish, 1, 512, 0, (const uint4*)d_src, (uint32_t)(bytes / 16), (const uint32_t*)c.d_flags,
                 reinterpret_cast<uint4*>(pinned + Ctx::kPinnedTables), reinterpret_cast<uint32_t*>(pinned),
                 ++c.flag_seq);
  return c.flag_seq;
}

void collect_checked(Ctx& c, uint32_t seq, size_t bytes, void* host) {
  if (seq != c.flag_seq) throw Error(APG_ERR_INTERNAL, "a result collected after another was published");
  c.wait_flag();
  memcpy(host, c.host_pinned() + Ctx::kPinnedTables, bytes);
  if (reinterpret_cast<const uint32_t*>(c.host_pinned())[1]) c.check_flags();  // clears the flags and throws
}

void fetch_checked(Ctx& c, const void* d_src, size_t bytes, void* host) {
  if (bytes <= Ctx::kPinnedBytes - Ctx::kPinnedTables && bytes % 16 == 0) {
    collect_checked(c, publish_checked(c, d_src, bytes), bytes, host);
    return;
  }
  c.copy(host, d_src, bytes, cudaMemcpyDeviceToHost);
  c.check_flags();
}

void upload_points_async(Ctx& c, const uint8_t* host, size_t n, Affine* dst) {
  if (n == 0) return;
  uint4* raw = c.scratch[S_TMP7].as<uint4>(4 * n);
  c.copy(raw, host, 64 * n, cudaMemcpyHostToDevice);
  launch(c, k_points_in, blocks_for<int>(n, 256), 256, 0, (const uint4*)raw, n, dst, c.d_flags);
}

void upload_points(Ctx& c, const uint8_t* host, size_t n, Affine* dst) {
  upload_points_async(c, host, n, dst);
  if (n) c.check_flags();
}

void download_points(Ctx& c, const Affine* src, size_t n, uint8_t* host) {
  if (n == 0) return;
  uint4* raw = c.scratch[S_TMP7].as<uint4>(4 * n);
  launch(c, k_points_out, blocks_for<int>(n, 256), 256, 0, src, n, raw);
  c.copy(host, raw, 64 * n, cudaMemcpyDeviceToHost);
  APG_CUDA(cudaStreamSynchronize(c.stream));
}

void generate_srs(Ctx& c, const uint8_t tau_canonical[32], size_t n, Affine* dst) {
  Fr* d_tau = c.scratch[S_TMP6].as<Fr>(1);
  c.copy(d_tau, tau_canonical, 32, cudaMemcpyHostToDevice);
  launch(c, k_fr_to_mont, 1, 1, 0, d_tau, (size_t)1, c.d_flags);
  c.check_flags();
  Fr tau_mont;
  c.copy(&tau_mont, d_tau, 32, cudaMemcpyDeviceToHost);
  APG_CUDA(cudaStreamSynchronize(c.stream));
  launch(c, k_srs_powers, blocks_for<int>(n, 128), 128, 0, tau_mont, n, dst, c.d_flags);
  APG_CUDA(cudaStreamSynchronize(c.stream));
}

static int default_window(size_t n, bool small) {
  int lg = 0;
  while (((size_t)1 << (lg + 1)) <= n) ++lg;
  int cb;
  if (lg <= 4) cb = 3;
  else if (lg <= 8) cb = 5;
  else if (lg <= 12) cb = 9;
  else if (lg <= 16) cb = 12;
  else if (lg <= 20) cb = 15;
  else cb = 16;
  if (small && cb > 11) cb = 11;  // 32-bit scalars: three windows
  return cb;
}

// Window width for n half scalars (127 bits). Eight bits make sixteen windows exactly.
// Swept on a GB300, us a call from host points and scalars, by the whole scalars'
// count: 2^12 at 7/8/9/12 bits 510/494/551/544, 2^14 at 8/12/13 639/621/633, 2^16 at
// 12/13/14 876/866/928, 2^18 at 12/13/16 1900/1746/1735.
static int split_window(size_t n) {
  return n < ((size_t)1 << 15) ? 8 : n < ((size_t)1 << 17) ? 12 : n < ((size_t)1 << 19) ? 13 : 16;
}

static int window_count(int bits, int cb) { return (bits + 1 + cb - 1) / cb; }

const SrsTable* srs_table(Ctx& c, int cbits, size_t need) {
  for (auto& t : c.tables)
    if (t.c == cbits && t.n >= need) return &t;
  if (!c.srs || c.srs_n < need) return nullptr;
  // A wide table covers the whole SRS, a narrower one the prefix that the
  // default rule reads it for until a caller needs more: of a width below 12 the
  // 2^16 points that the autotuner may time it over, of the others the SRS (5 bits
  // take 3.3 KB a point). The prefix's table then goes, with the last context that
  // shares it.
  size_t n = c.srs_n;
  for (size_t prefix : {cbits < 7 ? kNarrowTableMax : (size_t)0, cbits < 12 ? kNarrowWindowMax : (size_t)0,
                        cbits >= 12 && cbits < 16 ? kWideTableMin : (size_t)0})
    if (need <= prefix) n = std::min(n, prefix);
  for (auto it = c.tables.begin(); it != c.tables.end(); ++it)
    if (it->c == cbits) {
      APG_CUDA(cudaStreamSynchronize(c.stream));
      if (c.lane) {  // (a batch gives it the tables anew)
        APG_CUDA(cudaStreamSynchronize(c.lane->stream));
        c.lane->tables.clear();
      }
      c.tables.erase(it);
      break;
    }
  SrsTable t;
  t.c = cbits;
  t.windows = window_count(254, cbits);
  t.n = n;
  // Sorted references carry the table index in 31 bits.
  if ((size_t)t.windows * n >= ((size_t)1 << 31)) throw Error(APG_ERR_OUT_OF_MEMORY, "SRS window table too large");
  APG_CUDA(cudaMalloc(&t.tab, (size_t)t.windows * n * sizeof(Affine)));
  t.mem = std::shared_ptr<void>(t.tab, [](void* p) { cudaFree(p); });
  launch(c, k_window_table, blocks_for<int>(n, 128), 128, 0, (const Affine*)c.srs, n, cbits, t.windows, t.tab,
         c.d_flags);
  APG_CUDA(cudaStreamSynchronize(c.stream));
  c.tables.push_back(t);
  return &c.tables.back();
}

static int ceil_log2(size_t n) {
  int k = 0;
  while (((size_t)1 << k) < n) ++k;
  return k;
}

const SrsTable* srs_table_for(Ctx& c, size_t n, size_t cols, bool tuned) {
  const int cls = ceil_log2(n);
  if (tuned && cls < 64 && c.tuned_c[cls]) {
    const SrsTable* t = srs_table(c, c.tuned_c[cls], n);
    if (t) return t;
  }
  return srs_table(c, default_table_window(n, cols), n);
}

void msm_autotune(Ctx& c, const void* d_sample, size_t sample_len, int kmin, int kmax, const int* cands,
                  size_t ncands, int* chosen) {
  cudaEvent_t e0, e1;
  APG_CUDA(cudaEventCreate(&e0));
  APG_CUDA(cudaEventCreate(&e1));
  uint8_t* d_out = c.scratch[S_TMP4].as<uint8_t>(64);
  for (int k = kmin; k <= kmax; ++k) {
    const size_t n = (size_t)1 << k;
    int best_c = 0;
    float best_ms = 0;
    if (k < 64 && n <= sample_len && n <= c.srs_n) {
      for (size_t j = 0; j < ncands; ++j) {
        const int cb = cands[j];
        if (cb < 2 || cb > 20) continue;
        if (cb < 12 && n > kNarrowWindowMax) continue;
        const SrsTable* t = srs_table(c, cb, n);
        if (!t) continue;
        msm_device(c, nullptr, t, d_sample, false, false, n, d_out, nullptr);  // warm-up
        APG_CUDA(cudaEventRecord(e0, c.stream));
        for (int r = 0; r < 2; ++r) msm_device(c, nullptr, t, d_sample, false, false, n, d_out, nullptr);
        APG_CUDA(cudaEventRecord(e1, c.stream));
        APG_CUDA(cudaEventSynchronize(e1));
        float ms = 0;
        APG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        if (!best_c || ms < best_ms) {
          best_c = cb;
          best_ms = ms;
        }
      }
      c.check_flags();
      c.tuned_c[k] = best_c;
    }
    if (chosen) chosen[k - kmin] = best_c;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
}

MsmPlan msm_plan(size_t n, bool small_scalars, const SrsTable* table, int bits, int full_bits) {
  MsmPlan p;
  p.c = table ? table->c : full_bits < 254 ? split_window(n) : default_window(n, small_scalars);
  p.precomp = table != nullptr;
  p.windows = small_scalars ? window_count(bits, p.c) : table ? table->windows : window_count(full_bits, p.c);
  // A scalar narrower than the window has one digit, itself, and fills no
  // bucket past its own range (one-byte columns over 17-bit windows: 2^8 of
  // 2^16 buckets to scan and reduce).
  p.buckets = 1u << (p.c - 1);
  if (small_scalars && bits < p.c) p.buckets = std::min(p.buckets, 1u << bits);
  return p;
}

namespace {

// Scalars over the caller's own bases are split (k_split) up to this many halves. A
// call without a window table ends in Horner's chain over the windows, one doubling
// after another whatever the size: 254 of them took 520 us of the 750 that a GB300
// needed for 2484 points, half of that when split. us a call, whole -> split: 2^4
// 796 -> 412, 2^12 801 -> 494, 2^16 1140 -> 866, 2^19 2980 -> 2694; at 2^20 the gain
// is down to 5 % for twice the memory of the bases.
constexpr int kSplitBits = 127;
constexpr size_t kSplitMax = (size_t)1 << 20;

// Threads of k_bucket_acc resident on the whole device (one wave).
size_t acc_resident_threads(Ctx& c) {
  static std::once_flag once;
  static int per_sm = 0;
  std::call_once(once, [] {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bucket_acc, 128, 0) != cudaSuccess || per_sm < 1)
      per_sm = 1;
  });
  return (size_t)c.sm_count * (size_t)per_sm * 128;
}

size_t pair_resident_threads(Ctx& c) {
  static std::once_flag once;
  static int per_sm = 0;
  std::call_once(once, [] {
    int a = 0, b = 0;
    if (APG_PAIR_PF) {
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_pair_bwd_pf<true>, kPairThreads, 0) != cudaSuccess)
        a = 1;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_pair_bwd_pf<false>, kPairThreads, 0) != cudaSuccess)
        b = 1;
    } else {
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_pair_bwd<true>, kPairThreads, 0) != cudaSuccess) a = 1;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_pair_bwd<false>, kPairThreads, 0) != cudaSuccess)
        b = 1;
    }
    per_sm = std::max(1, std::min(a, b));
  });
  return (size_t)c.sm_count * (size_t)per_sm * kPairThreads;
}

constexpr size_t kMaxBins = (size_t)(kScanBlock - 1) * kScanBlock * kScanItems;  // one pass of the scan
constexpr size_t kMaxGroupEntries = (size_t)1 << 28;                           // 1 GiB of sorted references

// The accumulation's slices hold at least this many references: a group too
// small to fill the resident wave gets fewer, longer slices, trading serial
// additions a thread against items for the edge fold. Measured on a GB300: one
// 2^8-point uniform column 193 us at four and 215 at eight, one 2^12-point column
// 242 and 216, two 309 and 258.
inline size_t acc_slice_min(size_t entries) { return entries <= ((size_t)1 << 15) ? 4 : 8; }

// Round r's list of the pair rounds fits cap[r]: a round keeps ceil(len/2) of each
// run, so a list never grows and at most halves plus one point per bucket.
struct PairCaps {
  size_t cap[kPairRounds > 0 ? kPairRounds : 1];
};
inline PairCaps pair_caps(size_t emax, size_t nbins) {
  PairCaps p;
  p.cap[0] = std::min((emax + nbins + 1) / 2, kPairMaxPoints);
  for (int r = 1; r < kPairRounds; ++r) p.cap[r] = std::min(p.cap[r - 1], (p.cap[r - 1] + nbins + 1) / 2);
  return p;
}
inline bool takes_pair_rounds(size_t emax, bool uniform) {
  return kPairRounds > 0 && emax >= kPairMinEntries * (uniform ? 1 : 2);
}

// One group: columns share the plan, the bases and one pass of every kernel.
void msm_group(Ctx& c, const Affine* bases, const SrsTable* table, const MsmCols& cols, int ncols, size_t nmax,
               const MsmPlan& p, bool small_scalars, bool scalars_canonical, bool uniform, uint8_t* d_out) {
  const uint32_t K = p.buckets;
  const int spaces_per_col = p.precomp ? 1 : p.windows;
  const int nout = cols.shared ? 1 : ncols;  // results: one per column, or the stack's sum
  const int S = spaces_per_col * nout;
  const size_t nbins = (size_t)S * K;
  size_t emax = 0;
  for (int j = 0; j < ncols; ++j) emax += (size_t)p.windows * cols.len[j];
  const Affine* src = p.precomp ? table->tab : bases;
  const uint32_t tab_n = p.precomp ? (uint32_t)table->n : 0;

  const size_t scan_blocks = (nbins + kScanBlock * kScanItems - 1) / (kScanBlock * kScanItems);
  uint32_t* blk = c.scratch[S_SCANBLK].as<uint32_t>(kScanBlock + 1);
  uint32_t* total = blk + kScanBlock;  // (its own word: the pair rounds scan through blk as well)
  uint32_t* sorted = c.scratch[S_SORTED].as<uint32_t>(std::max<size_t>(emax, 1));
  // The buckets and, after them, their counts: what a group must find at zero.
  const size_t zero_bytes = nbins * sizeof(Xyzz) + (nbins + 1) * sizeof(uint32_t);
  Xyzz* buckets = reinterpret_cast<Xyzz*>(c.scratch[S_BUCKETS].get(zero_bytes));
  uint32_t* counts = reinterpret_cast<uint32_t*>(buckets + nbins);

  const size_t slice_min = acc_slice_min(emax);
  const size_t nseg =
      std::max<size_t>(1, std::min(acc_resident_threads(c), (emax + slice_min - 1) / slice_min));
  uint32_t* ikeys[2] = {c.scratch[S_HEAD].as<uint32_t>(2 * nseg), c.scratch[S_TAIL].as<uint32_t>(2 * nseg)};
  Xyzz* ipts[2] = {c.scratch[S_TMP0].as<Xyzz>(2 * nseg), c.scratch[S_TMP1].as<Xyzz>(2 * nseg)};
  uint8_t* ipres[2] = {c.scratch[S_FLAGS].as<uint8_t>(2 * nseg), c.scratch[S_TMP2].as<uint8_t>(2 * nseg)};

  const ReducePlan rp = reduce_plan(K, S, c.sm_count);
  Xyzz* tsum = c.scratch[S_TSUM].as<Xyzz>(S);
  Xyzz* lvlT = c.scratch[S_LEVEL_T].as<Xyzz>((size_t)S * rp.blocks);
  Xyzz* lvlR = c.scratch[S_LEVEL_A].as<Xyzz>((size_t)S * rp.blocks);

  cudaEvent_t t_total = c.timer_begin();
  c.fill(buckets, 0, zero_bytes);
  const int canon = scalars_canonical ? 1 : 0;
  // One pass over the digits: counted (place null) or placed.
  auto digits = [&](uint32_t* place) {
    const uint32_t few = (uint32_t)spaces_per_col * K;
    if (few <= kFewBins) {
      // Tiles of 256 scalars until they fill the device twice, then up to
      // eight times as long: a block's counters cost it one pass over them. Fewer
      // scalars a tile, down to 32, while there are fewer blocks than SMs and a
      // tile has as many digits as the block has counters.
      const size_t tiles = (std::max<size_t>(nmax, 1) + kFewChunk - 1) / kFewChunk;
      uint32_t tile = kFewChunk *
                      (uint32_t)std::min<size_t>(8, std::max<size_t>(1, tiles * ncols / (2 * (size_t)c.sm_count)));
      while (tile > 32 && tile <= kFewChunk && (nmax + tile - 1) / tile * ncols < (size_t)c.sm_count &&
             tile / 2 * (uint32_t)p.windows >= few)
        tile /= 2;
      const dim3 grid((unsigned)((std::max<size_t>(nmax, 1) + tile - 1) / tile), (unsigned)ncols);
      DigitBias bias{};
      for (int w = 0; w + 1 < p.windows; ++w) {
        const int at = w * p.c + p.c - 1;
        if (at < 256) bias.w[at >> 5] |= 1u << (at & 31);
      }
      const size_t smem = sizeof(uint32_t) * (few + (tile < kFewChunk ? (small_scalars ? 2 : 8) * tile : 0));
      void (*k)(MsmCols, int, int, int, uint32_t, uint32_t, int, uint32_t, DigitBias, uint32_t*, uint32_t*, uint32_t*) =
          small_scalars ? (place ? k_digits_few<true, true> : k_digits_few<true, false>)
                        : (place ? k_digits_few<false, true> : k_digits_few<false, false>);
      launch_chained(c, k, grid, 256, smem, cols, p.c, p.windows, (int)p.precomp, K, tab_n, canon, tile, bias, counts,
                     place, c.d_flags);
    } else {
      const dim3 grid(blocks_for<int>(std::max<size_t>(nmax, 1), kDigitThreads), (unsigned)ncols);
      void (*k)(MsmCols, int, int, int, uint32_t, uint32_t, int, uint32_t*, uint32_t*, uint32_t*) =
          small_scalars ? (place ? k_digits<true, true> : k_digits<true, false>)
                        : (place ? k_digits<false, true> : k_digits<false, false>);
      launch_chained(c, k, grid, kDigitThreads, 0, cols, p.c, p.windows, (int)p.precomp, K, tab_n, canon, counts, place,
                     c.d_flags);
    }
  };
  digits(nullptr);
  launch_chained(c, k_scan_local, (unsigned)scan_blocks, kScanBlock, 0, counts, nbins, scan_blocks > 1 ? blk : total);
  if (scan_blocks > 1)
    launch_chained(c, k_scan_add, (unsigned)scan_blocks, 256, 0, counts, nbins, (const uint32_t*)blk, total);
  digits(sorted);
  cudaEvent_t t_acc = c.timer_begin();
  const uint32_t* pair_mode = nullptr;
  const uint32_t* pair_ends = nullptr;
  const Affine* pair_pts = nullptr;
  if (takes_pair_rounds(emax, uniform)) {
    const PairCaps caps = pair_caps(emax, nbins);
    const size_t* cap = caps.cap;
    const size_t T = pair_resident_threads(c);
    Affine* lst[2] = {c.scratch[S_PAIR_A].as<Affine>(cap[0]),
                      c.scratch[S_PAIR_B].as<Affine>(kPairRounds > 1 ? cap[1] : 1)};
    // Running products (one a slot, j * T + s), the lanes' totals and, with
    // APG_PAIR_PF, the slot words (4 bytes a slot) after them.
    const size_t P = (cap[0] + T - 1) / T * T;
    Fq* pp = c.scratch[S_PAIR_PP].as<Fq>(P + T + (APG_PAIR_PF ? (P + 7) / 8 : 0));
    Fq* tot = pp + P;
    uint32_t* idx = APG_PAIR_PF ? reinterpret_cast<uint32_t*>(tot + T) : nullptr;
    uint32_t* cnt = c.scratch[S_PAIR_CNT].as<uint32_t>((size_t)kPairRounds * (nbins + 1) + 2);
    uint32_t* mode = cnt + (size_t)kPairRounds * (nbins + 1);
    c.fill(mode, 0, 2 * sizeof(uint32_t));
    const size_t scan_n = nbins + 1;
    const unsigned sblocks = (unsigned)((scan_n + kScanBlock * kScanItems - 1) / (kScanBlock * kScanItems));
    const uint32_t* ends_in = counts;
    const unsigned pblocks = (unsigned)((T + kPairThreads - 1) / kPairThreads);
    for (int r = 0; r < kPairRounds; ++r) {
      uint32_t* st = cnt + (size_t)r * scan_n;
      launch(c, k_halve_counts, blocks_for<int>(scan_n, 256), 256, 0, ends_in, (uint32_t)nbins, st);
      launch_chained(c, k_scan_local, sblocks, kScanBlock, 0, st, scan_n, blk);
      if (sblocks > 1) launch_chained(c, k_scan_add, sblocks, 256, 0, st, scan_n, (const uint32_t*)blk, mode + 1);
      const uint32_t* rr = r == 0 ? (const uint32_t*)sorted : (const uint32_t*)nullptr;
      const Affine* in = r == 0 ? src : lst[(r - 1) & 1];
      if (r == 0) {
        launch(c, k_pair_fwd<true>, pblocks, kPairThreads, 0, rr, in, ends_in, (const uint32_t*)st, (uint32_t)nbins,
               cap[0], mode, T, pp, tot, idx);
        if (APG_PAIR_PF)
          launch(c, k_pair_bwd_pf<true>, pblocks, kPairThreads, 0, rr, in, (const uint32_t*)idx, (const uint32_t*)st,
                 (uint32_t)nbins, (const uint32_t*)mode, T, (const Fq*)pp, (const Fq*)tot, lst[0], c.d_flags);
        else
          launch(c, k_pair_bwd<true>, pblocks, kPairThreads, 0, rr, in, ends_in, (const uint32_t*)st,
                 (uint32_t)nbins, (const uint32_t*)mode, T, (const Fq*)pp, (const Fq*)tot, lst[0], c.d_flags);
      } else {
        launch(c, k_pair_fwd<false>, pblocks, kPairThreads, 0, rr, in, ends_in, (const uint32_t*)st, (uint32_t)nbins,
               cap[r], mode, T, pp, tot, idx);
        if (APG_PAIR_PF)
          launch(c, k_pair_bwd_pf<false>, pblocks, kPairThreads, 0, rr, in, (const uint32_t*)idx,
                 (const uint32_t*)st, (uint32_t)nbins, (const uint32_t*)mode, T, (const Fq*)pp, (const Fq*)tot,
                 lst[r & 1], c.d_flags);
        else
          launch(c, k_pair_bwd<false>, pblocks, kPairThreads, 0, rr, in, ends_in, (const uint32_t*)st,
                 (uint32_t)nbins, (const uint32_t*)mode, T, (const Fq*)pp, (const Fq*)tot, lst[r & 1], c.d_flags);
      }
      ends_in = st + 1;
    }
    pair_mode = mode;
    pair_ends = ends_in;
    pair_pts = lst[(kPairRounds - 1) & 1];
  }
  launch_chained(c, k_bucket_acc, blocks_for<int>(nseg, 128), 128, 0, (const uint32_t*)sorted, (const uint32_t*)counts,
         (uint32_t)nbins, (const uint32_t*)total, nseg, src, buckets, ikeys[0], ipts[0], ipres[0], pair_mode,
         pair_ends, pair_pts);
  c.timer_end(APG_TIMER_MSM_ACCUMULATE, t_acc);
  for (size_t len = 2 * nseg, cur = 0; len > 2; cur ^= 1) {
    const FoldLevel f = fold_level(len);
    launch_chained(c, tail_kernel(k_fold_edges<1>, k_fold_edges<2>, f.blocks, c.sm_count), f.blocks, 4 * kFoldQuads, 0,
                   (const uint32_t*)ikeys[cur], (const Xyzz*)ipts[cur], (const uint8_t*)ipres[cur], len, f.per, buckets,
                   ikeys[cur ^ 1], ipts[cur ^ 1], ipres[cur ^ 1]);
    len = 2 * (size_t)f.blocks;
  }
  const bool two_levels = rp.last_scale > 0;
  if (two_levels)
    launch_chained(c, tail_kernel(k_reduce<1>, k_reduce<2>, (size_t)rp.blocks * S, c.sm_count), dim3(rp.blocks, S),
           4 * kReduceQuads, reduce_smem(kReduceQuads), (const Xyzz*)buckets,
           (const Xyzz*)nullptr, (int)K, rp.lf, 0, 0, lvlT, lvlR);
  launch_chained(c, tail_kernel(k_reduce<1>, k_reduce<2>, S, c.sm_count), dim3(1, S), 4 * rp.last_quads, reduce_smem(rp.last_quads),
         (const Xyzz*)(two_levels ? lvlR : buckets), (const Xyzz*)(two_levels ? lvlT : nullptr), rp.last_m, rp.last_lf,
         rp.last_scale, 1, tsum, (Xyzz*)nullptr);
  launch_chained(c, k_finish, (unsigned)nout, 32, 0, (const Xyzz*)tsum, spaces_per_col, p.c, (uint32_t*)d_out, c.d_flags);
  c.timer_end(APG_TIMER_MSM_TOTAL, t_total);
}

}  // namespace

size_t msm_scratch_bytes(size_t n, size_t cols, int window, bool uniform) {
  const size_t digits = (size_t)window_count(254, window) * n, K = (size_t)1 << (window - 1);
  const size_t fit = std::min(kMaxBins / K, kMaxGroupEntries / std::max<size_t>(digits, 1));
  const size_t g = std::max<size_t>(1, std::min(std::min(cols, (size_t)kMaxCols), fit)), emax = g * digits, nbins = g * K;
  const size_t resident = (size_t)152 * 1024;  // threads: no kernel here has more on a GB300
  const size_t nseg = std::min(resident, emax / acc_slice_min(emax) + 1);
  size_t b = emax * 4 + nbins * (sizeof(Xyzz) + 4)            // references, buckets, counts
             + 4 * nseg * (sizeof(Xyzz) + 5)                  // the fold's items: two lists of two a slice
             + nbins / kReduceQuads * 2 * sizeof(Xyzz);       // the reduction's first level
  if (takes_pair_rounds(emax, uniform)) {
    const PairCaps caps = pair_caps(emax, nbins);
    b += (caps.cap[0] + caps.cap[kPairRounds > 1 ? 1 : 0]) * sizeof(Affine) + (caps.cap[0] + 2 * resident) * sizeof(Fq) +
         kPairRounds * nbins * 4;
    if (APG_PAIR_PF) b += (caps.cap[0] + resident) * 4;
  }
  return b + b / 8 + ((size_t)1 << 20);  // (a buffer grows by an eighth more than it is asked for)
}

void msm_multi(Ctx& c, const Affine* bases, const SrsTable* table, const void* const* scalars, const size_t* lens,
               size_t k, bool small_scalars, bool scalars_canonical, uint8_t* d_out, const MsmBatchOpts& o) {
  // Field elements over the caller's bases: as halves, while they are few enough.
  if (!table && !small_scalars && o.full_bits == 254 && k <= (size_t)kMaxCols) {
    size_t n2 = 0, nmax = 0;
    for (size_t j = 0; j < k; ++j) {
      n2 = lens[j] > kSplitMax ? kSplitMax + 1 : std::min(kSplitMax + 1, n2 + 2 * lens[j]);
      nmax = std::max(nmax, lens[j]);
    }
    if (n2 > 0 && n2 <= kSplitMax) {
      Affine* sb = c.scratch[S_SPLIT_BASES].as<Affine>(n2);
      Fr* ss = c.scratch[S_SPLIT_SCALARS].as<Fr>(n2);
      SplitCols S{};
      const void* ptrs[kMaxCols];
      size_t len2[kMaxCols], offs[kMaxCols], at = 0;
      for (size_t j = 0; j < k; ++j) {
        S.in.s[j] = scalars[j];
        S.in.len[j] = (uint32_t)lens[j];
        S.in.off[j] = o.offs ? (uint32_t)o.offs[j] : 0u;
        S.at[j] = (uint32_t)at;
        ptrs[j] = ss + at;
        len2[j] = 2 * lens[j];
        offs[j] = at;
        at += len2[j];
      }
      launch(c, k_split, dim3(blocks_for<int>(nmax, 128), (unsigned)k), 128, 0, S, bases, scalars_canonical ? 1 : 0, sb,
             ss, c.d_flags);
      MsmBatchOpts o2 = o;
      o2.offs = offs;
      o2.full_bits = kSplitBits;
      return msm_multi(c, sb, nullptr, ptrs, len2, k, false, true, d_out, o2);
    }
  }
  // A stack sums its columns: every group writes one partial result, added
  // at the end when there is more than one.
  uint8_t* partial = nullptr;
  size_t ngroups = 0;
  if (o.stack) partial = c.scratch[S_TMP7].as<uint8_t>(64 * ((k + kMaxCols - 1) / kMaxCols + k));
  size_t j = 0;
  while (j < k) {
    // Grow the group while the plan, the bucket range and the sorted list fit.
    size_t nmax = 0;
    MsmPlan p{};
    size_t g = 0;
    while (j + g < k && g < (size_t)kMaxCols) {
      const size_t n = lens[j + g];
      if (n >= ((size_t)1 << 31)) throw Error(APG_ERR_INVALID_ARGUMENT, "MSM longer than 2^31 - 1 points");
      const size_t nm = std::max(nmax, n);
      const MsmPlan q = msm_plan(std::max<size_t>(nm, 1), small_scalars, table, o.bits, o.full_bits);
      const size_t spaces = q.precomp ? 1 : (size_t)q.windows;
      const size_t bins = (g + 1) * spaces * q.buckets;
      size_t e = 0;
      for (size_t t = 0; t <= g; ++t) e += (size_t)q.windows * lens[j + t];
      if (g > 0 && (bins > kMaxBins || e > kMaxGroupEntries || q.c != p.c || q.windows != p.windows)) break;
      if (bins > kMaxBins) throw Error(APG_ERR_INVALID_ARGUMENT, "too many buckets");
      p = q;
      nmax = nm;
      ++g;
    }
    MsmCols cols{};
    for (size_t t = 0; t < g; ++t) {
      cols.s[t] = scalars[j + t];
      cols.len[t] = (uint32_t)lens[j + t];
      cols.off[t] = o.offs ? (uint32_t)o.offs[j + t] : 0u;
    }
    cols.shared = o.stack ? 1 : 0;
    cols.bits = o.bits;
    uint8_t* dst = !o.stack ? d_out + 64 * j : g == k ? d_out : partial + 64 * ngroups;  // (one group: the sum itself)
    msm_group(c, bases, table, cols, (int)g, nmax, p, small_scalars, scalars_canonical, o.uniform, dst);
    ++ngroups;
    j += g;
  }
  if (o.stack) {
    if (ngroups == 0) c.fill(d_out, 0, 64);
    else if (ngroups > 1) launch(c, k_add_points, 1, 32, 0, (const uint32_t*)partial, (int)ngroups, (uint32_t*)d_out, c.d_flags);
  }
}

void msm_device(Ctx& c, const Affine* bases, const SrsTable* table, const void* scalars, bool small_scalars,
                bool scalars_canonical, size_t n, uint8_t* out64_device, uint8_t* host_out, const MsmBatchOpts& o) {
  if (n == 0) {
    if (out64_device) c.fill(out64_device, 0, 64);
    if (host_out) memset(host_out, 0, 64);
    return;
  }
  uint8_t* d_out = out64_device ? out64_device : c.scratch[S_RESULT].as<uint8_t>(64);
  msm_multi(c, bases, table, &scalars, &n, 1, small_scalars, scalars_canonical, d_out, o);
  if (host_out) {
    fetch_checked(c, d_out, 64, host_out);
  }
}

// ---------------------------------------------------------------------------
// The allocation-free MSM (apg_msm_noalloc).
//
// Some callers cannot let a library allocate device memory on their behalf:
// a serving loop that has already promised every byte of HBM to admitted
// requests (a cudaMalloc there can fail a request that was admitted, or push
// another tenant out of memory), or a latency-critical pipeline that cannot
// afford the device-wide synchronisation cudaMalloc and cudaFree imply. For
// them this variant of the MSM runs the same kernels with all of its scratch
// in one fixed array that lives in the module's global memory, reserved when
// the module is loaded on a device (with CUDA's lazy loading: the first call,
// or the first launch of any kernel of this file, on that device -- make it
// before the device's memory is promised) and held until the process exits.
// It calls no cudaMalloc, no cudaFree and no allocating library routine.
//
// Limit: at most kNoAllocMaxPoints bases. The plan is fixed: 9-bit signed
// windows (29 of them) with one bucket set per window, 16 entries per
// accumulation segment, so every buffer has a size known at compile time.
// ---------------------------------------------------------------------------

namespace {

constexpr size_t kNoAllocMaxPoints = 4096;
constexpr int kNoAllocC = 9;
constexpr int kNoAllocWindows = (254 + 1 + kNoAllocC - 1) / kNoAllocC;  // 29
constexpr int kNoAllocK = 1 << (kNoAllocC - 1);                          // 256 buckets a window
constexpr size_t kNoAllocBins = (size_t)kNoAllocWindows * kNoAllocK;
constexpr size_t kNoAllocEntries = (size_t)kNoAllocWindows * kNoAllocMaxPoints;
constexpr int kNoAllocSeg = 16;
constexpr size_t kNoAllocSegs = (kNoAllocEntries + kNoAllocSeg - 1) / kNoAllocSeg;
constexpr size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Byte offsets of every buffer inside the array.
constexpr size_t kOffFlags = 0;
constexpr size_t kOffTotal = kOffFlags + 256;
constexpr size_t kOffResult = kOffTotal + 256;
constexpr size_t kOffBases = kOffResult + 256;
constexpr size_t kOffEntries = kOffBases + align256(kNoAllocMaxPoints * sizeof(Affine));
constexpr size_t kOffSorted = kOffEntries + align256(kNoAllocEntries * 8);
constexpr size_t kOffCounts = kOffSorted + align256(kNoAllocEntries * 8);
constexpr size_t kOffScanBlk = kOffCounts + align256((kNoAllocBins + 1) * 4);
constexpr size_t kOffBuckets = kOffScanBlk + align256((kScanBlock + 1) * 4);
constexpr size_t kOffKeys0 = kOffBuckets + align256(kNoAllocBins * sizeof(Xyzz));
constexpr size_t kOffKeys1 = kOffKeys0 + align256(2 * kNoAllocSegs * 4);
constexpr size_t kOffPts0 = kOffKeys1 + align256(2 * kNoAllocSegs * 4);
constexpr size_t kOffPts1 = kOffPts0 + align256(2 * kNoAllocSegs * sizeof(Xyzz));
constexpr size_t kOffPres0 = kOffPts1 + align256(2 * kNoAllocSegs * sizeof(Xyzz));
constexpr size_t kOffPres1 = kOffPres0 + align256(2 * kNoAllocSegs);
constexpr size_t kOffTsum = kOffPres1 + align256(2 * kNoAllocSegs);
constexpr size_t kNoAllocBytes = kOffTsum + align256((size_t)kNoAllocWindows * sizeof(Xyzz));

}  // namespace

// The scratch itself (about 8.5 MB). In host code this name is only a
// stand-in for the device symbol: its device address comes from
// cudaGetSymbolAddress, once per device.
static __device__ __align__(256) uint8_t g_noalloc_scratch[kNoAllocBytes];

namespace {

std::mutex g_noalloc_mu;
void* g_noalloc_addr[256] = {nullptr};

// The array's device address, looked up once per device, on the first call
// made with that device current (the set-up step; with CUDA's lazy module
// loading that lookup, or the first launch of any other kernel of this file
// on the device, loads the module, which is when the array is reserved). The
// address belongs to the device's primary context, the one the CUDA runtime
// uses: the entry point assumes no cudaDeviceReset while the library is
// loaded and no other current context.
int noalloc_scratch(int device, uint8_t** out) {
  if (device < 0 || device >= 256) return APG_ERR_NO_DEVICE;
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_addr[device]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return APG_ERR_CUDA;
    g_noalloc_addr[device] = p;
  }
  *out = (uint8_t*)g_noalloc_addr[device];
  return APG_OK;
}

#define APG_NA(call)                                \
  do {                                              \
    if ((call) != cudaSuccess) return APG_ERR_CUDA; \
  } while (0)
#define APG_NA_LAUNCH()                                     \
  do {                                                      \
    if (cudaGetLastError() != cudaSuccess) return APG_ERR_CUDA; \
  } while (0)

int msm_noalloc(const void* d_bases, const void* d_scalars, size_t n, void* d_out, cudaStream_t st) {
  if (n > kNoAllocMaxPoints) return APG_ERR_NOALLOC_TOO_LARGE;
  if (!d_out || (n && (!d_bases || !d_scalars))) return APG_ERR_INVALID_ARGUMENT;
  int device = 0;
  APG_NA(cudaGetDevice(&device));
  uint8_t* s = nullptr;
  int rc = noalloc_scratch(device, &s);
  if (rc) return rc;
  if (n == 0) {
    APG_NA(cudaMemsetAsync(d_out, 0, 64, st));
    APG_NA(cudaStreamSynchronize(st));
    return APG_OK;
  }
  uint32_t* flags = (uint32_t*)(s + kOffFlags);
  uint32_t* total = (uint32_t*)(s + kOffTotal);
  Affine* bases = (Affine*)(s + kOffBases);
  uint64_t* entries = (uint64_t*)(s + kOffEntries);
  uint64_t* sorted = (uint64_t*)(s + kOffSorted);
  uint32_t* counts = (uint32_t*)(s + kOffCounts);
  uint32_t* blk = (uint32_t*)(s + kOffScanBlk);
  Xyzz* buckets = (Xyzz*)(s + kOffBuckets);
  uint32_t* ikeys[2] = {(uint32_t*)(s + kOffKeys0), (uint32_t*)(s + kOffKeys1)};
  Xyzz* ipts[2] = {(Xyzz*)(s + kOffPts0), (Xyzz*)(s + kOffPts1)};
  uint8_t* ipres[2] = {s + kOffPres0, s + kOffPres1};
  Xyzz* tsum = (Xyzz*)(s + kOffTsum);

  const int K = kNoAllocK, W = kNoAllocWindows, spaces = W;
  const size_t nbins = kNoAllocBins;
  const size_t E = (size_t)W * n;
  const size_t nseg = (E + kNoAllocSeg - 1) / kNoAllocSeg;
  const size_t scan_blocks = (nbins + kScanBlock * kScanItems - 1) / (kScanBlock * kScanItems);

  // What a call must find at zero: the error flag, the histogram, the buckets.
  APG_NA(cudaMemsetAsync(flags, 0, 4, st));
  APG_NA(cudaMemsetAsync(counts, 0, (nbins + 1) * sizeof(uint32_t), st));
  APG_NA(cudaMemsetAsync(buckets, 0, nbins * sizeof(Xyzz), st));
  k_points_in<<<blocks_for<int>(n, 256), 256, 0, st>>>((const uint4*)d_bases, n, bases, flags);
  APG_NA_LAUNCH();
  k_recode<false><<<blocks_for<int>(n, 256), 256, 0, st>>>(d_scalars, n, kNoAllocC, W, 0, 0, 0, entries, counts,
                                                            flags);
  APG_NA_LAUNCH();
  k_scan_local<<<(unsigned)scan_blocks, kScanBlock, 0, st>>>(counts, nbins, blk);
  static_assert(kNoAllocBins > (size_t)kScanBlock * kScanItems, "one block's scan leaves its total elsewhere");
  k_scan_add<<<(unsigned)scan_blocks, 256, 0, st>>>(counts, nbins, (const uint32_t*)blk, total);
  k_scatter<<<blocks_for<int>(E, 256), 256, 0, st>>>((const uint64_t*)entries, E, counts, sorted);
  APG_NA_LAUNCH();
  k_accumulate<<<blocks_for<int>(nseg, 128), 128, 0, st>>>((const uint64_t*)sorted, (const uint32_t*)total,
                                                            kNoAllocSeg, nseg, (const Affine*)bases, buckets,
                                                            ikeys[0], ipts[0], ipres[0]);
  APG_NA_LAUNCH();
  for (size_t len = 2 * nseg, cur = 0; len > 2; cur ^= 1) {
    const FoldLevel f = fold_level(len);
    k_fold_edges<1><<<f.blocks, 4 * kFoldQuads, 0, st>>>((const uint32_t*)ikeys[cur], (const Xyzz*)ipts[cur],
                                                      (const uint8_t*)ipres[cur], len, f.per, buckets, ikeys[cur ^ 1],
                                                      ipts[cur ^ 1], ipres[cur ^ 1]);
    APG_NA_LAUNCH();
    len = 2 * (size_t)f.blocks;
  }
  k_reduce<1><<<dim3(1, spaces), 4 * kReduceQuads, reduce_smem(kReduceQuads), st>>>(
      (const Xyzz*)buckets, (const Xyzz*)nullptr, K, 2, 0, 1, tsum, (Xyzz*)nullptr);
  APG_NA_LAUNCH();
  k_finish<<<1, 32, 0, st>>>((const Xyzz*)tsum, spaces, kNoAllocC, (uint32_t*)d_out, flags);
  APG_NA_LAUNCH();
  uint32_t f = 0;
  APG_NA(cudaMemcpyAsync(&f, flags, 4, cudaMemcpyDeviceToHost, st));
  APG_NA(cudaStreamSynchronize(st));
  if (f & DEV_NONCANONICAL) return APG_ERR_NONCANONICAL;
  if (f & DEV_OFF_CURVE) return APG_ERR_INVALID_POINT;
  if (f) return APG_ERR_INTERNAL;
  return APG_OK;
}

static_assert(kNoAllocK == 4 * kReduceQuads, "the reduction above is one block a window");

}  // namespace

}  // namespace apg

extern "C" int apg_msm_noalloc(const void* d_bases, const void* d_scalars, size_t n, void* d_out, void* stream) {
  return apg::msm_noalloc(d_bases, d_scalars, n, d_out, (cudaStream_t)stream);
}
