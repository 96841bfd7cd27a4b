// Mercury opening (crates/pcs/src/lib.rs:313-492) and the batched opening
// (:688-789) with the O(n) passes and every MSM on the device.
//
// Device: the restriction h (one warp per row of the b x b evaluation
// matrix), the column-parallel fold into q and g, the numerator and its
// division by (X - z) -- both linear recurrences, run as multi-level suffix
// Horner scans -- the size-2b transforms behind S, the batch combination and
// all eight MSMs over the resident SRS. Host: the batch's cm* over a few
// commitments (host_g1.hpp), the transcript and the O(1)
// and O(b) scalar glue of the BDFG20 step (crates/pcs-verify/src/bdfg.rs),
// exactly the reference's formulas.
#include <algorithm>

#include "host_g1.hpp"
#include "host_pairing.hpp"
#include "sumcheck.cuh"

namespace apg {

// Commitments a stacked opening sums on the host (host_g1.hpp) rather than
// through the device MSM.
constexpr size_t kHostMsmMax = 32;

using host::F;

namespace {

Fr dv(const F& a) {
  Fr r;
  memcpy(r.v, a.w, 32);
  return r;
}

// A lane's share of sum_i a[i] b[i], i from `first` in steps of `step`: fifteen
// products to a reduction.
__device__ __forceinline__ Fr dot_share(const Fr* a, const Fr* b, size_t n, size_t first, size_t step) {
  Fr acc = fe_zero<FrConsts>();
  for (size_t i = first; i < n;) {
    FeWide<FrConsts> w = wide_zero<FrConsts>();
    for (int k = 0; k < kWideProducts && i < n; ++k, i += step) wide_mac(w, ld_fe(&a[i]), ld_fe(&b[i]));
    acc = fe_add(acc, fe_from_wide(w));
  }
  return acc;
}

__device__ __forceinline__ Fr warp_total(Fr acc) {  // in lane 0
  for (int off = 16; off > 0; off >>= 1) {
    Fr o;
#pragma unroll
    for (int w = 0; w < 8; ++w) o.v[w] = __shfl_down_sync(0xffffffffu, acc.v[w], off);
    acc = fe_add(acc, o);
  }
  return acc;
}

// h_j = sum_i eq1[i] * f[j*b + i], one warp per row, for the columns of a table
// (`one`, when not null, in their place). Bound by its products: unreduced sums
// and all columns in one launch took 16 columns of 2^22 from 1.65 to 0.63 ms on a
// GB300.
__global__ void __launch_bounds__(256) k_row_dot(const Fr* const* cols, const Fr* one, const Fr* eq1, size_t b,
                                                 size_t rows, Fr* h) {
  chain_begin();
  const size_t row = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) / 32;
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const Fr* f = one ? one : cols[blockIdx.y];
  const Fr acc = warp_total(dot_share(eq1, f + row * b, b, lane, 32));
  if (lane == 0) st_fe(&h[blockIdx.y * rows + row], acc);
}

// out[j] = sum_i a[i] * b[j * n + i], a block each.
__global__ void __launch_bounds__(256) k_dot(const Fr* a, const Fr* b, size_t n, Fr* out) {
  chain_begin();
  __shared__ Fr red[8];
  const Fr acc = warp_total(dot_share(a, b + blockIdx.x * n, n, threadIdx.x, blockDim.x));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x != 0) return;
  Fr s = red[0];
  for (int w = 1; w < 8; ++w) s = fe_add(s, red[w]);
  st_fe(&out[blockIdx.x], s);
}

// Suffix Horner over `count` positions of `cols` interleaved columns
// (element j of column c at j*stride + c): acc_j = sum_{k>=j} x_k r^(k-j).
// Pass 1: every segment of L positions folds locally from its top and keeps
// its bottom value as the segment's aggregate.
__global__ void k_suffix_local(const Fr* in, Fr* out, size_t stride, size_t count, size_t cols, int L, Fr r,
                               Fr* agg) {
  chain_begin();
  const size_t id = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t nseg = (count + L - 1) / L;
  if (id >= nseg * cols) return;
  const size_t seg = id / cols, col = id % cols;
  const size_t lo = seg * L, hi = min(lo + (size_t)L, count);
  Fr acc = fe_zero<FrConsts>();
  for (size_t j = hi; j-- > lo;) {
    acc = fe_add(ld_fe(&in[j * stride + col]), fe_mul(r, acc));
    st_fe(&out[j * stride + col], acc);
  }
  st_fe(&agg[seg * cols + col], acc);
}

// The powers a level takes with its launch: r^0 .. r^L for the fix, or r^(2^s)
// for the scan.
constexpr int kSuffixMax = 32;
struct SuffixPowers {
  Fr p[kSuffixMax + 1];
};

// Pass 2: with upper[s] = acc at the bottom of segment s (the next level's
// result), acc_j = local_j + r^(lo_{s+1} - j) * upper[s+1].
__global__ void k_suffix_fix(Fr* out, size_t stride, size_t count, size_t cols, int L, const Fr* upper,
                             const __grid_constant__ SuffixPowers pows) {
  chain_begin();
  const size_t id = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (id >= count * cols) return;
  const size_t j = id / cols, col = id % cols;
  const size_t seg = j / L;
  const size_t nseg = (count + L - 1) / L;
  if (seg + 1 >= nseg) return;
  const size_t next = (seg + 1) * L;
  Fr carry = ld_fe(&upper[(seg + 1) * cols + col]);
  Fr* p = &out[j * stride + col];
  st_fe(p, fe_add(ld_fe(p), fe_mul(pows.p[next - j], carry)));
}

// A column of up to 1024 positions by one block: a thread runs Horner over its R
// positions, the threads' sums are scanned (acc_t += r^(R 2^s) acc_{t + 2^s} for s = 0,
// 1, ...) and what follows a thread's positions is added to them. One position a thread
// up to 256; four above, where a step over all positions would be eight warps a
// scheduler (1024 positions: 28 us, four a thread 14). pows holds r^(2^s), then r^3.
constexpr size_t kSuffixScanMax = 1024;
constexpr int kSuffixCube = 11;
template <int R>
__global__ void __launch_bounds__(256) k_suffix_scan(const Fr* in, Fr* out, size_t stride, int count,
                                                     const __grid_constant__ SuffixPowers pows) {
  chain_begin();
  __shared__ Fr sh[257];
  const int t = threadIdx.x, j = t * R;
  Fr a[R];
#pragma unroll
  for (int i = R - 1; i >= 0; --i) {
    a[i] = j + i < count ? ld_fe(&in[(j + i) * stride + blockIdx.x]) : fe_zero<FrConsts>();
    if (i + 1 < R) a[i] = fe_add(a[i], rmul(pows.p[0], a[i + 1]));
  }
  Fr acc = a[0];
  for (int s = R == 4 ? 2 : 0, off = 1; off * R < count; ++s, off <<= 1) {
    sh[t] = acc;
    __syncthreads();
    if (j + off * R < count) acc = fe_add(acc, rmul(pows.p[s], sh[t + off]));
    __syncthreads();
  }
  if (R == 1) {
    if (j < count) st_fe(&out[j * stride + blockIdx.x], acc);
    return;
  }
  sh[t] = acc;
  __syncthreads();
  const bool more = j + R < count;
  const Fr next = more ? sh[t + 1] : fe_zero<FrConsts>();
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int k = R - i;  // r^k: 4 and 2 are in the list, 3 at its end
    if (i > 0 && more) a[i] = fe_add(a[i], rmul(pows.p[k == 3 ? kSuffixCube : k == 2 ? 1 : 0], next));
    if (j + i < count) st_fe(&out[(j + i) * stride + blockIdx.x], i == 0 ? acc : a[i]);
  }
}

// out[i] = base^i.
__global__ void k_powers(Fr base, size_t count, Fr* out) {
  chain_begin();
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= count) return;
  Fr acc = fe_one<FrConsts>(), b = base;
  for (size_t e = i; e; e >>= 1) {
    if (e & 1) acc = fe_mul(acc, b);
    b = fe_sqr(b);
  }
  st_fe(&out[i], acc);
}

__global__ void k_bitrev(Fr* a, size_t m, int bits) {
  chain_begin();
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= m) return;
  size_t j = __brevll((unsigned long long)i) >> (64 - bits);
  if (i < j) {
    Fr x = ld_fe(&a[i]), y = ld_fe(&a[j]);
    st_fe(&a[i], y);
    st_fe(&a[j], x);
  }
}

// One radix-2 decimation-in-time stage at half-width `half` (the reference's
// butterflies, crates/pcs/src/fft.rs:100-134): tw holds w^k for k < m/2.
__global__ void k_fft_stage(Fr* a, size_t m, size_t half, const Fr* tw) {
  chain_begin();
  size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t >= m / 2) return;
  size_t start = (t / half) * 2 * half, k = t % half;
  Fr w = ld_fe(&tw[k * (m / (2 * half))]);
  Fr lo = ld_fe(&a[start + k]), hi = fe_mul(ld_fe(&a[start + k + half]), w);
  st_fe(&a[start + k], fe_add(lo, hi));
  st_fe(&a[start + k + half], fe_sub(lo, hi));
}

// ---- the O(b) polynomials of the BDFG step ---------------------------------------

// out[q] = poly_q(x_q), a block each: a thread runs Horner over a run of `run`
// coefficients, then the runs fold by doubling distances; pw[q] holds x and
// x^(run 2^s) for s = 0..7.
constexpr int kEvals = 6;
struct EvalArgs {
  const Fr* poly[kEvals];
  uint32_t len[kEvals];
  Fr pw[kEvals][9];
};
__global__ void __launch_bounds__(256) k_eval(const __grid_constant__ EvalArgs E, uint32_t run, Fr* out) {
  chain_begin();
  __shared__ Fr sh[256];
  const int q = blockIdx.x, t = threadIdx.x;
  const Fr* p = E.poly[q];
  const uint32_t lo = t * run, hi = min(lo + run, E.len[q]);
  Fr acc = fe_zero<FrConsts>();
  for (uint32_t i = hi; i-- > lo && lo < hi;) acc = fe_add(ld_fe(&p[i]), rmul(E.pw[q][0], acc));
  for (int s = 0; s < 8; ++s) {
    sh[t] = acc;
    __syncthreads();
    if (t + (1 << s) < 256) acc = fe_add(acc, rmul(E.pw[q][s + 1], sh[t + (1 << s)]));
    __syncthreads();
  }
  if (t == 0) st_fe(&out[q], acc);
}

// out[k] = sum_i sum_j mul[i][j] poly_i[k - j] + low[k]: the combination F of the
// four openings' numerators (multipliers of up to three coefficients, the
// interpolants folded into the five lowest), and with one coefficient each the
// linearization.
struct BdfgArgs {
  const Fr* poly[5];
  uint32_t len[5];
  Fr mul[5][3];
  int nmul[5];
  Fr low[5];
};
__global__ void __launch_bounds__(256) k_bdfg(const __grid_constant__ BdfgArgs B, uint32_t n, Fr* out) {
  chain_begin();
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  FeWide<FrConsts> s = wide_zero<FrConsts>();  // (at most fourteen products)
  for (int i = 0; i < 5; ++i)
    for (int j = 0; j < B.nmul[i]; ++j)
      if (k >= (uint32_t)j && k - j < B.len[i]) wide_mac(s, B.mul[i][j], ld_fe(&B.poly[i][k - j]));
  Fr v = fe_from_wide(s);
  if (k < 5) v = fe_add(v, B.low[k]);
  st_fe(&out[k], v);
}

// ---- transforms of up to 2^12 points in one block ------------------------------
//
// 4096 elements are 128 KB of shared memory, so a transform is one block and one
// launch: a launch a stage cost 4 us each, 60 of them in a 2^22 opening. Element
// i's 16-byte halves stand at sh[i] and sh[m + i].
constexpr size_t kFftBlockMax = 4096;

__device__ __forceinline__ Fr fft_ld(const uint4* sh, size_t m, size_t i) {
  const uint4 u = sh[i], v = sh[m + i];
  Fr r;
  r.v[0] = u.x, r.v[1] = u.y, r.v[2] = u.z, r.v[3] = u.w;
  r.v[4] = v.x, r.v[5] = v.y, r.v[6] = v.z, r.v[7] = v.w;
  return r;
}
__device__ __forceinline__ void fft_st(uint4* sh, size_t m, size_t i, const Fr& a) {
  sh[i] = make_uint4(a.v[0], a.v[1], a.v[2], a.v[3]);
  sh[m + i] = make_uint4(a.v[4], a.v[5], a.v[6], a.v[7]);
}

// The decimation-in-time stages over bit-reversed input. tw holds w^k for
// k < m/2; the inverse transform's w^-k is 1 or -w^(m/2 - k).
__device__ __forceinline__ void fft_stages(uint4* sh, size_t m, const Fr* tw, bool inverse) {
  for (size_t half = 1; half < m; half *= 2) {
    __syncthreads();
    for (size_t t = threadIdx.x; t < m / 2; t += blockDim.x) {
      const size_t k = t & (half - 1), at = 2 * (t - k) + k, e = k * (m / (2 * half));
      const Fr lo = fft_ld(sh, m, at);
      Fr hi = fft_ld(sh, m, at + half);
      if (e) hi = rmul(hi, ld_fe(&tw[inverse ? m / 2 - e : e]));
      if (e && inverse) hi = fe_neg(hi);
      fft_st(sh, m, at, fe_add(lo, hi));
      fft_st(sh, m, at + half, fe_sub(lo, hi));
    }
  }
  __syncthreads();
}

// The transforms of g, rev(eq1), h and rev(eq2), each b long in m = 2b, block q
// the q-th: out[q m ..].
struct SymOperands {
  const Fr* src[4];
};
__global__ void __launch_bounds__(1024) k_sym_fft(SymOperands S, size_t b, int bits, const Fr* tw, Fr* out) {
  chain_begin();
  extern __shared__ uint4 sh_fft[];
  const size_t m = 2 * b, q = blockIdx.x;
  const Fr* src = S.src[q];
  for (size_t i = threadIdx.x; i < m; i += blockDim.x) {
    const Fr v = i < b ? ld_fe(&src[q & 1 ? b - 1 - i : i]) : fe_zero<FrConsts>();
    fft_st(sh_fft, m, __brevll((unsigned long long)i) >> (64 - bits), v);
  }
  fft_stages(sh_fft, m, tw, false);
  for (size_t i = threadIdx.x; i < m; i += blockDim.x) st_fe(&out[q * m + i], fft_ld(sh_fft, m, i));
}

// R = IFFT(G P1 + gamma H P2), then S and D and symmetric_witness's two
// assertions (k_sym_out, k_reverse). scale = 1/m.
__global__ void __launch_bounds__(1024) k_sym_ifft(const Fr* t, size_t b, int bits, const Fr* tw, Fr gamma, Fr scale,
                                                   const Fr* h_alpha, Fr gamma_v, const Fr* g, Fr* S, Fr* D,
                                                   uint32_t* flags) {
  chain_begin();
  extern __shared__ uint4 sh_fft[];
  const size_t m = 2 * b;
  for (size_t i = threadIdx.x; i < m; i += blockDim.x) {
    FeWide<FrConsts> s = wide_zero<FrConsts>();
    wide_mac(s, ld_fe(&t[i]), ld_fe(&t[m + i]));
    wide_mac(s, gamma, rmul(ld_fe(&t[2 * m + i]), ld_fe(&t[3 * m + i])));
    fft_st(sh_fft, m, __brevll((unsigned long long)i) >> (64 - bits), fe_from_wide(s));
  }
  fft_stages(sh_fft, m, tw, true);
  if (threadIdx.x == 0 &&
      (!fe_is_zero(fft_ld(sh_fft, m, m - 1)) ||
       !fe_eq(rmul(scale, fft_ld(sh_fft, m, b - 1)), fe_add(ld_fe(h_alpha), gamma_v))))
    atomicOr(flags, (uint32_t)DEV_NONZERO_REM);
  for (size_t i = threadIdx.x; i < b; i += blockDim.x) {
    if (i + 1 < b)
      st_fe(&S[i], rmul(scale, fe_add(fft_ld(sh_fft, m, b + i), fft_ld(sh_fft, m, b - 2 - i))));
    st_fe(&D[i], ld_fe(&g[b - 1 - i]));
  }
}

// The four padded operands of S: g, rev(eq1), h, rev(eq2), each b long in 2b.
__global__ void k_sym_pad(const Fr* g, const Fr* eq1, const Fr* h, const Fr* eq2, size_t b, Fr* G, Fr* P1, Fr* H,
                          Fr* P2) {
  chain_begin();
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= 2 * b) return;
  const Fr z = fe_zero<FrConsts>();
  st_fe(&G[i], i < b ? ld_fe(&g[i]) : z);
  st_fe(&P1[i], i < b ? ld_fe(&eq1[b - 1 - i]) : z);
  st_fe(&H[i], i < b ? ld_fe(&h[i]) : z);
  st_fe(&P2[i], i < b ? ld_fe(&eq2[b - 1 - i]) : z);
}

__global__ void k_sym_mix(const Fr* G, const Fr* P1, const Fr* H, const Fr* P2, size_t m, Fr gamma, Fr* R) {
  chain_begin();
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= m) return;
  Fr a = fe_mul(ld_fe(&G[i]), ld_fe(&P1[i]));
  Fr c = fe_mul(gamma, fe_mul(ld_fe(&H[i]), ld_fe(&P2[i])));
  st_fe(&R[i], fe_add(a, c));
}

__global__ void k_scale(Fr* a, size_t m, Fr s) {
  chain_begin();
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < m) st_fe(&a[i], fe_mul(ld_fe(&a[i]), s));
}

// S[k - b] = R[k] + R[2b - 2 - k] for k in [b, 2b - 1); checks R[2b-1] = 0 and
// R[b-1] = h(alpha) + gamma v (symmetric_witness's two assertions).
__global__ void k_sym_out(const Fr* R, size_t b, const Fr* h_alpha, Fr gamma_v, Fr* S, uint32_t* flags) {
  chain_begin();
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i == 0) {
    if (!fe_is_zero(ld_fe(&R[2 * b - 1])) || !fe_eq(ld_fe(&R[b - 1]), fe_add(ld_fe(h_alpha), gamma_v)))
      atomicOr(flags, (uint32_t)DEV_NONZERO_REM);
  }
  if (i >= b - 1) return;
  size_t k = b + i;
  st_fe(&S[i], fe_add(ld_fe(&R[k]), ld_fe(&R[2 * b - 2 - k])));
}

__global__ void k_reverse(const Fr* src, size_t b, Fr* dst) {
  chain_begin();
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < b) st_fe(&dst[i], ld_fe(&src[b - 1 - i]));
}

// numerator = f - (z^b - alpha) q - g(z), with q the n - b coefficients.
__global__ void k_numerator(const Fr* f, const Fr* q, size_t n, size_t nq, Fr c, Fr gz, Fr* out) {
  chain_begin();
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  Fr v = ld_fe(&f[i]);
  if (i < nq) v = fe_sub(v, fe_mul(c, ld_fe(&q[i])));
  if (i == 0) v = fe_sub(v, gz);
  st_fe(&out[i], v);
}

// f* = sum_j w_j stack_j: stack j's column in slot s (cols[j * maxlen + s],
// null past the stack's end) covers entries [s * 2^width, (s + 1) * 2^width).
// Unreduced sums: 16 columns of 2^22 998 -> 664 us on a GB300.
__global__ void __launch_bounds__(256) k_combine_stacked(const Fr* const* cols, const Fr* w, int nstacks, size_t maxlen, int width,
                                  size_t n, Fr* out) {
  chain_begin();
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const size_t slot = i >> width, row = i & (((size_t)1 << width) - 1);
  Fr acc = fe_zero<FrConsts>();
  if (slot < maxlen)
    for (int j = 0; j < nstacks;) {
      FeWide<FrConsts> s = wide_zero<FrConsts>();
      for (int k = 0; k < kWideProducts && j < nstacks; ++k, ++j) {
        const Fr* col = cols[(size_t)j * maxlen + slot];
        if (col) wide_mac(s, ld_fe(&w[j]), ld_fe(&col[row]));
      }
      acc = fe_add(acc, fe_from_wide(s));
    }
  st_fe(&out[i], acc);
}

// The remainders x[0 .. n) of exact divisions.
__global__ void k_expect_zero(const Fr* x, uint32_t* flags) {
  chain_begin();
  if (!fe_is_zero(ld_fe(&x[threadIdx.x]))) atomicOr(flags, (uint32_t)DEV_NONZERO_REM);
}

inline unsigned nb(size_t n, int t) { return (unsigned)((n + t - 1) / t); }

// ---- host helpers -------------------------------------------------------------

std::vector<F> read_frs(Ctx& c, const Fr* d, size_t n) {
  std::vector<F> v(n);
  if (n) fetch_checked(c, d, 32 * n, v.data());
  return v;
}

// One or two MSMs of the first SRS powers against device scalars, two in one
// group (one sort, accumulation and bucket reduction for both): launched, and
// later fetched as canonical bytes, so that the transcript takes what it already
// has while they run. Openings' scalars are combinations at random points.
const uint8_t* srs_commit_start(Ctx& c, const Fr* d0, size_t len0, const Fr* d1 = nullptr, size_t len1 = 0) {
  const size_t k = d1 ? 2 : 1;
  const SrsTable* t = srs_table_for(c, std::max(len0, len1), k, false);
  if (!t) throw Error(APG_ERR_SRS_TOO_SMALL, "the SRS holds fewer powers than the polynomial has coefficients");
  MsmBatchOpts o;
  o.uniform = true;
  const void* ptrs[2] = {d0, d1};
  const size_t lens[2] = {len0, len1};
  uint8_t* d_out = c.scratch[S_RESULT].as<uint8_t>(128);
  msm_multi(c, nullptr, t, ptrs, lens, k, false, false, d_out, o);
  return d_out;
}

// acc_j = sum_{k >= j} x_k r^(k - j) for every position, in place or not: one
// block scan a column where a column fits a block; else segments (32 positions
// where there are enough to fill the device, 8 where the chain is what counts),
// the same over their aggregates, and a fix. `agg`: the aggregates of this level and
// those above it, one after another in the context's scratch.
bool suffix_one_block(size_t count, size_t cols) { return count <= kSuffixScanMax && cols < ((size_t)1 << 31); }
int suffix_segment(size_t count, size_t cols) { return count * cols >= ((size_t)1 << 20) ? kSuffixMax : 8; }

void suffix_horner(Ctx& c, const Fr* in, Fr* out, size_t stride, size_t count, size_t cols, const F& r,
                   Fr* agg = nullptr) {
  if (count == 0) return;
  SuffixPowers pows;
  if (suffix_one_block(count, cols)) {
    F p = r;
    for (int s = 0; s < 11; ++s) {
      pows.p[s] = dv(p);
      p = host::fsqr(p);
    }
    pows.p[kSuffixCube] = dv(host::fmul(host::fsqr(r), r));
    const size_t per = count > 256 ? 4 : 1, threads = ((count + per - 1) / per + 31) / 32 * 32;
    launch_chained(c, per == 4 ? k_suffix_scan<4> : k_suffix_scan<1>, (unsigned)cols, (unsigned)threads, 0, in, out,
                   stride, (int)count, pows);
    return;
  }
  const int L = suffix_segment(count, cols);
  const size_t nseg = (count + L - 1) / L;
  if (!agg) {
    size_t words = 0;
    for (size_t n = count; n > 1 && !suffix_one_block(n, cols);) {
      const size_t per = suffix_segment(n, cols);
      n = (n + per - 1) / per;
      words += n * cols;
    }
    agg = c.scratch[S_TMP3].as<Fr>(std::max(words, cols));
  }
  launch_chained(c, k_suffix_local, nb(nseg * cols, 128), 128, 0, in, out, stride, count, cols, L, dv(r), agg);
  if (nseg > 1) {
    F p = host::fone();
    for (int k = 0; k <= L; ++k) {
      pows.p[k] = dv(p);
      p = host::fmul(p, r);
    }
    F rL = host::fpow_u64(r, L);
    suffix_horner(c, agg, agg, cols, nseg, cols, rL, agg + nseg * cols);
    launch_chained(c, k_suffix_fix, nb(count * cols, 256), 256, 0, out, stride, count, cols, L, (const Fr*)agg, pows);
  }
}

// out[q] = poly_q(x_q) for up to kEvals polynomials.
void eval_polys(Ctx& c, int n, const Fr* const* poly, const size_t* len, const F* x, Fr* out) {
  EvalArgs E;
  memset(&E, 0, sizeof(E));
  size_t most = 1;
  for (int q = 0; q < n; ++q) most = std::max(most, len[q]);
  const size_t run = (most + 255) / 256;
  for (int q = 0; q < n; ++q) {
    E.poly[q] = poly[q];
    E.len[q] = (uint32_t)len[q];
    E.pw[q][0] = dv(x[q]);
    F p = host::fpow_u64(x[q], run);
    for (int s = 0; s < 8; ++s) {
      E.pw[q][s + 1] = dv(p);
      p = host::fsqr(p);
    }
  }
  launch_chained(c, k_eval, (unsigned)n, 256, 0, E, (uint32_t)run, out);
}

F two_adic_root() {
  // 5^((p - 1) / 2^28), derived rather than transcribed.
  uint64_t e[4] = {host::kP[0] - 1, host::kP[1], host::kP[2], host::kP[3]};
  for (int s = 0; s < 28; ++s) {
    for (int i = 0; i < 3; ++i) e[i] = (e[i] >> 1) | (e[i + 1] << 63);
    e[3] >>= 1;
  }
  return host::fpow(host::from_u64(5), e);
}

// w^k for k < m/2, w of order m = 2^log_m: kept by the context for the sizes that
// transform in one block (64 KB at most each).
const Fr* twiddles(Ctx& c, int log_m) {
  DevBuf& b = c.fft_tw[log_m];
  if (!b.p) {
    F w = two_adic_root();
    for (int i = log_m; i < 28; ++i) w = host::fsqr(w);
    const size_t half = (size_t)1 << (log_m - 1);
    Fr* tw = b.as<Fr>(half);
    launch_chained(c, k_powers, nb(half, 256), 256, 0, dv(w), half, tw);
  }
  return static_cast<const Fr*>(b.p);
}

void fft_inplace(Ctx& c, Fr* a, size_t m, const Fr* tw) {
  int bits = 0;
  while (((size_t)1 << bits) < m) ++bits;
  launch_chained(c, k_bitrev, nb(m, 256), 256, 0, a, m, bits);
  for (size_t half = 1; half < m; half *= 2) launch_chained(c, k_fft_stage, nb(m / 2, 256), 256, 0, a, m, half, tw);
}

// ---- univariate helpers on the host (O(b), crates/pcs-verify/src/uni.rs) -------

typedef std::vector<F> Poly;

F ueval(const Poly& p, const F& x) {
  F acc = host::fzero();
  for (size_t i = p.size(); i-- > 0;) acc = host::fadd(host::fmul(acc, x), p[i]);
  return acc;
}

Poly umul(const Poly& a, const Poly& b) {
  if (a.empty() || b.empty()) return {};
  Poly out(a.size() + b.size() - 1, host::fzero());
  for (size_t i = 0; i < a.size(); ++i)
    for (size_t j = 0; j < b.size(); ++j) out[i + j] = host::fadd(out[i + j], host::fmul(a[i], b[j]));
  return out;
}

void uadd_scaled(Poly& acc, const Poly& src, const F& k) {
  if (src.size() > acc.size()) acc.resize(src.size(), host::fzero());
  for (size_t i = 0; i < src.size(); ++i) acc[i] = host::fadd(acc[i], host::fmul(k, src[i]));
}

Poly uvanishing(const std::vector<F>& roots) {
  Poly out{host::fone()};
  for (auto& r : roots) out = umul(out, {host::fneg(r), host::fone()});
  return out;
}

Poly uinterpolate(const std::vector<std::pair<F, F>>& pts) {
  Poly out(pts.size(), host::fzero());
  for (size_t i = 0; i < pts.size(); ++i) {
    Poly num{host::fone()};
    F den = host::fone();
    for (size_t j = 0; j < pts.size(); ++j) {
      if (i == j) continue;
      num = umul(num, {host::fneg(pts[j].first), host::fone()});
      den = host::fmul(den, host::fsub(pts[i].first, pts[j].first));
    }
    uadd_scaled(out, num, host::fmul(pts[i].second, host::finv(den)));
  }
  return out;
}

F tensor_eval(const std::vector<F>& u, F x) {
  F acc = host::fone();
  for (auto& uk : u) {
    acc = host::fmul(acc, host::fadd(host::fmul(uk, x), host::fsub(host::fone(), uk)));
    x = host::fsqr(x);
  }
  return acc;
}

}  // namespace

// ---------------------------------------------------------------------------
// The verifier's field side (crates/pcs-verify/src/lib.rs:355-434) and the
// point checks around it (crates/pcs/src/lib.rs:509-548, 586-602): the
// opening's transcript schedule replayed, h(alpha) and D(z) derived, the
// BDFG20 batch at z', and the twelve accumulator entries of a deferred check.
// ---------------------------------------------------------------------------

namespace {

struct Entries {
  uint8_t side[12];
  F scalar[12];
  uint8_t point[12][64];
};

// pcs::accumulate (lib.rs:509-548) with pcs_verify::scalars (:366-434).
// `info` names the refused point: 0..7 the proof's points in field order
// (h, q, g, s, d, pi_z, w, w'), 8 the commitment.
int accumulate(const uint8_t cm[64], const std::vector<F>& u, const F& v, const uint8_t proof[704],
               host::Transcript& tr, Entries& out, uint64_t* info) {
  using namespace host;
  const size_t nv = u.size();
  if (nv < 2 || nv > 54 || nv % 2) return APG_ERR_UNSUPPORTED_NUM_VARS;
  for (int i = 0; i < 8; ++i)
    if (!host::g1::valid_encoding(proof + 64 * i)) {
      if (info) *info = (uint64_t)i;
      return APG_ERR_INVALID_POINT;
    }
  if (!host::g1::valid_encoding(cm)) {
    if (info) *info = 8;
    return APG_ERR_INVALID_POINT;
  }
  F ev[6];
  for (int i = 0; i < 6; ++i)
    if (!from_bytes(proof + 512 + 32 * i, ev[i])) return APG_ERR_NONCANONICAL;
  const size_t t = nv / 2, b = (size_t)1 << t;
  const std::vector<F> u1(u.begin(), u.begin() + t), u2(u.begin() + t, u.end());
  const uint8_t* pt[8];
  for (int i = 0; i < 8; ++i) pt[i] = proof + 64 * i;

  // The opening's schedule, step for step.
  tr.absorb(T_MERCURY_INSTANCE, std::vector<F>{from_u64((uint64_t)1 << nv)});
  tr.absorb_g1(T_COMMITMENT, cm, 1);
  std::vector<F> claim = u;
  claim.push_back(v);
  tr.absorb(T_EVALUATION_CLAIM, claim);
  tr.absorb_g1(T_PCS_OPENING, pt[0], 1);
  const F alpha = tr.challenge(T_MERCURY_ALPHA);
  tr.absorb_g1(T_PCS_OPENING, pt[1], 2);
  const F gamma = tr.challenge(T_MERCURY_GAMMA);
  tr.absorb_g1(T_PCS_OPENING, pt[3], 2);
  F z;
  do {
    z = tr.challenge(T_MERCURY_Z);
  } while (z.zero());
  if (fsqr(z) == fone() || z == alpha || fmul(z, alpha) == fone()) return APG_ERR_DEGENERATE_CHALLENGE;
  const F zi = finv(z);
  tr.absorb(T_PCS_OPENING, ev, 6);
  tr.absorb_g1(T_PCS_OPENING, pt[5], 1);
  const F delta = tr.challenge(T_BDFG_BATCH);
  tr.absorb_g1(T_PCS_OPENING, pt[6], 1);
  const F zp = tr.challenge(T_BDFG_POINT);
  tr.absorb_g1(T_PCS_OPENING, pt[7], 1);
  const F rho = tr.challenge(T_PAIRING_MERGE);

  // h(alpha) from the symmetrized identity at z (derive_h_alpha, :205-227)
  // and D(z) = z^(b-1) g(1/z).
  F inner = fadd(fadd(fmul(ev[0], tensor_eval(u1, zi)), fmul(ev[1], tensor_eval(u1, z))),
                 fmul(gamma, fsub(fsub(fadd(fmul(ev[2], tensor_eval(u2, zi)), fmul(ev[3], tensor_eval(u2, z))), v), v)));
  inner = fsub(fsub(inner, fmul(z, ev[4])), fmul(zi, ev[5]));
  const F h_alpha = fmul(inner, finv(from_u64(2)));
  const F d_z = fmul(fpow_u64(z, b - 1), ev[1]);
  // The BDFG20 batch at z' (bdfg::items, crates/pcs-verify/src/bdfg.rs):
  // c_i = delta^i Z_{T minus S_i}(z'), constant = sum_i c_i r_i(z').
  const Poly wa = uvanishing({alpha});
  const Poly zc[4] = {wa, Poly{fone()}, wa, uvanishing({zi, alpha})};
  const Poly rr[4] = {uinterpolate({{z, ev[0]}, {zi, ev[1]}}),
                      uinterpolate({{z, ev[2]}, {zi, ev[3]}, {alpha, h_alpha}}),
                      uinterpolate({{z, ev[4]}, {zi, ev[5]}}), Poly{d_z}};
  F c[4], constant = fzero(), dp = fone();
  for (int i = 0; i < 4; ++i) {
    c[i] = fmul(dp, ueval(zc[i], zp));
    constant = fadd(constant, fmul(c[i], ueval(rr[i], zp)));
    dp = fmul(dp, delta);
  }
  const F z_t = ueval(uvanishing({z, zi, alpha}), zp);
  const F z_pow_b = fpow_u64(z, b);
  // Check A (the fold identity at z) plus rho times check B (the batch).
  const F sc[12] = {fone(),
                    fmul(rho, c[1]),
                    fneg(fsub(z_pow_b, alpha)),
                    fmul(rho, c[0]),
                    fmul(rho, c[2]),
                    fmul(rho, c[3]),
                    z,
                    fneg(fmul(rho, z_t)),
                    fmul(rho, zp),
                    fneg(fadd(ev[0], fmul(rho, constant))),
                    fone(),
                    rho};
  // ENTRY_POINTS (:271-284): the points [cm, h, q, g, s, d, pi_z, w, w',
  // [1]_1], ten on the [1]_2 side, then pi_z and w' on the [x]_2 side.
  uint8_t gen[64] = {0};
  gen[0] = 1;
  gen[32] = 2;
  const uint8_t* at[10] = {cm, pt[0], pt[1], pt[2], pt[3], pt[4], pt[5], pt[6], pt[7], gen};
  const int idx[12] = {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 6, 8};
  for (int i = 0; i < 12; ++i) {
    out.side[i] = i < 10 ? 0 : 1;
    out.scalar[i] = sc[i];
    memcpy(out.point[i], at[idx[i]], 64);
  }
  return APG_OK;
}

void write_entries(const Entries& e, uint8_t* sides, uint8_t* scalars, uint8_t* points) {
  memcpy(sides, e.side, 12);
  memcpy(scalars, e.scalar, 12 * 32);
  memcpy(points, e.point, 12 * 64);
}

bool read_frs_mem(const uint8_t* p, size_t n, std::vector<F>& out) {
  out.resize(n);
  for (size_t i = 0; i < n; ++i) {
    memcpy(out[i].w, p + 32 * i, 32);
    if (!host::below_p(out[i].w)) return false;
  }
  return true;
}

}  // namespace

// pcs::verify_deferred (crates/pcs/src/lib.rs:632-641).
int mercury_verify_deferred_impl(const uint8_t cm[64], const uint8_t* u, size_t u_len, const uint8_t v[32],
                                 const uint8_t proof[704], uint8_t* transcript, uint8_t* sides, uint8_t* scalars,
                                 uint8_t* points, uint64_t* info) {
  if (info) *info = 0;
  if (!cm || (u_len && !u) || !v || !proof || !transcript || !sides || !scalars || !points)
    return APG_ERR_INVALID_ARGUMENT;
  std::vector<F> uu, vv;
  if (!read_frs_mem(u, u_len, uu) || !read_frs_mem(v, 1, vv)) return APG_ERR_NONCANONICAL;
  host::Transcript tr;
  if (!tr.load(transcript)) return APG_ERR_INVALID_ARGUMENT;
  Entries e;
  const int st = accumulate(cm, uu, vv[0], proof, tr, e, info);
  if (st) return st;
  write_entries(e, sides, scalars, points);
  tr.save(transcript);
  return APG_OK;
}

// pcs::batch_verify_deferred (crates/pcs/src/lib.rs:661-670) through
// batch_accumulate (:586-602): check_batch, every commitment validated, the
// preamble (the commitments as passed, u || vs, rho), cm* = sum rho^i cm_i
// and v* = sum rho^i v_i, then the single-instance core.
int mercury_batch_verify_deferred_impl(const uint8_t* cms, size_t k, const uint8_t* u, size_t u_len,
                                       const uint8_t* vs, size_t n_vs, const uint8_t proof[704], uint8_t* transcript,
                                       uint8_t* sides, uint8_t* scalars, uint8_t* points, uint64_t* info) {
  using namespace host;
  if (info) *info = 0;
  if ((k && !cms) || (u_len && !u) || (n_vs && !vs) || !proof || !transcript || !sides || !scalars || !points)
    return APG_ERR_INVALID_ARGUMENT;
  if (k == 0) return APG_ERR_EMPTY_BATCH;
  if (k != n_vs) return APG_ERR_BATCH_LENGTH_MISMATCH;
  if (u_len < 2 || u_len > 54 || u_len % 2) return APG_ERR_UNSUPPORTED_NUM_VARS;
  for (size_t j = 0; j < k; ++j)
    if (!host::g1::valid_encoding(cms + 64 * j)) {
      if (info) *info = 8;
      return APG_ERR_INVALID_POINT;
    }
  std::vector<F> uu, vals;
  if (!read_frs_mem(u, u_len, uu) || !read_frs_mem(vs, n_vs, vals)) return APG_ERR_NONCANONICAL;
  Transcript tr;
  if (!tr.load(transcript)) return APG_ERR_INVALID_ARGUMENT;
  // pcs_verify::batch_preamble (:333-347).
  tr.absorb_g1(T_COMMITMENT, cms, k);
  std::vector<F> claim = uu;
  claim.insert(claim.end(), vals.begin(), vals.end());
  tr.absorb(T_EVALUATION_CLAIM, claim);
  const F rho = tr.challenge(T_MERCURY_BATCH);
  std::vector<F> wts(k);
  F acc = fone(), vstar = fzero();
  for (size_t i = 0; i < k; ++i) {
    wts[i] = acc;
    vstar = fadd(vstar, fmul(acc, vals[i]));
    acc = fmul(acc, rho);
  }
  uint8_t cm_star[64];
  host::g1::msm_small(cms, wts.data(), k, cm_star);
  Entries e;
  const int st = accumulate(cm_star, uu, vstar, proof, tr, e, info);
  if (st) return st;
  write_entries(e, sides, scalars, points);
  tr.save(transcript);
  return APG_OK;
}


// ---------------------------------------------------------------------------
// The pairing step (crates/curve/src/pairing.rs, crates/pcs/src/accumulator.rs
// check_pairings :171-214): e(A, [1]_2) e(-B, [x]_2) == 1 with A and B the
// weighted sums of the entries on each side, over the verifier's SRS points
// (SrsVerifier, crates/srs/src/lib.rs:279-283: [1]_1 || [1]_2 || [x]_2).
// ---------------------------------------------------------------------------

namespace {

struct Vsrs {
  host::pairing::G2 g2_gen, g2_tau;
};

int read_vsrs(const uint8_t vsrs[320], Vsrs& out) {
  if (!host::g1::valid_encoding(vsrs)) return APG_ERR_INVALID_POINT;
  if (!host::pairing::g2from_bytes(vsrs + 64, out.g2_gen) || !host::pairing::g2from_bytes(vsrs + 192, out.g2_tau))
    return APG_ERR_INVALID_POINT;
  return APG_OK;
}

// -P for a canonical encoding (infinity stays infinity).
void g1_negate(const uint8_t p[64], uint8_t out[64]) {
  memcpy(out, p, 64);
  bool inf = true;
  for (int i = 0; i < 64; ++i) inf &= p[i] == 0;
  if (inf) return;
  uint64_t y[4];
  memcpy(y, p + 32, 32);
  if ((y[0] | y[1] | y[2] | y[3]) == 0) return;
  uint64_t br = 0;
  for (int i = 0; i < 4; ++i) {
    const host::u128 d = (host::u128)host::g1::kQ[i] - y[i] - br;
    y[i] = (uint64_t)d;
    br = (uint64_t)(d >> 127);
  }
  memcpy(out + 32, y, 32);
}

bool pairings_hold(const Vsrs& vk, const uint8_t a[64], const uint8_t b[64]) {
  uint8_t nb[64];
  g1_negate(b, nb);
  return host::pairing::pairing_check({a, nb}, {vk.g2_gen, vk.g2_tau});
}

// One deferred check with weight one: A and B summed on the host.
int check_entries(const Vsrs& vk, const Entries& e) {
  std::vector<uint8_t> pa, pb;
  std::vector<F> sa, sb;
  for (int i = 0; i < 12; ++i) {
    auto& pts = e.side[i] ? pb : pa;
    pts.insert(pts.end(), e.point[i], e.point[i] + 64);
    (e.side[i] ? sb : sa).push_back(e.scalar[i]);
  }
  uint8_t a[64], b[64];
  host::g1::msm_small(pa.data(), sa.data(), sa.size(), a);
  host::g1::msm_small(pb.data(), sb.data(), sb.size(), b);
  return pairings_hold(vk, a, b) ? APG_OK : APG_ERR_VERIFICATION_FAILED;
}

}  // namespace

int pairing_impl(const uint8_t p[64], const uint8_t q[128], uint8_t out[384]) {
  if (!p || !q || !out) return APG_ERR_INVALID_ARGUMENT;
  host::pairing::G2 qq;
  if (!host::g1::valid_encoding(p) || !host::pairing::g2from_bytes(q, qq)) return APG_ERR_INVALID_POINT;
  host::g1::Q x, y;
  bool inf;
  host::pairing::g1_affine(p, x, y, inf);
  host::pairing::f12to_bytes(host::pairing::final_exponentiation(host::pairing::miller_loop(x, y, inf, qq)), out);
  return APG_OK;
}

int g2_mul_impl(const uint8_t q[128], const uint8_t k[32], uint8_t out[128]) {
  if (!q || !k || !out) return APG_ERR_INVALID_ARGUMENT;
  host::pairing::G2 qq;
  if (!host::pairing::g2from_bytes(q, qq)) return APG_ERR_INVALID_POINT;
  host::pairing::Big kb(4);
  memcpy(kb.data(), k, 32);
  host::pairing::big_trim(kb);
  host::pairing::g2to_bytes(host::pairing::g2mul(qq, kb), out);
  return APG_OK;
}

int pairing_check_impl(const uint8_t* ps, const uint8_t* qs, size_t n, int* holds) {
  if ((n && (!ps || !qs)) || !holds) return APG_ERR_INVALID_ARGUMENT;
  std::vector<const uint8_t*> pp(n);
  std::vector<host::pairing::G2> qq(n);
  for (size_t i = 0; i < n; ++i) {
    pp[i] = ps + 64 * i;
    if (!host::g1::valid_encoding(pp[i]) || !host::pairing::g2from_bytes(qs + 128 * i, qq[i]))
      return APG_ERR_INVALID_POINT;
  }
  *holds = host::pairing::pairing_check(pp, qq) ? 1 : 0;
  return APG_OK;
}

// pcs::verify (crates/pcs/src/lib.rs:614-628): the deferred check, then its
// pairing.
int mercury_verify_impl(const uint8_t vsrs[320], const uint8_t cm[64], const uint8_t* u, size_t u_len,
                        const uint8_t v[32], const uint8_t proof[704], uint8_t* transcript, uint64_t* info) {
  if (!vsrs) return APG_ERR_INVALID_ARGUMENT;
  uint8_t snap[226], sides[12], scalars[12 * 32], points[12 * 64];
  if (!transcript) return APG_ERR_INVALID_ARGUMENT;
  memcpy(snap, transcript, 226);
  int st = mercury_verify_deferred_impl(cm, u, u_len, v, proof, snap, sides, scalars, points, info);
  if (st) return st;
  Vsrs vk;
  if ((st = read_vsrs(vsrs, vk))) return st;
  Entries e;
  memcpy(e.side, sides, 12);
  memcpy(e.scalar, scalars, sizeof(scalars));
  memcpy(e.point, points, sizeof(points));
  if ((st = check_entries(vk, e))) return st;
  memcpy(transcript, snap, 226);
  return APG_OK;
}

// pcs::batch_verify (lib.rs:648-658).
int mercury_batch_verify_impl(const uint8_t vsrs[320], const uint8_t* cms, size_t k, const uint8_t* u, size_t u_len,
                              const uint8_t* vs, size_t n_vs, const uint8_t proof[704], uint8_t* transcript,
                              uint64_t* info) {
  if (!vsrs || !transcript) return APG_ERR_INVALID_ARGUMENT;
  uint8_t snap[226], sides[12], scalars[12 * 32], points[12 * 64];
  memcpy(snap, transcript, 226);
  int st = mercury_batch_verify_deferred_impl(cms, k, u, u_len, vs, n_vs, proof, snap, sides, scalars, points, info);
  if (st) return st;
  Vsrs vk;
  if ((st = read_vsrs(vsrs, vk))) return st;
  Entries e;
  memcpy(e.side, sides, 12);
  memcpy(e.scalar, scalars, sizeof(scalars));
  memcpy(e.point, points, sizeof(points));
  if ((st = check_entries(vk, e))) return st;
  memcpy(transcript, snap, 226);
  return APG_OK;
}

// The pairing step of pcs::discharge (accumulator.rs:146-163) over the A and B
// its MSMs produced (apg_discharge_msms).
int discharge_pairing_impl(const uint8_t vsrs[320], const uint8_t a[64], const uint8_t b[64]) {
  if (!vsrs || !a || !b) return APG_ERR_INVALID_ARGUMENT;
  Vsrs vk;
  const int st = read_vsrs(vsrs, vk);
  if (st) return st;
  return pairings_hold(vk, a, b) ? APG_OK : APG_ERR_VERIFICATION_FAILED;
}

// ---------------------------------------------------------------------------

int mercury_open_impl(Ctx& c, const Fr* d_f, size_t nv, const uint8_t cm[64], const std::vector<F>& u,
                      host::Transcript& tr, F& v_out, uint8_t proof_out[704]) {
  using namespace host;
  if (nv < 2 || nv > 54 || nv % 2) return APG_ERR_UNSUPPORTED_NUM_VARS;
  if (u.size() != nv) return APG_ERR_POINT_LENGTH_MISMATCH;
  if (!c.srs) return APG_ERR_NO_SRS;
  const size_t n = (size_t)1 << nv;
  if (c.srs_n < n) return APG_ERR_SRS_TOO_SMALL;
  if (nv > 40) return APG_ERR_OUT_OF_MEMORY;
  const size_t t = nv / 2, b = (size_t)1 << t;
  std::vector<F> u1(u.begin(), u.begin() + t), u2(u.begin() + t, u.end());

  Fr* work;
  // eq1 | eq2 | h | g | S | D | acc(n) | num(n) | 4 x (2b) transforms | twiddles
  const size_t words = 6 * b + 2 * n + 8 * b + b + 16;
  c.alloc(&work, 32 * words);
  struct Guard {
    Ctx& c;
    Fr* p;
    ~Guard() { cudaFreeAsync(p, c.stream); }
  } guard{c, work};
  Fr *eq1 = work, *eq2 = eq1 + b, *h = eq2 + b, *g = h + b, *S = g + b, *D = S + b, *acc = D + b, *num = acc + n;
  Fr *TG = num + n, *TP1 = TG + 2 * b, *TH = TP1 + 2 * b, *TP2 = TH + 2 * b, *tw = TP2 + 2 * b, *tmp = tw + b;

  // Step 1: h, v. The claim goes into the transcript while h is committed.
  build_eq_table(c, u1, eq1);
  build_eq_table(c, u2, eq2);
  launch_chained(c, k_row_dot, nb(b * 32, 256), 256, 0, (const Fr* const*)nullptr, d_f, (const Fr*)eq1, b, b, h);
  launch_chained(c, k_dot, 1, 256, 0, (const Fr*)eq2, (const Fr*)h, b, tmp);
  const uint32_t v_there = publish_checked(c, tmp, 32);
  uint8_t pts[8][64];
  const uint8_t* d_pts = srs_commit_start(c, h, b);
  tr.absorb(T_MERCURY_INSTANCE, std::vector<F>{from_u64(n)});
  tr.absorb_g1(T_COMMITMENT, cm, 1);
  F v;
  collect_checked(c, v_there, 32, v.w);
  std::vector<F> claim = u;
  claim.push_back(v);
  tr.absorb(T_EVALUATION_CLAIM, claim);
  tr.open(T_PCS_OPENING, 4);
  fetch_checked(c, d_pts, 64, pts[0]);
  tr.observe_g1(pts[0], 1);
  F alpha = tr.challenge(T_MERCURY_ALPHA);

  // Step 2: the fold. acc rows: acc_j = sum_{k>=j} alpha^(k-j) row_k; q is
  // rows 1..b-1 of acc, g is row 0.
  cudaEvent_t tp = c.timer_begin();
  suffix_horner(c, d_f, acc, b, b, b, alpha);
  c.timer_end(APG_TIMER_MERCURY_PASS, tp);
  c.copy(g, acc, 32 * b, cudaMemcpyDeviceToDevice);
  const Fr* q = acc + b;
  const size_t nq = n - b;
  d_pts = srs_commit_start(c, q, nq, g, b);
  Fr *d_halpha = tmp + 1, *d_ev = tmp + 2;  // h(alpha), then the six values
  {
    const Fr* hp[1] = {h};
    eval_polys(c, 1, hp, &b, &alpha, d_halpha);
  }
  tr.open(T_PCS_OPENING, 8);
  fetch_checked(c, d_pts, 128, pts[1]);
  tr.observe_g1(pts[1], 2);
  F gamma = tr.challenge(T_MERCURY_GAMMA);

  // Step 3: S and D.
  {
    const size_t m = 2 * b;
    int k = 0;
    while (((size_t)1 << k) < m) ++k;
    const Fr gamma_v = dv(fmul(gamma, v));
    if (m <= kFftBlockMax) {
      const Fr* tws = twiddles(c, k);
      const unsigned threads = (unsigned)std::min<size_t>(1024, std::max<size_t>(32, m / 2));
      const size_t smem = 32 * m;
      APG_CUDA(cudaFuncSetAttribute(k_sym_fft, cudaFuncAttributeMaxDynamicSharedMemorySize, 32 * (int)kFftBlockMax));
      APG_CUDA(cudaFuncSetAttribute(k_sym_ifft, cudaFuncAttributeMaxDynamicSharedMemorySize, 32 * (int)kFftBlockMax));
      launch_chained(c, k_sym_fft, 4, threads, smem, SymOperands{{g, eq1, h, eq2}}, b, k, tws, TG);
      launch_chained(c, k_sym_ifft, 1, threads, smem, (const Fr*)TG, b, k, tws, dv(gamma), dv(finv(from_u64(m))),
             (const Fr*)d_halpha, gamma_v, (const Fr*)g, S, D, c.d_flags);
    } else {
      F w = two_adic_root();
      for (int i = k; i < 28; ++i) w = fsqr(w);
      launch_chained(c, k_sym_pad, nb(m, 256), 256, 0, (const Fr*)g, (const Fr*)eq1, (const Fr*)h, (const Fr*)eq2, b, TG, TP1,
             TH, TP2);
      launch_chained(c, k_powers, nb(m / 2, 256), 256, 0, dv(w), m / 2, tw);
      fft_inplace(c, TG, m, tw);
      fft_inplace(c, TP1, m, tw);
      fft_inplace(c, TH, m, tw);
      fft_inplace(c, TP2, m, tw);
      launch_chained(c, k_sym_mix, nb(m, 256), 256, 0, (const Fr*)TG, (const Fr*)TP1, (const Fr*)TH, (const Fr*)TP2, m,
             dv(gamma), TG);
      launch_chained(c, k_powers, nb(m / 2, 256), 256, 0, dv(finv(w)), m / 2, tw);
      fft_inplace(c, TG, m, tw);
      launch_chained(c, k_scale, nb(m, 256), 256, 0, TG, m, dv(finv(from_u64(m))));
      launch_chained(c, k_sym_out, nb(b, 256), 256, 0, (const Fr*)TG, b, (const Fr*)d_halpha, gamma_v, S,
             c.d_flags);
      launch_chained(c, k_reverse, nb(b, 256), 256, 0, (const Fr*)g, b, D);
    }
  }
  d_pts = srs_commit_start(c, S, b - 1, D, b);
  tr.open(T_PCS_OPENING, 8);
  fetch_checked(c, d_pts, 128, pts[3]);
  tr.observe_g1(pts[3], 2);
  F z;
  do {
    z = tr.challenge(T_MERCURY_Z);
  } while (z.zero());
  if (fsqr(z) == fone() || z == alpha || fmul(z, alpha) == fone()) {
    c.last_error = "degenerate challenge set {z, 1/z, alpha}";
    return APG_ERR_DEGENERATE_CHALLENGE;
  }
  F zi = finv(z);

  // Step 4: the six values, the numerator and its quotient by (X - z).
  {
    const Fr* polys[6] = {g, g, h, h, S, S};
    const size_t lens[6] = {b, b, b, b, b - 1, b - 1};
    const F at[6] = {z, zi, z, zi, z, zi};
    eval_polys(c, 6, polys, lens, at, d_ev);
  }
  const std::vector<F> evs = read_frs(c, d_halpha, 7);
  const F h_alpha = evs[0];
  const F* ev = evs.data() + 1;
  F zb = fpow_u64(z, b);
  launch_chained(c, k_numerator, nb(n, 256), 256, 0, d_f, q, n, nq, dv(fsub(zb, alpha)), dv(ev[0]), num);
  tp = c.timer_begin();
  suffix_horner(c, num, num, 1, n, 1, z);
  c.timer_end(APG_TIMER_MERCURY_PASS, tp);
  launch_chained(c, k_expect_zero, 1, 1, 0, (const Fr*)num, c.d_flags);  // the remainder f(z) - ... = 0
  d_pts = srs_commit_start(c, num + 1, n - 1);
  tr.absorb(T_PCS_OPENING, ev, 6);
  tr.open(T_PCS_OPENING, 4);
  fetch_checked(c, d_pts, 64, pts[5]);
  tr.observe_g1(pts[5], 1);

  // Step 4(e): BDFG20 over T = {z, 1/z, alpha} (crates/pcs-verify/src/bdfg.rs).
  F two_inv = finv(from_u64(2));
  F inner = fadd(fadd(fmul(ev[0], tensor_eval(u1, zi)), fmul(ev[1], tensor_eval(u1, z))),
                 fmul(gamma, fsub(fsub(fadd(fmul(ev[2], tensor_eval(u2, zi)), fmul(ev[3], tensor_eval(u2, z))), v), v)));
  inner = fsub(fsub(inner, fmul(z, ev[4])), fmul(zi, ev[5]));
  F ha = fmul(inner, two_inv);
  if (ha != h_alpha) throw Error(APG_ERR_INTERNAL, "h(alpha) does not re-derive from the six values");
  F d_z = fmul(fpow_u64(z, b - 1), ev[1]);
  std::vector<F> tset = {z, zi, alpha};
  Poly wa = uvanishing({alpha});
  Poly zc[4] = {wa, Poly{fone()}, wa, uvanishing({zi, alpha})};
  Poly rr[4] = {uinterpolate({{z, ev[0]}, {zi, ev[1]}}), uinterpolate({{z, ev[2]}, {zi, ev[3]}, {alpha, h_alpha}}),
                uinterpolate({{z, ev[4]}, {zi, ev[5]}}), Poly{d_z}};
  const F delta = tr.challenge(T_BDFG_BATCH);
  // F = sum_i delta^i Z_i (poly_i - r_i), b + 2 coefficients, and W = F / Z_T by
  // its three roots in turn: after a root's suffix Horner the remainder stands
  // first and the quotient after it.
  BdfgArgs B;
  memset(&B, 0, sizeof(B));
  const Fr* polys[4] = {g, h, S, D};
  const uint32_t lens[4] = {(uint32_t)b, (uint32_t)b, (uint32_t)(b - 1), (uint32_t)b};
  F low[5] = {fzero(), fzero(), fzero(), fzero(), fzero()}, pw = fone();
  for (int i = 0; i < 4; ++i) {
    B.poly[i] = polys[i];
    B.len[i] = lens[i];
    B.nmul[i] = (int)zc[i].size();
    for (size_t j = 0; j < zc[i].size(); ++j) B.mul[i][j] = dv(fmul(pw, zc[i][j]));
    const Poly zr = umul(zc[i], rr[i]);
    for (size_t k = 0; k < zr.size(); ++k) low[k] = fsub(low[k], fmul(pw, zr[k]));
    pw = fmul(pw, delta);
  }
  for (int k = 0; k < 5; ++k) B.low[k] = dv(low[k]);
  Fr* dF = TH;  // reuse a transform buffer (2b >= b + 2)
  launch_chained(c, k_bdfg, nb(b + 2, 256), 256, 0, B, (uint32_t)(b + 2), dF);
  for (int r = 0; r < 3; ++r) suffix_horner(c, dF + r, dF + r, 1, b + 2 - r, 1, tset[r]);
  launch_chained(c, k_expect_zero, 1, 3, 0, (const Fr*)dF, c.d_flags);
  const Fr* dW = dF + 3;
  d_pts = srs_commit_start(c, dW, b - 1);
  tr.open(T_PCS_OPENING, 4);
  fetch_checked(c, d_pts, 64, pts[6]);
  tr.observe_g1(pts[6], 1);
  F zp = tr.challenge(T_BDFG_POINT);
  // The linearization - Z_T(z') W + sum_i c_i poly_i - constant, and W' = it / (X - z').
  memset(&B, 0, sizeof(B));
  F cst = fzero();
  for (int i = 0; i < 4; ++i) {
    F cc = fmul(fpow_u64(delta, i), ueval(zc[i], zp));
    B.poly[i] = polys[i];
    B.len[i] = lens[i];
    B.nmul[i] = 1;
    B.mul[i][0] = dv(cc);
    cst = fadd(cst, fmul(cc, ueval(rr[i], zp)));
  }
  B.poly[4] = dW;
  B.len[4] = (uint32_t)(b - 1);
  B.nmul[4] = 1;
  B.mul[4][0] = dv(fneg(ueval(uvanishing(tset), zp)));
  B.low[0] = dv(fneg(cst));
  Fr* dL = TP2;
  launch_chained(c, k_bdfg, nb(b, 256), 256, 0, B, (uint32_t)b, dL);
  suffix_horner(c, dL, dL, 1, b, 1, zp);
  launch_chained(c, k_expect_zero, 1, 1, 0, (const Fr*)dL, c.d_flags);
  d_pts = srs_commit_start(c, dL + 1, b - 1);
  tr.open(T_PCS_OPENING, 4);
  fetch_checked(c, d_pts, 64, pts[7]);
  tr.observe_g1(pts[7], 1);
  (void)tr.challenge(T_PAIRING_MERGE);

  v_out = v;
  for (int i = 0; i < 8; ++i) memcpy(proof_out + 64 * i, pts[i], 64);
  for (int i = 0; i < 6; ++i) to_bytes(ev[i], proof_out + 512 + 32 * i);
  return APG_OK;
}

// batch_open_stacked (crates/pcs/src/lib.rs:705-789) past its refusals, which
// the caller has checked: stack j's columns (d_cols, stack after stack, each
// 2^width entries on the device) fill its first stack_lens[j] slots of a
// (width + |r|)-variable table. Each column's value at u comes from one row
// dot against eq(u_lo) and one dot against eq(u_hi); v_j = sum_s eq(r, s) *
// col_{j,s}(u); the preamble absorbs the commitments, u || r and the values
// and draws rho (:568-581); cm* = sum_j rho^j cm_j is a generic-base MSM and
// f* = sum_j rho^j stack_j is opened at u || r. batch_open is r = [] with one
// column a stack.
int mercury_batch_open_stacked_impl(Ctx& c, const Fr* const* d_cols, const size_t* stack_lens, size_t nstacks,
                                    size_t width, const uint8_t* cms, const std::vector<F>& u,
                                    const std::vector<F>& r, host::Transcript& tr, std::vector<F>& vs,
                                    uint8_t proof_out[704]) {
  using namespace host;
  const size_t nv = width + r.size();
  const size_t n = (size_t)1 << nv;
  size_t ncols = 0, maxlen = 0;
  for (size_t j = 0; j < nstacks; ++j) {
    ncols += stack_lens[j];
    maxlen = std::max(maxlen, stack_lens[j]);
  }
  const size_t w1 = width / 2, b1 = (size_t)1 << w1, b2 = (size_t)1 << (width - w1);
  std::vector<F> u1(u.begin(), u.begin() + w1), u2(u.begin() + w1, u.end());
  Fr* work;
  const size_t words = b1 + b2 + ncols * b2 + ncols + nstacks + n;
  c.alloc(&work, 32 * words);
  struct Guard {
    Ctx& c;
    Fr* p;
    ~Guard() { cudaFreeAsync(p, c.stream); }
  } guard{c, work};
  Fr *eq1 = work, *eq2 = eq1 + b1, *h = eq2 + b2, *cv = h + ncols * b2, *w = cv + ncols, *fstar = w + nstacks;
  // The columns' addresses: stack after stack, then by (stack, slot), null past a
  // stack's end.
  std::vector<const Fr*> table(d_cols, d_cols + ncols);
  table.resize(ncols + nstacks * maxlen, nullptr);
  for (size_t j = 0, idx = 0; j < nstacks; ++j)
    for (size_t s = 0; s < stack_lens[j]; ++s) table[ncols + j * maxlen + s] = d_cols[idx++];
  const Fr** d_table = c.scratch[S_TMP5].as<const Fr*>(table.size());
  c.copy(d_table, table.data(), sizeof(Fr*) * table.size(), cudaMemcpyHostToDevice);
  build_eq_table(c, u1, eq1);
  build_eq_table(c, u2, eq2);
  for (size_t c0 = 0; c0 < ncols; c0 += 32768) {
    const unsigned cn = (unsigned)std::min<size_t>(32768, ncols - c0);
    launch_chained(c, k_row_dot, dim3(nb(b2 * 32, 256), cn), 256, 0, (const Fr* const*)(d_table + c0), (const Fr*)nullptr,
           (const Fr*)eq1, b1, b2, h + c0 * b2);
    launch_chained(c, k_dot, cn, 256, 0, (const Fr*)eq2, (const Fr*)(h + c0 * b2), b2, cv + c0);
  }
  tr.absorb_g1(T_COMMITMENT, cms, nstacks);  // (while the columns are evaluated)
  const std::vector<F> vals = read_frs(c, cv, ncols);
  vs.assign(nstacks, fzero());
  for (size_t j = 0, idx = 0; j < nstacks; ++j)
    for (size_t s = 0; s < stack_lens[j]; ++s, ++idx) {
      F e = fone();  // eq(r, s): variable i is bit i of the slot
      for (size_t i = 0; i < r.size(); ++i) e = fmul(e, (s >> i) & 1 ? r[i] : fsub(fone(), r[i]));
      vs[j] = fadd(vs[j], fmul(e, vals[idx]));
    }
  std::vector<F> point = u;
  point.insert(point.end(), r.begin(), r.end());
  std::vector<F> claim = point;
  claim.insert(claim.end(), vs.begin(), vs.end());
  tr.absorb(T_EVALUATION_CLAIM, claim);
  F rho = tr.challenge(T_MERCURY_BATCH);
  std::vector<F> wts(nstacks);
  F acc = fone();
  for (size_t i = 0; i < nstacks; ++i) {
    wts[i] = acc;
    acc = fmul(acc, rho);
  }
  // cm* = sum rho^j cm_j (crates/pcs/src/lib.rs:568-581). The commitments
  // are validated on their way to the device (status codes of the general
  // MSM); a few of them are summed on the host, where the sum's chain of 252
  // doublings runs many times faster than in one device thread (eight
  // commitments: about 0.2 ms against 2.2 ms), more through the device MSM.
  Affine* d_cms = c.scratch[S_BASES].as<Affine>(nstacks);
  upload_points(c, cms, nstacks, d_cms);
  c.copy(w, wts.data(), 32 * nstacks, cudaMemcpyHostToDevice);
  launch_chained(c, k_combine_stacked, nb(n, 256), 256, 0, (const Fr* const*)(d_table + ncols), (const Fr*)w, (int)nstacks, maxlen,
         (int)width, n, fstar);
  uint8_t cm_star[64];
  if (nstacks <= kHostMsmMax)
    host::g1::msm_small(cms, wts.data(), nstacks, cm_star);
  else
    msm_device(c, d_cms, nullptr, w, false, false, nstacks, nullptr, cm_star);
  F v;
  int st = mercury_open_impl(c, fstar, nv, cm_star, point, tr, v, proof_out);
  if (st) return st;
  F vstar = fzero();
  for (size_t i = 0; i < nstacks; ++i) vstar = fadd(vstar, fmul(wts[i], vs[i]));
  if (v != vstar) throw Error(APG_ERR_INTERNAL, "the combined value is not the combination of the values");
  return APG_OK;
}

}  // namespace apg
