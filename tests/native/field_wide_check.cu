// Unreduced sums of products and their one reduction (wide_mac, fe_from_wide):
// reads "<q|r> <count>", then count times a number of products k (at most
// kWideProducts) and k pairs of 64-digit hex values below the modulus, and prints
// a line each: (sum of the products) / 2^256 as the device computes it.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../apogee-vm_gb300/csrc/field.cuh"

using namespace apg;

template <class C>
__global__ void k_sums(const Fe<C>* ab, const int* counts, int n, Fe<C>* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  FeWide<C> w = wide_zero<C>();
  for (int j = 0; j < counts[i]; ++j)
    wide_mac(w, ab[2 * (i * kWideProducts + j)], ab[2 * (i * kWideProducts + j) + 1]);
  out[i] = fe_from_wide(w);
}

static bool read_hex(uint32_t w[8]) {
  char s[80];
  if (scanf("%72s", s) != 1) return false;
  for (int k = 0; k < 8; ++k) {
    char part[9] = {0};
    for (int j = 0; j < 8; ++j) part[j] = s[8 * (7 - k) + j];
    w[k] = (uint32_t)strtoul(part, nullptr, 16);
  }
  return true;
}

template <class C>
static int run(int n) {
  std::vector<Fe<C>> ab(2 * (size_t)n * kWideProducts), out(n);
  std::vector<int> counts(n);
  for (int i = 0; i < n; ++i) {
    if (scanf("%d", &counts[i]) != 1 || counts[i] < 0 || counts[i] > kWideProducts) return 2;
    for (int j = 0; j < 2 * counts[i]; ++j)
      if (!read_hex(ab[2 * (size_t)i * kWideProducts + j].v)) return 2;
  }
  Fe<C>*dab, *dout;
  int* dcounts;
  if (cudaMalloc(&dab, ab.size() * 32) || cudaMalloc(&dout, 32 * (size_t)n) || cudaMalloc(&dcounts, 4 * (size_t)n)) return 3;
  cudaMemcpy(dab, ab.data(), ab.size() * 32, cudaMemcpyHostToDevice);
  cudaMemcpy(dcounts, counts.data(), 4 * (size_t)n, cudaMemcpyHostToDevice);
  k_sums<C><<<(n + 127) / 128, 128>>>(dab, dcounts, n, dout);
  if (cudaMemcpy(out.data(), dout, 32 * (size_t)n, cudaMemcpyDeviceToHost) != cudaSuccess) return 4;
  for (const auto& o : out) {
    for (int k = 7; k >= 0; --k) printf("%08x", o.v[k]);
    printf("\n");
  }
  return 0;
}

int main() {
  char f;
  int n;
  if (scanf(" %c %d", &f, &n) != 2 || n < 1 || n > 1 << 16) return 1;
  return f == 'q' ? run<FqConsts>(n) : run<FrConsts>(n);
}
