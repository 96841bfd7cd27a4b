// Products, squares and Montgomery reductions of the device field arithmetic:
// reads "<q|r> <count>", then count lines of two 64-digit hex values (each
// below the modulus), and prints per line a b / 2^256, a^2 / 2^256 and
// a / 2^256 as the device computes them.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../apogee-vm_gb300/csrc/field.cuh"

using namespace apg;

template <class C>
__global__ void k_ops(const Fe<C>* a, const Fe<C>* b, int n, Fe<C>* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[3 * i] = fe_mul(a[i], b[i]);
  out[3 * i + 1] = fe_sqr(a[i]);
  out[3 * i + 2] = fe_from_mont(a[i]);
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
  std::vector<Fe<C>> a(n), b(n), out(3 * (size_t)n);
  for (int i = 0; i < n; ++i)
    if (!read_hex(a[i].v) || !read_hex(b[i].v)) return 2;
  Fe<C>*da, *db, *dout;
  if (cudaMalloc(&da, 32 * (size_t)n) || cudaMalloc(&db, 32 * (size_t)n) || cudaMalloc(&dout, 96 * (size_t)n)) return 3;
  cudaMemcpy(da, a.data(), 32 * (size_t)n, cudaMemcpyHostToDevice);
  cudaMemcpy(db, b.data(), 32 * (size_t)n, cudaMemcpyHostToDevice);
  k_ops<C><<<(n + 127) / 128, 128>>>(da, db, n, dout);
  if (cudaMemcpy(out.data(), dout, 96 * (size_t)n, cudaMemcpyDeviceToHost) != cudaSuccess) return 4;
  for (size_t i = 0; i < out.size(); ++i) {
    for (int k = 7; k >= 0; --k) printf("%08x", out[i].v[k]);
    printf(i % 3 == 2 ? "\n" : " ");
  }
  return 0;
}

int main() {
  char f;
  int n;
  if (scanf(" %c %d", &f, &n) != 2 || n < 1 || n > 1 << 20) return 1;
  return f == 'q' ? run<FqConsts>(n) : run<FrConsts>(n);
}
