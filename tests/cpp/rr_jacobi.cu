// rrdev::jacobi on matrices from a file: count, then n and n x n doubles each; writes
// the eigenvalues and the eigenvectors (column j at n + n j) of each.  Arguments:
// input, output, 32 or 64 (the batched solver's block or the single one's).
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "common.cuh"
#include "rr_dev.cuh"

template <int NMAX, int NT>
__global__ void __launch_bounds__(NT) k_solve(const double *in, int n, double *out) {
  extern __shared__ double sm[];
  __shared__ sbdgb::rrdev::Scratch<NMAX, NT> work;
  const int nn = n * n;
  double *A = sm, *An = sm + nn, *V = sm + 2 * nn, *Vn = sm + 3 * nn;
  for (int t = threadIdx.x; t < nn; t += NT) {
    A[t] = in[t];
    V[t] = t % n == t / n ? 1.0 : 0.0;
  }
  __syncthreads();
  sbdgb::rrdev::jacobi<NMAX, NT>(n, A, An, V, Vn, work);
  __syncthreads();
  for (int t = threadIdx.x; t < nn; t += NT) {
    if (t < n) out[t] = A[t + n * t];
    out[n + t] = V[t];
  }
}

template <int NMAX, int NT>
void solve(const double *in, int n, double *out) {
  const size_t smem = 4 * sizeof(double) * n * n;
  SBDGB_CUDA(cudaFuncSetAttribute(k_solve<NMAX, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_solve<NMAX, NT><<<1, NT, smem>>>(in, n, out);
  SBDGB_CUDA(cudaGetLastError());
  SBDGB_CUDA(cudaDeviceSynchronize());
}

int main(int argc, char **argv) {
  if (argc != 4) return 2;
  const int nmax = std::atoi(argv[3]);
  FILE *f = std::fopen(argv[1], "rb"), *g = std::fopen(argv[2], "wb");
  if (!f || !g) return 2;
  double *d = nullptr;
  SBDGB_CUDA(cudaMalloc(&d, sizeof(double) * (2 * 64 * 64 + 64)));
  double x = 0.0;
  if (std::fread(&x, 8, 1, f) != 1) return 2;
  for (int i = (int)x; i > 0; --i) {
    if (std::fread(&x, 8, 1, f) != 1) return 2;
    const int n = (int)x;
    std::vector<double> a((size_t)n * n), out((size_t)n + (size_t)n * n);
    if (n < 1 || n > nmax || std::fread(a.data(), 8, a.size(), f) != a.size()) return 2;
    SBDGB_CUDA(cudaMemcpy(d, a.data(), 8 * a.size(), cudaMemcpyHostToDevice));
    if (nmax <= 32)
      solve<32, 256>(d, n, d + 64 * 64);
    else
      solve<64, 1024>(d, n, d + 64 * 64);
    SBDGB_CUDA(cudaMemcpy(out.data(), d + 64 * 64, 8 * out.size(), cudaMemcpyDeviceToHost));
    std::fwrite(out.data(), 8, out.size(), g);
  }
  std::fclose(f);
  std::fclose(g);
  cudaFree(d);
  return 0;
}
