// Kernel-level check of the FP64 tensor-pipe contraction (gemm) in its tile shapes against
// dot products in 128-bit floats on the CPU.
// Usage: gemm_check M N K batch transA transB; exits non-zero on a CUDA error or an entry
// outside K + 2 rounding errors of sum |a b| (the running sum is at most that, each of its
// K additions rounds once, the epilogue twice).
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "../../cc4s_b200/csrc/gemm_f64.cuh"
using namespace cc4s_b200;

int main(int argc, char** argv) {
  if (argc < 7) return 2;
  const int64_t M = atoll(argv[1]), N = atoll(argv[2]), K = atoll(argv[3]), B = atoll(argv[4]);
  const int tA = atoi(argv[5]), tB = atoi(argv[6]);
  std::vector<double> hA(M * K * B), hB(K * N * B), hC(M * N * B), r(M * N * B);
  srand(5);
  for (auto* h : {&hA, &hB, &hC})
    for (auto& x : *h) x = rand() / (double)RAND_MAX - 0.5;
  double *dA, *dB, *dC;
  GemmScratch gs; gs.elems = 1 << 22; cudaMalloc(&gs.p, gs.elems * 8);
  cudaMalloc(&dA, hA.size() * 8); cudaMalloc(&dB, hB.size() * 8); cudaMalloc(&dC, hC.size() * 8);
  cudaMemcpy(dA, hA.data(), hA.size() * 8, cudaMemcpyHostToDevice);
  cudaMemcpy(dB, hB.data(), hB.size() * 8, cudaMemcpyHostToDevice);
  for (double beta : {0.0, 1.0})
    for (int ct = 0; ct < 2; ++ct) {  // C stored row-major or transposed
      cudaMemcpy(dC, hC.data(), hC.size() * 8, cudaMemcpyHostToDevice);
      Contraction c; c.M = M; c.N = N; c.K = K; c.batch = B; c.alpha = -1.5; c.beta = beta;
      c.A = with_batch(tA ? tr(dA, M) : rm(dA, K), M * K);
      c.B = with_batch(tB ? tr(dB, K) : rm(dB, N), K * N);
      c.C = with_batch(ct ? tr(dC, M) : rm(dC, N), M * N);
      gemm(c, 0, gs);
      cudaMemcpy(r.data(), dC, r.size() * 8, cudaMemcpyDeviceToHost);
      const cudaError_t ce = cudaDeviceSynchronize();
      if (ce != cudaSuccess) { printf("%s\n", cudaGetErrorString(ce)); return 1; }
      double worst = 0;
      for (int64_t q = 0; q < 600; ++q) {
        const int64_t b = q % B;
        const int64_t m = q < 2 ? q * (M - 1) : (q * 7919) % M, n = q < 2 ? q * (N - 1) : (q * 104729) % N;
        __float128 x = 0;
        double a = 0;
        for (int64_t k = 0; k < K; ++k) {
          const double u = hA[b * M * K + (tA ? k * M + m : m * K + k)];
          const double v = hB[b * K * N + (tB ? n * K + k : k * N + n)];
          x += (__float128)u * v;
          a += std::fabs(u * v);
        }
        const int64_t at = b * M * N + (ct ? n * M + m : m * N + n);
        const double ref = (double)(-1.5 * x + beta * hC[at]);
        const double bound = (K + 2) * std::ldexp(1.5 * a + std::fabs(beta * hC[at]), -53);
        worst = std::fmax(worst, std::fabs(r[at] - ref) / bound);
      }
      if (!(worst <= 1.0)) { printf("beta=%g ct=%d: error %.3g of the bound\n", beta, ct, worst); return 1; }
      printf("beta=%g ct=%d ok: error %.3g of the bound\n", beta, ct, worst);
    }
  return 0;
}
