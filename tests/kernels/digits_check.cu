// Kernel-level check of the digit-form contractions (gemm_split with 4 and 7 digits)
// against dot products in 128-bit floats on the CPU.
// Usage: digits_check M N K transA transB; exits non-zero on a CUDA error, a bounded-wait
// error flag, an entry outside the bound, or a non-finite input that does not show.
//
// Bound, with a row of A below 2^ea and a column of B below 2^eb, D digits of 8 D - 2 bits:
// rounding the operands gives at most 2^-(8D-1) 2^(ea+eb) per product and operand; the
// digit products left out weigh 2^-12 2^(14 - 8 NG) each, fewer than 8 per k; the final
// rounding (beta = 1: of the sum too) 2^-52 of the value.  2^ea <= 2 amax, 2^eb <= 2 bmax.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "../../cc4s_b200/csrc/split_gemm.cuh"
using namespace cc4s_b200;

int main(int argc, char** argv) {
  if (argc < 6) return 2;
  const int64_t M = atoll(argv[1]), N = atoll(argv[2]), K = atoll(argv[3]);
  const int tA = atoi(argv[4]), tB = atoi(argv[5]);
  int* err; cudaMalloc(&err, 4); cudaMemset(err, 0, 4);
  SplitScratch ws; ws.bytes = size_t(1) << 30; cudaMalloc(&ws.p, ws.bytes); ws.error = err;
  std::vector<double> hA(M * K), hB(K * N), hC(M * N);
  srand(11);
  auto rnd = [] { return (rand() / (double)RAND_MAX - 0.5) * std::pow(2.0, rand() % 17 - 12); };
  for (auto& x : hA) x = rnd();
  for (auto& x : hB) x = rnd();
  for (auto& x : hC) x = rnd();
  double *A, *B, *C;
  cudaMalloc(&A, M * K * 8); cudaMalloc(&B, K * N * 8); cudaMalloc(&C, M * N * 8);
  auto at = [&](const std::vector<double>& h, bool t, int64_t rows, int64_t cols, int64_t r,
                int64_t c) { return t ? h[c * rows + r] : h[r * cols + c]; };
  for (int digits : {4, 7})
    for (double beta : {0.0, 1.0})
      for (int bad = 0; bad < 2; ++bad) {
        std::vector<double> a = hA;
        if (bad) a[tA ? (K - 1) * M + M / 2 : (M / 2) * K + K - 1] = bad ? HUGE_VAL : 0.0;
        cudaMemcpy(A, a.data(), M * K * 8, cudaMemcpyHostToDevice);
        cudaMemcpy(B, hB.data(), K * N * 8, cudaMemcpyHostToDevice);
        cudaMemcpy(C, hC.data(), M * N * 8, cudaMemcpyHostToDevice);
        Contraction c; c.M = M; c.N = N; c.K = K; c.alpha = -0.75; c.beta = beta; c.digits = digits;
        c.A = tA ? tr(A, M) : rm(A, K);
        c.B = tB ? tr(B, K) : rm(B, N);
        c.C = rm(C, N);
        gemm_split(c, 0, ws);
        const cudaError_t ce = cudaDeviceSynchronize();
        int herr = 0; cudaMemcpy(&herr, err, 4, cudaMemcpyDeviceToHost);
        if (ce != cudaSuccess || herr) { printf("%s errflag=%d\n", cudaGetErrorString(ce), herr); return 1; }
        std::vector<double> r(M * N);
        cudaMemcpy(r.data(), C, M * N * 8, cudaMemcpyDeviceToHost);
        double worst = 0;
        for (int64_t q = 0; q < 400; ++q) {  // corners and edges first, then a spread of entries
          const int64_t m = q == 0 ? 0 : q == 1 ? M - 1 : q < 20 ? M - 1 - (q % M) : (q * 7919) % M;
          const int64_t n = q == 0 ? 0 : q == 1 ? N - 1 : q < 20 ? N - 1 - (q % N) : (q * 104729) % N;
          const double got = r[m * N + n];
          if (bad && m == M / 2) {
            if (std::isfinite(got)) { printf("non-finite input lost\n"); return 1; }
            continue;
          }
          __float128 x = 0;
          double am = 0, bm = 0;
          for (int64_t k = 0; k < K; ++k) {
            const double p = at(a, tA, M, K, m, k), s = at(hB, tB, K, N, k, n);
            x += (__float128)p * s;
            am = std::fmax(am, std::fabs(p));
            bm = std::fmax(bm, std::fabs(s));
          }
          const double ref = (double)(-0.75 * x + beta * hC[m * N + n]);
          const int NG = digits == 7 ? 8 : 4;
          const double per_k = 2 * std::ldexp(1.0, -(8 * digits - 1)) + std::ldexp(8.0, 2 - 8 * NG);
          const double bound = 0.75 * K * per_k * 4 * am * bm +
                               std::ldexp(2 * std::fabs((double)x) + std::fabs(beta * hC[m * N + n]), -52);
          worst = std::fmax(worst, std::fabs(got - ref) / bound);
        }
        if (!(worst <= 1.0)) { printf("digits=%d beta=%g: error %.3g of the bound\n", digits, beta, worst); return 1; }
        printf("digits=%d beta=%g bad=%d errflag=0 error %.3g of the bound\n", digits, beta, bad, worst);
      }
  return 0;
}
