// Kernel-level check of the digit-form contractions (gemm_split with 4 and 8 digits)
// against dot products in 128-bit floats on the CPU, on operands with even rows, on graded
// ones (A falls and B rises along k by a factor of 1e6) and with an Inf in one row.
// Usage: digits_check M N K transA transB; exits non-zero on a CUDA error, a bounded-wait
// error flag, an entry outside the bound, a non-finite input that does not show, or
// even operands in eight digits that ran on the FP64 pipe (gemm()'s result bit by bit).
//
// Bounds.  Eight digits stand for FP64: |error| <= K 2^-53 sum_k |a_k b_k|, what an FP64
// accumulation is held to, whatever the rows look like.  Four digits, with a row of A below
// 2^ea and a column of B below 2^eb, 30 bits: rounding the operands gives at most
// 2^-31 2^(ea+eb) per product and operand; the digit products left out weigh
// 2^-12 2^(14 - 32) each, fewer than 8 per k; 2^ea <= 2 amax, 2^eb <= 2 bmax.  The final
// rounding adds 2^-52 of the value (beta = 1: of the sum too).
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "../../cc4s_b200/csrc/split_gemm.cuh"
using namespace cc4s_b200;

int main(int argc, char** argv) {
  if (argc < 6) return 2;
  const int64_t M = atoll(argv[1]), N = atoll(argv[2]), K = atoll(argv[3]);
  const int tA = atoi(argv[4]), tB = atoi(argv[5]);
  int* err; cudaMalloc(&err, 4); cudaMemset(err, 0, 4);
  SplitScratch ws; ws.bytes = size_t(1) << 30; cudaMalloc(&ws.p, ws.bytes); ws.error = err;
  ws.fp64.elems = 1 << 22; cudaMalloc(&ws.fp64.p, ws.fp64.elems * 8);
  std::vector<double> hA(M * K), hB(K * N), hC(M * N);
  srand(11);
  auto rnd = [] { return (rand() / (double)RAND_MAX - 0.5) * std::pow(2.0, rand() % 5 - 2); };
  for (auto& x : hA) x = rnd();
  for (auto& x : hB) x = rnd();
  for (auto& x : hC) x = rnd();
  double *A, *B, *C;
  cudaMalloc(&A, M * K * 8); cudaMalloc(&B, K * N * 8); cudaMalloc(&C, M * N * 8);
  auto ia = [&](int64_t m, int64_t k) { return tA ? k * M + m : m * K + k; };
  auto ib = [&](int64_t k, int64_t n) { return tB ? n * K + k : k * N + n; };
  enum { EVEN, GRADED, INFINITE };
  for (int digits : {4, 8}) {  // the k ranges of the launch, and S32 spans of a tile
    const int tn = digits == 8 ? 64 : 128;
    const int parts = split_k_parts((M + 127) / 128 * ((N + tn - 1) / tn), M, N, (K + 31) / 32 * 32, digits);
    printf("digits=%d parts=%d spans=%ld\n", digits, parts, (long)((K + parts * 16384 - 1) / (parts * 16384)));
  }
  for (int digits : {4, 8})
    for (double beta : {0.0, 1.0})
      for (int kind : {EVEN, GRADED, INFINITE}) {
        std::vector<double> a = hA, b = hB;
        if (kind == INFINITE) a[ia(M / 2, K - 1)] = HUGE_VAL;
        for (int64_t k = 0; kind == GRADED && k < K; ++k) {
          const double w = std::pow(1e-6, K > 1 ? double(k) / (K - 1) : 0.0);
          for (int64_t m = 0; m < M; ++m) a[ia(m, k)] *= w;
          for (int64_t n = 0; n < N; ++n) b[ib(k, n)] *= 1e-6 / w;
        }
        cudaMemcpy(A, a.data(), M * K * 8, cudaMemcpyHostToDevice);
        cudaMemcpy(B, b.data(), K * N * 8, cudaMemcpyHostToDevice);
        Contraction c; c.M = M; c.N = N; c.K = K; c.alpha = -0.75; c.beta = beta; c.digits = digits;
        c.A = tA ? tr(A, M) : rm(A, K);
        c.B = tB ? tr(B, K) : rm(B, N);
        c.C = rm(C, N);
        std::vector<double> r(M * N), pipe(M * N);
        for (int route = 0; route < 2; ++route) {
          cudaMemcpy(C, hC.data(), M * N * 8, cudaMemcpyHostToDevice);
          if (route) gemm_split(c, 0, ws);
          else gemm(c, 0, ws.fp64);
          const cudaError_t ce = cudaDeviceSynchronize();
          int herr = 0; cudaMemcpy(&herr, err, 4, cudaMemcpyDeviceToHost);
          if (ce != cudaSuccess || herr) { printf("%s errflag=%d\n", cudaGetErrorString(ce), herr); return 1; }
          cudaMemcpy(route ? r.data() : pipe.data(), C, M * N * 8, cudaMemcpyDeviceToHost);
        }
        const bool same = !std::memcmp(r.data(), pipe.data(), M * N * 8);
        if (digits == 8 && K >= 64 && kind == EVEN && same) {
          printf("kind %d ran on the wrong kernel\n", kind);
          return 1;
        }
        double worst = 0;
        for (int64_t q = 0; q < 400; ++q) {  // corners and edges first, then a spread of entries
          const int64_t m = q == 0 ? 0 : q == 1 ? M - 1 : q < 20 ? M - 1 - (q % M) : (q * 7919) % M;
          const int64_t n = q == 0 ? 0 : q == 1 ? N - 1 : q < 20 ? N - 1 - (q % N) : (q * 104729) % N;
          const double got = r[m * N + n];
          if (kind == INFINITE && m == M / 2) {
            if (std::isfinite(got)) { printf("non-finite input lost\n"); return 1; }
            continue;
          }
          __float128 x = 0;
          double am = 0, bm = 0, sum = 0;
          for (int64_t k = 0; k < K; ++k) {
            const double p = a[ia(m, k)], s = b[ib(k, n)];
            x += (__float128)p * s;
            sum += std::fabs(p * s);
            am = std::fmax(am, std::fabs(p));
            bm = std::fmax(bm, std::fabs(s));
          }
          const double ref = (double)(-0.75 * x + beta * hC[m * N + n]);
          const double form = digits == 8 ? std::ldexp(sum, -53)
                                          : (2 * std::ldexp(1.0, -31) + std::ldexp(8.0, 2 - 32)) * 4 * am * bm;
          const double bound = 0.75 * K * form +
                               std::ldexp(2 * std::fabs((double)x) + std::fabs(beta * hC[m * N + n]), -52);
          worst = std::fmax(worst, std::fabs(got - ref) / bound);
        }
        if (!(worst <= 1.0)) { printf("digits=%d beta=%g kind=%d: error %.3g of the bound\n", digits, beta, kind, worst); return 1; }
        printf("digits=%d beta=%g kind=%d errflag=0 error %.3g of the bound\n", digits, beta, kind, worst);
      }
  return 0;
}
