// Kernel-level check of the digit-form contractions on general operands, against dot products
// in 128-bit floats on the CPU: two-level rows, columns and k with every order of the strides,
// outputs contiguous along either index, a second output, every kind of beta; planar complex
// products with both conjugations and either operand the larger; a pre-sliced B; both operands
// pre-sliced with runs of rows; and operands of which some blocks are refused by eight digits.
// Usage: forms_check; exits non-zero on a CUDA error, an error flag, or an entry outside its
// bound, which is that of digits_check.cu (four digits of a complex product: over both planes).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "../../cc4s_b200/csrc/split_gemm.cuh"
using namespace cc4s_b200;

namespace {
double rnd() { return (rand() / (double)RAND_MAX - 0.5) * std::pow(2.0, rand() % 5 - 2); }

// Strides of (outer, inner) of two indices of a dense tensor whose axes lie in memory in the
// order `perm` (last contiguous) of {x outer, x inner, y outer, y inner}.
struct Strides { int64_t s[4]; };
Strides strides(const int64_t (&d)[4], const int* perm) {
  Strides r;
  int64_t s = 1;
  for (int k = 3; k >= 0; --k) { r.s[perm[k]] = s; s *= d[perm[k]]; }
  return r;
}
View view(double* p, const Strides& s) {
  View v;
  v.p = p; v.s_ro = s.s[0]; v.s_ri = s.s[1]; v.s_co = s.s[2]; v.s_ci = s.s[3];
  return v;
}
int64_t off(const View& v, int64_t x, int64_t xi, int64_t y, int64_t yi) {
  return x / xi * v.s_ro + x % xi * v.s_ri + y / yi * v.s_co + y % yi * v.s_ci;
}

struct Dev {
  double* p;
  std::vector<double> h;
  explicit Dev(size_t n) : p(nullptr), h(n) {
    if (cudaMalloc(&p, n * 8) != cudaSuccess) exit(3);
    for (auto& x : h) x = rnd();
  }
  Dev(const Dev&) = delete;
  ~Dev() { cudaFree(p); }
  void up() { cudaMemcpy(p, h.data(), h.size() * 8, cudaMemcpyHostToDevice); }
  std::vector<double> down() const {
    std::vector<double> r(h.size());
    cudaMemcpy(r.data(), p, r.size() * 8, cudaMemcpyDeviceToHost);
    return r;
  }
};

SplitScratch ws;
int failures = 0, checks = 0;
void settled(const char* what) {
  const cudaError_t ce = cudaDeviceSynchronize();
  int herr = 0;
  cudaMemcpy(&herr, ws.error, 4, cudaMemcpyDeviceToHost);
  if (ce != cudaSuccess || herr) { printf("%s: %s errflag=%d\n", what, cudaGetErrorString(ce), herr); exit(1); }
}

// One real term: alpha sum_k a b with sum |a b| and the maxima; terms of a complex product add.
struct Sum {
  __float128 x = 0;
  double abs = 0, am = 0, bm = 0;
  int64_t k = 0;
  void add(double w, double a, double b) {
    x += (__float128)(w * a) * b;
    abs += std::fabs(w * a * b);
    am = std::fmax(am, std::fabs(a));
    bm = std::fmax(bm, std::fabs(b));
    ++k;
  }
  void check(const char* what, int digits, double alpha, double beta, double old, double got) {
    ++checks;
    const double ref = (double)(alpha * x + (__float128)beta * old);
    const double form = digits == 8 ? std::ldexp(abs, -53)
                                    : (2 * std::ldexp(1.0, -31) + std::ldexp(8.0, -30)) * 4 * am * bm;
    const double bound = std::fabs(alpha) * k * form +
                         std::ldexp(2 * std::fabs(alpha * (double)x) + 2 * std::fabs(beta * old), -52);
    if (!(std::fabs(got - ref) <= bound) && failures++ < 20)
      printf("%s digits=%d beta=%g: %.17g instead of %.17g, bound %.3g\n", what, digits, beta, got, ref, bound);
  }
};

const int PERMS[6][4] = {{0, 1, 2, 3}, {2, 3, 0, 1}, {2, 0, 3, 1}, {0, 2, 1, 3}, {3, 1, 2, 0}, {1, 3, 0, 2}};

// Real contractions: every pair of operand and output orders below, optionally a second
// output; graded: some rows of A fall along k while B rises, so that blocks are refused.
void real_views(int64_t Mo, int64_t Mi, int64_t No, int64_t Ni, int64_t Ko, int64_t Ki, bool packed_b) {
  const int64_t M = Mo * Mi, N = No * Ni, K = Ko * Ki;
  Dev A(M * K), B(K * N), C(M * N), C2(M * N);
  for (int q = 0; q < 6; ++q)
    for (int digits : {4, 8})
      for (double beta : {0.0, 1.0, 0.5}) {
        const bool two = (q + (digits == 8)) & 1, graded = q % 3 == 2;
        Contraction c;
        c.M = M; c.N = N; c.K = K; c.Mi = Mi; c.Ni = Ni; c.Ki = Ki;
        c.alpha = -0.75; c.beta = beta; c.digits = digits;
        c.A = view(A.p, strides({Mo, Mi, Ko, Ki}, PERMS[q]));
        c.B = view(B.p, strides({Ko, Ki, No, Ni}, PERMS[(q + 1) % 6]));
        c.C = view(C.p, strides({Mo, Mi, No, Ni}, PERMS[(q + 2) % 6]));
        if (two) c.C2 = view(C2.p, strides({Mo, Mi, No, Ni}, PERMS[(q + 3) % 6]));
        for (auto& x : A.h) x = rnd();
        for (auto& x : B.h) x = rnd();
        if (graded)
          for (int64_t k = 0; k < K; ++k) {
            const double w = std::pow(1e-8, K > 1 ? double(k) / (K - 1) : 0.0);
            for (int64_t m = 0; m < std::min<int64_t>(M, 64); ++m) A.h[off(c.A, m, Mi, k, Ki)] *= w;
            for (int64_t n = 0; n < N; ++n) B.h[off(c.B, k, Ki, n, Ni)] *= 1e-8 / w;
          }
        A.up(); B.up(); C.up(); C2.up();
        if (packed_b && split_single_panel(c)) {
          void* dst = nullptr;
          if (cudaMalloc(&dst, split_packed_b_bytes(c)) != cudaSuccess) exit(3);
          const SplitPackedB pb = split_pack_b(c, dst, 0);
          gemm_split_packed_b(c, pb, 0, ws);
          settled("packed B");
          cudaFree(dst);
        } else {
          gemm_split(c, 0, ws);
          settled("views");
        }
        const std::vector<double> r = C.down(), r2 = C2.down();
        for (int s = 0; s < 60; ++s) {
          const int64_t m = s < 2 ? s * (M - 1) : rand() % M, n = s < 2 ? s * (N - 1) : rand() % N;
          Sum x;
          for (int64_t k = 0; k < K; ++k) x.add(1.0, A.h[off(c.A, m, Mi, k, Ki)], B.h[off(c.B, k, Ki, n, Ni)]);
          const int64_t o = off(c.C, m, Mi, n, Ni);
          x.check("view", digits, c.alpha, beta, C.h[o], r[o]);
          if (two) {
            const int64_t o2 = off(c.C2, m, Mi, n, Ni);
            x.check("second output", digits, c.alpha, beta, C2.h[o2], r2[o2]);
          }
        }
        if (!two)
          for (size_t k = 0; k < r2.size(); ++k)
            if (r2[k] != C2.h[k]) { ++failures; break; }
      }
}

// Planar complex products; graded as above.
void complex_views(int64_t Mo, int64_t Mi, int64_t N, int64_t Ko, int64_t Ki) {
  const int64_t M = Mo * Mi, K = Ko * Ki;
  Dev A(2 * M * K), B(2 * K * N), C(2 * M * N), C2(2 * M * N);
  for (int q = 0; q < 4; ++q)
    for (int digits : {4, 8})
      for (double beta : {0.0, 1.0}) {
        const bool cA = q & 1, cB = q & 2, two = q == 1 || q == 2, graded = q >= 2;
        const double sA = cA ? -1.0 : 1.0, sB = cB ? -1.0 : 1.0;
        Contraction c;
        c.M = M; c.N = N; c.K = K; c.Mi = Mi; c.Ki = Ki;
        c.alpha = 1.5; c.beta = beta; c.digits = digits;
        c.A = view(A.p, strides({Mo, Mi, Ko, Ki}, PERMS[q]));
        c.B = view(B.p, strides({Ko, Ki, 1, N}, PERMS[q + 1]));
        c.C = view(C.p, strides({Mo, Mi, 1, N}, PERMS[q]));
        if (two) c.C2 = view(C2.p, strides({Mo, Mi, 1, N}, PERMS[q + 2]));
        for (auto& x : A.h) x = rnd();
        for (auto& x : B.h) x = rnd();
        for (int64_t k = 0; graded && k < K; ++k) {
          const double w = std::pow(1e-8, K > 1 ? double(k) / (K - 1) : 0.0);
          for (int pl = 0; pl < 2; ++pl) {
            for (int64_t m = 0; m < std::min<int64_t>(M, 64); ++m) A.h[pl * M * K + off(c.A, m, Mi, k, Ki)] *= w;
            for (int64_t n = 0; n < N; ++n) B.h[pl * K * N + off(c.B, k, Ki, n, N)] *= 1e-8 / w;
          }
        }
        A.up(); B.up(); C.up(); C2.up();
        gemm_split_complex(c, M * K, K * N, M * N, cA, cB, 0, ws);
        settled("complex");
        const std::vector<double> r = C.down(), r2 = C2.down();
        for (int s = 0; s < 60; ++s) {
          const int64_t m = s < 2 ? s * (M - 1) : rand() % M, n = s < 2 ? s * (N - 1) : rand() % N;
          for (int im = 0; im < 2; ++im) {
            Sum x;
            for (int64_t k = 0; k < K; ++k) {
              const double* a = &A.h[off(c.A, m, Mi, k, Ki)];
              const double* b = &B.h[off(c.B, k, Ki, n, N)];
              const double ai = sA * a[M * K], bi = sB * b[K * N];
              if (im) { x.add(1.0, *a, bi); x.add(1.0, ai, *b); }
              else { x.add(1.0, *a, *b); x.add(-1.0, ai, bi); }
            }
            const int64_t o = im * M * N + off(c.C, m, Mi, n, N);
            x.check("complex", digits, c.alpha, beta, C.h[o], r[o]);
            if (two) {
              const int64_t o2 = im * M * N + off(c.C2, m, Mi, n, N);
              x.check("complex, second output", digits, c.alpha, beta, C2.h[o2], r2[o2]);
            }
          }
        }
      }
}

// Both operands pre-sliced, rows taken in runs.
void runs(int64_t K) {
  const int64_t RA = 5 * 90, RB = 4 * 77 + 3;
  Dev A(RA * K), B(RB * K);
  A.up(); B.up();
  for (int digits : {4, 8})
    for (double beta : {0.0, 1.0}) {
      void *da, *db;
      int* word;
      cudaMalloc(&da, split_operand_bytes(RA, K, digits));
      cudaMalloc(&db, split_operand_bytes(RB, K, digits));
      cudaMalloc(&word, 8);
      // A's rows in two levels: row r at (r % 5) * 90 K + (r / 5) K
      const SplitOperand a = split_pack_operand(A.p, RA, 5, K, 90 * K, K, 1, da, 0, digits);
      const SplitOperand b = split_pack_operand(B.p, RB, 0, 0, K, K, 1, db, 0, digits);
      if (digits == 8) {
        split_refused(a, b, word, 0);
        int w = 1;
        cudaMemcpy(&w, word, 4, cudaMemcpyDeviceToHost);
        if (w) { printf("even operands refused\n"); ++failures; }
      }
      SplitRuns ar, br;
      ar.base = 7; ar.run = 70; ar.stride = 101;    // 4 runs of 70 rows
      br.base = 3; br.run = 77; br.stride = 77;     // adjacent runs
      Contraction c;
      c.M = 4 * 70; c.N = 4 * 77; c.K = K; c.alpha = 0.5; c.beta = beta; c.digits = digits;
      Dev C(c.M * c.N);
      C.up();
      c.C = rm(C.p, c.N);
      gemm_split_prepacked(c, a, ar, b, br, 0, ws);
      settled("runs");
      const std::vector<double> r = C.down();
      for (int s = 0; s < 300; ++s) {
        const int64_t m = s < 2 ? s * (c.M - 1) : rand() % c.M, n = s < 2 ? s * (c.N - 1) : rand() % c.N;
        const int64_t pa = ar.base + m / ar.run * ar.stride + m % ar.run, pb = br.base + n;
        Sum x;
        for (int64_t k = 0; k < K; ++k)
          x.add(1.0, A.h[(pa % 5) * 90 * K + pa / 5 * K + k], B.h[pb * K + k]);
        x.check("runs", digits, c.alpha, beta, C.h[m * c.N + n], r[m * c.N + n]);
      }
      cudaFree(da); cudaFree(db); cudaFree(word);
    }
}
}  // namespace

int main() {
  cudaMalloc(&ws.error, 8);
  cudaMemset(ws.error, 0, 8);
  ws.bytes = size_t(1) << 29;
  cudaMalloc(&ws.p, ws.bytes);
  ws.fp64.elems = 1 << 22;
  cudaMalloc(&ws.fp64.p, ws.fp64.elems * 8);
  srand(5);
  real_views(3, 50, 5, 29, 4, 33, false);     // ragged everywhere
  real_views(2, 64, 1, 64, 1, 64, false);     // whole tiles
  real_views(1, 130, 2, 40, 9, 331, false);   // split over k
  real_views(3, 50, 5, 29, 4, 33, true);
  complex_views(3, 30, 200, 5, 21);           // the second forms on A's side
  complex_views(5, 41, 70, 2, 50);            // on B's
  complex_views(1, 121, 121, 3, 700);         // split over k
  runs(96);
  runs(100);
  printf("%d checks, %d failures\n", checks, failures);
  return failures != 0;
}
