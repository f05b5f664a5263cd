// TEST INFRASTRUCTURE ONLY: plain-loop CPU emulation of the device operations
// declared in cc4s_b200/csrc/ops.h and gemm_f64.cuh.
//
// It is linked with the product's schedule and driver sources into a separate
// test library (tests/emu/_build/libcc4s_emu.so) so that the index and stride
// bookkeeping of every contraction can be checked against the oracle on a
// machine without a GPU.  The product library never contains this file.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../cc4s_b200/csrc/ops.h"
#include "../../cc4s_b200/csrc/split_gemm.cuh"

namespace cc4s_b200 {

namespace {
struct Ax {
  int64_t inner, so, si;
  int64_t off(int64_t x) const { return (x / inner) * so + (x % inner) * si; }
};
Ax ax(int64_t inner, int64_t so, int64_t si) { return Ax{inner > 0 ? inner : 1, so, si}; }
uint64_t g_gemm = 0, g_ops = 0;
}  // namespace

uint64_t gemm_launch_count() { return g_gemm; }

void gemm(const Contraction& g, cudaStream_t, const GemmScratch&) {
  ++g_gemm;
  if (g.M <= 0 || g.N <= 0 || g.batch <= 0) return;
  const int64_t Mi = g.Mi > 0 ? g.Mi : g.M, Ni = g.Ni > 0 ? g.Ni : g.N;
  const int64_t Ki = g.Ki > 0 ? g.Ki : std::max<int64_t>(g.K, 1), Bi = g.Bi > 0 ? g.Bi : g.batch;
  Ax Am = ax(Mi, g.A.s_ro, g.A.s_ri), Ak = ax(Ki, g.A.s_co, g.A.s_ci);
  Ax Bk = ax(Ki, g.B.s_ro, g.B.s_ri), Bn = ax(Ni, g.B.s_co, g.B.s_ci);
  Ax Cm = ax(Mi, g.C.s_ro, g.C.s_ri), Cn = ax(Ni, g.C.s_co, g.C.s_ci);
  Ax C2m = ax(Mi, g.C2.s_ro, g.C2.s_ri), C2n = ax(Ni, g.C2.s_co, g.C2.s_ci);
  Ax Ab = ax(Bi, g.A.s_bo, g.A.s_bi), Bb = ax(Bi, g.B.s_bo, g.B.s_bi);
  Ax Cb = ax(Bi, g.C.s_bo, g.C.s_bi), C2b = ax(Bi, g.C2.s_bo, g.C2.s_bi);
  std::vector<int64_t> ak(g.K), bk(g.K);
  for (int64_t k = 0; k < g.K; ++k) { ak[k] = Ak.off(k); bk[k] = Bk.off(k); }
  for (int64_t b = 0; b < g.batch; ++b) {
    const double* A = g.A.p ? g.A.p + Ab.off(b) : nullptr;
    const double* B = g.B.p ? g.B.p + Bb.off(b) : nullptr;
    for (int64_t m = 0; m < g.M; ++m) {
      const int64_t am = Am.off(m);
      for (int64_t n = 0; n < g.N; ++n) {
        if (g.only && !g.only[b * g.only_bs + (m / 64) * g.only_ld + n / 64]) continue;
        const int64_t bn = Bn.off(n);
        double s = 0.0;
        for (int64_t k = 0; k < g.K; ++k) s += A[am + ak[k]] * B[bk[k] + bn];
        const double v = g.alpha * s;
        double* c = g.C.p + Cb.off(b) + Cm.off(m) + Cn.off(n);
        *c = g.beta != 0.0 ? v + g.beta * *c : v;
        if (g.C2.p) {
          double* c2 = g.C2.p + C2b.off(b) + C2m.off(m) + C2n.off(n);
          *c2 = g.beta != 0.0 ? v + g.beta * *c2 : v;
        }
      }
    }
  }
}

// Emulation of the digit-form contraction: the same row/column scaling, balanced
// base-256 digits and digit products (p + q < 4 of four digits, p + q < 8 of eight), each
// weight summed exactly as on the device, and the same blocks refused by eight digits.
static uint64_t g_split = 0, g_pack = 0;
// Test controls: every eligible FP64 contraction in the digit form, and the n-th digit
// contraction from now (0: the next) recording an expired wait.
static int g_force_digits = 0, g_fail_in = -1;
static uint64_t g_refused = 0;
extern "C" void emu_force_digits(int on) { g_force_digits = on; }
extern "C" void emu_fail_split_in(int n) { g_fail_in = n; }
extern "C" uint64_t emu_split_count() { return g_split; }
bool digits8_pays(const Contraction& c, bool cplx) {
  return g_force_digits && c.batch == 1 && c.M >= 64 && c.N >= 64 && c.K * (cplx ? 2 : 1) >= 64;
}
uint64_t split_launch_count() { return g_split; }
uint64_t split_pack_launch_count() { return g_pack; }
size_t gemm_split_scratch_bytes(const Contraction& g) { return size_t(g.digits) * (g.M + g.N) * g.K; }

extern "C" uint64_t emu_refused_count() { return g_refused; }

// The profiles of split_gemm.cuh: rows [R][K] -> [ceil(R / 64)][K].
static std::vector<float> profile(const std::vector<std::vector<double>>& rows, int64_t K) {
  const int64_t R = rows.size(), nI = (R + 63) / 64;
  std::vector<float> p(nI * K);
  for (int64_t I = 0; I < nI; ++I) {
    std::vector<double> least(K, 1.0);
    bool odd = false;
    for (int64_t g0 = 64 * I; g0 < std::min(R, 64 * I + 64); g0 += 8) {
      std::vector<double> sum(K, 0.0);
      int live = 0;
      for (int64_t r = g0; r < std::min(R, g0 + 8); ++r) {
        double m = 0.0;
        bool finite = true;
        for (double v : rows[r]) {
          finite = finite && std::isfinite(v);
          m = std::max(m, std::fabs(v));
        }
        if (!finite) { odd = true; continue; }
        if (m == 0.0) continue;
        int e;
        std::frexp(m, &e);
        odd = odd || std::abs(e) > kSplitMaxExponent;
        ++live;
        for (int64_t k = 0; k < K; ++k) sum[k] += std::ldexp(std::fabs(rows[r][k]), -e);
      }
      for (int64_t k = 0; live && k < K; ++k) least[k] = std::min(least[k], sum[k] / live);
    }
    for (int64_t k = 0; k < K; ++k) p[I * K + k] = odd ? NAN : static_cast<float>(least[k]);
  }
  return p;
}
// The blocks that eight digits refuse.
static std::vector<unsigned char> refused(const std::vector<std::vector<double>>& A,
                                          const std::vector<std::vector<double>>& B, int64_t K) {
  const std::vector<float> a = profile(A, K), b = profile(B, K);
  const int64_t nI = a.size() / K, nJ = b.size() / K;
  std::vector<unsigned char> map(nI * nJ);
  for (int64_t I = 0; I < nI; ++I)
    for (int64_t J = 0; J < nJ; ++J) {
      double v = 0.0;
      for (int64_t k = 0; k < K; ++k) v += double(a[I * K + k]) * b[J * K + k];
      map[I * nJ + J] = !(v >= split_profile_least(K));
    }
  return map;
}

void gemm_split(const Contraction& g, cudaStream_t s, SplitScratch& ws) {
  ++g_split;
  if (g_fail_in >= 0 && g_fail_in-- == 0) {
    *ws.error = 1;
    return;
  }
  g_pack += 2;  // the device slices both operands together (two launches)
  const int64_t Mi = g.Mi > 0 ? g.Mi : g.M, Ni = g.Ni > 0 ? g.Ni : g.N;
  const int64_t Ki = g.Ki > 0 ? g.Ki : std::max<int64_t>(g.K, 1);
  Ax Am = ax(Mi, g.A.s_ro, g.A.s_ri), Ak = ax(Ki, g.A.s_co, g.A.s_ci);
  Ax Bk = ax(Ki, g.B.s_ro, g.B.s_ri), Bn = ax(Ni, g.B.s_co, g.B.s_ci);
  Ax Cm = ax(Mi, g.C.s_ro, g.C.s_ri), Cn = ax(Ni, g.C.s_co, g.C.s_ci);
  Ax C2m = ax(Mi, g.C2.s_ro, g.C2.s_ri), C2n = ax(Ni, g.C2.s_co, g.C2.s_ci);
  const int D = g.digits == 8 ? 8 : 4, NG = D;
  using Digits = std::vector<std::vector<double>>;  // [digit][k]
  auto split = [&](const std::vector<double>& x, Digits& s, int& e) {
    double m = 0.0;
    for (double v : x) m = std::max(m, std::fabs(v));
    e = 0;
    if (m > 0.0) std::frexp(m, &e);
    s.assign(D, std::vector<double>(x.size(), 0.0));
    for (size_t k = 0; k < x.size(); ++k) {
      long long X = std::llrint(std::ldexp(x[k], 8 * D - 2 - e));
      for (int q = D - 1; q > 0; --q) {
        const auto d = static_cast<int8_t>(X & 255);
        s[q][k] = d;
        X = (X - d) >> 8;
      }
      s[0][k] = static_cast<double>(X);
    }
  };
  std::vector<Digits> as(g.M), bs(g.N);
  std::vector<int> ea(g.M), eb(g.N);
  std::vector<std::vector<double>> Ar(g.M, std::vector<double>(g.K)), Br(g.N, Ar[0]);
  for (int64_t m = 0; m < g.M; ++m) {
    for (int64_t k = 0; k < g.K; ++k) Ar[m][k] = g.A.p[Am.off(m) + Ak.off(k)];
    split(Ar[m], as[m], ea[m]);
  }
  for (int64_t n = 0; n < g.N; ++n) {
    for (int64_t k = 0; k < g.K; ++k) Br[n][k] = g.B.p[Bk.off(k) + Bn.off(n)];
    split(Br[n], bs[n], eb[n]);
  }
  std::vector<unsigned char> map((g.M + 63) / 64 * ((g.N + 63) / 64), 0);
  if (D == 8) map = refused(Ar, Br, g.K);
  for (int64_t m = 0; m < g.M; ++m)
    for (int64_t n = 0; n < g.N; ++n) {
      if (map[(m / 64) * ((g.N + 63) / 64) + n / 64]) continue;
      double sum = 0.0;
      for (int w = NG - 1; w >= 0; --w) {  // smallest weight first
        double grp = 0.0;
        for (int pa = std::max(0, w - D + 1); pa <= std::min(w, D - 1); ++pa) {
          const auto& x = as[m][pa];
          const auto& y = bs[n][w - pa];
          for (int64_t k = 0; k < g.K; ++k) grp += x[k] * y[k];
        }
        sum += std::ldexp(grp, -12 - 8 * w);
      }
      const double v = g.alpha * std::ldexp(sum, ea[m] + eb[n]);
      double* c = g.C.p + Cm.off(m) + Cn.off(n);
      *c = g.beta != 0.0 ? v + g.beta * *c : v;
      if (g.C2.p) {
        double* c2 = g.C2.p + C2m.off(m) + C2n.off(n);
        *c2 = g.beta != 0.0 ? v + g.beta * *c2 : v;
      }
    }
  if (std::count(map.begin(), map.end(), 0) < static_cast<int64_t>(map.size())) {
    ++g_refused;
    Contraction h = g;
    h.only = map.data();
    h.only_ld = (g.N + 63) / 64;
    gemm(h, s, ws.fp64);
  }
}

// The complex form: two real contractions over the planes side by side along k.
size_t gemm_split_complex_scratch_bytes(const Contraction& g) { return 4 * gemm_split_scratch_bytes(g); }
void gemm_split_complex(const Contraction& g, int64_t a_im, int64_t b_im, int64_t c_im, bool conjA,
                        bool conjB, cudaStream_t s, SplitScratch& ws) {
  const double sA = conjA ? -1.0 : 1.0, sB = conjB ? -1.0 : 1.0;
  const int64_t Mi = g.Mi > 0 ? g.Mi : g.M, Ni = g.Ni > 0 ? g.Ni : g.N, K = g.K;
  const int64_t Ki = g.Ki > 0 ? g.Ki : std::max<int64_t>(K, 1);
  const Ax Am = ax(Mi, g.A.s_ro, g.A.s_ri), Ak = ax(Ki, g.A.s_co, g.A.s_ci);
  const Ax Bk = ax(Ki, g.B.s_ro, g.B.s_ri), Bn = ax(Ni, g.B.s_co, g.B.s_ci);
  for (int part = 0; part < 2; ++part) {  // [Ar | Ai] on [Br ; -sA sB Bi] or [sB Bi ; sA Br]
    std::vector<double> A(g.M * 2 * K), B(2 * K * g.N);
    for (int64_t m = 0; m < g.M; ++m)
      for (int64_t k = 0; k < K; ++k)
        for (int h = 0; h < 2; ++h)
          A[m * 2 * K + h * K + k] = g.A.p[Am.off(m) + Ak.off(k) + h * a_im];
    for (int64_t n = 0; n < g.N; ++n)
      for (int64_t k = 0; k < K; ++k)
        for (int h = 0; h < 2; ++h) {
          const double w = part == 0 ? (h ? -sA * sB : 1.0) : (h ? sA : sB);
          B[n * 2 * K + h * K + k] = w * g.B.p[Bk.off(k) + Bn.off(n) + (h != part ? b_im : 0)];
        }
    Contraction c = g;
    c.K = 2 * K; c.Ki = 0;
    c.A.p = A.data(); c.A.s_ro = Mi * 2 * K; c.A.s_ri = 2 * K; c.A.s_co = 0; c.A.s_ci = 1;
    c.B.p = B.data(); c.B.s_ro = 0; c.B.s_ri = 1; c.B.s_co = Ni * 2 * K; c.B.s_ci = 2 * K;
    if (part) {
      c.C.p += c_im;
      if (c.C2.p) c.C2.p += c_im;
    }
    gemm_split(c, s, ws);
  }
}

// Pre-packed B: the emulation keeps a dense copy B[n][k] of the operand's values
// and slices it again in gemm_split (same values, same slices).
size_t split_packed_b_bytes(const Contraction& g) { return size_t(g.N) * g.K * 8 + 64; }
size_t split_scratch_bytes_packed_b(const Contraction& g) { return size_t(g.digits) * g.M * g.K; }
bool split_single_panel(const Contraction& g) { return g.batch == 1; }

SplitPackedB split_pack_b(const Contraction& g, void* dst, cudaStream_t) {
  const int64_t Ni = g.Ni > 0 ? g.Ni : g.N, Ki = g.Ki > 0 ? g.Ki : std::max<int64_t>(g.K, 1);
  Ax Bk = ax(Ki, g.B.s_ro, g.B.s_ri), Bn = ax(Ni, g.B.s_co, g.B.s_ci);
  double* d = static_cast<double*>(dst);
  for (int64_t n = 0; n < g.N; ++n)
    for (int64_t k = 0; k < g.K; ++k) d[n * g.K + k] = g.B.p[Bk.off(k) + Bn.off(n)];
  SplitPackedB b;
  b.slices = dst; b.N = g.N; b.K = g.K; b.Np = g.N; b.Kp = g.K; b.digits = g.digits;
  g_pack += 2;
  return b;
}

void gemm_split_packed_b(const Contraction& g, const SplitPackedB& b, cudaStream_t s,
                         SplitScratch& ws) {
  if (b.N != g.N || b.K != g.K || b.digits != g.digits) throw Error(ERR_INVALID_ARGUMENT, "pre-packed B of another shape");
  const int64_t Ni = g.Ni > 0 ? g.Ni : g.N, Ki = g.Ki > 0 ? g.Ki : std::max<int64_t>(g.K, 1);
  Contraction h = g;   // B(k, n) = copy[n * K + k] in the contraction's two-level k and n
  h.B.p = static_cast<double*>(b.slices);
  h.B.s_ro = Ki; h.B.s_ri = 1; h.B.s_co = Ni * g.K; h.B.s_ci = g.K;
  gemm_split(h, s, ws);
}

// Sliced operands: the emulation keeps the rows as a dense copy [R][K] and slices the
// rows a contraction reads again in gemm_split (same rows, same slices).
size_t split_operand_bytes(int64_t R, int64_t K, int) { return size_t(R) * K * 8 + 64; }

SplitOperand split_pack_operand(const double* src, int64_t R, int64_t Ri, int64_t s_ro,
                                int64_t s_ri, int64_t K, int64_t s_k, void* dst, cudaStream_t,
                                int digits) {
  if (R <= 0 || K <= 0) throw Error(ERR_BAD_SHAPE, "split_pack_operand: empty operand");
  Ax r = ax(Ri > 0 ? Ri : R, s_ro, s_ri);
  double* d = static_cast<double*>(dst);
  for (int64_t i = 0; i < R; ++i)
    for (int64_t k = 0; k < K; ++k) d[i * K + k] = src[r.off(i) + k * s_k];
  SplitOperand o;
  o.slices = dst; o.R = R; o.K = K; o.Rp = R; o.Kp = K; o.digits = digits;
  g_pack += 2;
  return o;
}

void split_refused(const SplitOperand& A, const SplitOperand& B, int* word, cudaStream_t) {
  auto rows = [](const SplitOperand& o) {
    const double* d = static_cast<const double*>(o.slices);
    std::vector<std::vector<double>> r;
    for (int64_t i = 0; i < o.R; ++i) r.emplace_back(d + i * o.K, d + (i + 1) * o.K);
    return r;
  };
  const std::vector<unsigned char> map = refused(rows(A), rows(B), A.K);
  std::memset(word, 0, 8);
  *word = std::count(map.begin(), map.end(), 0) < static_cast<int64_t>(map.size());
}

void gemm_split_prepacked(const Contraction& g, const SplitOperand& A, const SplitRuns& ar,
                          const SplitOperand& B, const SplitRuns& br, cudaStream_t s,
                          SplitScratch& ws) {
  if (g.M <= 0 || g.N <= 0) return;
  if (A.K != g.K || B.K != g.K || A.digits != B.digits)
    throw Error(ERR_INVALID_ARGUMENT, "gemm_split_prepacked: operands of another K");
  const int64_t K = g.K;
  auto rows = [&](const SplitOperand& o, const SplitRuns& r, int64_t X) {
    if (r.run <= 0) throw Error(ERR_INVALID_ARGUMENT, "gemm_split_prepacked: bad runs");
    std::vector<double> d(size_t(X) * K);
    const double* src = static_cast<const double*>(o.slices);
    for (int64_t x = 0; x < X; ++x) {
      const int64_t pr = r.base + (x / r.run) * r.stride + x % r.run;
      if (pr < 0 || pr >= o.R)
        throw Error(ERR_INVALID_ARGUMENT, "gemm_split_prepacked: runs leave the operand");
      for (int64_t k = 0; k < K; ++k) d[x * K + k] = src[pr * K + k];
    }
    return d;
  };
  std::vector<double> Ad = rows(A, ar, g.M), Bd = rows(B, br, g.N);
  g_pack -= 2;  // nothing is sliced here on the device (gemm_split below counts two)
  const int64_t Mi = g.Mi > 0 ? g.Mi : g.M, Ni = g.Ni > 0 ? g.Ni : g.N;
  Contraction h = g;
  h.Ki = 0;
  h.digits = A.digits;
  h.A.p = Ad.data(); h.A.s_ro = Mi * K; h.A.s_ri = K; h.A.s_co = 0; h.A.s_ci = 1;
  h.B.p = Bd.data(); h.B.s_ro = 0; h.B.s_ri = 1; h.B.s_co = Ni * K; h.B.s_ci = K;
  gemm_split(h, s, ws);
}

// Plain-loop stand-in for the allocation-free energy entry (host pointers).
int energy_noalloc(const double* T1, const double* T2, const double* V, int64_t o, int64_t v,
                   int cplx, double* out, cudaStream_t, const char** err) {
  if (!T1 || !T2 || !V || !out) { *err = "null pointer"; return ERR_INVALID_ARGUMENT; }
  if (o <= 0 || v <= 0) { *err = "No and Nv must be positive"; return ERR_BAD_SHAPE; }
  if (o * o > 65536) { *err = "No too large"; return ERR_BAD_SHAPE; }
  double acc[4] = {0, 0, 0, 0};
  for (int64_t j = 0; j < o; ++j)
    for (int64_t i = 0; i < o; ++i)
      for (int64_t b = 0; b < v; ++b)
        for (int64_t a = 0; a < v; ++a) {
          const int64_t e = a + v * (b + v * (i + o * j)), ex = b + v * (a + v * (i + o * j));
          const int64_t ai = a + v * i, bj = b + v * j;
          if (!cplx) {
            const double x = T2[e] + T1[ai] * T1[bj];
            acc[0] += x * V[e];
            acc[1] += x * V[ex];
          } else {
            const double xr = T2[2 * e] + T1[2 * ai] * T1[2 * bj] - T1[2 * ai + 1] * T1[2 * bj + 1];
            const double xi = T2[2 * e + 1] + T1[2 * ai] * T1[2 * bj + 1] + T1[2 * ai + 1] * T1[2 * bj];
            acc[0] += xr * V[2 * e] + xi * V[2 * e + 1];
            acc[1] += xr * V[2 * ex] + xi * V[2 * ex + 1];
            acc[2] += xi * V[2 * e] - xr * V[2 * e + 1];
            acc[3] += xi * V[2 * ex] - xr * V[2 * ex + 1];
          }
        }
  out[0] = 2 * acc[0]; out[1] = -acc[1]; out[2] = 2 * acc[2]; out[3] = -acc[3];
  return OK;
}

namespace ops {

// Test controls: single allocations of more than `bytes`, or all live ones together beyond
// `total`, find no memory (0: no limit).
static size_t g_alloc_limit = 0, g_total_limit = 0, g_live = 0, g_peak = 0;
static uint64_t g_alloc_failures = 0;
extern "C" void emu_alloc_limit(size_t bytes, size_t total) {
  g_alloc_limit = bytes;
  g_total_limit = total;
}
extern "C" uint64_t emu_alloc_failures() { return g_alloc_failures; }
extern "C" size_t emu_live_bytes() { return g_live; }
extern "C" size_t emu_peak_bytes(int reset) {
  const size_t p = g_peak;
  if (reset) g_peak = g_live;
  return p;
}

double* alloc(size_t elems) {  // the size in a header of 64 bytes
  const size_t bytes = std::max<size_t>(elems, 1) * sizeof(double);
  void* p = nullptr;
  if (!(g_alloc_limit && bytes > g_alloc_limit) && !(g_total_limit && g_live + bytes > g_total_limit))
    p = std::calloc(bytes + 64, 1);
  if (!p) {
    ++g_alloc_failures;
    throw Error(ERR_OUT_OF_MEMORY, "host allocation failed");
  }
  *static_cast<size_t*>(p) = bytes;
  g_live += bytes;
  g_peak = std::max(g_peak, g_live);
  return static_cast<double*>(p) + 8;
}
void release(void* p) {
  if (!p) return;
  size_t* h = static_cast<size_t*>(p) - 8;
  g_live -= *h;
  std::free(h);
}
void zero(double* p, size_t n, Stream) { std::memset(p, 0, n * sizeof(double)); }
void h2d(double* d, const double* s, size_t n, Stream) { std::memcpy(d, s, n * sizeof(double)); }
void d2h(double* d, const double* s, size_t n, Stream) { std::memcpy(d, s, n * sizeof(double)); }
void d2d(double* d, const double* s, size_t n, Stream) { std::memmove(d, s, n * sizeof(double)); }
void sync(Stream) {}
Stream stream_create(int) { return nullptr; }
void stream_destroy(Stream) {}
void* event_create() { return nullptr; }
void event_record(void*, Stream) {}
float event_ms(void*, void*) { return 0.f; }
void event_destroy(void*) {}
uint64_t launch_count() { return g_ops; }

void permute4(double* dst, const double* src, const int64_t d[4], const int perm[4],
              double alpha, double beta, Stream) {
  ++g_ops;
  int64_t ss[4];
  ss[3] = 1;
  for (int k = 2; k >= 0; --k) ss[k] = ss[k + 1] * d[k + 1];
  int64_t e[4], es[4];
  for (int k = 0; k < 4; ++k) { e[k] = d[perm[k]]; es[k] = ss[perm[k]]; }
  int64_t o = 0;
  for (int64_t i0 = 0; i0 < e[0]; ++i0)
    for (int64_t i1 = 0; i1 < e[1]; ++i1)
      for (int64_t i2 = 0; i2 < e[2]; ++i2)
        for (int64_t i3 = 0; i3 < e[3]; ++i3, ++o) {
          const double v = alpha * src[i0 * es[0] + i1 * es[1] + i2 * es[2] + i3 * es[3]];
          dst[o] = beta != 0.0 ? v + beta * dst[o] : v;
        }
}

void copy4(double* dst, const int64_t ds[4], const double* src, const int64_t ss[4],
           const int64_t e[4], double alpha, double beta, Stream) {
  ++g_ops;
  if (ds[3] != 1) throw Error(ERR_STATE, "copy4: the destination's inner stride must be 1");
  for (int64_t i0 = 0; i0 < e[0]; ++i0)
    for (int64_t i1 = 0; i1 < e[1]; ++i1)
      for (int64_t i2 = 0; i2 < e[2]; ++i2)
        for (int64_t i3 = 0; i3 < e[3]; ++i3) {
          const double v = alpha * src[i0 * ss[0] + i1 * ss[1] + i2 * ss[2] + i3 * ss[3]];
          double* d = dst + i0 * ds[0] + i1 * ds[1] + i2 * ds[2] + i3;
          *d = beta != 0.0 ? v + beta * *d : v;
        }
}

void axpby(double* out, double a, const double* x, double b, const double* y, double c,
           int64_t n, Stream) {
  ++g_ops;
  for (int64_t e = 0; e < n; ++e) {
    double v = a * x[e];
    if (y) v += b * y[e];
    if (c != 0.0) v += c * out[e];
    out[e] = v;
  }
}

void rank1(double* out, double a, const double* A, double b, const double* t, int64_t n,
           Stream) {
  ++g_ops;
  for (int64_t r = 0; r < n; ++r)
    for (int64_t c = 0; c < n; ++c) out[r * n + c] = a * A[r * n + c] + b * t[r] * t[c];
}

void zrank1(double* ore, double* oim, const double* are, const double* aim, const double* tre,
            const double* tim, double b, int64_t n, Stream) {
  ++g_ops;
  for (int64_t r = 0; r < n; ++r)
    for (int64_t c = 0; c < n; ++c) {
      const int64_t e = r * n + c;
      const double xr = tre[r] * tre[c] - tim[r] * tim[c];
      const double xi = tre[r] * tim[c] + tim[r] * tre[c];
      ore[e] = are[e] + b * xr;
      oim[e] = aim[e] + b * xi;
    }
}

void symmetrize(double* R, int64_t n, Stream) {
  ++g_ops;
  for (int64_t r = 0; r < n; ++r)
    for (int64_t c = r; c < n; ++c) {
      const double s = R[r * n + c] + R[c * n + r];
      R[r * n + c] = s;
      R[c * n + r] = s;
    }
}

void gather_vertex(double* out, const double* in, bool cplx, int part, int64_t NG, int64_t Np,
                   int64_t row0, int64_t nx, int64_t col0, int64_t ny, Stream) {
  ++g_ops;
  const int64_t es = cplx ? 2 : 1;
  for (int64_t g = 0; g < NG; ++g)
    for (int64_t x = 0; x < nx; ++x)
      for (int64_t y = 0; y < ny; ++y)
        out[(g * nx + x) * ny + y] = in[(g + NG * ((row0 + x) + Np * (col0 + y))) * es + part];
}

void jacobi(double* Tnew, double* dT, const double* R, const double* Told, const double* eh,
            const double* ep, const AmpShape& sh, double shift, Stream) {
  ++g_ops;
  const int64_t n1 = sh.n1();
  for (int64_t e = 0; e < sh.total(); ++e) {
    const int64_t q = e % sh.plane();
    double D;
    if (q < n1) {
      D = ep[q / sh.o] - eh[q % sh.o];
    } else {
      const int64_t r = q - n1, ai = r / n1, bj = r % n1;
      D = ep[ai / sh.o] - eh[ai % sh.o] + ep[bj / sh.o] - eh[bj % sh.o];
    }
    double rv = R[e];
    const double told = Told ? Told[e] : 0.0;
    if (Told && shift != 0.0) rv -= shift * told;
    const double tn = rv * (-1.0 / (D + shift));
    Tnew[e] = tn;
    dT[e] = Told ? tn - told : tn;
  }
}

void mp2_energy(const double* Vr, const double* Vi, const double* eh, const double* ep,
                int64_t o, int64_t v, double* out, double*, Stream) {
  ++g_ops;
  const int64_t n1 = v * o;
  double acc[2] = {0, 0};
  for (int64_t r = 0; r < n1; ++r)
    for (int64_t c = 0; c < n1; ++c) {
      const int64_t e = r * n1 + c, a = r / o, i = r % o, b = c / o, j = c % o;
      const double d = eh[i] + eh[j] - ep[a] - ep[b];
      const int64_t ex = (a * o + j) * n1 + b * o + i;
      acc[0] += (Vr[e] * Vr[e] + (Vi ? Vi[e] * Vi[e] : 0.0)) / d;
      acc[1] += (Vr[e] * Vr[ex] + (Vi ? Vi[e] * Vi[ex] : 0.0)) / d;
    }
  out[0] = 2.0 * acc[0];
  out[1] = -acc[1];
}

void energy(const double* T, const double* Vdr, const double* Vdi, const double* Ver,
            const double* Vei, const AmpShape& sh, double* out, double*, Stream) {
  ++g_ops;
  const int64_t n1 = sh.n1();
  const double* t1r = T;
  const double* t2r = T + n1;
  const double* t1i = sh.planes > 1 ? T + sh.plane() : nullptr;
  const double* t2i = sh.planes > 1 ? T + sh.plane() + n1 : nullptr;
  double acc[4] = {0, 0, 0, 0};
  for (int64_t r = 0; r < n1; ++r)
    for (int64_t c = 0; c < n1; ++c) {
      const int64_t e = r * n1 + c;
      // V_baij = Vd[(b,i),(a,j)] when no exchange tensor is given
      const int64_t ex = ((c / sh.o) * sh.o + r % sh.o) * n1 + (r / sh.o) * sh.o + c % sh.o;
      if (!t1i) {
        const double x = t2r[e] + t1r[r] * t1r[c];
        acc[0] += x * Vdr[e];
        acc[1] += x * (Ver ? Ver[e] : Vdr[ex]);
      } else {
        const double xr = t2r[e] + t1r[r] * t1r[c] - t1i[r] * t1i[c];
        const double xi = t2i[e] + t1r[r] * t1i[c] + t1i[r] * t1r[c];
        const double vdi = Vdi ? Vdi[e] : 0.0;
        const double ver = Ver ? Ver[e] : Vdr[ex];
        const double vei = Ver ? (Vei ? Vei[e] : 0.0) : (Vdi ? Vdi[ex] : 0.0);
        acc[0] += xr * Vdr[e] + xi * vdi;
        acc[1] += xr * ver + xi * vei;
        acc[2] += xi * Vdr[e] - xr * vdi;
        acc[3] += xi * ver - xr * vei;
      }
    }
  out[0] = 2.0 * acc[0]; out[1] = -acc[1]; out[2] = 2.0 * acc[2]; out[3] = -acc[3];
}

void dots(const double* x, const double* const* ys, int ny, int64_t n, double* out, double*,
          Stream) {
  ++g_ops;
  for (int k = 0; k < ny; ++k) {
    double s = 0.0;
    for (int64_t e = 0; e < n; ++e) s += x[e] * ys[k][e];
    out[k] = s;
  }
}

void diis_solve(double* B, const double* dots_dev, const int* valid, int N, int next, int count,
                double* coef, int* status, Stream) {
  ++g_ops;
  const int M = N + 1;
  int di = 0;
  for (int i = 0; i < N; ++i) {
    if (!valid[i]) continue;
    const double ov = 2.0 * dots_dev[di++];
    B[(i + 1) * M + next + 1] = ov;
    B[(next + 1) * M + i + 1] = ov;
  }
  const int dim = count + 1;
  std::vector<double> m(dim * dim), x(dim, 0.0);
  for (int r = 0; r < dim; ++r)
    for (int c = 0; c < dim; ++c) m[r * dim + c] = B[r * M + c];
  x[0] = -1.0;
  int singular = 0;
  for (int k = 0; k < dim; ++k) {
    int piv = k;
    double best = std::fabs(m[k * dim + k]);
    for (int r = k + 1; r < dim; ++r)
      if (std::fabs(m[r * dim + k]) > best) { best = std::fabs(m[r * dim + k]); piv = r; }
    if (!std::isfinite(best)) { singular = 2; break; }
    if (best == 0.0) { singular = 1; break; }
    if (piv != k) {
      for (int c = 0; c < dim; ++c) std::swap(m[k * dim + c], m[piv * dim + c]);
      std::swap(x[k], x[piv]);
    }
    for (int r = k + 1; r < dim; ++r) {
      const double f = m[r * dim + k] / m[k * dim + k];
      for (int c = k; c < dim; ++c) m[r * dim + c] -= f * m[k * dim + c];
      x[r] -= f * x[k];
    }
  }
  if (!singular) {
    for (int k = dim - 1; k >= 0; --k) {
      double s = x[k];
      for (int c = k + 1; c < dim; ++c) s -= m[k * dim + c] * x[c];
      x[k] = s / m[k * dim + k];
    }
    for (int j = 0; j < count; ++j) coef[j] = x[(next + N - j) % N + 1];
  }
  status[0] = singular;
}

void lincomb(double* out, const double* const* xs, const double* const* ys, const double* coef,
             int nx, int64_t n, double* norm2, double*, Stream) {
  ++g_ops;
  double s2 = 0.0;
  for (int64_t e = 0; e < n; ++e) {
    double v = 0.0, w = 0.0;
    for (int k = 0; k < nx; ++k) {
      v += coef[k] * xs[k][e];
      if (ys) w += coef[k] * ys[k][e];
    }
    out[e] = v;
    s2 += w * w;
  }
  if (ys && norm2) norm2[0] = s2;
}

void sum_partials_to(double* dst, const double* ws, int nparts, int nvals, Stream) {
  ++g_ops;
  for (int k = 0; k < nvals; ++k) {
    double v = 0.0;
    for (int b = 0; b < nparts; ++b) v += ws[b * nvals + k];
    dst[k] = v;
  }
}

HostStage::~HostStage() {}
void h2d_staged(double* dst, const double* src, int64_t n, int stride, HostStage&, Stream) {
  for (int64_t k = 0; k < n; ++k) dst[k] = src[k * stride];
}
void d2h_staged(double* dst, int stride, const double* src, int64_t n, HostStage&, Stream) {
  for (int64_t k = 0; k < n; ++k) dst[k * stride] = src[k];
}
void scatter_vertex(double* out, const double* in, bool cplx, int part, int64_t NG, int64_t Np,
                    int64_t row0, int64_t nx, int64_t col0, int64_t ny, Stream) {
  ++g_ops;
  for (int64_t g = 0; g < NG; ++g)
    for (int64_t x = 0; x < nx; ++x)
      for (int64_t y = 0; y < ny; ++y)
        out[(g + NG * (row0 + x + Np * (col0 + y))) * (cplx ? 2 : 1) + part] =
            in[(g * nx + x) * ny + y];
}
int scan_vertex(const double* p, int64_t n, bool complex_values, Stream) {
  ++g_ops;
  int f = 0;
  for (int64_t e = 0; e < n; ++e) {
    if (!std::isfinite(p[e])) f |= 1;
    if (complex_values && (e & 1) && p[e] != 0.0) f |= 2;
  }
  return f;
}

// Packed amplitude vectors: per plane [T1 | T2 rows r, columns r..n1-1].
static int64_t packed_index(const AmpShape& sh, int64_t pl, int64_t r, int64_t c) {
  const int64_t n1 = sh.n1();
  return pl * sh.packed_plane() + n1 + r * n1 - r * (r - 1) / 2 + (c - r);
}

void jacobi_packed(double* Tnew, double* dT, const double* R, const double* Told,
                   const double* eh, const double* ep, const AmpShape& sh, double shift,
                   Stream) {
  ++g_ops;
  const int64_t n1 = sh.n1();
  auto upd = [&](int64_t full, int64_t pk, double D) {
    double rv = R[full];
    const double told = Told ? Told[full] : 0.0;
    if (Told && shift != 0.0) rv -= shift * told;
    const double tn = rv * (-1.0 / (D + shift));
    Tnew[pk] = tn;
    dT[pk] = Told ? tn - told : tn;
  };
  for (int64_t pl = 0; pl < sh.planes; ++pl) {
    for (int64_t ai = 0; ai < n1; ++ai)
      upd(pl * sh.plane() + ai, pl * sh.packed_plane() + ai, ep[ai / sh.o] - eh[ai % sh.o]);
    for (int64_t r = 0; r < n1; ++r)
      for (int64_t c = r; c < n1; ++c)
        upd(pl * sh.plane() + n1 + r * n1 + c, packed_index(sh, pl, r, c),
            ep[r / sh.o] - eh[r % sh.o] + ep[c / sh.o] - eh[c % sh.o]);
  }
}

void dots_packed(const double* x, const double* const* ys, int ny, const AmpShape& sh,
                 double* out, double*, Stream) {
  ++g_ops;
  const int64_t n1 = sh.n1();
  for (int k = 0; k < ny; ++k) {
    double s = 0.0;
    for (int64_t pl = 0; pl < sh.planes; ++pl) {
      for (int64_t ai = 0; ai < n1; ++ai) {
        const int64_t e = pl * sh.packed_plane() + ai;
        s += x[e] * ys[k][e];
      }
      for (int64_t r = 0; r < n1; ++r)
        for (int64_t c = r; c < n1; ++c) {
          const int64_t e = packed_index(sh, pl, r, c);
          s += (c == r ? 1.0 : 2.0) * x[e] * ys[k][e];
        }
    }
    out[k] = s;
  }
}

void lincomb_packed(double* out, const double* const* xs, const double* const* ys,
                    const double* coef, int nx, const AmpShape& sh, double* norm2, double*,
                    Stream) {
  ++g_ops;
  const int64_t n1 = sh.n1();
  double s2 = 0.0;
  auto comb = [&](int64_t pk, double& w) {
    double v = 0.0;
    w = 0.0;
    for (int k = 0; k < nx; ++k) {
      v += coef[k] * xs[k][pk];
      if (ys) w += coef[k] * ys[k][pk];
    }
    return v;
  };
  for (int64_t pl = 0; pl < sh.planes; ++pl) {
    double* ob = out + pl * sh.plane();
    for (int64_t ai = 0; ai < n1; ++ai) {
      double w;
      ob[ai] = comb(pl * sh.packed_plane() + ai, w);
      s2 += w * w;
    }
    for (int64_t r = 0; r < n1; ++r)
      for (int64_t c = r; c < n1; ++c) {
        double w;
        const double v = comb(packed_index(sh, pl, r, c), w);
        ob[n1 + r * n1 + c] = v;
        ob[n1 + c * n1 + r] = v;
        s2 += (c == r ? 1.0 : 2.0) * w * w;
      }
  }
  if (ys && norm2) norm2[0] = s2;
}


void fsc_prepare_u(double* ore, double* oim, const double* U, const double* V, int64_t NGG,
                   int64_t NF, Stream) {
  ++g_ops;
  for (int64_t G = 0; G < NGG; ++G)
    for (int64_t F = 0; F < NF; ++F) {
      const int64_t e = F * NGG + G;
      const double re = U ? U[2 * e] : (G == F ? 1.0 : 0.0), im = U ? U[2 * e + 1] : 0.0;
      const double sc = V ? 1.0 / std::sqrt(V[G]) : 1.0;
      ore[G * NF + F] = re * sc;
      oim[G * NF + F] = im * sc;
    }
}

void fsc_stacked_to_complex(double* Qr, double* Qi, const double* Qs, int64_t NF, int parts,
                            Stream) {
  ++g_ops;
  const int64_t S2 = parts * NF;
  for (int64_t F = 0; F < NF; ++F)
    for (int64_t Fp = 0; Fp < NF; ++Fp) {
      const int64_t e = F * NF + Fp;
      if (parts == 2) {
        Qr[e] = Qs[F * S2 + Fp] + Qs[(F + NF) * S2 + Fp + NF];
        Qi[e] = Qs[F * S2 + Fp + NF] - Qs[(F + NF) * S2 + Fp];
      } else {
        Qr[e] = Qs[e];
        Qi[e] = 0.0;
      }
    }
}

static void fsc_direct_emu(const FscGeometry& g, const double v[3], double x[3]) {
  for (int d = 0; d < 3; ++d) x[d] = g.A[3 * d] * v[0] + g.A[3 * d + 1] * v[1] + g.A[3 * d + 2] * v[2];
}

void fsc_box(double* box, const double* S, const double* grid, const FscGeometry& g, Stream) {
  ++g_ops;
  std::memset(box, 0, sizeof(double) * g.dims[0] * g.dims[1] * g.dims[2]);
  for (int64_t e = 0; e < g.NG; ++e) {
    double x[3];
    fsc_direct_emu(g, grid + 3 * e, x);
    int64_t i[3];
    bool in = true;
    for (int d = 0; d < 3; ++d) {
      i[d] = static_cast<int64_t>(std::floor(x[d] + 0.5) - g.origin[d]);
      in = in && i[d] >= 0 && i[d] < g.dims[d];
    }
    if (in) box[i[0] + g.dims[0] * (i[1] + g.dims[1] * i[2])] = S[e];
  }
}

static double fsc_tricubic_emu(const double* box, const FscGeometry& g, const double x[3]) {
  static const double BL[4][4] = {{0.0, -0.5, 1.0, -0.5}, {1.0, 0.0, -2.5, 1.5},
                                  {0.0, 0.5, 2.0, -1.5}, {0.0, 0.0, -0.5, 0.5}};
  double w[3][4];
  int64_t base[3];
  for (int d = 0; d < 3; ++d) {
    const double t = x[d] - g.origin[d];
    int64_t i = static_cast<int64_t>(t);
    i = std::min<int64_t>(std::max<int64_t>(i, 0), g.dims[d] - 1);
    const double u = t - static_cast<double>(i);
    for (int r = 0; r < 4; ++r) w[d][r] = BL[r][0] + BL[r][1] * u + BL[r][2] * u * u + BL[r][3] * u * u * u;
    base[d] = i - 1;
  }
  auto cl = [](int64_t a, int64_t n) { return std::min<int64_t>(std::max<int64_t>(a, 0), n - 1); };
  double total = 0.0;
  for (int sl = 0; sl < 4; ++sl)
    for (int r = 0; r < 4; ++r)
      for (int c = 0; c < 4; ++c)
        total += w[0][c] * w[1][r] * w[2][sl] *
                 box[cl(base[0] + c, g.dims[0]) +
                     g.dims[0] * (cl(base[1] + r, g.dims[1]) + g.dims[1] * cl(base[2] + sl, g.dims[2]))];
  return total;
}

void fsc_sums(const double* box, const double* S, const double* grid, const FscGeometry& g,
              double*, double* out, Stream) {
  ++g_ops;
  double acc0 = 0.0, acc1 = 0.0;
  for (int64_t e = 0; e < g.NG; ++e) {
    const double* v = grid + 3 * e;
    const double n2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
    if (std::sqrt(n2) >= 1e-8) acc0 += g.f / n2 * S[e];
  }
  const int64_t n2N = 2 * static_cast<int64_t>(g.N);
  const double inv2N = 1.0 / static_cast<double>(n2N);
  for (int64_t a = -g.N; a < g.N; ++a)
    for (int64_t b = -g.N; b < g.N; ++b)
      for (int64_t c = -g.N; c < g.N; ++c)
        for (int64_t i = 0; i < g.NG; ++i) {
          double v[3];
          for (int d = 0; d < 3; ++d)
            v[d] = g.B[d] * inv2N * double(a) + g.B[3 + d] * inv2N * double(b) +
                   g.B[6 + d] * inv2N * double(c) + grid[3 * i + d];
          const double n2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
          if (std::sqrt(n2) < 1e-8) continue;
          double x[3];
          fsc_direct_emu(g, v, x);
          acc1 += g.f * fsc_tricubic_emu(box, g, x) / n2;
        }
  out[0] = acc0;
  out[1] = acc1;
}

struct TriplesC { double re, im; };

static TriplesC triples_singles_at(const double* t, const double* ti, const double* V,
                                   const double* Vi, int64_t n1, int64_t p1, int64_t p2,
                                   int64_t p3) {
  const int64_t pr[3][3] = {{p1, p2, p3}, {p2, p1, p3}, {p3, p1, p2}};  // t index, V row, V col
  TriplesC s{0.0, 0.0};
  for (const auto& k : pr) {
    const double tr = t[k[0]], tm = ti ? ti[k[0]] : 0.0;
    const double vr = V[k[1] * n1 + k[2]], vm = Vi ? Vi[k[1] * n1 + k[2]] : 0.0;
    s.re += tr * vr - tm * vm;
    s.im += tr * vm + tm * vr;
  }
  return s;
}

void triples_singles(double* S, double* S_im, const double* t1, const double* t1_im,
                     const double* V, const double* V_im, const TriplesBlock& b, Stream) {
  ++g_ops;
  for (int64_t q1 = 0; q1 < b.L[0]; ++q1)
    for (int64_t q2 = 0; q2 < b.L[1]; ++q2)
      for (int64_t q3 = 0; q3 < b.L[2]; ++q3) {
        const int64_t e = (q1 * b.L[1] + q2) * b.L[2] + q3;
        const TriplesC x = triples_singles_at(t1, t1_im, V, V_im, b.n1, b.P[0] + q1,
                                              b.P[1] + q2, b.P[2] + q3);
        S[e] = x.re;
        if (S_im) S_im[e] = x.im;
      }
}

void triples_energy(const double* S, const double* S_im, const double* t1, const double* t1_im,
                    const double* V, const double* V_im, const double* eh, const double* ep,
                    const TriplesBlock& b, const double coef[6], double*, double* out, Stream,
                    const double* M, const double* M_im) {
  ++g_ops;
  static const int perm[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
  const int64_t o = b.o;
  double acc[2] = {0.0, 0.0};
  for (int64_t q1 = 0; q1 < b.L[0]; ++q1)
    for (int64_t q2 = 0; q2 < b.L[1]; ++q2)
      for (int64_t q3 = 0; q3 < b.L[2]; ++q3) {
        const int64_t x[3] = {q1 / o, q2 / o, q3 / o};
        const int64_t y[3] = {q1 % o, q2 % o, q3 % o};
        auto at = [&](const double* A, int64_t r1, int64_t r2, int64_t r3) {
          return A[(r1 * b.L[1] + r2) * b.L[2] + r3];
        };
        const TriplesC sg = triples_singles_at(t1, t1_im, V, V_im, b.n1, b.P[0] + q1,
                                               b.P[1] + q2, b.P[2] + q3);
        double d = 0.0;
        for (int m = 0; m < 3; ++m) d += eh[y[m]] - ep[b.P[m] / o + x[m]];
        double yr = 0.0, yi = 0.0;
        for (int k = 0; k < 6; ++k) {
          const int64_t r1 = x[0] * o + y[perm[k][0]], r2 = x[1] * o + y[perm[k][1]],
                        r3 = x[2] * o + y[perm[k][2]];
          yr += coef[k] * at(S, r1, r2, r3);
          if (S_im) yi += coef[k] * at(S_im, r1, r2, r3);
        }
        const double wr = M ? at(M, q1, q2, q3) : at(S, q1, q2, q3) - sg.re;
        acc[0] += wr * yr / d;
        if (S_im) acc[1] += (M ? at(M_im, q1, q2, q3) : at(S_im, q1, q2, q3) - sg.im) * yi / d;
      }
  out[0] = acc[0];
  out[1] = acc[1];
}

bool triples_cube_fits(int64_t, bool) { return true; }
void triples_energy_connected(const double* W, const double* W_im, const double* t1,
                              const double* t1_im, const double* V, const double* V_im,
                              const double* eh, const double* ep, const TriplesBlock& b,
                              const double coef[6], double* ws, double* out, Stream s) {
  const int64_t n = b.L[0] * b.L[1] * b.L[2];
  std::vector<double> S(n), Si(W_im ? n : 0);
  triples_singles(S.data(), W_im ? Si.data() : nullptr, t1, t1_im, V, V_im, b, s);
  for (int64_t k = 0; k < n; ++k) S[k] += W[k];
  for (int64_t k = 0; k < (W_im ? n : 0); ++k) Si[k] += W_im[k];
  triples_energy(S.data(), W_im ? Si.data() : nullptr, t1, t1_im, V, V_im, eh, ep, b, coef, ws, out,
                 s, W, W_im);
}

void triples_cr_sums(const double* S, const double* S_im, const double* t1, const double* t1_im,
                     const double* T2, const double* T2_im, const double* eh, const double* ep,
                     const TriplesBlock& b, const double coef[6], double*, double* out, Stream) {
  ++g_ops;
  static const int perm[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
  const int64_t o = b.o;
  double acc[2] = {0.0, 0.0};
  for (int64_t q1 = 0; q1 < b.L[0]; ++q1)
    for (int64_t q2 = 0; q2 < b.L[1]; ++q2)
      for (int64_t q3 = 0; q3 < b.L[2]; ++q3) {
        const int64_t x[3] = {q1 / o, q2 / o, q3 / o};
        const int64_t y[3] = {q1 % o, q2 % o, q3 % o};
        auto at = [&](const double* A, int64_t r1, int64_t r2, int64_t r3) {
          return A[(r1 * b.L[1] + r2) * b.L[2] + r3];
        };
        const int64_t p[3] = {b.P[0] + q1, b.P[1] + q2, b.P[2] + q3};
        const TriplesC ts = triples_singles_at(t1, t1_im, T2, T2_im, b.n1, p[0], p[1], p[2]);
        double pr = t1[p[0]], pi = t1_im ? t1_im[p[0]] : 0.0;
        for (int m = 1; m < 3; ++m) {
          const double r = t1[p[m]], i = t1_im ? t1_im[p[m]] : 0.0;
          const double nr = pr * r - pi * i, ni = pr * i + pi * r;
          pr = nr; pi = ni;
        }
        double d = 0.0;
        for (int m = 0; m < 3; ++m) d += eh[y[m]] - ep[b.P[m] / o + x[m]];
        double zr = 0.0, zi = 0.0;
        for (int k = 0; k < 6; ++k) {
          const int64_t r1 = x[0] * o + y[perm[k][0]], r2 = x[1] * o + y[perm[k][1]],
                        r3 = x[2] * o + y[perm[k][2]];
          zr += coef[k] * at(S, r1, r2, r3);
          if (S_im) zi += coef[k] * at(S_im, r1, r2, r3);
        }
        acc[0] += (ts.re + pr) * zr / d;
        if (S_im) acc[1] += (ts.im + pi) * zi / d;
      }
  out[0] = acc[0];
  out[1] = acc[1];
}

}  // namespace ops
}  // namespace cc4s_b200

// Test-only entry: C = A B of row-major host operands in a digit form (0: the plain chain).
extern "C" void emu_gemm_split(const double* A, const double* B, double* C, int64_t M, int64_t N,
                               int64_t K, int digits) {
  using namespace cc4s_b200;
  Contraction c;
  c.M = M; c.N = N; c.K = K; c.digits = digits;
  c.A = rm(const_cast<double*>(A), K);
  c.B = rm(const_cast<double*>(B), N);
  c.C = rm(C, N);
  SplitScratch ws;
  if (digits) gemm_split(c, nullptr, ws);
  else gemm(c, nullptr, ws.fp64);
}
