// FP64 contraction in signed 8-bit digits on the tcgen05 tensor cores (kind::i8).
//
// Kernel layout (persistent, one CTA of 320 threads per SM, 128 x TN output tiles,
// TN = 128 with 4 digits, 64 with 8):
//   warp 0      TMA producer: per k-block all digit planes of the A rows and of the
//               B rows (two 3-D boxes, swizzled) into a shared-memory ring, completion
//               tracked by mbarriers;
//   warp 1      allocates 512 TMEM columns; one thread issues tcgen05.mma (M = 128,
//               N up to 256, K = 32) for the digit products of equal weight p + q into
//               one S32 accumulator each (TN columns at TN (p + q)): A digit p times
//               the adjacent B digits q is one MMA into adjacent groups;
//   warps 2..9  epilogue: tcgen05.ld of the groups, exact 64-bit integer combination of
//               four groups at a time, conversion to FP64, then scale and store of the
//               tile (through warp-private transposes where the columns are contiguous)
//               while the MMA issuer is on the next tile.
// Integer accumulation is exact, so a tile is drained once per 16384 of K.
// Every mbarrier wait is bounded; on expiry the kernel records an error flag
// and every role leaves its loop, so the kernel always terminates.
#include "split_gemm.cuh"

#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <climits>
#include <cstdlib>
#include <mutex>
#include <vector>

namespace cc4s_b200 {

namespace {

constexpr int TM = 128;
constexpr int KPAD = 32;                         // K step of one MMA: packed K granularity
// |digit product| <= 2^14, and 65 * 128 where the top digit takes part: at most 114944 per
// group and k (six products and two with the top digit), exact in S32 up to here
constexpr int KCHUNK = 16384;
constexpr uint32_t WAIT_LIMIT = 1u << 28;         // bounded mbarrier waits
constexpr uint32_t RASTER_M = 8;                 // tile rows per raster group
constexpr int WBUF_DOUBLES = 32 * 16;            // transpose buffer of one epilogue warp
constexpr int EXP_NONFINITE = INT_MAX;           // exponent of a row holding Inf or NaN

// Geometry of the two forms: NS digits, groups p + q < NG = NS, TN columns per tile (TN NG =
// the 512 TMEM columns), k-blocks of TK bytes (= the swizzle width), NST ring stages.
template <int NS_> struct Form;
template <> struct Form<4> {
  static constexpr int NS = 4, NG = 4, TN = 128, TK = 64, NST = 3;
};
template <> struct Form<8> {
  static constexpr int NS = 8, NG = 8, TN = 64, TK = 64, NST = 2;
};
template <class F> __host__ __device__ constexpr int a_bytes() { return F::NS * TM * F::TK; }
template <class F> __host__ __device__ constexpr int stage_bytes() { return F::NS * (TM + F::TN) * F::TK; }
template <class F> constexpr int smem_bytes() {
  return F::NST * stage_bytes<F>() + 8 * WBUF_DOUBLES * 8 + 1024 + 256;
}
int tile_n(int digits) { return digits == 8 ? Form<8>::TN : Form<4>::TN; }

std::atomic<uint64_t> g_split_launches{0};
std::atomic<uint64_t> g_pack_launches{0};

struct Ax {
  uint32_t inner;
  int64_t s_o, s_i;
  __host__ __device__ __forceinline__ int64_t off(uint32_t x) const {
    const uint32_t o = x / inner;
    return static_cast<int64_t>(o) * s_o + static_cast<int64_t>(x - o * inner) * s_i;
  }
};
Ax mkax(int64_t inner, int64_t s_o, int64_t s_i) {
  Ax a; a.inner = static_cast<uint32_t>(inner > 0 ? inner : 1); a.s_o = s_o; a.s_i = s_i; return a;
}

// ---------------------------------------------------------------------------
// Packing: operand element (r, k) -> NS signed 8-bit digits P[q][r][k]
// (row-padded to Rp, k-padded to Kp) and a per-row exponent.
struct PackArgs {
  const double* src;
  Ax ar, ak;              // two-level index maps of the row and k indices
  int64_t R, K, Rp, Kp;
  unsigned long long* rmax;  // per-row max |x| as IEEE bits (non-negative doubles)
  int* rexp;              // per-row exponent
  int8_t* dst;            // [NS][Rp][Kp]
  int r_contig;           // 1: the row index is the contiguous one in memory
  float* prof;            // [Rp / 64][Kp] profiles (eight digits)
  // Two planes of a complex operand side by side along k: k < K1 reads at offset off[0]
  // with sign[0], the others at off[1] with sign[1] (K1 = K: one plane).
  int64_t K1;
  int64_t off[2];
  double sign[2];
  __device__ __forceinline__ int64_t koff(int64_t k) const {
    return k < K1 ? off[0] + ak.off(static_cast<uint32_t>(k))
                  : off[1] + ak.off(static_cast<uint32_t>(k - K1));
  }
};
// One launch slices up to three operands: A and B of a contraction, one of them in two
// forms in a complex one.
struct PackSet {
  PackArgs op[3];
  uint32_t end[3];        // work items of the operands, cumulative; the last is the total
};

constexpr int PR = 64, PTHREADS = 256;  // rows of a work item

__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return static_cast<unsigned long long>(__double_as_longlong(fabs(x)));
}

// Row maxima |x| as IEEE bits of non-negative doubles (Inf and NaN order above every
// number).  A work item is 64 rows x `kstrip` k, read straight from memory with the lanes
// along the contiguous index and 16 loads in flight per thread; one atomicMax per row.
// Bound by latency until a few hundred items are in flight, which sets kstrip: strips of
// 1024 k left two 1024 x 1024 operands to 32 blocks (whole contraction 79 us,
// 63 us with strips of 128).
__global__ void __launch_bounds__(PTHREADS) pack_max_kernel(PackSet pp, int kstrip) {
  __shared__ unsigned long long part[8][PR];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint32_t it = blockIdx.x; it < pp.end[2]; it += gridDim.x) {
    const int which = it < pp.end[0] ? 0 : it < pp.end[1] ? 1 : 2;
    const PackArgs& a = pp.op[which];
    const uint32_t w = which ? it - pp.end[which - 1] : it;
    const uint32_t nks = static_cast<uint32_t>(a.K + kstrip - 1) / static_cast<uint32_t>(kstrip);
    const uint32_t wr = w / nks;
    const int64_t r0 = int64_t(wr) * PR, kbeg = int64_t(w - wr * nks) * kstrip;
    const int64_t kend = min(a.K, kbeg + kstrip);
    if (a.r_contig) {  // lanes on rows; the eight warps take every eighth k
      unsigned long long m[2] = {0, 0};
      const int64_t ra = r0 + lane, rb = ra + 32;
      const double* sa = a.src + (ra < a.R ? a.ar.off(static_cast<uint32_t>(ra)) : 0);
      const double* sb = a.src + (rb < a.R ? a.ar.off(static_cast<uint32_t>(rb)) : 0);
      for (int64_t k0 = kbeg + warp; k0 < kend; k0 += 64) {
        double x[2][8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int64_t k = k0 + 8 * j;
          const int64_t ko = k < kend ? a.koff(k) : 0;
          x[0][j] = k < kend && ra < a.R ? sa[ko] : 0.0;
          x[1][j] = k < kend && rb < a.R ? sb[ko] : 0.0;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 8; ++j) m[h] = max(m[h], abs_bits(x[h][j]));
      }
      part[warp][lane] = m[0];
      part[warp][lane + 32] = m[1];
      __syncthreads();
      if (threadIdx.x < PR) {
        unsigned long long v = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) v = max(v, part[q][threadIdx.x]);
        if (r0 + threadIdx.x < a.R && v != 0) atomicMax(&a.rmax[r0 + threadIdx.x], v);
      }
      __syncthreads();
    } else {           // lanes on k; every warp takes eight rows
      const int64_t rw = r0 + 8 * warp;
      unsigned long long m[8];
      const double* src[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        m[q] = 0;
        src[q] = rw + q < a.R ? a.src + a.ar.off(static_cast<uint32_t>(rw + q)) : nullptr;
      }
      for (int64_t k0 = kbeg + lane; k0 < kend; k0 += 64) {
        const int64_t k1 = k0 + 32;
        const int64_t o0 = a.koff(k0);
        const int64_t o1 = k1 < kend ? a.koff(k1) : o0;
        double x[2][8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          x[0][q] = src[q] ? src[q][o0] : 0.0;
          x[1][q] = src[q] ? src[q][o1] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) m[q] = max(m[q], max(abs_bits(x[0][q]), abs_bits(x[1][q])));
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) m[q] = max(m[q], __shfl_xor_sync(0xffffffffu, m[q], s));
        if (lane == q && src[q] && m[q] != 0) atomicMax(&a.rmax[rw + q], m[q]);
      }
    }
  }
}

// 2^e as an exact double: built from its exponent bits in the normal range.
__device__ __forceinline__ double pow2i(int e) {
  if (e >= -1022 && e <= 1023) return __longlong_as_double(static_cast<long long>(e + 1023) << 52);
  return ldexp(1.0, e);
}

// Digits of four elements: word q holds digit q of each, element 0 in the lowest byte.
// With 128 added to every digit but the top one, the bytes of the integer are the digits
// plus 128 (the carries of a balanced representation happen in the one addition).  Eight
// digits also add the magnitudes, in units of 2^-27 of the row's power of two, to sum.
template <int NS>
__device__ __forceinline__ void digits4(const double (&x)[4], double s1, double s2,
                                        uint32_t (&w)[NS], uint32_t (&sum)[4]) {
  uint32_t lo[4], hi[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if constexpr (NS == 4) {
      lo[j] = (static_cast<uint32_t>(__double2int_rn(x[j] * s1 * s2)) + 0x00808080u) ^ 0x00808080u;
      hi[j] = 0;
    } else {
      const long long v = __double2ll_rn(x[j] * s1 * s2);
      sum[j] += static_cast<uint32_t>(abs(static_cast<int>(v >> 32))) >> 3;
      const unsigned long long X =
          (static_cast<unsigned long long>(v) + 0x0080808080808080ull) ^ 0x0080808080808080ull;
      lo[j] = static_cast<uint32_t>(X);
      hi[j] = static_cast<uint32_t>(X >> 32);
    }
  }
  auto planes = [&](const uint32_t (&v)[4], int byte) {  // byte pair (byte, byte + 1) of each
    const uint32_t a = __byte_perm(v[0], v[1], byte ? 0x7362 : 0x5140);
    const uint32_t b = __byte_perm(v[2], v[3], byte ? 0x7362 : 0x5140);
    return make_uint2(__byte_perm(a, b, 0x5410), __byte_perm(a, b, 0x7632));
  };
  const uint2 l0 = planes(lo, 0), l2 = planes(lo, 2);
  w[NS - 1] = l0.x;
  w[NS - 2] = l0.y;
  w[NS - 3] = l2.x;
  w[NS - 4] = l2.y;
  if constexpr (NS == 8) {
    const uint2 h0 = planes(hi, 0), h2 = planes(hi, 2);
    w[3] = h0.x;
    w[2] = h0.y;
    w[1] = h2.x;
    w[0] = h2.y;
  }
}

// The digits of every element (row-padded to Rp, k-padded to Kp) and the per-row
// exponent: x = 2^e X 2^-(8 NS - 2) with |X| <= 2^(8 NS - 2) rounded to an integer and
// written in balanced base 256 (each digit in [-128, 127], the top one in [-64, 65]).
// A work item is 64 rows x 128 k (lanes on four k each, a warp per row, nothing staged, so
// 16 loads per thread stay in flight without a barrier) or, where the rows are contiguous
// in memory, 64 rows x 64 k through a shared-memory tile (stores of 16 bytes per row and
// lane straight from such loads were slower: 1.14 against 0.99 ms for 256 x 262144 x 256).
// Memory bound: 8 B read, NS B written per element.  Against tiles for both and digits
// extracted one by one, whole contractions (seven digits) of 2048^3 0.291 -> 0.275 ms,
// 4096 x 256 x 16384 0.92 -> 0.87 ms, 4096 x 1024 x 65536 8.06 -> 7.83 ms.
// Eight digits also leave the profile of the item's rows (the header says what for): sums
// over the 8 rows of a warp in registers, from the integers that are there, then the least
// of the eight warps' means through shared memory, which costs the unstaged items their
// only barrier.
constexpr int PK_K = 128, PK_R = 64;  // k per item, by the contiguous index
// Mean magnitudes over `live` rows (all-zero rows are exact and do not count).
__device__ __forceinline__ float4 means(const uint32_t (&s)[4], int live) {
  const float w = live ? 0x1p-27f / static_cast<float>(live) : 0.0f;
  const float none = live ? 0.0f : 1.0f;
  return make_float4(s[0] * w + none, s[1] * w + none, s[2] * w + none, s[3] * w + none);
}
// The least of the eight warps' means.
__device__ __forceinline__ float least(const float* part, int stride, bool odd) {
  float v = part[0];
#pragma unroll
  for (int q = 1; q < 8; ++q) v = fminf(v, part[q * stride]);
  return odd ? __int_as_float(0x7fc00000) : v;
}
template <int NS>
__global__ void __launch_bounds__(PTHREADS) pack_digits_kernel(PackSet pp) {
  __shared__ double tile[PR][81];  // k at k + k / 4: both directions free of bank conflicts
  __shared__ int64_t rows_off[PR], ks_off[PK_R];
  __shared__ float cpart[8][PK_R];
  int flip = 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint32_t it = blockIdx.x; it < pp.end[2]; it += gridDim.x) {
    const int which = it < pp.end[0] ? 0 : it < pp.end[1] ? 1 : 2;
    const PackArgs& a = pp.op[which];
    const uint32_t w = which ? it - pp.end[which - 1] : it;
    const int kw = a.r_contig ? PK_R : PK_K;
    const uint32_t nk = static_cast<uint32_t>(a.Kp + kw - 1) / kw, wr = w / nk;
    const int64_t pl = a.Rp * a.Kp, r0 = int64_t(wr) * PR, k0 = int64_t(w - wr * nk) * kw;
    // the row this lane answers for: its exponent, scale and offset
    const int64_t lr = r0 + 8 * warp + (lane & 7);
    double s1 = 0.0, s2 = 0.0;  // their product 2^(8 NS - 2 - e), each in the normal range
    int64_t roff = -1;
    bool live = false, odd = false;  // not all zero; neither finite nor within the exponents
    if (lr < a.R) {
      const unsigned long long mb = a.rmax[lr];
      int e = 0;
      if (mb >= 0x7ff0000000000000ull) {
        e = EXP_NONFINITE;
      } else if (mb != 0) {
        frexp(__longlong_as_double(static_cast<long long>(mb)), &e);
        const int sh = 8 * NS - 2 - e;
        s1 = pow2i(sh / 2);
        s2 = pow2i(sh - sh / 2);
      }
      if (k0 == 0) a.rexp[lr] = e;
      live = mb != 0;
      odd = e > kSplitMaxExponent || e < -kSplitMaxExponent;
      roff = a.ar.off(static_cast<uint32_t>(lr));
    }
    uint32_t sum[4] = {0, 0, 0, 0};  // magnitudes of the warp's rows, per k of the lane
    const int nlive = NS == 8 ? __popc(__ballot_sync(0xffffffffu, live) & 0xff) : 0;
    int any_odd = odd;
    if (a.r_contig) {
      if (lane < 8) rows_off[8 * warp + lane] = roff;
      else if (lane < 16) {
        const int64_t k = k0 + 8 * warp + (lane - 8);
        ks_off[8 * warp + lane - 8] = k < a.K ? a.koff(k) : -1;
      }
      __syncthreads();
    }
    if (a.r_contig) {  // lanes on rows for the loads, on k for the stores
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int64_t ro = rows_off[32 * h + lane];
        double x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int64_t ko = ks_off[8 * warp + j];
          x[j] = (ro >= 0 && ko >= 0) ? a.src[ro + ko] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int k = 8 * warp + j;
          tile[32 * h + lane][k + (k >> 2)] = x[j];
        }
      }
      __syncthreads();
      const int64_t kb = k0 + 4 * (lane & 15);
      double sg[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) sg[j] = a.sign[kb + j < a.K1 ? 0 : 1];
#pragma unroll
      for (int h = 0; h < 4; ++h) {  // two rows at a time, half a warp each
        const int r = 2 * h + (lane >> 4);
        const double t1 = __shfl_sync(0xffffffffu, s1, r), t2 = __shfl_sync(0xffffffffu, s2, r);
        double y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] = tile[8 * warp + r][5 * (lane & 15) + j] * sg[j];
        uint32_t q[NS];
        digits4<NS>(y, t1, t2, q, sum);
        if (kb < a.Kp) {
          int8_t* d = a.dst + (r0 + 8 * warp + r) * a.Kp + kb;
#pragma unroll
          for (int n = 0; n < NS; ++n) *reinterpret_cast<uint32_t*>(d + n * pl) = q[n];
        }
      }
      if (NS == 8) {
#pragma unroll
        for (int j = 0; j < 4; ++j) sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], 16);
        if (lane < 16)
          *reinterpret_cast<float4*>(&cpart[warp][4 * lane]) = means(sum, nlive);
        any_odd = __syncthreads_or(any_odd);
        if (threadIdx.x < PK_R && k0 + threadIdx.x < a.Kp)
          a.prof[int64_t(wr) * a.Kp + k0 + threadIdx.x] = least(&cpart[0][threadIdx.x], PK_R, any_odd);
      }
      __syncthreads();
    } else {
      const int64_t kb = k0 + 4 * lane;
      int64_t ko[4];
      double sg[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        ko[j] = kb + j < a.K ? a.koff(kb + j) : -1;
        sg[j] = a.sign[kb + j < a.K1 ? 0 : 1];
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {  // four rows at a time
        double x[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int64_t ro = __shfl_sync(0xffffffffu, roff, 4 * h + r);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            x[r][j] = (ro >= 0 && ko[j] >= 0) ? a.src[ro + ko[j]] * sg[j] : 0.0;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const double t1 = __shfl_sync(0xffffffffu, s1, 4 * h + r);
          const double t2 = __shfl_sync(0xffffffffu, s2, 4 * h + r);
          uint32_t q[NS];
          digits4<NS>(x[r], t1, t2, q, sum);
          if (kb < a.Kp) {
            int8_t* d = a.dst + (r0 + 8 * warp + 4 * h + r) * a.Kp + kb;
#pragma unroll
            for (int n = 0; n < NS; ++n) *reinterpret_cast<uint32_t*>(d + n * pl) = q[n];
          }
        }
      }
      if (NS == 8) {  // two buffers in turn, so that one barrier per item is enough
        float* part = reinterpret_cast<float*>(tile) + flip * 8 * PK_K;
        *reinterpret_cast<float4*>(part + warp * PK_K + 4 * lane) = means(sum, nlive);
        any_odd = __syncthreads_or(any_odd);
        if (threadIdx.x < PK_K && k0 + threadIdx.x < a.Kp)
          a.prof[int64_t(wr) * a.Kp + k0 + threadIdx.x] = least(part + threadIdx.x, PK_K, any_odd);
      }
    }
    if (NS == 8) flip ^= 1;
  }
}

// Product sums of the profiles of nI blocks of A and nJ of B: map[I][J] (and *any) tell the
// ones below `least`, or NaN.  A block takes one I and four J, its warps share k.  Small: 20
// flops per 64 x 64 x 4 products; the launch is most of it.
__global__ void profile_kernel(const float* A, const float* B, int64_t nI, int64_t nJ, int64_t Kp,
                               float least, unsigned char* map, int* any) {
  __shared__ float part[32][4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t nq = (nJ + 3) / 4;
  for (int64_t b = blockIdx.x; b < nI * nq; b += gridDim.x) {
    const int64_t I = b / nq, J = (b - I * nq) * 4;
    const float* a = A + I * Kp;
    const float* bs[4];
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < 4; ++q) bs[q] = B + min(J + q, nJ - 1) * Kp;
#pragma unroll 2
    for (int64_t k = 4 * threadIdx.x; k < Kp; k += 4 * blockDim.x) {
      const float4 x = *reinterpret_cast<const float4*>(a + k);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 y = *reinterpret_cast<const float4*>(bs[q] + k);
        s[q] += x.x * y.x + x.y * y.y + x.z * y.z + x.w * y.w;
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], d);
      if (lane == 0) part[warp][q] = s[q];
    }
    __syncthreads();
    if (threadIdx.x < 4 && J + threadIdx.x < nJ) {
      float v = 0.f;
      for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) v += part[w][threadIdx.x];
      const bool refused = !(v >= least);
      if (map) map[I * nJ + J + threadIdx.x] = refused;
      if (refused) *any = 1;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Device helpers (inline PTX for sm_100a).
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar));
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;\n" : "=l"(t));
  return t;
}
// Bounded wait for the phase with the given parity: gives up after
// WAIT_LIMIT polls or 2 seconds, whichever comes first; returns false then.  The clock
// is read only once 1024 polls have failed.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  uint64_t t0 = 0;
  for (uint32_t it = 0; it < WAIT_LIMIT; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
    if ((it & 1023) == 1023) {
      const uint64_t now = global_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > 2000000000ull) return false;
    }
  }
  return false;
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar,
                                            int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];\n"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// Shared-memory matrix descriptor: K-major, swizzled rows of ROW bytes (32, 64 or 128),
// 8-row groups 8 * ROW apart.
template <int ROW>
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr >> 4) & 0x3FFF);        // start address
  d |= static_cast<uint64_t>(1) << 16;                       // leading byte offset (16 B)
  d |= static_cast<uint64_t>((8 * ROW) >> 4) << 32;          // stride byte offset
  d |= static_cast<uint64_t>(1) << 46;                       // descriptor version (sm100)
  d |= static_cast<uint64_t>(ROW == 128 ? 2 : ROW == 64 ? 4 : 6) << 61;  // swizzle width
  return d;
}
// Instruction descriptor: D = S32, A = B = signed 8 bit, both K-major, M = 128.
__host__ __device__ constexpr uint32_t idesc_i8(int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(TM >> 4) << 24);
}

__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc,
                                     uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc));
}
// COLS columns of D at column d: A (one digit) times COLS consecutive rows of the B planes.
template <int COLS, int ROW>
__device__ __forceinline__ void umma_row(uint32_t d, uint64_t da, uint32_t b, uint32_t acc) {
#pragma unroll
  for (int c = 0; c < COLS; c += 256) {
    constexpr int W = 256;
    if (COLS - c >= W) umma(d + c, da, sdesc<ROW>(b + c * ROW), idesc_i8(W), acc);
    else umma(d + c, da, sdesc<ROW>(b + c * ROW), idesc_i8(COLS % W), acc);
  }
}
// All digit products with p + q < NG of one K step of 32: A digit p against B digits
// 0 .. NG - p - 1, into groups p and up.  `init` starts the accumulators: every group is
// first written by p = 0.
template <class F, int P>
__device__ __forceinline__ void umma_digits(uint32_t tmem, uint32_t a, uint32_t b, bool init) {
  if constexpr (P < F::NS) {
    umma_row<(F::NG - P) * F::TN, F::TK>(tmem + P * F::TN, sdesc<F::TK>(a + P * TM * F::TK), b,
                                         P == 0 && init ? 0u : 1u);
    umma_digits<F, P + 1>(tmem, a, b, init);
  }
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
               ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int (&r)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// The power of two of a packed row or column, NaN where it held a non-finite element.
__device__ __forceinline__ double row_scale(double alpha, int e, int shift) {
  if (e == EXP_NONFINITE) return __longlong_as_double(0x7ff8000000000000ll);
  return alpha * pow2i(e - shift);
}
// Four groups of neighbouring weight 2^-8 as one exact integer, in units of the last.
__device__ __forceinline__ long long combine4(int g0, int g1, int g2, int g3) {
  return ((static_cast<long long>(g0) * 256 + g1) * 256 + g2) * 256 + g3;
}
// Store of NB output elements, C = v + beta C.  Every element of an output has one writer
// per launch, so C += v (beta = 1, what nearly every accumulating contraction asks) goes
// out as a reduction that L2 performs: the same rounding and order as load, add, store,
// without the load's latency on the storing warp (7168 x 7168 x 288: 0.61 -> 0.51 ms in
// seven digits, 0.52 -> 0.37 ms in four; 8192 x 8192 x 1024 in four 0.89 -> 0.69 ms).
// Another beta loads every old value before the first store, so the NB reads are in flight
// together (a store followed by a load through another pointer would serialise them).
template <int NB>
__device__ __forceinline__ void store_out(double* const (&ptr)[NB], const double (&v)[NB],
                                          double beta) {
  if (beta == 1.0) {
#pragma unroll
    for (int j = 0; j < NB; ++j)
      if (ptr[j]) atomicAdd(ptr[j], v[j]);
  } else if (beta != 0.0) {
    double old[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) old[j] = ptr[j] ? *ptr[j] : 0.0;
#pragma unroll
    for (int j = 0; j < NB; ++j)
      if (ptr[j]) *ptr[j] = v[j] + beta * old[j];
  } else {
#pragma unroll
    for (int j = 0; j < NB; ++j)
      if (ptr[j]) *ptr[j] = v[j];
  }
}

struct SplitParams {
  int64_t M, N, K;                 // logical extents
  int64_t Kp;                      // packed K (a multiple of KPAD)
  int nkb;                         // k-blocks of TK
  Ax Cm, Cn, C2m, C2n;
  double* C; double* C2;
  double alpha, beta;
  const int* ea; const int* eb;    // exponents of the packed rows of A and of B
  int* error;
  const unsigned char* map;  // refused 64 x 64 blocks of the output, [ceil(M / 64)][map_ld]
  const int* any;            // (null: none), and whether there are some
  int64_t map_ld;
  __device__ __forceinline__ bool refused(int64_t m, int64_t n) const {
    return map && m < M && map[(m >> 6) * map_ld + (n >> 6)] != 0;
  }
  // nsplit ranges of kb_len k-blocks; range q stores at C + q part_stride.
  int nsplit, kb_len;
  int64_t part_stride;
  // Packed rows: logical row m of A is packed row
  //   a_base + (m / a_run) * a_stride + m % a_run,
  // and tiles never straddle a run (a_tiles tiles per run, nMt tile rows in all);
  // likewise n for B.  One run over the whole extent is the plain case.
  int64_t a_run, a_stride, a_base, a_tiles, nMt;
  int64_t b_run, b_stride, b_base, b_tiles, nNt;
};

// Tile t in the grouped raster order: logical origins (m0, n0), packed-row origins
// (pa, pb) and the valid extents (mlim, nlim) of the tile.
struct TileAt {
  int64_t m0, n0, pa, pb;
  int mlim, nlim;
  int kb0, nkb;     // k-blocks of the work item (none if the whole tile is refused)
  int64_t out;      // offset of its output
};
// (32-bit arithmetic: every role divides its way here once per tile, and a 64-bit division
// is a call of some hundred instructions; tiles and work items stay below 2^31.)
template <int TN>
__device__ __forceinline__ TileAt tile_at(const SplitParams& p, uint32_t t) {
  TileAt a;
  const uint32_t nM = static_cast<uint32_t>(p.nMt), nN = static_cast<uint32_t>(p.nNt);
  const uint32_t tiles = nM * nN, part = p.nsplit > 1 ? t / tiles : 0;
  t -= part * tiles;
  a.kb0 = static_cast<int>(part) * p.kb_len;
  a.nkb = min(p.kb_len, p.nkb - a.kb0);
  a.out = part * p.part_stride;
  const uint32_t per_group = RASTER_M * nN, group = t / per_group;
  const uint32_t first = group * RASTER_M;
  const uint32_t rows = nM - first < RASTER_M ? nM - first : RASTER_M;
  const uint32_t in = t - group * per_group;
  const uint32_t tn = in / rows, tm = first + in - tn * rows;
  const uint32_t at = static_cast<uint32_t>(p.a_tiles), bt = static_cast<uint32_t>(p.b_tiles);
  const uint32_t rm = tm / at, om = (tm - rm * at) * TM;
  const uint32_t rn = tn / bt, on = (tn - rn * bt) * TN;
  a.m0 = rm * p.a_run + om;
  a.n0 = rn * p.b_run + on;
  a.pa = p.a_base + rm * p.a_stride + om;
  a.pb = p.b_base + rn * p.b_stride + on;
  const int64_t ml = min(p.a_run - om, p.M - a.m0), nl = min(p.b_run - on, p.N - a.n0);
  a.mlim = static_cast<int>(ml < 0 ? 0 : (ml > TM ? TM : ml));
  a.nlim = static_cast<int>(nl < 0 ? 0 : (nl > TN ? TN : nl));
  if (p.refused(a.m0, a.n0) && (a.m0 + 64 >= p.M || p.refused(a.m0 + 64, a.n0))) a.nkb = 0;
  return a;
}

template <class F>
__global__ void __launch_bounds__(320)
split_kernel_persistent(const __grid_constant__ CUtensorMap tmA,
                        const __grid_constant__ CUtensorMap tmB, SplitParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  constexpr int TN = F::TN, TK = F::TK, NST = F::NST, STAGE = stage_bytes<F>();
  constexpr int COLS = TN / 2;  // columns of one epilogue warp
  double* wbufs = reinterpret_cast<double*>(base + NST * STAGE);
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + NST * STAGE + 8 * WBUF_DOUBLES * 8);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * NST + 2);
  __shared__ int abort_flag;
  volatile int* abort_v = &abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ntiles = static_cast<uint32_t>(p.nMt * p.nNt * p.nsplit);
  if (p.map && *p.any == 0) p.map = nullptr;
  constexpr int KB_PER_CHUNK = KCHUNK / TK;
  auto chunks_of = [](int nkb) { return (nkb + KB_PER_CHUNK - 1) / KB_PER_CHUNK; };

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < NST; ++s) {
      mbar_init(smem_u32(&bars[s]), 1);
      mbar_init(smem_u32(&bars[NST + s]), 1);
    }
    mbar_init(smem_u32(&bars[2 * NST]), 1);
    mbar_init(smem_u32(&bars[2 * NST + 1]), 256);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                 ::"r"(smem_u32(tmem_slot)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    // ---- TMA producer: every k-block of every tile of this CTA ----
    uint32_t it = 0;
    for (uint32_t t = blockIdx.x; t < ntiles && !*abort_v; t += gridDim.x) {
      const TileAt ta = tile_at<TN>(p, t);
      for (int kb = ta.kb0; kb < ta.kb0 + ta.nkb; ++kb, ++it) {
        const int s = it % NST;
        if (it >= NST && !mbar_wait(smem_u32(&bars[NST + s]), ((it / NST) - 1) & 1)) {
          atomicExch(&abort_flag, 1);
          break;
        }
        if (*abort_v) break;
        const uint32_t full = smem_u32(&bars[s]);
        mbar_expect_tx(full, STAGE);
        unsigned char* st = base + s * STAGE;
        tma_load_3d(smem_u32(st), &tmA, full, kb * TK, static_cast<int>(ta.pa), 0);
        tma_load_3d(smem_u32(st + a_bytes<F>()), &tmB, full, kb * TK, static_cast<int>(ta.pb), 0);
      }
    }
  } else if (warp == 1 && lane == 0) {
    // ---- MMA issuer: chunks of all tiles, global stage and chunk counters ----
    uint32_t it = 0, q = 0;
    for (uint32_t t = blockIdx.x; t < ntiles && !*abort_v; t += gridDim.x) {
      const TileAt ta = tile_at<TN>(p, t);
      const int nchunks = chunks_of(ta.nkb), kb_last = ta.kb0 + ta.nkb;
      int kb = ta.kb0;
      for (int c = 0; c < nchunks && !*abort_v; ++c, ++q) {
        if (q > 0 && !mbar_wait(smem_u32(&bars[2 * NST + 1]), (q - 1) & 1)) {
          atomicExch(&abort_flag, 1);
          break;
        }
        tc_fence_after();
        const int kb_end = min(kb_last, kb + KB_PER_CHUNK);
        bool first = true;
        for (; kb < kb_end; ++kb, ++it) {
          const int s = it % NST;
          if (!mbar_wait(smem_u32(&bars[s]), (it / NST) & 1)) { atomicExch(&abort_flag, 1); break; }
          tc_fence_after();
          const uint32_t st = smem_u32(base + s * STAGE);
#pragma unroll
          for (int kk = 0; kk < TK; kk += KPAD)
            if (kb * TK + kk < p.Kp)  // the last k-block may be a half one
              umma_digits<F, 0>(tmem, st + kk, st + a_bytes<F>() + kk, first && kk == 0);
          umma_commit(smem_u32(&bars[NST + s]));
          first = false;
        }
        umma_commit(smem_u32(&bars[2 * NST]));
      }
    }
  } else if (warp >= 2) {
    // ---- epilogue: per tile, FP64 accumulation of every chunk, then the store ----
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row = quad * 32 + lane;
    double* wb = wbufs + (warp - 2) * WBUF_DOUBLES;
    const bool m_major = p.Cm.s_i == 1 && p.Cm.inner > 1;  // output contiguous along rows
    uint32_t q = 0;
    for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
      if (__any_sync(0xffffffffu, *abort_v != 0)) break;
      const TileAt ta = tile_at<TN>(p, t);
      const int64_t m0 = ta.m0, n0 = ta.n0;
      double acc[COLS];  // in units of the fourth group
#pragma unroll
      for (int j = 0; j < COLS; ++j) acc[j] = 0.0;
      bool ok = true;
      const int nchunks = chunks_of(ta.nkb);
      for (int c = 0; c < nchunks; ++c, ++q) {
        const bool got = mbar_wait(smem_u32(&bars[2 * NST]), q & 1);
        if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int cb = 0; cb < COLS; cb += 8) {
          const uint32_t taddr = tmem + (static_cast<uint32_t>(quad * 32) << 16) +
                                 static_cast<uint32_t>(COLS * half + cb);
          int g[F::NG][8];
#pragma unroll
          for (int w = 0; w < F::NG; ++w) tmem_ld8(taddr + w * TN, g[w]);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            double x = static_cast<double>(combine4(g[0][j], g[1][j], g[2][j], g[3][j]));
            if constexpr (F::NG == 8)
              x = fma(static_cast<double>(combine4(g[4][j], g[5][j], g[6][j], g[7][j])), 0x1p-32, x);
            acc[cb + j] += x;
          }
        }
        tc_fence_before();
        mbar_arrive(smem_u32(&bars[2 * NST + 1]));  // TMEM free: the next chunk may start
      }
      if (!ok) { atomicExch(&abort_flag, 1); break; }
      // store this warp's 32 rows x COLS columns (the MMA issuer is already on the next tile).
      // The offset of a row belongs to the lane of that row; the offset and the
      // power-of-two scale of a column are computed by one lane per group of 32 (or 16)
      // columns; both reach the lanes that store an element through warp shuffles
      // (offset -1: outside the output).
      if (nchunks == 0 || p.refused(m0 + (row & 64), n0)) continue;
      const int64_t m = m0 + row;
      const bool mv = row < ta.mlim;
      // acc counts 2^-36: digit 0 weighs 2^-6 in each operand, the fourth group 2^-24 of the first
      const double sa = mv ? row_scale(p.alpha, p.ea[ta.pa + row], 18) : 0.0;
      const int64_t rowoff = mv ? ta.out + p.Cm.off(static_cast<uint32_t>(m)) : -1;
      const int64_t rowoff2 = (mv && p.C2) ? p.C2m.off(static_cast<uint32_t>(m)) : -1;
      if (m_major) {
        // lanes are consecutive rows: store column by column straight from registers
#pragma unroll
        for (int h2 = 0; h2 < COLS / 32; ++h2) {
          const int jl = COLS * half + 32 * h2 + lane;  // this lane's column of the group
          const int64_t colL = jl < ta.nlim ? p.Cn.off(static_cast<uint32_t>(n0 + jl)) : -1;
          const double scL = jl < ta.nlim ? row_scale(1.0, p.eb[ta.pb + jl], 18) : 0.0;
#pragma unroll
          for (int j0 = 0; j0 < 32; j0 += 4) {
            double* ptr[4];
            double val[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int64_t col = __shfl_sync(0xffffffffu, colL, j0 + j);
              const double sc = __shfl_sync(0xffffffffu, scL, j0 + j);
              val[j] = acc[32 * h2 + j0 + j] * sa * sc;
              ptr[j] = (rowoff >= 0 && col >= 0) ? p.C + rowoff + col : nullptr;
            }
            store_out<4>(ptr, val, p.beta);
            if (p.C2) {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const int jc = COLS * half + 32 * h2 + j0 + j;
                ptr[j] = (rowoff2 >= 0 && jc < ta.nlim)
                             ? p.C2 + rowoff2 + p.C2n.off(static_cast<uint32_t>(n0 + jc)) : nullptr;
              }
              store_out<4>(ptr, val, p.beta);
            }
          }
        }
      } else {
        // 16-column pieces through the warp's buffer; lanes then run along columns
#pragma unroll
        for (int piece = 0; piece < COLS / 16; ++piece) {
          const int cc = lane & 15;  // this lane's column within the piece
          const int jn = COLS * half + 16 * piece + cc;
          const int64_t nn = n0 + jn;
          const int64_t cn = jn < ta.nlim ? p.Cn.off(static_cast<uint32_t>(nn)) : -1;
          const double scL = jn < ta.nlim ? row_scale(1.0, p.eb[ta.pb + jn], 18) : 0.0;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const double sc = __shfl_sync(0xffffffffu, scL, j);
            wb[lane * 16 + (j ^ (lane & 15))] = acc[16 * piece + j] * sa * sc;
          }
          __syncwarp();
#pragma unroll 1
          for (int k0 = 0; k0 < 16; k0 += 4) {
            double* ptr[4];
            double val[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int r = 2 * (k0 + k) + (lane >> 4);  // row within the warp
              const int64_t ro = __shfl_sync(0xffffffffu, rowoff, r);
              val[k] = wb[r * 16 + (cc ^ (r & 15))];
              ptr[k] = (ro >= 0 && cn >= 0) ? p.C + ro + cn : nullptr;
            }
            store_out<4>(ptr, val, p.beta);
            if (p.C2) {
              const int64_t cn2 = jn < ta.nlim ? p.C2n.off(static_cast<uint32_t>(nn)) : -1;
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const int r = 2 * (k0 + k) + (lane >> 4);
                const int64_t r2 = __shfl_sync(0xffffffffu, rowoff2, r);
                ptr[k] = (r2 >= 0 && cn2 >= 0) ? p.C2 + r2 + cn2 : nullptr;
              }
              store_out<4>(ptr, val, p.beta);
            }
          }
          __syncwarp();
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) atomicExch(p.error, 1);
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
  }
}

// C = sum over the k ranges, in order, + beta C (C2 likewise).
__global__ void __launch_bounds__(256) split_k_sum_kernel(SplitParams p, const double* part) {
  if (p.map && *p.any == 0) p.map = nullptr;
  const int64_t total = p.M * p.N;
  for (int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const uint32_t m = static_cast<uint32_t>(e / p.N), n = static_cast<uint32_t>(e - m * p.N);
    if (p.refused(m, n)) continue;
    double v = 0.0;
#pragma unroll 4
    for (int q = 0; q < p.nsplit; ++q) v += part[q * total + e];
    double* c = p.C + p.Cm.off(m) + p.Cn.off(n);
    *c = p.beta != 0.0 ? v + p.beta * *c : v;
    if (p.C2) {
      c = p.C2 + p.C2m.off(m) + p.C2n.off(n);
      *c = p.beta != 0.0 ? v + p.beta * *c : v;
    }
  }
}

// ---------------------------------------------------------------------------
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                              const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeFn>(p);
  });
  if (!fn) throw Error(ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  return fn;
}

// 3-D map over the digit planes [digits][Rp][Kp], box tk (k) x rows x digits, rows of
// tk bytes swizzled like the MMA descriptors expect.  Rows and k beyond the operand
// read zero.
CUtensorMap make_map(void* base, int digits, int64_t Rp, int64_t Kp, int tk, int rows) {
  CUtensorMap m;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(Kp), static_cast<cuuint64_t>(Rp),
                              static_cast<cuuint64_t>(digits)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(Kp), static_cast<cuuint64_t>(Kp * Rp)};
  const cuuint32_t box[3] = {static_cast<cuuint32_t>(tk), static_cast<cuuint32_t>(rows),
                             static_cast<cuuint32_t>(digits)};
  const cuuint32_t es[3] = {1, 1, 1};
  CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, es,
                           CU_TENSOR_MAP_INTERLEAVE_NONE,
                           tk == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                           : tk == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw Error(ERR_CUDA, "cuTensorMapEncodeTiled failed");
  return m;
}

inline int64_t rup(int64_t x, int64_t a) { return (x + a - 1) / a * a; }

int digits_of(const Contraction& g) { return g.digits == 8 ? 8 : 4; }

// Partials of the k ranges of a contraction packed over Kp.
int parts_of(const Contraction& g, int64_t Kp) {
  const int D = digits_of(g);
  return split_k_parts(rup(g.M, TM) / TM * (rup(g.N, tile_n(D)) / tile_n(D)), g.M, g.N, Kp, D);
}
size_t part_bytes(const Contraction& g, int64_t Kp) {
  const int n = parts_of(g, Kp);
  return n > 1 ? rup(n * g.M * g.N * 8, 1024) : 0;
}
// The most any panel of the contraction may need (a shorter panel may take more parts).
size_t part_bound(const Contraction& g, int64_t Kp) {
  const int64_t n = split_k_most(g.M, g.N, Kp);
  return n > 1 ? rup(n * g.M * g.N * 8, 1024) : 0;
}

// Metadata of `rows` packed rows: whether a block is refused and the maxima (cleared by every
// slicing), exponents and, in eight digits, profiles.
struct Meta {
  int* any;
  unsigned long long* rmax;
  int* exps;
  float* prof;
};
size_t meta_clear_bytes(int64_t rows) { return 8 + rows * 8; }
size_t meta_head_bytes(int64_t rows) { return rup(meta_clear_bytes(rows) + rows * 4, 1024); }
size_t meta_bytes(int64_t rows, int64_t Kp, int digits) {
  return meta_head_bytes(rows) + (digits == 8 ? rup(rows / PR * Kp * 4, 1024) : 0);
}
Meta meta_at(void* p, int64_t rows) {
  unsigned char* b = static_cast<unsigned char*>(p);
  Meta m;
  m.any = reinterpret_cast<int*>(b);
  m.rmax = reinterpret_cast<unsigned long long*>(b + 8);
  m.exps = reinterpret_cast<int*>(b + meta_clear_bytes(rows));
  m.prof = reinterpret_cast<float*>(b + meta_head_bytes(rows));
  return m;
}
// The map of refused blocks of an M x N output.
size_t map_bytes(int64_t M, int64_t N, int digits) {
  return digits == 8 ? rup(rup(M, PR) / PR * (rup(N, PR) / PR), 1024) : 0;
}

struct Layout2 {
  int64_t Mp, Np, Kp;
  size_t a_bytes, b_bytes, meta, map, part_bytes;
};
Layout2 layout_of(const Contraction& g) {
  const int D = digits_of(g);
  Layout2 L;
  L.Mp = rup(g.M, TM);
  L.Np = rup(g.N, tile_n(D));
  L.Kp = rup(std::max<int64_t>(g.K, 1), KPAD);
  L.a_bytes = rup(static_cast<int64_t>(D * L.Mp * L.Kp), 1024);
  L.b_bytes = rup(static_cast<int64_t>(D * L.Np * L.Kp), 1024);
  L.meta = meta_bytes(L.Mp + L.Np, L.Kp, D);
  L.map = map_bytes(g.M, g.N, D);
  L.part_bytes = part_bytes(g, L.Kp);
  return L;
}

PackArgs pack_args(const View& v, bool rows_are_m, const Contraction& g, int64_t R, int64_t Rp,
                   int64_t Kp, void* dst, const Meta& m, int64_t row0) {
  const int64_t Mi = g.Mi > 0 ? g.Mi : g.M, Ni = g.Ni > 0 ? g.Ni : g.N;
  const int64_t Ki = g.Ki > 0 ? g.Ki : std::max<int64_t>(g.K, 1);
  PackArgs a;
  a.src = v.p;
  if (rows_are_m) {  // A(m, k): rows = m (s_ro, s_ri), k = cols (s_co, s_ci)
    a.ar = mkax(Mi, v.s_ro, v.s_ri);
    a.ak = mkax(Ki, v.s_co, v.s_ci);
    a.r_contig = (v.s_ri == 1 && v.s_ci != 1) ? 1 : 0;
  } else {           // B(k, n): rows of the packed operand = n (s_co, s_ci), k = (s_ro, s_ri)
    a.ar = mkax(Ni, v.s_co, v.s_ci);
    a.ak = mkax(Ki, v.s_ro, v.s_ri);
    a.r_contig = (v.s_ci == 1 && v.s_ri != 1) ? 1 : 0;
  }
  a.R = R; a.K = g.K; a.Rp = Rp; a.Kp = Kp;
  a.rmax = m.rmax + row0; a.rexp = m.exps + row0; a.dst = static_cast<int8_t*>(dst);
  a.prof = m.prof + row0 / PR * Kp;
  a.K1 = a.K; a.off[0] = a.off[1] = 0; a.sign[0] = a.sign[1] = 1.0;
  if (Rp % PR || Kp % 16) throw Error(ERR_BAD_SHAPE, "gemm_split: packed extents not tiled");
  return a;
}

// Row maxima and digits of one to three operands, whose rows share one block of metadata of
// `rows` rows (cleared here).
void pack(const PackArgs* const* ops, int n, const Meta& m, int64_t rows, int digits,
          cudaStream_t s) {
  CC_CHECK(cudaMemsetAsync(m.any, 0, meta_clear_bytes(rows), s));
  PackSet pp;
  for (int k = 0; k < 3; ++k) pp.op[k] = *ops[std::min(k, n - 1)];
  // strips of k for the maxima: the longest of 128 .. 1024 that gives 148 x 6 work items
  int64_t kstrip = 1024;
  auto strips = [&](const PackArgs& x) { return (x.Rp / PR) * ((x.K + kstrip - 1) / kstrip); };
  auto tiles = [](const PackArgs& x) {
    const int kw = x.r_contig ? PK_R : PK_K;
    return (x.Rp / PR) * ((x.Kp + kw - 1) / kw);
  };
  auto items = [&](auto&& count) {
    int64_t t = 0;
    for (int k = 0; k < 3; ++k) pp.end[k] = static_cast<uint32_t>(t += k < n ? count(pp.op[k]) : 0);
    if (t >= (int64_t(1) << 31)) throw Error(ERR_BAD_SHAPE, "gemm_split: operand too large");
    return t;
  };
  int64_t work = items(strips);
  while (kstrip > 128 && work < 148 * 6) {
    kstrip /= 2;
    work = items(strips);
  }
  pack_max_kernel<<<static_cast<unsigned>(std::min<int64_t>(work, 148 * 8)), PTHREADS, 0, s>>>(
      pp, static_cast<int>(kstrip));
  CC_LAUNCH_CHECK();
  work = items(tiles);
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>(work, 148 * 8));
  if (digits == 8) pack_digits_kernel<8><<<grid, PTHREADS, 0, s>>>(pp);
  else pack_digits_kernel<4><<<grid, PTHREADS, 0, s>>>(pp);
  CC_LAUNCH_CHECK();
  g_pack_launches.fetch_add(2);
}
void pack_one(const PackArgs& a, const Meta& m, int64_t rows, int digits, cudaStream_t s) {
  const PackArgs* op = &a;
  pack(&op, 1, m, rows, digits, s);
}

// The refused blocks of an M x N output from the profiles of its operands.
void profiles(const float* A, const float* B, int64_t M, int64_t N, int64_t K, int64_t Kp,
              unsigned char* map, int* any, cudaStream_t s) {
  const int64_t nI = rup(M, PR) / PR, nJ = rup(N, PR) / PR, work = nI * ((nJ + 3) / 4);
  int threads = 32;  // more warps share k where there are few pairs of blocks
  while (threads < 1024 && work * threads < 148 * 2048 && threads * 4 < Kp) threads *= 2;
  profile_kernel<<<static_cast<unsigned>(std::min<int64_t>(work, 148 * 32)), threads, 0, s>>>(
      A, B, nI, nJ, Kp, split_profile_least(K), map, any);
  CC_LAUNCH_CHECK();
  g_pack_launches.fetch_add(1);
}

// Packed slices of both operands are limited to this many bytes: a longer K is
// cut into panels (multiples of KCHUNK where possible), each packed and
// multiplied in turn and accumulated into C in FP64.
constexpr size_t kPanelBytes = size_t(3) << 30;  // 3 GiB: one panel for the ladder contractions

// CC4S_SPLIT_PANEL_BYTES (at least 1 MiB) overrides the limit, e.g. to trade
// scratch memory for fewer, longer panels.
size_t panel_bytes() {
  if (const char* e = std::getenv("CC4S_SPLIT_PANEL_BYTES")) {
    const long long v = std::atoll(e);
    if (v >= (1ll << 20)) return static_cast<size_t>(v);
  }
  return kPanelBytes;
}

int64_t panel_len(const Contraction& g) {
  const int D = digits_of(g);
  const int64_t per_k = D * (rup(g.M, TM) + rup(g.N, tile_n(D)));  // bytes per k
  int64_t P = static_cast<int64_t>(panel_bytes()) / per_k;
  if (P >= KCHUNK) P = P / KCHUNK * KCHUNK;
  else P = std::max<int64_t>(2 * KPAD, P / KPAD * KPAD);
  return P;
}

struct Panel { int64_t k0, kl, ki, a_off, b_off; };

// K panels of length <= P.  A two-level K index (inner extent Ki) is cut either
// into groups of whole inner runs (Ki <= P) or inside each run (Ki > P); the
// operand views are shifted to the panel start.
std::vector<Panel> panels_of(const Contraction& g, int64_t P) {
  std::vector<Panel> out;
  const int64_t K = g.K, Ki = g.Ki > 0 ? g.Ki : K;
  if (K <= P) {
    out.push_back({0, K, g.Ki, 0, 0});
  } else if (Ki >= K) {
    for (int64_t k0 = 0; k0 < K; k0 += P)
      out.push_back({k0, std::min(P, K - k0), 0, k0 * g.A.s_ci, k0 * g.B.s_ri});
  } else if (Ki <= P) {
    const int64_t runs = P / Ki;
    for (int64_t q0 = 0; q0 * Ki < K; q0 += runs)
      out.push_back({q0 * Ki, std::min(runs * Ki, K - q0 * Ki), Ki, q0 * g.A.s_co, q0 * g.B.s_ro});
  } else {
    for (int64_t q = 0; q * Ki < K; ++q)
      for (int64_t r0 = 0; r0 < Ki && q * Ki + r0 < K; r0 += P)
        out.push_back({q * Ki + r0, std::min(std::min(P, Ki - r0), K - q * Ki - r0), 0,
                       q * g.A.s_co + r0 * g.A.s_ci, q * g.B.s_ro + r0 * g.B.s_ri});
  }
  return out;
}

void split_panel(const Contraction& g, cudaStream_t s, SplitScratch& ws,
                 const SplitPackedB* pb = nullptr);

}  // namespace

// FP64 contractions: the eight-digit form where its time (launches, slicing at 24 bytes per
// element, waves of one tile per SM) is below the FP64 tensor pipe's.  The constants follow
// measured contractions that accumulate (FP64 pipe, eight digits, us): 512 x 512 x 512 31 and
// 54, 1024 x 1024 x 256 47 and 46, x 1024 107 and 65; 128 x 8192 x 1024 108 and 126,
// 64 x 32768 x 1024 184 and 376 (slicing of an operand used 64 times), 1067 x 1067 x 512 68
// and 64, 2048 x 2048 x 256 157 and 75, 256 x 256 x 16384 112 and 139; complex, four real
// ones and the digit form: 512 x 512 x 256 82 and 91, 512 x 512 x 512 122 and 114,
// 1024 x 1024 x 64 64 and 67, x 256 186 and 86, 64 x 32768 x 1024 737 and 944.
bool digits8_pays(const Contraction& c, bool cplx) {
  if (c.batch != 1 || c.M < 64 || c.N < 64 || c.K * (cplx ? 2 : 1) < 64) return false;
  const double M = double(c.M), N = double(c.N), K = double(c.K), P = cplx ? 2.0 : 1.0;
  auto up = [](double x, double t) { return std::ceil(x / t) * t; };
  const double tiles = up(M, 128) * up(N, 64) / (128 * 64);
  const double rows = cplx ? M + N + std::min(M, N) : M + N;
  const int parts = split_k_parts(static_cast<int64_t>(tiles), c.M, c.N, c.K * (cplx ? 2 : 1), 8);
  const double d8 = (cplx ? 58.0 : 36.0) + 24.0 * rows * P * K / 3.5e6 +
                    P * ((parts > 1 ? 6.0 : 0.0) +
                         std::ceil(tiles * parts / 148.0) * (3.3 + 0.021 * up(P * K, 32) / parts));
  // (outputs beyond 2^22 elements no longer stay in L2 between their load and their store)
  const double dmma = P * P * (15.0 + 2.0 * up(M, 64) * up(N, 64) * K / 24.5e6 +
                               std::max(0.0, M * N - 4194304.0) / 1.6e5);
  return d8 < dmma;
}

uint64_t split_launch_count() { return g_split_launches.load(); }
uint64_t split_pack_launch_count() { return g_pack_launches.load(); }

size_t gemm_split_scratch_bytes(const Contraction& g) {
  Contraction h = g;
  h.K = std::min(g.K, panel_len(g));
  const Layout2 L = layout_of(h);
  return L.a_bytes + L.b_bytes + L.meta + L.map + part_bound(g, L.Kp);
}

size_t split_packed_b_bytes(const Contraction& g) {
  const Layout2 L = layout_of(g);
  return L.b_bytes + meta_bytes(L.Np, L.Kp, digits_of(g));
}

size_t split_scratch_bytes_packed_b(const Contraction& g) {
  const Layout2 L = layout_of(g);
  return L.a_bytes + L.meta + L.map + part_bound(g, L.Kp);
}

bool split_single_panel(const Contraction& g) { return g.K <= panel_len(g) && g.batch == 1; }

SplitPackedB split_pack_b(const Contraction& g, void* dst, cudaStream_t s) {
  if (!split_single_panel(g)) throw Error(ERR_UNSUPPORTED, "split_pack_b: K beyond one panel");
  const Layout2 L = layout_of(g);
  unsigned char* p = static_cast<unsigned char*>(dst);
  SplitPackedB b;
  b.slices = p;
  const Meta m = meta_at(p + L.b_bytes, L.Np);
  b.exps = m.exps;
  b.N = g.N; b.K = g.K; b.Np = L.Np; b.Kp = L.Kp; b.digits = digits_of(g);
  b.prof = m.prof;
  pack_one(pack_args(g.B, false, g, g.N, L.Np, L.Kp, b.slices, m, 0), m, L.Np, b.digits, s);
  return b;
}

void gemm_split_packed_b(const Contraction& g, const SplitPackedB& b, cudaStream_t s,
                         SplitScratch& ws) {
  if (g.M <= 0 || g.N <= 0) return;
  if (!split_single_panel(g)) throw Error(ERR_UNSUPPORTED, "gemm_split_packed_b: K beyond one panel");
  split_panel(g, s, ws, &b);
}

void gemm_split(const Contraction& g, cudaStream_t s, SplitScratch& ws) {
  if (g.M <= 0 || g.N <= 0) return;
  if (g.batch != 1) throw Error(ERR_UNSUPPORTED, "gemm_split: batched contraction");
  if (g.K <= 0) throw Error(ERR_UNSUPPORTED, "gemm_split: empty K");
  const std::vector<Panel> ps = panels_of(g, panel_len(g));
  for (size_t i = 0; i < ps.size(); ++i) {
    Contraction h = g;
    h.K = ps[i].kl;
    h.Ki = ps[i].ki;
    h.A.p = g.A.p + ps[i].a_off;
    h.B.p = g.B.p + ps[i].b_off;
    if (i > 0) h.beta = 1.0;
    split_panel(h, s, ws);
  }
}

namespace {

template <class F>
void launch_form(const CUtensorMap& ta, const CUtensorMap& tb, SplitParams sp, double* part,
                 cudaStream_t s) {
  static std::atomic<int> sms{0};
  int n = sms.load();
  if (!n) {
    int dev = 0;
    CC_CHECK(cudaGetDevice(&dev));
    CC_CHECK(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    CC_CHECK(cudaFuncSetAttribute(split_kernel_persistent<F>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<F>()));
    sms.store(n);
  }
  sp.nkb = static_cast<int>((sp.Kp + F::TK - 1) / F::TK);
  sp.kb_len = sp.nkb;
  sp.part_stride = 0;
  SplitParams out = sp;
  if (part) {
    sp.kb_len = (sp.nkb + sp.nsplit - 1) / sp.nsplit;
    sp.nsplit = (sp.nkb + sp.kb_len - 1) / sp.kb_len;
    out.nsplit = sp.nsplit;
    sp.part_stride = sp.M * sp.N;
    sp.C = part;
    sp.C2 = nullptr;
    sp.Cm = mkax(sp.M, 0, sp.N);
    sp.Cn = mkax(sp.N, 0, 1);
    sp.beta = 0.0;
  }
  const dim3 grid(static_cast<unsigned>(std::min<int64_t>(sp.nMt * sp.nNt * sp.nsplit, n)));
  split_kernel_persistent<F><<<grid, 320, smem_bytes<F>(), s>>>(ta, tb, sp);
  CC_LAUNCH_CHECK();
  g_split_launches.fetch_add(1);
  if (part) {
    split_k_sum_kernel<<<grid_for(out.M * out.N, 256), 256, 0, s>>>(out, part);
    CC_LAUNCH_CHECK();
    g_split_launches.fetch_add(1);
  }
}

// The output side of a contraction and the runs of its packed rows -> one launch, or with
// room for partials (part_bytes) one launch over the k ranges and their sum; of the
// blocks that the contraction's map does not leave to gemm().
void launch(const Contraction& g, int digits, void* Apk, const int* ea, int64_t Ap,
            const SplitRuns& ar, int64_t nra, void* Bpk, const int* eb, int64_t Bp,
            const SplitRuns& br, int64_t nrb, int64_t Kp, double* part, cudaStream_t s,
            SplitScratch& ws) {
  const int tn = tile_n(digits), tk = digits == 8 ? Form<8>::TK : Form<4>::TK;
  const CUtensorMap ta = make_map(Apk, digits, Ap, Kp, tk, TM);
  const CUtensorMap tb = make_map(Bpk, digits, Bp, Kp, tk, tn);
  const int64_t Mi = g.Mi > 0 ? g.Mi : g.M, Ni = g.Ni > 0 ? g.Ni : g.N;
  SplitParams sp;
  sp.M = g.M; sp.N = g.N; sp.K = g.K; sp.Kp = Kp; sp.nkb = 0;
  sp.Cm = mkax(Mi, g.C.s_ro, g.C.s_ri);
  sp.Cn = mkax(Ni, g.C.s_co, g.C.s_ci);
  sp.C2m = mkax(Mi, g.C2.s_ro, g.C2.s_ri);
  sp.C2n = mkax(Ni, g.C2.s_co, g.C2.s_ci);
  sp.C = g.C.p; sp.C2 = g.C2.p;
  sp.alpha = g.alpha; sp.beta = g.beta;
  sp.ea = ea; sp.eb = eb;
  sp.error = ws.error;
  sp.map = g.only; sp.any = g.only_any;
  sp.map_ld = g.only_ld;
  sp.nsplit = part ? parts_of(g, Kp) : 1;
  sp.a_run = ar.run; sp.a_stride = ar.stride; sp.a_base = ar.base;
  sp.a_tiles = (ar.run + TM - 1) / TM; sp.nMt = nra * sp.a_tiles;
  sp.b_run = br.run; sp.b_stride = br.stride; sp.b_base = br.base;
  sp.b_tiles = (br.run + tn - 1) / tn; sp.nNt = nrb * sp.b_tiles;
  if (sp.nMt * sp.nNt * sp.nsplit >= (int64_t(1) << 31) || Ap >= (int64_t(1) << 31) ||
      Bp >= (int64_t(1) << 31) || Kp >= (int64_t(1) << 31))
    throw Error(ERR_BAD_SHAPE, "gemm_split: extent too large");
  if (digits == 8) launch_form<Form<8>>(ta, tb, sp, part, s);
  else launch_form<Form<4>>(ta, tb, sp, part, s);
}

void split_panel(const Contraction& g, cudaStream_t s, SplitScratch& ws, const SplitPackedB* pb) {
  const Layout2 L = layout_of(g);
  const int D = digits_of(g);
  // with a pre-packed B the scratch holds A and the metadata only
  const size_t base = L.a_bytes + (pb ? 0 : L.b_bytes) + L.meta + L.map;
  if (base + L.part_bytes > ws.bytes)
    throw Error(ERR_OUT_OF_MEMORY, "gemm_split: scratch too small");
  unsigned char* p = static_cast<unsigned char*>(ws.p);
  void* Apk = p;
  void* Bpk = p + L.a_bytes;
  unsigned char* meta = p + L.a_bytes + (pb ? 0 : L.b_bytes);
  const Meta m = meta_at(meta, L.Mp + L.Np);
  const int* bexp = m.exps + L.Mp;
  const float* bprof = m.prof + L.Mp / PR * L.Kp;
  const PackArgs pa = pack_args(g.A, true, g, g.M, L.Mp, L.Kp, Apk, m, 0);
  if (pb) {   // B sliced before, by split_pack_b, for this N, K and padding
    if (pb->N != g.N || pb->K != g.K || pb->Np != L.Np || pb->Kp != L.Kp || pb->digits != D)
      throw Error(ERR_INVALID_ARGUMENT, "gemm_split: pre-packed B of another shape");
    Bpk = pb->slices;
    bexp = pb->exps;
    bprof = pb->prof;
    pack_one(pa, m, L.Mp, D, s);
  } else {
    const PackArgs pbk = pack_args(g.B, false, g, g.N, L.Np, L.Kp, Bpk, m, L.Mp);
    const PackArgs* both[2] = {&pa, &pbk};
    pack(both, 2, m, L.Mp + L.Np, D, s);
  }
  Contraction h = g;
  if (D == 8) {
    unsigned char* map = meta + L.meta;
    profiles(m.prof, bprof, g.M, g.N, g.K, L.Kp, map, m.any, s);
    h.only = map;
    h.only_any = m.any;
    h.only_ld = rup(g.N, PR) / PR;
  }
  SplitRuns ar, br;
  ar.run = g.M;
  br.run = g.N;
  double* part = L.part_bytes ? reinterpret_cast<double*>(p + base) : nullptr;
  launch(h, D, Apk, m.exps, L.Mp, ar, 1, Bpk, bexp, L.Np, br, 1, L.Kp, part, s, ws);
  if (D == 8) gemm(h, s, ws.fp64);
}

}  // namespace
namespace {
// Scratch of one complex panel: the operand with more rows as one form of K' = 2 K, the
// other as two.
struct ComplexLayout {
  int64_t Mp, Np, Kp;
  int na, nb;            // forms of A and of B
  size_t a_bytes, b_bytes, meta, map, part_bytes;  // slices per form, meta of all, map per plane
};
ComplexLayout complex_layout(const Contraction& g, int64_t K) {
  const int D = digits_of(g);
  ComplexLayout L;
  L.Mp = rup(g.M, TM);
  L.Np = rup(g.N, tile_n(D));
  L.Kp = rup(2 * std::max<int64_t>(K, 1), KPAD);
  L.na = g.M < g.N ? 2 : 1;
  L.nb = 3 - L.na;
  L.a_bytes = rup(D * L.Mp * L.Kp, 1024);
  L.b_bytes = rup(D * L.Np * L.Kp, 1024);
  L.meta = meta_bytes(L.na * L.Mp + L.nb * L.Np, L.Kp, D);
  L.map = map_bytes(g.M, g.N, D);
  L.part_bytes = part_bytes(g, L.Kp);
  return L;
}
int64_t complex_panel_len(const Contraction& g) {
  const ComplexLayout L = complex_layout(g, 1);
  const int64_t per_k = 2 * digits_of(g) * (L.na * L.Mp + L.nb * L.Np);
  const int64_t P = static_cast<int64_t>(panel_bytes()) / per_k;
  return std::max<int64_t>(KPAD, P / KPAD * KPAD);
}
size_t complex_bytes(const ComplexLayout& L) {
  return L.na * L.a_bytes + L.nb * L.b_bytes + L.meta + 2 * L.map + L.part_bytes;
}
}  // namespace

size_t gemm_split_complex_scratch_bytes(const Contraction& g) {
  const ComplexLayout L = complex_layout(g, std::min(g.K, complex_panel_len(g)));
  return complex_bytes(L) - L.part_bytes + part_bound(g, L.Kp);
}

void gemm_split_complex(const Contraction& g, int64_t a_im, int64_t b_im, int64_t c_im, bool conjA,
                        bool conjB, cudaStream_t s, SplitScratch& ws) {
  if (g.M <= 0 || g.N <= 0) return;
  if (g.batch != 1) throw Error(ERR_UNSUPPORTED, "gemm_split_complex: batched contraction");
  if (g.K <= 0) throw Error(ERR_UNSUPPORTED, "gemm_split_complex: empty K");
  const int D = digits_of(g);
  const double sA = conjA ? -1.0 : 1.0, sB = conjB ? -1.0 : 1.0;
  for (const Panel& pn : panels_of(g, complex_panel_len(g))) {
    Contraction h = g;
    h.K = pn.kl;
    h.Ki = pn.ki;
    h.A.p = g.A.p + pn.a_off;
    h.B.p = g.B.p + pn.b_off;
    if (pn.k0 > 0) h.beta = 1.0;
    const ComplexLayout L = complex_layout(h, h.K);
    if (complex_bytes(L) > ws.bytes)
      throw Error(ERR_OUT_OF_MEMORY, "gemm_split_complex: scratch too small");
    unsigned char* p = static_cast<unsigned char*>(ws.p);
    const int64_t rows = L.na * L.Mp + L.nb * L.Np;
    const Meta m = meta_at(p + L.na * L.a_bytes + L.nb * L.b_bytes, rows);
    PackArgs op[3];
    const PackArgs* ops[3] = {&op[0], &op[1], &op[2]};
    int64_t r = 0;
    for (int k = 0; k < 3; ++k) {
      const bool isA = k < L.na;
      const int form = isA ? k : k - L.na;
      void* dst = isA ? p + k * L.a_bytes : p + L.na * L.a_bytes + form * L.b_bytes;
      op[k] = pack_args(isA ? h.A : h.B, isA, h, isA ? h.M : h.N, isA ? L.Mp : L.Np, L.Kp, dst,
                        m, r);
      r += isA ? L.Mp : L.Np;
      const int64_t im = isA ? a_im : b_im;
      op[k].K = 2 * h.K;
      op[k].K1 = h.K;
      op[k].off[1] = im;
      if ((isA ? L.na : L.nb) == 2) {
        // C_re = [Ar | Ai] [Br ; -sA sB Bi],  C_im = [Ar | Ai] [sB Bi ; sA Br], or the same
        // with the two forms on the A side: [Ar | -sA sB Ai], [sA Ai | sB Ar] on [Br ; Bi]
        if (form == 0) {
          op[k].sign[1] = -sA * sB;
        } else {
          op[k].off[0] = im;
          op[k].off[1] = 0;
          op[k].sign[0] = isA ? sA : sB;
          op[k].sign[1] = isA ? sB : sA;
        }
      }
    }
    pack(ops, 3, m, rows, D, s);
    unsigned char* maps = p + L.na * L.a_bytes + L.nb * L.b_bytes + L.meta;
    const int64_t map1 = static_cast<int64_t>(L.map);
    double* part_mem = L.part_bytes ? reinterpret_cast<double*>(maps + 2 * L.map) : nullptr;
    SplitRuns ar, br;
    ar.run = h.M;
    br.run = h.N;
    for (int part = 0; part < 2; ++part) {
      const PackArgs& A = op[L.na == 2 ? part : 0];
      const PackArgs& B = op[L.na + (L.nb == 2 ? part : 0)];
      Contraction c = h;
      c.K = 2 * h.K;
      if (part) {
        c.C.p = g.C.p + c_im;
        if (g.C2.p) c.C2.p = g.C2.p + c_im;
      }
      if (D == 8) {
        c.only = maps + part * map1;
        c.only_any = m.any;
        c.only_ld = rup(h.N, PR) / PR;
        profiles(A.prof, B.prof, h.M, h.N, c.K, L.Kp, maps + part * map1, m.any, s);
      }
      launch(c, D, A.dst, A.rexp, L.Mp, ar, 1, B.dst, B.rexp, L.Np, br, 1, L.Kp,
             part_mem, s, ws);
    }
    // The refused blocks: Re A and then Im A on both planes of B, the planes of the output
    // as a batch of two.
    for (int term = 0; D == 8 && term < 2; ++term) {
      Contraction c = h;
      c.batch = 2;
      c.A.s_bi = c.A.s_bo = 0;
      if (term) c.A.p += a_im;
      if (term) c.B.p += b_im;
      c.B.s_bi = term ? -b_im : b_im;
      c.C.s_bi = c.C2.s_bi = c_im;
      c.alpha1 = c.alpha * (term ? sA : sB);
      if (term) c.alpha *= -sA * sB;
      if (term) c.beta = 1.0;
      c.only = maps;
      c.only_any = m.any;
      c.only_ld = rup(h.N, PR) / PR;
      c.only_bs = map1;
      gemm(c, s, ws.fp64);
    }
  }
}

size_t split_operand_bytes(int64_t R, int64_t K, int digits) {
  const int64_t Rp = rup(std::max<int64_t>(R, 1), TM), Kp = rup(std::max<int64_t>(K, 1), KPAD);
  return static_cast<size_t>(rup(digits * Rp * Kp, 1024)) + meta_bytes(Rp, Kp, digits);
}

SplitOperand split_pack_operand(const double* src, int64_t R, int64_t Ri, int64_t s_ro,
                                int64_t s_ri, int64_t K, int64_t s_k, void* dst, cudaStream_t s,
                                int digits) {
  if (R <= 0 || K <= 0) throw Error(ERR_BAD_SHAPE, "split_pack_operand: empty operand");
  SplitOperand o;
  o.R = R; o.K = K; o.digits = digits;
  o.Rp = rup(R, TM);
  o.Kp = rup(K, KPAD);
  if (o.Rp >= (int64_t(1) << 31) || o.Kp >= (int64_t(1) << 31))
    throw Error(ERR_BAD_SHAPE, "split_pack_operand: extent too large");
  unsigned char* p = static_cast<unsigned char*>(dst);
  const int64_t sb = rup(digits * o.Rp * o.Kp, 1024);
  o.slices = p;
  const Meta m = meta_at(p + sb, o.Rp);
  o.exps = m.exps;
  o.prof = m.prof;
  Contraction g;
  g.M = R; g.Mi = Ri; g.K = K;
  g.A.p = const_cast<double*>(src);
  g.A.s_ro = s_ro; g.A.s_ri = s_ri; g.A.s_co = 0; g.A.s_ci = s_k;
  pack_one(pack_args(g.A, true, g, R, o.Rp, o.Kp, o.slices, m, 0), m, o.Rp, digits, s);
  return o;
}

void split_refused(const SplitOperand& A, const SplitOperand& B, int* word, cudaStream_t s) {
  if (A.digits != 8 || B.digits != 8 || A.K != B.K)
    throw Error(ERR_INVALID_ARGUMENT, "split_refused: operands of another form");
  CC_CHECK(cudaMemsetAsync(word, 0, 8, s));
  profiles(A.prof, B.prof, A.R, B.R, A.K, A.Kp, nullptr, word, s);
}

void gemm_split_prepacked(const Contraction& g, const SplitOperand& A, const SplitRuns& ar,
                          const SplitOperand& B, const SplitRuns& br, cudaStream_t s,
                          SplitScratch& ws) {
  if (g.M <= 0 || g.N <= 0) return;
  if (A.K != g.K || B.K != g.K || A.Kp != B.Kp || A.digits != B.digits)
    throw Error(ERR_INVALID_ARGUMENT, "gemm_split_prepacked: operands of another K");
  // every packed row that a valid logical row reads lies inside the operand
  auto check = [](const SplitRuns& r, int64_t X, int64_t R, const char* what) {
    if (r.run <= 0 || r.base < 0 || r.stride < 0)
      throw Error(ERR_INVALID_ARGUMENT, std::string("gemm_split_prepacked: bad runs of ") + what);
    const int64_t nr = (X + r.run - 1) / r.run;
    const int64_t last = r.base + (nr - 1) * r.stride + std::min(r.run, X - (nr - 1) * r.run) - 1;
    const int64_t full_last = nr > 1 ? r.base + (nr - 2) * r.stride + r.run - 1 : -1;
    if (last >= R || full_last >= R)
      throw Error(ERR_INVALID_ARGUMENT, std::string("gemm_split_prepacked: runs of ") + what +
                                            " leave the operand");
    return nr;
  };
  const int64_t nra = check(ar, g.M, A.R, "A"), nrb = check(br, g.N, B.R, "B");
  launch(g, A.digits, A.slices, A.exps, A.Rp, ar, nra, B.slices, B.exps, B.Rp, br, nrb, A.Kp,
         nullptr, s, ws);
}

}  // namespace cc4s_b200
