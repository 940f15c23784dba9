// Complex GEMM on the B200's integer tensor cores, exact up to the rounding of
// its operands to fixed point (tcgen05 kind::i8 + TMA + TMEM).
//
//   C (m x n) = alpha A (m x k) B (k x n) + beta C     (complex64 / complex128, row views)
//
// Every row of A and every column of B is scaled by a power of two so that its
// 2-norm is at most 2^alpha and rounded to integers.  The integer product,
// |C_ij| <= |a_i| |b_j| <= 2^(2 alpha) by Cauchy-Schwarz, is computed modulo N
// pairwise coprime p <= 241 with 2^(2 alpha) < P / 2, P = prod p, and
// recovered by the Chinese remainder theorem (the residue scheme of Ozaki,
// Uchino and Imamura, "Ozaki scheme II", 2025).  All p have only prime factors
// = 1 mod 4, so w^2 = -1 has a solution modulo p and the complex product
// splits into TWO real ones: with u = re + w im and v = re - w im,
//   X = u(A) u(B),  Y = v(A) v(B),  re C = (X + Y) / 2,  im C = (X - Y) / (2 w)   (mod p).
// So a product takes 2 N int8 products with int32 accumulation, all exact:
//   complex64 : N = 7,  2 alpha = 53 (26-bit operands relative to the row norm)
//   complex128: N = 16, 2 alpha = 116 (58 bits: more than a double's 53)
// The rounding of the operands is the only error before the final rounding, and
// the result does not depend on any summation order.  The scaled norms lie in
// [2^(alpha - 1), 2^alpha] and every real component is rounded by at most half a
// unit, so |dC_ij| <= sqrt(2 k) 2^(1 - alpha) |a_i| |b_j| in the worst case, about
// 2^-alpha |a_i| |b_j| for roundings of random sign.  That is a bound in norms; an
// FMA product is bounded by sum_k |a_ik| |b_kj| instead, which is smaller where the
// large entries of a_i meet small ones of b_j.  A scaling of the operands does not
// blow the norms up: rows of A and columns of B have their own scales, and one
// along the summation index, (A D)(D^-1 B), is undone by powers of two
// (rns_balance).  Within a balanced vector, entries below 2^-4 (complex128; 2^-2
// complex64) of its norm still keep fewer bits than the type holds.
//
// Launches per product: rns_balance (powers of two along k), rns_split (scales
// and residue planes, K-major, of A and B), rns_gemm (2 N int8 products, residues
// of the accumulators), rns_merge (CRT, alpha, beta).
#include <algorithm>
#include <climits>
#include <cmath>
#include <cuda.h>
#include <type_traits>

#include "dense.cuh"

namespace bem200 {

namespace rns {

// ------------------------------------------------------------------ moduli
constexpr int kMaxMod = 16;
// pairwise coprime, every prime factor = 1 mod 4 (221 = 13 x 17, 205 = 5 x 41)
constexpr int kModuli[kMaxMod] = {241, 233, 229, 221, 205, 197, 193, 181, 173, 157, 149, 137, 113, 109, 101, 97};

template <typename C> struct Traits;
template <> struct Traits<float2> {
  static constexpr int N = 7;           // log2 P = 54.29
  static constexpr int kTwoAlpha = 53;
  static constexpr int kWords = 1;      // 32-bit words of an operand's base-256 digits
  static constexpr int kFrac = 2;       // 32-bit words of the CRT fractions
  static constexpr int kBlock = 6144;   // largest block of m and n per pass (workspace bound)
  static constexpr int kExpMax = 250;   // entries are scaled by at most 2^+-kExpMax, in two factors
};
template <> struct Traits<double2> {
  static constexpr int N = 16;          // log2 P = 117.68
  static constexpr int kTwoAlpha = 116;
  static constexpr int kWords = 2;
  static constexpr int kFrac = 3;
  static constexpr int kBlock = 3072;
  static constexpr int kExpMax = 2040;
};
// Largest k per pass: accumulators stay below 121^2 x 3072 < 2^25.5, where the
// FP32 quotient of the epilogue leaves residues of at most 126 (see there).
constexpr int kBlockK = 3072;

constexpr float kMagic = 12582912.0f;  // 1.5 2^23: a float this size holds its integer in the low mantissa bits

struct SplitMod {  // residues of an operand from its signed base-256 digits
  int32_t w[2];    // 256^l mod p, a signed byte per digit
  int32_t ww[2];   // w 256^l mod p (w^2 = -1)
  int32_t bias;    // bits of the float K = 256 p i near 1.5 2^23
  int32_t p;
  float pinv, c;   // 1 / p, kMagic - K / p
};
struct SplitTab { SplitMod mod[kMaxMod]; };
struct MergeMod {
  uint32_t u[3], v[3];  // CRT weights of X + Y and X - Y as fractions of P: little-endian words of 32 kFrac bits
};
struct MergeTab {
  MergeMod mod[kMaxMod];
  uint32_t u0[3], v0[3];  // minus the contribution of the byte offsets (256 per X + Y, 255 per X - Y)
  double scale;           // P 2^(-32 kFrac)
};
struct ModTab {
  int32_t p[kMaxMod];
  float pinv[kMaxMod];
};

struct Tables {
  SplitTab split;
  MergeTab merge;
  ModTab mod;
};

static int symmetric(int x, int p) {
  x %= p;
  if (x < 0) x += p;
  return 2 * x > p ? x - p : x;
}
static int invmod(int a, int p) {
  a %= p;
  if (a < 0) a += p;
  for (int x = 1; x < p; ++x)
    if (a * x % p == 1) return x;
  return 0;
}

template <typename C>
static Tables make_tables() {
  using T = Traits<C>;
  Tables t{};
  double P = 1.0;
  for (int i = 0; i < T::N; ++i) P *= kModuli[i];
  unsigned __int128 su = 0, sv = 0;
  for (int i = 0; i < T::N; ++i) {
    const int p = kModuli[i];
    int w = 1;
    while ((w * w + 1) % p) ++w;
    int pi = 1;  // P / p mod p
    for (int j = 0; j < T::N; ++j)
      if (j != i) pi = pi * kModuli[j] % p;
    const int q = invmod(pi, p);
    const int c1 = invmod(2, p) * q % p;          // (X + Y) c1 (P / p) is re C's CRT term
    const int c2 = invmod(2 * w % p, p) * q % p;  // (X - Y) c2 (P / p) is im C's
    SplitMod& s = t.split.mod[i];
    s.p = p;
    s.pinv = 1.0f / (float)p;
    const int K = (int)(12582912.0 / (256.0 * p) + 0.5) * 256 * p;
    s.bias = 0x4B000000 + (K - (1 << 23));
    s.c = 12582912.0f - (float)(K / p);
    int pw = 1;
    for (int l = 0; l < 8; ++l) {
      const int sh = 8 * (l & 3);
      s.w[l >> 2] |= (int32_t)((uint32_t)(symmetric(pw, p) & 0xff) << sh);
      s.ww[l >> 2] |= (int32_t)((uint32_t)(symmetric(pw * w, p) & 0xff) << sh);
      pw = pw * 256 % p;
    }
    MergeMod& g = t.merge.mod[i];
    const unsigned __int128 one = (unsigned __int128)1 << (32 * T::kFrac);
    const unsigned __int128 u = (one * c1 + p / 2) / p, v = (one * c2 + p / 2) / p;
    su += u;
    sv += v;
    for (int k = 0; k < T::kFrac; ++k) {
      g.u[k] = (uint32_t)(u >> (32 * k));
      g.v[k] = (uint32_t)(v >> (32 * k));
    }
    t.mod.p[i] = p;
    t.mod.pinv[i] = 1.0f / (float)p;
  }
  su = ~(su * 256) + 1;
  sv = ~(sv * 255) + 1;
  for (int k = 0; k < T::kFrac; ++k) {
    t.merge.u0[k] = (uint32_t)(su >> (32 * k));
    t.merge.v0[k] = (uint32_t)(sv >> (32 * k));
  }
  t.merge.scale = ldexp(P, -32 * T::kFrac);
  return t;
}

template <typename C>
static const Tables& tables() {
  static const Tables t = make_tables<C>();
  return t;
}

// ------------------------------------------------------------------ scales
// Exponent e of a vector's scale 2^e: the norm times 2^e is at most 2^alpha.
// kNonFinite marks a vector with an infinity or a NaN: its integers are 0 and
// its row or column of the product becomes NaN.
constexpr int kNonFinite = INT_MIN;

// norm^2 = ss of the vector times 2^d per entry
__device__ __forceinline__ int scale_exponent(double ss, int two_alpha) {
  if (!(ss < INFINITY)) return kNonFinite;
  return ss > 0.0 ? (two_alpha - 1 - ilogb(ss * (1.0 + 1e-12))) >> 1 : 0;  // floor; norm^2 < 2^(ilogb + 1)
}
// complex64: squares and their sums stay in the range of doubles
__device__ __forceinline__ void norm_add(float2 v, int d, double& ss) {
  const double x = v.x, y = v.y;
  ss = fma(fma(x, x, y * y), __hiloint2double((2 * d + 1023) << 20, 0), ss);  // a NaN entry stays in ss
}
__device__ __forceinline__ void norm_add(double2 v, int d, double& ss) {
  const double f = __hiloint2double((d + 1023) << 20, 0), x = v.x * f, y = v.y * f;
  ss = fma(x, x, fma(y, y, ss));
}
// complex128 squares out of range (or a vector of zeros): the norm taken again, kLowShift powers of two
// lower if the sum overflowed; where squares vanish, norm^2 <= 2 k max^2
constexpr int kLowShift = 600;
__device__ __forceinline__ bool norm_unsafe(float2*, double) { return false; }
__device__ __forceinline__ bool norm_unsafe(double2*, double ss) { return !(ss > 1e-270 && ss < 1e290); }
template <typename C>
__device__ __forceinline__ void norm_add_wide(C v, int d, bool low, double& mx, double& ss) {
  const double g = low ? __hiloint2double((1023 - kLowShift) << 20, 0) : 1.0, f = __hiloint2double((d + 1023) << 20, 0);
  const double x = fabs((double)v.x) * g * f, y = fabs((double)v.y) * g * f;
  mx = fmax(mx, fmax(x, y));
  ss = fma(x, x, fma(y, y, ss));
}
__device__ __forceinline__ int scale_exponent_wide(double mx, double ss, int k, bool low, int two_alpha) {
  if (!(ss >= 0.0) || !(mx < INFINITY)) return kNonFinite;
  if (!(mx > 0.0)) return 0;
  const int e2 = mx > 1e-140 && mx < 1e140 ? ilogb(ss * (1.0 + 1e-12)) : 2 * (ilogb(mx) + 1) + ilogb((double)(2 * k));
  return ((two_alpha - 1 - e2) >> 1) - (low ? kLowShift : 0);
}

// ------------------------------------------------------------------ residue planes
// x 2^e rounded to an integer, as signed base-256 digits: adding 128 to every
// digit below the top one and flipping its high bit back turns the bytes of
// the two's complement integer into digits in [-128, 127]
__device__ __forceinline__ void digits(float x, int e, int32_t (&d)[1]) {
  const int e1 = e >> 1, e2 = e - e1;
  const float s = x * __int_as_float((e1 + 127) << 23) * __int_as_float((e2 + 127) << 23);
  d[0] = (__float2int_rn(s) + 0x00808080) ^ 0x00808080;
}
__device__ __forceinline__ void digits(double x, int e, int32_t (&d)[2]) {
  const int e1 = e >> 1, e2 = e - e1;
  const double s = x * __hiloint2double((e1 + 1023) << 20, 0) * __hiloint2double((e2 + 1023) << 20, 0);
  const long long v = (__double2ll_rn(s) + 0x0080808080808080LL) ^ 0x0080808080808080LL;
  d[0] = (int32_t)v;
  d[1] = (int32_t)(v >> 32);
}

// ------------------------------------------------------------------ balance
// (A D)(D^-1 B) = A B for any diagonal D, but with D far from constant the large
// columns of A meet small rows of B, and scales taken from the norms leave few
// bits for the entries that make up the product.  So column k of A is multiplied
// by 2^d[k] and row k of B by 2^-d[k], d[k] half the difference of their mean
// exponents over 32 rows of A and 32 columns of B (evenly spaced over all of
// them; zeros and non-finite entries do not count).  A diagonal scaling of
// either operand shows in every row and column and shifts these means exactly;
// the means are little moved by the peaks of single entries, so that operands
// without a grading stay as they are to within a bit.  A k without an entry in
// the sample takes the mean over 32 other k.  One CTA per 32 k; 3 to 4 us, latency
// bound.  (Exact column and row maxima recorded by the split, and a second split
// where they differ, cost 9 - 25 % of a solve: the maxima of BEM blocks differ by
// 5 to 10 bits along k through single entries.)
constexpr int kSample = 32;

// exponent of the larger component; false for zeros and non-finite entries
__device__ __forceinline__ bool entry_exponent(float2 v, int& e) {
  const int b = max(__float_as_int(v.x) & INT_MAX, __float_as_int(v.y) & INT_MAX);
  e = b >> 23;
  if (e == 0) e = 9 - __clz(b);  // subnormal
  e -= 127;
  return b != 0 && b < 0x7f800000;
}
__device__ __forceinline__ bool entry_exponent(double2 v, int& e) {
  const double m = fmax(fabs(v.x), fabs(v.y));
  const bool ok = m > 0.0 && m < INFINITY && v.x == v.x && v.y == v.y;
  e = ok ? ilogb(m) : 0;
  return ok;
}

template <typename C>
__global__ void __launch_bounds__(256) rns_balance_kernel(int m, int n, int k, RowView<C> A, RowView<C> B,
                                                          int* __restrict__ d) {
  __shared__ int as[8][32], ac[8][32], bs[32], bc[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, k0 = 32 * blockIdx.x;
  const int na = min(kSample, m), nb = min(kSample, n);
  // mean exponents of 32 columns of A (k from col(0..31), along the lanes) and of the same rows of B, into
  // warp 0's lanes; false where either has no entry
  auto difference = [&](auto col, float& v) -> bool {
    int sum = 0, cnt = 0;
    C va[4], vb[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = 4 * wid + j, ca = col(lane), cb = col(r);
      va[j] = r < na && ca < k ? A.at((int)((2LL * r + 1) * m / (2 * na)), ca) : czero<C>();
      vb[j] = lane < nb && cb < k ? B.at(cb, (int)((2LL * lane + 1) * n / (2 * nb))) : czero<C>();
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int e;
      if (entry_exponent(va[j], e)) {
        sum += e;
        ++cnt;
      }
      const bool ok = entry_exponent(vb[j], e);
      const int s = __reduce_add_sync(0xffffffffu, ok ? e : 0), c = __popc(__ballot_sync(0xffffffffu, ok));
      if (lane == 0) {
        bs[4 * wid + j] = s;
        bc[4 * wid + j] = c;
      }
    }
    as[wid][lane] = sum;
    ac[wid][lane] = cnt;
    __syncthreads();
    bool ok = false;
    if (wid == 0) {
      for (int w = 1; w < 8; ++w) {
        sum += as[w][lane];
        cnt += ac[w][lane];
      }
      ok = cnt > 0 && bc[lane] > 0;
      v = ok ? 0.5f * ((float)bs[lane] / bc[lane] - (float)sum / cnt) : 0.f;
    }
    __syncthreads();
    return ok;
  };
  float v = 0.f;
  const bool ok = difference([&](int i) { return k0 + i; }, v);
  if (__syncthreads_or(wid == 0 && !ok && k0 + lane < k)) {
    float t = 0.f;
    const bool any = difference([&](int i) { return (int)((2LL * i + 1) * k / 64); }, t);
    if (wid == 0) {
      const int c = __popc(__ballot_sync(0xffffffffu, any));
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (!ok) v = c ? t / c : 0.f;
    }
  }
  constexpr int lim = sizeof(C) == 8 ? 300 : 1020;  // 2^(2 d) and 2^d are normal doubles
  if (wid == 0 && k0 + lane < k) d[k0 + lane] = max(-lim, min(lim, __float2int_rn(v)));
}

__device__ __forceinline__ uint32_t pack4(const uint32_t (&b)[4]) {
  return __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
}

// u = re + w im and v = re - w im of four entries modulo p, as signed bytes.
// The digit sums (below 2^18) are formed on top of the bits of a float K, a
// multiple of p, so that one FFMA gives the quotient in the low mantissa bits:
// K and the magic constant are 0 modulo 256, and only the low byte is kept.
template <int W>
__device__ __forceinline__ void residues4(const int4 (&re)[W], const int4 (&im)[W], const SplitMod& t, uint32_t& u4,
                                          uint32_t& v4) {
  uint32_t u[4], v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    int a = t.bias, b = 0;
#pragma unroll
    for (int l = 0; l < W; ++l) {
      a = __dp4a((&re[l].x)[j], t.w[l], a);
      b = __dp4a((&im[l].x)[j], t.ww[l], b);
    }
    const int x = a + b, y = a - b;
    const int qx = __float_as_int(fmaf(__int_as_float(x), t.pinv, t.c));
    const int qy = __float_as_int(fmaf(__int_as_float(y), t.pinv, t.c));
    u[j] = (uint32_t)(x - qx * t.p);
    v[j] = (uint32_t)(y - qy * t.p);
  }
  u4 = pack4(u);
  v4 = pack4(v);
}

// the residues of four consecutive k (digits at shared quads `re`, `im`) to all planes
template <typename C>
__device__ __forceinline__ void emit(const int4 (&re)[Traits<C>::kWords], const int4 (&im)[Traits<C>::kWords],
                                     uint8_t* out, size_t plane, const SplitTab& tab) {
  // complex64: unrolled, the table's entries become constant operands; the
  // complex128 body is too long for that (a 5768-face LU loses 0.5 %)
  constexpr int kUnroll = Traits<C>::N <= 8 ? Traits<C>::N : 1;
#pragma unroll kUnroll
  for (int t = 0; t < Traits<C>::N; ++t) {
    uint32_t u, v;
    residues4<Traits<C>::kWords>(re, im, tab.mod[t], u, v);
    *reinterpret_cast<uint32_t*>(out) = u;
    *reinterpret_cast<uint32_t*>(out + plane) = v;
    out += 2 * plane;
  }
}

// Scales and residue planes, plane 2 i (u) and 2 i + 1 (v) of modulus i, K
// contiguous.  The digits are exchanged through shared memory so that global
// reads run along the rows and a warp writes 128 contiguous bytes per plane.
// Blocks [0, ablocks): 8 / wpr rows of A, wpr warps per row, each holding its
// 128-entry chunks of the row in registers between the norm and the digits
// ([rows][Kp]; the columns k..Kp are 0).  Blocks beyond: 8 columns of B, read
// once for the norms and again (from L2) in tiles of 128 rows, written
// transposed ([columns of B][Kp]; the K padding of B is not written, it meets
// A's zeros).  Instruction issue (64 % of the slots) and latency at half
// occupancy bound it: 13 (complex64) / 15 (complex128) instructions per entry
// and modulus; 2884^3 complex64 operands take 120 us with the moduli unrolled,
// 133 with a loop over them.  Norms summed in FP32 do not help.  Entries take the
// powers of two of rns_balance on top of their vector's scale (2884^3 products:
// complex64 449 us, 447 without them; complex128 1072 and 1064).
// exponent of the scale of one entry: 2^e of its vector times 2^d; clamped where the scaled entry is
// 0 or rounds to 0 anyway
template <typename C>
__device__ __forceinline__ int entry_scale(int e, int d) {
  return e == kNonFinite ? 0 : max(-Traits<C>::kExpMax, min(Traits<C>::kExpMax, e + d));
}
constexpr int kRowChunks = kBlockK / 128 / 8;  // chunks per warp of the longest row
template <typename C>
__global__ void __launch_bounds__(256, sizeof(C) == 16 ? 3 : 4) rns_split_kernel(int m, int n, int k, RowView<C> A, RowView<C> B, int Mp, int Np,
                                                        int Kp, int ablocks, int wpr, const int* __restrict__ pw, int* __restrict__ sa,
                                                        int* __restrict__ sb, uint8_t* __restrict__ pa,
                                                        uint8_t* __restrict__ pb,
                                                        const __grid_constant__ SplitTab tab) {
  using T = Traits<C>;
  constexpr int W = T::kWords;
  __shared__ __align__(16) int32_t sh[8][2 * W][128];  // A: per warp; B: per column
  __shared__ double rmx[8][8], rss[8][8];
  __shared__ int esh[8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int4 re[W], im[W];
  if ((int)blockIdx.x < ablocks) {
    const int chunks = Kp / 128, share = wid % wpr;
    const int i = blockIdx.x * (8 / wpr) + wid / wpr;
    C v[kRowChunks][4];
    int d[kRowChunks][4];
    double mx = 0.0, ss = 0.0;
    // sum over the lanes and the row's warps
    auto row_sum = [&](int buf) {
      for (int o = 16; o > 0; o >>= 1) {
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
      }
      if (lane == 0) {
        rmx[buf][wid] = mx;
        rss[buf][wid] = ss;
      }
      __syncthreads();
      mx = ss = 0.0;
      for (int w = 0; w < wpr; ++w) {
        mx = fmax(mx, rmx[buf][wid - share + w]);
        ss += rss[buf][wid - share + w];
      }
    };
    if (i < m) {
      const C* row = &A.at(i, 0);
#pragma unroll
      for (int g = 0; g < kRowChunks; ++g)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int c = (share + g * wpr) * 128 + lane + 32 * j;
          v[g][j] = c < k ? row[c] : czero<C>();
          d[g][j] = c < k ? pw[c] : 0;
        }
#pragma unroll
      for (int g = 0; g < kRowChunks; ++g)
#pragma unroll
        for (int j = 0; j < 4; ++j) norm_add(v[g][j], d[g][j], ss);
    }
    row_sum(0);
    int e = scale_exponent(ss, T::kTwoAlpha);
    if constexpr (sizeof(C) == 16) {
      const bool redo = i < m && norm_unsafe((C*)nullptr, ss), low = ss >= 1e290;
      if (__syncthreads_or(redo)) {
        mx = ss = 0.0;
        if (redo) {
#pragma unroll
          for (int g = 0; g < kRowChunks; ++g)
#pragma unroll
            for (int j = 0; j < 4; ++j) norm_add_wide(v[g][j], d[g][j], low, mx, ss);
        }
        row_sum(1);
        if (redo) e = scale_exponent_wide(mx, ss, k, low, T::kTwoAlpha);
      }
    }
    if (i >= m) return;
    if (share == 0 && lane == 0) sa[i] = e;
#pragma unroll
    for (int g = 0; g < kRowChunks; ++g) {
      const int ch = share + g * wpr;
      if (ch >= chunks) break;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        int32_t dr[W], di[W];
        const int t = entry_scale<C>(e, d[g][j]);
        digits(v[g][j].x, t, dr);
        digits(v[g][j].y, t, di);
#pragma unroll
        for (int l = 0; l < W; ++l) {
          sh[wid][l][lane + 32 * j] = e == kNonFinite ? 0 : dr[l];
          sh[wid][W + l][lane + 32 * j] = e == kNonFinite ? 0 : di[l];
        }
      }
      __syncwarp();
#pragma unroll
      for (int l = 0; l < W; ++l) {
        re[l] = *reinterpret_cast<const int4*>(&sh[wid][l][4 * lane]);
        im[l] = *reinterpret_cast<const int4*>(&sh[wid][W + l][4 * lane]);
      }
      __syncwarp();
      emit<C>(re, im, pa + (size_t)i * Kp + ch * 128 + 4 * lane, (size_t)Mp * Kp, tab);
    }
    return;
  }
  const int q0 = (blockIdx.x - ablocks) * 8;
  const int c = threadIdx.x & 7, rg = threadIdx.x >> 3, q = q0 + c;  // column, row group (0..31)
  {
    double mx = 0.0, ss = 0.0;
    // sum over the row groups, to threads 0 .. 7
    auto column_sum = [&]() {
      for (int o = 16; o >= 8; o >>= 1) {
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
      }
      if (lane < 8) {
        rmx[wid][lane] = mx;
        rss[wid][lane] = ss;
      }
      __syncthreads();
      mx = ss = 0.0;
      for (int w = 0; w < 8; ++w) {
        mx = fmax(mx, rmx[w][c]);
        ss += rss[w][c];
      }
      __syncthreads();
    };
    if (q < n) {
#pragma unroll 8
      for (int p = rg; p < k; p += 32) norm_add(B.at(p, q), -pw[p], ss);
    }
    column_sum();
    int e = scale_exponent(ss, T::kTwoAlpha);
    if constexpr (sizeof(C) == 16) {
      const bool redo = q < n && norm_unsafe((C*)nullptr, ss), low = ss >= 1e290;
      if (__syncthreads_or(redo)) {
        mx = ss = 0.0;
        if (redo)
          for (int p = rg; p < k; p += 32) norm_add_wide(B.at(p, q), -pw[p], low, mx, ss);
        column_sum();
        if (redo) e = scale_exponent_wide(mx, ss, k, low, T::kTwoAlpha);
      }
    }
    if (threadIdx.x < 8) {
      esh[c] = e;
      if (q < n) sb[q] = e;
    }
    __syncthreads();
  }
  const int e = esh[c];
  const size_t plane = (size_t)Np * Kp;
  C v[4];
  int d[4];
  auto fetch = [&](int p0) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int p = p0 + 4 * rg + j;
      v[j] = (p < k && q < n) ? B.at(p, q) : czero<C>();
      d[j] = p < k ? -pw[p] : 0;
    }
  };
  fetch(0);
  for (int p0 = 0; p0 < k; p0 += 128) {
    int4 dr[W], di[W];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int32_t r[W], s[W];
      const int t = entry_scale<C>(e, d[j]);
      digits(v[j].x, t, r);
      digits(v[j].y, t, s);
#pragma unroll
      for (int l = 0; l < W; ++l) {
        (&dr[l].x)[j] = e == kNonFinite ? 0 : r[l];
        (&di[l].x)[j] = e == kNonFinite ? 0 : s[l];
      }
    }
    __syncthreads();  // the previous tile's digits have been read
#pragma unroll
    for (int l = 0; l < W; ++l) {  // quads swizzled by the column: conflict-free 16-byte stores
      *reinterpret_cast<int4*>(&sh[c][l][4 * (rg ^ c)]) = dr[l];
      *reinterpret_cast<int4*>(&sh[c][W + l][4 * (rg ^ c)]) = di[l];
    }
    __syncthreads();
    if (p0 + 128 < k) fetch(p0 + 128);
    if (q0 + wid < n) {  // warp w: column q0 + w, lane l: quad l of the tile
#pragma unroll
      for (int l = 0; l < W; ++l) {
        re[l] = *reinterpret_cast<const int4*>(&sh[wid][l][4 * (lane ^ wid)]);
        im[l] = *reinterpret_cast<const int4*>(&sh[wid][W + l][4 * (lane ^ wid)]);
      }
      emit<C>(re, im, pb + (size_t)(q0 + wid) * Kp + p0 + 4 * lane, plane, tab);
    }
  }
}

// ------------------------------------------------------------------ int8 product
constexpr int BM = 128;          // output tile rows (TMEM lanes)
constexpr int BN = 256;          // output tile columns
constexpr int BK = 128;          // bytes per K slab: one 128-byte swizzle row
constexpr int STAGES = 4;        // 48 KB each: three slabs in flight behind the one multiplied
constexpr int kGroupM = 16;      // tile rows per band of the grouped tile order
constexpr int UMMA_K = 32;
constexpr int A_TILE = BM * BK;  // 16 KB
constexpr int B_TILE = BN * BK;  // 32 KB
constexpr int STAGE_BYTES = A_TILE + B_TILE;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024;
constexpr int THREADS = 256;
constexpr long long kMaxSpin = 1LL << 26;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait; false (and *err set) on timeout, or once another role gave up
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err, volatile int* abort_flag) {
  for (long long i = 0; i < kMaxSpin; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if (i > 32) {
      if (*abort_flag) return false;
      __nanosleep(20);
    }
  }
  atomicExch(err, BEM200_ERR_TIMEOUT);
  *abort_flag = 1;
  return false;
}

__device__ __forceinline__ void tma_load_2d(const CUtensorMap* map, uint64_t* bar, void* dst, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

// K-major, 128-byte swizzled operand tile: rows of 128 B, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;             // leading-dimension offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;   // stride-dimension offset: 8 rows x 128 B
  d |= (uint64_t)1 << 46;             // descriptor version for tcgen05
  d |= (uint64_t)2 << 61;             // 128-byte swizzle
  return d;
}

// instruction descriptor: D s32, A/B s8, both K-major, M = BM, N = BN
constexpr uint32_t kIdesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);

__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(kIdesc), "r"(accum));
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

struct GemmArgs {
  int m;            // rows stored
  int tm, tn;       // tiles per plane
  int tiles;        // planes x tm x tn
  int nk;           // K slabs
  int Mp, Np;       // rows per plane of the operands
  uint8_t* C;       // [plane][m][Np] residues + 128
  int* status;
  ModTab mod;
};

// Persistent: CTA b takes tiles b, b + gridDim.x, ... of the list of 2 N planes x
// output tiles (planes outermost, so that one plane's operands stay in L2).
// Warp 0 loads (TMA), warp 1 issues the MMAs (one thread), warps 4..7 read
// the accumulator of the previous tile (two accumulators of 256 columns in
// TMEM), reduce it modulo p and store bytes.
__global__ void __launch_bounds__(THREADS, 1) rns_gemm_kernel(const __grid_constant__ CUtensorMap mA,
                                                              const __grid_constant__ CUtensorMap mB,
                                                              const __grid_constant__ GemmArgs args) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_sh;
  __shared__ volatile int abort_sh, never_sh;
  __shared__ volatile int issued_sh, consumed_sh;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4);
    }
    abort_sh = 0;
    never_sh = 0;
    issued_sh = 0;
    consumed_sh = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                 "r"(2 * BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_sh;
  const int per_plane = args.tm * args.tn;
  // grouped order within a plane: consecutive tiles sweep a band of kGroupM tile rows
  auto decode = [&](int t, int& plane, int& tile_m, int& tile_n) {
    plane = t / per_plane;
    const int lin = t - plane * per_plane;
    const int per_group = kGroupM * args.tn;
    const int grp = lin / per_group, first_m = grp * kGroupM;
    const int rows = min(kGroupM, args.tm - first_m);
    const int local = lin - grp * per_group;
    tile_m = first_m + local % rows;
    tile_n = local / rows;
  };

  if (warp == 0 && lane == 0) {
    // ---------------- TMA producer
    int it = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < args.tiles && ok; t += gridDim.x) {
      int plane, tile_m, tile_n;
      decode(t, plane, tile_m, tile_n);
      const int ya = plane * args.Mp + tile_m * BM, yb = plane * args.Np + tile_n * BN;
      for (int kb = 0; kb < args.nk; ++kb, ++it) {
        const int s = it % STAGES;
        if (it >= STAGES && !mbar_wait(&empty_bar[s], ((it / STAGES) & 1) ^ 1, args.status, &abort_sh)) {
          ok = false;
          break;
        }
        unsigned char* st = base + s * STAGE_BYTES;
        mbar_expect_tx(&full_bar[s], STAGE_BYTES);
        tma_load_2d(&mA, &full_bar[s], st, kb * BK, ya);
        tma_load_2d(&mB, &full_bar[s], st + A_TILE, kb * BK, yb);
        issued_sh = it + 1;
      }
    }
  } else if (warp == 1 && lane == 0) {
    // ---------------- MMA issuer
    int it = 0, i = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < args.tiles && ok; t += gridDim.x, ++i) {
      const int buf = i & 1;
      if (i >= 2 && !mbar_wait(&acc_empty[buf], ((i >> 1) & 1) ^ 1, args.status, &abort_sh)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem + buf * BN;
      for (int kb = 0; kb < args.nk; ++kb, ++it) {
        const int s = it % STAGES;
        if (!mbar_wait(&full_bar[s], (it / STAGES) & 1, args.status, &abort_sh)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a = smem_u32(base + s * STAGE_BYTES), b = a + A_TILE;
#pragma unroll
        for (int kk = 0; kk < BK / UMMA_K; ++kk)
          umma_i8(acc, sdesc(a + kk * UMMA_K), sdesc(b + kk * UMMA_K), (kb | kk) ? 1u : 0u);
        umma_commit(&empty_bar[s]);  // stage free once these MMAs retire
        consumed_sh = it + 1;
      }
      umma_commit(&acc_full[buf]);  // accumulator complete (or abandoned)
    }
  } else if (warp >= 4) {
    // ---------------- epilogue: accumulator mod p -> bytes.  Thread = one TMEM lane = one output row.
    const int ew = warp - 4;
    int i = 0;
    for (int t = blockIdx.x; t < args.tiles; t += gridDim.x, ++i) {
      const int buf = i & 1;
      if (!mbar_wait(&acc_full[buf], (i >> 1) & 1, args.status, &abort_sh)) break;
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      int plane, tile_m, tile_n;
      decode(t, plane, tile_m, tile_n);
      // x mod p in bytes: x / p from the FP32 value of x (|x| < 2^25.5: off by at
      // most 2 / p) times the rounded 1 / p (off by 2^-24 |x| / p), so the quotient
      // is that of x / p within 0.52 and |x - q p| <= 126
      const int p = args.mod.p[plane >> 1];
      const float pinv = args.mod.pinv[plane >> 1];
      const int row = tile_m * BM + ew * 32 + lane;
      uint8_t* out = args.C + ((size_t)plane * args.m + row) * args.Np + tile_n * BN;
#pragma unroll 1
      for (int cb = 0; cb < BN / 32; ++cb) {
        uint32_t r[32];
        tmem_ld32(tmem + buf * BN + ((uint32_t)(ew * 32) << 16) + cb * 32, r);
        uint32_t w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          uint32_t b[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int x = (int)r[4 * j + c];
            b[c] = (uint32_t)(x - __float_as_int(fmaf(__int2float_rn(x), pinv, kMagic)) * p);
          }
          w[j] = pack4(b) ^ 0x80808080u;
        }
        if (row < args.m) {
          uint4* o = reinterpret_cast<uint4*>(out + cb * 32);
          o[0] = make_uint4(w[0], w[1], w[2], w[3]);
          o[1] = make_uint4(w[4], w[5], w[6], w[7]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_sh && threadIdx.x == 0) {
    // drain (bounded): loads issued but never consumed must land, committed
    // MMAs must retire (the last commit to a stage signals its empty barrier)
    const int iss = issued_sh, con = consumed_sh;
    for (int s = con; s < iss; ++s) mbar_wait(&full_bar[s % STAGES], (s / STAGES) & 1, args.status, &never_sh);
    if (con > 0) mbar_wait(&empty_bar[(con - 1) % STAGES], ((con - 1) / STAGES) & 1, args.status, &never_sh);
  }
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN));
  }
}

// ------------------------------------------------------------------ CRT
// C = alpha (CRT of the residues) + beta C.  A warp merges 128 columns of one
// row, 4 per lane (2 N coalesced 4-byte reads), and exchanges the results
// through shared memory so that C is read and written along the row.  The
// weights are fractions of P modulo 1 in 32 kFrac bits, so the sum's
// wrap-around is the reduction modulo P.  Memory bound: 2 N bytes read per
// entry besides C.
template <typename C>
__global__ void __launch_bounds__(256) rns_merge_kernel(int m, int n, int Np, const uint8_t* __restrict__ res,
                                                        const int* __restrict__ sa, const int* __restrict__ sb,
                                                        C alpha, C beta, RowView<C> Cv, int nsplit, C alpha2, C beta2,
                                                        const __grid_constant__ MergeTab tab) {
  using T = Traits<C>;
  __shared__ __align__(16) C sh[8][128];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int chunks = (n + 127) / 128;
  const long long item = (long long)blockIdx.x * 8 + wid;
  const int i = (int)(item / chunks), q0 = (int)(item % chunks) * 128;
  if (i >= m) return;
  const uint8_t* src = res + (size_t)i * Np + q0 + 4 * lane;
  const size_t plane = (size_t)m * Np;
  uint32_t x4[T::N], y4[T::N];
#pragma unroll
  for (int t = 0; t < T::N; ++t) {
    x4[t] = __ldcs(reinterpret_cast<const uint32_t*>(src + (2 * t) * plane));
    y4[t] = __ldcs(reinterpret_cast<const uint32_t*>(src + (2 * t + 1) * plane));
  }
  const int ea = sa[i];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    double fr, fi;
    if constexpr (T::kFrac == 2) {
      uint64_t r0 = tab.u0[0] | ((uint64_t)tab.u0[1] << 32), i0 = tab.v0[0] | ((uint64_t)tab.v0[1] << 32);
      uint32_t r1 = 0, i1 = 0;
#pragma unroll
      for (int t = 0; t < T::N; ++t) {
        const uint32_t x = (x4[t] >> (8 * j)) & 0xffu, y = (y4[t] >> (8 * j)) & 0xffu;
        const uint32_t s = x + y, d = x + 255u - y;
        r0 += (uint64_t)s * tab.mod[t].u[0];
        i0 += (uint64_t)d * tab.mod[t].v[0];
        r1 += s * tab.mod[t].u[1];
        i1 += d * tab.mod[t].v[1];
      }
      fr = (double)(long long)(r0 + ((uint64_t)r1 << 32));
      fi = (double)(long long)(i0 + ((uint64_t)i1 << 32));
    } else {
      uint64_t r0 = tab.u0[0], r1 = tab.u0[1], i0 = tab.v0[0], i1 = tab.v0[1];
      uint32_t r2 = tab.u0[2], i2 = tab.v0[2];
#pragma unroll
      for (int t = 0; t < T::N; ++t) {
        const uint32_t x = (x4[t] >> (8 * j)) & 0xffu, y = (y4[t] >> (8 * j)) & 0xffu;
        const uint32_t s = x + y, d = x + 255u - y;
        r0 += (uint64_t)s * tab.mod[t].u[0];
        i0 += (uint64_t)d * tab.mod[t].v[0];
        r1 += (uint64_t)s * tab.mod[t].u[1];
        i1 += (uint64_t)d * tab.mod[t].v[1];
        r2 += s * tab.mod[t].u[2];
        i2 += d * tab.mod[t].v[2];
      }
      r1 += r0 >> 32;  // carries
      i1 += i0 >> 32;
      fr = fma((double)(int32_t)(r2 + (uint32_t)(r1 >> 32)), 18446744073709551616.0,
               fma((double)(uint32_t)r1, 4294967296.0, (double)(uint32_t)r0));
      fi = fma((double)(int32_t)(i2 + (uint32_t)(i1 >> 32)), 18446744073709551616.0,
               fma((double)(uint32_t)i1, 4294967296.0, (double)(uint32_t)i0));
    }
    // times P 2^(-32 kFrac) 2^-(ea + eb), the power of two in two factors
    const int q = q0 + 4 * lane + j;
    const int eb = q < n ? sb[q] : 0;
    const int h = max(-1400, min(1400, -(ea + eb))), h1 = h >> 1;
    const bool finite = ea != kNonFinite && eb != kNonFinite;
    const double f1 = finite ? __hiloint2double((h1 + 1023) << 20, 0) * tab.scale : NAN;
    const double f2 = __hiloint2double((h - h1 + 1023) << 20, 0);
    sh[wid][4 * lane + j] = cmake<C>(fr * f1 * f2, fi * f1 * f2);
  }
  __syncwarp();
  C* out = &Cv.at(i, q0);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = lane + 32 * j;
    if (q0 + c >= n) break;
    const bool lo = q0 + c < nsplit;
    const C be = lo ? beta : beta2;
    C v = cmul(lo ? alpha : alpha2, sh[wid][c]);
    if (be.x != 0 || be.y != 0) v = cadd(v, cmul(be, out[c]));
    out[c] = v;
  }
}

// ------------------------------------------------------------------ host
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeFn encode_fn() {
  static EncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<EncodeFn>(p);
    return (EncodeFn) nullptr;
  }();
  return fn;
}

static int make_map(CUtensorMap* m, void* ptr, long long rows, int cols, int box_rows) {
  EncodeFn fn = encode_fn();
  BEM_REQUIRE(fn, BEM200_ERR_CUDA, "gemm: cuTensorMapEncodeTiled unavailable");
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  BEM_REQUIRE(r == CUDA_SUCCESS, BEM200_ERR_CUDA, "gemm: tensor map encode failed (%d)", (int)r);
  return BEM200_OK;
}

static size_t up256(size_t b) { return (b + 255) & ~size_t(255); }

constexpr size_t kBalanceBytes = sizeof(int) * kBlockK;
static_assert(kBalanceBytes % 256 == 0, "workspace layout");

struct Plan {
  int Mp, Np, Kp;
  size_t a, b, c, sa, sb, total;
};

template <typename C>
static Plan plan(int m, int n, int k) {
  constexpr size_t planes = 2 * Traits<C>::N;
  Plan p;
  p.Mp = ceil_div(m, BM) * BM;
  p.Np = ceil_div(n, BN) * BN;
  p.Kp = ceil_div(k, BK) * BK;
  p.a = planes * p.Mp * p.Kp;
  p.b = planes * p.Np * p.Kp;
  p.c = up256(planes * m * (size_t)p.Np);
  p.sa = up256(sizeof(int) * (size_t)m);
  p.sb = up256(sizeof(int) * (size_t)n);
  p.total = kBalanceBytes + p.a + p.b + p.c + p.sa + p.sb + 256;
  return p;
}

// Largest blocks of m, n, k whose planes fit `bytes` (0 when nothing does):
// the largest extent is halved until they do, down to one tile.
template <typename C>
static bool fit_blocks(int m, int n, int k, size_t bytes, int& mb, int& nb, int& kb) {
  constexpr int cap = Traits<C>::kBlock;
  auto even = [](int x, int lim, int q) {  // x in equal parts of at most lim, multiples of q
    const int parts = ceil_div(x, lim);
    return std::min(x, ceil_div(ceil_div(x, parts), q) * q);
  };
  int lm = cap, ln = cap, lk = kBlockK;
  while (true) {
    mb = even(m, lm, BM);
    nb = even(n, ln, BN);
    kb = even(k, lk, BK);
    if (plan<C>(mb, nb, kb).total <= bytes) return true;
    if (mb <= BM && nb <= BN && kb <= BK) return false;
    if (kb >= mb && kb >= nb && kb > BK) lk = std::max(BK, kb / 2);
    else if (nb >= mb && nb > BN) ln = std::max(BN, nb / 2);
    else if (mb > BM) lm = std::max(BM, mb / 2);
    else if (nb > BN) ln = std::max(BN, nb / 2);
    else lk = std::max(BK, kb / 2);
  }
}

}  // namespace rns

template <typename C>
size_t gemm_tc_workspace(int m, int n, int k, GemmEngine e) {
  if (e == GemmEngine::kSimt || m <= 0 || n <= 0 || k <= 0) return 0;
  int mb, nb, kb;
  rns::fit_blocks<C>(m, n, k, ~size_t(0), mb, nb, kb);
  return rns::plan<C>(mb, nb, kb).total;
}

// the caller's workspace from its first 256-byte boundary on
static char* operand_space(const LaContext& ctx, size_t& bytes) {
  const uintptr_t p = reinterpret_cast<uintptr_t>(ctx.ws), a = (p + 255) & ~uintptr_t(255);
  bytes = ctx.ws && ctx.ws_bytes > a - p ? ctx.ws_bytes - (a - p) : 0;
  return reinterpret_cast<char*>(a);
}

template <typename C>
bool gemm_tc_fits(const LaContext& ctx, int m, int n, int k) {
  int mb, nb, kb;
  size_t bytes;
  operand_space(ctx, bytes);
  return rns::fit_blocks<C>(m, n, k, bytes, mb, nb, kb);
}

template <typename C>
bool gemm_tc_in_place(const LaContext& ctx, int m, int n, int k) {
  int mb, nb, kb;
  size_t bytes;
  operand_space(ctx, bytes);
  return rns::fit_blocks<C>(m, n, k, bytes, mb, nb, kb) && mb == m && kb == k;
}

template <typename C>
int gemm_tc(const LaContext& ctx, int m, int n, int k, C alpha, RowView<C> A, RowView<C> B, C beta, RowView<C> Cv,
            int nsplit, C alpha2, C beta2) {
  using namespace rns;
  using T = Traits<C>;
  BEM_REQUIRE(ctx.engine == GemmEngine::kTc, BEM200_ERR_UNSUPPORTED, "gemm: the TF32 tensor-core engine is not built");
  int mb, nb, kb;
  size_t bytes;
  char* w = operand_space(ctx, bytes);
  BEM_REQUIRE(fit_blocks<C>(m, n, k, bytes, mb, nb, kb), BEM200_ERR_ARG,
              "gemm: workspace of %zu bytes needed for %d x %d x %d (have %zu)", plan<C>(m, n, k).total, m, n, k,
              ctx.ws_bytes);
  const Tables& tab = tables<C>();
  BEM_CUDA_CHECK(set_kernel_attrs_once(rns_gemm_kernel, SMEM_BYTES, false));
  for (int k0 = 0; k0 < k; k0 += kb)
    for (int m0 = 0; m0 < m; m0 += mb)
      for (int n0 = 0; n0 < n; n0 += nb) {
        const int mm = std::min(mb, m - m0), nn = std::min(nb, n - n0), kk = std::min(kb, k - k0);
        const Plan p = plan<C>(mm, nn, kk);
        // the powers of two stay for all blocks of this k, A's scales and planes for the other blocks of n
        int* pw = reinterpret_cast<int*>(w);
        int* sa = reinterpret_cast<int*>(w + kBalanceBytes);
        uint8_t* pa = reinterpret_cast<uint8_t*>(w) + kBalanceBytes + p.sa;
        uint8_t* pb = pa + p.a;
        uint8_t* pc = pb + p.b;
        int* sb = reinterpret_cast<int*>(pc + p.c);
        // without a status of the caller's, a place that is written on a timeout and never read
        int* status = ctx.dstatus ? ctx.dstatus : reinterpret_cast<int*>(pc + p.c + p.sb);
        const RowView<C> Ab = A.sub(m0, k0), Bb = B.sub(k0, n0), Cb = Cv.sub(m0, n0);
        const int chunks = p.Kp / 128, wpr = chunks >= 8 ? 8 : (chunks >= 4 ? 4 : (chunks >= 2 ? 2 : 1));
        const int ablocks = n0 == 0 ? ceil_div(mm, 8 / wpr) : 0;
        if (m0 == 0 && n0 == 0) {
          rns_balance_kernel<C><<<ceil_div(kk, 32), 256, 0, ctx.stream>>>(m, n, kk, A.sub(0, k0), B.sub(k0, 0), pw);
          BEM_LAUNCH_CHECK();
        }
        rns_split_kernel<C><<<ablocks + ceil_div(nn, 8), 256, 0, ctx.stream>>>(
            mm, nn, kk, Ab, Bb, p.Mp, p.Np, p.Kp, ablocks, wpr, pw, sa, sb, pa, pb, tab.split);
        BEM_LAUNCH_CHECK();
        CUtensorMap ma, mbm;
        int st;
        if ((st = make_map(&ma, pa, (long long)2 * T::N * p.Mp, p.Kp, BM))) return st;
        if ((st = make_map(&mbm, pb, (long long)2 * T::N * p.Np, p.Kp, BN))) return st;
        GemmArgs ga;
        ga.m = mm;
        ga.tm = p.Mp / BM;
        ga.tn = p.Np / BN;
        ga.tiles = 2 * T::N * ga.tm * ga.tn;
        ga.nk = p.Kp / BK;
        ga.Mp = p.Mp;
        ga.Np = p.Np;
        ga.C = pc;
        ga.status = status;
        ga.mod = tab.mod;
        rns_gemm_kernel<<<std::min(ga.tiles, 148), THREADS, SMEM_BYTES, ctx.stream>>>(ma, mbm, ga);
        BEM_LAUNCH_CHECK();
        const C b0 = k0 == 0 ? beta : cmake<C>(1.0, 0.0);
        rns_merge_kernel<C><<<ceil_div((long long)mm * ((nn + 127) / 128), 8), 256, 0, ctx.stream>>>(
            mm, nn, p.Np, pc, sa, sb, alpha, b0, Cb, nsplit - n0, alpha2, k0 == 0 ? beta2 : cmake<C>(1.0, 0.0),
            tab.merge);
        BEM_LAUNCH_CHECK();
      }
  return BEM200_OK;
}

#define RNS_INST(C)                                                                                              \
  template size_t gemm_tc_workspace<C>(int, int, int, GemmEngine);                                               \
  template bool gemm_tc_fits<C>(const LaContext&, int, int, int);                                                \
  template bool gemm_tc_in_place<C>(const LaContext&, int, int, int);                                            \
  template int gemm_tc<C>(const LaContext&, int, int, int, C, RowView<C>, RowView<C>, C, RowView<C>, int, C, C);
RNS_INST(float2)
RNS_INST(double2)

}  // namespace bem200
