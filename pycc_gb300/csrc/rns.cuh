// FP64 products on the BF16 tensor cores in residue arithmetic: what contract_rns.cu (pairwise
// contractions) and triples_rns.cu (the connected triples) share -- operands to residues, the
// GEMM over residues, residues to FP64.  contract_rns.cu describes the method.
#pragma once
#include "tc_common.cuh"
#include <cuda_bf16.h>
#include <algorithm>
#include <cmath>
#include <cstring>

namespace pcg {
namespace rns {

using namespace pcg::tc;

// Sixteen pairwise coprime moduli whose nearest residues fit a signed byte (255 would reach
// +128).  The rounding of the scaled integers, relative to the sum, grows with sqrt(K) and with
// the spread of a row's magnitudes; measured against 113-bit sums, 15 moduli (2^-58.5 |a| |b|)
// fall behind the FP64 kernel at K = 50000 with magnitudes spread over e^+-4 (8.7e-16 against
// 5.8e-16 of the sums' norm), 16 stay ahead of it everywhere.
constexpr int NM = 16;
constexpr int kModuli[NM] = {256, 253, 251, 247, 241, 239, 233, 229,
                             227, 223, 217, 211, 199, 197, 193, 191};
// Planes of a packed operand and of a product: the residues, then magnitudes.  A row is rounded to
// integers at one power of two, so an output's error is a fixed number of units: 0.29 sqrt(|a'|^2
// + |b'|^2) <= 2^60.6 of them (root mean square).  Where large entries of a row meet small or zero
// ones, that can be all of a sum of small products.  So |a'| and |b'|, truncated to BF16, go
// through the GEMM as well and give sum |a'||b'|; an output whose sum is not zero and below kDoubt
// units is computed again in FP64.  Elsewhere the error is at most 2^-53.4 sum |a||b| (root mean
// square) and sqrt(K) 2^-52 sum |a||b| in the worst case, against K 2^-53 for FP64 multiply-adds.
constexpr int NP = NM + 1;
constexpr float kDoubt = 0x1p114f;
// The magnitude of an entry that rounds to zero and is not: large enough that the product of two of
// them is a normal FP32 number, so that sum |a'||b'| is zero for outputs without a product only.
constexpr unsigned kTinyBf16 = (127 - 60) << 7;
constexpr int kBits2 = 123;         // |a'|^2 |b'|^2 <= 2^(2 * 123.75); log2(product / 2) = 123.95
constexpr int kSumBits = 123;       // sums of up to 2^kSumBits are certain to be in range
// The product of the moduli above 2^(kSumBits + 1) times 2^0.9: room for kBits2's 0.75 bits too.
constexpr bool moduli_hold_sums() {
  double half = 0.5;
  for (int p : kModuli) half *= p;
  for (int b = 0; b < kSumBits; ++b) half *= 0.5;
  return half > 1.866;  // 2^0.9
}
static_assert(moduli_hold_sums(), "half the product of the moduli exceeds 2^(kSumBits + 0.9)");
// first bit of the four digits of a scaled integer (16, 15, 15 and 16 bits): with residues of
// the powers of at most 127, a digit sum stays below 2^16 + 127 * 2^17 < 2^24, exact in FP32
__host__ __device__ constexpr int digit_bit(int q) {
  return q == 0 ? 0 : (q == 4 ? 62 : 1 + 15 * q);
}
constexpr int kChunk = 15;          // 64-K blocks per exact FP32 accumulation: 960 K
constexpr float kMagic = 12582912.f;  // 1.5 * 2^23: adding it rounds to an integer

// Per modulus: p, 1/p and the residues of 2^16, 2^31, 2^46 (symmetric).  The magnitudes' p and 1/p
// are zero: nothing is taken off their sums.
struct ModTab {
  float p[NP], inv[NP], c1[NM], c2[NM], c3[NM];
};
// ModTab's entries twice each (np: -p), for arithmetic on pairs.
struct PairTab {
  unsigned long long np[NM], inv[NM], c1[NM], c2[NM], c3[NM];
};
// Per modulus floor(2^96 q / p), q = ((P / p)^-1 mod p), in three 32-bit words; b: what the
// bias of the stored bytes adds, negated; scale = P 2^-96.
struct CrtTab {
  unsigned c0[NM], c1[NM], c2[NM], b0, b1, b2;
  double scale;
};
static_assert(NM * 8 <= 128, "the product fits a 128-bit integer");

// Four residues as bytes r + 128 (modulo 256).
__device__ __forceinline__ unsigned residue_bytes(float a, float b, float c, float d) {
  constexpr float bias = 8388608.f + 128.f;
  return __byte_perm(
      __byte_perm(__float_as_uint(a + bias), __float_as_uint(b + bias), 0x0040),
      __byte_perm(__float_as_uint(c + bias), __float_as_uint(d + bias), 0x0040), 0x5410);
}

// Exponent bits of four sums of magnitudes (not negative, below 2^128).
__device__ __forceinline__ unsigned exponent_bytes(float a, float b, float c, float d) {
  return (__float_as_uint(a) >> 23) | (__float_as_uint(b) >> 23 << 8) |
         (__float_as_uint(c) >> 23 << 16) | (__float_as_uint(d) >> 23 << 24);
}
// A sum of magnitudes, to a factor of two, from byte e of a word of them.
__device__ __forceinline__ float magnitude_sum(unsigned w, int e) {
  return __uint_as_float(__byte_perm(w, 0u, 0x4440u + e) << 23);
}

// Two FP32 values in one register pair; each half is rounded as the scalar operation's.
__device__ __forceinline__ unsigned long long pair(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpair(unsigned long long v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma_pair(unsigned long long a, unsigned long long b,
                                                       unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long add_pair(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// Nearest residues of two integer-valued t, |t| < 2^24, with (-p, -p) and (1/p, 1/p): FP32's 1/p is
// off by at most 2^-24.4 relative, so the quotient is off its nearest integer by less than 0.5 +
// 0.0027 and |r| <= 127 (128 for p = 256).
__device__ __forceinline__ unsigned long long mod_near_pair(unsigned long long t,
                                                            unsigned long long np,
                                                            unsigned long long inv) {
  const unsigned long long q =
      add_pair(fma_pair(t, inv, pair(kMagic, kMagic)), pair(-kMagic, -kMagic));
  return fma_pair(np, q, t);
}

struct Operand {
  const double* X;
  SubIdx r;             // rows: s0 = strides in X, s1 = strides in C
  long long R;          // rows
  long long* off;       // [R] element offset of each row in X
  long long* coff;      // [R] element offset of each row (or column) in C
  int* walk;            // [R] rows in an order whose neighbours are close in X
  unsigned long long* norm;  // [R] the row's largest exponent and sum of squares (RowNorm)
  const int* shift;     // one power of two for all rows, or null: each row its own
  int* sh;              // [R] the rows' powers of two as the pack used them (kNotFinite: the row
                        // holds an Inf or a NaN), or null
  const long long* k;   // [K] element offset of each K index in X
  long long kstep;      // > 0: k[i] = i * kstep
  int wq;               // sub-index that the walk has innermost
  int kfast;            // gathered along K (otherwise along the rows)
};

struct TableArgs {
  Operand a, b;
  SubIdx k;
  long long K;
  long long *ka, *kb;
  int* status;
};

__device__ __forceinline__ void fill_row(const Operand& o, long long r) {
  long long o0, o1;
  sub_offsets(o.r, r, o0, o1);
  o.off[r] = o0;
  if (o.coff) o.coff[r] = o1;
  // r as a position of the walk: the same sub-indices with wq moved innermost
  const int n = o.r.n;
  long long x[kMaxSub], rr = r;
  x[o.wq] = rr % o.r.ext[o.wq];
  rr /= o.r.ext[o.wq];
  for (int q = n - 1; q >= 0; --q) {
    if (q == o.wq) continue;
    x[q] = rr % o.r.ext[q];
    rr /= o.r.ext[q];
  }
  long long row = 0;
  for (int q = 0; q < n; ++q) row = row * o.r.ext[q] + x[q];
  o.walk[r] = (int)row;
}

static __global__ void rns_tables_kernel(const TableArgs t) {
  const long long total = t.a.R + t.b.R + t.K;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    if (i == 0 && t.status) *t.status = 0;
    if (i < t.a.R) {
      fill_row(t.a, i);
      t.a.norm[i] = 0;
    } else if (i < t.a.R + t.b.R) {
      fill_row(t.b, i - t.a.R);
      t.b.norm[i - t.a.R] = 0;
    } else if (t.ka) {
      const long long k = i - t.a.R - t.b.R;
      long long ka, kb;
      sub_offsets(t.k, k, ka, kb);
      t.ka[k] = ka;
      t.kb[k] = kb;
    }
  }
}

__device__ __forceinline__ long long k_offset(const Operand& o, long long k) {
  return o.kstep > 0 ? k * o.kstep : o.k[k];
}

// Sum of squares of a row's |x| 2^(1023 - top), |x| truncated to 20 mantissa bits; top: the biased
// exponent of the largest, at least 1 (2047: an Inf or a NaN).  With an exponent of its own the sum
// holds for rows of any magnitude, where a plain FP32 one holds norms of 2^-40 to 2^50.  Subnormal
// numbers, and zeros of rows below 2^-900, count as more than they are.
struct RowNorm {
  int top = 1;
  float s = 0.f;
  __device__ __forceinline__ void raise(int t) {
    if (t > top) {
      const int d = 127 - 2 * (t - top);
      s *= d > 0 ? __int_as_float(d << 23) : 0.f;
      top = t;
    }
  }
  // h: the upper words of finite doubles or not, without their signs
  template <int N>
  __device__ __forceinline__ void add(const unsigned (&h)[N]) {
    unsigned m = 0;
#pragma unroll
    for (int u = 0; u < N; ++u) m = max(m, h[u]);
    raise((int)(m >> 20));
    const int off = (top - 127) * (1 << 20);
    float t = 0.f;
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const float f = __uint_as_float((unsigned)max((int)h[u] - off, 0) << 3);
      t = fmaf(f, f, t);
    }
    s += t;
  }
  __device__ __forceinline__ void add(RowNorm r) {
    raise(r.top);
    r.raise(top);
    s += r.s;
  }
  __device__ __forceinline__ void reduce() {  // over a warp
    raise(__reduce_max_sync(0xffffffffu, top));
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  }
  __device__ __forceinline__ unsigned long long bits() const {
    return (unsigned long long)top << 32 | __float_as_uint(s);
  }
  static __device__ __forceinline__ RowNorm from(unsigned long long b) {
    RowNorm r;
    r.top = max((int)(b >> 32), 1);
    r.s = __uint_as_float((unsigned)b);
    return r;
  }
  // floor(log2) of the sum in units of one, with 2^-7 for its truncation and summation, and the
  // significand's upper bits
  __device__ __forceinline__ int log2(unsigned& frac) const {
    const unsigned u = __float_as_uint(s * 1.0078125f);
    frac = u & 0x7fffffu;
    return (int)(u >> 23) - 127 + 2 * (top - 1023);
  }
};

// Norms of the rows over K indices [k0, k1): one read of the operand, bound by HBM.  Gathered
// along K (KF: a warp per row) or along the rows (a thread per row, or, of few rows, one per row
// and slice of K: the eight warps of a block then share 32 rows), eight loads in flight per lane.
// Block by of segs has K indices [k0 + by seg, ..).
template <bool KF>
__device__ __forceinline__ void norm_rows(const Operand& o, unsigned long long* part, long long k0,
                                          long long k1, bool slices, long long seg, long long segs,
                                          long long bx, long long by) {
  __shared__ unsigned long long sums[8][32];
  long long kb = k0 + by * seg, ke = min(k1, kb + seg);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long w = KF ? bx * 8 + warp : (slices ? bx * 32 + lane : bx * 256 + threadIdx.x);
  if (w >= o.R && !slices) return;
  if (slices) {
    const long long each = (seg + 7) / 8;
    kb = min(ke, kb + warp * each);
    ke = min(ke, kb + each);
  }
  constexpr int STEP = KF ? 32 : 1;
  const int row = o.walk[min(w, o.R - 1)];
  const double* x = o.X + o.off[row];
  RowNorm n;
  long long k = kb + (KF ? lane : 0);
  for (; k + 7 * STEP < ke; k += 8 * STEP) {
    unsigned h[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      h[u] = (unsigned)__double2hiint(__ldg(x + k_offset(o, k + STEP * u))) & 0x7fffffffu;
    n.add(h);
  }
  if (k < ke) {  // zeros past the end
    unsigned h[7];
#pragma unroll
    for (int u = 0; u < 7; ++u)
      h[u] = k + STEP * u < ke
                 ? (unsigned)__double2hiint(__ldg(x + k_offset(o, k + STEP * u))) & 0x7fffffffu
                 : 0u;
    n.add(h);
  }
  if (KF) n.reduce();
  if (slices) {
    sums[warp][lane] = n.bits();
    __syncthreads();
    if (warp > 0 || w >= o.R) return;
    for (int q = 1; q < 8; ++q) n.add(RowNorm::from(sums[q][lane]));
  }
  if (segs == 1) {
    if (!KF || lane == 0) o.norm[row] = n.bits();
    return;
  }
  // the last of the row's parts adds them up (norm, zero before, counts them)
  bool last = false;
  if (!KF || lane == 0) {
    part[by * o.R + row] = n.bits();
    __threadfence();
    last = atomicAdd(o.norm + row, 1ull) + 1 == (unsigned long long)segs;
    if (last) __threadfence();
  }
  if (KF ? !__shfl_sync(0xffffffffu, last, 0) : !last) return;
  RowNorm sum;
  for (int q0 = KF ? lane : 0; q0 < segs; q0 += 8 * STEP) {  // eight loads in flight here too
    unsigned long long r[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      r[u] = q0 + STEP * u < segs ? __ldcg(part + (q0 + STEP * u) * o.R + row) : 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) sum.add(RowNorm::from(r[u]));
  }
  if (KF) sum.reduce();
  if (!KF || lane == 0) o.norm[row] = sum.bits();
}

struct NormArgs {
  Operand o[2];
  long long gx[2], blocks[2], seg[2], segs[2];  // row blocks, blocks, K segment and their number
  bool slices[2];                               // a block's warps have K slices of 32 rows
  unsigned long long* part[2];                  // [segs][R] sums of the segments
  long long k0, k1;
};

// Both operands in one launch: the first blocks take A, the others B.
static __global__ void __launch_bounds__(256, 8)
    rns_norm_kernel(const __grid_constant__ NormArgs p) {
  const int side = blockIdx.x >= p.blocks[0];
  const long long b = (long long)blockIdx.x - (side ? p.blocks[0] : 0);
  const long long bx = b % p.gx[side], by = b / p.gx[side];
  if (p.o[side].kfast)
    norm_rows<true>(p.o[side], p.part[side], p.k0, p.k1, false, p.seg[side], p.segs[side], bx, by);
  else
    norm_rows<false>(p.o[side], p.part[side], p.k0, p.k1, p.slices[side], p.seg[side], p.segs[side],
                     bx, by);
}

constexpr int kNotFinite = 1 << 20;

// Power of two s of a row: |x| 2^s has a 2-norm of at most 2^61.9 (and of at least 2^60.3, where
// its entries are normal numbers).  A zero row may take any.
__device__ __forceinline__ int row_shift(const Operand& o, long long row) {
  if (o.shift) return *o.shift;
  unsigned frac;
  const int e = RowNorm::from(o.norm[row]).log2(frac);
  // log2 of the sum of squares <= e + 0.75 or e + 1.75; scaled() takes up to 1083
  return min((frac < 0x570000u ? kBits2 - e : kBits2 - 1 - e) >> 1, 1083);
}
__device__ __forceinline__ bool not_finite(const Operand& o, long long row) {
  return o.norm[row] >> 32 == 2047u;
}

// The magnitude of x 2^s rounded to an integer of at most 62 bits, and its sign as +-1.
__device__ __forceinline__ unsigned long long scaled(double x, int s, unsigned flip, float& sign) {
  const unsigned hi = (unsigned)__double2hiint(x) ^ flip, lo = (unsigned)__double2loint(x);
  const unsigned ex = (hi >> 20) & 0x7ffu;
  const unsigned mh = (hi & 0xfffffu) | (ex ? 1u << 20 : 0u);
  // |x| 2^s = m 2^sh, sh = max(ex, 1) - 1075 + s at most 9 since |x| 2^s <= 2^61.9: shifted left
  // by 9 - sh from 10 bits up, then rounded off by the last.  A shift past 63 leaves 0, as does
  // the exponent of an infinity or a NaN, whose row takes its outputs from FP64 dot products.
  const unsigned r = min((unsigned)(9 + 1075 - s - (int)max(ex, 1u)), 63u);
  const unsigned long long m = (((unsigned long long)mh << 32) | lo) << 10;
  sign = __uint_as_float(0x3f800000u | (hi & 0x80000000u));
  return ((m >> r) + 1ull) >> 1;
}

// The four digits (with the sign) of two such integers.
__device__ __forceinline__ void digits(double x, double y, int s, unsigned flip,
                                       unsigned long long (&d)[4]) {
  float sx, sy;
  const unsigned long long m = scaled(x, s, flip, sx), n = scaled(y, s, flip, sy);
  const unsigned long long sign = pair(sx, sy), low = pair(-8388608.f * sx, -8388608.f * sy);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const unsigned mask = (1u << (digit_bit(q + 1) - digit_bit(q))) - 1;
    d[q] = fma_pair(pair(__uint_as_float(0x4b000000u | ((unsigned)(m >> digit_bit(q)) & mask)),
                         __uint_as_float(0x4b000000u | ((unsigned)(n >> digit_bit(q)) & mask))),
                    sign, low);
  }
}

struct PackSide {
  Operand o;
  long long w0, nrow;  // rows of this panel: walk positions [w0, w0 + nrow); nrow 0: none
  __nv_bfloat16* out;  // [plane][row][ld]
  long long plane;     // 16-byte units from a plane to the next
  unsigned flip;       // 0x80000000: the negated operand
  long long blocks;
};

struct PackArgs {
  PackSide s[2];
  long long k0, K;      // K indices [k0, k0 + K)
  long long width, ld;  // columns written, zeros from K on, of each row's ld (multiples of 8)
  PairTab t;
};

__device__ __forceinline__ bool not_zero(double x) {
  return ((unsigned)__double2hiint(x) << 1 | (unsigned)__double2loint(x)) != 0u;
}

// Magnitudes and residues of eight neighbouring K entries, two to an instruction and one 128-bit
// store per plane: an integer of at most 8 bits is exact in the upper half of its FP32 word, which
// is BF16.
__device__ __forceinline__ void store_residues(const PackArgs& p, const PackSide& o,
                                               const double (&x)[8], int s, long long at) {
  unsigned long long d[4][4];
#pragma unroll
  for (int e = 0; e < 4; ++e) digits(x[2 * e], x[2 * e + 1], s, o.flip, d[e]);
  uint4* out = reinterpret_cast<uint4*>(o.out + at);
  const long long plane = o.plane;
  unsigned r[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float a, b;
    unpair(fma_pair(d[e][3], pair(0x1p46f, 0x1p46f),
                    fma_pair(d[e][2], pair(0x1p31f, 0x1p31f),
                             fma_pair(d[e][1], pair(0x1p16f, 0x1p16f), d[e][0]))), a, b);
    r[e] = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632) & 0x7fff7fffu;
    if ((r[e] & 0xffffu) == 0u && not_zero(x[2 * e])) r[e] |= kTinyBf16;
    if ((r[e] >> 16) == 0u && not_zero(x[2 * e + 1])) r[e] |= kTinyBf16 << 16;
  }
  __stcs(out + NM * plane, make_uint4(r[0], r[1], r[2], r[3]));
#pragma unroll
  for (int l = 0; l < NM; ++l, out += plane) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float a, b;
      const unsigned long long t =
          fma_pair(d[e][3], p.t.c3[l],
                   fma_pair(d[e][2], p.t.c2[l], fma_pair(d[e][1], p.t.c1[l], d[e][0])));
      unpair(mod_near_pair(t, p.t.np[l], p.t.inv[l]), a, b);
      r[e] = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
    }
    __stcs(out, make_uint4(r[0], r[1], r[2], r[3]));
  }
}

// Operand -> residues: 8 bytes read and 2 NP written per element, about 95 instructions; bound by
// the writes.  A quarter warp takes 64 K of a row, eight neighbouring K a lane.  Gathered along K
// it loads them straight from global memory; otherwise a tile of 64 walked rows x 64 K goes
// through shared memory, read along the rows.  One launch packs a panel of each operand: the first
// blocks take A's, the others B's.  163e6 elements: 1.12 ms (6.1 TB/s), 1.07 before the plane of
// magnitudes, against 1.15 with one element to an instruction and 1.20 with four K a lane as well.
static __global__ void __launch_bounds__(256, 4)
    rns_pack_kernel(const __grid_constant__ PackArgs p) {
  __shared__ double tile[64][65];
  __shared__ long long off[64], kof[64];
  __shared__ int srow[64], ssh[64];
  const int side = blockIdx.x >= p.s[0].blocks;
  const PackSide& ps = p.s[side];
  const Operand& o = ps.o;
  const unsigned b = blockIdx.x - (side ? (unsigned)p.s[0].blocks : 0u);
  const unsigned nk = (unsigned)((p.width + 63) >> 6), bw = b / nk;
  const long long w = (long long)bw * (o.kfast ? 32 : 64);  // first row of the block
  const long long kk0 = (long long)(b - bw * nk) * 64;      // first K, in the panel
  const int half = threadIdx.x >> 3, kk = 8 * (threadIdx.x & 7);
  if (o.kfast) {
    if (w + half < ps.nrow && kk0 + kk < p.width) {
      const int row = o.walk[ps.w0 + w + half];
      const double* q = o.X + o.off[row];
      double x[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const long long k = kk0 + kk + e;
        x[e] = k < p.K ? __ldg(q + k_offset(o, p.k0 + k)) : 0.0;
      }
      const int sh = row_shift(o, row);
      if (o.sh && kk0 + kk == 0) o.sh[row] = not_finite(o, row) ? kNotFinite : sh;
      store_residues(p, ps, x, sh, (row - ps.w0) * p.ld + kk0 + kk);
    }
  } else {
    if (threadIdx.x < 64) {
      kof[threadIdx.x] = kk0 + threadIdx.x < p.K ? k_offset(o, p.k0 + kk0 + threadIdx.x) : 0;
      if (w + threadIdx.x < ps.nrow) {
        const int r = o.walk[ps.w0 + w + threadIdx.x];
        srow[threadIdx.x] = r;
        off[threadIdx.x] = o.off[r];
        const int sh = row_shift(o, r);
        ssh[threadIdx.x] = sh;
        if (o.sh && kk0 == 0) o.sh[r] = not_finite(o, r) ? kNotFinite : sh;
      }
    }
    __syncthreads();
    const int rr = threadIdx.x & 63;
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int k = (threadIdx.x >> 6) + 4 * u;
      v[u] = (w + rr < ps.nrow && kk0 + k < p.K) ? __ldg(o.X + off[rr] + kof[k]) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) tile[rr][(threadIdx.x >> 6) + 4 * u] = v[u];
    __syncthreads();
#pragma unroll 1
    for (int r = half; r < 64 && w + r < ps.nrow && kk0 + kk < p.width; r += 32) {
      double x[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = tile[r][kk + e];
      store_residues(p, ps, x, ssh[r], (srow[r] - ps.w0) * p.ld + kk0 + kk);
    }
  }
}

// ---- GEMM over the residues -------------------------------------------------------------
// Output tiles and K of a launch.  Plain: C[split][plane] = A B^T over K blocks
// [split kb_per_split, ...).  Triples (TRIP): group g = 3 t + q is orientation q of triple t,
// the sum of two products of row blocks (csrc/triples_rns.cu).
struct GemmArgs {
  long long M, N;    // rows of A and of B in this panel (TRIP: v^2 and v)
  long long mt, nt;  // 128-row and bs-column tiles
  int gm;            // M tiles per raster group
  int bs;            // columns per N tile, a multiple of 16
  int planes;        // splits, or groups
  int nkb, kb_per_split;
  long long ld;        // bytes of one output row: N rounded up to 16
  unsigned char* out;  // [split or group][NP][M][ld]: bytes of residues, exponents of magnitudes
  int* status;
  unsigned long long wait_ns;
  ModTab t;
  // TRIP (T3Plan in triples_rns.cu)
  const int* ijk;           // [triples][3]
  int kc;                   // K blocks of a product over e and m
  int blocks_a, pairs;      // blocks of v^2 rows of an A matrix, pairs (blocks of v rows) of B
  int c, first[3], width[3];  // of i, j, k: slots of c occupied indices from first on, width of
                              // them present; c = 0: one slot for all of them
};

struct GemmMaps {
  CUtensorMap a[2];  // TRIP: [VT | TM], [VN | TMT]
  CUtensorMap b[1];  // TRIP: [T2P | OB]
};

constexpr int kEpiWarps = 8;
constexpr int kGemmThreads = 64 + 32 * kEpiWarps;

template <int BN>
struct RSmem {
  static constexpr int A_BYTES = BM * KBYTES, B_BYTES = BN * KBYTES;
  static constexpr int STAGE = A_BYTES + B_BYTES;
  static constexpr int TAIL = 256;
  static constexpr int FIT = (232448 - 1024 - TAIL) / STAGE;
  static constexpr int STAGES = FIT > 8 ? 8 : FIT;
  static constexpr int TOTAL = 1024 + STAGES * STAGE + TAIL;
  static constexpr unsigned TMEM_COLS = 2 * BN;
  static_assert(BN == 64 || BN == 128 || BN == 256, "two accumulators in a power of two columns");
};

// One unit of work: an output tile of one plane, the sum of up to two runs of K blocks.
struct Unit {
  int plane, mod, n0, blocks;  // plane: split or group; blocks: K blocks in all
  long long m0;
  int ma[2], mb[2], ya[2], yb[2], kb[2], nk[2];
};

// The two products of orientation q of a triple, in indices 0, 1, 2 for i, j, k: [VT | TM] (swap 0)
// or [VN | TMT] of occupied index a, with [T2P | OB] of the pair (bx, by).  [VT | TM] meets i and j
// only, [VN | TMT] j and k.
struct T3Product {
  int swap, a, bx, by;
};
__device__ __forceinline__ T3Product t3_product(int q, int s) {
  T3Product t;
  t.swap = (q == 2) != (s == 1);
  t.a = s == 0 ? (q == 2 ? 2 : 0) : (q == 1 ? 2 : 1);
  t.bx = 2 - q;
  t.by = s == 0 ? (q == 1 ? 2 : 1) : (q == 2 ? 2 : 0);
  return t;
}

// Unit u -> (plane, split or group, tile): neighbouring groups share row blocks of one plane (mod:
// a modulus, or NM for the magnitudes).  The tile order within a plane is tc_gemm_kernel's raster
// (groups of gm M tiles, M fastest), so a wave shares the row blocks of both operands in L2.
template <bool TRIP, bool SEGS>
__device__ __forceinline__ Unit decode_unit(const GemmArgs& p, unsigned u) {
  // 32-bit divisions: in 64 bits the chain took longer than the MMAs of a short-K unit
  const unsigned mt = (unsigned)p.mt, nt = (unsigned)p.nt, per = mt * nt, gm = (unsigned)p.gm;
  Unit x;
  const unsigned g = u / per, r = u - g * per;
  x.mod = (int)(g / (unsigned)p.planes);
  x.plane = (int)(g - (unsigned)x.mod * (unsigned)p.planes);
  const unsigned group = r / (gm * nt), rg = r - group * gm * nt;
  const unsigned here = min(gm, mt - group * gm), n = rg / here;
  x.m0 = (long long)(group * gm + (rg - n * here)) * BM;
  x.n0 = (int)n * p.bs;
  if (!TRIP) {
    x.kb[0] = x.plane * p.kb_per_split;
    x.blocks = x.nk[0] = min(p.nkb, x.kb[0] + p.kb_per_split) - x.kb[0];
    if (SEGS) {
      x.ma[0] = x.mb[0] = 0;
      x.ya[0] = (int)(x.mod * p.M + x.m0);
      x.yb[0] = (int)(x.mod * p.N + x.n0);
    }
    return x;
  }
  x.blocks = 2 * p.kc;
  if (SEGS) {
    const int q = x.plane % 3;
    int at[3];  // place of i, j, k in their slots
#pragma unroll
    for (int r = 0; r < 3; ++r) at[r] = p.ijk[x.plane - q + r] - p.first[r];
    auto of = [](const int (&v)[3], int r) { return r == 0 ? v[0] : (r == 1 ? v[1] : v[2]); };
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const T3Product t = t3_product(q, s);
      const int block = (t.a - t.swap) * p.c + of(at, t.a);
      const int pair = (3 * t.bx + t.by) * p.c * p.c + of(at, t.bx) * of(p.width, t.by) +
                       of(at, t.by);
      x.ma[s] = t.swap;
      x.mb[s] = 0;
      x.ya[s] = (int)(((long long)x.mod * p.blocks_a + block) * p.M + x.m0);
      x.yb[s] = (int)(((long long)x.mod * p.pairs + pair) * p.N + x.n0);
      x.kb[s] = 0;
      x.nk[s] = p.kc;
    }
  }
  return x;
}

// Persistent and warp-specialised: warp 0 TMA, warp 1 MMA, warps 2-9 epilogue (a TMEM lane
// quarter and a column half each).  The two TMEM accumulators alternate between chunks of
// kChunk K blocks; the epilogue warps add each chunk to their running residues (BN / 2
// registers per thread) and reduce modulo p while the other accumulator fills: two FP32
// instructions per element and chunk.  Sixteen planes of 3600 x 3600 x 3600: 921 us (1.62 PFLOP/s)
// against 993 with four, of 3600 x 3600 x 400 159 against 180 (seventeen: 169).  Every wait is
// bounded; an expired one leaves its code in *status and the caller's outputs become NaN.
template <int BN, bool TRIP>
static __global__ void __launch_bounds__(kGemmThreads, 1)
    rns_gemm_kernel(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmArgs p,
                    unsigned units) {
  using L = RSmem<BN>;
  constexpr int S = L::STAGES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint8_t* sA = base;
  uint8_t* sB = base + S * L::A_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(base + S * L::STAGE);
  uint64_t* empty = full + S;
  uint64_t* tfull = empty + S;
  uint64_t* tempty = tfull + 2;
  uint64_t* mdone = tempty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mdone + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], kEpiWarps);
    }
    mbar_init(mdone, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(L::TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      bool stop = false;
      const uint32_t bytes = (uint32_t)(BM + p.bs) * KBYTES;
      for (unsigned u = blockIdx.x; u < units && !stop; u += gridDim.x) {
        const Unit x = decode_unit<TRIP, true>(p, u);
#pragma unroll
        for (int g = 0; g < (TRIP ? 2 : 1); ++g) {
          const CUtensorMap* ta = &maps.a[x.ma[g]];
          const CUtensorMap* tb = &maps.b[x.mb[g]];
          for (int kb = x.kb[g]; kb < x.kb[g] + x.nk[g] && !stop; ++kb, ++it) {
            const int s = it % S;
            if (it >= S && !mbar_wait(&empty[s], ((it / S) - 1) & 1, p.wait_ns)) {
              atomicExch(p.status, kStatusTimeoutEmpty);
              *abort_flag = 1;
            }
            if (*abort_flag) {
              stop = true;
              break;
            }
            mbar_expect_tx(&full[s], bytes);
            tma_load_2d(ta, &full[s], sA + s * L::A_BYTES, kb * 64, x.ya[g]);
            tma_load_2d(tb, &full[s], sB + s * L::B_BYTES, kb * 64, x.yb[g]);
          }
        }
      }
      if (stop)  // copies in flight land before the CTA gives up its shared memory
        for (int j = max(0, it - S); j < it; ++j)
          mbar_wait(&full[j % S], (j / S) & 1, p.wait_ns);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) |
                             ((uint32_t)(p.bs >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
      int it = 0, c = 0;
      bool stop = false;
      for (unsigned u = blockIdx.x; u < units && !stop; u += gridDim.x) {
        const int blocks = decode_unit<TRIP, false>(p, u).blocks;
        for (int k0 = 0; k0 < blocks && !stop; k0 += kChunk, ++c) {
          const int b = c & 1;
          if (c >= 2 && !mbar_wait(&tempty[b], ((c >> 1) - 1) & 1, p.wait_ns)) {
            atomicExch(p.status, kStatusTimeoutEmpty);
            *abort_flag = 1;
          }
          if (*abort_flag) {
            stop = true;
            break;
          }
          tc_fence_after();
          const uint32_t d = tmem + (uint32_t)(b * BN);
          uint32_t acc = 0u;
          const int n = min(kChunk, blocks - k0);
          for (int kb = 0; kb < n; ++kb, ++it) {
            const int s = it % S;
            if (!mbar_wait(&full[s], (it / S) & 1, p.wait_ns)) {
              atomicExch(p.status, kStatusTimeoutFull);
              *abort_flag = 1;
            }
            if (*abort_flag) {
              stop = true;
              break;
            }
            tc_fence_after();
            const uint64_t da = sw128_desc(smem_u32(sA + s * L::A_BYTES));
            const uint64_t db = sw128_desc(smem_u32(sB + s * L::B_BYTES));
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              umma_f16(d, da + 2 * k, db + 2 * k, idesc, acc);
              acc = 1u;
            }
            umma_commit(&empty[s]);
          }
          umma_commit(&tfull[b]);
        }
      }
      umma_commit(mdone);
      mbar_wait(mdone, 0, p.wait_ns);  // every MMA retired before TMEM is released
    }
    __syncwarp();
  } else {
    const int q = warp & 3, h = (warp - 2) >> 2;
    constexpr int HB = BN / 2;  // columns of this warp: [h HB, (h + 1) HB) of the tile
    int c = 0;
    bool stop = false;
    for (unsigned u = blockIdx.x; u < units && !stop; u += gridDim.x) {
      const Unit x = decode_unit<TRIP, false>(p, u);
      const unsigned long long np = pair(-p.t.p[x.mod], -p.t.p[x.mod]),
                               inv = pair(p.t.inv[x.mod], p.t.inv[x.mod]);
      unsigned long long r[HB / 2];  // two columns each
#pragma unroll
      for (int j = 0; j < HB / 2; ++j) r[j] = 0;
      for (int k0 = 0; k0 < x.blocks; k0 += kChunk, ++c) {
        const int b = c & 1;
        int okw = 1;
        if (lane == 0) {
          okw = mbar_wait_sleep(&tfull[b], (c >> 1) & 1, p.wait_ns) ? 1 : 0;
          if (!okw) {
            atomicExch(p.status, kStatusTimeoutDone);
            *abort_flag = 1;
          }
          if (*abort_flag) okw = 0;
        }
        if (!__shfl_sync(0xffffffffu, okw, 0)) {  // warp-uniform: tcgen05.ld is .sync.aligned
          stop = true;
          break;
        }
        tc_fence_after();
        const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BN + h * HB);
#pragma unroll
        for (int f = 0; f < HB / 32; ++f) {
          if (h * HB + 32 * f >= p.bs) break;  // columns the tile does not have
          uint32_t v[32];
          tmem_ld32(tbase + 32 * f, v);
#pragma unroll
          for (int j = 0; j < 16; ++j)
            r[16 * f + j] = mod_near_pair(
                add_pair(pair(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])),
                         r[16 * f + j]),
                np, inv);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty[b]);
      }
      if (stop) break;
      const long long row = x.m0 + q * 32 + lane;
      if (row < p.M) {
        unsigned char* o = p.out + (((long long)x.plane * NP + x.mod) * p.M + row) * p.ld;
        const bool mags = x.mod == NM;
#pragma unroll
        for (int f = 0; f < HB / 16; ++f) {
          const int cj = h * HB + 16 * f;  // 16 columns: inside the tile and the row, or not at all
          if (cj < p.bs && x.n0 + cj < p.ld) {
            float e[16];
#pragma unroll
            for (int j = 0; j < 8; ++j) unpair(r[8 * f + j], e[2 * j], e[2 * j + 1]);
            uint4 w;
            if (mags)
              w = make_uint4(exponent_bytes(e[0], e[1], e[2], e[3]),
                             exponent_bytes(e[4], e[5], e[6], e[7]),
                             exponent_bytes(e[8], e[9], e[10], e[11]),
                             exponent_bytes(e[12], e[13], e[14], e[15]));
            else
              w = make_uint4(residue_bytes(e[0], e[1], e[2], e[3]),
                             residue_bytes(e[4], e[5], e[6], e[7]),
                             residue_bytes(e[8], e[9], e[10], e[11]),
                             residue_bytes(e[12], e[13], e[14], e[15]));
            *reinterpret_cast<uint4*>(o + x.n0 + cj) = w;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(L::TMEM_COLS));
  }
}

// ---- residues -> FP64 ---------------------------------------------------------------------
// Four outputs' sums of residue times floor(2^96 q / p), in three words of 64-bit accumulators.
struct CrtSum {
  unsigned long long s0[4], s1[4], s2[4];
  __device__ __forceinline__ CrtSum(const CrtTab& t) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      s0[e] = t.b0;
      s1[e] = t.b1;
      s2[e] = t.b2;
    }
  }
  // w[l]: the four outputs' bytes of plane l
  __device__ __forceinline__ void add(const CrtTab& t, const unsigned (&w)[NP]) {
#pragma unroll
    for (int l = 0; l < NM; ++l)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const unsigned r = __byte_perm(w[l], 0u, 0x4440u + e);
        s0[e] += (unsigned long long)r * t.c0[l];
        s1[e] += (unsigned long long)r * t.c1[l];
        s2[e] += (unsigned long long)r * t.c2[l];
      }
  }
  // output e: the signed fraction of P (their integer part fell out modulo 2^96) times 2^ex times
  // t.scale, rounded to FP64 in integer arithmetic (GB300's FP64 pipe converts two values per
  // clock and SM) and multiplied once; exponents that could make the intermediate subnormal
  // scale last
  __device__ __forceinline__ double value(const CrtTab& t, int e, int ex) const {
    const unsigned long long t1 = s1[e] + (s0[e] >> 32);
    const unsigned w2 = (unsigned)s2[e] + (unsigned)(t1 >> 32);
    unsigned long long hi = ((unsigned long long)w2 << 32) | (unsigned)t1;
    unsigned lo = (unsigned)s0[e];
    const bool neg = (w2 >> 31) != 0;
    if (neg) {  // two's complement of the 96 bits
      lo = ~lo + 1u;
      hi = ~hi + (lo == 0u ? 1ull : 0ull);
    }
    double v;
    if (hi == 0 || ex < -800 || ex > 800) {
      v = scalbn(fma(__ull2double_rn(hi), 4294967296.0, __uint2double_rn(lo)) * t.scale, ex);
    } else {
      const int lz = __clzll((long long)hi);
      const unsigned long long top =
          lz ? (hi << lz) | (((unsigned long long)lo << 32) >> (64 - lz)) : hi;
      unsigned long long m = top >> 11;
      const unsigned rest = (unsigned)top & 0x7ffu;
      m += (rest > 0x400u || (rest == 0x400u && (m & 1ull))) ? 1ull : 0ull;
      // top 2^(32 - lz) = m 2^(43 - lz), with m's leading bit added into the exponent field
      v = __longlong_as_double(
              (long long)(m + ((unsigned long long)(1023 + 94 - lz + ex) << 52))) * t.scale;
    }
    return __longlong_as_double(__double_as_longlong(v) ^
                                (neg ? (long long)0x8000000000000000ull : 0ll));
  }
};

// ---- host side --------------------------------------------------------------------------
struct Tables {
  ModTab mod;
  PairTab pairs;
  CrtTab crt;
};

inline const Tables& tables() {
  static const Tables t = [] {
    Tables x{};
    unsigned __int128 P = 1;
    for (int p : kModuli) P *= (unsigned)p;
    for (int l = 0; l < NM; ++l) {
      const int p = kModuli[l];
      auto sym = [p](long long r) { r %= p; return (float)(2 * r > p ? r - p : r); };
      x.mod.p[l] = (float)p;
      x.mod.inv[l] = 1.0f / (float)p;
      x.mod.c1[l] = sym(1ll << digit_bit(1));
      x.mod.c2[l] = sym(1ll << digit_bit(2));
      x.mod.c3[l] = sym(1ll << digit_bit(3));
      auto twice = [](float f) {
        unsigned u;
        std::memcpy(&u, &f, 4);
        return (unsigned long long)u << 32 | u;
      };
      x.pairs.np[l] = twice(-x.mod.p[l]);
      x.pairs.inv[l] = twice(x.mod.inv[l]);
      x.pairs.c1[l] = twice(x.mod.c1[l]);
      x.pairs.c2[l] = twice(x.mod.c2[l]);
      x.pairs.c3[l] = twice(x.mod.c3[l]);
      const unsigned m = (unsigned)((P / (unsigned)p) % (unsigned)p);
      unsigned q = 1;
      while ((q * m) % p != 1) ++q;
      unsigned long long rem = q;
      unsigned* w[3] = {x.crt.c2, x.crt.c1, x.crt.c0};
      for (auto* word : w) {
        word[l] = (unsigned)((rem << 32) / p);
        rem = (rem << 32) % p;
      }
    }
    x.crt.scale = std::ldexp((double)P, -96);
    return x;
  }();
  return t;
}

// The tables of a join that adds up `planes` planes of biased bytes and scales by alpha.
inline CrtTab crt_tab(int planes, double alpha) {
  CrtTab t = tables().crt;
  unsigned __int128 sum = 0;
  for (int l = 0; l < NM; ++l)
    sum += ((unsigned __int128)t.c2[l] << 64) | ((unsigned __int128)t.c1[l] << 32) | t.c0[l];
  const unsigned __int128 b = -(sum * 128 * (unsigned)planes);
  t.b0 = (unsigned)b;
  t.b1 = (unsigned)(b >> 32);
  t.b2 = (unsigned)(b >> 64);
  t.scale *= alpha;
  return t;
}

inline long long up(long long x, long long m) { return (x + m - 1) / m * m; }

inline int blocks_for(long long n, int per) {
  return (int)std::max(1LL, std::min((n + per - 1) / per, 16LL * num_sms()));
}

// Scratch for the sums of K segments: `bytes` of each operand's panel, which is packed later.
struct NormScratch {
  void* at[2];
  long long bytes[2];
};

inline int run_norm(const Operand& a, const Operand& b, long long k0, long long k1,
                    const NormScratch& scratch, cudaStream_t st) {
  NormArgs p{};
  p.o[0] = a;
  p.o[1] = b;
  p.k0 = k0;
  p.k1 = k1;
  const long long K = k1 - k0;
  for (int s = 0; s < 2; ++s) {
    const Operand& o = p.o[s];
    if (o.R == 0) continue;
    p.slices[s] = !o.kfast && K >= 512 && o.R < 256LL * 8 * num_sms();
    const int rows = o.kfast ? 8 : (p.slices[s] ? 32 : 256);
    p.gx[s] = (o.R + rows - 1) / rows;
    // about eight blocks per SM; each a few hundred K, and few enough parts to add up at the end
    const long long most = o.kfast ? K / 512 : (p.slices[s] ? std::min(K / 256, 128LL) : K / 32);
    const long long segs = std::max(1LL, std::min({(8LL * num_sms() + p.gx[s] - 1) / p.gx[s], most,
                                                   scratch.bytes[s] / (8 * o.R)}));
    p.seg[s] = (K + segs - 1) / segs;
    p.segs[s] = (K + p.seg[s] - 1) / p.seg[s];
    p.blocks[s] = p.gx[s] * p.segs[s];
    p.part[s] = (unsigned long long*)scratch.at[s];
  }
  rns_norm_kernel<<<(unsigned)(p.blocks[0] + p.blocks[1]), 256, 0, st>>>(p);
  PCG_CHECK_LAUNCH("rns norm");
  return 0;
}

inline int run_pack(PackArgs& p, cudaStream_t st) {
  for (PackSide& s : p.s) {
    const int rows = s.o.kfast ? 32 : 64;
    s.blocks = ((p.width + 63) >> 6) * ((s.nrow + rows - 1) / rows);
  }
  rns_pack_kernel<<<(unsigned)(p.s[0].blocks + p.s[1].blocks), 256, 0, st>>>(p);
  PCG_CHECK_LAUNCH("rns pack");
  return 0;
}

template <int BN, bool TRIP>
inline int run_gemm(const GemmMaps& maps, const GemmArgs& a, cudaStream_t st) {
  const int smem = RSmem<BN>::TOTAL;
  cudaFuncSetAttribute(rns_gemm_kernel<BN, TRIP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       smem);
  const long long units = a.mt * a.nt * NP * a.planes;
  if (units > 0x7fffffffLL) {
    set_error("rns gemm: %lld units of work", units);
    return -1;
  }
  rns_gemm_kernel<BN, TRIP>
      <<<(unsigned)std::min<long long>(units, num_sms()), kGemmThreads, smem, st>>>(
          maps, a, (unsigned)units);
  PCG_CHECK_LAUNCH("rns gemm");
  return 0;
}

}  // namespace rns
}  // namespace pcg
