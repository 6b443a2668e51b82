// FP64 strided contraction on the BF16 tensor cores, in residue arithmetic.
//
//   C[m, n] = beta * C[m, n] + alpha * sum_k A[m, k] * B[n, k]        (all FP64)
//
// GB300 multiplies FP64 at about 1.2 TFLOP/s and BF16 at about 1.9 PFLOP/s, so an FP64 product
// that is taken apart into exact BF16 products is cheaper than one on the FP64 pipe even at
// sixteen BF16 products each.  The method is the Chinese-remainder form of the Ozaki scheme
// (Ozaki, Uchino, Imamura 2025: integer matrix products modulo many small moduli):
//
// 1. Every row of A and of B is scaled by a power of two, so that its 2-norm is at most
//    2^61.9, and rounded to integers.  This is the only rounding before step 4: it leaves
//    about 2^-62.5 |a_i| |b_j|, where FP64 multiply-adds leave 2^-55 (K = 64) to 2^-58 (K = 50000).
// 2. The integers are reduced modulo 16 pairwise coprime moduli p <= 256 to residues
//    |r| <= 128, which BF16 holds exactly.
// 3. For each modulus a tcgen05 GEMM multiplies the residues.  A chunk of 960 K adds up to at
//    most 960 * 2^14 < 2^24, so the FP32 accumulator in TMEM is exact; the epilogue warps
//    reduce every chunk modulo p and keep the running residue in registers.
// 4. The integer sum is at most |a'_i| |b'_j| (Cauchy-Schwarz), below half the product of the
//    moduli (2^125.4), so the residues determine it exactly.  It is rebuilt as a 96-bit
//    fraction of that product, rounded to FP64, scaled back and added into C.
//
// A row with an infinity or a NaN (or a column of B) takes its outputs from a plain FP64
// dot product in step 4, so non-finite inputs give what FP64 arithmetic gives.
//
// Measured on GB300 against the FP64 kernel (contract_f64.cu), no = 20, nv = 180: the ladder
// 'ijef,abef->ijab' 882 -> 22.9 ms (GEMM 11.7, residues 9.8), a ring 'imae,mbej->ijab' 90.8 ->
// 1.50 ms; at no = 9, nv = 53 3.2 -> 0.18 ms and 0.46 -> 0.09 ms.
//
// The offsets of strided rows, columns and K indices are expanded into tables once per call;
// operands larger than the workspace go through in panels of rows, columns or K.
#include "tc_common.cuh"
#include <cuda_bf16.h>
#include <algorithm>
#include <cmath>

namespace pcg {
namespace rns {

using namespace pcg::tc;

// The largest 16 pairwise coprime moduli that BF16 residues allow.  The rounding of the scaled
// integers, relative to the sum, grows with sqrt(K) and with the spread of a row's magnitudes;
// measured against 113-bit sums, 15 moduli (2^-58.5 |a| |b|) fall behind the FP64 kernel at
// K = 50000 with magnitudes spread over e^+-4 (8.7e-16 against 5.8e-16 of the sums' norm), 16
// stay ahead of it everywhere.
constexpr int NM = 16;
constexpr int kModuli[NM] = {256, 255, 253, 251, 247, 241, 239, 233,
                             229, 227, 223, 217, 211, 199, 197, 193};
constexpr int kBits2 = 123;         // |a'|^2 |b'|^2 <= 2^(2 * 123.75); log2(product / 2) = 124.4
// first bit of the four digits of a scaled integer (16, 15, 15 and 16 bits): with residues of
// the powers of at most 127, a digit sum stays below 2^16 + 127 * 2^17 < 2^24, exact in FP32
__host__ __device__ constexpr int digit_bit(int q) { return q == 0 ? 0 : (q == 4 ? 62 : 1 + 15 * q); }
constexpr int kChunk = 15;          // 64-K blocks per exact FP32 accumulation: 960 K
constexpr float kMagic = 12582912.f;  // 1.5 * 2^23: adding it rounds to an integer

// Per modulus: p, 1/p and the residues of 2^16, 2^31, 2^46 (symmetric).
struct ModTab {
  float p[NM], inv[NM], c1[NM], c2[NM], c3[NM];
};
// Per modulus floor(2^96 q / p), q = ((P / p)^-1 mod p), in three 32-bit words; scale = P 2^-96.
struct CrtTab {
  unsigned c0[NM], c1[NM], c2[NM];
  double scale;
};
static_assert(NM * 8 <= 128, "the product fits a 128-bit integer");

// Nearest residue of an integer-valued t, |t| < 2^24: t / p is below 2^17 and FP32's 1/p is
// off by 2^-25 relative, so the quotient is off its nearest integer by less than 0.51 and
// |r| <= 128 for every p <= 256.
__device__ __forceinline__ float mod_near(float t, float p, float inv) {
  const float q = fmaf(t, inv, kMagic) - kMagic;
  return fmaf(-p, q, t);
}

struct Operand {
  const double* X;
  SubIdx r;             // rows: s0 = strides in X, s1 = strides in C
  long long R;          // rows
  long long* off;       // [R] element offset of each row in X
  long long* coff;      // [R] element offset of each row (or column) in C
  int* walk;            // [R] rows in an order whose neighbours are close in X
  unsigned* top;        // [R] biased exponent of the row's largest |x| (2047: Inf or NaN)
  float* norm2;         // [R] sum of the row's squares, each term truncated to 20 bits
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
  o.coff[r] = o1;
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

__global__ void rns_tables_kernel(const TableArgs t) {
  const long long total = t.a.R + t.b.R + t.K;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    if (i == 0) *t.status = 0;
    if (i < t.a.R) {
      fill_row(t.a, i);
      t.a.top[i] = 0;
      t.a.norm2[i] = 0.f;
    } else if (i < t.a.R + t.b.R) {
      fill_row(t.b, i - t.a.R);
      t.b.top[i - t.a.R] = 0;
      t.b.norm2[i - t.a.R] = 0.f;
    } else {
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

// |x| as FP32 from the upper word of a double (20 mantissa bits, truncated); below FP32's
// range 0, above it infinity.
__device__ __forceinline__ float abs_hi_f32(unsigned h) {
  h &= 0x7fffffffu;
  if (h < (897u << 20)) return 0.f;
  return h < (1151u << 20) ? __uint_as_float((h - (896u << 20)) << 3)
                           : __uint_as_float(0x7f800000u);
}

// Largest exponent and sum of squares of each row over K indices [k0, k1): one read of the
// operand, bound by HBM.  Gathered along K (KF: a warp per row) or along the rows (a thread
// per row), eight loads in flight per lane; blockIdx.y cuts K.
template <bool KF>
__device__ __forceinline__ void norm_rows(const Operand& o, long long k0, long long k1,
                                          long long seg, long long bx, long long by) {
  const long long kb = k0 + by * seg, ke = min(k1, kb + seg);
  const int lane = threadIdx.x & 31;
  const long long w = KF ? bx * 8 + (threadIdx.x >> 5) : bx * 256 + threadIdx.x;
  if (w >= o.R) return;
  constexpr int STEP = KF ? 32 : 1;
  const int row = o.walk[w];
  const double* x = o.X + o.off[row];
  unsigned m = 0;
  float s = 0.f;
  long long k = kb + (KF ? lane : 0);
  for (; k + 7 * STEP < ke; k += 8 * STEP) {
    unsigned h[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      h[u] = (unsigned)__double2hiint(__ldg(x + k_offset(o, k + STEP * u)));
    float t = 0.f;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float f = abs_hi_f32(h[u]);
      m = max(m, h[u] & 0x7fffffffu);
      t = fmaf(f, f, t);
    }
    s += t;
  }
  for (; k < ke; k += STEP) {
    const unsigned h = (unsigned)__double2hiint(__ldg(x + k_offset(o, k)));
    const float f = abs_hi_f32(h);
    m = max(m, h & 0x7fffffffu);
    s = fmaf(f, f, s);
  }
  if (KF) {
    for (int d = 16; d > 0; d >>= 1) {
      m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
      s += __shfl_xor_sync(0xffffffffu, s, d);
    }
    if (lane != 0) return;
  }
  atomicMax(o.top + row, m >> 20);
  atomicAdd(o.norm2 + row, s);
}

struct NormArgs {
  Operand o[2];
  long long gx[2], blocks[2], seg[2];  // row blocks, blocks and K segment of each operand
  long long k0, k1;
};

// Both operands in one launch: the first blocks take A, the others B.
__global__ void __launch_bounds__(256) rns_norm_kernel(const __grid_constant__ NormArgs p) {
  const int side = blockIdx.x >= p.blocks[0];
  const long long b = (long long)blockIdx.x - (side ? p.blocks[0] : 0);
  const long long bx = b % p.gx[side], by = b / p.gx[side];
  if (p.o[side].kfast)
    norm_rows<true>(p.o[side], p.k0, p.k1, p.seg[side], bx, by);
  else
    norm_rows<false>(p.o[side], p.k0, p.k1, p.seg[side], bx, by);
}

// Power of two s of a row: |x| 2^s has a 2-norm of at most 2^61.9.  From the sum of squares
// where FP32 holds it (1 + 2^-7 covers its truncation and summation), else from the largest
// element and K.  A zero row may take any.
__device__ __forceinline__ int row_shift(const Operand& o, long long row, int log2k) {
  const float n2 = o.norm2[row] * 1.0078125f;
  if (n2 >= 0x1p-80f && n2 <= 0x1p100f) {
    const unsigned u = __float_as_uint(n2);
    const int e = (int)(u >> 23) - 127;
    // log2 n2 <= e + 0.75 or e + 1.75
    return ((u & 0x7fffffu) < 0x570000u ? kBits2 - e : kBits2 - 1 - e) >> 1;
  }
  return (kBits2 - log2k - 2 * (max((int)o.top[row], 1) - 1022)) >> 1;
}

// The four digits (with the sign) of x 2^s rounded to an integer of at most 62 bits.
__device__ __forceinline__ void digits(double x, int s, float (&d)[4]) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  int ex = (int)((hi >> 20) & 0x7ffu);
  unsigned long long m = ((unsigned long long)(hi & 0xfffffu) << 32) | lo;
  if (ex)
    m |= 1ull << 52;
  else
    ex = 1;
  const int sh = ex - 1075 + s;  // at most 9, since |x| 2^s <= 2^61.9
  if (ex == 2047)
    m = 0;  // the row's outputs come from the FP64 dot product
  else if (sh >= 0)
    m <<= sh;
  else if (sh > -55)
    m = (m + (1ull << (-sh - 1))) >> -sh;
  else
    m = 0;
  const unsigned sign = hi & 0x80000000u;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const unsigned v = (unsigned)(m >> digit_bit(q)) & ((1u << (digit_bit(q + 1) - digit_bit(q))) - 1);
    d[q] = __uint_as_float(__float_as_uint(__uint_as_float(0x4b000000u | v) - 8388608.f) ^ sign);
  }
}

struct PackSide {
  Operand o;
  long long w0, nrow;  // rows of this panel: walk positions [w0, w0 + nrow); nrow 0: none
  __nv_bfloat16* out;  // [modulus][nrow][Kp]
  long long blocks;
};

struct PackArgs {
  PackSide s[2];
  long long k0, K, Kp;  // K indices [k0, k0 + K), padded with zeros to Kp
  int log2k;            // ceil(log2 K)
  ModTab t;
};

// Residues of two neighbouring K entries for every modulus, one 32-bit store per modulus: an
// integer of at most 8 bits is exact in the upper half of its FP32 word, which is BF16.
__device__ __forceinline__ void store_residues(const PackArgs& p, const PackSide& o, double x0,
                                               double x1, int s, long long at) {
  float a[4], b[4];
  digits(x0, s, a);
  digits(x1, s, b);
  unsigned* out = reinterpret_cast<unsigned*>(o.out + at);
  const long long plane = (o.nrow * p.Kp) >> 1;
#pragma unroll
  for (int l = 0; l < NM; ++l) {
    const float t0 = fmaf(a[3], p.t.c3[l], fmaf(a[2], p.t.c2[l], fmaf(a[1], p.t.c1[l], a[0])));
    const float t1 = fmaf(b[3], p.t.c3[l], fmaf(b[2], p.t.c2[l], fmaf(b[1], p.t.c1[l], b[0])));
    const float r0 = mod_near(t0, p.t.p[l], p.t.inv[l]), r1 = mod_near(t1, p.t.p[l], p.t.inv[l]);
    out[l * plane] = __byte_perm(__float_as_uint(r0), __float_as_uint(r1), 0x7632);
  }
}

// Operand -> residues: 8 bytes read and 2 NM written per element, about 7 NM FP32
// instructions; bound by the writes (9.8 ms at 1.05e9 elements, 4.3 of 6.8 TB/s).  Gathered along K, a
// warp takes 64 K of a row, four rows at a time, straight from global memory.  Otherwise a tile
// of 64 walked rows x 64 K goes through shared memory, read along the rows.  One launch packs a
// panel of each operand: the first blocks take A's, the others B's.
__global__ void __launch_bounds__(256, 5) rns_pack_kernel(const __grid_constant__ PackArgs p) {
  __shared__ double tile[64][65];
  __shared__ long long off[64], kof[64];
  __shared__ int srow[64], ssh[64];
  const int side = blockIdx.x >= p.s[0].blocks;
  const PackSide& ps = p.s[side];
  const Operand& o = ps.o;
  const long long b = (long long)blockIdx.x - (side ? p.s[0].blocks : 0);
  const long long nk = p.Kp >> 6;
  const long long w = (b / nk) * (o.kfast ? 32 : 64);  // first row of the block
  const long long kk0 = (b % nk) * 64;                 // first K, in the panel
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (o.kfast) {
    const long long ka = kk0 + 2 * lane, kb = ka + 1;
    const long long oa = ka < p.K ? k_offset(o, p.k0 + ka) : 0;
    const long long ob = kb < p.K ? k_offset(o, p.k0 + kb) : 0;
    const long long w1 = w + 4 * warp;
    double x[4], y[4];
    int row[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      x[u] = y[u] = 0.0;
      row[u] = 0;
      if (w1 + u < ps.nrow) {
        row[u] = o.walk[ps.w0 + w1 + u];
        const double* q = o.X + o.off[row[u]];
        if (ka < p.K) x[u] = __ldg(q + oa);
        if (kb < p.K) y[u] = __ldg(q + ob);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (w1 + u < ps.nrow)
        store_residues(p, ps, x[u], y[u], row_shift(o, row[u], p.log2k),
                       (row[u] - ps.w0) * p.Kp + kk0 + 2 * lane);
  } else {
    if (threadIdx.x < 64) {
      kof[threadIdx.x] = kk0 + threadIdx.x < p.K ? k_offset(o, p.k0 + kk0 + threadIdx.x) : 0;
      if (w + threadIdx.x < ps.nrow) {
        const int r = o.walk[ps.w0 + w + threadIdx.x];
        srow[threadIdx.x] = r;
        off[threadIdx.x] = o.off[r];
        ssh[threadIdx.x] = row_shift(o, r, p.log2k);
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
    for (int r = warp; r < 64 && w + r < ps.nrow; r += 8)
      store_residues(p, ps, tile[r][2 * lane], tile[r][2 * lane + 1], ssh[r],
                     (srow[r] - ps.w0) * p.Kp + kk0 + 2 * lane);
  }
}

// ---- GEMM over the residues -------------------------------------------------------------
struct GemmArgs {
  long long M, N;    // rows of A and of B in this panel
  long long mt, nt;  // 128-row and bs-column tiles
  int gm;            // M tiles per raster group
  int bs;            // columns per N tile, a multiple of 16
  int splits, nkb, kb_per_split;
  long long ld;      // bytes of one output row: N rounded up to 16
  unsigned char* out;  // [split][modulus][M][ld]
  int* status;
  unsigned long long wait_ns;
  ModTab t;
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

struct Unit {
  int split, mod, n0;
  long long m0;
};

// Unit u -> (split, modulus, tile); the tile order within a modulus is tc_gemm_kernel's raster
// (groups of gm M tiles, M fastest), so a wave shares the row blocks of both operands in L2.
__device__ __forceinline__ Unit decode_unit(const GemmArgs& p, long long u) {
  const long long per = p.mt * p.nt;
  Unit x;
  const long long g = u / per, r = u % per;
  x.mod = (int)(g % NM);
  x.split = (int)(g / NM);
  const long long group = r / ((long long)p.gm * p.nt), rg = r % ((long long)p.gm * p.nt);
  const long long here = min((long long)p.gm, p.mt - group * p.gm);
  x.m0 = (group * p.gm + rg % here) * BM;
  x.n0 = (int)((rg / here) * p.bs);
  return x;
}

// Persistent and warp-specialised: warp 0 TMA, warp 1 MMA, warps 2-9 epilogue (a TMEM lane
// quarter and a column half each).  The two TMEM accumulators alternate between chunks of
// kChunk K blocks; the epilogue warps add each chunk to their running residues (BN / 2
// registers per thread) and reduce modulo p while the other accumulator fills: four FP32
// instructions per element and chunk, an eighth of the chunk's MMA time.  Every wait is
// bounded; an expired one leaves its code in *status and the caller's outputs become NaN.
template <int BN>
__global__ void __launch_bounds__(kGemmThreads, 1)
    rns_gemm_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
                    const __grid_constant__ GemmArgs p) {
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
  const long long units = p.mt * p.nt * NM * p.splits;

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
      for (long long u = blockIdx.x; u < units && !stop; u += gridDim.x) {
        const Unit x = decode_unit(p, u);
        const int ya = (int)(x.mod * p.M + x.m0), yb = (int)(x.mod * p.N + x.n0);
        const int kb1 = min(p.nkb, (x.split + 1) * p.kb_per_split);
        for (int kb = x.split * p.kb_per_split; kb < kb1; ++kb, ++it) {
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
          tma_load_2d(&ta, &full[s], sA + s * L::A_BYTES, kb * 64, ya);
          tma_load_2d(&tb, &full[s], sB + s * L::B_BYTES, kb * 64, yb);
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
      for (long long u = blockIdx.x; u < units && !stop; u += gridDim.x) {
        const Unit x = decode_unit(p, u);
        const int kb1 = min(p.nkb, (x.split + 1) * p.kb_per_split);
        for (int kc = x.split * p.kb_per_split; kc < kb1 && !stop; kc += kChunk, ++c) {
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
          const int ke = min(kb1, kc + kChunk);
          for (int kb = kc; kb < ke; ++kb, ++it) {
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
    for (long long u = blockIdx.x; u < units && !stop; u += gridDim.x) {
      const Unit x = decode_unit(p, u);
      const float pm = p.t.p[x.mod], inv = p.t.inv[x.mod];
      const int kb1 = min(p.nkb, (x.split + 1) * p.kb_per_split);
      float r[HB];
#pragma unroll
      for (int j = 0; j < HB; ++j) r[j] = 0.f;
      for (int kc = x.split * p.kb_per_split; kc < kb1; kc += kChunk, ++c) {
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
          uint32_t v[32];
          tmem_ld32(tbase + 32 * f, v);
#pragma unroll
          for (int j = 0; j < 32; ++j)
            r[32 * f + j] = mod_near(__uint_as_float(v[j]) + r[32 * f + j], pm, inv);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty[b]);
      }
      if (stop) break;
      const long long row = x.m0 + q * 32 + lane;
      if (row < p.M) {
        unsigned char* o = p.out + (((long long)x.split * NM + x.mod) * p.M + row) * p.ld;
#pragma unroll
        for (int f = 0; f < HB / 16; ++f) {
          const int cj = h * HB + 16 * f;  // 16 columns: inside the tile and the row, or not at all
          if (cj < p.bs && x.n0 + cj < p.ld) {
            unsigned w[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              unsigned e[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float v = r[16 * f + 4 * g + j];
                e[j] = __float_as_uint((v < 0.f ? v + pm : v) + 8388608.f);
              }
              w[g] = __byte_perm(__byte_perm(e[0], e[1], 0x0040), __byte_perm(e[2], e[3], 0x0040),
                                 0x5410);
            }
            *reinterpret_cast<uint4*>(o + x.n0 + cj) = make_uint4(w[0], w[1], w[2], w[3]);
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

// ---- residues -> C --------------------------------------------------------------------
struct JoinArgs {
  Operand a, b;
  long long m0, n0, M, N;  // this panel's rows and columns
  long long k0, K;
  int splits, log2k;
  long long ld;
  const unsigned char* res;  // [split][modulus][M][ld]
  double alpha, beta;
  double* C;
  const int* status;
  CrtTab t;  // t.scale: P 2^-96 alpha
};

// FP64 dot product of one output whose row or column holds an Inf or a NaN.
__device__ __noinline__ double plain_dot(const JoinArgs& p, long long row, long long col) {
  const double* x = p.a.X + p.a.off[row];
  const double* y = p.b.X + p.b.off[col];
  double s = 0.0;
  for (long long k = p.k0; k < p.k0 + p.K && !isnan(s); ++k)
    s = fma(x[k_offset(p.a, k)], y[k_offset(p.b, k)], s);
  return s;
}

// The 96-bit magnitude (hi, lo) times 2^ex times scale: rounded to FP64 in integer arithmetic
// (GB300's FP64 pipe converts two values per clock and SM) and multiplied once.  Exponents that
// could make the intermediate subnormal scale last.
__device__ __forceinline__ double scaled_f64(unsigned long long hi, unsigned lo, int ex,
                                             double scale) {
  if (hi == 0 || ex < -800 || ex > 800)
    return scalbn(fma(__ull2double_rn(hi), 4294967296.0, __uint2double_rn(lo)) * scale, ex);
  const int lz = __clzll((long long)hi);
  const unsigned long long top = lz ? (hi << lz) | (((unsigned long long)lo << 32) >> (64 - lz)) : hi;
  unsigned long long m = top >> 11;
  const unsigned rest = (unsigned)top & 0x7ffu;
  m += (rest > 0x400u || (rest == 0x400u && (m & 1ull))) ? 1ull : 0ull;
  // top 2^(32 - lz) = m 2^(43 - lz), with m's leading bit added into the exponent field
  return __longlong_as_double((long long)(m + ((unsigned long long)(1023 + 94 - lz + ex) << 52))) *
         scale;
}

// Four columns of one row per thread: for every modulus the residues times the three words of
// floor(2^96 q / p) are summed in 64-bit accumulators (their integer part falls out modulo
// 2^96), the signed fraction is rounded to FP64 and scaled.  Bound by the 64-bit multiply-adds
// (3 NM per element) and, for short K, by the residues' and C's bytes.
__global__ void __launch_bounds__(256) rns_join_kernel(const __grid_constant__ JoinArgs p) {
  const unsigned nc = (unsigned)((p.N + 3) >> 2);
  const unsigned total = (unsigned)(p.M * nc);  // below 2^31 (host check)
  const bool failed = *p.status != 0;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const unsigned row = i / nc, col = 4 * (i - row * nc);
    unsigned long long s0[4] = {0, 0, 0, 0}, s1[4] = {0, 0, 0, 0}, s2[4] = {0, 0, 0, 0};
    for (int sp = 0; sp < p.splits; ++sp) {
      const unsigned char* src = p.res + ((long long)sp * NM * p.M + row) * p.ld + col;
      unsigned w[NM];
#pragma unroll
      for (int l = 0; l < NM; ++l)
        w[l] = __ldg(reinterpret_cast<const unsigned*>(src + (long long)l * p.M * p.ld));
#pragma unroll
      for (int l = 0; l < NM; ++l)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const unsigned r = (w[l] >> (8 * e)) & 0xffu;
          s0[e] += (unsigned long long)r * p.t.c0[l];
          s1[e] += (unsigned long long)r * p.t.c1[l];
          s2[e] += (unsigned long long)r * p.t.c2[l];
        }
    }
    const long long grow = p.m0 + row;
    const bool bad_row = p.a.top[grow] == 2047u;
    const int sa = row_shift(p.a, grow, p.log2k);
    double* crow = p.C + p.a.coff[grow];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (col + e >= p.N) break;
      const long long gcol = p.n0 + col + e;
      const unsigned long long t1 = s1[e] + (s0[e] >> 32);
      const unsigned w2 = (unsigned)s2[e] + (unsigned)(t1 >> 32);
      unsigned long long hi = ((unsigned long long)w2 << 32) | (unsigned)t1;
      unsigned lo = (unsigned)s0[e];
      const bool neg = (w2 >> 31) != 0;
      if (neg) {  // two's complement of the 96 bits
        lo = ~lo + 1u;
        hi = ~hi + (lo == 0u ? 1ull : 0ull);
      }
      double v = scaled_f64(hi, lo, -sa - row_shift(p.b, gcol, p.log2k), p.t.scale);
      v = __longlong_as_double(__double_as_longlong(v) ^ (neg ? 0x8000000000000000ll : 0ll));
      if (bad_row || p.b.top[gcol] == 2047u) v = p.alpha * plain_dot(p, grow, gcol);
      if (failed) v = __longlong_as_double(0x7ff8000000000000ll);
      double* dst = crow + p.b.coff[gcol];
      *dst = p.beta == 0.0 ? v : p.beta * *dst + v;
    }
  }
}

// ---- host side --------------------------------------------------------------------------
struct Tables {
  ModTab mod;
  CrtTab crt;
};

const Tables& tables() {
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

// How one call is cut: panels of M, N and K, and the workspace's layout.
struct Plan {
  long long PM, PN, PK, Kp;  // panel sizes (Kp: PK rounded up to the 64-K block)
  long long np_m, np_n, np_k;
  int splits, kb_per_split, bs, BN;
  long long nt, ld;
  long long tables, panel_a, panel_b, res, total;  // bytes
};

long long up(long long x, long long m) { return (x + m - 1) / m * m; }

bool size_plan(Plan& p, long long M, long long N, long long K) {
  p.PM = p.np_m == 1 ? M : up((M + p.np_m - 1) / p.np_m, BM);
  p.PN = p.np_n == 1 ? N : up((N + p.np_n - 1) / p.np_n, 64);
  p.PK = p.np_k == 1 ? K : up((K + p.np_k - 1) / p.np_k, 64);
  p.Kp = up(p.PK, 64);
  p.BN = p.PN > 128 ? 256 : (p.PN > 64 ? 128 : 64);
  p.nt = (p.PN + p.BN - 1) / p.BN;
  p.bs = (int)(16 * (((p.PN + 15) / 16 + p.nt - 1) / p.nt));
  p.ld = up(p.PN, 16);
  const long long nkb = p.Kp / 64, units = (p.PM + BM - 1) / BM * p.nt * NM;
  const int sms = num_sms();
  // fewer units than SMs: cut K (each part at least a chunk), the residues add up in the join
  int splits = 1;
  if (units < sms) splits = (int)std::max(1LL, std::min<long long>(sms / units, nkb / kChunk));
  splits = std::min(splits, 8);
  p.kb_per_split = (int)((nkb + splits - 1) / splits);
  p.splits = (int)((nkb + p.kb_per_split - 1) / p.kb_per_split);
  p.tables = up((M + N) * (8 + 8 + 4 + 4 + 4) + 16 * K + 256, 256);
  p.panel_a = up(p.PM * p.Kp * 2 * NM, 256);
  p.panel_b = up(p.PN * p.Kp * 2 * NM, 256);
  p.res = up((long long)p.splits * NM * p.PM * p.ld, 256);
  p.total = p.tables + p.panel_a + p.panel_b + p.res;
  return p.PM * NM < 0x7fffffffLL - BM && p.PN * NM < 0x7fffffffLL - 256 &&
         p.PM * (p.PN + 3) < 0x7fffffffLL &&
         (p.PM / 32 + p.PN / 32 + 4) * (p.Kp / 64) < 0x7fffffffLL;
}

// The fewest panels whose workspace fits in `limit` bytes: the larger operand panel is halved,
// K last (every K panel costs another pass over C).
bool make_plan(Plan& p, long long M, long long N, long long K, long long limit) {
  p = Plan{};
  p.np_m = p.np_n = p.np_k = 1;
  for (int it = 0; it < 64; ++it) {
    const bool ok = size_plan(p, M, N, K);
    if (ok && p.total <= limit) return true;
    if (p.PM > 256 && p.PM >= p.PN)
      p.np_m *= 2;
    else if (p.PN > 256)
      p.np_n *= 2;
    else if (p.PK > 1024)
      p.np_k *= 2;
    else
      return false;
  }
  return false;
}

bool fill_group(SubIdx& d, int n, const long long* ext, const long long* s0, const long long* s1,
                const char* what) {
  if (n < 0 || n > kMaxSub) {
    set_error("pcg_contract_rns_f64: %s has %d sub-indices (max %d)", what, n, kMaxSub);
    return false;
  }
  if (n > 0 && (!ext || !s0 || !s1)) {
    set_error("pcg_contract_rns_f64: %s extents or strides missing", what);
    return false;
  }
  d.n = std::max(n, 1);
  d.ext[0] = 1;
  d.s0[0] = d.s1[0] = 0;
  for (int q = 0; q < n; ++q) {
    if (ext[q] <= 0) {
      set_error("pcg_contract_rns_f64: %s extent %lld must be positive", what, ext[q]);
      return false;
    }
    d.ext[q] = ext[q];
    d.s0[q] = s0[q];
    d.s1[q] = s1[q];
  }
  return true;
}

// Smallest |stride| of a group's sub-indices with more than one element, and which it is.
long long near_stride(const SubIdx& d, bool second, int* at) {
  long long best = 0;
  for (int q = 0; q < d.n; ++q) {
    const long long s = llabs(second ? d.s1[q] : d.s0[q]);
    if (d.ext[q] > 1 && s > 0 && (best == 0 || s < best)) {
      best = s;
      if (at) *at = q;
    }
  }
  return best;
}

int blocks_for(long long n, int per) {
  return (int)std::max(1LL, std::min((n + per - 1) / per, 16LL * num_sms()));
}

int run_norm(const Operand& a, const Operand& b, long long k0, long long k1, cudaStream_t st) {
  NormArgs p{};
  p.o[0] = a;
  p.o[1] = b;
  p.k0 = k0;
  p.k1 = k1;
  const long long K = k1 - k0;
  for (int s = 0; s < 2; ++s) {
    const Operand& o = p.o[s];
    p.gx[s] = o.kfast ? (o.R + 7) / 8 : (o.R + 255) / 256;
    const long long most = std::max(1LL, K / (o.kfast ? 512 : 32));
    const long long segs = std::max(1LL, std::min((8LL * num_sms() + p.gx[s] - 1) / p.gx[s], most));
    p.seg[s] = (K + segs - 1) / segs;
    p.blocks[s] = p.gx[s] * ((K + p.seg[s] - 1) / p.seg[s]);
  }
  rns_norm_kernel<<<(unsigned)(p.blocks[0] + p.blocks[1]), 256, 0, st>>>(p);
  PCG_CHECK_LAUNCH("pcg_contract_rns_f64/norm");
  return 0;
}

int run_pack(PackArgs& p, cudaStream_t st) {
  for (PackSide& s : p.s) {
    const int rows = s.o.kfast ? 32 : 64;
    s.blocks = (p.Kp >> 6) * ((s.nrow + rows - 1) / rows);
  }
  rns_pack_kernel<<<(unsigned)(p.s[0].blocks + p.s[1].blocks), 256, 0, st>>>(p);
  PCG_CHECK_LAUNCH("pcg_contract_rns_f64/pack");
  return 0;
}

template <int BN>
int run_gemm(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& a, cudaStream_t st) {
  const int smem = RSmem<BN>::TOTAL;
  cudaFuncSetAttribute(rns_gemm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  const long long units = a.mt * a.nt * NM * a.splits;
  rns_gemm_kernel<BN><<<(unsigned)std::min<long long>(units, num_sms()), kGemmThreads, smem, st>>>(
      ta, tb, a);
  PCG_CHECK_LAUNCH("pcg_contract_rns_f64/gemm");
  return 0;
}

}  // namespace rns
}  // namespace pcg

using namespace pcg;
using namespace pcg::rns;

// Bytes of workspace for one M x N x K contraction within `limit` bytes, 0 when its panels
// cannot be cut to fit.
extern "C" int pcg_contract_rns_f64_work(long long M, long long N, long long K, long long limit,
                                         long long* bytes) {
  if (!bytes || M <= 0 || N <= 0 || K <= 0) {
    set_error("pcg_contract_rns_f64_work: bad arguments");
    return -1;
  }
  // the call may take either side as the columns
  Plan p, q;
  *bytes = 0;
  if (M < 0x7fffffffLL && N < 0x7fffffffLL && make_plan(p, M, N, K, limit) &&
      make_plan(q, N, M, K, limit))
    *bytes = std::max(p.total, q.total);
  return 0;
}

extern "C" int pcg_contract_rns_f64(int m_n, const long long* m_ext, const long long* m_sa,
                                    const long long* m_sc, int n_n, const long long* n_ext,
                                    const long long* n_sb, const long long* n_sc, int k_n,
                                    const long long* k_ext, const long long* k_sa,
                                    const long long* k_sb, double alpha, const double* A,
                                    const double* B, double beta, double* C, void* work,
                                    long long work_len, void* stream) {
  SubIdx m{}, n{}, k{};
  if (!fill_group(m, m_n, m_ext, m_sa, m_sc, "M") || !fill_group(n, n_n, n_ext, n_sb, n_sc, "N") ||
      !fill_group(k, k_n, k_ext, k_sa, k_sb, "K"))
    return -1;
  if (!A || !B || !C || !work || ((uintptr_t)work & 255u)) {
    set_error("pcg_contract_rns_f64: null operand, or a workspace not 256-byte aligned");
    return -1;
  }
  // the side with the output's unit stride becomes the columns, so that C is written along it
  const long long cm = near_stride(m, true, nullptr), cn = near_stride(n, true, nullptr);
  if (cm != 0 && (cn == 0 || cm < cn)) {
    std::swap(m, n);
    std::swap(A, B);
    std::swap(k.s0, k.s1);
  }
  const long long M = sub_total(m), N = sub_total(n), K = sub_total(k);
  Plan p;
  if (M >= 0x7fffffffLL || N >= 0x7fffffffLL || !make_plan(p, M, N, K, work_len)) {
    set_error("pcg_contract_rns_f64: %lld bytes of workspace do not hold a panel of %lld x %lld x "
              "%lld", work_len, M, N, K);
    return -1;
  }
  cudaStream_t st = (cudaStream_t)stream;
  // workspace: tables, panels of A and B, residues of the products
  unsigned char* w = (unsigned char*)work;
  unsigned char* tb = w;
  auto take = [&](long long bytes) {
    unsigned char* r = tb;
    tb += bytes;
    return r;
  };
  Operand a{}, b{};
  int* status = (int*)take(256);
  a.off = (long long*)take(8 * M);
  a.coff = (long long*)take(8 * M);
  b.off = (long long*)take(8 * N);
  b.coff = (long long*)take(8 * N);
  long long* ka = (long long*)take(8 * K);
  long long* kb = (long long*)take(8 * K);
  a.walk = (int*)take(4 * M);
  a.top = (unsigned*)take(4 * M);
  b.walk = (int*)take(4 * N);
  b.top = (unsigned*)take(4 * N);
  a.norm2 = (float*)take(4 * M);
  b.norm2 = (float*)take(4 * N);
  __nv_bfloat16* pa = (__nv_bfloat16*)(w + p.tables);
  __nv_bfloat16* pb = (__nv_bfloat16*)(w + p.tables + p.panel_a);
  unsigned char* res = w + p.tables + p.panel_a + p.panel_b;
  for (int side = 0; side < 2; ++side) {
    Operand& o = side ? b : a;
    o.X = side ? B : A;
    o.r = side ? n : m;
    o.R = side ? N : M;
    o.k = side ? kb : ka;
    o.kstep = k.n == 1 ? (side ? k.s1[0] : k.s0[0]) : 0;
    // gathered along K when the operand is at least as dense along it as along the rows
    o.wq = o.r.n - 1;
    int near = o.wq;
    const long long rs = near_stride(o.r, false, &near), ks = near_stride(k, side == 1, nullptr);
    o.kfast = rs == 0 || (ks != 0 && ks <= rs);
    // rows walked with their densest sub-index innermost, where one panel holds them all
    if (!o.kfast && (side ? p.np_n : p.np_m) == 1) o.wq = near;
  }
  const Tables& t = tables();
  TableArgs ta{a, b, k, K, ka, kb, status};
  rns_tables_kernel<<<blocks_for(M + N + K, 256), 256, 0, st>>>(ta);
  PCG_CHECK_LAUNCH("pcg_contract_rns_f64/tables");
  for (long long k0 = 0; k0 < K; k0 += p.PK) {
    const long long kn = std::min(p.PK, K - k0);
    int log2k = 0;
    while ((1LL << log2k) < kn) ++log2k;
    if (k0 > 0) {
      cudaMemsetAsync(a.top, 0, 4 * M, st);
      cudaMemsetAsync(b.top, 0, 4 * N, st);
      cudaMemsetAsync(a.norm2, 0, 4 * M, st);
      cudaMemsetAsync(b.norm2, 0, 4 * N, st);
    }
    if (run_norm(a, b, k0, k0 + kn, st)) return -2;
    for (long long n0 = 0; n0 < N; n0 += p.PN) {
      const long long nn = std::min(p.PN, N - n0);
      for (long long m0 = 0; m0 < M; m0 += p.PM) {
        const long long mm = std::min(p.PM, M - m0);
        // B's panel is packed with the first panel of A
        PackArgs q{{{a, m0, mm, pa, 0}, {b, n0, m0 == 0 ? nn : 0, pb, 0}}, k0, kn, p.Kp, log2k,
                   t.mod};
        if (run_pack(q, st)) return -2;
        GemmArgs g{};
        g.M = mm;
        g.N = nn;
        g.mt = (mm + BM - 1) / BM;
        g.bs = p.bs;
        g.nt = (nn + p.bs - 1) / p.bs;
        
        g.splits = p.splits;
        g.nkb = (int)(p.Kp / 64);
        g.kb_per_split = p.kb_per_split;
        g.ld = up(nn, 16);
        g.out = res;
        g.status = status;
        g.wait_ns = wait_limit_ns();
        g.t = t.mod;
        const long long W = std::min<long long>(g.mt * g.nt, num_sms());
        long long gm = (long long)std::llround(std::sqrt((double)W * p.bs / BM));
        gm = std::max(1LL, std::min(gm, g.mt));
        if (g.nt * gm <= W) gm = 1;
        g.gm = (int)gm;
        CUtensorMap tma, tmb;
        if (!make_map(&tma, pa, mm * NM, 2 * p.Kp, 2 * p.Kp, 2, BM) ||
            !make_map(&tmb, pb, nn * NM, 2 * p.Kp, 2 * p.Kp, 2, p.bs))
          return -1;
        const int rc = p.BN == 256   ? run_gemm<256>(tma, tmb, g, st)
                       : p.BN == 128 ? run_gemm<128>(tma, tmb, g, st)
                                     : run_gemm<64>(tma, tmb, g, st);
        if (rc) return rc;
        JoinArgs j{a, b, m0, n0, mm, nn, k0, kn, p.splits, log2k, g.ld, res, alpha,
                   k0 > 0 ? 1.0 : beta, C, status, t.crt};
        j.t.scale *= alpha;
        rns_join_kernel<<<blocks_for(mm * ((nn + 3) / 4), 256), 256, 0, st>>>(j);
        PCG_CHECK_LAUNCH("pcg_contract_rns_f64/join");
      }
    }
  }
  return 0;
}
