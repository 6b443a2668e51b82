// FP64 strided tensor contraction on the FP64 tensor pipe (DMMA, mma.sync m8n8k4 f64).
//
//   C[m, n] = beta * C[m, n] + alpha * sum_k A[m, k] * B[n, k]
//
// m, n and k are flat indices over up to four sub-indices each; every sub-index carries
// its own element stride in both tensors that hold it, so index permutations of the
// operands and of the output (the einsum strings of the CCSD residual, e.g.
// 'imae,mbej->ijab') are folded into address generation and never materialised.
// This is the oracle-grade GPU path of the engine: exact FP64 products, FP64 sums.
#include "common.cuh"
#include <algorithm>

namespace pcg {
namespace {

constexpr int BM = 64, BN = 64, BK = 16, NT = 128;

struct F64Args {
  SubIdx m, n, k;  // m: (A, C) strides; n: (B, C) strides; k: (A, B) strides
  long long M, N, K;
  long long k_per_split;
  double alpha, beta;
  const double* A;
  const double* B;
  double* C;
  int atomic_out;
};

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// Offsets of flat index r in both tensors; I is the type of the index arithmetic (32-bit
// division where the totals allow it, a third of the 64-bit sequence).
template <typename I>
__device__ __forceinline__ void sub_offsets_as(const SubIdx& d, I r, long long& o0,
                                               long long& o1) {
  o0 = 0;
  o1 = 0;
  for (int q = d.n - 1; q >= 0; --q) {
    const I e = (I)d.ext[q];
    const long long x = (long long)(r % e);
    r /= e;
    o0 += x * d.s0[q];
    o1 += x * d.s1[q];
  }
}

// A warp computes 8 FM x 8 FN outputs over a slice of K, its DMMA fragments read straight from
// global memory (L1 holds the rows; the 8 x 4 fragment of a lane pattern is whole sectors
// whichever index is unit-stride).  A quarter of an SM's FP64 pipe takes about 512 clocks for one
// m8n8k4, so loads cost little next to it; what bounds a small product is how evenly the
// multiply-adds spread over the 608 quarters.  Blocks of 64 x 64 tiles left most of them idle.
// Here kw of the block's 8 warps share an output tile and split K, blocks split K further (FP64
// atomics), and a tile is 16 x 16, 8 x 32 or 32 x 8 where one side has at most 8 entries, or
// 8 x 8 where there would be fewer 16-K steps than would keep every quarter busy.
// Device time against 64 x 64 tiles in shared memory, us: no = 5, nv = 19 ring 138 -> 11, small
// products 45-60 -> 6-8; no = 9, nv = 53 'nb,mnej->mbej' 41 -> 15, 'mief,maef->ia' 490 -> 59; the
// large ladder of no = 20, nv = 180 882 -> 770 ms (1.09 TFLOP/s).
template <int FM, int FN, typename I>
__global__ void __launch_bounds__(256) contract_f64_kernel(const F64Args p, int kw,
                                                           long long tiles_n, long long tiles) {
  constexpr int NF = 2 * FM * FN;
  __shared__ double red[8][NF][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int ks = warp % kw;
  const long long tile = (long long)blockIdx.x * (8 / kw) + warp / kw;
  const bool live = tile < tiles;
  const long long m0 = (live ? tile / tiles_n : 0) * (8 * FM);
  const long long n0 = (live ? tile % tiles_n : 0) * (8 * FN);
  const long long kbeg = (long long)blockIdx.y * p.k_per_split;
  const long long kend = live ? min(p.K, kbeg + p.k_per_split) : 0;

  long long ao[FM], bo[FN], cm[FM];
  bool aok[FM], bok[FN];
#pragma unroll
  for (int i = 0; i < FM; ++i) {
    const long long r = m0 + 8 * i + g;
    aok[i] = r < p.M;
    ao[i] = cm[i] = 0;
    if (aok[i]) sub_offsets_as<I>(p.m, (I)r, ao[i], cm[i]);
  }
#pragma unroll
  for (int j = 0; j < FN; ++j) {
    const long long r = n0 + 8 * j + g;
    long long unused;
    bok[j] = r < p.N;
    bo[j] = 0;
    if (bok[j]) sub_offsets_as<I>(p.n, (I)r, bo[j], unused);
  }
  double acc[FM][FN][2];
#pragma unroll
  for (int i = 0; i < FM; ++i)
#pragma unroll
    for (int j = 0; j < FN; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  for (long long k0 = kbeg + 16 * ks; k0 < kend; k0 += 16 * kw) {
    double a[4][FM], b[4][FN];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const long long k = k0 + 4 * s + t4;
      const bool ok = k < kend;
      long long ka = 0, kb = 0;
      if (ok) sub_offsets_as<I>(p.k, (I)k, ka, kb);
#pragma unroll
      for (int i = 0; i < FM; ++i) a[s][i] = (ok && aok[i]) ? __ldg(p.A + ao[i] + ka) : 0.0;
#pragma unroll
      for (int j = 0; j < FN; ++j) b[s][j] = (ok && bok[j]) ? __ldg(p.B + bo[j] + kb) : 0.0;
    }
    if (k0 + 12 < kend) {
#pragma unroll
      for (int s = 0; s < 4; ++s)
#pragma unroll
        for (int i = 0; i < FM; ++i)
#pragma unroll
          for (int j = 0; j < FN; ++j) dmma(acc[i][j], a[s][i], b[s][j]);
    } else {  // the last step multiplies the K it has
#pragma unroll
      for (int s = 0; s < 3; ++s)
        if (k0 + 4 * s < kend)
#pragma unroll
          for (int i = 0; i < FM; ++i)
#pragma unroll
            for (int j = 0; j < FN; ++j) dmma(acc[i][j], a[s][i], b[s][j]);
    }
  }

  if (kw > 1) {  // the K slices of a tile add up in its first warp
    if (ks > 0)
#pragma unroll
      for (int f = 0; f < NF; ++f) red[warp][f][lane] = acc[f / (2 * FN)][(f / 2) % FN][f % 2];
    __syncthreads();
    if (ks > 0) return;
    for (int w = warp + 1; w < warp + kw; ++w)
#pragma unroll
      for (int f = 0; f < NF; ++f) acc[f / (2 * FN)][(f / 2) % FN][f % 2] += red[w][f][lane];
  }
  if (!live) return;
#pragma unroll
  for (int j = 0; j < FN; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long c = n0 + 8 * j + 2 * t4 + h;
      if (c >= p.N) continue;
      long long unused, cn;
      sub_offsets_as<I>(p.n, (I)c, unused, cn);
#pragma unroll
      for (int i = 0; i < FM; ++i) {
        if (!aok[i]) continue;
        double* dst = p.C + cm[i] + cn;
        const double v = p.alpha * acc[i][j][h];
        if (p.atomic_out)
          atomicAdd(dst, v);
        else
          *dst = p.beta == 0.0 ? v : p.beta * *dst + v;
      }
    }
}

// C[m, n] *= beta over the strided M x N range (used before a split-K accumulation).
__global__ void scale_strided_kernel(SubIdx m, SubIdx n, long long M, long long N, double beta,
                                     double* C) {
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = M * N;
  for (; idx < total; idx += (long long)gridDim.x * blockDim.x) {
    long long r = idx / N, c = idx % N, a0, a1, b0, b1;
    sub_offsets(m, r, a0, a1);
    sub_offsets(n, c, b0, b1);
    double* dst = C + a1 + b1;
    *dst = (beta == 0.0) ? 0.0 : beta * *dst;
  }
}

// Stores one partial (or the whole) dot product of an output element: with K split across
// blocks (blockIdx.y) the partials are atomic FP64 adds onto C, which the host scaled by
// beta first.
__device__ __forceinline__ void gemv_store(const F64Args& p, double* dst, double acc) {
  const double v = p.alpha * acc;
  if (p.atomic_out)
    atomicAdd(dst, v);
  else
    *dst = (p.beta == 0.0) ? v : p.beta * *dst + v;
}

// Outputs with a degenerate free dimension (matrix-vector shapes such as 'nf,mnef->me', and
// full dot products): one warp per output element and K slice (blockIdx.y), a warp-wide FP64
// dot over the slice, four products a lane in flight and (I) 32-bit index arithmetic where the
// totals allow it.  'ijab,jb->ia' at no = 11, nv = 83: 17 us against 24 with one product in
// flight and 64-bit divisions.
template <typename I>
__global__ void __launch_bounds__(256) contract_gemv_kernel(const F64Args p) {
  const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long total = p.M * p.N;
  const long long kbeg = (long long)blockIdx.y * p.k_per_split;
  const long long kend = min(p.K, kbeg + p.k_per_split);
  for (long long o = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; o < total;
       o += warps) {
    const long long m = (long long)((I)o / (I)p.N), n = o - m * p.N;
    long long am, cm, bn, cn;
    sub_offsets_as<I>(p.m, (I)m, am, cm);
    sub_offsets_as<I>(p.n, (I)n, bn, cn);
    const double *A = p.A + am, *B = p.B + bn;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (long long k = kbeg + lane; k < kend; k += 128) {
      double a[4], b[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        a[u] = b[u] = 0.0;
        if (k + 32 * u < kend) {
          long long ka, kb;
          if (p.k.n == 1) {
            ka = (k + 32 * u) * p.k.s0[0];
            kb = (k + 32 * u) * p.k.s1[0];
          } else {
            sub_offsets_as<I>(p.k, (I)(k + 32 * u), ka, kb);
          }
          a[u] = __ldg(A + ka);
          b[u] = __ldg(B + kb);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[u] = fma(a[u], b[u], acc[u]);
    }
    double sum = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
    if (lane == 0) gemv_store(p, p.C + cm + cn, sum);
  }
}

// Matrix-vector shapes whose operand B is unit-stride along the output's innermost
// sub-index: one thread per output, consecutive threads on consecutive outputs (coalesced
// B reads); the K offsets are staged in shared memory once per block; blockIdx.y is the K
// slice.
__global__ void __launch_bounds__(256) contract_gemv_thread_kernel(const F64Args p) {
  __shared__ long long ka[256], kb[256];
  const long long o = (long long)blockIdx.x * 256 + threadIdx.x;
  const bool valid = o < p.M * p.N;
  const long long kbeg = (long long)blockIdx.y * p.k_per_split;
  const long long kend = min(p.K, kbeg + p.k_per_split);
  long long am = 0, cm = 0, bn = 0, cn = 0;
  if (valid) {
    sub_offsets(p.m, o / p.N, am, cm);
    sub_offsets(p.n, o % p.N, bn, cn);
  }
  double acc = 0.0;
  for (long long k0 = kbeg; k0 < kend; k0 += 256) {
    __syncthreads();
    const long long k = k0 + threadIdx.x;
    if (k < kend) sub_offsets(p.k, k, ka[threadIdx.x], kb[threadIdx.x]);
    __syncthreads();
    const int kn = (int)min((long long)256, kend - k0);
    if (valid)
      for (int j = 0; j < kn; ++j) acc += p.A[am + ka[j]] * p.B[bn + kb[j]];
  }
  if (valid) gemv_store(p, p.C + cm + cn, acc);
}

// K slices for a matrix-vector launch of `blocks` output blocks: enough blocks for about
// eight per SM, each slice at least `kmin` long; beta is applied up front when split.  kmin is
// 64 for a thread per output (with 1024, 'mf,mafe->ae' at no = 9, nv = 53 ran 11 blocks for
// 79 us; 11 us now) and 512 for a warp.
long long gemv_splits(const F64Args& p, long long blocks, long long kmin);

// Reorder sub-indices by decreasing |stride| in the operand (s0), unit stride innermost.
void sort_by_operand_stride(SubIdx& d) {
  for (int i = 0; i < d.n; ++i)
    for (int j = i + 1; j < d.n; ++j)
      if (llabs(d.s0[j]) > llabs(d.s0[i])) {
        std::swap(d.ext[i], d.ext[j]);
        std::swap(d.s0[i], d.s0[j]);
        std::swap(d.s1[i], d.s1[j]);
      }
}

// C[m, n] *= beta ahead of a split K.  A zero fill of a C without gaps is a memset.
int scale_output(const F64Args& p, const SubIdx& m, const SubIdx& n, long long M, long long N,
                 double beta, cudaStream_t st) {
  if (beta == 1.0) return 0;
  if (beta == 0.0 && dense_output(m.n, m.ext, m.s1, n.n, n.ext, n.s1)) {
    if (cudaMemsetAsync(p.C, 0, (size_t)(8 * M * N), st) == cudaSuccess) return 0;
    set_error("pcg_contract_f64: clearing the output failed");
    return -2;
  }
  scale_strided_kernel<<<(int)std::min<long long>((M * N + 255) / 256, 4096), 256, 0, st>>>(
      m, n, M, N, beta, p.C);
  PCG_CHECK_LAUNCH("pcg_contract_f64/scale");
  return 0;
}

bool fill_sub(SubIdx& d, int n, const long long* ext, const long long* s0, const long long* s1,
              const char* what) {
  if (n < 0 || n > kMaxSub) {
    set_error("pcg_contract_f64: %s has %d sub-indices (max %d)", what, n, kMaxSub);
    return false;
  }
  if (n > 0 && (!ext || !s0 || !s1)) {
    set_error("pcg_contract_f64: %s extents or strides missing", what);
    return false;
  }
  d.n = n;
  for (int q = 0; q < n; ++q) {
    if (ext[q] <= 0) {
      set_error("pcg_contract_f64: %s extent %lld must be positive", what, ext[q]);
      return false;
    }
    d.ext[q] = ext[q];
    d.s0[q] = s0[q];
    d.s1[q] = s1[q];
  }
  if (n == 0) {  // an empty group is a single index of extent 1
    d.n = 1;
    d.ext[0] = 1;
    d.s0[0] = 0;
    d.s1[0] = 0;
  }
  return true;
}

long long gemv_splits(const F64Args& p, long long blocks, long long kmin) {
  const long long want = 8LL * 152;
  if (blocks >= want || p.K < 2 * kmin) return 1;
  long long splits = std::min((want + blocks - 1) / blocks, p.K / kmin);
  return std::max(1LL, std::min(splits, 65535LL));
}

int num_sms() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  return sms;
}

}  // namespace
}  // namespace pcg

extern "C" int pcg_contract_f64(int m_n, const long long* m_ext, const long long* m_sa,
                                const long long* m_sc, int n_n, const long long* n_ext,
                                const long long* n_sb, const long long* n_sc, int k_n,
                                const long long* k_ext, const long long* k_sa,
                                const long long* k_sb, double alpha, const double* A,
                                const double* B, double beta, double* C, void* stream) {
  using namespace pcg;
  F64Args p{};
  if (!fill_sub(p.m, m_n, m_ext, m_sa, m_sc, "M") || !fill_sub(p.n, n_n, n_ext, n_sb, n_sc, "N") ||
      !fill_sub(p.k, k_n, k_ext, k_sa, k_sb, "K"))
    return -1;
  if (!A || !B || !C) {
    set_error("pcg_contract_f64: null operand pointer");
    return -1;
  }
  p.M = sub_total(p.m);
  p.N = sub_total(p.n);
  p.K = sub_total(p.k);
  p.alpha = alpha;
  p.beta = beta;
  p.A = A;
  p.B = B;
  p.C = C;
  cudaStream_t st = (cudaStream_t)stream;
  if (p.M == 1 || p.N == 1) {
    // one free side: enumerate the outputs along the big operand's unit-stride index
    F64Args q = p;
    if (q.M == 1) {
      sort_by_operand_stride(q.n);
    } else {  // N == 1: swap roles so the free index is on the B side
      std::swap(q.m, q.n);
      std::swap(q.M, q.N);
      std::swap(q.A, q.B);
      for (int i = 0; i < q.k.n; ++i) std::swap(q.k.s0[i], q.k.s1[i]);
      sort_by_operand_stride(q.n);
    }
    if (q.n.s0[q.n.n - 1] == 1 && q.M * q.N >= 1024) {
      const long long blocks = (q.M * q.N + 255) / 256;
      const long long splits = gemv_splits(q, blocks, 64);
      q.k_per_split = (q.K + splits - 1) / splits;
      q.atomic_out = splits > 1;
      if (q.atomic_out)
        if (const int rc = scale_output(q, q.m, q.n, q.M, q.N, beta, st)) return rc;
      contract_gemv_thread_kernel<<<dim3((unsigned)blocks, (unsigned)splits), 256, 0, st>>>(q);
      PCG_CHECK_LAUNCH("pcg_contract_f64/gemv_thread");
      return 0;
    }
  }
  if (p.M == 1 || p.N == 1) {
    long long warps = p.M * p.N;
    int blocks = (int)std::min<long long>((warps * 32 + 255) / 256, 152LL * 64);
    const long long splits = gemv_splits(p, blocks, 512);
    p.k_per_split = (p.K + splits - 1) / splits;
    p.atomic_out = splits > 1;
    if (p.atomic_out)
      if (const int rc = scale_output(p, p.m, p.n, p.M, p.N, beta, st)) return rc;
    const dim3 grid((unsigned)blocks, (unsigned)splits);
    if (p.M * p.N > 0x7fffffffLL || p.K > 0x7fffffffLL - 128)
      contract_gemv_kernel<unsigned long long><<<grid, 256, 0, st>>>(p);
    else
      contract_gemv_kernel<unsigned><<<grid, 256, 0, st>>>(p);
    PCG_CHECK_LAUNCH("pcg_contract_f64/gemv");
    return 0;
  }
  // tiles of 16 x 16 outputs per warp, 8 x 32 or 32 x 8 where a side has at most 8, 8 x 8 where
  // 16 x 16 tiles would leave fewer than two K steps for each quarter of an SM
  const long long steps = (p.K + 15) / 16;
  int fm = p.M <= 8 ? 1 : (p.N <= 8 ? 4 : 2), fn = 4 / fm;
  if ((p.M + 15) / 16 * ((p.N + 15) / 16) * steps < 8LL * num_sms()) fm = fn = 1;
  const long long nt = (p.N + 8 * fn - 1) / (8 * fn), mt = (p.M + 8 * fm - 1) / (8 * fm);
  const long long tiles = mt * nt;
  // warps per tile: K's 16-wide steps over up to 8 warps while that fills the chip (16 warps on
  // each SM), then over blocks, each at least two steps a warp
  const long long want = 16LL * num_sms();
  int kw = 1;
  while (kw < 8 && 2 * kw <= steps && tiles * kw < want) kw *= 2;
  long long splits = 1;
  if (kw == 8 && tiles * 8 < want)
    splits = std::max(1LL, std::min((want + tiles * 8 - 1) / (tiles * 8), steps / 16));
  long long kps = ((p.K + splits - 1) / splits + 15) / 16 * 16;
  splits = (p.K + kps - 1) / kps;
  p.k_per_split = kps;
  p.atomic_out = splits > 1;
  const long long blocks = (tiles + 8 / kw - 1) / (8 / kw);
  if (blocks > 0x7fffffffLL) {
    set_error("pcg_contract_f64: M=%lld x N=%lld too large", p.M, p.N);
    return -1;
  }
  if (p.atomic_out)
    if (const int rc = scale_output(p, p.m, p.n, p.M, p.N, beta, st)) return rc;
  const dim3 grid((unsigned)blocks, (unsigned)splits);
  const bool wide = p.M > 0x7fffffffLL || p.N > 0x7fffffffLL || p.K > 0x7fffffffLL;
  auto go = [&](auto kernel) { kernel<<<grid, 256, 0, st>>>(p, kw, nt, tiles); };
  if (fm == 1 && fn == 1)
    wide ? go(contract_f64_kernel<1, 1, unsigned long long>) : go(contract_f64_kernel<1, 1, unsigned>);
  else if (fm == 1)
    wide ? go(contract_f64_kernel<1, 4, unsigned long long>) : go(contract_f64_kernel<1, 4, unsigned>);
  else if (fm == 2)
    wide ? go(contract_f64_kernel<2, 2, unsigned long long>) : go(contract_f64_kernel<2, 2, unsigned>);
  else
    wide ? go(contract_f64_kernel<4, 1, unsigned long long>) : go(contract_f64_kernel<4, 1, unsigned>);
  PCG_CHECK_LAUNCH("pcg_contract_f64");
  return 0;
}

// ---------------------------------------------------------------------------------------
// Sum of up to four FP64 contractions into one output tile:
//   C[m, n] = beta * C[m, n] + sum_t alpha_t * sum_k A_t[m, k] * B_t[n, k]
// All terms share the M / N extents and the C strides; each term has its own operands, A / B
// strides and K range.  Used where several einsum terms land on the same output (the four
// terms of one orientation of the connected triples), so the output is written once.
// ---------------------------------------------------------------------------------------
namespace pcg {
namespace {
constexpr int kMaxTerms = 4;

struct MultiArgs {
  int nterm;
  SubIdx m, n;                 // ext + C strides (s1); s0 unused
  long long ma[kMaxTerms][kMaxSub];  // per-term A strides of the M sub-indices
  long long nb[kMaxTerms][kMaxSub];  // per-term B strides of the N sub-indices
  SubIdx k[kMaxTerms];         // per-term K (A strides s0, B strides s1)
  long long K[kMaxTerms];
  double alpha[kMaxTerms];
  const double* A[kMaxTerms];
  const double* B[kMaxTerms];
  long long M, N;
  double beta;
  double* C;
};

__device__ __forceinline__ long long strided_offset(const SubIdx& d, const long long* s,
                                                    long long r) {
  long long o = 0;
  for (int q = d.n - 1; q >= 0; --q) {
    const long long e = d.ext[q];
    o += (r % e) * s[q];
    r /= e;
  }
  return o;
}

__global__ void __launch_bounds__(NT) contract_multi_f64_kernel(const MultiArgs p) {
  __shared__ double As[BK][BM + 2];
  __shared__ double Bs[BK][BN + 2];
  __shared__ long long aoff[BM], coffm[BM], boff[BN], coffn[BN];
  __shared__ long long akoff[BK], bkoff[BK];
  const int tid = threadIdx.x;
  const long long m0 = (long long)blockIdx.y * BM;
  const long long n0 = (long long)blockIdx.x * BN;
  const int warp = tid >> 5, lane = tid & 31;
  const int wm = warp >> 1, wn = warp & 1;
  const int g = lane >> 2, t4 = lane & 3;
  double acc[4][4][2];
  if (tid < BM) {
    const long long r = m0 + tid;
    coffm[tid] = (r < p.M) ? strided_offset(p.m, p.m.s1, r) : 0;
  } else {
    const int t = tid - BM;
    const long long r = n0 + t;
    coffn[t] = (r < p.N) ? strided_offset(p.n, p.n.s1, r) : 0;
  }
  double out[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) out[i][j][0] = out[i][j][1] = 0.0;

  for (int term = 0; term < p.nterm; ++term) {
    __syncthreads();
    if (tid < BM) {
      const long long r = m0 + tid;
      aoff[tid] = (r < p.M) ? strided_offset(p.m, p.ma[term], r) : 0;
    } else {
      const int t = tid - BM;
      const long long r = n0 + t;
      boff[t] = (r < p.N) ? strided_offset(p.n, p.nb[term], r) : 0;
    }
    const SubIdx& kd = p.k[term];
    const long long K = p.K[term];
    const double* Ap = p.A[term];
    const double* Bp = p.B[term];
    const int a_kfast = (kd.s0[kd.n - 1] == 1);
    const int b_kfast = (kd.s1[kd.n - 1] == 1);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    for (long long kt = 0; kt < K; kt += BK) {
      __syncthreads();
      if (tid < BK) {
        long long o0 = 0, o1 = 0;
        if (kt + tid < K) sub_offsets(kd, kt + tid, o0, o1);
        akoff[tid] = o0;
        bkoff[tid] = o1;
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int e = tid + NT * i;
        int mm, kk;
        if (a_kfast) { kk = e % BK; mm = e / BK; } else { mm = e % BM; kk = e / BM; }
        As[kk][mm] = (m0 + mm < p.M && kt + kk < K) ? __ldg(Ap + aoff[mm] + akoff[kk]) : 0.0;
        int nn;
        if (b_kfast) { kk = e % BK; nn = e / BK; } else { nn = e % BN; kk = e / BN; }
        Bs[kk][nn] = (n0 + nn < p.N && kt + kk < K) ? __ldg(Bp + boff[nn] + bkoff[kk]) : 0.0;
      }
      __syncthreads();
#pragma unroll
      for (int ks = 0; ks < BK; ks += 4) {
        double a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = As[ks + t4][wm * 32 + i * 8 + g];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = Bs[ks + t4][wn * 32 + j * 8 + g];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) dmma(acc[i][j], a[i], b[j]);
      }
    }
    const double al = p.alpha[term];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        out[i][j][0] += al * acc[i][j][0];
        out[i][j][1] += al * acc[i][j][1];
      }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = wm * 32 + i * 8 + g;
    if (m0 + row >= p.M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int col = wn * 32 + j * 8 + 2 * t4 + h;
        if (n0 + col >= p.N) continue;
        double* dst = p.C + coffm[row] + coffn[col];
        *dst = (p.beta == 0.0) ? out[i][j][h] : p.beta * *dst + out[i][j][h];
      }
  }
}
}  // namespace
}  // namespace pcg

// C = beta*C + sum_t alpha[t] * A_t . B_t^T over nterm (<= 4) terms.  The M / N sub-index
// extents (m_ext, n_ext) and C strides (m_sc, n_sc) are common; per term t: A strides of the
// M sub-indices m_sa[t*4 + q], B strides of the N sub-indices n_sb[t*4 + q], and its K
// group k_n[t], k_ext[t*4 + q], k_sa[t*4 + q], k_sb[t*4 + q].
extern "C" int pcg_contract_multi_f64(int nterm, int m_n, const long long* m_ext,
                                      const long long* m_sc, const long long* m_sa, int n_n,
                                      const long long* n_ext, const long long* n_sc,
                                      const long long* n_sb, const int* k_n,
                                      const long long* k_ext, const long long* k_sa,
                                      const long long* k_sb, const double* alpha,
                                      const double* const* A, const double* const* B,
                                      double beta, double* C, void* stream) {
  using namespace pcg;
  if (nterm < 1 || nterm > kMaxTerms || m_n < 0 || m_n > kMaxSub || n_n < 0 || n_n > kMaxSub ||
      !C || !k_n || !alpha || !A || !B || (m_n > 0 && !m_sa) || (n_n > 0 && !n_sb) ||
      !k_ext || !k_sa || !k_sb) {
    set_error("pcg_contract_multi_f64: bad term / sub-index counts or missing arrays");
    return -1;
  }
  MultiArgs p{};
  p.nterm = nterm;
  const long long zero[kMaxSub] = {0, 0, 0, 0};
  if (!fill_sub(p.m, m_n, m_ext, zero, m_sc, "M") || !fill_sub(p.n, n_n, n_ext, zero, n_sc, "N"))
    return -1;
  for (int t = 0; t < nterm; ++t) {
    for (int q = 0; q < kMaxSub; ++q) {
      p.ma[t][q] = (q < m_n) ? m_sa[t * kMaxSub + q] : 0;
      p.nb[t][q] = (q < n_n) ? n_sb[t * kMaxSub + q] : 0;
    }
    if (!fill_sub(p.k[t], k_n[t], k_ext + t * kMaxSub, k_sa + t * kMaxSub, k_sb + t * kMaxSub,
                  "K"))
      return -1;
    p.K[t] = sub_total(p.k[t]);
    p.alpha[t] = alpha[t];
    p.A[t] = A[t];
    p.B[t] = B[t];
    if (!A[t] || !B[t]) {
      set_error("pcg_contract_multi_f64: null operand of term %d", t);
      return -1;
    }
  }
  p.M = sub_total(p.m);
  p.N = sub_total(p.n);
  p.beta = beta;
  p.C = C;
  const long long mt = (p.M + BM - 1) / BM, nt = (p.N + BN - 1) / BN;
  if (mt > 65535) {
    set_error("pcg_contract_multi_f64: M=%lld too large", p.M);
    return -1;
  }
  dim3 grid((unsigned)nt, (unsigned)mt);
  contract_multi_f64_kernel<<<grid, NT, 0, (cudaStream_t)stream>>>(p);
  PCG_CHECK_LAUNCH("pcg_contract_multi_f64");
  return 0;
}
