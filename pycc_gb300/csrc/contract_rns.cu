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
//    A seventeenth GEMM, of the integers' magnitudes in BF16, gives sum |a'||b'|, 2 % low at most.
// 4. The integer sum is at most |a'_i| |b'_j| (Cauchy-Schwarz), below half the product of the
//    moduli (2^123.95), so the residues determine it exactly.  It is rebuilt as a 96-bit
//    fraction of that product, rounded to FP64, scaled back and added into C.
//
// Where large entries of a row meet small or zero ones of a column, the rounding of step 1 can be
// as large as the sum.  Step 4 sees this from the sum of magnitudes (kDoubt in rns.cuh) and takes
// such outputs from FP64 dot products, so every output's error is bounded in terms of sum |a||b|,
// as that of FP64 multiply-adds.  So are the outputs of a row (or a column of B) with an infinity
// or a NaN, and non-finite inputs give what FP64 arithmetic gives.
//
// Measured on GB300 against the FP64 pipe at its peak rate, no = 20, nv = 180: the ladder
// 'ijef,abef->ijab' 727 -> 21.9 ms (GEMM 12.8, packs 7.7), a ring 'imae,mbej->ijab' 81 -> 1.40 ms;
// at no = 9, nv = 53 2.2 -> 0.16 ms for the ladder.
//
// The offsets of strided rows, columns and K indices are expanded into tables once per call;
// operands larger than the workspace go through in panels of rows, columns or K.
#include "rns.cuh"

namespace pcg {
namespace rns {

// ---- residues -> C --------------------------------------------------------------------
struct JoinArgs {
  Operand a, b;
  long long m0, n0, M, N;  // this panel's rows and columns
  long long k0, K;
  int splits;
  int beta_zero, beta_one;
  long long ld;
  const unsigned char* res;  // [split][plane][M][ld]
  unsigned items;            // groups of four columns per block and step: 8, 16, .. 256
  double alpha, beta;
  double* C;
  const int* status;
  CrtTab t;
};

// This lane's part of the FP64 dot product of one output: K indices k0, k0 + step, ..., four in
// flight.  A warp leaves when its sum is a NaN, which nothing changes any more.
__device__ __forceinline__ double lane_dot(const JoinArgs& p, long long row, long long col,
                                           int part, int step) {
  const int lane = threadIdx.x & 31;
  const double* x = p.a.X + p.a.off[row];
  const double* y = p.b.X + p.b.off[col];
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (long long k = 32 * part; k < p.K; k += 4 * step) {
    double u[4], v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const long long kk = k + lane + q * step;
      u[q] = kk < p.K ? __ldg(x + k_offset(p.a, p.k0 + kk)) : 0.0;
      v[q] = kk < p.K ? __ldg(y + k_offset(p.b, p.k0 + kk)) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) s[q] = fma(u[q], v[q], s[q]);
    if (__any_sync(0xffffffffu, isnan(s[0]))) break;
  }
  double r = (s[0] + s[1]) + (s[2] + s[3]);
  for (int d = 16; d > 0; d >>= 1) r += __shfl_xor_sync(0xffffffffu, r, d);
  return r;
}

__device__ __forceinline__ void put(const JoinArgs& p, double* dst, double v) {
  if (!p.beta_zero) v = p.beta_one ? *dst + v : fma(p.beta, *dst, v);
  *dst = v;
}

struct Redo {
  int count;
  unsigned short todo[4 * 256];
  double part[4][256];
};

// All outputs of the block's items: a thread has an item's four columns and every slices-th K, two
// in flight.
__device__ __forceinline__ void dense_sums(const JoinArgs& p, Redo& s, unsigned i0, unsigned nc) {
  const int slices = 256 / (int)p.items;
  const unsigned i = min(i0 + threadIdx.x % p.items, (unsigned)(p.M * nc) - 1), row = i / nc;
  const double* x = p.a.X + p.a.off[p.m0 + row];
  const double* y[4];
#pragma unroll
  for (int e = 0; e < 4; ++e)
    y[e] = p.b.X + p.b.off[p.n0 + min(4ll * (i - row * nc) + e, p.N - 1)];
  double sum[2][4] = {};
  for (long long k = threadIdx.x / p.items; k < p.K; k += 2 * slices) {
    double u[2], v[2][4];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const bool in = k + q * slices < p.K;
      const long long kk = p.k0 + (in ? k + q * slices : k);
      const long long ka = k_offset(p.a, kk), kb = k_offset(p.b, kk);
      u[q] = in ? __ldg(x + ka) : 0.0;
#pragma unroll
      for (int e = 0; e < 4; ++e) v[q][e] = in ? __ldg(y[e] + kb) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) sum[q][e] = fma(u[q], v[q][e], sum[q][e]);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) s.part[e][threadIdx.x] = sum[0][e] + sum[1][e];
}

// The four columns of one item by a warp with the lanes along K; returns column `lane >> 3`'s sum.
__device__ __forceinline__ double item_sum(const JoinArgs& p, unsigned row, unsigned col) {
  const int lane = threadIdx.x & 31;
  const double* x = p.a.X + p.a.off[p.m0 + row];
  const double* y[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) y[e] = p.b.X + p.b.off[p.n0 + min((long long)col + e, p.N - 1)];
  double s[4] = {};
  for (long long k = lane; k < p.K; k += 64) {
    double u[2], v[2][4];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const bool in = k + 32 * q < p.K;
      const long long kk = p.k0 + (in ? k + 32 * q : k);
      const long long ka = k_offset(p.a, kk), kb = k_offset(p.b, kk);
      u[q] = in ? __ldg(x + ka) : 0.0;
#pragma unroll
      for (int e = 0; e < 4; ++e) v[q][e] = in ? __ldg(y[e] + kb) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[e] = fma(u[q], v[q][e], s[e]);
  }
  // by halves: six FP64 additions, where five for each column would be twenty
#pragma unroll
  for (int h = 2, d = 16; h > 0; h >>= 1, d >>= 1)
#pragma unroll
    for (int j = 0; j < h; ++j) {
      const double give = lane & d ? s[j] : s[j + h], keep = lane & d ? s[j + h] : s[j];
      s[j] = keep + __shfl_xor_sync(0xffffffffu, give, d);
    }
  for (int d = 4; d > 0; d >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], d);
  return s[0];
}

// The outputs of this block's items i0, i0 + 1, ... that their threads marked (bit e of `doubt`:
// column e).  A few: a warp each with the lanes along K, or, along a long K, all eight warps.
// That takes up to four times an FP64 kernel's time for an output, so from a third of the block's
// outputs on an item's four columns are computed together, by a thread or, where B is contiguous
// along K, by a warp.  The whole call, with no output, one output of each row and every output
// marked: 1600 x 1600 x 1600 0.20, 0.30 and 7.4 ms (FP64 kernel 6.7), 477 x 477 x 477 42, 46 and
// 274 us (201), 53 x 53 x 4293 53, 57 and 89 us (36).
__device__ __noinline__ void redo_marked(const JoinArgs& p, Redo& s, unsigned i0, unsigned nc,
                                         unsigned doubt) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) s.count = 0;
  __syncthreads();
  for (int e = 0; e < 4; ++e)
    if (doubt >> e & 1) s.todo[atomicAdd(&s.count, 1)] = (unsigned short)(4 * threadIdx.x + e);
  __syncthreads();
  if (3 * s.count > 4 * (int)p.items && p.b.kfast) {
    __syncthreads();
    s.todo[threadIdx.x] = (unsigned short)doubt;
    __syncthreads();
    for (unsigned it = warp; it < p.items; it += 8) {
      const unsigned marked = s.todo[it], i = i0 + it, row = i / nc, col = 4 * (i - row * nc);
      if (!marked) continue;
      const double v = item_sum(p, row, col);
      if ((lane & 7) == 0 && (marked >> (lane >> 3) & 1))
        put(p, p.C + p.a.coff[p.m0 + row] + p.b.coff[p.n0 + col + (lane >> 3)], p.alpha * v);
    }
    __syncthreads();
    return;
  }
  if (3 * s.count > 4 * (int)p.items) {
    dense_sums(p, s, i0, nc);
    __syncthreads();
    if (doubt) {
      const unsigned i = i0 + threadIdx.x, row = i / nc;
      const long long c = p.n0 + 4 * (i - row * nc);
      for (int e = 0; e < 4; ++e)
        if (doubt >> e & 1) {
          double v = 0.0;
          for (int t = threadIdx.x; t < 256; t += p.items) v += s.part[e][t];
          put(p, p.C + p.a.coff[p.m0 + row] + p.b.coff[c + e], p.alpha * v);
        }
    }
    __syncthreads();
    return;
  }
  const int parts = p.K >= 4096 ? 8 : 1, at = 8 / parts;
  for (int q0 = 0; q0 < s.count; q0 += at) {
    const int q = q0 + warp / parts, part = warp % parts;
    double v = 0.0;
    double* dst = nullptr;
    if (q < s.count) {  // the same for all of a warp
      const unsigned i = i0 + s.todo[q] / 4, row = i / nc;
      const long long r = p.m0 + row, c = p.n0 + 4 * (i - row * nc) + s.todo[q] % 4;
      v = lane_dot(p, r, c, part, 32 * parts);
      dst = p.C + p.a.coff[r] + p.b.coff[c];
    }
    if (parts > 1) {
      if (lane == 0) s.part[0][warp] = v;
      __syncthreads();
      if (warp == 0)
        for (int w = 1; w < parts; ++w) v += s.part[0][w];
      __syncthreads();
    }
    if (dst && part == 0 && lane == 0) put(p, dst, p.alpha * v);
  }
  __syncthreads();  // the list is filled anew
}

// Four columns of one row per thread: for every modulus the residues times the three words of
// floor(2^96 q / p) are summed in 64-bit accumulators (their integer part falls out modulo 2^96),
// the signed fraction is rounded to FP64 and scaled.  About 200 integer instructions and two FP64
// ones per output; four resident blocks hide the loads' latency.  At 13.0e6 outputs 134 us,
// against 175 at 66 registers with each column's scale computed where it is read; on another day
// 121, and 131 with the sums of magnitudes, a seventeenth byte per output, and their check.
__global__ void __launch_bounds__(256, 4) rns_join_kernel(const __grid_constant__ JoinArgs p) {
  __shared__ Redo redo;
  const unsigned nc = (unsigned)((p.N + 3) >> 2);
  const unsigned total = (unsigned)(p.M * nc);  // below 2^31 (host check)
  const bool failed = *p.status != 0;
  for (unsigned i0 = blockIdx.x * p.items; i0 < total; i0 += gridDim.x * p.items) {
    const unsigned i = i0 + threadIdx.x;
    unsigned doubt = 0;
    if (threadIdx.x < p.items && i < total) {
      const unsigned row = i / nc, col = 4 * (i - row * nc);
      CrtSum sum(p.t);
      float mag[4] = {0.f, 0.f, 0.f, 0.f};
      for (int sp = 0; sp < p.splits; ++sp) {
        const unsigned char* src = p.res + ((long long)sp * NP * p.M + row) * p.ld + col;
        unsigned w[NP];
#pragma unroll
        for (int l = 0; l < NP; ++l)
          w[l] = __ldg(reinterpret_cast<const unsigned*>(src + (long long)l * p.M * p.ld));
        sum.add(p.t, w);
#pragma unroll
        for (int e = 0; e < 4; ++e) mag[e] += magnitude_sum(w[NM], e);
      }
      const long long grow = p.m0 + row, gcol = p.n0 + col;  // gcol: a multiple of four
      const int sa = p.a.sh[grow];
      const int4 sb = *reinterpret_cast<const int4*>(p.b.sh + gcol);
      const longlong2 o0 = *reinterpret_cast<const longlong2*>(p.b.coff + gcol);
      const longlong2 o1 = *reinterpret_cast<const longlong2*>(p.b.coff + gcol + 2);
      double* crow = p.C + p.a.coff[grow];
      const int sbe[4] = {sb.x, sb.y, sb.z, sb.w};
      const long long off[4] = {o0.x, o0.y, o1.x, o1.y};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (col + e >= p.N) break;
        double v = sum.value(p.t, e, -sa - sbe[e]);
        const bool again = (mag[e] > 0.f && mag[e] < kDoubt) || sa == kNotFinite ||
                           sbe[e] == kNotFinite;
        if (failed) v = __longlong_as_double(0x7ff8000000000000ll);
        if (again && !failed)
          doubt |= 1u << e;
        else
          put(p, crow + off[e], v);
      }
    }
    if (__syncthreads_or((int)doubt)) redo_marked(p, redo, i0, nc, doubt);
  }
}

// ---- host side --------------------------------------------------------------------------
// How one call is cut: panels of M, N and K, and the workspace's layout.
struct Plan {
  long long PM, PN, PK, Kp;  // panel sizes (Kp: PK rounded up to the 64-K block)
  long long np_m, np_n, np_k;
  int splits, kb_per_split, bs, BN;
  long long nt, ld;
  long long tables, panel_a, panel_b, res, total;  // bytes
};

bool size_plan(Plan& p, long long M, long long N, long long K) {
  p.PM = p.np_m == 1 ? M : up((M + p.np_m - 1) / p.np_m, BM);
  p.PN = p.np_n == 1 ? N : up((N + p.np_n - 1) / p.np_n, 64);
  p.PK = p.np_k == 1 ? K : up((K + p.np_k - 1) / p.np_k, 64);
  p.Kp = up(p.PK, 64);
  p.BN = p.PN > 128 ? 256 : (p.PN > 64 ? 128 : 64);
  p.nt = (p.PN + p.BN - 1) / p.BN;
  p.bs = (int)(16 * (((p.PN + 15) / 16 + p.nt - 1) / p.nt));
  p.ld = up(p.PN, 16);
  const long long nkb = p.Kp / 64, units = (p.PM + BM - 1) / BM * p.nt * NP;
  const int sms = num_sms();
  // fewer units than SMs: cut K (each part at least a chunk), the residues add up in the join
  int splits = 1;
  if (units < sms) splits = (int)std::max(1LL, std::min<long long>(sms / units, nkb / kChunk));
  splits = std::min(splits, 8);
  p.kb_per_split = (int)((nkb + splits - 1) / splits);
  p.splits = (int)((nkb + p.kb_per_split - 1) / p.kb_per_split);
  p.tables = up((M + N) * (8 + 8 + 4 + 4 + 4 + 4) + 16 * K + 256 + 14 * 16, 256);
  p.panel_a = up(p.PM * p.Kp * 2 * NP, 256);
  p.panel_b = up(p.PN * p.Kp * 2 * NP, 256);
  p.res = up((long long)p.splits * NP * p.PM * p.ld, 256);
  p.total = p.tables + p.panel_a + p.panel_b + p.res;
  return p.PM * NP < 0x7fffffffLL - BM && p.PN * NP < 0x7fffffffLL - 256 &&
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
  auto take = [&](long long bytes) {  // every array 16-byte aligned
    unsigned char* r = tb;
    tb += up(bytes, 16);
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
  a.norm = (unsigned long long*)take(8 * M);
  b.norm = (unsigned long long*)take(8 * N);
  a.walk = (int*)take(4 * M);
  b.walk = (int*)take(4 * N);
  a.sh = (int*)take(4 * M);
  b.sh = (int*)take(4 * N);
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
    if (k0 > 0) {
      cudaMemsetAsync(a.norm, 0, 8 * M, st);
      cudaMemsetAsync(b.norm, 0, 8 * N, st);
    }
    if (run_norm(a, b, k0, k0 + kn, {{pa, pb}, {p.panel_a, p.panel_b}}, st)) return -2;
    for (long long n0 = 0; n0 < N; n0 += p.PN) {
      const long long nn = std::min(p.PN, N - n0);
      for (long long m0 = 0; m0 < M; m0 += p.PM) {
        const long long mm = std::min(p.PM, M - m0);
        // B's panel is packed with the first panel of A
        PackArgs q{{{a, m0, mm, pa, mm * p.Kp / 8, 0, 0},
                    {b, n0, m0 == 0 ? nn : 0, pb, nn * p.Kp / 8, 0, 0}},
                   k0, kn, p.Kp, p.Kp, t.pairs};
        if (run_pack(q, st)) return -2;
        GemmArgs g{};
        g.M = mm;
        g.N = nn;
        g.mt = (mm + BM - 1) / BM;
        g.bs = p.bs;
        g.nt = (nn + p.bs - 1) / p.bs;
        g.planes = p.splits;
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
        GemmMaps maps{};
        if (!make_map(&maps.a[0], pa, mm * NP, 2 * p.Kp, 2 * p.Kp, 2, BM) ||
            !make_map(&maps.b[0], pb, nn * NP, 2 * p.Kp, 2 * p.Kp, 2, p.bs))
          return -1;
        const int rc = p.BN == 256   ? run_gemm<256, false>(maps, g, st)
                       : p.BN == 128 ? run_gemm<128, false>(maps, g, st)
                                     : run_gemm<64, false>(maps, g, st);
        if (rc) return rc;
        const double bt = k0 > 0 ? 1.0 : beta;
        // few outputs go to many blocks, whose warps share those that are computed again
        const long long quads = mm * ((nn + 3) / 4);
        unsigned items = 8;
        while (items < 256 && items * 4LL * num_sms() < quads) items *= 2;
        JoinArgs j{a, b, m0, n0, mm, nn, k0, kn, p.splits, bt == 0.0, bt == 1.0, g.ld, res, items,
                   alpha, bt, C, status, crt_tab(p.splits, alpha)};
        rns_join_kernel<<<blocks_for(quads, (int)items), 256, 0, st>>>(j);
        PCG_CHECK_LAUNCH("pcg_contract_rns_f64/join");
      }
    }
  }
  return 0;
}
