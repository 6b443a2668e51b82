// FP64 strided tensor contraction on the FP64 pipe.
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

// Stores one partial (or the whole) sum of products of an output element: with K split across
// blocks (blockIdx.y) the partials are atomic FP64 adds onto C, which the host scaled by
// beta first.
__device__ __forceinline__ void store_sum(const F64Args& p, double* dst, double acc) {
  const double v = p.alpha * acc;
  if (p.atomic_out)
    atomicAdd(dst, v);
  else
    *dst = (p.beta == 0.0) ? v : p.beta * *dst + v;
}

// Clusters of `cy` blocks along K: the first block's first warp adds up what the others' first
// warps left in their shared memory (`mine` there, one value per lane and entry).  All threads of
// all blocks come here.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ double cluster_load(const double* p, int rank) {
  unsigned a = (unsigned)__cvta_generic_to_shared(p);
  double v;
  asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
template <int N>
__device__ __forceinline__ void cluster_sums(double (&x)[N], double* mine, int stride, int cy,
                                             bool first_warp) {
  if (first_warp)
#pragma unroll
    for (int i = 0; i < N; ++i) mine[i * stride] = x[i];
  cluster_barrier();
  if (first_warp && blockIdx.y % cy == 0)
    for (int c = 1; c < cy; ++c)
#pragma unroll
      for (int i = 0; i < N; ++i) x[i] += cluster_load(mine + i * stride, c);
  cluster_barrier();  // no block leaves before its sums are read
}

// A warp computes 32 x R outputs over a slice of K: a lane per index of the long side (m), R
// entries of the other side (n), FP64 multiply-adds with all operands straight from global
// memory.  An SM quarter takes 64 clocks for a warp's FP64 multiply-add, so a step's R + 1 loads
// (the R ones are broadcasts) cost little next to it; what bounds a product is how evenly the
// multiply-adds spread over the 608 quarters and how many of them are padding.  Neither side is
// padded to 8 x 8 fragments as mma.m8n8k4 needs, which has the same FP64 rate.  kw warps of a
// block share a tile and split K, clusters of cy blocks split it further, and clusters beyond that
// (FP64 atomics, each a rounding of the output: without the clusters they were most of the
// rounding error of the singles' residual).
// Device time against 16 x 16 mma tiles, us: no = 9, nv = 53 'ijae,be->ijab' 45 -> 29, 'ie,abej->
// ijab' 62 -> 29, no = 11, nv = 83 'nb,mnej->mbej' 40 -> 26, 'ie,abej->ijab' 215 -> 143, no = 20,
// nv = 180 'mi,mjab->ijab' 959 -> 512 (1.0 TFLOP/s); no = 5, nv = 19 6 -> 4.6-6.
template <int R, typename I>
__global__ void __launch_bounds__(256) contract_f64_kernel(const F64Args p, int kw, int cy,
                                                           long long tiles_n, long long tiles) {
  constexpr int U = 4;  // K steps whose loads are in flight
  __shared__ double red[8][R][32];
  __shared__ longlong2 koff[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ks = warp % kw;
  const long long tile = (long long)blockIdx.x * ((int)(blockDim.x >> 5) / kw) + warp / kw;
  const bool live = tile < tiles;
  const long long tm = live ? tile / tiles_n : 0, n0 = (live ? tile % tiles_n : 0) * R;
  const long long row = tm * 32 + lane;
  const long long bbeg = (long long)blockIdx.y * p.k_per_split;
  const long long bend = live ? min(p.K, bbeg + p.k_per_split) : 0;
  const long long slice = (p.k_per_split + kw - 1) / kw;
  const long long kbeg = min(bend, bbeg + ks * slice), kend = min(bend, kbeg + slice);

  // entries past the end repeat the last one; only the store leaves them out
  long long ao, cm, cn[R];
  sub_offsets_as<I>(p.m, (I)min(row, p.M - 1), ao, cm);
  const double *A = p.A + ao, *B[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    long long bo;
    sub_offsets_as<I>(p.n, (I)min(n0 + r, p.N - 1), bo, cn[r]);
    B[r] = p.B + bo;
  }
  double acc[R], odd[R];  // even and odd steps apart: shorter chains, smaller rounding errors
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r] = odd[r] = 0.0;

  for (long long k0 = kbeg; k0 < kend; k0 += 32) {
    long long ka = 0, kb = 0;
    if (k0 + lane < kend) sub_offsets_as<I>(p.k, (I)(k0 + lane), ka, kb);
    __syncwarp();
    koff[warp][lane] = make_longlong2(ka, kb);
    __syncwarp();
    const int kn = (int)min(32LL, kend - k0);
    for (int u0 = 0; u0 < kn; u0 += U) {
      double a[U], b[U][R];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const longlong2 o = koff[warp][min(u0 + u, kn - 1)];
        a[u] = __ldg(A + o.x);
#pragma unroll
        for (int r = 0; r < R; ++r) b[u][r] = __ldg(B[r] + o.y);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u0 + u < kn)
#pragma unroll
          for (int r = 0; r < R; ++r) {
            double& x = u & 1 ? odd[r] : acc[r];
            x = fma(a[u], b[u][r], x);
          }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r] += odd[r];

  if (kw > 1) {  // the K slices of a tile add up in its first warp
    if (ks > 0)
#pragma unroll
      for (int r = 0; r < R; ++r) red[warp][r][lane] = acc[r];
    __syncthreads();
    if (ks == 0)
      for (int w = warp + 1; w < warp + kw; ++w)
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] += red[w][r][lane];
    if (cy > 1) cluster_sums(acc, &red[0][0][lane], 32, cy, warp == 0);
    if (ks > 0 || blockIdx.y % cy > 0) return;
  }
  if (!live || row >= p.M) return;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (n0 + r >= p.N) break;
    store_sum(p, p.C + cm + cn[r], acc[r]);
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

// The same product with the lanes along K: a warp computes T x T outputs over a slice of K, so
// that a few outputs of a long K are not padded to 32 rows, and adds its lanes' sums up by halves
// (16 FP64 additions for up to 16 outputs; five for each would cost more than the products of a
// short slice).  us, against 16 x 16 mma tiles: no = 9, nv = 53 'ijef,mnef->mnij' 94 -> 43,
// 'ijab,mjab->im' 35 -> 17; no = 11, nv = 83 'mief,maef->ia' 333 -> 168, 'mnef,mnaf->ae' 263 ->
// 133; no = 14, nv = 60 'ijef,mnef->mnij' 412 -> 241 (1.15 TFLOP/s).
template <int T, typename I>
__global__ void __launch_bounds__(256) contract_dot_kernel(const F64Args p, int kw, int cy,
                                                           long long tiles_n, long long tiles) {
  constexpr int U = 2, NV = 16;
  __shared__ double red[8][NV];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, per = 8 / kw, ks = warp % kw;
  const long long kbeg = (long long)blockIdx.y * p.k_per_split;
  const long long kend = min(p.K, kbeg + p.k_per_split);
  const long long t = (long long)blockIdx.x * per + warp / kw, tc = min(t, tiles - 1);
  const long long tm = (long long)((I)tc / (I)tiles_n), m0 = tm * T, n0 = (tc - tm * tiles_n) * T;
  const double *A[T], *B[T];
#pragma unroll
  for (int r = 0; r < T; ++r) {  // entries past the end repeat the last one
    long long o, unused;
    sub_offsets_as<I>(p.m, (I)min(m0 + r, p.M - 1), o, unused);
    A[r] = p.A + o;
    sub_offsets_as<I>(p.n, (I)min(n0 + r, p.N - 1), o, unused);
    B[r] = p.B + o;
  }
  double v[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) v[j] = 0.0;
  for (long long k = kbeg + 32 * U * ks + lane; k < kend; k += 32 * U * kw) {
    double a[U][T], b[U][T];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool ok = k + 32 * u < kend;
      long long ka = 0, kb = 0;
      if (ok) sub_offsets_as<I>(p.k, (I)(k + 32 * u), ka, kb);
#pragma unroll
      for (int r = 0; r < T; ++r) {
        a[u][r] = ok ? __ldg(A[r] + ka) : 0.0;
        b[u][r] = ok ? __ldg(B[r] + kb) : 0.0;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) v[i * T + j] = fma(a[u][i], b[u][j], v[i * T + j]);
  }
  int out = 0;  // this lane's output of the tile
#pragma unroll
  for (int h = NV / 2, s = 16; h > 0; h >>= 1, s >>= 1) {
    const bool up = lane & s;
    out += up ? h : 0;
#pragma unroll
    for (int j = 0; j < h; ++j) {
      const double give = up ? v[j] : v[j + h], keep = up ? v[j + h] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, give, s);
    }
  }
  double x[1] = {v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1)};
  if (kw > 1) {
    if (ks > 0) red[warp][out] = x[0];
    __syncthreads();
    if (ks == 0)
      for (int w = warp + 1; w < warp + kw; ++w) x[0] += red[w][out];
    if (cy > 1) cluster_sums(x, &red[0][out], 0, cy, warp == 0);
    if (ks > 0 || blockIdx.y % cy > 0) return;
  }
  const long long m = m0 + out / T, n = n0 + out % T;
  if (!(lane & 1) && t < tiles && out < T * T && m < p.M && n < p.N) {
    long long unused, cm, cn;
    sub_offsets_as<I>(p.m, (I)m, unused, cm);
    sub_offsets_as<I>(p.n, (I)n, unused, cn);
    store_sum(p, p.C + cm + cn, x[0]);
  }
}

// Outputs with a degenerate or short free dimension (matrix-vector shapes such as 'nf,mnef->me', and
// full dot products): kw warps of a block share an output and a K slice (blockIdx.y), a lane holds
// four products in flight and (I) 32-bit index arithmetic where the totals allow it.  With one
// warp per output the index divisions of K / 32 products were a serial chain.  us: 'ijab,jb->ia'
// no = 11, nv = 83 15 -> 10; 'ijab,ijab->' no = 5, nv = 19 6.2 -> 5.0, no = 40, nv = 300 1730 ->
// 380-430 (5.3-6 TB/s).
template <typename I>
__global__ void __launch_bounds__(256) contract_gemv_kernel(const F64Args p, int kw) {
  __shared__ double red[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, per = 8 / kw, ks = warp % kw;
  const long long total = p.M * p.N;
  const long long kbeg = (long long)blockIdx.y * p.k_per_split;
  const long long kend = min(p.K, kbeg + p.k_per_split);
  for (long long o0 = (long long)blockIdx.x * per; o0 < total; o0 += (long long)gridDim.x * per) {
    const long long o = o0 + warp / kw, oc = min(o, total - 1);
    const long long m = (long long)((I)oc / (I)p.N), n = oc - m * p.N;
    long long am, cm, bn, cn;
    sub_offsets_as<I>(p.m, (I)m, am, cm);
    sub_offsets_as<I>(p.n, (I)n, bn, cn);
    const double *A = p.A + am, *B = p.B + bn;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (long long k = kbeg + ks * 128 + lane; k < kend; k += 128 * kw) {
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
    if (kw > 1) {
      if (lane == 0) red[warp] = sum;
      __syncthreads();
      if (ks == 0)
        for (int w = warp + 1; w < warp + kw; ++w) sum += red[w];
      __syncthreads();  // the next output's sums go to the same place
    }
    if (lane == 0 && ks == 0 && o < total) store_sum(p, p.C + cm + cn, sum);
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
  if (valid) store_sum(p, p.C + cm + cn, acc);
}

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
  if (beta == 0.0 && dense_output(M * N, m.n, m.ext, m.s1, n.n, n.ext, n.s1)) {
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

// How a product is cut: R entries of the n side per warp (lanes along m), or T x T outputs
// (lanes along K); kw warps per tile, blocks of nw warps, K over `splits` blocks in clusters of cy.
struct F64Plan {
  int R, T, kw, nw, cy;
  bool swap;  // the operands exchanged
  long long splits, tiles_n, tiles, blocks;
  double clocks;
};

// Fills in the rest of a cut and keeps it if it is estimated to be the fastest yet, in clocks of
// the SM with the most blocks: on each quarter's FP64 pipe `step` clocks per K step and `fixed`
// per warp; and, only partly hidden by the other warps, the chain of a warp with `wait` more per
// step.  The sums of a cluster cost 2000 and 800 per warp, K split over s of them a pass
// over C and s atomic additions to each output (5000 + 200 s).
void consider(F64Plan& best, F64Plan q, long long steps, double step, double wait, double fixed) {
  const long long sms = num_sms();
  q.nw = q.T ? 8 : std::max(4, q.kw);
  q.blocks = (q.tiles * q.kw + q.nw - 1) / q.nw;
  const long long top = q.kw < 8 ? 1 : std::max(1LL, std::min(steps / (q.T ? 16 : 64), 65528LL));
  const long long fill = (4 * sms + q.blocks - 1) / q.blocks;
  const long long tries[4] = {1, std::min(top, 8LL), std::min(top, fill / 2), std::min(top, fill)};
  for (int i = 0; i < (top > 1 ? 4 : 1); ++i) {
    if (i > 0 && tries[i] < 2) continue;
    q.cy = tries[i] >= 8 ? 8 : 1;
    q.splits = tries[i] / q.cy * q.cy;
    const double ks = (double)((steps + q.splits * q.kw - 1) / (q.splits * q.kw));
    const double warps = (double)((q.blocks * q.splits + sms - 1) / sms) * q.nw / 4;
    const double each = fixed + (q.cy > 1 ? 800 : 0);
    const double sums = 64.0 * (q.T ? 1 : q.R) * (q.kw - 1);  // of a tile's K slices
    q.clocks = warps * (step * ks + each + sums / q.kw) +
               0.4 * (1000 + ks * (step + wait) + each + sums) + (q.cy > 1 ? 2000 : 0) +
               (q.splits > q.cy ? 5000 + 200.0 * q.splits / q.cy : 0);
    if (best.clocks == 0 || q.clocks < best.clocks) best = q;
  }
}

// Lanes along the first side, with every R and kw.
void consider_rows(F64Plan& best, long long M, long long N, long long K, bool wide, bool swap) {
  const int r0 = wide ? 4 : 2, r1 = wide ? 4 : 6;
  F64Plan q{};
  q.swap = swap;
  for (q.R = r0; q.R <= r1; ++q.R) {
    q.tiles_n = (N + q.R - 1) / q.R;
    q.tiles = (M + 31) / 32 * q.tiles_n;
    for (q.kw = 1; q.kw <= 8 && (q.kw == 1 || K >= 4 * q.kw); q.kw *= 2)
      consider(best, q, K, 64.0 * q.R, 150, 250);
  }
}

// Lanes along K.  Where K is not unit-stride a load touches 32 rows of the L1, which all four
// quarters share.
void consider_dots(F64Plan& best, const F64Args& p) {
  const int la = p.k.s0[p.k.n - 1] == 1 ? 2 : 32, lb = p.k.s1[p.k.n - 1] == 1 ? 2 : 32;
  F64Plan q{};
  const long long steps = (p.K + 31) / 32;
  for (q.T = 3; q.T <= 4; ++q.T) {
    q.tiles_n = (p.N + q.T - 1) / q.T;
    q.tiles = (p.M + q.T - 1) / q.T * q.tiles_n;
    for (q.kw = 1; q.kw <= 8 && q.kw <= steps; q.kw *= 2)
      consider(best, q, steps, std::max(64 * q.T * q.T, 4 * q.T * (la + lb)), 400, 1300);
  }
}

// The cut of a product with M >= N > 1.  It depends on the sizes and on K's strides being one or
// not; each thread keeps its last ones (a search takes a few us, as long as a small product).
F64Plan f64_plan(const F64Args& p, bool wide) {
  struct Known {
    long long M, N, K;
    int unit;
    F64Plan q;
  };
  static thread_local Known known[64];
  const int unit = (p.k.s0[p.k.n - 1] == 1) + 2 * (p.k.s1[p.k.n - 1] == 1);
  Known& e = known[(unsigned long long)(p.M * 31 + p.N * 17 + p.K * 7 + unit) % 64];
  if (e.M != p.M || e.N != p.N || e.K != p.K || e.unit != unit) {
    F64Plan q{};
    consider_rows(q, p.M, p.N, p.K, wide, false);
    if (!wide && p.M < 512) {
      if (p.M < 256) consider_rows(q, p.N, p.M, p.K, wide, true);  // may pad less
      if (p.K >= 128) consider_dots(q, p);
    }
    e = {p.M, p.N, p.K, unit, q};
  }
  return e.q;
}

// Blocks of contract_gemv_kernel, and the warps kw that share an output: more while its 128-wide
// steps of K suffice and fewer than `want` warps run.
long long gemv_blocks(long long outputs, long long K, long long want, int& kw) {
  const long long steps = (K + 127) / 128;
  for (kw = 1; kw < 8 && 2 * kw <= steps && outputs * kw < want;) kw *= 2;
  return std::min((outputs * kw + 7) / 8, 64LL * num_sms());
}

// the two operands exchanged
F64Args swapped(F64Args p) {
  std::swap(p.m, p.n);
  std::swap(p.M, p.N);
  std::swap(p.A, p.B);
  for (int i = 0; i < p.k.n; ++i) std::swap(p.k.s0[i], p.k.s1[i]);
  return p;
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
  const bool wide = p.M > 0x7fffffffLL || p.N > 0x7fffffffLL || p.K > 0x7fffffffLL - 256;
  if (p.M == 1) p = swapped(p);
  if (p.N == 1) {
    // one free side.  At least 1024 outputs along the operand's unit-stride index: a thread each,
    // K in slices of 64 or more until there are about eight blocks per SM (with slices of 1024,
    // 'mf,mafe->ae' at no = 9, nv = 53 ran 11 blocks for 79 us; 11 us now).  Otherwise warps,
    // about six for each SM quarter: over K's 128-wide steps in a block, then over blocks.
    p = swapped(p);
    sort_by_operand_stride(p.n);
    const bool threads = p.n.s0[p.n.n - 1] == 1 && p.N >= 1024;
    long long blocks, splits = 1;
    int kw = 1;
    if (threads) {
      blocks = (p.N + 255) / 256;
      const long long want = 8LL * num_sms();
      if (blocks < want && p.K >= 128) splits = std::min((want + blocks - 1) / blocks, p.K / 64);
    } else {
      const long long steps = (p.K + 127) / 128, want = 20LL * num_sms();
      blocks = gemv_blocks(p.N, p.K, want, kw);
      if (kw == 8) splits = std::min(want / 8 / blocks, steps / 8);
    }
    splits = std::max(1LL, std::min(splits, 65535LL));
    p.k_per_split = (p.K + splits - 1) / splits;
    p.atomic_out = splits > 1;
    if (p.atomic_out)
      if (const int rc = scale_output(p, p.m, p.n, p.M, p.N, beta, st)) return rc;
    const dim3 grid((unsigned)blocks, (unsigned)splits);
    if (threads)
      contract_gemv_thread_kernel<<<grid, 256, 0, st>>>(p);
    else if (wide)
      contract_gemv_kernel<unsigned long long><<<grid, 256, 0, st>>>(p, kw);
    else
      contract_gemv_kernel<unsigned><<<grid, 256, 0, st>>>(p, kw);
    PCG_CHECK_LAUNCH("pcg_contract_f64/gemv");
    return 0;
  }
  if (p.M < p.N) p = swapped(p);
  // A side below eight, and few outputs or rows of K contiguous in both operands: an output per
  // warp, or per up to eight, without staged offsets or tiles.  A long K is cut over up to eight
  // blocks where the outputs alone leave SMs idle.  us in a graph, here / by the kernels below: 5 x
  // 2 x 52 3.4 / 6.5, 322 x 7 x 111 3.8 / 7.8, 1024 x 7 x 1000 21 / 25, 40 x 2 x 4000 6 / 12; but
  // 4096 x 2 x 111 10.0 / 8.0 and, with K not contiguous, 1024 x 7 x 4000 128 / 75.
  const bool k_rows = p.k.s0[p.k.n - 1] == 1 && p.k.s1[p.k.n - 1] == 1;
  const long long outputs = p.M * p.N;
  if (p.N < 8 && !wide &&
      ((outputs <= 4096 && p.K <= 8192) ||
       (k_rows && p.K >= 256 && (p.K <= 8192 || outputs >= 48)))) {
    const long long want = (p.K >= 2048 ? 20LL : 8LL) * num_sms();
    int kw = 1;
    const long long blocks = gemv_blocks(outputs, p.K, want, kw);
    const long long splits =
        p.K > 8192 ? std::max(1LL, std::min({want / 8 / blocks, p.K / 4096, 8LL})) : 1;
    p.k_per_split = (p.K + splits - 1) / splits;
    p.atomic_out = splits > 1;
    if (p.atomic_out)
      if (const int rc = scale_output(p, p.m, p.n, p.M, p.N, beta, st)) return rc;
    contract_gemv_kernel<unsigned><<<dim3((unsigned)blocks, (unsigned)splits), 256, 0, st>>>(p, kw);
    PCG_CHECK_LAUNCH("pcg_contract_f64/gemv");
    return 0;
  }
  const F64Plan q = f64_plan(p, wide);
  if (q.swap) p = swapped(p);
  if (q.blocks > 0x7fffffffLL) {
    set_error("pcg_contract_f64: M=%lld x N=%lld too large", p.M, p.N);
    return -1;
  }
  p.k_per_split = (p.K + q.splits - 1) / q.splits;
  p.atomic_out = q.splits > q.cy;
  if (p.atomic_out)
    if (const int rc = scale_output(p, p.m, p.n, p.M, p.N, beta, st)) return rc;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = attr.val.clusterDim.z = 1;
  attr.val.clusterDim.y = (unsigned)q.cy;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)q.blocks, (unsigned)q.splits);
  cfg.blockDim = dim3(32 * q.nw);
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = q.cy > 1 ? 1 : 0;
  auto go = [&](auto kernel) {
    cudaLaunchKernelEx(&cfg, kernel, (const F64Args)p, q.kw, q.cy, q.tiles_n, q.tiles);
  };
  if (q.T == 3)
    go(contract_dot_kernel<3, unsigned>);
  else if (q.T == 4)
    go(contract_dot_kernel<4, unsigned>);
  else if (wide)
    go(contract_f64_kernel<4, unsigned long long>);
  else if (q.R == 2)
    go(contract_f64_kernel<2, unsigned>);
  else if (q.R == 3)
    go(contract_f64_kernel<3, unsigned>);
  else if (q.R == 4)
    go(contract_f64_kernel<4, unsigned>);
  else if (q.R == 5)
    go(contract_f64_kernel<5, unsigned>);
  else
    go(contract_f64_kernel<6, unsigned>);
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
