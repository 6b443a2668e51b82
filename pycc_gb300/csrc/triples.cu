// (T) energy from the connected triples of a batch of (i, j, k) triples, i >= j >= k.
//
// The connected triples W[a,b,c] of one triple arrive as three partial tensors, one per
// orientation of the twelve t3 terms (the terms of an orientation share their output
// layout, so each partial is written once by a single contraction).  Each is the output of
// a GEMM with rows (two virtual indices) and one column index, stored column-major:
//   orientation 1: rows (a,b), column c  ->  P1[c][a][b]
//   orientation 2: rows (a,c), column b  ->  P2[b][a][c]
//   orientation 3: rows (b,c), column a  ->  P3[a][b][c]
//   W[a,b,c] = P1[c][a][b] + P2[b][a][c] + P3[a][b][c]
// The Lee-Rendell energy of the reference (pycc/cctriples.py:177-240) is then evaluated
// for a >= b >= c with the same weights; one block per (triple, a), one FP64 partial per
// block (deterministic reduction by pcg_reduce_sum_f64).
#include "tc_common.cuh"
#include <algorithm>

namespace pcg {
namespace {

constexpr int TE_THREADS = 256;

template <typename T>
struct TripArgs {
  const T* P1;
  const T* P2;
  const T* P3;
  long long pstride;  // elements between consecutive triples' partials
  const int* ijk;     // [ntrip][3]
  int ntrip;
  const double* eps;  // [nmo]
  const T* eoovv;     // <ij|ab> [o][o][v][v], in the partials' type
  const double* t1;   // [o][v]
  const T* t2;        // [o][o][v][v], in the partials' type
  const double* fov;  // [o][v] or null (canonical)
  long long no, nv;
  double* part;       // [ntrip][nv]
};

template <typename T>
__device__ __forceinline__ T wval(const TripArgs<T>& p, const T* P1, const T* P2, const T* P3,
                                  long long x, long long y, long long z) {
  const long long v = p.nv;
  return P1[(z * v + x) * v + y] + P2[(y * v + x) * v + z] + P3[(x * v + y) * v + z];
}

// disconnected triples (pycc/cctriples.py:133-140) at (x, y, z), in the arithmetic type T
// (FP32 for the tensor-core path: the FP64 pipe of GB300 is ~60x slower than FP32)
template <typename T>
__device__ __forceinline__ T dval(const TripArgs<T>& p, int i, int j, int k, long long x,
                                  long long y, long long z) {
  const long long o = p.no, v = p.nv;
  auto E = [&](int a, int b, long long c, long long d) {
    return (T)p.eoovv[((a * o + b) * v + c) * v + d];
  };
  auto A2 = [&](int a, int b, long long c, long long d) {
    return (T)p.t2[((a * o + b) * v + c) * v + d];
  };
  T d = E(i, j, x, y) * (T)p.t1[k * v + z] + E(i, k, x, z) * (T)p.t1[j * v + y] +
        E(j, k, y, z) * (T)p.t1[i * v + x];
  if (p.fov)
    d += A2(i, j, x, y) * (T)p.fov[k * v + z] + A2(i, k, x, z) * (T)p.fov[j * v + y] +
         A2(j, k, y, z) * (T)p.fov[i * v + x];
  return d;
}

template <typename T>
__global__ void __launch_bounds__(TE_THREADS) triples_energy_kernel(const TripArgs<T> p) {
  const int t = blockIdx.y;
  const long long a = blockIdx.x;
  const int i = p.ijk[3 * t], j = p.ijk[3 * t + 1], k = p.ijk[3 * t + 2];
  const T* P1 = p.P1 + t * p.pstride;
  const T* P2 = p.P2 + t * p.pstride;
  const T* P3 = p.P3 + t * p.pstride;
  const long long o = p.no;
  const double eo = p.eps[i] + p.eps[j] + p.eps[k];
  const double fac = 2.0 - ((i == j) + (i == k) + (j == k));
  const long long npair = (a + 1) * (a + 2) / 2;
  T acc_t = 0;  // per-thread partial (a few hundred terms); the block sum is FP64
  for (long long q = threadIdx.x; q < npair; q += TE_THREADS) {
    // q -> (b, c) with a >= b >= c
    long long b = (long long)((sqrtf(8.0f * (float)q + 1.0f) - 1.0f) * 0.5f);
    while (b * (b + 1) / 2 > q) --b;
    while ((b + 1) * (b + 2) / 2 <= q) ++b;
    const long long c = q - b * (b + 1) / 2;
    const long long idx[6][3] = {{a, b, c}, {a, c, b}, {b, a, c}, {b, c, a}, {c, a, b}, {c, b, a}};
    // 1 + d_ab + d_ac + d_bc is 1, 2 or 4: the division by it is an exact product (six FP64
    // divisions were half of the FP64 kernel's time)
    const int same = (a == b) + (a == c) + (b == c);
    const T rw = same == 0 ? (T)1 : (same == 1 ? (T)0.5 : (T)0.25);
    T W[6], V[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) {
      W[s] = wval(p, P1, P2, P3, idx[s][0], idx[s][1], idx[s][2]);
      V[s] = (W[s] + dval(p, i, j, k, idx[s][0], idx[s][1], idx[s][2])) * rw;
    }
    // perms: 0 abc, 1 acb, 2 bac, 3 bca, 4 cab, 5 cba
    T X = 0;
#pragma unroll
    for (int s = 0; s < 6; ++s) X += W[s] * V[s];
    const T Y = V[0] + V[3] + V[4];
    const T Z = V[1] + V[2] + V[5];
    const T Wc = W[0] + W[3] + W[4];
    const T Wa = W[1] + W[2] + W[5];
    const T S = (Y - (T)2 * Z) * Wc + (Z - (T)2 * Y) * Wa + (T)3 * X;
    const T D = (T)(eo - p.eps[o + a] - p.eps[o + b] - p.eps[o + c]);
    acc_t += S / D;
  }
  double acc = (double)acc_t;
  __shared__ double red[TE_THREADS / 32];
  for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = (threadIdx.x < TE_THREADS / 32) ? red[threadIdx.x] : 0.0;
    for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
    if (threadIdx.x == 0) p.part[(long long)t * p.nv + a] = fac * v;
  }
}

// ---- FP32 path: tiles of the (a, b, c) cube -------------------------------------------
// One block per (triple, tile triple A >= B >= C) of TT^3 tiles.  W at the six orderings of
// the tile sets, W[XYZ][x][y][z] with (X, Y, Z) = (A,B,C), (A,C,B), (B,A,C), (B,C,A),
// (C,A,B), (C,B,A), is staged in shared memory from the column-major partials, each read
// as aligned runs of TT consecutive floats (one 32-byte sector): P3[x][y][z] and P2[y][x][z]
// along z, P1[z][x][y] along y.  <ij|xy>, <ik|xz>, <jk|yz> (and t2 when f_ov is present)
// over the 3 TT indices of A, B and C, the t1 rows and the orbital energies are staged
// too.  The block then evaluates every a >= b >= c of its tiles with the same weights and
// formula as the per-(triple, a) kernel, in FP32, and writes one FP64 partial.
constexpr int TT = 8;
constexpr int TT3 = 3 * TT;
constexpr int TE2_THREADS = 256;

struct TiledStage {
  float w[6][TT][TT][TT + 1];
  float e[3][TT3][TT3 + 1];   // <ij|..>, <ik|..>, <jk|..> over the union of A, B, C
  float d2[3][TT3][TT3 + 1];  // t2_ij.., t2_ik.., t2_jk.. (non-canonical only)
  float t1r[3][TT3];          // t1[i], t1[j], t1[k] over the union
  float fr[3][TT3];           // f_ov[i], f_ov[j], f_ov[k] over the union
  float ev[TT3];              // eps of the virtual orbitals of the union
  double red[TE2_THREADS / 32];
};

// Tile triple u -> (A, B, C), A >= B >= C, in the order u = A(A+1)(A+2)/6 + B(B+1)/2 + C:
// root estimates, then exact integer corrections (u < 2^31).
__device__ __forceinline__ void tile_triple(long long u, int& A, int& B, int& C) {
  auto tet = [](long long a) { return a * (a + 1) * (a + 2) / 6; };
  auto tri = [](long long b) { return b * (b + 1) / 2; };
  long long a = (long long)cbrtf(6.0f * (float)u);
  while (a > 0 && tet(a) > u) --a;
  while (tet(a + 1) <= u) ++a;
  const long long r = u - tet(a);
  long long b = (long long)((sqrtf(8.0f * (float)r + 1.0f) - 1.0f) * 0.5f);
  while (b > 0 && tri(b) > r) --b;
  while (tri(b + 1) <= r) ++b;
  A = (int)a;
  B = (int)b;
  C = (int)(r - tri(b));
}

__device__ __forceinline__ float dval_tiled(const TiledStage& s, bool fov, int lx, int ly,
                                            int lz) {
  float d = s.e[0][lx][ly] * s.t1r[2][lz] + s.e[1][lx][lz] * s.t1r[1][ly] +
            s.e[2][ly][lz] * s.t1r[0][lx];
  if (fov)
    d += s.d2[0][lx][ly] * s.fr[2][lz] + s.d2[1][lx][lz] * s.fr[1][ly] +
         s.d2[2][ly][lz] * s.fr[0][lx];
  return d;
}

// orderings of the tile sets (A, B, C), so = 0..5: (A,B,C), (A,C,B), (B,A,C), (B,C,A),
// (C,A,B), (C,B,A); kord(so, q) is the set in position q, two bits per entry
__host__ __device__ constexpr int kord(int so, int q) {
  return (int)((0x192261624ULL >> (2 * (3 * so + q))) & 3u);
}

// five resident blocks per SM (48 registers): short, latency-bound blocks gain more from the
// extra block than they lose to the few spilled registers of the staging phase
__global__ void __launch_bounds__(TE2_THREADS, 5) triples_energy_tiled_kernel(
    const TripArgs<float> p, long long ntt) {
  __shared__ TiledStage s;
  const int t = blockIdx.y;
  const long long u = blockIdx.x;
  int A, B, C;
  tile_triple(u, A, B, C);
  const long long org[3] = {(long long)A * TT, (long long)B * TT, (long long)C * TT};
  const int i = p.ijk[3 * t], j = p.ijk[3 * t + 1], k = p.ijk[3 * t + 2];
  const float* P1 = p.P1 + t * p.pstride;
  const float* P2 = p.P2 + t * p.pstride;
  const float* P3 = p.P3 + t * p.pstride;
  const long long o = p.no, v = p.nv;
  const int tid = threadIdx.x;
  constexpr int NE = TT * TT * TT / TE2_THREADS;  // tile elements per thread and ordering
  static_assert(TT * TT * TT % TE2_THREADS == 0, "whole tile elements per thread");
  // orbital of staged-union index l (8 q + r is orbital org[q] + r)
  auto uorb = [&](int l) -> long long {
    return (l < TT ? org[0] : (l < 2 * TT ? org[1] : org[2])) + (l % TT);
  };
  // Every global load of the block is issued before the first shared-memory store:
  // P3[x][y][z] + P2[y][x][z] (runs along z), P1[z][x][y] (runs along y), the integral
  // and amplitude slices.  The ordering index is unrolled, so the tile origins are
  // registers; offsets are 32-bit (v^3 < 2^31, checked by the host), and a thread's
  // repeats differ by a constant stride (TE2_THREADS / TT^2 steps of the slowest index).
  const int vv = (int)v, v2 = vv * vv;
  const bool full = (vv % TT) == 0;  // every tile inside the cube: no bounds checks
  constexpr int RS = TE2_THREADS / (TT * TT);
  const int e0 = tid;
  const int s_hi = e0 / (TT * TT), s_mid = (e0 / TT) % TT, s_lo = e0 % TT;
  float p32[6][NE], p1v[6][NE];
#pragma unroll
  for (int so = 0; so < 6; ++so) {
    const int X0 = (int)org[kord(so, 0)], Y0 = (int)org[kord(so, 1)], Z0 = (int)org[kord(so, 2)];
    // pass-1 mapping (x, y, z) = (hi, mid, lo); pass-2 mapping (z, x, y) = (hi, mid, lo)
    const int x1 = X0 + s_hi, y1 = Y0 + s_mid, z1 = Z0 + s_lo;
    const int z2 = Z0 + s_hi, x2 = X0 + s_mid, y2 = Y0 + s_lo;
    const int o3 = (x1 * vv + y1) * vv + z1, o2 = (y1 * vv + x1) * vv + z1;
    const int o1 = (z2 * vv + x2) * vv + y2;
#pragma unroll
    for (int rep = 0; rep < NE; ++rep) {
      const int d = rep * RS;  // steps of the slowest index
      if (full) {
        p32[so][rep] = P3[o3 + d * v2] + P2[o2 + d * vv];
        p1v[so][rep] = P1[o1 + d * v2];
      } else {
        p32[so][rep] = (x1 + d < vv && y1 < vv && z1 < vv)
                           ? P3[o3 + d * v2] + P2[o2 + d * vv] : 0.f;
        p1v[so][rep] = (z2 + d < vv && x2 < vv && y2 < vv) ? P1[o1 + d * v2] : 0.f;
      }
    }
  }
  // <ij|xy>, <ik|xz>, <jk|yz> (and t2) over the union of the tiles, FP32: per pair and
  // row, three runs of TT orbitals, read as float4 when the tiles are whole (v % TT == 0
  // keeps every run 16-byte aligned)
  constexpr int QPR = TT / 4;                      // float4 per run
  constexpr int NSEG = 3 * TT3 * 3 * QPR;          // pairs x rows x runs x float4
  constexpr int NS = (NSEG + TE2_THREADS - 1) / TE2_THREADS;
  float4 ev[NS], tv[NS];
#pragma unroll
  for (int rp = 0; rp < NS; ++rp) {
    const int e = tid + rp * TE2_THREADS;
    ev[rp] = make_float4(0.f, 0.f, 0.f, 0.f);
    tv[rp] = ev[rp];
    if (e < NSEG) {
      const int pr = e / (TT3 * 3 * QPR), r = e % (TT3 * 3 * QPR);
      const int l1 = r / (3 * QPR), c = r % (3 * QPR);
      const long long x = uorb(l1), y = uorb((c / QPR) * TT) + 4 * (c % QPR);
      const int a0 = pr == 2 ? j : i, a1 = pr == 0 ? j : k;  // pairs ij, ik, jk
      const long long at = ((a0 * o + a1) * v + x) * v + y;
      if (full) {
        ev[rp] = *reinterpret_cast<const float4*>(p.eoovv + at);
        if (p.fov) tv[rp] = *reinterpret_cast<const float4*>(p.t2 + at);
      } else if (x < v) {
        float* pe = &ev[rp].x;
        float* pt = &tv[rp].x;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (y + q < v) {
            pe[q] = p.eoovv[at + q];
            if (p.fov) pt[q] = p.t2[at + q];
          }
      }
    }
  }
  if (tid < 3 * TT3) {
    const int q = tid / TT3, l = tid % TT3;
    const long long x = uorb(l);
    const int occ = q == 0 ? i : (q == 1 ? j : k);
    s.t1r[q][l] = x < v ? f64_to_f32(p.t1[occ * v + x]) : 0.f;
    s.fr[q][l] = (x < v && p.fov) ? f64_to_f32(p.fov[occ * v + x]) : 0.f;
    if (q == 0) s.ev[l] = x < v ? f64_to_f32(p.eps[o + x]) : 0.f;
  }
#pragma unroll
  for (int so = 0; so < 6; ++so)
#pragma unroll
    for (int rep = 0; rep < NE; ++rep) {
      const int e = tid + rep * TE2_THREADS;
      s.w[so][e / (TT * TT)][(e / TT) % TT][e % TT] = p32[so][rep];
    }
#pragma unroll
  for (int rp = 0; rp < NS; ++rp) {
    const int e = tid + rp * TE2_THREADS;
    if (e < NSEG) {
      const int pr = e / (TT3 * 3 * QPR), r = e % (TT3 * 3 * QPR);
      const int l1 = r / (3 * QPR), c = r % (3 * QPR);
      const int l2 = (c / QPR) * TT + 4 * (c % QPR);
      const float* pe = &ev[rp].x;
      const float* pt = &tv[rp].x;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        s.e[pr][l1][l2 + q] = pe[q];
        s.d2[pr][l1][l2 + q] = pt[q];
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int so = 0; so < 6; ++so)
#pragma unroll
    for (int rep = 0; rep < NE; ++rep) {
      const int e = tid + rep * TE2_THREADS;
      s.w[so][(e / TT) % TT][e % TT][e / (TT * TT)] += p1v[so][rep];
    }
  __syncthreads();
  const float eo = f64_to_f32(p.eps[i] + p.eps[j] + p.eps[k]);
  const bool fov = p.fov != nullptr;
  float acc = 0.f;
#pragma unroll
  for (int rep = 0; rep < NE; ++rep) {
    const int e = tid + rep * TE2_THREADS;
    const int al = e / (TT * TT), bl = (e / TT) % TT, cl = e % TT;
    const long long a = org[0] + al, b = org[1] + bl, c = org[2] + cl;
    if (a >= v || b > a || c > b) continue;
    const int la = al, lb = TT + bl, lc = 2 * TT + cl;  // indices in the staged union
    float W[6], V[6];
    W[0] = s.w[0][al][bl][cl];
    W[1] = s.w[1][al][cl][bl];
    W[2] = s.w[2][bl][al][cl];
    W[3] = s.w[3][bl][cl][al];
    W[4] = s.w[4][cl][al][bl];
    W[5] = s.w[5][cl][bl][al];
    const float wt = (float)(1 + (a == b) + (a == c) + (b == c));
    const float rw = 1.f / wt;
    V[0] = (W[0] + dval_tiled(s, fov, la, lb, lc)) * rw;
    V[1] = (W[1] + dval_tiled(s, fov, la, lc, lb)) * rw;
    V[2] = (W[2] + dval_tiled(s, fov, lb, la, lc)) * rw;
    V[3] = (W[3] + dval_tiled(s, fov, lb, lc, la)) * rw;
    V[4] = (W[4] + dval_tiled(s, fov, lc, la, lb)) * rw;
    V[5] = (W[5] + dval_tiled(s, fov, lc, lb, la)) * rw;
    float X = 0.f;
#pragma unroll
    for (int q = 0; q < 6; ++q) X += W[q] * V[q];
    const float Y = V[0] + V[3] + V[4], Z = V[1] + V[2] + V[5];
    const float Wc = W[0] + W[3] + W[4], Wa = W[1] + W[2] + W[5];
    const float S = (Y - 2.f * Z) * Wc + (Z - 2.f * Y) * Wa + 3.f * X;
    const float D = eo - s.ev[la] - s.ev[lb] - s.ev[lc];
    acc += S / D;
  }
  // warp sums as an FP32 tree (a few combinations per thread), the block's eight warp
  // sums in FP64
  float wsum = acc;
  for (int sh = 16; sh > 0; sh >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, sh);
  if ((tid & 31) == 0) s.red[tid >> 5] = f32_to_f64(wsum);
  __syncthreads();
  if (tid < 32) {
    double r = (tid < TE2_THREADS / 32) ? s.red[tid] : 0.0;
    for (int sh = 16; sh > 0; sh >>= 1) r += __shfl_xor_sync(0xffffffffu, r, sh);
    const double fac = 2.0 - ((i == j) + (i == k) + (j == k));
    if (tid == 0) p.part[(long long)t * ntt + u] = fac * r;
  }
}

long long tile_triples(long long nv) {
  const long long nt = (nv + TT - 1) / TT;
  return nt * (nt + 1) * (nt + 2) / 6;
}

// ---- FP32 path, partials with a 16-byte pitch: tiles by TMA ------------------------------
// One block per (triple, tile triple A >= B >= C) as above, but the six orderings of the tile sets
// of each partial arrive as 8 x 8 x 8 boxes by TMA (18 boxes of 2 KB, zeros beyond nv) and W is
// summed where it is used.  The 8 x 8 blocks of integrals and amplitudes are the threads' own
// loads: 36 more small copies by TMA, which takes 2.6 clocks for a 32-byte row, made the kernel
// 15 % slower.  The staging of the kernel above cost about 500 instructions a thread and, at a pitch
// that is no multiple of 32 bytes, two sectors for each 32-byte run; what bounds this one is
// shared-memory reads, so a warp takes 2 x 4 x 4 elements (a, b, c), which keeps the boxes'
// 256-byte slices at two to four reads to a bank.  At nv = 121, 32 triples: 260 us against 400.
struct CubeArgs {
  const int* ijk;      // [ntrip][3]
  const double* eps;   // [nmo]
  const float *eoovv, *t2;  // <ij|ab> and t2, [o][o][v][pitch]
  long long pitch;
  const double* t1;    // [o][v]
  const double* fov;   // [o][v] or null (canonical)
  int no, nv;
  unsigned ntt;
  double* part;        // [ntrip][ntt]
  int* status;
  unsigned long long wait_ns;
};

// ordered pairs of the tile sets A, B, C (0, 1, 2): AB, AC, BA, BC, CA, CB
__host__ __device__ constexpr int pair_first(int q) { return q >> 1; }
__host__ __device__ constexpr int pair_second(int q) {
  return (q >> 1) == 0 ? 1 + (q & 1) : ((q & 1) ? 3 - (q >> 1) : 0);
}

template <bool FOV>
struct CubeStage {
  float box[3][6][TT * TT * TT];      // partial, ordering of (slow, middle, fast) as kord
  float e[3][6][TT][TT];              // <ij|..>, <ik|..>, <jk|..> over the ordered pairs
  float d2[FOV ? 3 : 1][FOV ? 6 : 1][TT][TT];
  float t1r[3][TT3], fr[3][TT3];      // t1 and f_ov of i, j, k over the union
  float ev[TT3];
  double red[TE2_THREADS / 32];
  uint64_t bar;
  int ok;
};

template <bool FOV>
__global__ void __launch_bounds__(TE2_THREADS, 4)
    triples_energy_cube_kernel(const __grid_constant__ CUtensorMap map, const CubeArgs p) {
  __shared__ __align__(128) CubeStage<FOV> s;
  const int t = blockIdx.y, tid = threadIdx.x;
  const int v = p.nv;
  const int i = p.ijk[3 * t], j = p.ijk[3 * t + 1], k = p.ijk[3 * t + 2];
  int org[3];
  {  // tile triple blockIdx.x -> A >= B >= C, 32-bit (nv^3 < 2^31)
    const unsigned u = blockIdx.x;
    auto tet = [](unsigned a) { return a * (a + 1) * (a + 2) / 6; };
    auto tri = [](unsigned b) { return b * (b + 1) / 2; };
    unsigned a = (unsigned)cbrtf(6.0f * (float)u);
    while (a > 0 && tet(a) > u) --a;
    while (tet(a + 1) <= u) ++a;
    const unsigned r = u - tet(a);
    unsigned b = (unsigned)((sqrtf(8.0f * (float)r + 1.0f) - 1.0f) * 0.5f);
    while (b > 0 && tri(b) > r) --b;
    while (tri(b + 1) <= r) ++b;
    org[0] = (int)a * TT;
    org[1] = (int)b * TT;
    org[2] = (int)(r - tri(b)) * TT;
  }
  if (tid == 0) {
    tc::mbar_init(&s.bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc::mbar_expect_tx(&s.bar, 18 * TT * TT * TT * 4);
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int o = 0; o < 6; ++o)
        tc::tma_load_4d(&map, &s.bar, s.box[q][o], org[kord(o, 2)], org[kord(o, 1)],
                        org[kord(o, 0)], 3 * t + q);
  }
  {
    // the 3 x 6 blocks of 8 x 8, a 64-thread group each: of the ordered pair sp of tile sets in
    // matrix pr (ij, ik, jk)
    const int r = (tid / TT) % TT, c = tid % TT, grp = tid / (TT * TT);
#pragma unroll
    for (int rep = 0; rep < 5; ++rep) {
      const int x = 4 * rep + grp;
      if (x < 18) {
        const int pr = x / 6, sp = x - 6 * pr, f = sp >> 1, g = pair_second(sp);
        const int row = (f == 0 ? org[0] : (f == 1 ? org[1] : org[2])) + r;
        const int col = (g == 0 ? org[0] : (g == 1 ? org[1] : org[2])) + c;
        const unsigned slab = (unsigned)((pr == 2 ? j : i) * p.no + (pr == 0 ? j : k));
        const bool in = row < v && col < v;
        const long long at = (long long)(slab * (unsigned)v + row) * p.pitch + col;
        s.e[pr][sp][r][c] = in ? __ldg(p.eoovv + at) : 0.f;
        if (FOV) s.d2[pr][sp][r][c] = in ? __ldg(p.t2 + at) : 0.f;
      }
    }
  }
  if (tid < 3 * TT3) {
    const int q = tid / TT3, l = tid % TT3;
    const int x = (l < TT ? org[0] : (l < 2 * TT ? org[1] : org[2])) + l % TT;
    const int occ = q == 0 ? i : (q == 1 ? j : k);
    s.t1r[q][l] = x < v ? f64_to_f32(p.t1[(long long)occ * v + x]) : 0.f;
    if (FOV) s.fr[q][l] = x < v ? f64_to_f32(p.fov[(long long)occ * v + x]) : 0.f;
    if (q == 0) s.ev[l] = x < v ? f64_to_f32(p.eps[p.no + x]) : 0.f;
  }
  if (tid == 0) {
    const bool ok = tc::mbar_wait(&s.bar, 0, p.wait_ns);
    if (!ok) {
      atomicExch(p.status, kStatusTimeoutFull);
      tc::mbar_wait(&s.bar, 0, p.wait_ns);  // the copies in flight, again with a limit
    }
    s.ok = ok;
  }
  __syncthreads();
  if (!s.ok) {
    if (tid == 0)
      p.part[(long long)t * p.ntt + blockIdx.x] = __longlong_as_double(0x7ff8000000000000ll);
    return;
  }
  // the TMA's writes: every thread observes the completed phase itself
  tc::mbar_wait(&s.bar, 0, p.wait_ns);
  const int lane = tid & 31, warp = tid >> 5;
  const int bl = ((lane >> 2) & 3) | (((warp >> 1) & 1) << 2), cl = (lane & 3) | ((warp >> 2) << 2);
  const int b = org[1] + bl, c = org[2] + cl;
  float acc = 0.f;
  const float eo = f64_to_f32(p.eps[i] + p.eps[j] + p.eps[k]);
  auto lin = [](int o, int la, int lb, int lc) {  // place of (la, lb, lc) in a box of ordering o
    const int st[3] = {TT * TT, TT, 1};
    int at = 0;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int set = kord(o, q);
      at += st[q] * (set == 0 ? la : (set == 1 ? lb : lc));
    }
    return at;
  };
#pragma unroll
  for (int rep = 0; rep < 2; ++rep) {
    const int al = (lane >> 4) | (rep << 1) | ((warp & 1) << 2);
    const int a = org[0] + al;
    if (a >= v || b > a || c > b) continue;
    int at[6];
#pragma unroll
    for (int o = 0; o < 6; ++o) at[o] = lin(o, al, bl, cl);
    // W[x, y, z] = P3[x][y][z] + P2[y][x][z] + P1[z][x][y] for the orderings of (a, b, c); the
    // orderings of the boxes' (slow, middle, fast) per ordering of W
    constexpr int o2[6] = {2, 4, 0, 5, 1, 3}, o1[6] = {4, 2, 5, 0, 3, 1};
    const int loc[3] = {al, bl, cl};
    float W[6], V[6];
    const float wt = (float)(1 + (a == b) + (a == c) + (b == c));
    const float rw = 1.f / wt;
#pragma unroll
    for (int o = 0; o < 6; ++o) {
      W[o] = s.box[2][o][at[o]] + s.box[1][o2[o]][at[o2[o]]] + s.box[0][o1[o]][at[o1[o]]];
      const int X = kord(o, 0), Y = kord(o, 1), Z = kord(o, 2);
      auto pr = [](int f, int g) { return 2 * f + (f == 0 ? g - 1 : (f == 1 ? (g == 2) : g)); };
      const int lx = loc[X], ly = loc[Y], lz = loc[Z];
      const int ux = X * TT + lx, uy = Y * TT + ly, uz = Z * TT + lz;
      float d = s.e[0][pr(X, Y)][lx][ly] * s.t1r[2][uz] + s.e[1][pr(X, Z)][lx][lz] * s.t1r[1][uy] +
                s.e[2][pr(Y, Z)][ly][lz] * s.t1r[0][ux];
      if (FOV)
        d += s.d2[0][pr(X, Y)][lx][ly] * s.fr[2][uz] + s.d2[1][pr(X, Z)][lx][lz] * s.fr[1][uy] +
             s.d2[2][pr(Y, Z)][ly][lz] * s.fr[0][ux];
      V[o] = (W[o] + d) * rw;
    }
    float X = 0.f;
#pragma unroll
    for (int q = 0; q < 6; ++q) X += W[q] * V[q];
    const float Y = V[0] + V[3] + V[4], Z = V[1] + V[2] + V[5];
    const float Wc = W[0] + W[3] + W[4], Wa = W[1] + W[2] + W[5];
    const float S = (Y - 2.f * Z) * Wc + (Z - 2.f * Y) * Wa + 3.f * X;
    const float D = eo - s.ev[al] - s.ev[TT + bl] - s.ev[2 * TT + cl];
    acc += S / D;
  }
  for (int sh = 16; sh > 0; sh >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, sh);
  if (lane == 0) s.red[warp] = f32_to_f64(acc);
  __syncthreads();
  if (tid == 0) {
    double r = 0.0;
    for (int q = 0; q < TE2_THREADS / 32; ++q) r += s.red[q];
    const double fac = 2.0 - ((i == j) + (i == k) + (j == k));
    p.part[(long long)t * p.ntt + blockIdx.x] = fac * r;
  }
}

__global__ void reduce_sum_kernel(const double* x, long long n, double* out) {
  __shared__ double red[TE_THREADS / 32];
  double acc = 0.0;
  for (long long q = threadIdx.x; q < n; q += TE_THREADS) acc += x[q];
  for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = (threadIdx.x < TE_THREADS / 32) ? red[threadIdx.x] : 0.0;
    for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
    if (threadIdx.x == 0) *out += v;
  }
}

}  // namespace
}  // namespace pcg

using namespace pcg;

// (T) energy contributions of ntrip triples (see top of file).  fp32 selects FP32 partial
// tensors and FP32 element arithmetic (the tensor-core path, tiled kernel); otherwise FP64
// throughout.  Writes pcg_triples_part_len(fp32, nv) FP64 partials per triple; the caller
// sums them.  pycc/cctriples.py:177-240.
extern "C" int pcg_triples_energy(int fp32, const void* P1, const void* P2, const void* P3,
                                  long long pstride, const int* ijk, int ntrip,
                                  const double* eps, const void* eoovv, const double* t1,
                                  const void* t2, const double* fov, long long no,
                                  long long nv, double* part, void* stream) {
  if (ntrip < 1 || ntrip > 65535 || nv < 1 || nv > 0x7fffffff || !P1 || !P2 || !P3 || !ijk ||
      !eps || !eoovv || !t1 || !t2 || !part) {
    set_error("pcg_triples_energy: bad arguments (ntrip=%d)", ntrip);
    return -1;
  }
  dim3 grid((unsigned)nv, (unsigned)ntrip);
  cudaStream_t st = (cudaStream_t)stream;
  if (fp32) {
    const long long ntt = tile_triples(nv);
    if (ntt > 0x7fffffffLL || nv * nv * nv > 0x7fffffffLL) {
      set_error("pcg_triples_energy: nv=%lld too large", nv);
      return -1;
    }
    if (((uintptr_t)eoovv & 15u) || ((uintptr_t)t2 & 15u)) {
      set_error("pcg_triples_energy: FP32 eoovv and t2 must be 16-byte aligned");
      return -1;
    }
    TripArgs<float> a{(const float*)P1, (const float*)P2, (const float*)P3, pstride, ijk, ntrip,
                      eps, (const float*)eoovv, t1, (const float*)t2, fov, no, nv, part};
    triples_energy_tiled_kernel<<<dim3((unsigned)ntt, (unsigned)ntrip), TE2_THREADS, 0, st>>>(
        a, ntt);
  } else {
    TripArgs<double> a{(const double*)P1, (const double*)P2, (const double*)P3, pstride, ijk,
                       ntrip, eps, (const double*)eoovv, t1, (const double*)t2, fov, no, nv,
                       part};
    triples_energy_kernel<double><<<grid, TE_THREADS, 0, st>>>(a);
  }
  PCG_CHECK_LAUNCH("pcg_triples_energy");
  return 0;
}

// The FP32 path with the partials P[triple][orientation][nv][nv][pitch] and eoovv, t2 of
// [o][o][nv][pitch], pitch a multiple of four floats (16 bytes): the partials' tiles come by TMA.
// *status: a device word that an expired wait sets (the partial is NaN then).  Partials as
// pcg_triples_energy(fp32 = 1) writes them.
extern "C" int pcg_triples_energy_pitched(const float* P, long long pitch, const int* ijk, int ntrip,
                                          const double* eps, const float* eoovv, const double* t1,
                                          const float* t2, const double* fov, long long no,
                                          long long nv, double* part, int* status, void* stream) {
  if (!P || !ijk || !eps || !eoovv || !t1 || !t2 || !part || !status || ntrip < 1 || ntrip > 65535 ||
      no < 1 || nv < 1 || pitch < nv || pitch % 4 != 0 ||
      (((uintptr_t)P | (uintptr_t)eoovv | (uintptr_t)t2) & 15u)) {
    set_error("pcg_triples_energy_pitched: bad arguments (ntrip=%d, pitch=%lld)", ntrip, pitch);
    return -1;
  }
  const long long ntt = tile_triples(nv);
  if (ntt > 0x7fffffffLL || nv * nv * nv > 0x7fffffffLL) {
    set_error("pcg_triples_energy_pitched: nv=%lld too large", nv);
    return -1;
  }
  CUtensorMap map;
  if (!tc::make_map_cube8(&map, P, nv, pitch, 3LL * ntrip)) return -1;
  CubeArgs a{ijk, eps, eoovv, t2, pitch, t1, fov, (int)no, (int)nv, (unsigned)ntt, part, status,
             wait_limit_ns()};
  const dim3 grid((unsigned)ntt, (unsigned)ntrip);
  if (fov)
    triples_energy_cube_kernel<true><<<grid, TE2_THREADS, 0, (cudaStream_t)stream>>>(map, a);
  else
    triples_energy_cube_kernel<false><<<grid, TE2_THREADS, 0, (cudaStream_t)stream>>>(map, a);
  PCG_CHECK_LAUNCH("pcg_triples_energy_pitched");
  return 0;
}

// FP64 partials per triple written by pcg_triples_energy: one per virtual index a (FP64),
// one per tile triple of the (a, b, c) cube (FP32).
extern "C" long long pcg_triples_part_len(int fp32, long long nv) {
  return fp32 ? tile_triples(nv) : nv;
}

// *out += sum(x[0:n]) in FP64, one block (deterministic order).
extern "C" int pcg_reduce_sum_f64(const double* x, long long n, double* out, void* stream) {
  if (!x || !out || n < 0) {
    set_error("pcg_reduce_sum_f64: bad arguments");
    return -1;
  }
  reduce_sum_kernel<<<1, TE_THREADS, 0, (cudaStream_t)stream>>>(x, n, out);
  PCG_CHECK_LAUNCH("pcg_reduce_sum_f64");
  return 0;
}
