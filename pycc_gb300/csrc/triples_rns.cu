// The connected triples t3c_ijk (pycc/cctriples.py:27-72) in FP64 on the BF16 tensor cores, by
// the residue arithmetic of contract_rns.cu.
//
// The twelve terms of a triple are products of six operand matrices, turned into residues once
// for one set of amplitudes:
//   A side (rows (x, p, q)):  VT = <qp|ex>,  VN = <pq|ex>  (K = e);  TM = t2_xmpq,
//                             TMT = t2_xmqp  (K = m)
//   B side (rows (x, y, p)):  T2P = t2_xype  (K = e);  OB = -<mp|xy>  (K = m)
// An orientation is a sum of four products (pycc_gb300/triples.py, orientation_terms), in which VT
// meets T2P's rows (y, z) where TM of the same index meets OB's (z, y), and VN and TMT likewise.
// So the residues are stored side by side along K, [VT | TM], [VN | TMT] and [T2P | OB with x and y
// exchanged], and an orientation is two products of K = nv + no: at no = 7, nv = 45 two 64-K
// blocks in place of four.  The residue of the sum is the sum's when all four products carry the
// same scale, so a matrix has one power of two for all its rows, chosen from its largest row norm
// so that the sum of the four stays below half the product of the moduli; a partial whose products
// are small at that scale is computed again in FP64 (kDoubt in rns.cuh).  One GEMM launch computes
// the three orientations of a batch of triples, a second kernel rebuilds the partials in FP64, in
// the layout the energy kernel reads.  E(T) at no = 7, nv = 45: 63.4 ms with one FP64 launch per
// triple and orientation (46.6 ms on a few SMs' FP64 pipes, a host synchronisation per triple),
// 1.34 ms here (GEMM 0.45, by half more with the four products apart; rebuild 0.20, energy 0.32).
#include "rns.cuh"

namespace pcg {
namespace rns {
namespace {

struct T3Shift {
  int sh[4];  // V, T2P, t2 (rows of TM), OB
  int total;  // sh[0] + sh[1] = sh[2] + sh[3]
  int bad;    // an operand holds an Inf or a NaN
};

struct T3MaxArgs {
  const unsigned long long* norm[4];
  long long R[4];
  unsigned* out;  // [4] largest log2 of a squared row norm, rounded up, + kT3Bias (0: no row is above
                  // zero); [1] an Inf or a NaN
};
constexpr int kT3Bias = 1 << 16;

__global__ void __launch_bounds__(256) t3_max_kernel(const T3MaxArgs p) {
  const int q = blockIdx.y;
  unsigned m = 0, bad = 0;
  for (long long r = (long long)blockIdx.x * 256 + threadIdx.x; r < p.R[q];
       r += (long long)gridDim.x * 256) {
    const RowNorm n = RowNorm::from(p.norm[q][r]);
    unsigned frac;
    if (n.s > 0.f) m = max(m, (unsigned)(n.log2(frac) + 1 + kT3Bias));
    bad |= n.top == 2047;
  }
  m = __reduce_max_sync(0xffffffffu, m);
  bad = __reduce_or_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(p.out + q, m);
    if (bad) p.out[4] = 1;
  }
}

// Powers of two that keep every product of two row norms at or below 2^kT3Bits.  By Cauchy-Schwarz
// the four products of an orientation sum to at most 4 2^kT3Bits = 2^123, and the residues
// determine a sum of up to half the product of the moduli, 2^123.95.
constexpr int kT3Bits = 121;
static_assert(kT3Bits + 2 <= kSumBits, "four products stay in the range of the residues");
__global__ void t3_shift_kernel(const unsigned* mx, T3Shift* out) {
  int e[4];  // row norms are at most 2^e
  for (int q = 0; q < 4; ++q) e[q] = mx[q] ? ((int)mx[q] - kT3Bias + 1) >> 1 : -1000;
  const int s1 = kT3Bits - e[0] - e[1], s2 = kT3Bits - e[2] - e[3], s = min(s1, s2);
  out->sh[0] = kT3Bits / 2 - e[0] - ((s1 - s) >> 1);
  out->sh[1] = s - out->sh[0];
  out->sh[2] = kT3Bits / 2 - e[2] - ((s2 - s) >> 1);
  out->sh[3] = s - out->sh[2];
  out->total = s;
  out->bad = mx[4] != 0;
}

struct T3JoinArgs {
  const unsigned char* res;  // [group][plane][v^2][ld]
  long long ld;
  int nv, groups;
  double* P;  // [group][z][x][y]
  const T3Shift* shift;
  const int* status;
  CrtTab t;
  // operands for partials that are computed again in FP64, or null: none is
  const double *V, *O, *t2;
  const int* ijk;
  int no;
};

// One partial, orientation g % 3 of triple g / 3, by a warp with the lanes along K (e, then m).
__device__ __noinline__ double t3_dot(const T3JoinArgs& p, int g, long long row, int z) {
  const int q = g % 3, lane = threadIdx.x & 31;
  const int i = p.ijk[g - q], j = p.ijk[g - q + 1], k = p.ijk[g - q + 2];
  const long long o = p.no, v = p.nv, x = row / v, y = row - x * v;
  double s = 0.0;
  for (int part = 0; part < 2; ++part) {  // [VT | TM] or [VN | TMT], as decode_unit has them
    const T3Product t = t3_product(q, part, i, j, k);
    const long long a = t.swap ? x : y, b = t.swap ? y : x;  // VT = <qp|ex>, VN = <pq|ex>
    const double* V = p.V + (a * v + b) * v * o + t.a;
    const double* T = p.t2 + ((t.bx * o + t.by) * v + z) * v;
    for (long long e = lane; e < v; e += 32) s = fma(__ldg(V + e * o), __ldg(T + e), s);
    const double* M = p.t2 + t.a * o * v * v + b * v + a;    // TM = t2_xmpq, TMT = t2_xmqp
    const double* O = p.O + (z * o + t.by) * o + t.bx;
    for (long long m = lane; m < o; m += 32)
      s = fma(-__ldg(M + m * v * v), __ldg(O + m * v * o * o), s);
  }
  for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  return s;
}

// Lanes along the rows (x, y), which are P's unit stride; four columns z per thread.  A partial
// whose products are small against the norms behind its scale (kDoubt in rns.cuh) is computed again
// in FP64, a warp each, and so are all of them with an Inf or a NaN in an operand: at most a third of the time of one FP64 launch per triple and orientation.
__global__ void __launch_bounds__(256, 4) t3_join_kernel(const __grid_constant__ T3JoinArgs p) {
  const long long M = (long long)p.nv * p.nv;
  const long long row0 = (long long)blockIdx.x * 32, row = row0 + threadIdx.x;
  const int col = 4 * (int)(blockIdx.y * 8 + threadIdx.y);
  if (col >= p.nv) return;  // a whole warp
  const bool failed = *p.status != 0, bad = p.shift->bad;
  const int ex = -p.shift->total;
  for (int g = blockIdx.z; g < p.groups; g += gridDim.z) {
    double* out = p.P + ((long long)g * p.nv + col) * M + row;
    unsigned doubt = 0;
    if (row < M) {
      const unsigned char* src = p.res + ((long long)g * NP * M + row) * p.ld + col;
      unsigned w[NP];
#pragma unroll
      for (int l = 0; l < NP; ++l)
        w[l] = __ldg(reinterpret_cast<const unsigned*>(src + (long long)l * M * p.ld));
      CrtSum sum(p.t);
      sum.add(p.t, w);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float mag = magnitude_sum(w[NM], e);
        if (col + e < p.nv) {
          out[e * M] =
              failed || bad ? __longlong_as_double(0x7ff8000000000000ll) : sum.value(p.t, e, ex);
          if (p.V && !failed && (bad || (mag > 0.f && mag < kDoubt))) doubt |= 1u << e;
        }
      }
    }
    if (__any_sync(0xffffffffu, doubt != 0u))
      for (int e = 0; e < 4; ++e)
        for (unsigned m = __ballot_sync(0xffffffffu, doubt >> e & 1u); m; m &= m - 1) {
          const int l = __ffs((int)m) - 1;
          const double v = t3_dot(p, g, row0 + l, col + e);
          if (threadIdx.x == l) out[e * M] = v;
        }
  }
}

// Workspace of a wave function: status and shifts, the residues of the matrices, then each
// batch's products (during packing the rows' tables lie there instead).
struct T3Plan {
  long long no, nv, rows_a, rows_b, ld;
  long long c0, kc;          // first column of the m part, a multiple of 8; columns in 64-K blocks
  long long a1, a2, b, fixed;  // byte offsets; fixed: the end of the residues
  long long tables, per_triple;
};

bool t3_plan(T3Plan& p, long long no, long long nv) {
  if (no < 1 || nv < 1 || no > 2048 || nv > 8192) return false;
  p.no = no;
  p.nv = nv;
  p.rows_a = no * nv * nv;
  p.rows_b = no * no * nv;
  p.c0 = up(nv, 8);
  p.kc = up(p.c0 + no, 64);
  p.ld = up(nv, 16);
  const long long a = up(NP * p.rows_a * p.kc * 2, 256);
  p.a1 = 256;
  p.a2 = p.a1 + a;
  p.b = p.a2 + a;
  p.fixed = p.b + up(NP * p.rows_b * p.kc * 2, 256);
  p.tables = (4 * p.rows_a + 2 * p.rows_b) * (8 + 8 + 4) + 6 * 3 * 16;
  p.per_triple = 3 * NP * nv * nv * p.ld;
  return NP * p.rows_a < 0x7fffffffLL - BM && NP * p.rows_b < 0x7fffffffLL - 256 &&
         (p.rows_a / 64 + p.rows_b / 32 + 4) * (p.kc / 64) < 0x7fffffffLL;
}

}  // namespace
}  // namespace rns
}  // namespace pcg

using namespace pcg;
using namespace pcg::rns;

extern "C" int pcg_t3_rns_work(long long no, long long nv, int batch, long long* bytes) {
  T3Plan p;
  if (!bytes || batch < 1) {
    set_error("pcg_t3_rns_work: bad arguments");
    return -1;
  }
  *bytes = t3_plan(p, no, nv) ? p.fixed + std::max(p.tables, batch * p.per_triple) : 0;
  return 0;
}

extern "C" int pcg_t3_rns_pack(const double* V, const double* O, const double* t2, long long no,
                               long long nv, void* work, long long work_len, void* stream) {
  T3Plan p;
  if (!V || !O || !t2 || !work || ((uintptr_t)work & 255u) || !t3_plan(p, no, nv) ||
      work_len < p.fixed + p.tables) {
    set_error("pcg_t3_rns_pack: bad arguments, or too little workspace");
    return -1;
  }
  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* w = (unsigned char*)work;
  unsigned* mx = (unsigned*)(w + 64);
  T3Shift* shift = (T3Shift*)(w + 128);
  unsigned char* tb = w + p.fixed;
  auto take = [&](long long bytes) {  // every array 16-byte aligned
    unsigned char* r = tb;
    tb += up(bytes, 16);
    return r;
  };
  const long long o = no, v = nv;
  auto operand = [&](const double* X, long long e0, long long s0, long long e1, long long s1,
                     long long e2, long long s2, long long kstep, int near, int which) {
    Operand x{};
    x.X = X;
    x.r.n = 3;
    x.r.ext[0] = e0;
    x.r.ext[1] = e1;
    x.r.ext[2] = e2;
    x.r.s0[0] = s0;
    x.r.s0[1] = s1;
    x.r.s0[2] = s2;
    x.R = e0 * e1 * e2;
    x.off = (long long*)take(8 * x.R);
    x.norm = (unsigned long long*)take(8 * x.R);
    x.walk = (int*)take(4 * x.R);
    x.kstep = kstep;
    x.kfast = kstep == 1;
    x.wq = near;
    x.shift = &shift->sh[which];
    return x;
  };
  const Operand vt = operand(V, o, 1, v, v * o, v, v * v * o, o, 0, 0);
  const Operand vn = operand(V, o, 1, v, v * v * o, v, v * o, o, 0, 0);
  const Operand tm = operand(t2, o, o * v * v, v, v, v, 1, v * v, 2, 2);
  const Operand tmt = operand(t2, o, o * v * v, v, 1, v, v, v * v, 1, 2);
  const Operand t2p = operand(t2, o, o * v * v, o, v * v, v, v, 1, 2, 1);
  const Operand ob = operand(O, o, 1, o, o, v, o * o, v * o * o, 0, 3);
  const Operand none{};
  struct {
    Operand a, b;
    long long K, c0, width, pa, pb;  // columns [c0, c0 + width) of the panels at pa and pb
  } pass[4] = {{vt, t2p, v, 0, p.c0, p.a1, p.b}, {tm, ob, o, p.c0, p.kc - p.c0, p.a1, p.b},
               {vn, none, v, 0, p.c0, p.a2, 0}, {tmt, none, o, p.c0, p.kc - p.c0, p.a2, 0}};
  cudaMemsetAsync(w, 0, 256, st);
  for (auto& x : pass) {
    TableArgs t{x.a, x.b, SubIdx{}, 0, nullptr, nullptr, nullptr};
    rns_tables_kernel<<<blocks_for(x.a.R + x.b.R, 256), 256, 0, st>>>(t);
    PCG_CHECK_LAUNCH("pcg_t3_rns_pack/tables");
  }
  const NormScratch scratch{{w + p.a1, w + p.b}, {p.a2 - p.a1, p.fixed - p.b}};
  for (int q = 0; q < 2; ++q)
    if (run_norm(pass[q].a, pass[q].b, 0, pass[q].K, scratch, st)) return -2;
  T3MaxArgs m{{vt.norm, t2p.norm, tm.norm, ob.norm}, {vt.R, t2p.R, tm.R, ob.R}, mx};
  t3_max_kernel<<<dim3(num_sms(), 4), 256, 0, st>>>(m);
  PCG_CHECK_LAUNCH("pcg_t3_rns_pack/max");
  t3_shift_kernel<<<1, 1, 0, st>>>(mx, shift);
  PCG_CHECK_LAUNCH("pcg_t3_rns_pack/shift");
  for (auto& x : pass) {
    PackArgs a{{{x.a, 0, x.a.R, (__nv_bfloat16*)(w + x.pa) + x.c0, 0, 0},
                {x.b, 0, x.b.R, (__nv_bfloat16*)(w + x.pb) + x.c0, x.b.X == O ? 0x80000000u : 0u, 0}},
               0, x.K, x.width, p.kc, tables().pairs};
    if (run_pack(a, st)) return -2;
  }
  return 0;
}

namespace {
int t3_partials(const double* V, const double* O, const double* t2, long long no, long long nv,
                const int* ijk, int ntrip, double* P, void* work, long long work_len, void* stream,
                const char* who) {
  T3Plan p;
  if (!ijk || ntrip < 1 || ntrip > 21845 || !P || !work || ((uintptr_t)work & 255u) ||
      !t3_plan(p, no, nv) || work_len < p.fixed + ntrip * p.per_triple) {
    set_error("%s: bad arguments, or too little workspace", who);
    return -1;
  }
  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* w = (unsigned char*)work;
  GemmArgs g{};
  g.M = nv * nv;
  g.N = nv;
  g.mt = (g.M + BM - 1) / BM;
  const int BN = nv > 128 ? 256 : (nv > 64 ? 128 : 64);
  g.nt = (nv + BN - 1) / BN;
  g.bs = (int)(16 * (((nv + 15) / 16 + g.nt - 1) / g.nt));
  g.gm = 1;
  g.planes = 3 * ntrip;
  g.ld = p.ld;
  g.out = w + p.fixed;
  g.status = (int*)w;
  g.wait_ns = wait_limit_ns();
  g.t = tables().mod;
  g.ijk = ijk;
  g.no = (int)no;
  g.kc = (int)(p.kc / 64);
  GemmMaps maps{};
  if (!make_map(&maps.a[0], w + p.a1, NP * p.rows_a, 2 * p.kc, 2 * p.kc, 2, BM) ||
      !make_map(&maps.a[1], w + p.a2, NP * p.rows_a, 2 * p.kc, 2 * p.kc, 2, BM) ||
      !make_map(&maps.b[0], w + p.b, NP * p.rows_b, 2 * p.kc, 2 * p.kc, 2, g.bs))
    return -1;
  const int rc = BN == 256   ? run_gemm<256, true>(maps, g, st)
                 : BN == 128 ? run_gemm<128, true>(maps, g, st)
                             : run_gemm<64, true>(maps, g, st);
  if (rc) return rc;
  T3JoinArgs j{w + p.fixed, p.ld, (int)nv, g.planes, P, (const T3Shift*)(w + 128),
               (const int*)w, crt_tab(1, 1.0), V, O, t2, ijk, (int)no};
  const dim3 grid((unsigned)((g.M + 31) / 32), (unsigned)((nv + 31) / 32), (unsigned)g.planes);
  t3_join_kernel<<<grid, dim3(32, 8), 0, st>>>(j);
  PCG_CHECK_LAUNCH(who);
  return 0;
}
}  // namespace

extern "C" int pcg_t3_rns_partials(long long no, long long nv, const int* ijk, int ntrip, double* P,
                                   void* work, long long work_len, void* stream) {
  return t3_partials(nullptr, nullptr, nullptr, no, nv, ijk, ntrip, P, work, work_len, stream,
                     "pcg_t3_rns_partials");
}

extern "C" int pcg_t3_rns_partials_of(const double* V, const double* O, const double* t2, long long no,
                                      long long nv, const int* ijk, int ntrip, double* P, void* work,
                                      long long work_len, void* stream) {
  if (!V || !O || !t2) {
    set_error("pcg_t3_rns_partials_of: null operand");
    return -1;
  }
  return t3_partials(V, O, t2, no, nv, ijk, ntrip, P, work, work_len, stream,
                     "pcg_t3_rns_partials_of");
}
