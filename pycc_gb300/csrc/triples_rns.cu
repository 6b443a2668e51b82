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
  const unsigned long long* norm[2];
  long long R[2];
  int which[2];   // entry of `out`
  unsigned* out;  // [4] largest log2 of a squared row norm, rounded up, + kT3Bias (0: no row is
                  // above zero); [1] an Inf or a NaN
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
    atomicMax(p.out + p.which[q], m);
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
__device__ __forceinline__ double t3_dot(const T3JoinArgs& p, int g, long long row, int z) {
  const int q = g % 3, lane = threadIdx.x & 31;
  const int i = p.ijk[g - q], j = p.ijk[g - q + 1], k = p.ijk[g - q + 2];
  const long long o = p.no, v = p.nv, x = row / v, y = row - x * v;
  double s = 0.0;
  for (int part = 0; part < 2; ++part) {  // [VT | TM] or [VN | TMT], as decode_unit has them
    const T3Product t = t3_product(q, part);
    auto of = [=](int r) { return r == 0 ? i : (r == 1 ? j : k); };
    const long long w = of(t.a), bx = of(t.bx), by = of(t.by);
    const long long a = t.swap ? x : y, b = t.swap ? y : x;  // VT = <qp|ex>, VN = <pq|ex>
    const double* V = p.V + (a * v + b) * v * o + w;
    const double* T = p.t2 + ((bx * o + by) * v + z) * v;
    for (long long e = lane; e < v; e += 32) s = fma(__ldg(V + e * o), __ldg(T + e), s);
    const double* M = p.t2 + w * o * v * v + b * v + a;      // TM = t2_xmpq, TMT = t2_xmqp
    const double* O = p.O + (z * o + by) * o + bx;
    for (long long m = lane; m < o; m += 32)
      s = fma(-__ldg(M + m * v * v), __ldg(O + m * v * o * o), s);
  }
  for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  return s;
}

// The partials that the lanes of a warp (rows row0, row0 + 1, ...) marked: bit e, column col + e.
__device__ __noinline__ void t3_redo(const T3JoinArgs& p, int g, long long row0, int col,
                                     unsigned doubt) {
  const long long M = (long long)p.nv * p.nv;
  for (int e = 0; e < 4; ++e)
    for (unsigned m = __ballot_sync(0xffffffffu, doubt >> e & 1u); m; m &= m - 1) {
      const int l = __ffs((int)m) - 1;
      const double v = t3_dot(p, g, row0 + l, col + e);
      if (threadIdx.x == l) p.P[((long long)g * p.nv + col + e) * M + row0 + l] = v;
    }
}

// Lanes along the rows (x, y), which are P's unit stride; four columns z per thread.  A partial
// whose products are small against the norms behind its scale (kDoubt in rns.cuh) is computed again
// in FP64, a warp each, and so are all of them with an Inf or a NaN in an operand (E(T) at no = 7,
// nv = 45 then takes 18 ms, at no = 9, nv = 70 133; with one FP64 launch per triple and orientation
// 50 and 256).  Five resident blocks: no = 9, nv = 70 1.38 ms, with four or six 1.53.
__global__ void __launch_bounds__(256, 5) t3_join_kernel(const __grid_constant__ T3JoinArgs p) {
  const long long M = (long long)p.nv * p.nv;
  const long long row0 = (long long)blockIdx.x * 32, row = row0 + threadIdx.x;
  const int col = 4 * (int)(blockIdx.y * 8 + threadIdx.y);
  if (col >= p.nv) return;  // a whole warp
  const bool failed = *p.status != 0, bad = p.shift->bad;
  const int ex = -p.shift->total;
  for (int g = blockIdx.z; g < p.groups; g += gridDim.z) {
    unsigned doubt = 0;
    if (row < M) {
      double* out = p.P + ((long long)g * p.nv + col) * M + row;
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
    if (__any_sync(0xffffffffu, doubt != 0u)) t3_redo(p, g, row0, col, doubt);
  }
}

// Workspace: status and shifts, the residues of the matrices, then each batch's products (while
// operands are prepared, the rows' tables lie there instead).  The residues of all occupied
// orbitals take 17 * 4 no nv^2 kc bytes (38 GB at no = 30, nv = 240), so a caller may go through
// the triples in windows: i, j and k each in a slot of c orbitals, of which [VT | TM] holds i's
// and j's and [VN | TMT] j's and k's.  c = no: one slot for all three.
struct T3Plan {
  long long no, nv, c;
  bool windows;
  long long blocks_a, pairs, rows_a, rows_b, ld;
  long long c0, kc;          // first column of the m part, a multiple of 8; columns in 64-K blocks
  long long a1, a2, b, fixed;  // byte offsets; fixed: the end of the residues
  long long tables, per_triple;
};

bool t3_plan(T3Plan& p, long long no, long long nv, long long c) {
  if (no < 1 || nv < 1 || no > 2048 || nv > 8192 || c < 1 || c > no) return false;
  p.no = no;
  p.nv = nv;
  p.c = c;
  p.windows = c < no;
  p.blocks_a = p.windows ? 2 * c : no;
  p.pairs = p.windows ? 9 * c * c : no * no;
  p.rows_a = p.blocks_a * nv * nv;
  p.rows_b = p.pairs * nv;
  p.c0 = up(nv, 8);
  p.kc = up(p.c0 + no, 64);
  p.ld = up(nv, 16);
  const long long a = up(NP * p.rows_a * p.kc * 2, 256);
  p.a1 = 256;
  p.a2 = p.a1 + a;
  p.b = p.a2 + a;
  p.fixed = p.b + up(NP * p.rows_b * p.kc * 2, 256);
  p.tables = 2 * (c * nv * std::max(nv, no) * (8 + 8 + 4) + 3 * 16);
  p.per_triple = 3 * NP * nv * nv * p.ld;
  return NP * p.rows_a < 0x7fffffffLL - BM && NP * p.rows_b < 0x7fffffffLL - 256 &&
         (p.rows_a / 64 + p.rows_b / 32 + 4) * (p.kc / 64) < 0x7fffffffLL &&
         c * nv * std::max(nv, no) < 0x7fffffffLL;
}

// Rows of one of the matrices.
struct T3Rows {
  const double* X;
  long long e[3], s[3], kstep;
  int near, which;  // sub-index walked innermost, scale
  unsigned flip;
};
enum T3Matrix { kVT, kVN, kTM, kTMT, kT2P, kOB };

// Occupied indices [x0, x0 + nx) and, on the B side, [y0, y0 + ny).
T3Rows t3_rows(T3Matrix m, const double* V, const double* O, const double* t2, long long o,
               long long v, long long x0, long long nx, long long y0, long long ny) {
  switch (m) {
    case kVT: return {V + x0, {nx, v, v}, {1, v * o, v * v * o}, o, 0, 0, 0};
    case kVN: return {V + x0, {nx, v, v}, {1, v * v * o, v * o}, o, 0, 0, 0};
    case kTM: return {t2 + x0 * o * v * v, {nx, v, v}, {o * v * v, v, 1}, v * v, 2, 2, 0};
    case kTMT: return {t2 + x0 * o * v * v, {nx, v, v}, {o * v * v, 1, v}, v * v, 1, 2, 0};
    case kT2P:
      return {t2 + (x0 * o + y0) * v * v, {nx, ny, v}, {o * v * v, v * v, v}, 1, 2, 1, 0};
    default: return {O + y0 * o + x0, {nx, ny, v}, {1, o, o * o}, v * o * o, 0, 3, 0x80000000u};
  }
}

// The header's parts and operands whose tables lie behind the residues, one pair at a time.
struct T3Work {
  const T3Plan& p;
  unsigned char* w;
  cudaStream_t st;
  unsigned* mx() const { return (unsigned*)(w + 64); }
  T3Shift* shift() const { return (T3Shift*)(w + 128); }
  // builds the tables of one or two row sets (b null: one)
  int tables(const T3Rows& ra, const T3Rows* rb, Operand& a, Operand& b) const {
    unsigned char* tb = w + p.fixed;
    auto take = [&](long long bytes) {  // every array 16-byte aligned
      unsigned char* r = tb;
      tb += up(bytes, 16);
      return r;
    };
    auto operand = [&](const T3Rows& r) {
      Operand x{};
      x.X = r.X;
      x.r.n = 3;
      x.R = 1;
      for (int q = 0; q < 3; ++q) {
        x.r.ext[q] = r.e[q];
        x.r.s0[q] = r.s[q];
        x.R *= r.e[q];
      }
      x.off = (long long*)take(8 * x.R);
      x.norm = (unsigned long long*)take(8 * x.R);
      x.walk = (int*)take(4 * x.R);
      x.kstep = r.kstep;
      x.kfast = r.kstep == 1;
      x.wq = r.near;
      x.shift = &shift()->sh[r.which];
      return x;
    };
    a = operand(ra);
    b = rb ? operand(*rb) : Operand{};
    TableArgs t{a, b, SubIdx{}, 0, nullptr, nullptr, nullptr};
    rns_tables_kernel<<<blocks_for(a.R + b.R, 256), 256, 0, st>>>(t);
    PCG_CHECK_LAUNCH("pcg_t3_rns/tables");
    return 0;
  }
};

bool t3_arguments(T3Plan& p, const void* work, long long work_len, long long no, long long nv,
                  long long c, long long batch, const char* who) {
  if (!work || ((uintptr_t)work & 255u) || !t3_plan(p, no, nv, c) ||
      work_len < p.fixed + std::max(p.tables, batch * p.per_triple)) {
    set_error("%s: bad arguments, or too little workspace", who);
    return false;
  }
  return true;
}

// The scales of the four operands, from the norms of all their rows; clears the status.
int t3_scales(const T3Plan& p, const double* V, const double* O, const double* t2, unsigned char* w,
              cudaStream_t st) {
  const T3Work k{p, w, st};
  const long long o = p.no, v = p.nv;
  const NormScratch scratch{{w + p.a1, w + p.b}, {p.a2 - p.a1, p.fixed - p.b}};
  cudaMemsetAsync(w, 0, 256, st);
  for (long long x0 = 0; x0 < o; x0 += p.c)
    for (int q = 0; q < 2; ++q) {
      const long long nx = std::min(p.c, o - x0);
      const T3Rows ra = t3_rows(q ? kTM : kVT, V, O, t2, o, v, x0, nx, 0, o);
      const T3Rows rb = t3_rows(q ? kOB : kT2P, V, O, t2, o, v, x0, nx, 0, o);
      Operand a, b;
      if (k.tables(ra, &rb, a, b) || run_norm(a, b, 0, q ? o : v, scratch, st)) return -2;
      T3MaxArgs m{{a.norm, b.norm}, {a.R, b.R}, {ra.which, rb.which}, k.mx()};
      t3_max_kernel<<<dim3(num_sms(), 2), 256, 0, st>>>(m);
      PCG_CHECK_LAUNCH("pcg_t3_rns/max");
    }
  t3_shift_kernel<<<1, 1, 0, st>>>(k.mx(), k.shift());
  PCG_CHECK_LAUNCH("pcg_t3_rns/shift");
  return 0;
}

// Occupied indices in the slot that starts at `first`.
long long t3_width(const T3Plan& p, long long first) { return std::min(p.c, p.no - first); }

// Residues of the slots in `changed` (bits 0, 1, 2: i, j, k) and of their pairs.
int t3_pack(const T3Plan& p, const double* V, const double* O, const double* t2, const int* first,
            unsigned changed, unsigned char* w, cudaStream_t st) {
  struct Item {
    T3Rows rows;
    unsigned char* panel;
    long long row, plane;  // first row in the panel, rows of a plane
  };
  const T3Work k{p, w, st};
  const long long o = p.no, v = p.nv;
  Item items[2][16];  // over e, over m
  int n = 0;
  auto add = [&](T3Matrix e, T3Matrix m, unsigned char* panel, long long row, long long plane,
                 long long x0, long long nx, long long y0, long long ny) {
    items[0][n] = {t3_rows(e, V, O, t2, o, v, x0, nx, y0, ny), panel, row, plane};
    items[1][n++] = {t3_rows(m, V, O, t2, o, v, x0, nx, y0, ny), panel, row, plane};
  };
  if (!p.windows) {
    add(kVT, kTM, w + p.a1, 0, p.rows_a, 0, o, 0, 0);
    add(kT2P, kOB, w + p.b, 0, p.rows_b, 0, o, 0, o);
    add(kVN, kTMT, w + p.a2, 0, p.rows_a, 0, o, 0, 0);
  } else {
    for (int r = 0; r < 3; ++r) {
      if (!(changed >> r & 1)) continue;
      const long long f = first[r], nr = t3_width(p, f);
      if (r < 2) add(kVT, kTM, w + p.a1, r * p.c * v * v, p.rows_a, f, nr, 0, 0);
      if (r > 0) add(kVN, kTMT, w + p.a2, (r - 1) * p.c * v * v, p.rows_a, f, nr, 0, 0);
    }
    for (int r = 0; r < 3; ++r)
      for (int s = 0; s < 3; ++s)
        if (r != s && ((changed >> r | changed >> s) & 1))
          add(kT2P, kOB, w + p.b, (3 * r + s) * p.c * p.c * v, p.rows_b, first[r],
              t3_width(p, first[r]), first[s], t3_width(p, first[s]));
  }
  for (int q = 0; q < 2; ++q)
    for (int i = 0; i < n; i += 2) {
      const Item *a = &items[q][i], *b = i + 1 < n ? &items[q][i + 1] : nullptr;
      const long long col = q ? p.c0 : 0;
      Operand oa, ob;
      if (k.tables(a->rows, b ? &b->rows : nullptr, oa, ob)) return -2;
      auto side = [&](const Item& x, const Operand& op) {
        return PackSide{op, 0, op.R, (__nv_bfloat16*)x.panel + x.row * p.kc + col,
                        x.plane * p.kc / 8, x.rows.flip, 0};
      };
      PackArgs args{{side(*a, oa), b ? side(*b, ob) : PackSide{}}, 0, q ? o : v,
                    q ? p.kc - p.c0 : p.c0, p.kc, tables().pairs};
      if (run_pack(args, st)) return -2;
    }
  return 0;
}

int t3_partials(const T3Plan& p, const double* V, const double* O, const double* t2,
                const int* first, const int* ijk, int ntrip, double* P, unsigned char* w,
                cudaStream_t st, const char* who) {
  const long long nv = p.nv;
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
  g.kc = (int)(p.kc / 64);
  g.blocks_a = (int)p.blocks_a;
  g.pairs = (int)p.pairs;
  g.c = p.windows ? (int)p.c : 0;
  for (int r = 0; r < 3; ++r) {
    g.first[r] = p.windows ? first[r] : 0;
    g.width[r] = p.windows ? (int)t3_width(p, first[r]) : (int)p.no;
  }
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
               (const int*)w, crt_tab(1, 1.0), V, O, t2, ijk, (int)p.no};
  const dim3 grid((unsigned)((g.M + 31) / 32), (unsigned)((nv + 31) / 32), (unsigned)g.planes);
  t3_join_kernel<<<grid, dim3(32, 8), 0, st>>>(j);
  PCG_CHECK_LAUNCH(who);
  return 0;
}

bool t3_operands(const double* V, const double* O, const double* t2, const char* who) {
  if (V && O && t2) return true;
  set_error("%s: null operand", who);
  return false;
}
bool t3_batch(const int* ijk, int ntrip, const double* P, const char* who) {
  if (ijk && P && ntrip >= 1 && ntrip <= 21845) return true;
  set_error("%s: bad triples (%d of them) or no output", who, ntrip);
  return false;
}
// Slots are at multiples of c; the first of i's, j's and k's do not increase.
bool t3_first(const T3Plan& p, const int* first, const char* who) {
  bool ok = first != nullptr;
  for (int r = 0; ok && r < 3; ++r)
    ok = first[r] >= 0 && first[r] < p.no && first[r] % p.c == 0 &&
         (r == 0 || first[r] <= first[r - 1]);
  if (!ok) set_error("%s: bad first indices of the window's slots", who);
  return ok;
}

}  // namespace
}  // namespace rns
}  // namespace pcg

using namespace pcg;
using namespace pcg::rns;

namespace {
int work_entry(const char* who, long long no, long long nv, long long c, int batch,
               long long* bytes) {
  T3Plan p;
  if (!bytes || batch < 1 || c < 1) {
    set_error("%s: bad arguments", who);
    return -1;
  }
  *bytes = t3_plan(p, no, nv, c) ? p.fixed + std::max(p.tables, batch * p.per_triple) : 0;
  return 0;
}

int partials_entry(const char* who, const double* V, const double* O, const double* t2,
                   long long no, long long nv, long long c, const int* first, const int* ijk,
                   int ntrip, double* P, void* work, long long work_len, void* stream) {
  T3Plan p;
  if (!t3_operands(V, O, t2, who) || !t3_batch(ijk, ntrip, P, who) ||
      !t3_arguments(p, work, work_len, no, nv, c, ntrip, who) || !t3_first(p, first, who))
    return -1;
  return t3_partials(p, V, O, t2, first, ijk, ntrip, P, (unsigned char*)work, (cudaStream_t)stream,
                     who);
}

const int kNoFirst[3] = {0, 0, 0};
}  // namespace

extern "C" int pcg_t3_rns_window_work(long long no, long long nv, long long c, int batch,
                                      long long* bytes) {
  return work_entry("pcg_t3_rns_window_work", no, nv, c, batch, bytes);
}

extern "C" int pcg_t3_rns_scales(const double* V, const double* O, const double* t2, long long no,
                                 long long nv, long long c, void* work, long long work_len,
                                 void* stream) {
  T3Plan p;
  if (!t3_operands(V, O, t2, "pcg_t3_rns_scales") ||
      !t3_arguments(p, work, work_len, no, nv, c, 0, "pcg_t3_rns_scales"))
    return -1;
  return t3_scales(p, V, O, t2, (unsigned char*)work, (cudaStream_t)stream);
}

extern "C" int pcg_t3_rns_window_pack(const double* V, const double* O, const double* t2,
                                      long long no, long long nv, long long c, const int* first,
                                      int changed, void* work, long long work_len, void* stream) {
  T3Plan p;
  if (!t3_operands(V, O, t2, "pcg_t3_rns_window_pack") ||
      !t3_arguments(p, work, work_len, no, nv, c, 0, "pcg_t3_rns_window_pack") ||
      !t3_first(p, first, "pcg_t3_rns_window_pack"))
    return -1;
  return t3_pack(p, V, O, t2, first, (unsigned)changed, (unsigned char*)work, (cudaStream_t)stream);
}

extern "C" int pcg_t3_rns_window_partials(const double* V, const double* O, const double* t2,
                                          long long no, long long nv, long long c, const int* first,
                                          const int* ijk, int ntrip, double* P, void* work,
                                          long long work_len, void* stream) {
  return partials_entry("pcg_t3_rns_window_partials", V, O, t2, no, nv, c, first, ijk, ntrip, P,
                        work, work_len, stream);
}

// The same with all occupied orbitals in one window.
extern "C" int pcg_t3_rns_work(long long no, long long nv, int batch, long long* bytes) {
  return work_entry("pcg_t3_rns_work", no, nv, std::max(no, 1LL), batch, bytes);
}

extern "C" int pcg_t3_rns_pack(const double* V, const double* O, const double* t2, long long no,
                               long long nv, void* work, long long work_len, void* stream) {
  T3Plan p;
  if (!t3_operands(V, O, t2, "pcg_t3_rns_pack") ||
      !t3_arguments(p, work, work_len, no, nv, no, 0, "pcg_t3_rns_pack"))
    return -1;
  unsigned char* w = (unsigned char*)work;
  const int rc = t3_scales(p, V, O, t2, w, (cudaStream_t)stream);
  return rc ? rc : t3_pack(p, V, O, t2, kNoFirst, 7, w, (cudaStream_t)stream);
}

extern "C" int pcg_t3_rns_partials_of(const double* V, const double* O, const double* t2,
                                      long long no, long long nv, const int* ijk, int ntrip,
                                      double* P, void* work, long long work_len, void* stream) {
  return partials_entry("pcg_t3_rns_partials_of", V, O, t2, no, nv, no, kNoFirst, ijk, ntrip, P,
                        work, work_len, stream);
}

extern "C" int pcg_t3_rns_partials(long long no, long long nv, const int* ijk, int ntrip, double* P,
                                   void* work, long long work_len, void* stream) {
  T3Plan p;
  const char* who = "pcg_t3_rns_partials";
  if (!t3_batch(ijk, ntrip, P, who) || !t3_arguments(p, work, work_len, no, nv, no, ntrip, who))
    return -1;
  return t3_partials(p, nullptr, nullptr, nullptr, nullptr, ijk, ntrip, P, (unsigned char*)work,
                     (cudaStream_t)stream, who);
}
