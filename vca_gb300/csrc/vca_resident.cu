// vca_resident.cu -- whole Lanczos runs in one launch.
//
// A Lanczos step by separate launches costs eleven of them (product, two
// reductions with their scalar kernels, update, scaling), 25-30 us however
// small the sector.  Where a vector fits shared memory one thread-block
// cluster keeps a run there from its start vector to its last step:
//  * every block holds the whole current vector X of its column (the hops of
//    both spins gather from it) and one more vector of its own rows: the
//    product, then the residual (FP64: on top of the previous vector; fixed
//    point keeps that one in an L2-resident scratch, since its update rounds
//    a x + b x_prev once).  Only the new X crosses to the other blocks of the
//    column, through distributed shared memory;
//  * a thread keeps one fast-index configuration and takes RS_CH slow-index
//    ones at a time: the fast hop word is read once for RS_CH gathers, and a
//    warp's slow hops are the same for (nearly) all its lanes, so those gathers
//    are conflict free.  Rows are taken in order of decreasing hop count,
//    dealt round to the blocks, so that the rows of one pass loop equally
//    long (padding points at a zero row);
//  * the loops over rows stay rolled: a form with all of a thread's rows in
//    registers ran at half the instruction rate, for misses in the
//    instruction cache (48 us a step of the 3x3 cluster's 15,876 states);
//  * the two scalars of a step are summed by warp shuffles, across the
//    cluster by one 16-byte remote store a block, and formed by one lane a
//    block (GB300 FP64: ~64 cycles a warp instruction, so no warp repeats it).
// Fixed point: the arithmetic of vca_fx.cu operation by operation (exact hop
// sums and dot products), so alpha and beta are the same bits as by the
// separate launches.  FP64: real or complex vectors; a hop takes one FMA per
// component, complex amplitudes as a real and an imaginary hop.
// Bound: fixed point by instruction issue (0.4-0.6 a cycle and quarter SM, ~370
// instructions an element and step), FP64 by its pipe (84 % busy).
// Measured, chain stage by separate launches -> resident: 2x2 (4 groups) 5.4 ->
// 0.29 ms, 3x3 200 steps 72 -> 43 ms, BHZ 2x2 200 steps 115 -> 63 ms; search
// stage 2x2 4.0 -> 0.6 ms, 3x3 16.2 -> 8.5 ms, BHZ 15.4 -> 12.3 ms.
#include "vca_resident.cuh"
#include "vca_tri.cuh"

#include <cooperative_groups.h>

namespace vca {

void count_launch_external();

namespace cg = cooperative_groups;
typedef __int128 i128;
typedef unsigned long long u64;

namespace {

#define RS_SMEM_MAX (226 * 1024)
#define RS_MAX_C 8

// round-half-up arithmetic shift (as rshift_round of vca_fx.cu); 1..63 on the
// two words
__device__ __noinline__ i64 rs_shift_any(i128 p, int s) {
  if (s <= 0) return (i64)p;
  p += ((i128)1) << (s - 1);
  return (i64)(p >> s);
}
__device__ __forceinline__ i64 rs_shift(i128 p, int s) {
  if ((unsigned)(s - 1) < 63u) {
    u64 lo = (u64)p, hi = (u64)(p >> 64);
    const u64 r = 1ull << (s - 1);
    lo += r;
    hi += lo < r ? 1ull : 0ull;
    return (i64)((lo >> s) | (hi << (64 - s)));
  }
  return rs_shift_any(p, s);
}
// multiplier and shift of x -> x * f * 2^(so - si) (as k_fx_mult)
__device__ __forceinline__ void rs_mult(double x, int si, int so, i64& mul, int& sh) {
  if (x == 0.0 || !isfinite(x)) { mul = 0; sh = 0; return; }
  const int e = (int)((__double_as_longlong(x) >> 52) & 2047) - 1022;  // frexp's exponent (x normal)
  int E = 60 - e;
  int shift = E + si - so;
  if (shift > 120) { E -= shift - 120; shift = 120; }
  if (shift < 0) { E -= shift; shift = 0; }
  mul = __double2ll_rn(ldexp(x, E));
  sh = shift;
}
__device__ __forceinline__ i64 rs_mixed(const FxView& f, unsigned u, unsigned d) {
  i64 s = f.c0fx;
  for (int o = 0; o < f.norb; o++) s += f.Ufx[o] * (i64)__popc(u & d & f.omask[o]);
  int c = 0;
  for (int o = 0; o < f.norb; o++)
    for (int q = o + 1; q < f.norb; q++)
      c += __popc(u & f.omask[o] & (d >> (q - o))) + __popc(u & f.omask[q] & (d << (q - o)));
  return s + f.Ustfx * (i64)c;
}
__device__ __forceinline__ uint64_t rs_splitmix64(uint64_t x) {
  uint64_t z = x + 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
// rank of an occupied word among the ascending words of its filling
__device__ __forceinline__ int rs_rank(const int* words, int n, unsigned w) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if ((unsigned)words[mid] < w) lo = mid + 1; else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ i128 rs_shfl_sum(i128 v) {
  u64 lo = (u64)v;
  i64 hi = (i64)(v >> 64);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const u64 lo2 = __shfl_xor_sync(0xffffffffu, lo, off);
    const i64 hi2 = __shfl_xor_sync(0xffffffffu, hi, off);
    const u64 sl = lo + lo2;
    hi = hi + hi2 + (sl < lo ? 1 : 0);
    lo = sl;
  }
  return (i128)(((unsigned __int128)(u64)hi << 64) | lo);
}

// what a block's scalar lane leaves for all its threads, and the cluster's
// exchange slots
struct RsShared {
  i128 warp[32];
  i128 part[3][RS_MAX_C];  // [start | alpha | beta^2][block of the cluster]
  i64 a, b, mul;
  int sh, active, done;
  double bnow, norm2, alpha, scale;
};

#define RS_CH 4  // slow rows a thread takes at a time

template <int K, bool CPLX>
struct RsTypes {
  typedef i64 V;     // element
  typedef i128 Acc;  // dot products
};
template <>
struct RsTypes<0, false> {
  typedef double V;
  typedef double Acc;
};
template <>
struct RsTypes<0, true> {
  typedef double2 V;
  typedef double Acc;
};

__device__ __forceinline__ double rs_shfl_sum(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}
__device__ __forceinline__ double rs_total(const RsShared* S, int which, int ncol, int CP, double) {
  double s = 0.0;
  for (int c = 0; c < ncol * CP; c++) s += ((const double*)&S->part[which][c])[0];
  return s;
}
// exact sums per column, scaled by `down`, then over the columns as k_chain_sum
__device__ __forceinline__ double rs_total(const RsShared* S, int which, int ncol, int CP, double down, i128) {
  double s = 0.0;
  for (int c = 0; c < ncol; c++) {
    i128 v = 0;
    for (int q = 0; q < CP; q++) v += S->part[which][c * CP + q];
    const bool neg = v < 0;
    unsigned __int128 u = neg ? (unsigned __int128)(-v) : (unsigned __int128)v;
    const double d = ((double)(u64)(u >> 64) * 18446744073709551616.0 + (double)(u64)u) * down;
    s += neg ? -d : d;
  }
  return s;
}

__device__ __forceinline__ double rs_pow2(int e) { return __longlong_as_double((i64)(1023 + e) << 52); }  // |e| < 1000

__device__ __forceinline__ double rs_re(double a, double b) { return a * b; }
__device__ __forceinline__ double rs_re(double2 a, double2 b) { return fma(a.y, b.y, a.x * b.x); }
__device__ __forceinline__ double rs_axpy(double y, double s, double x) { return fma(-s, x, y); }
__device__ __forceinline__ double2 rs_axpy(double2 y, double s, double2 x) {
  return make_double2(fma(-s, x.x, y.x), fma(-s, x.y, y.y));
}
__device__ __forceinline__ double rs_mulv(double f, double x) { return f * x; }
__device__ __forceinline__ double2 rs_mulv(double f, double2 x) { return make_double2(f * x.x, f * x.y); }
__device__ __forceinline__ double rs_addv(double a, double s, double x) { return fma(s, x, a); }
__device__ __forceinline__ double2 rs_addv(double2 a, double s, double2 x) {
  return make_double2(fma(s, x.x, a.x), fma(s, x.y, a.y));
}
// sign and zero tests on the bits, off the FP64 pipe
__device__ __forceinline__ double rs_negif(double a, bool neg) {
  return __hiloint2double(__double2hiint(a) ^ (neg ? 0x80000000 : 0), __double2loint(a));
}
__device__ __forceinline__ bool rs_zero(double a) { return ((__double2hiint(a) << 1) | __double2loint(a)) == 0; }
// one hop of amplitude a, turned by i when rot is set (ar = -a then, else a)
__device__ __forceinline__ double rs_hop(double acc, double, double a, bool, double x) { return fma(a, x, acc); }
__device__ __forceinline__ double2 rs_hop(double2 acc, double ar, double a, bool rot, double2 x) {
  return make_double2(fma(ar, rot ? x.y : x.x, acc.x), fma(a, rot ? x.x : x.y, acc.y));
}
__device__ __forceinline__ void rs_set(double& x, double re, double) { x = re; }
__device__ __forceinline__ void rs_set(double2& x, double re, double im) { x = make_double2(re, im); }

// Shared-memory layout of a block, the same for the kernel and the host.
struct RsLayout {
  size_t x, y, row, word, cnt, e1, off, amp, ford, ab, w32, bytes;
};
__host__ __device__ __forceinline__ RsLayout rs_layout(int df, int ds, int sp, int wd, int es, bool fx, bool search) {
  RsLayout l;
  size_t b = (sizeof(RsShared) + 15) & ~(size_t)15;
  l.x = b;
  b += (size_t)es * df * (ds + 1);  // and a zero row
  l.y = b;
  b += (size_t)es * df * sp;
  b = (b + 15) & ~(size_t)15;
  l.e1 = b;
  b += 8 * (size_t)sp;  // fixed point: one-body energies; FP64: unused
  l.amp = b;
  if (!fx) b += 8 * (size_t)sp * wd;
  l.off = b;
  b += 4 * (size_t)sp * wd;
  l.row = b;
  b += 4 * (size_t)sp;
  l.word = b;
  b += 4 * (size_t)sp;
  l.cnt = b;
  b += 8 * (size_t)sp;  // hops, and negative hops per class (4 x 8 bits)
  l.ford = b;
  if (!fx) b += 4 * (size_t)df;
  b = (b + 15) & ~(size_t)15;
  l.ab = b;
  l.w32 = b;
  if (search) {
    b += 8 * (2 * RS_NMAX + 2);
    l.w32 = b;
    b += sizeof(float2) * 2 * TRI_MAX;
  }
  l.bytes = b;
  return l;
}
// padded slow hop width: FP64 complex hops may take two entries
__host__ __device__ __forceinline__ int rs_width(int wd, int split) { return (wd * split + 1) & ~1; }

// place of row r among n rows by decreasing count (stable)
__device__ __forceinline__ int rs_order(const int* cnt, int n, int r) {
  const int c = cnt[r];
  int q = 0;
  for (int i = 0; i < n; i++) {
    const int d = cnt[i];
    q += d > c || (d == c && i < r);
  }
  return q;
}

// sum over the block, to slot `which` of every block of the cluster; returns
// after the cluster (C > 1) has met; with C == 1 warp 0 alone holds it
template <typename Acc>
__device__ __forceinline__ void rs_reduce(cg::cluster_group& cl, RsShared* S, Acc v, int which, int C, int rank) {
  v = rs_shfl_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (lane == 0) ((Acc*)S->warp)[warp] = v;
  __syncthreads();
  if (warp == 0) {
    Acc s = lane < nw ? ((Acc*)S->warp)[lane] : (Acc)0;
    s = rs_shfl_sum(s);
    if (lane < C) {
      RsShared* R = C > 1 ? cl.map_shared_rank(S, lane) : S;
      *(Acc*)&R->part[which][rank] = s;
    }
  }
  if (C > 1) cl.sync();
}

template <int K, bool CPLX, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT <= 256 ? 2 : 1) k_rs(RsParams P) {
  constexpr bool FX = K > 0;
  constexpr int KA = FX ? K : 1;
  typedef typename RsTypes<K, CPLX>::V V;
  typedef typename RsTypes<K, CPLX>::Acc Acc;
  extern __shared__ __align__(16) unsigned char rs_sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const RsTask& tk = P.tasks[blockIdx.x / C];
  const RsSpace& sp = P.spaces[tk.space];
  const SectorView& sv = sp.sv;
  const FxView& fv = sp.fv;
  // what the step loop reads of them, out of memory that its stores could alias
  const unsigned* __restrict__ fhop = fv.up_rhop;
  const int* __restrict__ fsrc = sv.up_src;
  const double2* __restrict__ famp = sv.up_amp;
  const bool one = fv.norb == 1;
  const i64 U0 = fv.Ufx[0], c0 = fv.c0fx;
  const unsigned m0sk = fv.omask[0];
  i64 afx[KA];
#pragma unroll
  for (int q = 0; q < KA; q++) afx[q] = fv.afx[q];
  const int fshift = fv.shift;
  const int swap = sp.swap, mode = P.mode;
  const int64_t nat_up = sp.nat_up;
  const int ncol = tk.ncol, CP = C / ncol, col = rank / CP, part = rank % CP;
  const int DF = sv.dimup, DS = sv.dimdw;
  const int SP = (DS + CP - 1) / CP;
  const int ns = (DS - part + CP - 1) / CP;  // own rows: every CP-th of the slow order
  const int WD = rs_width(sv.wdw, P.split);
  const RsLayout L = rs_layout(DF, DS, SP, WD, (int)sizeof(V), FX, P.mode != RS_CHAIN);
  RsShared* S = (RsShared*)rs_sm;
  V* X = (V*)(rs_sm + L.x);
  V* Y = (V*)(rs_sm + L.y);
  i64* es = (i64*)(rs_sm + L.e1);
  double* amps = (double*)(rs_sm + L.amp);
  unsigned* offs = (unsigned*)(rs_sm + L.off);
  int* rows = (int*)(rs_sm + L.row);
  unsigned* wsl = (unsigned*)(rs_sm + L.word);
  int2* cnts = (int2*)(rs_sm + L.cnt);
  int* ford = (int*)(rs_sm + L.ford);
  double* At = (double*)(rs_sm + L.ab);  // a search's alpha, beta
  double* Bs = At + RS_NMAX;
  float2* w32 = (float2*)(rs_sm + L.w32);
  // own rows of x_prev (fixed point) or of the diagonal (FP64), in L2
  i64* scr = P.scratch + (size_t)blockIdx.x * P.scratch_block;
  const FxScales& fs = P.fx;
  const bool search = mode != RS_CHAIN;
  const unsigned ZERO = (unsigned)(DS * DF);  // element offset of the zero row

  if (!FX) {  // rows by decreasing hop count (fixed point: from the tables)
    for (int r = threadIdx.x; r < DF; r += blockDim.x) ford[rs_order(sv.up_cnt, DF, r)] = r;
    for (int r = threadIdx.x; r < DS; r += blockDim.x) {
      const int q = rs_order(sv.dw_cnt, DS, r);
      if (q % CP == part) rows[q / CP] = r;
    }
    __syncthreads();
  }
  // slow tables of the own rows
  for (int j = threadIdx.x; j < ns; j += blockDim.x) {
    const int r = FX ? sp.slow_order[j * CP + part] : rows[j];
    const int n = sv.dw_cnt[r];
    if (FX) rows[j] = r;
    wsl[j] = (unsigned)sv.dw_words[r];
    int m = 0, neg = 0;
    for (int h = 0; h < n; h++) {
      if (FX) {
        const unsigned hw = fv.dw_hop[(size_t)h * DS + r];
        offs[j * WD + m++] = ((hw & 0xFFFFFFu) * (unsigned)DF) | (hw & 0xFF000000u);
        if (hw >> 31) neg += 1 << (8 * ((hw >> 24) & 3u));
      } else {
        const unsigned o = (unsigned)sv.dw_src[(size_t)h * DS + r] * (unsigned)DF;
        const double2 a = sv.dw_amp[(size_t)h * DS + r];
        if (a.x != 0.0 || !CPLX) {
          amps[j * WD + m] = a.x;
          offs[j * WD + m++] = o;
        }
        if (CPLX && a.y != 0.0) {
          amps[j * WD + m] = a.y;
          offs[j * WD + m++] = o | 0x80000000u;
        }
      }
    }
    cnts[j] = make_int2(m, neg);
    for (; m < WD; m++) {
      offs[j * WD + m] = ZERO;
      if (!FX) amps[j * WD + m] = 0.0;
    }
    if (FX) es[j] = fv.dw_e1[r];
  }
  for (int t = threadIdx.x; t < DF; t += blockDim.x) {
    if constexpr (FX) X[ZERO + t] = 0; else rs_set(X[ZERO + t], 0.0, 0.0);
  }
  if (C > 1) cl.sync(); else __syncthreads();  // every block of the cluster is there

  const int G = blockDim.x / DF;
  const int g = threadIdx.x / DF;
  const bool on = g < G;
  int f = threadIdx.x - g * DF;
  const int j0 = on ? g : ns;  // this thread's rows j0, j0 + G, ...
  unsigned wf = 0;
  i64 ef = 0;
  int nu = 0, fnat = f;
  i64 negf[KA];
#pragma unroll
  for (int q = 0; q < KA; q++) negf[q] = 0;
  if (on) {
    if (FX) {  // the fast role in its hop-count order (FxView::up_rhop)
      wf = (unsigned)fv.up_pword[f];
      ef = fv.up_pe1[f];
      nu = fv.up_pcnt[f];
      fnat = fv.up_perm[f];
      for (int h = 0; h < nu; h++) {
        const unsigned hw = fv.up_rhop[(size_t)h * DF + f];
#pragma unroll
        for (int q = 0; q < KA; q++)
          if ((hw >> 31) && (K == 1 || q == (int)((hw >> 24) & 3u))) negf[q]++;
      }
    } else {  // vectors in natural order; lanes take the fast rows by hop count
      f = ford[f];
      fnat = f;
      wf = (unsigned)sv.up_words[f];
      nu = sv.up_cnt[f];
    }
  }
  auto natural = [&](int r) {  // natural index of the element (fast f, slow row r)
    return swap ? (int64_t)r + (int64_t)fnat * nat_up : (int64_t)fnat + (int64_t)r * nat_up;
  };

  // ---- start vector --------------------------------------------------------
  Acc acc = 0;
  for (int j = j0; j < ns; j += G) {
    const int r = rows[j];
    const int iup = sp.swap ? r : fnat, idw = sp.swap ? fnat : r;
    V x;
    if constexpr (FX) x = 0; else rs_set(x, 0.0, 0.0);
    if (search) {
      const uint64_t i = (uint64_t)iup + (uint64_t)idw * (uint64_t)sp.nat_up;
      const uint64_t z = rs_splitmix64(P.seed + 0xD1B54A32D192ED03ull * (uint64_t)tk.isector + i);
      const double d = (double)(z >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
      if constexpr (FX) x = __double2ll_rn(ldexp(d, 40)); else rs_set(x, d, 0.0);
    } else {
      const bool fast = (tk.spin == 0) != (sp.swap != 0);  // the changed spin is the fast index
      const unsigned w = fast ? wf : wsl[j];
      double vr = 0.0, vi = 0.0;
      for (int q = 0; q < tk.nterm; q++) {
        const int pos = tk.pos[q];
        const bool occ = (w >> pos) & 1u;
        if (tk.dag ? !occ : occ) continue;
        const unsigned ws = w ^ (1u << pos);
        const bool neg = __popc(ws & ((1u << pos) - 1u)) & 1;
        const int rs = rs_rank(tk.src_words, tk.src_dim, ws);
        const int64_t si = tk.spin == 0 ? (int64_t)rs + (int64_t)idw * tk.src_dimup
                                        : (int64_t)iup + (int64_t)rs * tk.src_dimup;
        if constexpr (FX) {
          const i64 gv = ((const i64*)tk.gs)[si];
          x += (i64)(col == 0 ? tk.cre[q] : tk.cim[q]) * (neg ? -gv : gv);
        } else {
          double gr, gi = 0.0;
          if constexpr (CPLX) {
            const double2 gv = ((const double2*)tk.gs)[si];
            gr = gv.x;
            gi = gv.y;
          } else {
            gr = ((const double*)tk.gs)[si];
          }
          const double ar = neg ? -tk.cre[q] : tk.cre[q], ai = neg ? -tk.cim[q] : tk.cim[q];
          vr += ar * gr - ai * gi;
          vi += ar * gi + ai * gr;
        }
      }
      if constexpr (!FX) {
        if constexpr (CPLX) x = make_double2(vr, vi); else x = col == 0 ? vr : vi;
      }
    }
    if constexpr (FX) {
      acc += (i128)x * x;
    } else {
      acc += rs_re(x, x);
      // the diagonal of the own elements
      double d = sv.up_e1[f].x + sv.dw_e1[r].x + mixed_diag(P.md, wf, wsl[j]);
      scr[(size_t)j * DF + f] = __double_as_longlong(d);
    }
    Y[j * DF + f] = x;
  }
  rs_reduce(cl, S, acc, 0, C, rank);
  if (threadIdx.x == 0) {
    double n2;
    if constexpr (FX) n2 = rs_total(S, 0, ncol, CP, rs_pow2(search ? -80 : -2 * fs.F), (i128)0);
    else n2 = rs_total(S, 0, ncol, CP, 1.0);
    const double inv = n2 > 0.0 ? 1.0 / sqrt(n2) : 0.0;
    S->norm2 = n2;
    S->active = n2 > 0.0 ? 1 : 0;
    S->bnow = 0.0;
    S->b = 0;
    if (FX) rs_mult(inv, search ? 40 : fs.F, fs.F, S->mul, S->sh);
    S->scale = inv;
  }
  __syncthreads();
  int len = 0;
  bool live = S->active != 0;
  // X <- Y scaled, own rows here and in the column's other blocks; the old X
  // is kept for the next step
  auto spread = [&](bool keep) {
    const i64 mul = S->mul;
    const int sh = S->sh;
    const double f64 = S->scale;
#pragma unroll 2
    for (int j = j0; j < ns; j += G) {
      const int at = rows[j] * DF + f, o = j * DF + f;
      const V old = X[at];
      V xn;
      if constexpr (FX) {
        xn = rs_shift((i128)mul * Y[o], sh);
        if (keep) __stcg((long long*)scr + o, (long long)old);
      } else {
        xn = rs_mulv(f64, Y[o]);
        if (keep) Y[o] = old;
      }
      X[at] = xn;
      for (int q = 1; q < CP; q++) cl.map_shared_rank(X, col * CP + (part + q) % CP)[at] = xn;
    }
    if (C > 1) cl.sync(); else __syncthreads();
  };
  if (live) spread(false);

  const int last = mode == RS_VECTOR ? *tk.mconv : tk.nlanc;
  if (mode == RS_VECTOR) {  // Ritz coefficients of the search's tridiagonal
    if (rank == 0 && threadIdx.x < 32) {
      for (int j = threadIdx.x; j < last; j += 32) {
        At[j] = tk.svec[5 * RS_NMAX + j];
        Bs[j] = tk.svec[6 * RS_NMAX + j];
      }
      __syncwarp();
      if (last > 1) tri_invit(At, Bs, last, tk.theta[0], tk.svec);
      else if (threadIdx.x == 0) tk.svec[0] = 1.0;
      __threadfence();
    }
    if (C > 1) cl.sync(); else __syncthreads();
  }
  for (int k = 1; live && k <= last; k++) {
    if (mode == RS_VECTOR) {  // psi += s_k x
      const double sk = __ldcg(tk.svec + k - 1);
      V* psi = (V*)tk.psi;
      for (int j = j0; j < ns; j += G) {
        const int r = rows[j];
        const V x = X[r * DF + f];
        V& p = psi[natural(r)];
        if constexpr (FX) p += rs_shift((i128)__double2ll_rn(ldexp(sk, 61)) * x, 61);
        else p = rs_addv(p, sk, x);
      }
      if (k == last) break;
    }
    // ---- y = H x of the own rows (FP64: - b x_prev), <x, y> -----------------
    acc = 0;
    const double bprev = S->bnow;
    for (int jc = j0; jc < ns; jc += RS_CH * G) {
      unsigned ro[RS_CH];  // element offsets of the rows; past the end: the zero row
      const unsigned* tr[RS_CH];
#pragma unroll
      for (int i = 0; i < RS_CH; i++) {
        const int j = jc + i * G;
        const bool in = j < ns;
        ro[i] = in ? (unsigned)(rows[j] * DF) : ZERO;
        tr[i] = offs + (in ? j : jc) * WD;
      }
      const V* Xf = X + f;
      if constexpr (FX) {
        i64 hs[KA][RS_CH];
#pragma unroll
        for (int i = 0; i < RS_CH; i++) {
          const int ng = cnts[jc + i * G < ns ? jc + i * G : jc].y;
#pragma unroll
          for (int q = 0; q < KA; q++) hs[q][i] = negf[q] + ((ng >> (8 * q)) & 255);
        }
        // -v = ~v + 1: the complements here, the ones above
        for (int h = 0; h < nu; h++) {
          const unsigned hw = fhop[h * DF + f];
          const V* xb = X + (hw & 0xFFFFFFu);
          const i64 m = (i64)((int)hw >> 31);
          const int cls = (int)((hw >> 24) & 3u);
#pragma unroll
          for (int i = 0; i < RS_CH; i++) {
            const i64 xv = xb[ro[i]] ^ m;
#pragma unroll
            for (int q = 0; q < KA; q++) hs[q][i] += (K == 1 || q == cls) ? xv : 0;
          }
        }
        const int nd = cnts[jc].x;  // the most of these rows
        for (int h = 0; h < nd; h += 2) {
#pragma unroll
          for (int i = 0; i < RS_CH; i++) {
            const uint2 t2 = *(const uint2*)(tr[i] + h);
            const i64 m0 = (i64)((int)t2.x >> 31), m1 = (i64)((int)t2.y >> 31);
            const i64 x0 = Xf[t2.x & 0xFFFFFFu] ^ m0, x1 = Xf[t2.y & 0xFFFFFFu] ^ m1;
#pragma unroll
            for (int q = 0; q < KA; q++) {
              if (K == 1) {
                hs[q][i] += x0 + x1;
              } else {
                if (q == (int)((t2.x >> 24) & 3u)) hs[q][i] += x0;
                if (q == (int)((t2.y >> 24) & 3u)) hs[q][i] += x1;
              }
            }
          }
        }
#pragma unroll
        for (int i = 0; i < RS_CH; i++) {
          const int j = jc + i * G;
          if (j >= ns) break;
          const i64 x = Xf[ro[i]];
          const unsigned ws = wsl[j];
          const i64 d = ef + es[j] + (one ? c0 + U0 * (i64)__popc(wf & ws & m0sk) : rs_mixed(fv, wf, ws));
          i128 p = (i128)d * x;
#pragma unroll
          for (int q = 0; q < KA; q++) p += (i128)afx[q] * hs[q][i];
          const i64 y = rs_shift(p, fshift);
          Y[j * DF + f] = y;
          acc += (i128)x * y;
        }
      } else {
        V hs[RS_CH];
#pragma unroll
        for (int i = 0; i < RS_CH; i++) {
          const int j = jc + i * G;
          const V x = Xf[ro[i]];
          const double d = j < ns ? __longlong_as_double(__ldcg((const long long*)scr + (size_t)j * DF + f)) : 0.0;
          hs[i] = rs_mulv(d, x);
          if (CPLX && P.diag_im) {
            const double e = j < ns ? sv.up_e1[f].y + sv.dw_e1[rows[j]].y : 0.0;
            hs[i] = rs_hop(hs[i], -e, e, true, x);
          }
        }
        for (int h = 0; h < nu; h++) {
          const V* xb = X + fsrc[h * DF + f];
          const double2 a = famp[h * DF + f];
          const bool rot = CPLX && rs_zero(a.x);
          const double s = rot ? a.y : a.x, sr = rs_negif(s, rot);
#pragma unroll
          for (int i = 0; i < RS_CH; i++) hs[i] = rs_hop(hs[i], sr, s, rot, xb[ro[i]]);
          if (CPLX && P.split > 1 && !rot && !rs_zero(a.y)) {
#pragma unroll
            for (int i = 0; i < RS_CH; i++) hs[i] = rs_hop(hs[i], -a.y, a.y, true, xb[ro[i]]);
          }
        }
#pragma unroll
        for (int i = 0; i < RS_CH; i++) {
          const int j = jc + i * G;
          if (j >= ns) break;
          const int nd = cnts[j].x;
          const double* ta = amps + (size_t)j * WD;
#pragma unroll 2
          for (int h = 0; h < nd; h++) {
            const unsigned o = tr[i][h];
            const bool rot = CPLX && (o >> 31);
            hs[i] = rs_hop(hs[i], rs_negif(ta[h], rot), ta[h], rot, Xf[o & 0x7FFFFFFFu]);
          }
          const int at = j * DF + f;
          if (k > 1) hs[i] = rs_axpy(hs[i], bprev, Y[at]);
          Y[at] = hs[i];
          acc += rs_re(Xf[ro[i]], hs[i]);
        }
      }
    }
    rs_reduce(cl, S, acc, 1, C, rank);
    double alpha = 0.0;  // of the scalar lane
    if (threadIdx.x == 0) {
      if constexpr (FX) {
        alpha = rs_total(S, 1, ncol, CP, rs_pow2(-(fs.F + fs.G)), (i128)0);
        S->a = __double2ll_rn(alpha * rs_pow2(fs.C));
      } else {
        alpha = rs_total(S, 1, ncol, CP, 1.0);
        S->alpha = alpha;
      }
    }
    __syncthreads();
    // ---- w = y - a x (fixed point: - b x_prev) ------------------------------
    acc = 0;
    if constexpr (FX) {
      const i64 a = S->a, b = S->b;
      const int sh = fs.C + fs.F - fs.G;
#pragma unroll 2
      for (int j = j0; j < ns; j += G) {
        const int o = j * DF + f;
        i128 p = (i128)a * X[rows[j] * DF + f];
        if (k > 1) p += (i128)b * (i64)__ldcg((const long long*)scr + o);
        const i64 w = Y[o] - rs_shift(p, sh);
        Y[o] = w;
        acc += (i128)w * w;
      }
    } else {
      const double a = S->alpha;
#pragma unroll 2
      for (int j = j0; j < ns; j += G) {
        const int o = j * DF + f;
        const V w = rs_axpy(Y[o], a, X[rows[j] * DF + f]);
        Y[o] = w;
        acc += rs_re(w, w);
      }
    }
    rs_reduce(cl, S, acc, 2, C, rank);
    if (threadIdx.x == 0) {  // as k_lanczos_record
      double b2;
      if constexpr (FX) b2 = rs_total(S, 2, ncol, CP, rs_pow2(-2 * fs.G), (i128)0);
      else b2 = rs_total(S, 2, ncol, CP, 1.0);
      const double b = sqrt(fmax(b2, 0.0));
      double invb = 0.0;
      int act = 1;
      if (b < P.beta_tol) {
        act = 0;
      } else {
        if (k >= tk.nlanc) act = 0;
        invb = 1.0 / b;
      }
      if (FX) rs_mult(invb, fs.G, fs.F, S->mul, S->sh);
      S->scale = invb;
      S->active = mode == RS_VECTOR ? 1 : act;  // the vector pass repeats the search's steps
      S->bnow = b;
      if (FX) S->b = __double2ll_rn(b * rs_pow2(fs.C));
      const bool more = b >= P.beta_tol && k < tk.nlanc;
      if (mode == RS_CHAIN) {
        if (rank == 0) {
          P.cs.A[(size_t)tk.store * P.cs.ld + k - 1] = alpha;
          if (more) P.cs.B[(size_t)tk.store * P.cs.ld + k] = b;
        }
      } else if (mode == RS_SEARCH) {
        At[k - 1] = alpha;
        if (more) Bs[k] = b;
      }
    }
    __syncthreads();
    len = k;
    live = S->active != 0;
    if (mode == RS_SEARCH && (!live || k % P.check_every == 0)) {
      if (rank == 0 && threadIdx.x < 32) {
        double* th = tk.theta;
        const bool full = warp_tri_lowest(At, Bs, k, S->bnow, P.resid_tol, !live, false, w32, th, tk.svec, th + 1);
        const bool stop = full && (!live || th[1] <= P.resid_tol * fmax(1.0, fabs(th[0])));
        if (stop)
          for (int j = threadIdx.x; j < k; j += 32) {  // for the vector pass
            tk.svec[5 * RS_NMAX + j] = At[j];
            tk.svec[6 * RS_NMAX + j] = j ? Bs[j] : 0.0;
          }
        if (threadIdx.x == 0) {
          if (stop) *tk.mconv = k;
          for (int q = 0; q < C; q++) (C > 1 ? cl.map_shared_rank(S, q) : S)->done = stop ? 1 : 0;
        }
      }
      if (C > 1) cl.sync(); else __syncthreads();
      if (S->done) break;
    }
    if (!live) break;
    spread(true);
  }
  if (mode == RS_CHAIN) {
    if (rank == 0) {
      for (int j = len + threadIdx.x; j < P.cs.ld; j += blockDim.x) {
        P.cs.A[(size_t)tk.store * P.cs.ld + j] = 0.0;
        P.cs.B[(size_t)tk.store * P.cs.ld + j] = 0.0;
      }
      if (threadIdx.x == 0) {
        P.cs.B[(size_t)tk.store * P.cs.ld] = 0.0;
        P.cs.n[tk.store] = len;
        P.cs.pes[tk.store] = S->norm2 * tk.boltz / tk.zeta;
        P.cs.isign[tk.store] = tk.isign;
        P.cs.wfac[tk.store] = tk.wfac;
        P.cs.Ei[tk.store] = tk.Ei;
      }
    }
  } else if (mode == RS_SEARCH) {
    if (len == 0 && rank == 0 && threadIdx.x == 0) {  // zero start vector
      tk.theta[0] = INFINITY;
      *tk.mconv = 0;
    }
  } else {  // psi to unit norm
    V* psi = (V*)tk.psi;
    acc = 0;
    for (int j = j0; j < ns; j += G) {
      const V p = psi[natural(rows[j])];
      if constexpr (FX) acc += (i128)p * p; else acc += rs_re(p, p);
    }
    __syncthreads();
    rs_reduce(cl, S, acc, 0, C, rank);
    if (threadIdx.x == 0) {
      double n2;
      if constexpr (FX) n2 = rs_total(S, 0, ncol, CP, rs_pow2(-2 * fs.F), (i128)0);
      else n2 = rs_total(S, 0, ncol, CP, 1.0);
      const double inv = n2 > 0.0 ? 1.0 / sqrt(n2) : 0.0;
      if (FX) rs_mult(inv, fs.F, fs.F, S->mul, S->sh);
      S->scale = inv;
    }
    __syncthreads();
    for (int j = j0; j < ns; j += G) {
      V& p = psi[natural(rows[j])];
      if constexpr (FX) p = rs_shift((i128)S->mul * p, S->sh);
      else p = rs_mulv(S->scale, p);
    }
  }
  if (C > 1) cl.sync();  // no block leaves while another may write to it
}

template <int K, bool CPLX, int MAXT>
int rs_go(const RsParams& p, int ntask, const RsShape& s, cudaStream_t st) {
  static bool set = false;  // per instantiation, process-wide (every device is sm_103a)
  if (!set) {
    if (cudaFuncSetAttribute(k_rs<K, CPLX, MAXT>, cudaFuncAttributeMaxDynamicSharedMemorySize, RS_SMEM_MAX) !=
        cudaSuccess)
      return 1;
    set = true;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(ntask * s.C));
  cfg.blockDim = dim3((unsigned)s.T);
  cfg.dynamicSmemBytes = s.smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)s.C;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_rs<K, CPLX, MAXT>, p) == cudaSuccess ? 0 : 1;
}
template <int K, bool CPLX>
int rs_go_t(const RsParams& p, int ntask, const RsShape& s, cudaStream_t st) {
  if (s.T <= 256) return rs_go<K, CPLX, 256>(p, ntask, s, st);
  return s.T <= 512 ? rs_go<K, CPLX, 512>(p, ntask, s, st) : rs_go<K, CPLX, 1024>(p, ntask, s, st);
}

}  // namespace

// Cluster size: the one of 1, 2, 4 and 8 blocks, among those that are a multiple
// of every task's columns and whose blocks' shared memory holds their tasks,
// with the least estimated time.  A block's step costs its elements plus a
// fixed part (reductions, scalars, meeting points) worth about RS_FIXED
// elements; blocks that fit twice on an SM hide one another's fixed part (a
// quarter more work a second); the end of the launch costs half a block.
// Large clusters win when tasks are few (a search), small ones when many.
// Block size: the smallest of 64 .. 512 threads (256 where two blocks share an
// SM) that takes each task's rows in one pass, more where a fast dimension
// needs more.
RsShape rs_shape(const RsDims* dims, size_t n, int es, bool fx, int split, bool search) {
  const double RS_FIXED = 1000.0, SMS = 152.0;
  RsShape best;
  double tbest = 0.0;
  for (int C = 1; n && C <= RS_MAX_C; C *= 2) {
    RsShape s;
    s.C = C;
    bool ok = true;
    double work = 0.0, longest = 0.0;
    for (size_t i = 0; i < n && ok; i++) {
      const RsDims& d = dims[i];
      if (C % d.ncol || d.df > 1024) { ok = false; break; }
      const int CP = C / d.ncol, sp = (d.ds + CP - 1) / CP;
      s.smem = std::max(s.smem, rs_layout(d.df, d.ds, sp, rs_width(d.wd, split), es, fx, search).bytes);
      s.own = std::max(s.own, (size_t)d.df * sp);
      const double block = (double)d.df * sp + RS_FIXED;
      work += block * C * d.count;
      longest = std::max(longest, block);
    }
    if (!ok || s.smem > RS_SMEM_MAX) continue;
    const bool two = s.smem <= RS_SMEM_MAX / 2;
    s.T = 64;
    for (size_t i = 0; i < n; i++) {
      const RsDims& d = dims[i];
      const int CP = C / d.ncol, sp = (d.ds + CP - 1) / CP;
      while (s.T < d.df || (s.T < (two ? 256 : 512) && (int64_t)s.T * RS_CH < (int64_t)d.df * sp)) s.T *= 2;
    }
    const double speed = two && s.T <= 256 ? 1.25 : 1.0;
    if (speed > 1.0) longest *= 2.0 / speed;
    const double t = std::max(longest, work / (SMS * speed) + 0.5 * longest);
    if (!best.C || t < tbest) {
      best = s;
      tbest = t;
    }
  }
  return best;
}

int rs_launch(const RsParams& p, int ntask, const RsShape& s, int K, bool cplx, cudaStream_t st) {
  if (ntask <= 0) return 0;
  count_launch_external();
  if (K == 1) return rs_go_t<1, false>(p, ntask, s, st);
  if (K == 2) return rs_go_t<2, false>(p, ntask, s, st);
  return cplx ? rs_go_t<0, true>(p, ntask, s, st) : rs_go_t<0, false>(p, ntask, s, st);
}

}  // namespace vca
