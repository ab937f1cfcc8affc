// FP64 column kernels: the evaluation of FP64 contexts and the derivative
// products, on the search and the block walk of pmb200_columns.cuh -- clusters
// of 8 atoms against blocks of 32 staged atoms, each pair once.  The search and
// the pair masks are the mixed kernels' (fractions, FP32 box tests with a
// margin); positions, pair arithmetic and sums are FP64.
//
// Sums: each lane's i terms in registers (added over the lane groups in a fixed
// order), j terms travelling with the walk; both reach acc[8][n] (by rank,
// rows hi x, hi y, hi z, hi q, lo x, lo y, lo z, lo q) as the exact two-word
// fixed point of fix2_add, so the results are bitwise reproducible.
#pragma once
#include "pmb200_columns.cuh"

namespace pmb200 {

// Staged entries: {x, y} and {z, q} FP64 in arrays of their own (16 bytes an entry:
// no bank conflicts), {meta, rank} (8), for products the direction {x, y}, {z, 0};
// meta: type | pair mask << 16 | modified mask << 24.
template <bool kW>
struct ColLayout64 {
  static constexpr unsigned half = 16 * kColCap;  // {x, y} to {z, q}
  static constexpr unsigned pos = 0, mg = 2 * half, w = mg + 8 * kColCap,
                            mol = w + (kW ? 2 * half : 0), runs = mol + 32,
                            bytes = (runs + 256 + 511) / 512 * 512;
};

__device__ __forceinline__ double2 lds2d(unsigned a) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts2d(unsigned a, double x, double y) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(x), "d"(y) : "memory");
}

// v into word q (0..3) of the atom of rank r (fix2_add's split)
__device__ __forceinline__ void fix2_add_rank(unsigned long long *__restrict__ acc, size_t n, int r,
                                              int q, double v, int *__restrict__ err) {
  if (v == 0.0) return;
  if (!(fabs(v) < kFix2Max)) {
    atomicOr(err, 2);
    return;
  }
  const double s = v * kFix2Hi;
  const double h = rint(s);
  atomicAdd(&acc[q * n + r], (unsigned long long)(long long)h);
  atomicAdd(&acc[(4 + q) * n + r], (unsigned long long)__double2ll_rn((s - h) * kFix2Lo));
}

// 1/sqrt(x) from the FP32 approximation y and one Halley step, y (1 + e/2 + 3 e^2/8)
// with e = 1 - x y^2: e is about 2e-7, what is left out e^3 < 1e-20, so only the
// step's roundings remain (about one unit in the last place).  x in FP32's range.
__device__ __forceinline__ double col_rsqrt64(double x) {
  const double y = (double)col_rsqrt((float)x);
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// The walk common to both kernels.  Pair: a functor with
//   pair(front, a16, a8)   this lane's atom against the entry there
//   start()                zero the j terms
//   shift(to)              the j terms moved to the lane `to` away
//   join(to)               the j terms of the lane `to` away added
//   finish(a8)             the j terms (whole) added to the entry's atom
template <bool kW, bool kSplit, class Pair>
struct ColWalk64 {
  using Lay = ColLayout64<kW>;
  unsigned sb;
  Pair &pair;
  int nl = 0, nn = 0;  // staged entries from the front, from the back

  // half: the block's first 16 entries, four per lane group -- two lanes then
  // meet one entry, each with its own part of the j terms, and four steps are
  // enough (3% of the derivative kernels' time; the mixed kernel, with shorter
  // steps, lost as much to the choice as it gained)
  template <class Tag>
  __device__ __forceinline__ void block(Tag tag, int e0, bool half) {
    const int lane = threadIdx.x & 31;
    const unsigned e = (unsigned)(e0 + (half ? 4 * (lane >> 3) + (lane & 3) : lane));
    unsigned a16 = sb + Lay::pos + 16 * e, a8 = sb + Lay::mg + 8 * e;
    pair.start();
#pragma unroll 1
    for (int h = half ? 2 : 0; h < 4; h++) {
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const unsigned to = k == 0 ? 1u : ((h & 1) && !half ? 7u : 3u);
        pair(tag, a16, a8);
        pair.shift((int)to);
        a16 ^= to << 4;
        a8 ^= to << 3;
      }
    }
    if (half) pair.join(4);
    if (!half || !(lane & 4)) pair.finish(a8);
  }
  // (what a flush moves and what it overwrites lie apart, see col_task)
  __device__ __forceinline__ void copy(int from, int to) {
    for (unsigned h = 0; h <= Lay::half; h += Lay::half) {
      const double2 d = lds2d(sb + Lay::pos + 16 * from + h);
      sts2d(sb + Lay::pos + 16 * to + h, d.x, d.y);
      if (kW) {
        const double2 v = lds2d(sb + Lay::w + 16 * from + h);
        sts2d(sb + Lay::w + 16 * to + h, v.x, v.y);
      }
    }
    const int2 m = lds2(sb + Lay::mg + 8 * from);
    sts2(sb + Lay::mg + 8 * to, m.x, m.y);
  }
  // whole blocks evaluated, the rest kept (last: all, the back's rest and then
  // filler behind the front entries)
  __device__ __forceinline__ void flush(bool last) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    const int bn = kSplit ? nn & ~(kColBlk - 1) : 0;
    if (kSplit)
      for (int t = 0; t < bn; t += kColBlk) block(std::false_type{}, kColCap - kColBlk - t, false);
    const int r = nn - bn;
    int fn = nl & ~(kColBlk - 1);
    if (last) {
      if (lane < r) copy(kColCap - 1 - (bn + lane), nl + lane);
      nl += r;
      fn = (nl + kColBlk - 1) & ~(kColBlk - 1);
      if (nl + lane < fn) {
        const int e = nl + lane;
        for (unsigned h = 0; h <= Lay::half; h += Lay::half) {
          sts2d(sb + Lay::pos + 16 * e + h, 0.0, 0.0);
          if (kW) sts2d(sb + Lay::w + 16 * e + h, 0.0, 0.0);
        }
        sts2(sb + Lay::mg + 8 * e, 0, 0);
      }
      __syncwarp();
    }
    for (int t = 0; t < fn; t += kColBlk) block(std::true_type{}, t, last && nl - t <= 16);
    __syncwarp();
    if (last) {
      nl = nn = 0;
    } else {
      const int rf = nl - fn;
      if (bn > 0 && lane < r) copy(kColCap - 1 - (bn + lane), kColCap - 1 - lane);
      if (fn > 0 && lane < rf) copy(fn + lane, lane);
      nn = r;
      nl = rf;
    }
    __syncwarp();
  }
};

// The cluster's atoms, one per lane and lane group, and its search.
struct ColAtom64 {
  int4 m;           // smeta (atom -1: none)
  double4 p;        // wrapped position, charge
  unsigned bit;     // this lane's bit of an entry's pair mask
  bool wrap;        // pairs take their own minimum image
  ColBox box;
  ColExcl excl;
};
__device__ __forceinline__ ColAtom64 col_atom64(const ColGrid &g, const ColArrays &A, int cl,
                                                unsigned smol) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, ia = lane & (kColI - 1);
  const size_t at = (size_t)cl * kColI + ia;
  ColAtom64 a;
  a.m = A.smeta[at];
  const int4 p0 = A.spos[at];
  const bool active = a.m.z >= 0;
  int4 pi = p0;
  const int4 first = make_int4(__shfl_sync(full, p0.x, 0), __shfl_sync(full, p0.y, 0),
                               __shfl_sync(full, p0.z, 0), 0);
  if (!active) pi = first;
  a.p = A.spos64[active ? at : (size_t)cl * kColI];
  a.bit = active ? 0x10000u << ia : 0u;
  a.excl = col_exclusions(lane, a.m.z, A.ex_start, A.ex);
  a.box = col_box(g, pi);
  // an atom within the cutoff of the box has one image for all of the cluster
  // where the cutoff and the box's half extent fit half the edge
  a.wrap = a.box.hx > g.hmax[0] || a.box.hy > g.hmax[1] || a.box.hz > g.hmax[2];
  __syncwarp();
  if (lane < kColI) sts1(smol + 4 * lane, active ? a.m.y : -2);
  __syncwarp();
  return a;
}

// The edge multiple that brings fraction p (of a staged atom) to the image
// nearest the cluster's centre c: its unsigned difference against the signed one.
__device__ __forceinline__ double col_image(unsigned p, unsigned c, double edge) {
  const int d = (int)(p - c);
  return d < 0 ? (p > c ? -edge : 0.0) : (p < c ? edge : 0.0);
}

// What staging reads of a slot.
template <bool kW>
struct ColSlot64 {
  double4 p, w;
};

// The search with FP64 staging: positions moved to the cluster's image (or, in
// wrap clusters, as they are).
template <bool kW, bool kSplit, class Walk>
__device__ __forceinline__ void col_search64(const ColGrid &g, const ColArrays &A,
                                             const ColAtom64 &a, int cl, int part0, int pstride,
                                             Walk &walk) {
  using Lay = ColLayout64<kW>;
  const unsigned sb = walk.sb, full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  col_search(
      g, A, a.box, a.excl, a.m.z, sb + Lay::mol, sb + Lay::runs, cl, part0, pstride,
      [&](int slot, bool valid) {
        ColSlot64<kW> x{};
        if (valid) {
          x.p = A.spos64[slot];
          if (kW) x.w = A.w[slot];
        }
        return x;
      },
      [&](bool keep, const int4 &p, const int4 &m, const int2 &pmask, const ColSlot64<kW> &x,
          bool last) {
        const bool front = !kSplit || (m.x & 0x10000);
        const unsigned kf = __ballot_sync(full, keep && front);
        const unsigned kb = __ballot_sync(full, keep && !front);
        if (keep) {
          const unsigned below = (1u << lane) - 1u;
          const int e = front ? walk.nl + __popc(kf & below)
                              : kColCap - 1 - (walk.nn + __popc(kb & below));
          double3 s = make_double3(0.0, 0.0, 0.0);
          if (!a.wrap)
            s = make_double3(col_image((unsigned)p.x, a.box.xc, g.edge[0]),
                             col_image((unsigned)p.y, a.box.yc, g.edge[1]),
                             col_image((unsigned)p.z, a.box.zc, g.edge[2]));
          sts2d(sb + Lay::pos + 16 * e, x.p.x + s.x, x.p.y + s.y);
          sts2d(sb + Lay::pos + 16 * e + Lay::half, x.p.z + s.z, x.p.w);
          if (kW) {
            sts2d(sb + Lay::w + 16 * e, x.w.x, x.w.y);
            sts2d(sb + Lay::w + 16 * e + Lay::half, x.w.z, 0.0);
          }
          sts2(sb + Lay::mg + 8 * e, (m.x & 0xfff) | (pmask.x << 16) | (pmask.y << 24), m.w);
        }
        walk.nl += __popc(kf);
        walk.nn += __popc(kb);
        bool fuller;  // (see col_task)
        do {
          fuller = walk.nl + walk.nn > kColCap - 32;
          if (fuller || last) walk.flush(last && !fuller);
        } while (fuller && last);
      });
}

// The difference staged - own at the pair's image, and its square.
__device__ __forceinline__ double col_diff64(const ColGrid &g, const ColAtom64 &a, double x,
                                             double y, double z, double d[3]) {
  d[0] = x - a.p.x;
  d[1] = y - a.p.y;
  d[2] = z - a.p.z;
  if (a.wrap) {
#pragma unroll
    for (int k = 0; k < 3; k++) d[k] = fma(-g.edge[k], rint(d[k] * g.inv[k]), d[k]);
  }
  return fma(d[0], d[0], fma(d[1], d[1], d[2] * d[2]));
}

// ---------------------------------------------------------------------------
// Evaluation.
// ---------------------------------------------------------------------------
// Cutoff form: one reciprocal square root serves 1/r^2 and the Coulomb terms,
// E S = q q (1/r - 1.5/rc + 0.5 r^2/rc^3) and F S - E dS over r = q q (1/r^3 -
// 1/rc^3); the other forms take fp64_pair.  kFull: both switches end at the
// cutoff and no pair is modified.
template <int kForm, bool kEnergy, bool kFull>
struct ColPair64 {
  const ColGrid &g;
  const Fp64Consts &mc;
  const ColArrays &A;
  const ColAtom64 &a;
  const double4 *lj;  // [ntypes^2] from this atom's row on
  int ti;
  unsigned long long *acc;
  double fx = 0, fy = 0, fz = 0, eL = 0, eC = 0;  // eC: per unit of this atom's charge
  int np = 0;
  double jx, jy, jz;

  __device__ __forceinline__ void start() { jx = jy = jz = 0.0; }
  template <class Tag>
  __device__ __forceinline__ void operator()(Tag, unsigned a16, unsigned a8) {
    constexpr bool kLj = Tag::value;
    const double2 d0 = lds2d(a16), d1 = lds2d(a16 + ColLayout64<false>::half);
    const int mj = lds1(a8);
    double d[3];
    double r2 = col_diff64(g, a, d0.x, d0.y, d1.x, d);
    const bool ok = (mj & a.bit) && r2 <= mc.cut2;
    const int ia = threadIdx.x & (kColI - 1);
    const int kind = kFull ? 0 : (mj >> (24 + ia)) & 1;
    double f = 0.0;
    if constexpr (kForm == FORM_CUTOFF) {
      r2 = ok ? r2 : 1.0;
      double qj = ok ? d1.y : 0.0;
      if (!kFull) qj *= kind ? mc.csf : 1.0;
      const double ir = col_rsqrt64(r2), is = ir * ir;
      f = a.p.w * qj * fma(is, ir, -2.0 * mc.c05_3);
      double e = fma(mc.c05_3, r2, ir - mc.c15_1);
      if (!kFull) {
        const bool in = r2 <= mc.rcc2;
        f = in ? f : 0.0;
        e = in ? e : 0.0;
      }
      if (kEnergy) eC = fma(qj, e, eC);
      if (kLj) {
        const double4 p = lj[mj & 0xffff];
        double Aij = kind ? p.z : p.x, Bij = kind ? p.w : p.y;
        Aij = ok ? Aij : 0.0;
        Bij = ok ? Bij : 0.0;
        const double i6 = is * is * is;
        const double t = Aij * i6;
        double el = (t - Bij) * i6;
        // 12 A r^-12 - 6 B r^-6 = 6 (A r^-12 + el)
        double fl = fma(t, i6, el) * (6.0 * is);
        if (!kFull && r2 > mc.rclj2) {
          el = 0.0;
          fl = 0.0;
        } else if (r2 >= mc.ron2) {
          const double c2 = mc.rclj2 - r2;
          const double c4 = c2 * fma(2.0, r2, mc.s2);
          fl = fma(fl, mc.s1 * (c2 * c4), -el * (mc.s3 * fma(c2, c2, -c4)));
          el *= mc.s1 * (c2 * c4);
        }
        f += fl;
        if (kEnergy) eL += el;
      }
      if (kEnergy) np += ok ? 1 : 0;
    } else {
      if (ok) {
        double e1, e2;
        fp64_pair<kForm>(mc, lj - ti, ti, mj & 0xffff, kind, r2, a.p.w, d1.y, f, e1, e2);
        if (kEnergy) {
          eL += e1;
          eC += e2;
          np++;
        }
      }
    }
    fx = fma(-d[0], f, fx);
    fy = fma(-d[1], f, fy);
    fz = fma(-d[2], f, fz);
    jx = fma(d[0], f, jx);
    jy = fma(d[1], f, jy);
    jz = fma(d[2], f, jz);
  }
  __device__ __forceinline__ void shift(int to) {
    jx = __shfl_xor_sync(0xffffffffu, jx, to);
    jy = __shfl_xor_sync(0xffffffffu, jy, to);
    jz = __shfl_xor_sync(0xffffffffu, jz, to);
  }
  __device__ __forceinline__ void join(int to) {
    jx += __shfl_xor_sync(0xffffffffu, jx, to);
    jy += __shfl_xor_sync(0xffffffffu, jy, to);
    jz += __shfl_xor_sync(0xffffffffu, jz, to);
  }
  __device__ __forceinline__ void finish(unsigned a8) {
    const int r = lds1(a8 + 4);
    fix2_add_rank(acc, A.n, r, 0, jx, A.err);
    fix2_add_rank(acc, A.n, r, 1, jy, A.err);
    fix2_add_rank(acc, A.n, r, 2, jz, A.err);
  }
};

// (41,472 atoms, forces / with energies at 14, 16, 18, 20, 22, 24 blocks: 139 / 148,
// 141 / 149, 129 / 139, 133 / 139, 125 / 133, 125 / 133 us)
#ifndef PMB200_COL64_BLOCKS
#define PMB200_COL64_BLOCKS 20
#endif
// LJ tables up to this size in shared memory (forces of 41,472 atoms with 4, 8, 12
// and 16 types: 145, 148, 150 and 166 us from shared memory, where large tables
// cost residency, 145, 146, 148 and 149 through L1)
constexpr int kCol64LjTypes = 8;

// (launch, clusters and parts as k_col_pair; dynamic shared memory: the entries,
// then the LJ table)
template <int kForm, bool kEnergy, bool kFull>
__global__ void __launch_bounds__(32, PMB200_COL64_BLOCKS)
k_col_pair64(const ColGrid g, const Fp64Consts mc, int ntypes, const double4 *__restrict__ lj64,
             const ColArrays A, unsigned long long *__restrict__ acc,
             const int *__restrict__ ctl, int *__restrict__ count, int lsplit,
             double *__restrict__ partial) {
  constexpr bool kSplit = kForm == FORM_CUTOFF;
  using Lay = ColLayout64<false>;
  extern __shared__ __align__(512) unsigned char s_cdyn[];
  const int lane = threadIdx.x;
  const double4 *lj = lj64;
  if (ntypes <= kCol64LjTypes) {
    double4 *s_lj = reinterpret_cast<double4 *>(s_cdyn + Lay::bytes);
    for (int k = lane; k < ntypes * ntypes; k += 32) s_lj[k] = lj64[k];
    lj = s_lj;
  }
  __syncwarp();
  const unsigned sb = __shfl_sync(0xffffffffu, (unsigned)__cvta_generic_to_shared(s_cdyn), 0);
  pdl_wait();
  for (int c = blockIdx.x * 32 + lane; c < g.ncol; c += gridDim.x * 32) count[c] = 0;
  const int cl = blockIdx.x >> lsplit;
  if (cl >= *(const volatile int *)ctl) return;  // uniform per block
  const ColAtom64 a = col_atom64(g, A, cl, sb + Lay::mol);
  const int ti = (a.m.x & 0xffff) * ntypes;
  ColPair64<kForm, kEnergy, kFull> pair{g, mc, A, a, lj + ti, ti, acc};
  ColWalk64<false, kSplit, decltype(pair)> walk{sb, pair};
  col_search64<false, kSplit>(g, A, a, cl, (int)(blockIdx.x & ((1u << lsplit) - 1u)), 1 << lsplit,
                              walk);
#pragma unroll
  for (int off = kColI; off < 32; off <<= 1) {
    pair.fx += __shfl_xor_sync(0xffffffffu, pair.fx, off);
    pair.fy += __shfl_xor_sync(0xffffffffu, pair.fy, off);
    pair.fz += __shfl_xor_sync(0xffffffffu, pair.fz, off);
  }
  const int js = lane / kColI;
  if (a.m.z >= 0 && js < 3)
    fix2_add_rank(acc, A.n, a.m.w, js, js == 0 ? pair.fx : (js == 1 ? pair.fy : pair.fz), A.err);
  if (kEnergy) {
    double v[ACC_MV];
#pragma unroll
    for (int k = 0; k < ACC_MV; k++) v[k] = 0.0;
    v[ACC_ECOUL] = kForm == FORM_CUTOFF ? a.p.w * pair.eC : pair.eC;
    v[ACC_ELJ] = pair.eL;
    v[ACC_PAIRS] = (double)pair.np;
    if (a.m.z < 0) v[ACC_ECOUL] = v[ACC_ELJ] = v[ACC_PAIRS] = 0.0;
    write_partial_row<ACC_E>(v, lane, partial + (size_t)blockIdx.x * kNacc);
  }
}

// ---------------------------------------------------------------------------
// Derivatives of the cutoff form (see k_deriv_fp64_half, whose per-pair terms
// these are): H w, and with kParams dE/dq and the table sums.
// ---------------------------------------------------------------------------
template <int kMode, bool kParams>
struct ColDeriv64 {
  static constexpr bool kVjp = kMode == DERIV_VJP;
  const ColGrid &g;
  const Fp64Consts &mc;
  const ColArrays &A;
  const ColAtom64 &a;
  const double4 *lj;
  int ntypes, ti;
  unsigned long long *acc;
  double *tab;          // the block's table sums (shared memory): modified pairs
  double wx, wy, wz;    // this atom's direction
  double hx = 0, hy = 0, hz = 0, gq = 0;
  double ta[kDerivRegTypes] = {0, 0, 0, 0}, tb[kDerivRegTypes] = {0, 0, 0, 0};
  double jx, jy, jz, jq;

  __device__ __forceinline__ void start() { jx = jy = jz = jq = 0.0; }
  template <class Tag>
  __device__ __forceinline__ void operator()(Tag, unsigned a16, unsigned a8) {
    constexpr bool kLj = Tag::value;
    using Lay = ColLayout64<kVjp>;
    const double2 d0 = lds2d(a16), d1 = lds2d(a16 + Lay::half);
    const int mj = lds1(a8);
    double d[3];
    double s = col_diff64(g, a, d0.x, d0.y, d1.x, d);
    const bool ok = (mj & a.bit) && s <= mc.cut2 && s > 0.0;
    s = ok ? s : 1.0;
    const int kind = (mj >> (24 + (threadIdx.x & (kColI - 1)))) & 1;
    const int tj = mj & 0xffff;
    double Us, Uss;
    DerivTerms u;
    if (kLj) {
      u = deriv_terms(mc, lj, ti + tj, kind, s, d1.y, col_rsqrt64(s));
      Us = u.Ss * u.E + u.S * u.Es + a.p.w * u.qf * u.phis;
      Uss = u.Sss * u.E + 2.0 * u.Ss * u.Es + u.S * u.Ess + a.p.w * u.qf * u.phiss;
    } else {  // no Lennard-Jones term (and no parameters asked for)
      const double ir = col_rsqrt64(s), is = ir * ir;
      const bool in = s <= mc.rcc2;
      const double qq = in ? a.p.w * d1.y * (kind ? mc.csf : 1.0) : 0.0;
      Us = qq * (-0.5 * ir * is + mc.c05_3);
      Uss = qq * (0.75 * ir * is * is);
    }
    double T = 0.0;
    if (kVjp) {
      const double2 w0 = lds2d(a16 + (Lay::w - Lay::pos)),
                    w1 = lds2d(a16 + (Lay::w - Lay::pos) + Lay::half);
      const double e0 = wx - w0.x, e1 = wy - w0.y, e2 = wz - w1.x;  // w_i - w_j
      const double dd = fma(d[0], e0, fma(d[1], e1, d[2] * e2));
      const double p = 2.0 * Us, q = 4.0 * Uss * dd;
      // (selected, not multiplied by zero: a direction need not be finite)
      const double vx = ok ? fma(p, e0, q * d[0]) : 0.0, vy = ok ? fma(p, e1, q * d[1]) : 0.0,
                   vz = ok ? fma(p, e2, q * d[2]) : 0.0;
      hx += vx;
      hy += vy;
      hz += vz;
      jx -= vx;
      jy -= vy;
      jz -= vz;
      T = -2.0 * dd;
    }
    if (kParams && ok) {
      const double c = kVjp ? u.phis * T : u.phi;
      gq = fma(u.qf, c, gq);                               // f q_j c
      jq = fma(a.p.w * (kind ? mc.csf : 1.0), c, jq);      // f q_i c
      double va, vb;
      if (kVjp) {
        va = 0.5 * T * (u.Ss * u.is6 - 6.0 * u.S * u.is6 * u.is);
        vb = 0.5 * T * (-u.Ss * u.is3 + 3.0 * u.S * u.is3 * u.is);
      } else {
        va = 0.5 * u.S * u.is6;
        vb = -0.5 * u.S * u.is3;
      }
      if (kind == 0) {
#pragma unroll
        for (int k = 0; k < kDerivRegTypes; k++)
          if (k == tj) { ta[k] += va; tb[k] += vb; }
      } else {  // a modified pair: entries 2, 3 of both orders
        const int mi = a.m.x & 0xffff;
        const int e1 = (ti + tj) * 4 + 2, e2 = (tj * ntypes + mi) * 4 + 2;
        atomicAdd(&tab[e1], va);
        atomicAdd(&tab[e1 + 1], vb);
        atomicAdd(&tab[e2], va);
        atomicAdd(&tab[e2 + 1], vb);
      }
    }
  }
  __device__ __forceinline__ void shift(int to) {
    if (kVjp) {
      jx = __shfl_xor_sync(0xffffffffu, jx, to);
      jy = __shfl_xor_sync(0xffffffffu, jy, to);
      jz = __shfl_xor_sync(0xffffffffu, jz, to);
    }
    if (kParams) jq = __shfl_xor_sync(0xffffffffu, jq, to);
  }
  __device__ __forceinline__ void join(int to) {
    if (kVjp) {
      jx += __shfl_xor_sync(0xffffffffu, jx, to);
      jy += __shfl_xor_sync(0xffffffffu, jy, to);
      jz += __shfl_xor_sync(0xffffffffu, jz, to);
    }
    if (kParams) jq += __shfl_xor_sync(0xffffffffu, jq, to);
  }
  __device__ __forceinline__ void finish(unsigned a8) {
    const int r = lds1(a8 + 4);
    if (kVjp) {
      fix2_add_rank(acc, A.n, r, 0, jx, A.err);
      fix2_add_rank(acc, A.n, r, 1, jy, A.err);
      fix2_add_rank(acc, A.n, r, 2, jz, A.err);
    }
    if (kParams) fix2_add_rank(acc, A.n, r, 3, jq, A.err);
  }
};

// (a product of 41,472 atoms at 12, 14, 16, 18, 20 blocks 213, 189, 193, 178, 178 us;
// dE/dparams at 8, 10, 12, 14, 16 blocks 234, 234, 233, 199, 199, both together 420,
// 326, 322, 285, 285)
#ifndef PMB200_COLD_BLOCKS
#define PMB200_COLD_BLOCKS 16
#endif
#ifndef PMB200_COLD_PARAM_BLOCKS
#define PMB200_COLD_PARAM_BLOCKS 12
#endif
// At most kDerivRegTypes types with kParams (any number without).  tpart
// [entry][block]: the block's table sums (zero beyond the last cluster).
template <int kMode, bool kParams>
__global__ void __launch_bounds__(32, kParams ? PMB200_COLD_PARAM_BLOCKS : PMB200_COLD_BLOCKS)
k_col_deriv64(const ColGrid g, const Fp64Consts mc, int ntypes,
              const double4 *__restrict__ lj64, const ColArrays A,
              unsigned long long *__restrict__ acc, const int *__restrict__ ctl,
              int *__restrict__ count, int lsplit, double *__restrict__ tpart) {
  constexpr bool kVjp = kMode == DERIV_VJP;
  using Lay = ColLayout64<kVjp>;
  extern __shared__ __align__(512) unsigned char s_cdyn[];
  __shared__ double s_tab[kParams ? kDerivTab : 1];
  const int lane = threadIdx.x;
  const double4 *lj = lj64;
  if (ntypes <= kCol64LjTypes) {
    double4 *s_lj = reinterpret_cast<double4 *>(s_cdyn + Lay::bytes);
    for (int k = lane; k < ntypes * ntypes; k += 32) s_lj[k] = lj64[k];
    lj = s_lj;
  }
  const int nt4 = ntypes * ntypes * 4;
  if (kParams)
    for (int k = lane; k < nt4; k += 32) s_tab[k] = 0.0;
  __syncwarp();
  const unsigned sb = __shfl_sync(0xffffffffu, (unsigned)__cvta_generic_to_shared(s_cdyn), 0);
  pdl_wait();
  for (int c = blockIdx.x * 32 + lane; c < g.ncol; c += gridDim.x * 32) count[c] = 0;
  const int cl = blockIdx.x >> lsplit;
  if (cl < *(const volatile int *)ctl) {  // uniform per block
    const ColAtom64 a = col_atom64(g, A, cl, sb + Lay::mol);
    const int mi = a.m.x & 0xffff, ti = mi * ntypes;
    double4 wi = make_double4(0.0, 0.0, 0.0, 0.0);
    if (kVjp && a.m.z >= 0) wi = A.w[(size_t)cl * kColI + (lane & (kColI - 1))];
    ColDeriv64<kMode, kParams> pair{g, mc, A, a, lj, ntypes, ti, acc, s_tab, wi.x, wi.y, wi.z};
    ColWalk64<kVjp, !kParams, decltype(pair)> walk{sb, pair};
    col_search64<kVjp, !kParams>(g, A, a, cl, (int)(blockIdx.x & ((1u << lsplit) - 1u)),
                                 1 << lsplit, walk);
#pragma unroll
    for (int off = kColI; off < 32; off <<= 1) {
      if (kVjp) {
        pair.hx += __shfl_xor_sync(0xffffffffu, pair.hx, off);
        pair.hy += __shfl_xor_sync(0xffffffffu, pair.hy, off);
        pair.hz += __shfl_xor_sync(0xffffffffu, pair.hz, off);
      }
      if (kParams) pair.gq += __shfl_xor_sync(0xffffffffu, pair.gq, off);
    }
    const int js = lane / kColI;
    if (a.m.z >= 0) {
      if (kVjp && js < 3)
        fix2_add_rank(acc, A.n, a.m.w, js, js == 0 ? pair.hx : (js == 1 ? pair.hy : pair.hz),
                      A.err);
      if (kParams && js == 3) fix2_add_rank(acc, A.n, a.m.w, 3, pair.gq, A.err);
    }
    if (kParams) {
      // the lanes' register sums to both orders of the types, lane by lane (a
      // fixed order)
      for (int l = 0; l < 32; l++) {
        if (l == lane && a.m.z >= 0) {
#pragma unroll
          for (int k = 0; k < kDerivRegTypes; k++) {
            if (k >= ntypes) break;
            s_tab[(ti + k) * 4] += pair.ta[k];
            s_tab[(ti + k) * 4 + 1] += pair.tb[k];
            s_tab[(k * ntypes + mi) * 4] += pair.ta[k];
            s_tab[(k * ntypes + mi) * 4 + 1] += pair.tb[k];
          }
        }
        __syncwarp();
      }
    }
  }
  if (kParams) {
    __syncwarp();
    for (int k = lane; k < nt4; k += 32) tpart[(size_t)k * gridDim.x + blockIdx.x] = s_tab[k];
  }
}

}  // namespace pmb200
