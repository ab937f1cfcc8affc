// Column kernels: the evaluation path of orthogonal periodic boxes.
//
// Positions are 32-bit fractions of the box edge (x = 2^32 (r - lower) / L
// modulo 2^32, one quantum = 2e-8 A on a 75 A box), so the difference of two
// coordinates, taken as a signed 32-bit integer, is the minimum image.
//
//   k_col_index  each atom's fractions; atoms counted and listed per column of
//                the x-y plane (a column is about the edge of a cube of kColI
//                atoms wide and the box high)
//   k_col_sort   one block per column: its atoms in order of height, padded to
//                whole clusters of kColI atoms, and for every slab of about
//                1.25 A the first atom at or above it
//   pair kernel  one cluster (kColI = 8 atoms, a box of about 4 A) against
//                single j atoms: per part of the neighbouring columns, the atoms
//                within the cutoff of the cluster's box are staged in shared
//                memory and evaluated in blocks of 32 (see col_task)
//   k_col_finalize*  fixed-point sums -> forces, energies
//
// Layout in HBM (n atoms, S slots: every column padded to whole clusters):
//   ipos[n]     int4  {x, y, z fractions, charge (FP32 bits)}, caller order
//   bucket[ncol][cap] int  atoms of a column in arrival order
//   spos[S]     int4  ipos in column / height order
//   smeta[S]    int4  {type | LJ-active << 16, molecule, atom (-1: pad), rank}; rank:
//                     the atom's place in column / height order without the pads
//   sidx[n]     int   the atom of each rank
//   sq[S]       double charge (FP64; energies)
//   dpos[n], spos64[S] double4 {wrapped position (A), charge} (FP64 kernels)
//   zs[ncol][nsz + 1] int  first slot of a column at or above a slab's bottom
//   facc[3][n]  int64 fixed-point forces, by rank (a block's atoms lie close
//               together: in the caller's order its atomics took four times the
//               memory wavefronts)
#pragma once
#include "pmb200_kernels.cuh"

namespace pmb200 {

constexpr int kColI = 8;          // atoms per cluster (i side of a tile)
constexpr int kColBlk = 32;       // j atoms per block
constexpr int kColCap = 128;      // staged j atoms per flush
constexpr int kColMaxCls = 256;   // neighbour-column classes
constexpr int kColSortCap = 1536; // atoms a column sort holds in shared memory,
constexpr int kColSortCapS = 384; // and in a batch of small boxes (k_col_sort_batch)
constexpr int kColMaxSlabs = 1024;
constexpr int kColScan = 12000;   // columns from which on k_col_scan sums the counts
constexpr int kColSortThreads = 256, kColSortThreadsS = 128;

struct ColGrid {
  int ncx, ncy, ncol, nsz;   // columns along x and y, slabs per column
  int cap;                   // bucket capacity per column
  int nslot;                 // upper bound of the slots in use
  int nparts;                // parts the neighbour columns are dealt into
  double boxmin[3], edge[3], inv[3];  // lower corner, edges (A), 1 / edge
  float q[3];                // length units per quantum
  double qd[3];              // the same in FP64
  float wx, wy;              // column widths (units)
  float hmax[3];             // half extents of a cluster up to which an atom within the
                             // cutoff of its box has one image for all its atoms
  float rc2;                 // squared cutoff with the box tests' margin (units^2)
  float inv_hs;              // slabs per unit
  double inv_unit;           // 1 / unit (1 / A)
  float qscale;              // FP32 charge scale: 1 / sqrt(unit)
};

// A share of the clusters: [total lo / of, total hi / of).
struct ColShare {
  int lo, hi, of;
  __device__ int first(int total) const { return (int)((long long)total * lo / of); }
  __device__ int end(int total) const { return (int)((long long)total * hi / of); }
};

// Neighbour columns as offsets modulo the grid, every unordered pair of
// columns reached from one side only; offsets that are their own negative
// carry bit 15 of y (the pair is then listed by its lower column).
struct ColStencil {
  int n = 0;
  short2 off[kColMaxCls];
};

// ---------------------------------------------------------------------------
// Build
// ---------------------------------------------------------------------------

// The fractions of one position (wrapped, if asked: the same position in the
// image the fractions are of, from the lower corner); false for a non-finite
// coordinate.
__device__ __forceinline__ bool col_fraction(const ColGrid &g, const double *x, unsigned u[3],
                                             double *wrapped = nullptr) {
  bool ok = true;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    double d = x[a] - g.boxmin[a];
    double w = d * g.inv[a];
    if (!isfinite(w)) { ok = false; w = 0.0; d = 0.0; }
    double image = floor(w);
    w -= image;
    const unsigned long long v = __double2ull_rn(w * 4294967296.0);
    u[a] = (unsigned)v;  // (2^32 wraps to 0, the next image)
    if (wrapped) {
      if (v >> 32) image += 1.0;
      wrapped[a] = fma(-image, g.edge[a], d);
    }
  }
  return ok;
}

__device__ __forceinline__ int col_of(const ColGrid &g, unsigned x, unsigned y) {
  return (int)__umulhi(x, (unsigned)g.ncx) * g.ncy + (int)__umulhi(y, (unsigned)g.ncy);
}

// Molecules whose centres the molecular virial needs, as fractions.
struct ColMols {
  int n;
  const int *start, *atoms;
  const double *mass;
  int4 *centre;
};

// clear: nclear x n words of the force accumulator zeroed on the way.  kMols: the
// blocks after the atoms' take a molecule a thread (two launches of their own
// were 8 of the 89 us of an evaluation with virials of 15,009 atoms).
template <bool kMols>
static __global__ void k_col_index(int n, const double *__restrict__ pos, ColGrid g,
                            const double *__restrict__ q, int4 *__restrict__ ipos,
                            int *__restrict__ count, int *__restrict__ bucket,
                            unsigned long long *__restrict__ clear, int nclear,
                            int *__restrict__ err, double4 *__restrict__ dpos, ColMols mols) {
  pdl_trigger();
  if (kMols && blockIdx.x >= (unsigned)(n + 255) / 256) {
    const int m = (int)((blockIdx.x - (unsigned)(n + 255) / 256) * blockDim.x + threadIdx.x);
    if (m >= mols.n) return;
    double c[3];
    molecule_centre(mols.atoms, mols.mass, pos, mols.start[m], mols.start[m + 1], c);
    unsigned u[3];
    col_fraction(g, c, u);
    mols.centre[m] = make_int4((int)u[0], (int)u[1], (int)u[2], 0);
    return;
  }
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int k = 0; k < nclear; k++) clear[(size_t)k * n + i] = 0;
  const double x[3] = {pos[3 * (size_t)i], pos[3 * (size_t)i + 1], pos[3 * (size_t)i + 2]};
  unsigned u[3];
  double wr[3];
  if (!col_fraction(g, x, u, dpos ? wr : nullptr)) atomicOr(err, 1);
  if (dpos) dpos[i] = make_double4(wr[0], wr[1], wr[2], q[i]);
  const int col = col_of(g, u[0], u[1]);
  // one add per column and warp: neighbours in the caller's order are often
  // neighbours in space (and a few hundred counters take all the atoms)
  const unsigned peers = __match_any_sync(__activemask(), col);
  const int lane = threadIdx.x & 31, lead = __ffs((int)peers) - 1;
  int slot = 0;
  if (lane == lead) slot = atomicAdd(&count[col], __popc(peers));
  slot = __shfl_sync(peers, slot, lead) + __popc(peers & ((1u << lane) - 1u));
  if (slot < g.cap) bucket[(size_t)col * g.cap + slot] = i;
  ipos[i] = make_int4((int)u[0], (int)u[1], (int)u[2], __float_as_int((float)q[i] * g.qscale));
}

// One column's sort by one block: base is its first slot, rank0 its first rank.  Order: slab, height,
// atom index (the layout, and every sum over it, is the same on every run).
// A counting sort by slab, then ranks among the few atoms of a slab; the slabs'
// first slots come with it.  (Ranks counted against the whole column took 50 us
// on the 327k-atom box.)  In shared memory where the column fits, else through
// the column's slots of a slot-sized list in global memory (scratch).  A column of
// more than cap atoms, whose bucket is incomplete, finds them in the whole list
// i0 .. i0 + n - 1, which it reads twice.
template <int kCap>
struct ColSortSmem {
  unsigned long long key[kCap];
  int list[kCap];
  int first[kColMaxSlabs + 1];
  int warp[8];
};
template <int kThreads, int kCap>
__device__ __forceinline__ void col_sort_column(
    const ColGrid &g, int col, int cnt, int base, int rank0, int i0, int n, const int4 *__restrict__ ipos,
    const int *__restrict__ bucket, const int *__restrict__ type, const int *__restrict__ mol,
    const unsigned char *__restrict__ ljact, const double *__restrict__ q,
    int4 *__restrict__ spos, int4 *__restrict__ smeta, double *__restrict__ sq,
    int *__restrict__ sidx, int *__restrict__ zs, int *scratch, ColSortSmem<kCap> &sm,
    const double4 *__restrict__ dpos = nullptr, double4 *__restrict__ spos64 = nullptr,
    const double *__restrict__ w = nullptr, double4 *__restrict__ sw = nullptr) {
  constexpr int T = kThreads;
  const int t = threadIdx.x, lane = t & 31, wp = t >> 5;
  const unsigned nsz = (unsigned)g.nsz;
  auto put = [&](int i, int rank, const int4 &p) {
    const int ty = type[i], mo = mol[i];
    const double qi = q[i];
    spos[base + rank] = p;
    smeta[base + rank] = make_int4(ty | ((int)ljact[ty] << 16), mo, i, rank0 + rank);
    sidx[rank0 + rank] = i;
    sq[base + rank] = qi;
    if (spos64) spos64[base + rank] = dpos[i];
    if (sw)
      sw[base + rank] = make_double4(w[3 * (size_t)i], w[3 * (size_t)i + 1], w[3 * (size_t)i + 2], 0.0);
  };
  // the column's atoms: from its bucket, or from the whole list
  const bool whole = cnt > g.cap, shared = !whole && cnt <= kCap;
  auto each = [&](auto &&f) {
    if (!whole) {
      for (int k = t; k < cnt; k += T) {
        const int i = bucket[k];
        f(k, i, (unsigned)ipos[i].z);
      }
    } else {
#pragma unroll 4
      for (int k = t; k < n; k += T) {
        const int4 p = ipos[i0 + k];
        if (col_of(g, (unsigned)p.x, (unsigned)p.y) == col) f(k, i0 + k, (unsigned)p.z);
      }
    }
  };
  for (int k = t; k < g.nsz; k += T) sm.first[k] = 0;
  __syncthreads();
  each([&](int k, int i, unsigned z) {
    if (shared) sm.key[k] = ((unsigned long long)z << 32) | (unsigned)i;
    atomicAdd(&sm.first[__umulhi(z, nsz)], 1);
  });
  __syncthreads();
  // slab counts -> first entries (exclusive), a block-sized piece at a time
  for (int c0 = 0, carry = 0; c0 < g.nsz; c0 += T) {
    const int v = c0 + t < g.nsz ? sm.first[c0 + t] : 0;
    int incl = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += u;
    }
    if (lane == 31) sm.warp[wp] = incl;
    __syncthreads();
    int before = carry, total = 0;
    for (int w = 0; w < T / 32; w++) {
      if (w < wp) before += sm.warp[w];
      total += sm.warp[w];
    }
    if (c0 + t < g.nsz) {
      sm.first[c0 + t] = before + incl - v;
      zs[c0 + t] = base + before + incl - v;
    }
    carry += total;
    __syncthreads();
  }
  if (t == 0) zs[g.nsz] = base + cnt;
  // scattered to their slabs in any order (first then holds each slab's end), then
  // ranked among the slab's atoms
  if (shared) {
    for (int k = t; k < cnt; k += T)
      sm.list[atomicAdd(&sm.first[__umulhi((unsigned)(sm.key[k] >> 32), nsz)], 1)] = k;
    __syncthreads();
    for (int e = t; e < cnt; e += T) {
      const unsigned long long me = sm.key[sm.list[e]];
      const int s = (int)__umulhi((unsigned)(me >> 32), nsz);
      const int lo = s ? sm.first[s - 1] : 0, hi = sm.first[s];
      int rank = lo;
      for (int m = lo; m < hi; m++) rank += sm.key[sm.list[m]] < me;
      const int i = (int)(unsigned)me;
      put(i, rank, ipos[i]);
    }
  } else {
    int *list = scratch + base;
    each([&](int, int i, unsigned z) { list[atomicAdd(&sm.first[__umulhi(z, nsz)], 1)] = i; });
    __syncthreads();
    for (int e = t; e < cnt; e += T) {
      const int i = list[e];
      const int4 p = ipos[i];
      const unsigned z = (unsigned)p.z;
      const int s = (int)__umulhi(z, nsz);
      const int lo = s ? sm.first[s - 1] : 0, hi = sm.first[s];
      int rank = lo;
      for (int m = lo; m < hi; m++) {
        const int o = list[m];
        const unsigned zo = (unsigned)ipos[o].z;
        rank += zo < z || (zo == z && o < i);
      }
      put(i, rank, p);
    }
  }
  const int end = (cnt + kColI - 1) / kColI * kColI;
  for (int k = cnt + t; k < end; k += T) {
    spos[base + k] = make_int4(0, 0, 0, 0);
    smeta[base + k] = make_int4(0, -1, -1, 0);
  }
}

// The clusters and atoms of the columns before `col`: each block of the sort sums
// them itself where the counts are few, else k_col_scan has (kColScan).
template <int kThreads, int kCap>
__device__ __forceinline__ void col_before(const int *__restrict__ count, int col, int &clusters,
                                           int &atoms, ColSortSmem<kCap> &sm) {
  constexpr int T = kThreads;
  const int t = threadIdx.x;
  int s = 0, a = 0;
  for (int c = t; c < col; c += T) {
    const int v = count[c];
    a += v;
    s += (v + kColI - 1) / kColI;
  }
  s = __reduce_add_sync(0xffffffffu, s);
  a = __reduce_add_sync(0xffffffffu, a);
  if ((t & 31) == 0) {
    sm.warp[t >> 5] = s;
    sm.list[t >> 5] = a;
  }
  __syncthreads();
  clusters = atoms = 0;
#pragma unroll
  for (int w = 0; w < T / 32; w++) {
    clusters += sm.warp[w];
    atoms += sm.list[w];
  }
}

// Exclusive prefix sums {clusters, atoms} over all columns, one block of 1024
// threads, four columns a thread and round.  The blocks' own sums are quadratic in
// the columns: forces of water films 20 A thick (8,464 / 16,900 / 26,244 / 126,736
// columns) 461 / 918 / 1,427 / 8,127 us, with this launch 463 / 909 / 1,392 /
// 6,680.
static __global__ void __launch_bounds__(1024)
k_col_scan(int ncol, const int *__restrict__ count, int2 *__restrict__ before) {
  pdl_trigger();
  pdl_wait();
  __shared__ int2 sh[32];
  const int t = threadIdx.x, lane = t & 31, wp = t >> 5;
  int2 carry = make_int2(0, 0);
  for (int c0 = 0; c0 < ncol; c0 += 4096) {
    const int c = c0 + 4 * t;
    int v[4];
    int2 sum = make_int2(0, 0);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      v[k] = c + k < ncol ? count[c + k] : 0;
      sum.x += (v[k] + kColI - 1) / kColI;
      sum.y += v[k];
    }
    int2 incl = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl.x, off);
      const int y = __shfl_up_sync(0xffffffffu, incl.y, off);
      if (lane >= off) {
        incl.x += x;
        incl.y += y;
      }
    }
    if (lane == 31) sh[wp] = incl;
    __syncthreads();
    int2 at = make_int2(carry.x + incl.x - sum.x, carry.y + incl.y - sum.y);
#pragma unroll 8
    for (int w = 0; w < 32; w++) {
      const int2 s = sh[w];
      if (w < wp) {
        at.x += s.x;
        at.y += s.y;
      }
      carry.x += s.x;
      carry.y += s.y;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (c + k < ncol) before[c + k] = at;
      at.x += (v[k] + kColI - 1) / kColI;
      at.y += v[k];
    }
    __syncthreads();
  }
}

// One block per column.  ctl[0]: the number of clusters.  sums: k_col_scan's, or null.
static __global__ void __launch_bounds__(kColSortThreads)
k_col_sort(int n, ColGrid g, const int4 *__restrict__ ipos, const int *__restrict__ count,
           const int *__restrict__ bucket, const int *__restrict__ type,
           const int *__restrict__ mol, const unsigned char *__restrict__ ljact,
           const double *__restrict__ q, int4 *__restrict__ spos, int4 *__restrict__ smeta,
           double *__restrict__ sq, int *__restrict__ sidx, int *__restrict__ zs,
           int *__restrict__ scratch, int *__restrict__ ctl, const double4 *__restrict__ dpos,
           double4 *__restrict__ spos64, const double *__restrict__ w,
           double4 *__restrict__ sw, const int2 *__restrict__ sums) {
  pdl_trigger();
  pdl_wait();
  __shared__ ColSortSmem<kColSortCap> sm;
  const int col = blockIdx.x, t = threadIdx.x;
  int before, atoms;
  if (sums) {
    before = sums[col].x;
    atoms = sums[col].y;
  } else {
    col_before<kColSortThreads>(count, col, before, atoms, sm);
  }
  const int cnt = count[col];
  if (col == g.ncol - 1 && t == 0) ctl[0] = before + (cnt + kColI - 1) / kColI;
  __syncthreads();
  col_sort_column<kColSortThreads>(g, col, cnt, before * kColI, atoms, 0, n, ipos, bucket + (size_t)col * g.cap,
                  type, mol, ljact, q, spos, smeta, sq, sidx, zs + (size_t)col * (g.nsz + 1), scratch, sm,
                  dpos, spos64, w, sw);
}

// ---------------------------------------------------------------------------
// The search of one cluster's partners (shared by the pair kernels).
// ---------------------------------------------------------------------------

struct ColBox {  // one cluster's bounding box (uniform over the warp)
  unsigned xc, yc, zc;         // centre (fractions)
  float hx, hy, hz;            // half extents (units, rounded up)
  int colx, coly, col;
  float ulx, uhx, uly, uhy;    // x and y extent from the column's lower corner
  int sl, sh;                  // slabs of its lowest and highest atom
  float fl, fh;                // their heights within the slab, in slabs
};

// p: this lane's atom (lanes without one hold the cluster's first atom).
__device__ __forceinline__ ColBox col_box(const ColGrid &g, const int4 &p) {
  ColBox b;
  const unsigned full = 0xffffffffu;
  const unsigned xl = __reduce_min_sync(full, (unsigned)p.x);
  const unsigned xh = __reduce_max_sync(full, (unsigned)p.x);
  const unsigned yl = __reduce_min_sync(full, (unsigned)p.y);
  const unsigned yh = __reduce_max_sync(full, (unsigned)p.y);
  const unsigned zl = __reduce_min_sync(full, (unsigned)p.z);
  const unsigned zh = __reduce_max_sync(full, (unsigned)p.z);
  constexpr float up = 1.0f + 1e-6f;
  b.xc = xl + ((xh - xl) >> 1);
  b.yc = yl + ((yh - yl) >> 1);
  b.zc = zl + ((zh - zl) >> 1);
  b.hx = (float)(xh - b.xc) * (g.q[0] * up);
  b.hy = (float)(yh - b.yc) * (g.q[1] * up);
  b.hz = (float)(zh - b.zc) * (g.q[2] * up);
  b.colx = (int)__umulhi(xl, (unsigned)g.ncx);
  b.coly = (int)__umulhi(yl, (unsigned)g.ncy);
  b.col = b.colx * g.ncy + b.coly;
  constexpr float s32 = 1.0f / 4294967296.0f;
  b.ulx = (float)(xl * (unsigned)g.ncx) * (g.wx * s32);
  b.uhx = (float)(xh * (unsigned)g.ncx) * (g.wx * s32);
  b.uly = (float)(yl * (unsigned)g.ncy) * (g.wy * s32);
  b.uhy = (float)(yh * (unsigned)g.ncy) * (g.wy * s32);
  b.sl = (int)__umulhi(zl, (unsigned)g.nsz);
  b.sh = (int)__umulhi(zh, (unsigned)g.nsz);
  b.fl = (float)(zl * (unsigned)g.nsz) * s32;
  b.fh = (float)(zh * (unsigned)g.nsz) * s32;
  return b;
}

// Squared distance of fraction p from the box (units; rounding is covered by
// the margin of g.rc2).
__device__ __forceinline__ float col_gap2(const ColGrid &g, const ColBox &b, const int4 &p) {
  const float dx = fmaxf(fabsf((float)(int)((unsigned)p.x - b.xc)) * g.q[0] - b.hx, 0.f);
  const float dy = fmaxf(fabsf((float)(int)((unsigned)p.y - b.yc)) * g.q[1] - b.hy, 0.f);
  const float dz = fmaxf(fabsf((float)(int)((unsigned)p.z - b.zc)) * g.q[2] - b.hz, 0.f);
  return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

// Shared memory as 32-bit addresses: the walk keeps its own running addresses.
__device__ __forceinline__ int4 lds4(unsigned a) {
  int4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ int2 lds2(unsigned a) {
  int2 v;
  asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ int lds1(unsigned a) {
  int v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ double lds1d(unsigned a) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts4(unsigned a, int4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z),
               "r"(v.w) : "memory");
}
__device__ __forceinline__ void sts2(unsigned a, int x, int y) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void sts1(unsigned a, int x) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(x) : "memory");
}
__device__ __forceinline__ void sts1d(unsigned a, double x) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(x) : "memory");
}

// approximate 1/sqrt and sqrt (one instruction each; the arguments lie far
// from the denormal range)
__device__ __forceinline__ float col_rsqrt(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float col_sqrt(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The runs of slots that one group of up to 16 columns (classes q0 + k stride)
// offers: those whose slabs come within the cutoff of the box, each column's
// below and above the periodic wrap.  Packed into `runs` (256 bytes of shared
// memory: per non-empty run its first candidate and slot - candidate).
// `after`: first slot after the cluster (its own column is searched upwards
// from there: each pair of clusters once).  Returns the number of candidates;
// begin: the first candidate of this lane's run.
__device__ __forceinline__ int col_runs(const ColGrid &g, const ColBox &b,
                                        const short2 *__restrict__ st, int st_n, int q0,
                                        int stride, int after, const int *__restrict__ zs,
                                        unsigned runs, int &begin) {
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu;
  // lane = 2 k + s: run s of the k-th column
  const int q = q0 + (lane >> 1) * stride;
  int a = 0, cnt = 0;
  if (q < st_n) {
    const short2 o = st[q];
    const int mx = o.x, my = o.y & 0x7fff;
    int jx = b.colx + mx, jy = b.coly + my;
    jx -= jx >= g.ncx ? g.ncx : 0;
    jy -= jy >= g.ncy ? g.ncy : 0;
    const int jc = jx * g.ncy + jy;
    const float gx = mx ? fmaxf(fminf((float)mx * g.wx - b.uhx,
                                      (float)(g.ncx - mx - 1) * g.wx + b.ulx), 0.f) : 0.f;
    const float gy = my ? fmaxf(fminf((float)my * g.wy - b.uhy,
                                      (float)(g.ncy - my - 1) * g.wy + b.uly), 0.f) : 0.f;
    const float rz2 = g.rc2 - fmaf(gx, gx, gy * gy);
    if (rz2 > 0.f && (o.y >= 0 || b.col < jc)) {
      const float rz = fmaf(col_sqrt(rz2), g.inv_hs, 1e-3f);
      int lo = b.sl + (int)floorf(b.fl - rz), hi = b.sh + (int)floorf(b.fh + rz) + 1;
      const int *z = zs + (size_t)jc * (g.nsz + 1);
      // slabs [lo, hi): all of the column, one run, or two across the wrap
      const bool all = hi - lo >= g.nsz, under = lo < 0, over = hi > g.nsz;
      if (lane & 1) {  // the wrapped part
        hi = all ? 0 : (under ? g.nsz : (over ? hi - g.nsz : 0));
        lo = all || !under ? 0 : lo + g.nsz;
      } else {
        lo = all || under ? 0 : lo;
        hi = all || over ? g.nsz : hi;
      }
      a = z[lo];
      const int e = z[hi];
      if (jc == b.col) a = max(a, after);
      cnt = max(e - a, 0);
    }
  }
  int incl = cnt;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int v = __shfl_up_sync(full, incl, off);
    if (lane >= off) incl += v;
  }
  const unsigned some = __ballot_sync(full, cnt > 0);
  __syncwarp();
  if (cnt > 0) {
    const int r = __popc(some & ((1u << lane) - 1u));
    sts2(runs + 8 * r, incl - cnt, a - (incl - cnt));
  }
  __syncwarp();
  begin = lane < __popc(some) ? lds1(runs + 8 * lane) : 0x40000000;
  return __shfl_sync(full, incl, 31);
}

// The slot of candidate f0 + lane (past the last: not a slot); run: the last
// run that starts before f0 (-1 at first), advanced.
__device__ __forceinline__ int col_slot(int f0, int begin, unsigned runs, int &run) {
  const int lane = threadIdx.x & 31;
  // the runs that start in this round, one bit each
  const unsigned at = (unsigned)(begin - f0);
  const unsigned m = __reduce_or_sync(0xffffffffu, at < 32u ? 1u << at : 0u);
  const int r = run + __popc(m & (0xffffffffu >> (31 - lane)));
  run += __popc(m);
  return f0 + lane + lds1(runs + 8 * max(r, 0) + 4);
}

// e^{-(h + l)}, l the rounding error of h: n = rint(-h log2 e), the remainder r by
// Cody and Waite's two-part ln 2 (Software Manual for the Elementary Functions,
// 1980), the Taylor polynomial to r^7 / 7! (|r| <= ln 2 / 2: 5e-9 left out), whose
// last step rounds to nearest.  expf of the rounded square left nine tenths of
// the Ewald energy's error (a bias of its last bit, and up to 4e-7 of the
// exponential from the square's).  h >= 0; from 87 on e^{-87}, 1.6e-38, which no sum
// here tells from zero (the exponent bits below would wrap).
__device__ __forceinline__ float col_exp_neg(float h, float l) {
  h = fminf(h, 87.0f);
  const float t = fmaf(-h, 1.44269504f, 12582912.0f);  // 1.5 2^23: rint in the low bits
  const float n = t - 12582912.0f;
  float r = fmaf(n, -0.693359375f, -h);
  r = fmaf(n, 2.12194440e-4f, r) - l;
  float p = fmaf(r, 1.0f / 5040.0f, 1.0f / 720.0f);
  p = fmaf(r, p, 1.0f / 120.0f);
  p = fmaf(r, p, 1.0f / 24.0f);
  p = fmaf(r, p, 1.0f / 6.0f);
  p = fmaf(r, p, 0.5f);
  p = fmaf(r, p, 1.0f);
  p = fmaf(r, p, 1.0f);
  return __int_as_float(__float_as_int(p) + (__float_as_int(t) << 23));
}

// A cluster's exclusions: one entry per lane (partner atom; bit ia, or bit
// 8 + ia for a modified pair) where there are at most 32, else looked up.
struct ColExcl {
  int partner, bits;
  bool fits;
};

// Pair masks of the lanes' j atoms (molecule molj, atom atomj; need: the lane
// holds one to stage) against the cluster: bit ia set in .x where the pair is
// evaluated, in .y where it is a modified (1-4) pair.  The exclusion lists
// hold pairs of one molecule only, so the molecules tell which atoms to look
// up; those are few, and each is compared with the whole cluster's list by
// the warp (lists read from global memory per atom took 18 of the pair
// kernel's 95 us on the 41k-atom water box).  smol: the eight molecules.
__device__ __forceinline__ int2 col_pair_mask(unsigned smol, const ColExcl &x, bool need, int molj,
                                              int atomj, int my_atom,
                                              const int *__restrict__ ex_start,
                                              const int2 *__restrict__ ex) {
  const unsigned full = 0xffffffffu;
  int2 m = make_int2((1 << kColI) - 1, 0);
  const int4 m0 = lds4(smol), m1 = lds4(smol + 16);
  const bool any = need && (m0.x == molj || m0.y == molj || m0.z == molj || m0.w == molj ||
                            m1.x == molj || m1.y == molj || m1.z == molj || m1.w == molj);
  unsigned look = __ballot_sync(full, any);
  const int lane = threadIdx.x & 31;
  while (look) {
    const int src = __ffs((int)look) - 1;
    look &= look - 1u;
    const int aj = __shfl_sync(full, atomj, src);
    int hit = 0;
    if (x.fits) {
      hit = x.partner == aj ? x.bits : 0;
    } else if (lane < kColI && my_atom >= 0) {
      const int kind = excl_kind(ex, ex_start[my_atom], ex_start[my_atom + 1], aj);
      hit = kind == 2 ? 1 << lane : (kind == 1 ? 0x100 << lane : 0);
    }
    const int bits = (int)__reduce_or_sync(full, (unsigned)hit);
    if (lane == src) {
      m.x &= ~bits;
      m.y = bits >> 8;
    }
  }
  return m;
}

// (the entry of lane l: found over the atoms' list lengths)
__device__ __forceinline__ ColExcl col_exclusions(int lane, int my_atom,
                                                  const int *__restrict__ ex_start,
                                                  const int2 *__restrict__ ex) {
  const unsigned full = 0xffffffffu;
  int lo = 0, cnt = 0;
  if (my_atom >= 0 && lane < kColI) {
    lo = ex_start[my_atom];
    cnt = ex_start[my_atom + 1] - lo;
  }
  int incl = cnt;
#pragma unroll
  for (int off = 1; off < kColI; off <<= 1) {
    const int v = __shfl_up_sync(full, incl, off);
    if (lane >= off) incl += v;
  }
  const int total = __shfl_sync(full, incl, kColI - 1);
  ColExcl x{-1, 0, total <= 32};
  if (x.fits) {
    int k = 0;  // lists that end at or before this lane's entry
#pragma unroll
    for (int step = 4; step > 0; step >>= 1) {
      const int v = __shfl_sync(full, incl, k + step - 1);
      if (v <= lane) k += step;
    }
    const int at = __shfl_sync(full, lo - (incl - cnt), k & 7) + lane;
    if (lane < total) {
      const int2 e = ex[at];
      x.partner = e.x;
      x.bits = e.y == 2 ? 1 << k : 0x100 << k;
    }
  }
  return x;
}

struct ColArrays {  // per system (single) or batch-wide
  const int4 *spos, *smeta;
  const double *sq;
  const double4 *spos64;     // FP64 kernels: wrapped position (A) and charge
  const double4 *w;          // direction of a Hessian-vector product, slot order
  const int *zs;
  const short2 *st;          // neighbour-column classes
  int st_n;
  const int *ex_start;
  const int2 *ex;
  const int4 *icom;
  unsigned long long *facc;  // [3][n]
  int n;
  int *err;
};

// The search of cluster cl over parts part0, part0 + pstride, ... by one warp:
// its own atoms (each against those before it), then the candidates 32 at a
// time.  pre(slot, valid) loads what the caller wants of a lane's slot beside
// its position; round(keep, slot, p, m, pmask, x, last) gets every lane's atom p,
// m, whether it is within the cutoff of the box, its pair masks and pre's
// result; last: the part's last round.  Everything goes through this one loop
// (several inlined copies of a pair walk overflow the instruction cache: 0.57 ms
// instead of 0.07 for the virial instance on a 15k-atom box).
template <class Pre, class Round>
__device__ __forceinline__ void col_search(const ColGrid &g, const ColArrays &A,
                                           const ColBox &box, const ColExcl &excl, int my_atom,
                                           unsigned smol, unsigned runs, int cl, int part0,
                                           int pstride, Pre &&pre, Round &&round) {
  const int lane = threadIdx.x & 31;
  const int after = (cl + 1) * kColI;
  for (int part = part0; part < g.nparts; part += pstride)
    for (int q0 = part; q0 < A.st_n; q0 += 16 * g.nparts) {
      int begin, run = -1;
      const int total = col_runs(g, box, A.st, A.st_n, q0, g.nparts, after, A.zs, runs, begin);
      const bool last_group = q0 + 16 * g.nparts >= A.st_n;
      for (int f0 = q0 == 0 ? -32 : 0;;) {
        const bool own = f0 < 0;  // (the own column's class is the first)
        int slot = cl * kColI + lane;
        bool valid = lane < kColI;
        if (!own) {
          slot = col_slot(f0, begin, runs, run);
          valid = f0 + lane < total;
        }
        int4 p = make_int4(0, 0, 0, 0), m = make_int4(0, -1, -1, 0);
        if (valid) {
          p = A.spos[slot];
          m = A.smeta[slot];
        }
        const auto x = pre(slot, valid);
        bool keep = m.z >= 0 && col_gap2(g, box, p) <= g.rc2;
        int2 pmask =
            col_pair_mask(smol, excl, keep, m.y, m.z, my_atom, A.ex_start, A.ex);
        if (own) {  // atom j against the cluster's atoms before it
          pmask.x &= (1 << lane) - 1;
          keep = keep && pmask.x;
        }
        f0 += 32;
        const bool done = f0 >= total;
        round(keep, p, m, pmask, x, done && last_group);
        if (done) break;
      }
    }
}

// ---------------------------------------------------------------------------
// Mixed-precision pair kernel.
// ---------------------------------------------------------------------------
constexpr float kColFix = 4294967296.0f;        // 2^32 per unit force
constexpr float kColForceLim = 1.0e9f;          // summed force component (unit force)

// Whether the last flush of a walk with at most `most` staged entries overwrites
// none that it moves: the back's rest goes behind the front entries, the filler up
// to the next whole block behind it (no barrier orders the lanes in between).
constexpr bool col_last_flush_apart(int most) {
  for (int nl = 0; nl <= most; nl++)
    for (int nn = 0; nl + nn <= most; nn++) {
      const int r = nn % kColBlk, end = (nl + r + kColBlk - 1) / kColBlk * kColBlk;
      if (r > 0 && end > kColCap - nn) return false;
    }
  return true;
}
static_assert(col_last_flush_apart(kColCap - 32) && !col_last_flush_apart(kColCap),
              "a full buffer needs a flush of its whole blocks before the last one");

// One warp's shared memory: kColCap staged entries -- fractions and charge (16
// bytes), {meta, force offset} (8), for the exact energies the FP64 charge (8), for
// the molecular virial the molecule's centre (16) -- then the cluster's molecules
// and the candidate runs.  meta: 16 type | pair mask << 16 | modified mask << 24;
// force offset: 8 rank.
template <bool kExactE, bool kMolVir>
struct ColLayout {
  static constexpr unsigned pos = 0, mg = 16 * kColCap, qd = mg + 8 * kColCap,
                            com = qd + (kExactE ? 8 * kColCap : 0),
                            mol = com + (kMolVir ? 16 * kColCap : 0), runs = mol + 32,
                            bytes = (runs + 256 + 511) / 512 * 512;
};

// One task: cluster cl, parts part0, part0 + pstride, ... of the grid's
// nparts, in one warp.  sb: its shared memory (512-byte aligned).
//
// Lane 8 s + ia holds atom ia of the cluster.  Staged atoms are evaluated in
// blocks of 32, lane group s taking eight of them: at step k its lane ia meets
// atom ia ^ k, so no two lanes of a group share one; the j force travels in
// registers, exchanged by shuffles so that it is always with the lane that adds
// to it, and after eight steps every lane holds the whole force on one j atom.
// (Reducing each step's j forces over the eight lanes instead took 11 more
// instructions a step of about 50.)  Atoms without a Lennard-Jones term (two
// thirds of a water box) are staged from the other end of the buffer and
// evaluated without its arithmetic; the remainder of both meets the general body.
//
// i forces: FP32 within a flush, then int64; j forces: FP32 sums of eight, then
// int64 atomics.  Integer sums, so the result does not depend on the order.
// kFull: both switches end at the pair cutoff.  kMod: modified pairs exist.
template <int kForm, bool kEnergy, bool kVirial, bool kMolVir, bool kFull, bool kMod>
__device__ __forceinline__ void col_task(const ColGrid &g, const MixedConsts &mc, int ntypes,
                                         const float4 *lj, const double2 *ljd, int cl, int part0,
                                         int pstride, const ColArrays &A, unsigned sb,
                                         double *__restrict__ row) {
  constexpr bool kHasLj = kForm == FORM_CUTOFF || kForm == FORM_GENERIC;
  constexpr bool kExactE = kEnergy && kForm == FORM_CUTOFF;
  using Lay = ColLayout<kExactE, kMolVir>;
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int ia = lane & (kColI - 1), js = lane / kColI;
  const int4 mi = A.smeta[(size_t)cl * kColI + ia];
  const int4 pi0 = A.spos[(size_t)cl * kColI + ia];
  const bool active = mi.z >= 0;
  const double qown = kExactE && active ? A.sq[(size_t)cl * kColI + ia] : 0.0;
  const unsigned lanebit = active ? 0x10000u << ia : 0u;
  int4 pi = pi0;  // (lanes without an atom: the cluster's first)
  const int4 first = make_int4(__shfl_sync(full, pi0.x, 0), __shfl_sync(full, pi0.y, 0),
                               __shfl_sync(full, pi0.z, 0), __shfl_sync(full, pi0.w, 0));
  if (!active) pi = first;
  const float qi = __int_as_float(pi.w);
  const int ti = (mi.x & 0xffff) * ntypes;
  const ColExcl excl = col_exclusions(lane, mi.z, A.ex_start, A.ex);
  const ColBox box = col_box(g, pi);
  // (constants of the walk in registers where g and mc lie in shared memory)
  const float qx = g.q[0], qy = g.q[1], qz = g.q[2], cut2 = mc.cut2;
  const float cc = -2.0f * mc.c05_3, lrc2 = mc.rclj2, lron2 = mc.ron2;
  const float ls1 = mc.s1, ls2 = mc.s2, ls3 = mc.s3;
  const char *lji = reinterpret_cast<const char *>(lj + ti);
  const char *ljdi = reinterpret_cast<const char *>(ljd + ti);
  const unsigned ljmod = 16u * (unsigned)(ntypes * ntypes);  // to the modified pairs' records
  __syncwarp();
  if (lane < kColI) sts1(sb + Lay::mol + 4 * lane, active ? mi.y : -2);
  int4 ci = make_int4(0, 0, 0, 0);
  if (kMolVir && active) ci = A.icom[mi.y];
  __syncwarp();

  long long fx = 0, fy = 0, fz = 0;
  double eU = 0.0, eL = 0.0;
  double w[6] = {0, 0, 0, 0, 0, 0}, mw[6] = {0, 0, 0, 0, 0, 0};
  int npair = 0;
  KahanF kU;
  float px = 0.f, py = 0.f, pz = 0.f, pE = 0.f;
  float pw[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, pm[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  float jx, jy, jz;  // force on the j atom with this lane

  int nl = 0, nn = 0;  // staged LJ atoms (from the front) and others (from the back)

  // This lane's atom against the staged atom at a16 (16 bytes an entry), a8 (8).
  auto pair = [&](auto ljtag, unsigned a16, unsigned a8) {
    [[maybe_unused]] constexpr bool kLj = decltype(ljtag)::value;
    const int4 pj = lds4(a16);
    const int mj = lds1(a8);
    // (signed differences of fractions: the minimum image.  Differences of FP32
    // positions staged relative to the cluster cost six instructions less, but
    // ran no faster and with 1.1 times the force error)
    const int dxi = pj.x - pi.x, dyi = pj.y - pi.y, dzi = pj.z - pi.z;
    const float ddx = __fmul_rn((float)dxi, qx), ddy = __fmul_rn((float)dyi, qy),
                ddz = __fmul_rn((float)dzi, qz);
    float r2 = fmaf(ddx, ddx, fmaf(ddy, ddy, __fmul_rn(ddz, ddz)));
    const bool ok = (mj & lanebit) && r2 <= cut2;
    // (masked pairs: finite terms where they meet a sum; a force is selected)
    if (kEnergy) r2 = ok ? r2 : 1.0f;
    const int kind = kMod ? (mj >> (24 + ia)) & 1 : 0;
    float qj = __int_as_float(pj.w);
    if (kMod) qj *= kind ? mc.csf : 1.0f;
    // 1/r: hardware reciprocal square root refined by one Newton-Raphson step
    float rinv = col_rsqrt(r2);
    rinv = fmaf(0.5f * rinv, fmaf(-r2 * rinv, rinv, 1.0f), rinv);
    const float r2inv = rinv * rinv;
    float f = 0.f;
    if constexpr (kForm == FORM_CUTOFF) {
      const bool inC = kFull || r2 <= mc.rcc2;
      // E S = q q (1/r - 1.5/rc + 0.5 r^2/rc^3): F S - E dS over r is
      // q q (1/r^3 - 1/rc^3)
      f = __fmul_rn(__fmul_rn(qi, qj), fmaf(r2inv, rinv, cc));
      if (!kFull) f = inC ? f : 0.f;
      double rid = 0.0;
      if (kExactE) {
        // q_j g(r) from the FP64 distance (the total cancels to ~1e-4 of the
        // pair magnitudes); 1/r by one Newton-Raphson step from the FP32 one
        const double ex = (double)dxi * g.qd[0], ey = (double)dyi * g.qd[1],
                     ez = (double)dzi * g.qd[2];
        const double r2d = fma(ex, ex, fma(ey, ey, ez * ez));
        rid = (double)rinv;
        rid = rid * fma(-0.5 * r2d, rid * rid, 1.5);
        const double gd = fma(mc.e05, r2d, rid - mc.e15);
        double qjd = lds1d(a8 + (Lay::qd - Lay::mg));
        if (kMod) qjd *= kind ? (double)mc.csf : 1.0;
        qjd = (ok && inC) ? qjd : 0.0;
        eU = fma(qjd, gd, eU);
      }
      if (kLj) {
        const float4 p = *reinterpret_cast<const float4 *>(lji + (mj & 0xffff));
        const float Aij = kMod && kind ? p.z : p.x, Bij = kMod && kind ? p.w : p.y;
        const float r6 = r2inv * r2inv * r2inv;
        const float elj = __fmul_rn(fmaf(Aij, r6, -Bij), r6);
        // 12 A r^-12 - 6 B r^-6 = 6 (A r^-12 + elj)
        const float flj = __fmul_rn(fmaf(__fmul_rn(Aij, r6), r6, elj), 6.0f * r2inv);
        const float c2 = lrc2 - r2;
        const float c4 = c2 * fmaf(2.0f, r2, ls2);
        const bool on = r2 >= lron2;
        float sv = on ? ls1 * (c2 * c4) : 1.0f;
        float sd = on ? ls3 * fmaf(c2, c2, -c4) : 0.0f;
        if (!kFull) {
          const bool in = r2 <= lrc2;
          sv = in ? sv : 0.f;
          sd = in ? sd : 0.f;
        }
        f = __fadd_rn(f, fmaf(flj, sv, -elj * sd));
        if (kExactE) {
          const double2 pd = *reinterpret_cast<const double2 *>(
              ljdi + (mj & 0xffff) + (kMod && kind ? ljmod : 0u));
          const double i2 = rid * rid, i6 = i2 * i2 * i2;
          eL = fma(fma(pd.x, i6, -pd.y) * i6, ok ? (double)sv : 0.0, eL);
        }
      }
    } else if constexpr (kForm == FORM_GENERIC) {
      if (ok) {
        if (kLj && mc.swl.kind != SW_OFF) {
          const float4 p = *reinterpret_cast<const float4 *>(lji + (mj & 0xffff));
          const float Aij = kind ? p.z : p.x, Bij = kind ? p.w : p.y;
          const float r6 = r2inv * r2inv * r2inv;
          const float elj = fmaf(Aij, r6, -Bij) * r6;
          const float flj = fmaf(12.0f * Aij, r6, -6.0f * Bij) * r6 * r2inv;
          float S, dS;
          switch_eval(mc.swl, r2, rinv, S, dS);
          f = fmaf(flj, S, -elj * dS);
          if (kEnergy) pE = fmaf(elj, S, pE);
        }
        if (mc.swc.kind != SW_OFF) {
          const float ec = qi * qj * rinv;
          float S, dS;
          switch_eval(mc.swc, r2, rinv, S, dS);
          f = __fadd_rn(f, fmaf(ec * r2inv, S, -ec * dS));
          if (kEnergy) kU.add(__fmul_rn(qj * rinv, S));
        }
      }
    } else {
      // real-space Ewald (NonbondedFullEwaldSystemForce.h:803-823)
      const float x = mc.ea * (r2 * rinv);
      const float xx = mc.ea2 * r2;
      const float ex = col_exp_neg(xx, fmaf(mc.ea2, r2, -xx));
      float gg;
      if constexpr (kForm == FORM_EWALD_POLY5) {
        const float t = __fdividef(1.0f, fmaf((float)kAsP, x, 1.0f));
        gg = t * fmaf(t, fmaf(t, fmaf(t, fmaf(t, (float)kAsA5, (float)kAsA4), (float)kAsA3),
                              (float)kAsA2), (float)kAsA1) * ex * rinv;
      } else {
        gg = erfcf(x) * rinv;
      }
      f = __fmul_rn(__fmul_rn(qi * qj, fmaf(mc.ea2pi, ex, gg)), r2inv);
      if (kEnergy) kU.add(ok ? __fmul_rn(qj, gg) : 0.f);
    }
    f = ok ? f : 0.f;
    if (kEnergy) npair += ok ? 1 : 0;
    // (every product that meets a sum does so in an explicit fmaf, so that all
    // kernels instantiating this body round a pair alike)
    px = fmaf(-ddx, f, px);
    py = fmaf(-ddy, f, py);
    pz = fmaf(-ddz, f, pz);
    jx = fmaf(ddx, f, jx);
    jy = fmaf(ddy, f, jy);
    jz = fmaf(ddz, f, jz);
    if (kVirial) {
      const float ox = __fmul_rn(ddx, f), oy = __fmul_rn(ddy, f), oz = __fmul_rn(ddz, f);
      pw[0] = fmaf(ox, ddx, pw[0]); pw[1] = fmaf(ox, ddy, pw[1]); pw[2] = fmaf(ox, ddz, pw[2]);
      pw[3] = fmaf(oy, ddy, pw[3]); pw[4] = fmaf(oy, ddz, pw[4]); pw[5] = fmaf(oz, ddz, pw[5]);
      if (kMolVir) {
        // comDiff: the minimal image of the molecule centres (zero within one)
        const int4 cj = lds4(a16 + (Lay::com - Lay::pos));
        const float cx = (float)(cj.x - ci.x) * qx, cy = (float)(cj.y - ci.y) * qy,
                    cz = (float)(cj.z - ci.z) * qz;
        pm[0] = fmaf(ox, cx, pm[0]); pm[1] = fmaf(ox, cy, pm[1]); pm[2] = fmaf(ox, cz, pm[2]);
        pm[3] = fmaf(oy, cy, pm[3]); pm[4] = fmaf(oy, cz, pm[4]); pm[5] = fmaf(oz, cz, pm[5]);
      }
    }
  };

  float vmax = 0.f;  // largest j force component so far (a NaN shows in px..pz)
  // the block of 32 entries from e0 (a multiple of 32) on
  auto block = [&](auto ljtag, int e0) {
    const unsigned e = (unsigned)(e0 + lane);
    unsigned a16 = sb + Lay::pos + 16 * e, a8 = sb + Lay::mg + 8 * e;
    jx = jy = jz = 0.f;
    // step k meets atom ia ^ k; the j force then moves to the lane that meets
    // its atom next, ia ^ k ^ (k + 1): 1, 3, 1, 7 away, and after the eighth step
    // 7 away to its own lane
    auto step = [&](unsigned to) {
      pair(ljtag, a16, a8);
      jx = __shfl_xor_sync(full, jx, (int)to);
      jy = __shfl_xor_sync(full, jy, (int)to);
      jz = __shfl_xor_sync(full, jz, (int)to);
      a16 ^= to << 4;
      a8 ^= to << 3;
    };
    // (two steps of code: with more, the kernel's instructions no longer fit the
    // nearest cache, and its issue rate fell by a tenth at eight)
#pragma unroll 1
    for (int h = 0; h < 4; h++) {
      step(1);
      step(h & 1 ? 7 : 3);
    }
    const unsigned off = (unsigned)lds1(a8 + 4);
    const float v = fmaxf(fmaxf(fabsf(jx), fabsf(jy)), fabsf(jz));
    vmax = fmaxf(vmax, v);
    if (v != 0.f) {
      unsigned long long *f = reinterpret_cast<unsigned long long *>(
          reinterpret_cast<char *>(A.facc) + off);
      atomicAdd(f, (unsigned long long)__float2ll_rn(jx * kColFix));
      atomicAdd(f + A.n, (unsigned long long)__float2ll_rn(jy * kColFix));
      atomicAdd(f + 2 * (size_t)A.n, (unsigned long long)__float2ll_rn(jz * kColFix));
    }
  };
  // (no lane writes an entry that another still reads: what a flush moves and what
  // it overwrites lie apart, in the last one because at most kColCap - 32 entries
  // are left when it comes)
  auto copy_entry = [&](int from, int to) {
    sts4(sb + Lay::pos + 16 * to, lds4(sb + Lay::pos + 16 * from));
    const int2 m = lds2(sb + Lay::mg + 8 * from);
    sts2(sb + Lay::mg + 8 * to, m.x, m.y);
    if (kExactE) sts1d(sb + Lay::qd + 8 * to, lds1d(sb + Lay::qd + 8 * from));
    if (kMolVir) sts4(sb + Lay::com + 16 * to, lds4(sb + Lay::com + 16 * from));
  };
  // evaluate the staged entries: whole blocks, the rest kept (last: all, the
  // others' rest and then filler behind the LJ entries)
  auto flush = [&](bool last) {
    __syncwarp();
    const int bn = kHasLj ? nn & ~(kColBlk - 1) : 0;
    if (kHasLj)
      for (int t = 0; t < bn; t += kColBlk) block(std::false_type{}, kColCap - kColBlk - t);
    const int r = nn - bn;
    int fn = nl & ~(kColBlk - 1);
    if (last) {
      if (lane < r) copy_entry(kColCap - 1 - (bn + lane), nl + lane);
      nl += r;
      fn = (nl + kColBlk - 1) & ~(kColBlk - 1);
      if (nl + lane < fn) {
        const int e = nl + lane;
        sts4(sb + Lay::pos + 16 * e, make_int4(0, 0, 0, 0));
        sts2(sb + Lay::mg + 8 * e, 0, 0);
        if (kExactE) sts1d(sb + Lay::qd + 8 * e, 0.0);
        if (kMolVir) sts4(sb + Lay::com + 16 * e, make_int4(0, 0, 0, 0));
      }
      __syncwarp();
    }
    for (int t = 0; t < fn; t += kColBlk) block(std::true_type{}, t);
    __syncwarp();
    if (last) {
      nl = nn = 0;
    } else {
      const int rf = nl - fn;
      if (bn > 0 && lane < r) copy_entry(kColCap - 1 - (bn + lane), kColCap - 1 - lane);
      if (fn > 0 && lane < rf) copy_entry(fn + lane, lane);
      nn = r;
      nl = rf;
    }
    // the flush's FP32 sums into the wide ones
    fx += __float2ll_rn(px * kColFix);
    fy += __float2ll_rn(py * kColFix);
    fz += __float2ll_rn(pz * kColFix);
    // (sum, not maximum: a NaN must show)
    if (!(fabsf(px) + fabsf(py) + fabsf(pz) + vmax < kColForceLim)) atomicOr(A.err, 2);
    px = py = pz = 0.f;
    if (kEnergy) { eL += (double)pE; pE = 0.f; }
    if (kEnergy && !kExactE) {  // (per flush: grouped alike however the parts are dealt)
      eU += (double)kU.s - (double)kU.c;
      kU = KahanF();
    }
    if (kVirial)
#pragma unroll
      for (int k = 0; k < 6; k++) { w[k] += (double)pw[k]; pw[k] = 0.f; }
    if (kMolVir)
#pragma unroll
      for (int k = 0; k < 6; k++) { mw[k] += (double)pm[k]; pm[k] = 0.f; }
    __syncwarp();
  };
  col_search(
      g, A, box, excl, mi.z, sb + Lay::mol, sb + Lay::runs, cl, part0, pstride,
      [&](int slot, bool valid) { return kExactE && valid ? A.sq[slot] : 0.0; },
      [&](bool keep, const int4 &p, const int4 &m, const int2 &pmask, double qd, bool last) {
        const bool front = !kHasLj || (m.x & 0x10000);
        const unsigned kf = __ballot_sync(full, keep && front);
        const unsigned kb = __ballot_sync(full, keep && !front);
        if (keep) {
          const unsigned below = (1u << lane) - 1u;
          const int e = front ? nl + __popc(kf & below) : kColCap - 1 - (nn + __popc(kb & below));
          sts4(sb + Lay::pos + 16 * e, p);
          if (kExactE) sts1d(sb + Lay::qd + 8 * e, qd);
          sts2(sb + Lay::mg + 8 * e, ((m.x & 0xfff) << 4) | (pmask.x << 16) | (pmask.y << 24),
               (int)(8u * (unsigned)m.w));
          if (kMolVir) sts4(sb + Lay::com + 16 * e, A.icom[m.y]);
        }
        nl += __popc(kf);
        nn += __popc(kb);
        // (a fuller buffer empties its whole blocks before the last flush, so that
        // the rest moved to the front and the filler behind it end below the first
        // entry to be moved)
        bool fuller;
        do {
          fuller = nl + nn > kColCap - 32;
          if (fuller || last) flush(last && !fuller);
        } while (fuller && last);
      });

  // i forces over the lane groups, one component per group
#pragma unroll
  for (int off = kColI; off < 32; off <<= 1) {
    fx += __shfl_xor_sync(full, fx, off);
    fy += __shfl_xor_sync(full, fy, off);
    fz += __shfl_xor_sync(full, fz, off);
  }
  if (active && js < 3) {
    const long long v = js == 0 ? fx : (js == 1 ? fy : fz);
    if (v) atomicAdd(&A.facc[(size_t)js * A.n + mi.w], (unsigned long long)v);
  }
  if (kEnergy || kVirial) {
    double v[ACC_MV];
#pragma unroll
    for (int k = 0; k < ACC_MV; k++) v[k] = 0.0;
    if (kEnergy && active) {
      // weighted by q_i: the exact form in FP64 charges (1 / unit for 1 / r)
      v[ACC_ECOUL] = kExactE ? qown * g.inv_unit * eU
                             : (double)qi * eU;
      v[ACC_ELJ] = eL;
      v[ACC_PAIRS] = (double)npair;
    }
#pragma unroll
    for (int k = 0; k < 6; k++) { v[ACC_W + k] = w[k]; v[ACC_MW + k] = mw[k]; }
    write_partial_row<kVirial ? ACC_MV : ACC_E>(v, lane, row);
  }
}

// One warp per block, each its own task (a warp that finishes early frees its
// slot): block b takes cluster b >> lsplit, parts (b & (2^lsplit - 1)) + k 2^lsplit.
// share: the part of the clusters that this launch takes.
// Dynamic shared memory: the warp's entries, then the LJ tables (for exact
// energies double2 {A, B} [and {A14, B14}], float4; up to kMaxTypes types).
#ifndef PMB200_COL_BLOCKS
#define PMB200_COL_BLOCKS 24
#endif
#ifndef PMB200_COL_BLOCKS_V
// with virials (15,009 atoms with both, 12 / 13 / 14 / 16 blocks: 81.3 / 77.0 / 75.3 /
// 75.3 us an evaluation; the Ewald form 77.7 / 69.4 / 69.5 / 70.6)
#define PMB200_COL_BLOCKS_V 14
#endif
#ifndef PMB200_COL_BLOCKS_E
#define PMB200_COL_BLOCKS_E 20
#endif
template <int kForm, bool kEnergy, bool kVirial, bool kMolVir, bool kFull, bool kMod, bool kGlobalLj>
__global__ void __launch_bounds__(32, kVirial   ? PMB200_COL_BLOCKS_V
                                      : kEnergy ? PMB200_COL_BLOCKS_E
                                                : PMB200_COL_BLOCKS)
k_col_pair(const ColGrid g, const MixedConsts mc, int ntypes, const float4 *__restrict__ lj32,
           const double2 *__restrict__ lj64, const ColArrays A, const int *__restrict__ ctl,
           int *__restrict__ count, int lsplit, ColShare share,
           double *__restrict__ partial) {
  constexpr bool kHasLj = kForm == FORM_CUTOFF || kForm == FORM_GENERIC;
  constexpr bool kExactE = kEnergy && kForm == FORM_CUTOFF;
  using Lay = ColLayout<kExactE, kMolVir>;
  extern __shared__ __align__(512) unsigned char s_cdyn[];
  const int nlj = kHasLj && !kGlobalLj ? ntypes * ntypes : 0;
  constexpr int kRec = kExactE ? (kMod ? 2 : 1) : 0;
  double2 *s_ljd = reinterpret_cast<double2 *>(s_cdyn + Lay::bytes);
  float4 *s_lj = reinterpret_cast<float4 *>(s_ljd + kRec * nlj);
  const int lane = threadIdx.x;
  for (int k = lane; k < nlj; k += 32) s_lj[k] = lj32[k];
  for (int k = lane; k < kRec * nlj; k += 32) s_ljd[k] = lj64[k];
  __syncwarp();
  // (through a shuffle, so that the address is kept in a register and not
  // formed anew wherever it is used)
  const unsigned sb =
      __shfl_sync(0xffffffffu, (unsigned)__cvta_generic_to_shared(s_cdyn), 0);
  // (an overlapping launch waits here for the build: its prologue reads only
  // what was written before that started)
  pdl_wait();
  // the build's counts cleared for the next one
  for (int c = blockIdx.x * 32 + lane; c < g.ncol; c += gridDim.x * 32) count[c] = 0;
  int c1 = *(const volatile int *)ctl;
  int cl = blockIdx.x >> lsplit;
  if (share.of > 1) {
    cl += share.first(c1);
    c1 = share.end(c1);
  }
  if (cl >= c1) return;  // uniform per block
  col_task<kForm, kEnergy, kVirial, kMolVir, kFull, kMod>(
      g, mc, ntypes, kGlobalLj ? lj32 : s_lj, kGlobalLj ? lj64 : s_ljd, cl,
      (int)(blockIdx.x & ((1u << lsplit) - 1u)), 1 << lsplit, A, sb,
      partial + (size_t)blockIdx.x * kNacc);
}

// Component q of the force on the atom of rank r from the fixed-point sums: [3][n]
// (mixed; scale 2^-32 / unit) or the FP64 kernels' two words [8][n] (unscaled; q =
// 3: dq).
template <bool k64>
__device__ __forceinline__ double col_force(const unsigned long long *__restrict__ facc, size_t n,
                                            int r, int q, double scale) {
  if (!k64) return (double)(long long)facc[q * n + r] * scale;
  const double hi = (double)(long long)facc[q * n + r];
  const double lo = (double)(long long)facc[(4 + q) * n + r];
  return (hi + lo * (1.0 / kFix2Lo)) * (1.0 / kFix2Hi);
}

// Forces (or H w) in the caller's order, accumulated or overwritten; dq (FP64
// kernels, or null).
template <bool k64>
__global__ void __launch_bounds__(256)
k_col_finalize(int n, const unsigned long long *__restrict__ facc, const int *__restrict__ sidx,
               double scale, int accumulate, double *__restrict__ forces,
               double *__restrict__ dq) {
  pdl_wait();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int o = sidx[r];
  if (forces) {
    double *f = forces + 3 * (size_t)o;
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const double v = col_force<k64>(facc, n, r, q, scale);
      f[q] = accumulate ? f[q] + v : v;
    }
  }
  if (k64 && dq) dq[o] = col_force<k64>(facc, n, r, 3, scale);
}

// k_reduce1 over the rows of a share's clusters.
__device__ __forceinline__ int col_rows(const int *ctl, int lsplit, const ColShare &share) {
  const int ncl = *(const volatile int *)ctl;
  return (share.end(ncl) - share.first(ncl)) << lsplit;
}
static __global__ void k_col_reduce1(const int *__restrict__ ctl, int lsplit, ColShare share,
                              const double *__restrict__ partial, double *__restrict__ red,
                              int ns) {
  __shared__ double sh[8][ACC_MV];
  reduce1_block(blockIdx.x, col_rows(ctl, lsplit, share), partial, red, ns, sh);
}

// k_col_finalize, k_col_reduce1 and k_reduce2 in one launch of
// max(ceil(n / 256), kRedBlocks) blocks (see k_finalize_reduce: the same sums
// in the same order as the separate kernels).  f32: the forces go there in FP32
// instead.  tail (or null): receives the 20 results and the error flag.
template <bool k64>
__global__ void __launch_bounds__(256)
k_col_finalize_reduce(int n, const unsigned long long *__restrict__ facc,
                      const int *__restrict__ sidx, double scale, int accumulate,
                      double *__restrict__ forces, const int *__restrict__ ctl, int lsplit, const double *__restrict__ partial, double *red,
                      unsigned *__restrict__ arrivals, double *__restrict__ out,
                      double *__restrict__ pairs_out, int ns, float *__restrict__ f32,
                      double *tail, const int *err) {
  pdl_wait();
  __shared__ double sh[8][ACC_MV];
  __shared__ double col[ACC_MV];
  __shared__ unsigned s_arrived;
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n) {
    const size_t o = 3 * (size_t)sidx[r];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const double v = col_force<k64>(facc, n, r, q, scale);
      if (f32) f32[o + q] = (float)v;
      else forces[o + q] = accumulate ? forces[o + q] + v : v;
    }
  }
  if (blockIdx.x >= kRedBlocks) return;  // uniform per block
  reduce1_block(blockIdx.x, col_rows(ctl, lsplit, ColShare{0, 1, 1}), partial, red, ns, sh);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_arrived = atomicInc(arrivals, kRedBlocks - 1);
  __syncthreads();
  if (s_arrived != kRedBlocks - 1) return;  // uniform per block
  __threadfence();
  reduce2_block(kRedBlocks, red, 1.0, out, pairs_out, ns, col);
  if (tail && threadIdx.x == 0) {  // (out was written by this thread, and may be tail)
    if (tail != out)
      for (int q = 0; q < 20; q++) tail[q] = out[q];
    *reinterpret_cast<int *>(tail + 20) = *(const volatile int *)err;
  }
}

// ---------------------------------------------------------------------------
// Batches of systems: the same kernels over concatenated arrays.  Atom indices
// and ranks (ipos, smeta, facc, the exclusion lists) are batch-wide; slots, columns and
// clusters count from each system's first.
// ---------------------------------------------------------------------------
struct ColBatchSys {
  ColGrid g;
  MixedConsts mc;
  double fscale;            // fixed point -> force: 2^-32 / unit
  int atom0, natoms, col0, slot0, zs0;
  long long bucket0;
  int st0, st_n;            // neighbour-column classes
  int lj0, act0, ntypes;    // LJ tables (float4; double2 at 2 lj0), LJ-active flags
};

static __global__ void k_col_index_batch(int N, const double *__restrict__ pos,
                                         const ColBatchSys *__restrict__ sys,
                                         const int *__restrict__ atom_sys,
                                         const double *__restrict__ q, int4 *__restrict__ ipos,
                                         int *__restrict__ count, int *__restrict__ bucket,
                                         unsigned long long *__restrict__ clear,
                                         int *__restrict__ err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  for (int k = 0; k < 3; k++) clear[(size_t)k * N + i] = 0;
  const ColBatchSys &b = sys[atom_sys[i]];
  const double x[3] = {pos[3 * (size_t)i], pos[3 * (size_t)i + 1], pos[3 * (size_t)i + 2]};
  unsigned u[3];
  if (!col_fraction(b.g, x, u)) atomicOr(err, 1);
  const int col = col_of(b.g, u[0], u[1]);
  const int slot = atomicAdd(&count[b.col0 + col], 1);
  if (slot < b.g.cap) bucket[b.bucket0 + (size_t)col * b.g.cap + slot] = i;
  ipos[i] = make_int4((int)u[0], (int)u[1], (int)u[2], __float_as_int((float)q[i] * b.g.qscale));
}

// One block per column of the batch; col_sys: its system.  ctl[s]: clusters.
// Bound by each block's chain of loads and barriers; what helps is blocks in
// flight.  Where twice every system's mean column and 64 fit kColSortCapS atoms
// (longer ones go through global memory) blocks take kColSortThreadsS threads
// and 9 KB instead of 22 KB: an evaluation of 512 boxes of 300 to 6,000 atoms
// 2,208 -> 2,172 us (32 and 64 threads the same within 5).
template <int kThreads, int kCap>
static __global__ void __launch_bounds__(kThreads)
k_col_sort_batch(const ColBatchSys *__restrict__ sys, const int *__restrict__ col_sys,
                 const int4 *__restrict__ ipos, const int *__restrict__ count,
                 const int *__restrict__ bucket, const int *__restrict__ type,
                 const int *__restrict__ mol, const unsigned char *__restrict__ ljact,
                 const double *__restrict__ q, int4 *__restrict__ spos,
                 int4 *__restrict__ smeta, double *__restrict__ sq, int *__restrict__ sidx,
                 int *__restrict__ zs, int *__restrict__ scratch, int *__restrict__ ctl,
                 const int2 *__restrict__ sums) {
  __shared__ ColSortSmem<kCap> sm;
  const int s = col_sys[blockIdx.x], t = threadIdx.x;
  const ColBatchSys &b = sys[s];
  const int col = (int)blockIdx.x - b.col0;
  int before, atoms;
  if (sums) {  // (over all systems)
    const int2 first = sums[b.col0], here = sums[blockIdx.x];
    before = here.x - first.x;
    atoms = here.y - first.y;
  } else {
    col_before<kThreads>(count + b.col0, col, before, atoms, sm);
  }
  const int cnt = count[blockIdx.x];
  if (col == b.g.ncol - 1 && t == 0) ctl[s] = before + (cnt + kColI - 1) / kColI;
  __syncthreads();
  col_sort_column<kThreads>(b.g, col, cnt, before * kColI, b.atom0 + atoms, b.atom0, b.natoms, ipos,
                  bucket + b.bucket0 + (size_t)col * b.g.cap, type, mol, ljact + b.act0, q,
                  spos + b.slot0, smeta + b.slot0, sq + b.slot0, sidx,
                  zs + b.zs0 + (size_t)col * (b.g.nsz + 1), scratch + b.slot0, sm);
}

// Persistent: each one-warp block takes tasks {system, cluster, part, parts} from
// the counter (tasks of clusters beyond a system's last write an empty row).
// Dynamic shared memory: the warp's entries, the system, its LJ tables (at most
// lj_max type pairs).
template <int kForm, bool kEnergy, bool kVirial, bool kFull, bool kMod>
__global__ void __launch_bounds__(32, kVirial   ? PMB200_COL_BLOCKS_V
                                      : kEnergy ? PMB200_COL_BLOCKS_E
                                                : PMB200_COL_BLOCKS)
k_col_pair_batch(const ColBatchSys *__restrict__ sys, const int4 *__restrict__ tasks, int ntasks,
                 int *__restrict__ counter, const short2 *__restrict__ st,
                 const float4 *__restrict__ lj32, const double2 *__restrict__ lj64,
                 const ColArrays A0, const int *__restrict__ ctl, int *__restrict__ count,
                 int ncol, int lj_max, double *__restrict__ partial) {
  constexpr bool kHasLj = kForm == FORM_CUTOFF || kForm == FORM_GENERIC;
  constexpr bool kExactE = kEnergy && kForm == FORM_CUTOFF;
  constexpr int kRec = kExactE ? (kMod ? 2 : 1) : 0;
  using Lay = ColLayout<kExactE, false>;
  extern __shared__ __align__(512) unsigned char s_cdyn[];
  ColBatchSys &b = *reinterpret_cast<ColBatchSys *>(s_cdyn + Lay::bytes);
  double2 *s_ljd = reinterpret_cast<double2 *>(s_cdyn + Lay::bytes +
                                               (sizeof(ColBatchSys) + 15) / 16 * 16);
  float4 *s_lj = reinterpret_cast<float4 *>(s_ljd + kRec * lj_max);
  const unsigned sb = __shfl_sync(0xffffffffu, (unsigned)__cvta_generic_to_shared(s_cdyn), 0);
  const int lane = threadIdx.x;
  for (int c = blockIdx.x * 32 + lane; c < ncol; c += gridDim.x * 32) count[c] = 0;
  int loaded = -1;
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(counter, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= ntasks) break;  // uniform per warp
    const int4 tk = tasks[t];
    double *row = partial + (size_t)t * kNacc;
    if (tk.y >= ctl[tk.x]) {
      if ((kEnergy || kVirial) && lane < kNacc) row[lane] = 0.0;
      continue;
    }
    if (tk.x != loaded) {
      __syncwarp();
      const int *src = reinterpret_cast<const int *>(&sys[tk.x]);
      int *dst = reinterpret_cast<int *>(&b);
      for (int k = lane; k < (int)(sizeof(ColBatchSys) / sizeof(int)); k += 32) dst[k] = src[k];
      loaded = tk.x;
      __syncwarp();
      if (kHasLj) {
        const int t2 = b.ntypes * b.ntypes;
        for (int k = lane; k < t2; k += 32) s_lj[k] = lj32[b.lj0 + k];
        for (int k = lane; k < kRec * t2; k += 32) s_ljd[k] = lj64[2 * (size_t)b.lj0 + k];
      }
      __syncwarp();
    }
    ColArrays A = A0;
    A.spos += b.slot0;
    A.smeta += b.slot0;
    A.sq += b.slot0;
    A.zs += b.zs0;
    A.st = st + b.st0;
    A.st_n = b.st_n;
    col_task<kForm, kEnergy, kVirial, false, kFull, kMod>(b.g, b.mc, b.ntypes, s_lj, s_ljd, tk.y,
                                                          tk.z, tk.w, A, sb, row);
  }
}

static __global__ void __launch_bounds__(256)
k_col_finalize_batch(int N, const unsigned long long *__restrict__ facc,
                     const int *__restrict__ sidx, const int *__restrict__ atom_sys,
                     const ColBatchSys *__restrict__ sys, int accumulate,
                     double *__restrict__ forces) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= N) return;
  const int o = sidx[r];
  const double scale = sys[atom_sys[r]].fscale;  // (a system's ranks are its atoms' range)
  double *f = forces + 3 * (size_t)o;
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const double v = col_force<false>(facc, N, r, q, scale);
    f[q] = accumulate ? f[q] + v : v;
  }
}

}  // namespace pmb200
