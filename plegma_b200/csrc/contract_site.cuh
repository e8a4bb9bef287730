// Site contraction fused with the projection's sums over x, one site per lane:
// what the nucleon and meson kernel and the Delta kernel share.
//
// A position buffer costs 8 (split form) or 16 bytes (plain form) per site and
// component, written and read again.  Here a CTA walks over whole x rows,
// keeps the outputs of a tile in shared memory and adds them, times the x
// phases of project_axes.cu, into register sums that leave once per row: R1 /
// Lx of the buffer.
//
// A CTA has 16 roles of kS threads, thread = (role, site): split form (R =
// float) 16 warps and tiles of 32 consecutive sites of a unit of whole rows,
// plain form (R = double) 8 warps, whose half-warps are roles, and 16 sites.
// The roles share the work of a site and exchange partial sums through shared
// memory; lane = site makes a spin block's nine entries conflict-free loads,
// keeps the control uniform and needs no shuffles.  The next tile is
// prefetched into L2 during a tile's contraction; its u half is loaded into
// registers before the last phase of the contraction, its d half before the
// sums over x, so that both latencies are covered.  A row's sites are added
// in order by one thread, in the split form by fours that count from the
// slice's first site, so a row's sum does not depend on the launch shape.
// The x phases are kernel parameters: they come through the constant bank and
// cost no shared-memory wavefronts (copied to shared memory the plain form was
// 14 % slower).
//
// Why 16 warps of 32 sites: two CTAs of 16 sites per SM, whose phases overlap,
// took the same time for the mesons and 4 % more for the Delta (roles in half-
// warps load half the shared-memory bytes per wavefront in the products).  A
// slice without a rotation converts whole spin blocks; the groups of four
// blocks that a rotation mixes cost 680 instructions per site against 70, which
// was 8 % of the mesons' time.
// Measured on B200 against the position buffer and the sums over x from it, 123
// momenta: nucleon + 16 x 16 mesons, split, 48^3 x 8 slices 2.48 -> 2.24 ms; plain,
// 24^3 x 24 1.90 -> 1.59 ms; with both Deltas, split, 32^3 x 12 4.36 -> 3.59 ms, 48^3
// x 8 9.50 -> 7.86 ms.
#pragma once
#include "kernels.cuh"
#include "launch_util.h"
#include "site_contract.cuh"

namespace p2 {
namespace site {

constexpr int kRoles = 16;
template <typename R>
struct Cfg {
  static constexpr int kS = sizeof(R) == 4 ? 32 : 16;  // sites per tile
  static constexpr int kTh = kRoles * kS;
  static constexpr int kWarps = kTh / 32;
  static constexpr int kOutStride = kS + 1;  // odd: reads of consecutive positions of one site hit all banks
  static constexpr int kTileBytes = 32 * 9 * kS * (int)sizeof(Cx<R>);
};

// ---- sums over x -----------------------------------------------------------------
// [Lx][phase_stride(RT)]
template <typename R>
struct __align__(16) XPhases {
  R t[kRowsMaxPhases];
};
__host__ __device__ constexpr int phase_stride(int RT) { return (RT + 3) / 4 * 4; }

// Sums of one output position for N units of phase rows: FP32 a unit is a
// packed pair of rows (one paired FMA for both), FP64 one row.  FP32 sums take
// four sites at a time, whose sum is formed first (kSumGroup in kernels.cuh
// says why; it costs an addition per sum and four sites).
template <typename R, int N>
struct RowSums;
template <int N>
struct RowSums<float, N> {
  static constexpr int kRows = 2;  // rows per unit
  f32x2 re[N], im[N];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < N; i++) re[i] = im[i] = f2pack(0.f, 0.f);
  }
  // sites v[0..4) with the phases f[j * stride]; the first m of them (the others' values are zero)
  __device__ __forceinline__ void add4(const float* f, int stride, const Cx<float> (&v)[4], int m = 4) {
    f32x2 a[N], b[N];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const unsigned long long* q = reinterpret_cast<const unsigned long long*>(f + min(j, m - 1) * stride);
      const f32x2 vx = f2pack(v[j].x, v[j].x), vy = f2pack(v[j].y, v[j].y);
#pragma unroll
      for (int i = 0; i < N; i++) {
        a[i] = j ? f2fma(q[i], vx, a[i]) : f2mul(q[i], vx);
        b[i] = j ? f2fma(q[i], vy, b[i]) : f2mul(q[i], vy);
      }
    }
#pragma unroll
    for (int i = 0; i < N; i++) {
      re[i] = f2add(re[i], a[i]);
      im[i] = f2add(im[i], b[i]);
    }
  }
  __device__ __forceinline__ void write(Cx<float>* o, int row, int R1, long long K) {
#pragma unroll
    for (int i = 0; i < N; i++) {
      float a, b, c, d;
      f2unpack(re[i], a, b);
      f2unpack(im[i], c, d);
      const int r = row + 2 * i;
      if (r < R1) o[(long long)r * K] = cx<float>(a, c);
      if (r + 1 < R1) o[(long long)(r + 1) * K] = cx<float>(b, d);
    }
    clear();
  }
};
template <int N>
struct RowSums<double, N> {
  static constexpr int kRows = 1;
  Cx<double> s[N];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < N; i++) s[i] = czero<double>();
  }
  __device__ __forceinline__ void add(const double* f, Cx<double> v) {
#pragma unroll
    for (int i = 0; i < N; i++) {
      s[i].x = fma(f[i], v.x, s[i].x);
      s[i].y = fma(f[i], v.y, s[i].y);
    }
  }
  __device__ __forceinline__ void add4(const double* f, int stride, const Cx<double> (&v)[4]) {
#pragma unroll
    for (int j = 0; j < 4; j++) add(f + j * stride, v[j]);
  }
  __device__ __forceinline__ void write(Cx<double>* o, int row, int R1, long long K) {
#pragma unroll
    for (int i = 0; i < N; i++)
      if (row + i < R1) o[(long long)(row + i) * K] = s[i];
    clear();
  }
};
// units of a thread when `share` threads split the RT rows of a position
template <typename R>
constexpr int row_units(int RT, int share) {
  return ((sizeof(R) == 4 ? (RT + 1) / 2 : RT) + share - 1) / share;
}

// A CTA's walk over units of a.unit whole rows (the last unit of a slice
// fewer), each in tiles of up to kS consecutive sites.  The units of all slices
// are numbered through and a CTA takes every gridDim.x-th.
// Split form: the sites that are added together (add_x) are the fours of the
// slice's sites within a row, and a tile ends with one, so that their sum is
// never carried from tile to tile: that made the kernels 4 to 12 % slower (in
// registers by spills, in shared memory by a smaller L1, in the result by the
// loads).  Only a unit's first tile is shorter by it, by up to three sites.
template <typename R>
struct Cursor {
  static constexpr int kS = Cfg<R>::kS;
  int tl, unit, x0, n;  // slice, unit, first site of the tile in the slice, sites of the tile
  int row, x;           // of the first site
  __device__ __forceinline__ int end(const ContractArgs& a) const { return min(a.V3, (unit + 1) * a.unit * a.Lx); }
  __device__ __forceinline__ void fit(const ContractArgs& a) {
    const int left = end(a) - x0;
    n = min(kS - (sizeof(R) == 4 ? x0 & 3 : 0), left);
  }
  __device__ __forceinline__ void place(const ContractArgs& a) {
    row = unit * a.unit;
    x = 0;
    x0 = row * a.Lx;
    fit(a);
  }
  __device__ __forceinline__ void first(const ContractArgs& a) {
    tl = (int)(blockIdx.x / (unsigned)a.upt);
    unit = (int)(blockIdx.x % (unsigned)a.upt);
    place(a);
  }
  __device__ __forceinline__ bool valid(const ContractArgs& a) const { return tl < a.ntau; }
  __device__ __forceinline__ void next(const ContractArgs& a) {
    if (x0 + n < end(a)) {
      x0 += n;
      for (x += n; x >= a.Lx; x -= a.Lx) row++;
      fit(a);
    } else {  // gridDim.x units further, without a division
      tl += a.step_slice;
      unit += a.step_unit;
      if (unit >= a.upt) {
        unit -= a.upt;
        tl++;
      }
      place(a);
    }
  }
};

// Adds the tile's values of one output position (val(s), sites 0..n-1) into
// its sums for the phase rows from `first` on, writing every x row that ends.
template <typename R, int RT, int N, typename Val>
__device__ __forceinline__ void add_x(const ContractArgs& a, const R* ph, RowSums<R, N>& acc, int first,
                                      const Cursor<R>& c, int k, Val&& val) {
  constexpr int kStride = phase_stride(RT);
  const int rows = a.V3 / a.Lx;
  int row = c.row, x = c.x, s = 0;
  while (s < c.n) {
    const int end = min(c.n, s + a.Lx - x);  // the sites of this row
    const R* f = ph + x * kStride + first;
    x += end - s;
    if constexpr (sizeof(R) == 4) {
      // one to three sites before the first of the slice's fours, and after the last
      auto some = [&](int m) {
        Cx<R> v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = i < m ? val(s + i) : czero<R>();
        acc.add4(f, kStride, v, m);
        s += m;
        f += m * kStride;
      };
      const int head = min(end - s, -(c.x0 + s) & 3);
      if (head) some(head);
#pragma unroll 1
      for (; s + 4 <= end; s += 4, f += 4 * kStride) {
        Cx<R> v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = val(s + i);
        acc.add4(f, kStride, v);
      }
      if (s < end) some(end - s);
    } else {
#pragma unroll 1
      for (; s + 4 <= end; s += 4, f += 4 * kStride) {
        Cx<R> v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = val(s + i);
        acc.add4(f, kStride, v);
      }
#pragma unroll 1
      for (; s < end; s++, f += kStride) acc.add(f, val(s));
    }
    if (x == a.Lx) {
      acc.write((Cx<R>*)a.out + ((long long)c.tl * rows + row) * a.R1 * a.K + k, first, a.R1, a.K);
      x = 0;
      row++;
    }
  }
}

// ---- the tile ----------------------------------------------------------------------
// FP32: four colour pairs as 16-byte units [block][4][sites], then colour 8
// [block][sites]; FP64: [block][9][sites].  Blocks 16 f + 4 mu + nu.
template <typename R>
struct Tile;
template <>
struct Tile<float> {
  static constexpr int kS = Cfg<float>::kS;
  float4* q;
  Cx<float>* last;
  __device__ __forceinline__ Tile(unsigned char* sm, int site)
      : q((float4*)sm + site), last((Cx<float>*)((float4*)sm + 32 * 4 * kS) + site) {}
  __device__ __forceinline__ void load9(int blk, Cx<float> (&v)[9]) const {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float4 x = q[(blk * 4 + k) * kS];
      v[2 * k] = cx<float>(x.x, x.y);
      v[2 * k + 1] = cx<float>(x.z, x.w);
    }
    v[8] = last[blk * kS];
  }
  __device__ __forceinline__ void store9(int blk, const Cx<float> (&v)[9]) const {
#pragma unroll
    for (int k = 0; k < 4; k++) q[(blk * 4 + k) * kS] = make_float4(v[2 * k].x, v[2 * k].y, v[2 * k + 1].x, v[2 * k + 1].y);
    last[blk * kS] = v[8];
  }
  __device__ __forceinline__ void put(int blk, int col, Cx<float> v) const {
    Cx<float>* o = col == 8 ? last + blk * kS : (Cx<float>*)(q + (blk * 4 + (col >> 1)) * kS) + (col & 1);
    *o = v;
  }
};
template <>
struct Tile<double> {
  static constexpr int kS = Cfg<double>::kS;
  Cx<double>* p;
  __device__ __forceinline__ Tile(unsigned char* sm, int site) : p((Cx<double>*)sm + site) {}
  __device__ __forceinline__ void load9(int blk, Cx<double> (&v)[9]) const {
#pragma unroll
    for (int i = 0; i < 9; i++) v[i] = p[(blk * 9 + i) * kS];
  }
  __device__ __forceinline__ void store9(int blk, const Cx<double> (&v)[9]) const {
#pragma unroll
    for (int i = 0; i < 9; i++) p[(blk * 9 + i) * kS] = v[i];
  }
  __device__ __forceinline__ void put(int blk, int col, Cx<double> v) const { p[(blk * 9 + col) * kS] = v; }
};

// Fills one flavour of the tile: load() takes a role's share into registers, so
// that other work can cover the latency, store() converts it.  A role's share
// is a spin block (its column of nine colours); a rotated slice (prop_xf_code)
// mixes the blocks b, b + 2, b + 8, b + 10 and is shared out as 36 groups of
// them, two to a role and the last four to roles 0..3.  g5 from the left is a
// permutation of the blocks, the sign a factor.
template <typename R, typename Tin>
struct Loader {
  static constexpr int kS = Cfg<R>::kS;
  Cx<Tin> raw[9];
  const Cx<Tin>* p;  // colour 0 of block 0 at this site
  long long vol;
  int xf, f;

  __device__ __forceinline__ void group(int g, int i0) {
    const Cx<Tin>* q = p + (9 * ((g / 18) * 4 + (g / 9 & 1)) + g % 9) * vol;
#pragma unroll
    for (int i = 0; i < 4; i++) raw[i0 + i] = q[9 * group_blk(i) * vol];
  }
  __device__ __forceinline__ void put_group(const Tile<R>& t, int g, int i0, double sc) {
    Cx<double> v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = cx<double>((double)raw[i0 + i].x, (double)raw[i0 + i].y);
    prop_group_transform(v[0], v[1], v[2], v[3], xf);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (sizeof(R) == 4) v[i] = cscale(v[i], sc);
      t.put(16 * f + (g / 18) * 4 + (g / 9 & 1) + group_blk(i), g % 9, cx<R>((R)v[i].x, (R)v[i].y));
    }
  }
  // sites past the tile's last one read the first (their sums are not used)
  __device__ __forceinline__ void load(const ContractArgs& a, const Cursor<R>& c, int flavour, int role, int site) {
    if (!c.valid(a)) return;
    const SliceDesc* sd = a.sl + c.tl;
    f = flavour;
    vol = f ? sd->vol_d : sd->vol_u;
    p = (const Cx<Tin>*)(f ? sd->d : sd->u) + (f ? sd->off_d : sd->off_u) + c.x0 + (site < c.n ? site : 0);
    xf = sd->xf[f];
    if (xf & 3) {
      group(role, 0);
      group(role + kRoles, 4);
    } else {
      const Cx<Tin>* q = p + 9 * (role ^ (xf & 4 ? 8 : 0)) * vol;
#pragma unroll
      for (int i = 0; i < 9; i++) raw[i] = q[i * vol];
    }
  }
  // split form: scaled by 2^-E (in double: exact, no intermediate leaves the range)
  __device__ __forceinline__ void store(const ContractArgs& a, const Cursor<R>& c, const Tile<R>& t, int role) {
    if (!c.valid(a)) return;
    double sc = 1.0;
    if (sizeof(R) == 4) {
      const int E = a.exps[2 * c.tl + f];
      sc = abs(E) < 1000 ? __longlong_as_double((long long)(1023 - E) << 52) : ldexp(1.0, -E);
    }
    if (xf & 3) {
      put_group(t, role, 0, sc);
      put_group(t, role + kRoles, 4, sc);
      if (role + 2 * kRoles < 36) {
        group(role + 2 * kRoles, 0);
        put_group(t, role + 2 * kRoles, 0, sc);
      }
    } else {
      if (xf & 8) sc = -sc;
      Cx<R> v[9];
#pragma unroll
      for (int i = 0; i < 9; i++) v[i] = cx<R>((R)((double)raw[i].x * sc), (R)((double)raw[i].y * sc));
      t.store9(16 * f + role, v);
    }
  }
};

// The tile's 288 rows of kS sites into L2; a role takes its block of both flavours.
template <typename R, typename Tin>
__device__ __forceinline__ void prefetch(const ContractArgs& a, const Cursor<R>& c, int role, int site) {
  if (!c.valid(a)) return;
  constexpr int kS = Cfg<R>::kS, kLine = 128 / (int)sizeof(Cx<Tin>), kLines = kS / kLine;  // sites per line, lines per row
  const SliceDesc* sd = a.sl + c.tl;
#pragma unroll
  for (int f = 0; f < 2; f++) {
    const long long vol = f ? sd->vol_d : sd->vol_u;
    const Cx<Tin>* p =
        (const Cx<Tin>*)(f ? sd->d : sd->u) + (f ? sd->off_d : sd->off_u) + c.x0 + 9 * role * vol;
    for (int l = site; l < 9 * kLines; l += kS) {
      const int s = (l % kLines) * kLine;
      if (s < c.n) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + (l / kLines) * vol + s));
    }
  }
}

// The warp's number, known to the compiler to be the same in all lanes: what
// derives from it (shares of the phase rows, roles of the split form) stays in
// uniform registers, and the phases are read as uniform constants.
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }
// thread = (role, site)
template <typename R>
__device__ __forceinline__ int role_of(int warp) {
  constexpr int kS = Cfg<R>::kS;
  return kS == 32 ? warp : warp * (32 / kS) + ((int)threadIdx.x & 31) / kS;
}
// Barrier of the warps that hold some of the roles (ids 1.. ; 0 is __syncthreads)
__device__ __forceinline__ void warps_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// acc = sum over the nine colours; FP64 in three partial sums (cdot9)
template <typename R>
__device__ __forceinline__ Cx<R> dot_conj(const Cx<R> (&u)[9], const Cx<R> (&d)[9]) {
  constexpr int N = sizeof(R) == 8 ? 3 : 1;
  Cx<R> m[N];
#pragma unroll
  for (int i = 0; i < N; i++) m[i] = czero<R>();
#pragma unroll
  for (int i = 0; i < 9; i++) cmac_conj(m[i % N], u[i], d[i]);
  if constexpr (N == 3) m[0] = m[0] + m[1] + m[2];
  return m[0];
}

// q += SG eps eps x y
template <int SG, typename R>
__device__ __forceinline__ void diquark_add(const Cx<R> (&x)[9], const Cx<R> (&y)[9], Cx<R> (&q)[9]) {
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
#pragma unroll
    for (int e = 0; e < 3; e++) {
      const int e1 = (e + 1) % 3, e2 = (e + 2) % 3;
      Cx<R>& r = q[c * 3 + e];
      if (SG > 0) {
        cmac(r, x[c1 * 3 + e1], y[c2 * 3 + e2]);
        cmsub(r, x[c1 * 3 + e2], y[c2 * 3 + e1]);
        cmsub(r, x[c2 * 3 + e1], y[c1 * 3 + e2]);
        cmac(r, x[c2 * 3 + e2], y[c1 * 3 + e1]);
      } else {
        cmsub(r, x[c1 * 3 + e1], y[c2 * 3 + e2]);
        cmac(r, x[c1 * 3 + e2], y[c2 * 3 + e1]);
        cmac(r, x[c2 * 3 + e1], y[c1 * 3 + e2]);
        cmsub(r, x[c2 * 3 + e2], y[c1 * 3 + e1]);
      }
    }
  }
}

// xt: [Lx][R1] phase rows; one CTA per SM (its shared memory and registers fill it)
template <typename R, typename K>
cudaError_t launch_tiles(K kernel, const ContractArgs& a0, const double* xt, int RT, int smem, int nsm,
                         cudaStream_t s) {
  constexpr int kS = Cfg<R>::kS;
  ContractArgs a = a0;
  const int stride = phase_stride(RT);
  if (a.Lx * stride > kRowsMaxPhases || a.R1 > RT) return cudaErrorInvalidValue;
  XPhases<R> ph;
  for (int i = 0; i < a.Lx; i++)
    for (int r = 0; r < stride; r++) ph.t[i * stride + r] = r < a.R1 ? (R)xt[i * a.R1 + r] : R(0);
  // rows per unit: the fewest tiles per CTA, the smaller unit on a tie (a unit
  // of several rows fills its last tile better, fewer units balance worse)
  const int rows = a.V3 / a.Lx;
  long long best = -1;
  for (int m = 1; m <= kS && m <= rows; m++) {
    const long long units = (long long)((rows + m - 1) / m) * a.ntau;
    const int cut = sizeof(R) == 4 && m * a.Lx % 4 ? 3 : 0;  // of a unit's first tile
    const long long cost = (units + nsm - 1) / nsm * ((m * a.Lx + cut + kS - 1) / kS);
    if (best < 0 || cost < best) {
      best = cost;
      a.unit = m;
    }
  }
  a.upt = (rows + a.unit - 1) / a.unit;
  const long long units = (long long)a.upt * a.ntau;
  const unsigned grid = (unsigned)(units < nsm ? units : nsm);
  a.step_slice = (int)(grid / (unsigned)a.upt);
  a.step_unit = (int)(grid % (unsigned)a.upt);
  cudaError_t e = ensure_smem((const void*)kernel, smem);
  if (e != cudaSuccess) return e;
  kernel<<<grid, Cfg<R>::kTh, smem, s>>>(a, ph);
  return cudaGetLastError();
}

}  // namespace site
}  // namespace p2
