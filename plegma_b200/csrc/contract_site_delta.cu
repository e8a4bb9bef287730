// Delta C g_k (both isospins), one site per lane, fused with the sums over x
// (contract_site.cuh).
//
// The sums are those of delta_site (site_contract.cuh): for a flavour pair p
// and the symmetric diquarks G_g(r, s),
//   T[g, Z][m][r] = 4 sum_s s_g(s) G_g(r, s) . Z[m][z_g(s)] + 2 D_g . Z[m][r],
//   D_g = sum_s s_g(s) G_g(z_g(s), s).
// G_g(r, s) = G_g(s, r), so a role takes an unordered pair {r, s}, serving
// T[.][r] and T[.][s] with one diquark (10 diquarks where the lanes of a
// half-warp form 16): roles 0..5 the six with r < s for C g_1 and C g_2
// together (they share their products and z(s) = s, so each load of Z serves
// both), roles 6..11 the same six for C g_3, roles 12..15 the diagonal ones
// for all three.  D_g is a slot term too: z_g(s) = r in T[.][r] exactly for the
// diquarks that D_g sums over (the diagonal ones; {0, 1} and {2, 3} for C g_3),
// so their roles form D_g among themselves and add s_g D_g / 2 to their
// diquark before its slot terms.  Per flavour pair:
//   A   the role's diquarks, its slot terms to sP
//   B   role (r, m): the sums of four slot terms of every g and Z, in registers
// and after the three pairs the outputs to the output tile and, X, the sums
// over x.
// Bound: FMA issue and, in A, the shared-memory loads (18 wavefronts of a
// block against 36 issue slots of the dots it feeds): split form 1791 clk/site
// with 3897 warp instructions and 1024 wavefronts; plain form 3357 clk/site,
// FP64 pipe 47 %.  At 128 registers the split form with FP64 propagators and
// seven rows spills 332 bytes a thread, with FP32 propagators 104, the plain form at
// 255 registers 368 (the outputs o, the row sums and the next tile's nine values live through a flavour pair).
#include "contract_site.cuh"

namespace p2 {
namespace site {
namespace {

constexpr int kOut = 192;  // iso-1/2 0..95, iso-3/2 96..191
constexpr int kP3 = 256;   // entries of C g_1, C g_2 in sP: [r][4 contributions][g, Z, m]; then C g_3: [r][4][Z, m]
template <typename R>
struct Mem {
  static constexpr int kP = (kP3 + 128) * Cfg<R>::kS * (int)sizeof(Cx<R>);
  static constexpr int kD = (72 + 18) * Cfg<R>::kS * (int)sizeof(Cx<R>);  // parts of D_g: [4][g][9], C g_3 [2][9]
  static constexpr int kAll = Cfg<R>::kTileBytes + kP + kD;
  static_assert(kAll <= 232448 && kOut * Cfg<R>::kOutStride * (int)sizeof(Cx<R>) <= kP, "shared memory of a CTA");
};

// Source tables as used below: z(s) = s for C g_1 and C g_2, s ^ 1 for C g_3
__host__ __device__ constexpr int delta_sign(int g, int s) {
  return g == 0 ? (s == 0 || s == 3 ? 1 : -1) : (s < 2 ? 1 : -1);
}
constexpr bool delta_tables_ok() {
  for (int g = 0; g < 3; g++)
    for (int s = 0; s < 4; s++)
      if (kDeltaLane[g][s][0] != (g == 2 ? s ^ 1 : s) || kDeltaLane[g][s][1] != delta_sign(g, s)) return false;
  for (int i = 0; i < 4; i++) {
    if (kDeltaSink[0][i][0] != i || kDeltaSink[0][i][1] != i || kDeltaSink[0][i][2] != (i == 0 || i == 3 ? 1 : -1) ||
        kDeltaSink[1][i][0] != i || kDeltaSink[1][i][1] != i || kDeltaSink[1][i][2] != (i < 2 ? 1 : -1) ||
        kDeltaSink[2][i][0] != i || kDeltaSink[2][i][1] != (i ^ 1) || kDeltaSink[2][i][2] != (i < 2 ? 1 : -1))
      return false;
  }
  return true;
}
static_assert(delta_tables_ok() && delta_sign(2, 0) == delta_sign(2, 1) && delta_sign(2, 2) == delta_sign(2, 3) && delta_lane_symmetric(kDeltaLane[0]) && delta_lane_symmetric(kDeltaLane[1]) &&
                  delta_lane_symmetric(kDeltaLane[2]),
              "Delta tables in another form");

// q += SG eps eps X[xb] Y[yb]
template <int SG, typename R>
__device__ __forceinline__ void product(const Tile<R>& t, int xb, int yb, Cx<R> (&q)[9]) {
  asm volatile("" ::: "memory");  // keeps the loads of later products from being moved up (registers)
  Cx<R> x[9], y[9];
  t.load9(xb, x);
  t.load9(yb, y);
  diquark_add<SG>(x, y, q);
}

// C g_1 and C g_2 of the pair {r, s} (r = s: the diagonal one)
template <typename R>
__device__ __forceinline__ void pair_g12(const Tile<R>& t, int p, int X, int Y, int r, int s, Cx<R>* sP,
                                         Cx<R>* sD) {
  constexpr int kS = Cfg<R>::kS;
  const bool diag = r == s;
  Cx<R> G[2][9];
#pragma unroll
  for (int i = 0; i < 9; i++) G[0][i] = G[1][i] = czero<R>();
#pragma unroll 1
  for (int o = 0; o < (p == 1 && !diag ? 2 : 1); o++) {
    const int xs = X + (o ? s : r), ys = Y + (o ? r : s);
    product<1>(t, xs, ys, G[0]);
    product<-1>(t, xs + 8, ys + 8, G[0]);
    product<1>(t, xs + 4, ys + 4, G[1]);
    product<-1>(t, xs + 12, ys + 12, G[1]);
  }
  const R f = p == 1 && diag ? R(2) : R(1);
#pragma unroll
  for (int i = 0; i < 9; i++) {
    const Cx<R> v = G[0][i];
    G[0][i] = cscale(v - G[1][i], f);
    G[1][i] = cscale(v + G[1][i], f);
  }
  if (diag) {
    const R f0 = (R)delta_sign(0, r), f1 = (R)delta_sign(1, r);
#pragma unroll
    for (int i = 0; i < 9; i++) {
      sD[((r * 2 + 0) * 9 + i) * kS] = cscale(G[0][i], R(0.5) * f0);
      sD[((r * 2 + 1) * 9 + i) * kS] = cscale(G[1][i], R(0.5) * f1);
    }
    warps_sync(1, 4 * kS);
#pragma unroll
    for (int g = 0; g < 2; g++)
#pragma unroll
      for (int i = 0; i < 9; i++) {
        const Cx<R>* d = sD + (g * 9 + i) * kS;
        G[g][i] = G[g][i] + cscale((d[0] + d[18 * kS]) + (d[36 * kS] + d[54 * kS]), g ? f1 : f0);
      }
  }
#pragma unroll 1
  for (int o = 0; o < (diag ? 1 : 2); o++) {  // target r with the line's spin s, then the reverse
    const int tr = o ? s : r, ts = o ? r : s;
    const R f0 = (R)delta_sign(0, ts), f1 = (R)delta_sign(1, ts);
#pragma unroll 1
    for (int z = 0; z < 2; z++) {
      Cx<R>* d = sP + ((tr * 4 + ts) * 16 + 4 * z) * kS;
#pragma unroll
      for (int m = 0; m < 4; m++) {
        Cx<R> v[9], p0 = czero<R>(), p1 = p0;
        t.load9(16 * z + 4 * m + ts, v);
        cdot9_acc(p0, G[0], v);
        cdot9_acc(p1, G[1], v);
        d[m * kS] = cscale(p0, f0);
        d[(8 + m) * kS] = cscale(p1, f1);
      }
    }
  }
}

// C g_3 of the pair {r, s}
template <typename R>
__device__ __forceinline__ void pair_g3(const Tile<R>& t, int p, int X, int Y, int r, int s, Cx<R>* sP,
                                        Cx<R>* sD) {
  constexpr int kS = Cfg<R>::kS;
  const bool diag = r == s;
  Cx<R> G[9];
#pragma unroll
  for (int i = 0; i < 9; i++) G[i] = czero<R>();
  // P_{01} - P_{23} of (r, s) and (s, r); for ud also P_{10} - P_{32}
#pragma unroll 1
  for (int o = 0; o < (p == 1 ? 4 : 2); o += diag ? 2 : 1) {
    const int xs = X + ((o & 1) ? s : r) + (o & 2 ? 4 : 0), ys = Y + ((o & 1) ? r : s) + (o & 2 ? 0 : 4);
    product<1>(t, xs, ys, G);
    product<-1>(t, xs + 8, ys + 8, G);
  }
  // {0, 1}, {2, 3}, whose two slot signs are equal: s (G(r, s) + G(s, r)) / 2
  const bool cls = r == (s ^ 1);
  if (kS == 32 ? cls : __any_sync(0xffffffffu, cls)) {
    const R f = (R)delta_sign(2, s);
    if (cls) {
#pragma unroll
      for (int i = 0; i < 9; i++) sD[(72 + (r >> 1) * 9 + i) * kS] = cscale(G[i], f);
    }
    warps_sync(2, 64);  // the two warps that hold these roles
    if (cls) {
#pragma unroll
      for (int i = 0; i < 9; i++) G[i] = G[i] + cscale(sD[(72 + i) * kS] + sD[(81 + i) * kS], f);
    }
  }
  const R f2 = diag ? R(2) : R(1);
#pragma unroll 1
  for (int o = 0; o < (diag ? 1 : 2); o++) {
    const int tr = o ? s : r, ts = o ? r : s;
    const R f = f2 * (R)delta_sign(2, ts);
#pragma unroll 1
    for (int z = 0; z < 2; z++) {
      Cx<R>* d = sP + (kP3 + (tr * 4 + ts) * 8 + 4 * z) * kS;
#pragma unroll
      for (int m = 0; m < 4; m++) {
        Cx<R> v[9], p0 = czero<R>();
        t.load9(16 * z + 4 * m + (ts ^ 1), v);
        cdot9_acc(p0, G, v);
        d[m * kS] = cscale(p0, f);
      }
    }
  }
}

template <typename R, typename Tin, int RT>
__global__ void __launch_bounds__(Cfg<R>::kTh, 1)
    k_site_delta(const ContractArgs a, const __grid_constant__ XPhases<R> ph) {
  constexpr int kS = Cfg<R>::kS, kOutStride = Cfg<R>::kOutStride;
  extern __shared__ __align__(16) unsigned char sm[];
  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid % kS, w = role_of<R>(warp);  // site, role
  const Tile<R> t(sm, lane);
  Cx<R>* const so = (Cx<R>*)(sm + Cfg<R>::kTileBytes);  // output tile, over sP
  Cx<R>* const sP = so + lane;
  Cx<R>* const sD = (Cx<R>*)(sm + Cfg<R>::kTileBytes + Mem<R>::kP) + lane;
  // the pair of roles 0..11, the diagonal of roles 12..15
  const int i6 = w < 6 ? w : w - 6;
  const int r = w >= 12 ? w - 12 : i6 < 3 ? 0 : i6 < 5 ? 1 : 2;
  const int s = w >= 12 ? r : i6 < 3 ? i6 + 1 : i6 < 5 ? i6 - 1 : 3;
  // sums over x: position tid % 192, share warp / 6 of the phase rows
  constexpr int kShare = Cfg<R>::kTh / kOut, NU = row_units<R>(RT, kShare);
  RowSums<R, NU> acc;
  acc.clear();

  Cursor<R> cur, nx;
  cur.first(a);
#pragma unroll 1
  for (int f = 0; f < 2; f++) {
    Loader<R, Tin> ld;
    ld.load(a, cur, f, w, lane);
    ld.store(a, cur, t, w);
  }
  __syncthreads();
  for (; cur.valid(a); cur = nx) {
    nx = cur;
    nx.next(a);
    prefetch<R, Tin>(a, nx, w, lane);
    // outputs of (m, r) = (w & 3, w >> 2): o[g][j], j = 0 Delta+, 1 Delta0, 2 Delta++, 3 Delta-
    Cx<R> o[3][4];
#pragma unroll 1
    for (int p = 0; p < 3; p++) {
      const int X = p == 2 ? 16 : 0, Y = p == 0 ? 0 : 16;
      if (w < 6 || w >= 12) pair_g12(t, p, X, Y, r, s, sP, sD);
      if (w >= 6) pair_g3(t, p, X, Y, r, s, sP, sD);
      __syncthreads();
      const int mr = w >> 2, mm = w & 3;
      Cx<R> x[2][3];  // [Z][g]
#pragma unroll
      for (int z = 0; z < 2; z++)
#pragma unroll
        for (int g = 0; g < 3; g++) {
          const Cx<R>* src = g < 2 ? sP + (mr * 64 + 8 * g + 4 * z + mm) * kS : sP + (kP3 + mr * 32 + 4 * z + mm) * kS;
          const int st = (g < 2 ? 16 : 8) * kS;
          x[z][g] = (src[0] + src[st]) + (src[2 * st] + src[3 * st]);
        }
      // uu feeds Delta++ (Z = u) and Delta+ (Z = d), ud + du Delta+ and Delta0, dd Delta0 and Delta-
#pragma unroll
      for (int g = 0; g < 3; g++) {
        if (p == 0) {
          o[g][2] = cscale(x[0][g], R(4));
          o[g][0] = x[1][g];
        } else if (p == 1) {
          o[g][0] = cscale(o[g][0] + x[0][g], R(4) / R(3));
          o[g][1] = x[1][g];
        } else {
          o[g][1] = cscale(o[g][1] + x[0][g], R(4) / R(3));
          o[g][3] = cscale(x[1][g], R(4));
        }
      }
      __syncthreads();  // sP, sD and (last pair) the tile are read
    }
    Loader<R, Tin> ld;
    ld.load(a, nx, 0, w, lane);
#pragma unroll
    for (int g = 0; g < 3; g++)
#pragma unroll
      for (int j = 0; j < 4; j++)
        so[((j >= 2 ? 96 : 0) + (g * 2 + (j & 1)) * 16 + 4 * (w & 3) + (w >> 2)) * kOutStride + lane] = o[g][j];
    __syncthreads();
    // ---- X, with the next tile's d half in flight ----
    ld.store(a, nx, t, w);
    ld.load(a, nx, 1, w, lane);
    {
      const int share = warp / (kOut / 32), pos = tid % kOut;
      if (share < kShare && (a.what & (pos < 96 ? 2u : 4u)))
        add_x<R, RT>(a, ph.t, acc, share * NU * decltype(acc)::kRows, cur, pos < 96 ? a.k.diso12 + pos : a.k.diso32 + pos - 96,
                        [&](int i) { return so[pos * kOutStride + i]; });
    }
    ld.store(a, nx, t, w);
    __syncthreads();
  }
}

template <typename R, typename Tin, int RT>
cudaError_t go(const ContractArgs& a, const double* xt, int nsm, cudaStream_t s) {
  return launch_tiles<R>(k_site_delta<R, Tin, RT>, a, xt, RT, Mem<R>::kAll, nsm, s);
}

template <typename R, typename Tin>
cudaError_t go_rows(const ContractArgs& a, const double* xt, int nsm, cudaStream_t s) {
  return a.R1 <= 3   ? go<R, Tin, 3>(a, xt, nsm, s)
         : a.R1 <= 7 ? go<R, Tin, 7>(a, xt, nsm, s)
                     : go<R, Tin, 9>(a, xt, nsm, s);
}

}  // namespace
}  // namespace site

cudaError_t launch_site_delta(const ContractArgs& a, const double* xt, int plain, int fp32_in, int nsm,
                              cudaStream_t s) {
  if (plain) return site::go_rows<double, double>(a, xt, nsm, s);
  return fp32_in ? site::go_rows<float, float>(a, xt, nsm, s) : site::go_rows<float, double>(a, xt, nsm, s);
}

}  // namespace p2
