// Nucleon C g5 and the 16 x 16 mesons (their colour products M; k_meson_gamma
// forms the Gamma sums after the projection), one site per lane, fused with
// the sums over x (contract_site.cuh).
//
// Role (x', y') evaluates, for the tile's sites, what lane (x', y') of a site's
// half-warp does in site_contract.cuh: the diquark Q = G^{ud}(x', y'), its slot
// terms, and the products M_{al de}[x'][y'] = sum_colour u[al][x']
// conj(d[de][y']), which need the same eight blocks u[.][x'], d[.][y'] as Q, so
// one load of them serves both.  The sums over lanes of the half-warp form
// become sums over roles through shared memory:
//   A   every role: Q, M to the output tile, slot terms to sT
//   B   role (m, r): the nucleon's T[m][r] of both datasets, four slot terms each
//   X   sums over x: thread (position, share of the phase rows)
// The type-a term D . Z[m][r], D = sum over the class of s Q, is a slot term
// of the class itself: z(s) = r in T[m][r] exactly for the class role (r,
// r ^ 1), so that role adds s D to its Q before its slot terms.  The four
// roles of the class form D among themselves, the others do not wait.
// Bound, split form: issue with four warps per scheduler, 668 clk/site (54 %
// of the slots, 1439 warp instructions, 296 shared-memory wavefronts); half of
// it is A.  Plain form: FP64 latency at 8 warps per SM, 1175 clk/site (FP64
// pipe 41 %).  The HBM floor is 196 clk/site.
#include "contract_site.cuh"

namespace p2 {
namespace site {
namespace {

// The nucleon's tables as used below: sink entries (nu, nu ^ 1, + for even nu),
// z(s) = s ^ 1, s(s) = - for even s, type-a class y' = x' ^ 1 with sign + for odd y'.
constexpr bool nucleon_tables_ok() {
  for (int i = 0; i < 4; i++)
    if (kNucSink[i][0] != i || kNucSink[i][1] != (i ^ 1) || kNucSink[i][2] != (i % 2 == 0 ? 1 : -1)) return false;
  for (int l = 0; l < 16; l++) {
    const int x = l >> 2, y = l & 3;
    if (kNucLane[l][0] != (y ^ 1) || kNucLane[l][1] != (y % 2 ? 1 : -1) ||
        kNucLane[l][6] != (y == (x ^ 1) ? (y % 2 ? 1 : -1) : 0))
      return false;
  }
  return true;
}
static_assert(nucleon_tables_ok(), "nucleon tables in another form");

template <typename R>
struct Mem {
  static constexpr int kOut = 288 * Cfg<R>::kOutStride * (int)sizeof(Cx<R>);
  static constexpr int kT = 16 * 8 * Cfg<R>::kS * (int)sizeof(Cx<R>);
  static constexpr int kD = 4 * 9 * Cfg<R>::kS * (int)sizeof(Cx<R>);
  static constexpr int kAll = Cfg<R>::kTileBytes + kOut + kT + kD;
  static_assert(kAll <= 232448, "shared memory of a CTA");
};

template <typename R, typename Tin, int RT>
__global__ void __launch_bounds__(Cfg<R>::kTh, 1)
    k_site_mesons(const ContractArgs a, const __grid_constant__ XPhases<R> ph) {
  constexpr int kS = Cfg<R>::kS, kOutStride = Cfg<R>::kOutStride, kWarps = Cfg<R>::kWarps;
  extern __shared__ __align__(16) unsigned char sm[];
  const int tid = threadIdx.x, warp = uniform_warp(), site = tid % kS, role = role_of<R>(warp), xp = role >> 2,
            yp = role & 3;
  const bool cls = yp == (xp ^ 1);  // type-a class
  const Tile<R> t(sm, site);
  Cx<R>* const so = (Cx<R>*)(sm + Cfg<R>::kTileBytes);
  Cx<R>* const sT = (Cx<R>*)(sm + Cfg<R>::kTileBytes + Mem<R>::kOut) + site;
  Cx<R>* const sD = (Cx<R>*)(sm + Cfg<R>::kTileBytes + Mem<R>::kOut + Mem<R>::kT) + site;
  const bool nuc = (a.what & 1u) != 0, mes = (a.what & 8u) != 0;

  // sums over x: product position tid % 256, share warp / 8 of the phase rows
  constexpr int kShare = Cfg<R>::kTh / 256, NU = row_units<R>(RT, kShare);
  RowSums<R, NU> acc;
  acc.clear();
  constexpr int kNR = (RT + kWarps - 1) / kWarps;
  Cx<R> accn[kNR];  // nucleon: component tid % 32, phase rows warp, warp + kWarps
#pragma unroll
  for (int i = 0; i < kNR; i++) accn[i] = czero<R>();
  const int rows = a.V3 / a.Lx;

  Cursor<R> cur, nx;
  cur.first(a);
#pragma unroll 1
  for (int f = 0; f < 2; f++) {
    Loader<R, Tin> ld;
    ld.load(a, cur, f, role, site);
    ld.store(a, cur, t, role);
  }
  __syncthreads();
  for (; cur.valid(a); cur = nx) {
    nx = cur;
    nx.next(a);
    prefetch<R, Tin>(a, nx, role, site);
    // ---- A ----
    {
      Cx<R> Q[9];
#pragma unroll
      for (int i = 0; i < 9; i++) Q[i] = czero<R>();
      // two d blocks at a time (four do not fit beside u and Q)
#pragma unroll
      for (int dh = 0; dh < 2; dh++) {
        Cx<R> d[2][9];
        t.load9(16 + 8 * dh + yp, d[0]);
        t.load9(16 + 8 * dh + 4 + yp, d[1]);
#pragma unroll
        for (int nu = 0; nu < 4; nu++) {
          asm volatile("" ::: "memory");  // keeps the loads of later blocks from being moved up (registers)
          Cx<R> u[9];
          t.load9(4 * nu + xp, u);
          if (mes) {
#pragma unroll
            for (int de = 0; de < 2; de++)
              so[(16 * (4 * nu + 2 * dh + de) + role) * kOutStride + site] = dot_conj(u, d[de]);
          }
          if (nuc && nu / 2 == dh) {  // the sink entry (nu, nu ^ 1)
            if (nu % 2 == 0)
              diquark_add<1>(u, d[1], Q);
            else
              diquark_add<-1>(u, d[0], Q);
          }
        }
      }
      if (nuc) {
        // slot terms: proton s(y') Q . u[m][z(y')], neutron -s(x') Q . d[m][z(x')]
        const R s1 = (yp & 1) ? R(1) : R(-1), s2 = (xp & 1) ? R(-1) : R(1);
        // (equal signs in the class: y' = x' ^ 1)
        if (kS == 32 ? cls : __any_sync(0xffffffffu, cls)) {
          if (cls) {
#pragma unroll
            for (int i = 0; i < 9; i++) sD[(xp * 9 + i) * kS] = cscale(Q[i], s1);
          }
          warps_sync(1, 128);  // four warps hold a class role
          if (cls) {
#pragma unroll
            for (int i = 0; i < 9; i++)
              Q[i] = Q[i] + cscale((sD[i * kS] + sD[(9 + i) * kS]) + (sD[(18 + i) * kS] + sD[(27 + i) * kS]), s1);
          }
        }
#pragma unroll
        for (int f = 0; f < 2; f++) {
#pragma unroll
          for (int m = 0; m < 4; m++) {
            asm volatile("" ::: "memory");
            Cx<R> z[9], q = czero<R>();
            t.load9(16 * f + 4 * m + ((f ? xp : yp) ^ 1), z);
            cdot9_acc(q, Q, z);
            sT[(role * 8 + 4 * f + m) * kS] = cscale(q, f ? s2 : s1);
          }
        }
      }
    }
    __syncthreads();
    Loader<R, Tin> ld;
    ld.load(a, nx, 0, role, site);
    if (nuc) {
      // ---- B: (m, r) = (xp, yp) ----
      Cx<R> t1[4], t2[4];
#pragma unroll
      for (int s = 0; s < 4; s++) {
        t1[s] = sT[((yp * 4 + s) * 8 + xp) * kS];
        t2[s] = sT[((s * 4 + yp) * 8 + 4 + xp) * kS];
      }
      so[(256 + role) * kOutStride + site] = (t1[0] + t1[1]) + (t1[2] + t1[3]);
      so[(272 + role) * kOutStride + site] = (t2[0] + t2[1]) + (t2[2] + t2[3]);
    }
    __syncthreads();  // the outputs are complete and the tile is dead
    // ---- X, with the next tile's d half in flight ----
    ld.store(a, nx, t, role);
    ld.load(a, nx, 1, role, site);
    if (mes)
      add_x<R, RT>(a, ph.t, acc, warp / 8 * NU * decltype(acc)::kRows, cur, a.k.g16 + tid % 256,
                   [&](int s) { return so[(tid % 256) * kOutStride + s]; });
    if (nuc) {
      const int lane = tid & 31, w = warp;
      int row = cur.row, x = cur.x, s = 0;
      const Cx<R>* src = so + (256 + lane) * kOutStride;
      while (s < cur.n) {
        const int end = min(cur.n, s + a.Lx - x);
        if constexpr (sizeof(R) == 4) {
          // fours as in add_x
          auto some = [&](int m) {
            Cx<R> g = czero<R>();
#pragma unroll
            for (int i = 0; i < 4; i++)
              if (i < m && w < RT) {
                const Cx<R> v = src[s + i];
                const R f = ph.t[(x + i) * phase_stride(RT) + w];
                g.x = fma(f, v.x, g.x);
                g.y = fma(f, v.y, g.y);
              }
            accn[0] = accn[0] + g;
            s += m;
            x += m;
          };
          const int head = min(end - s, -(cur.x0 + s) & 3);
          if (head) some(head);
#pragma unroll 2
          for (; s + 4 <= end;) some(4);
          if (s < end) some(end - s);
        } else {
#pragma unroll 8
          for (; s < end; s++, x++) {
            const Cx<R> v = src[s];
#pragma unroll
            for (int i = 0; i < kNR; i++) {
              const int r = w + kWarps * i;
              if (r < RT) {
                const R f = ph.t[x * phase_stride(RT) + r];
                accn[i].x = fma(f, v.x, accn[i].x);
                accn[i].y = fma(f, v.y, accn[i].y);
              }
            }
          }
        }
        if (x == a.Lx) {
          Cx<R>* o = (Cx<R>*)a.out + ((long long)cur.tl * rows + row) * a.R1 * a.K + a.k.nuc + lane;
#pragma unroll
          for (int i = 0; i < kNR; i++) {
            const int r = w + kWarps * i;
            if (r < a.R1) o[(long long)r * a.K] = accn[i];
            accn[i] = czero<R>();
          }
          x = 0;
          row++;
        }
      }
    }
    ld.store(a, nx, t, role);
    __syncthreads();
  }
}

template <typename R, typename Tin, int RT>
cudaError_t go(const ContractArgs& a, const double* xt, int nsm, cudaStream_t s) {
  return launch_tiles<R>(k_site_mesons<R, Tin, RT>, a, xt, RT, Mem<R>::kAll, nsm, s);
}

// Instantiated for three, seven and nine phase rows: five run as seven, which
// takes no longer (48^3 x 12 slices, split, this kernel's us: three rows 3021, five
// 3127, seven 3126), one as three.
template <typename R, typename Tin>
cudaError_t go_rows(const ContractArgs& a, const double* xt, int nsm, cudaStream_t s) {
  return a.R1 <= 3   ? go<R, Tin, 3>(a, xt, nsm, s)
         : a.R1 <= 7 ? go<R, Tin, 7>(a, xt, nsm, s)
                     : go<R, Tin, 9>(a, xt, nsm, s);
}

}  // namespace
}  // namespace site

cudaError_t launch_site_mesons(const ContractArgs& a, const double* xt, int plain, int fp32_in, int nsm,
                               cudaStream_t s) {
  if (plain) return site::go_rows<double, double>(a, xt, nsm, s);
  return fp32_in ? site::go_rows<float, float>(a, xt, nsm, s) : site::go_rows<float, double>(a, xt, nsm, s);
}

}  // namespace p2
