// Table-driven baryon two-point functions: the reference's UDSC set
// (contractBaryonsUDSC, lib/PLEGMA_Correlator.cu:137-189, kernels
// lib/kernels/PLEGMA_baryons_udsc.cu:85-309), both forms.
//
// A flavour product (e.g. "uud") has up to 16 datasets (interpolator and
// projector variants); dataset d of a site is
//   sum_entries w * sum_{eps eps'} P1[s0 s1][a a'] P2[s2 s3][b b'] P3[s4 s5][c c']
// over the spin tables of plegma_b200/udsc.py (real weights, each rounded to
// single precision like the reference's, the sums of merged ones in double,
// in the split form rounded again; the reference spends 108 complex products
// per entry).  udsc.site_program turns a product's entries into a program:
// entries that differ by an exchange of equal flavours are merged, every
// distinct triple of spin blocks is evaluated once for all datasets, as a
// diquark of two of its blocks (36 complex products) dotted with the third
// (9 products), and a greedy cover keeps the diquarks few.  For "uud" that is
// 133 diquarks and 424 dots for 848 weights, against 240 diquarks and 1100
// dots of the entries as they stand.
//
// One site per lane: the eight warps of a block take 32 sites of one slice
// and an eighth of the program each, so the control flow is the same for all
// lanes (the program is read from constant memory), a block's nine entries
// are conflict-free loads, and nothing moves between lanes.  The datasets'
// partial sums of the eight warps meet in shared memory once per product.
// Products on the same one or two flavours run in one launch on the same
// staged tile.  The sums go to a [slice][dataset][site] buffer that the
// projection consumes.
// Measured on B200 against one instruction stream per lane over the unmerged
// entries (16 lanes of a site in divergent loops): split form, 32^3 x 16, u and
// d (28 datasets), 123 momenta 20.6 -> 3.8 ms; plain form, 16^3 x 16, all 200
// datasets, 33 momenta 33.9 -> 7.4 ms.
// Bound: the latency of a warp's chain program word -> block -> products, with
// 16 (split) or 8 (plain) warps per SM: 65 % of the issue slots, FMA pipe 40 %
// (split, 2029 clk/site), 35 % and FP64 pipe 42 % (plain, 3736 clk/site).
#include <algorithm>
#include <cstring>
#include <map>
#include <numeric>
#include <string>
#include <vector>

#include "ctx.h"
#include "launch_util.h"
#include "site_contract.cuh"
#include "udsc_tables.h"

using namespace p2host;

namespace p2 {
namespace {

constexpr int kThreadsU = 32 * kUdscWarps;
constexpr int kSitesU = 32;  // sites of a tile, one per lane
// datasets of a launch's largest product: 16 with three flavours, 10 with fewer
template <int NF>
constexpr int kMaxDs = NF == 3 ? 16 : 10;
constexpr int kMaxProgs = 4; // products on one pair of flavours: aab, abb, aaa, bbb

__constant__ unsigned c_code[kUdscCodeWords] = P2_INIT_UDSC_CODE;
__constant__ double c_weight[kUdscWeights] = P2_INIT_UDSC_WEIGHTS;
__constant__ float c_weight32[kUdscWeights] = P2_INIT_UDSC_WEIGHTS;
template <typename R>
__device__ __forceinline__ R weight(int i) {
  if constexpr (sizeof(R) == 8)
    return c_weight[i];
  else
    return c_weight32[i];
}

struct UdscSlice {
  long long off[3];  // element offset of the slice inside each of the views
  int xf[3];         // load-time transform of each view on this slice (PropXf)
  int pad;
};

// One flavour product of a launch.
struct UdscProg {
  int start[kUdscWarps];  // first record of each warp
  int nd, k0;             // datasets and their first component in the output
  int boff;               // added to the program's blocks (16 x the view of its first flavour)
};

struct UdscArgs {
  const void* p[3];  // views of the launch's NF flavours
  long long vol[3];  // component strides
  const UdscSlice* sl;
  int ntau, V3, K;   // slices, sites, components of the output
  int nprog;
  UdscProg prog[kMaxProgs];
  int* e3;           // split form: [ntau][3], view v of slice t is staged times 2^-e3[3t+v]
  int* es;           // split form: [ntau][2], what the components' exponents (kexp) multiply
  void* out;         // [ntau][K][V3] complex double (plain) or complex float (split)
  int* cmax;         // split form: [ntau][K] max |Re|, |Im| as float bits, or null
};

// ---- a tile's propagators in shared memory, the site in the lane -----------
// FP64: [16 f + block][9 colours][32 sites]; FP32: four pairs of colours as
// 16-byte units [16 f + block][4][32 sites], then colour 8 [16 f + block][32 sites].
template <typename R, int NF>
struct SiteTile;
template <int NF>
struct SiteTile<double, NF> {
  static constexpr int kBytes = NF * 144 * kSitesU * 16;
  Cx<double>* p;
  __device__ __forceinline__ SiteTile(unsigned char* sm, int lane) : p((Cx<double>*)sm + lane) {}
  __device__ __forceinline__ void load9(int blk, Cx<double> (&v)[9]) const {
#pragma unroll
    for (int i = 0; i < 9; i++) v[i] = p[(blk * 9 + i) * kSitesU];
  }
};
template <int NF>
struct SiteTile<float, NF> {
  static constexpr int kBytes = NF * 144 * kSitesU * 8;
  float4* q;
  Cx<float>* last;
  __device__ __forceinline__ SiteTile(unsigned char* sm, int lane)
      : q((float4*)sm + lane), last((Cx<float>*)((float4*)sm + NF * 16 * 4 * kSitesU) + lane) {}
  __device__ __forceinline__ void load9(int blk, Cx<float> (&v)[9]) const {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float4 x = q[(blk * 4 + k) * kSitesU];
      v[2 * k] = cx<float>(x.x, x.y);
      v[2 * k + 1] = cx<float>(x.z, x.w);
    }
    v[8] = last[blk * kSitesU];
  }
};

// FP64: the tile by cp.async, the load-time transforms in place.
template <int NF>
__device__ __forceinline__ void stage_tile(const UdscArgs& a, const SiteTile<double, NF>& t, int tl, int x, bool ok) {
  const int warp = threadIdx.x >> 5;
  const UdscSlice& sd = a.sl[tl];
#pragma unroll
  for (int f = 0; f < NF; f++) {
    const Cx<double>* src = (const Cx<double>*)a.p[f] + sd.off[f] + (ok ? x : 0);
#pragma unroll 6
    for (int c = warp; c < 144; c += kUdscWarps)
      cp_async16(t.p + (144 * f + c) * kSitesU, src + c * a.vol[f], ok ? 16 : 0);
  }
  cp_async_commit();
  cp_async_wait<0>();
  if (sd.xf[0] | sd.xf[1] | sd.xf[2]) {  // uniform over the block
    __syncthreads();
    for (int q = warp; q < 36 * NF; q += kUdscWarps) {
      const int f = q / 36;
      int comp[4];
      prop_group_comps(q - 36 * f, comp);
      Cx<double>* r = t.p + 144 * f * kSitesU;
      prop_group_transform(r[comp[0] * kSitesU], r[comp[1] * kSitesU], r[comp[2] * kSitesU], r[comp[3] * kSitesU],
                           sd.xf[f]);
    }
  }
}

// FP32: loaded, transformed, scaled by 2^-E (in double: exact, no intermediate
// leaves the range) and converted in registers; two blocks per SM overlap the
// loads of one with the contraction of the other.
template <typename Tin, int NF>
__device__ __forceinline__ void stage_tile(const UdscArgs& a, const SiteTile<float, NF>& t, int tl, int x, bool ok) {
  const int warp = threadIdx.x >> 5;
  const UdscSlice& sd = a.sl[tl];
#pragma unroll
  for (int f = 0; f < NF; f++) {
    const Cx<Tin>* src = (const Cx<Tin>*)a.p[f] + sd.off[f] + (ok ? x : 0);
    const long long vol = a.vol[f];
    const double sc = ldexp(1.0, -a.e3[3 * tl + f]);
    const int xf = sd.xf[f];
    // groups 0..15: (first block b of 0, 1, 4, 5; colours 2k, 2k + 1); 16..19: (b, colour 8)
#pragma unroll 1
    for (int g = warp; g < 20; g += kUdscWarps) {
      const int bq = g & 3, b = (bq >> 1) * 4 + (bq & 1);
      if (g < 16) {
        const int k = g >> 2;
        Cx<Tin> raw[2][4];
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
          for (int i = 0; i < 4; i++)
            raw[c][i] = ok ? src[(9 * (b + group_blk(i)) + 2 * k + c) * vol] : czero<Tin>();
        Cx<double> v[2][4];
#pragma unroll
        for (int c = 0; c < 2; c++) {
#pragma unroll
          for (int i = 0; i < 4; i++) v[c][i] = cx<double>((double)raw[c][i].x, (double)raw[c][i].y);
          prop_group_transform(v[c][0], v[c][1], v[c][2], v[c][3], xf);
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
          t.q[((16 * f + b + group_blk(i)) * 4 + k) * kSitesU] =
              make_float4((float)(v[0][i].x * sc), (float)(v[0][i].y * sc), (float)(v[1][i].x * sc),
                          (float)(v[1][i].y * sc));
      } else {
        Cx<double> v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const Cx<Tin> r = ok ? src[(9 * (b + group_blk(i)) + 8) * vol] : czero<Tin>();
          v[i] = cx<double>((double)r.x, (double)r.y);
        }
        prop_group_transform(v[0], v[1], v[2], v[3], xf);
#pragma unroll
        for (int i = 0; i < 4; i++)
          t.last[(16 * f + b + group_blk(i)) * kSitesU] = cx<float>((float)(v[i].x * sc), (float)(v[i].y * sc));
      }
    }
  }
}

// G[c][e] = sum eps_abc eps_xye A[a][x] B[b][y]
template <typename R>
__device__ __forceinline__ void site_diquark(const Cx<R> (&a)[9], const Cx<R> (&b)[9], Cx<R> (&g)[9]) {
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int e = 0; e < 3; e++) {
      const int c1 = (c + 1) % 3, c2 = (c + 2) % 3, e1 = (e + 1) % 3, e2 = (e + 2) % 3;
      Cx<R> r = cmul(a[c1 * 3 + e1], b[c2 * 3 + e2]);
      cmsub(r, a[c1 * 3 + e2], b[c2 * 3 + e1]);
      cmsub(r, a[c2 * 3 + e1], b[c1 * 3 + e2]);
      cmac(r, a[c2 * 3 + e2], b[c1 * 3 + e1]);
      g[c * 3 + e] = r;
    }
}

// This warp's part of a program on its lanes' sites, from record q (see
// udsc.encode_programs) to the ending one.  A record comes from constant
// memory an iteration before it is used.  A dot's datasets are one case of a
// generated switch (one uniform branch per dot, the accumulators in
// registers).
template <typename R, int NF>
__device__ __forceinline__ void run_program(const SiteTile<R, NF>& t, int q, int boff, Cx<R> (&acc)[kMaxDs<NF>]) {
  Cx<R> A[9], g[9];
#pragma unroll
  for (int i = 0; i < 9; i++) A[i] = g[i] = czero<R>();
  unsigned rec = c_code[q], next = c_code[q + 1];
  q += 2;  // two records follow the last program's end
  auto advance = [&]() {
    rec = next;
    next = c_code[q++];
  };
  auto block = [&](unsigned r) { return (int)(r >> 2 & 63) + boff; };
#pragma unroll 1
  while ((rec & 3) != 3) {
    if ((rec & 3) == 0) {
      t.load9(block(rec), A);
      advance();
    }
    {
      Cx<R> B[9];
      t.load9(block(rec), B);
      advance();
      site_diquark(A, B, g);
    }
#pragma unroll 1
    while ((rec & 3) == 2) {
      Cx<R> z[9];
      t.load9(block(rec), z);
      const int cs = (int)(rec >> 8 & 255), wi = (int)(rec >> 16);
      advance();
      // FP64 three, FP32 two partial sums: chains of dependent FMAs in flight
      constexpr int NV = sizeof(R) == 8 ? 3 : 2;
      Cx<R> vs[NV];
#pragma unroll
      for (int i = 0; i < 9; i++) {
        if (i < NV)
          vs[i] = cmul(g[i], z[i]);
        else
          cmac(vs[i % NV], g[i], z[i]);
      }
      Cx<R> v = vs[0] + vs[1];
      if constexpr (NV == 3) v = v + vs[2];
#define P2_ADD(d, i)                                   \
  {                                                    \
    const R f = weight<R>(wi + i);                     \
    acc[d].x = fma(f, v.x, acc[d].x);                  \
    acc[d].y = fma(f, v.y, acc[d].y);                  \
  }
      if constexpr (NF == 3) {
        switch (cs) { P2_UDSC_CASES_16 }
      } else {
        switch (cs) { P2_UDSC_CASES_10 }
      }
#undef P2_ADD
    }
  }
}

// Shared memory: the tile, then (with more than one program) the warps'
// partial sums; a single program's go over the tile, which is dead by then
// (three FP64 flavours fill the shared memory).
template <typename R, int NF>
constexpr int udsc_smem(int nprog, int nd) {
  const int red = kUdscWarps * nd * kSitesU * 2 * (int)sizeof(R);
  return nprog > 1 ? SiteTile<R, NF>::kBytes + red : SiteTile<R, NF>::kBytes > red ? SiteTile<R, NF>::kBytes : red;
}

template <typename R, typename Tin, int NF>
__global__ void __launch_bounds__(kThreadsU, sizeof(R) == 4 ? 2 : 1) k_contract_udsc(const UdscArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const SiteTile<R, NF> tile(smem_raw, lane);
  Cx<R>* red = (Cx<R>*)(a.nprog > 1 ? smem_raw + SiteTile<R, NF>::kBytes : smem_raw);
  const int tpt = (a.V3 + kSitesU - 1) / kSitesU;
  const long long ntile = (long long)tpt * a.ntau;
  for (long long i = blockIdx.x; i < ntile; i += gridDim.x) {
    const int tl = (int)(i / tpt), x = (int)(i % tpt) * kSitesU + lane;
    const bool ok = x < a.V3;
    if constexpr (sizeof(R) == 8)
      stage_tile<NF>(a, tile, tl, x, ok);
    else
      stage_tile<Tin, NF>(a, tile, tl, x, ok);
    __syncthreads();
#pragma unroll 1
    for (int p = 0; p < a.nprog; p++) {
      const UdscProg& pg = a.prog[p];
      Cx<R> acc[kMaxDs<NF>];
#pragma unroll
      for (int d = 0; d < kMaxDs<NF>; d++) acc[d] = czero<R>();
      run_program(tile, pg.start[warp], pg.boff, acc);
      __syncthreads();  // the tile (single program) or the previous program's sums are read
#pragma unroll
      for (int d = 0; d < kMaxDs<NF>; d++)
        if (d < pg.nd) red[(warp * pg.nd + d) * kSitesU + lane] = acc[d];
      __syncthreads();
      for (int d = warp; d < pg.nd; d += kUdscWarps) {
        Cx<R> v = czero<R>();
#pragma unroll
        for (int w = 0; w < kUdscWarps; w++) v = v + red[(w * pg.nd + d) * kSitesU + lane];
        const long long row = (long long)tl * a.K + pg.k0 + d;
        if (ok) ((Cx<R>*)a.out)[row * a.V3 + x] = v;
        if constexpr (sizeof(R) == 4)
          if (a.cmax) {
            const unsigned m = __reduce_max_sync(0xffffffffu, ok ? __float_as_uint(fmaxf(fabsf(v.x), fabsf(v.y))) : 0u);
            if (lane == 0) atomicMax(a.cmax + row, (int)m);
          }
      }
    }
    __syncthreads();  // the sums are read and the tile is dead
  }
}

// Per slice and view the exponent of a sample (sample_exponent), plus one when
// the view is rotated.  One block per (slice, view).
template <typename Tin>
__global__ void __launch_bounds__(kSampleThreads) k_sample_udsc(const UdscArgs a, int nf) {
  const int tl = blockIdx.x, f = blockIdx.y;
  const UdscSlice& sd = a.sl[tl];
  const int E0 = sample_exponent((const Cx<Tin>*)a.p[f] + sd.off[f], a.vol[f], a.V3);
  if (threadIdx.x == 0) {
    const int E = E0 + ((sd.xf[f] & 3) ? 1 : 0);
    a.e3[3 * tl + f] = E;
    // one or two flavours: es holds their exponents; three: each component carries all three once
    if (nf <= 2) {
      a.es[2 * tl + f] = E;
      if (nf == 1) a.es[2 * tl + 1] = 0;
    } else if (f < 2) {
      a.es[2 * tl + f] = 0;
    }
  }
}
// three flavours: the sum of the view exponents (after k_sample_udsc)
__global__ void k_sum_udsc(const UdscArgs a) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < a.ntau) a.es[2 * t] = a.e3[3 * t] + a.e3[3 * t + 1] + a.e3[3 * t + 2];
}

template <typename R, typename Tin, int NF>
cudaError_t launch_udsc_t(const UdscArgs& a, int nsm, cudaStream_t s) {
  int nd = 0;
  for (int p = 0; p < a.nprog; p++) nd = std::max(nd, a.prog[p].nd);
  if (nd > kMaxDs<NF>) return cudaErrorInvalidValue;
  const int smem = udsc_smem<R, NF>(a.nprog, nd);
  cudaError_t e = ensure_smem((const void*)k_contract_udsc<R, Tin, NF>, smem);
  if (e != cudaSuccess) return e;
  const long long tiles = (long long)((a.V3 + kSitesU - 1) / kSitesU) * a.ntau;
  const int grid = (int)std::min<long long>(tiles, (long long)nsm * (sizeof(R) == 4 ? 2 : 1));
  k_contract_udsc<R, Tin, NF><<<grid, kThreadsU, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_contract_udsc(const UdscArgs& a, int nf, int nsm, cudaStream_t s) {
  return nf == 1   ? launch_udsc_t<double, double, 1>(a, nsm, s)
         : nf == 2 ? launch_udsc_t<double, double, 2>(a, nsm, s)
                   : launch_udsc_t<double, double, 3>(a, nsm, s);
}

template <typename Tin>
cudaError_t launch_udsc_split_t(const UdscArgs& a, int nf, int nsm, cudaStream_t s) {
  k_sample_udsc<Tin><<<dim3(a.ntau, nf), kSampleThreads, 0, s>>>(a, nf);
  if (nf == 3) k_sum_udsc<<<(a.ntau + 255) / 256, 256, 0, s>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return nf == 1   ? launch_udsc_t<float, Tin, 1>(a, nsm, s)
         : nf == 2 ? launch_udsc_t<float, Tin, 2>(a, nsm, s)
                   : launch_udsc_t<float, Tin, 3>(a, nsm, s);
}

// Products a request runs, in the reference's order and with its filters
// (lib/PLEGMA_Correlator.cu:152-177).
std::vector<int> products_of(const p2_udsc_request& r) {
  std::vector<int> todo;
  for (int i = 0; i < kUdscProducts; i++) {
    const std::string f = kUdscProduct[i];
    auto has = [&](char c) { return f.find(c) != std::string::npos; };
    if ((r.prop_u < 0 && has('u')) || (r.prop_d < 0 && has('d')) || (r.prop_s < 0 && has('s')) ||
        (r.prop_c < 0 && has('c')))
      continue;
    if (r.only_st && !has('s')) continue;
    if (r.only_ch && !has('c')) continue;
    todo.push_back(i);
  }
  return todo;
}

int prop_of(const p2_udsc_request& r, char f) {
  return f == 'u' ? r.prop_u : f == 'd' ? r.prop_d : f == 's' ? r.prop_s : r.prop_c;
}

}  // namespace
}  // namespace p2

// Flavour products of a request that run in one launch: same one or two
// flavours (a product of a single flavour joins a pair with it when both hold
// the same slices), or one product of three.
namespace p2 {
namespace {
struct UdscGroup {
  std::string flavours;     // distinct, in the order u d s c
  std::vector<int> prods;
  std::vector<int> ds_off;  // first dataset of each product in the result
  std::vector<int> taus;    // local slices held by all the views
  std::vector<UdscSlice> sl;
  int K = 0;                // datasets of the group
  size_t o_sl = 0, o_desc = 0, o_kexp = 0;  // byte offsets in the call's upload
};
}  // namespace
}  // namespace p2

struct p2_udsc_cache {
  p2host::DevBuf args;    // slices, descriptors and component multiplicities of a call's groups
  p2host::DevBuf e3, es;  // split form: view exponents, un-scaling exponents
  ~p2_udsc_cache() {
    for (p2host::DevBuf* b : {&args, &e3, &es}) b->release();
  }
};

void p2_udsc_release(p2_ctx* c) {
  delete c->udsc;
  c->udsc = nullptr;
}

extern "C" {

int p2_udsc_datasets(const p2_udsc_request* r, char* names, size_t cap) {
  if (!r) return -1;
  std::string s;
  int n = 0;
  for (int p : p2::products_of(*r))
    for (int d = kUdscDsBegin[p]; d < kUdscDsBegin[p + 1]; d++, n++) {
      s += kUdscName[d];
      s += '\n';
    }
  if (names && cap) {
    const size_t m = std::min(cap - 1, s.size());
    std::memcpy(names, s.data(), m);
    names[m] = 0;
  }
  return n;
}

p2_status p2_contract_udsc(p2_ctx* c, const p2_prop* props, int nprops, const p2_udsc_request* r) {
  using namespace p2;
  if (!c) return P2_ERR_INVALID_ARG;
  if (!props || nprops < 1 || !r) return c->fail(P2_ERR_INVALID_ARG, "p2_contract_udsc: empty props or request");
  for (int f : {r->prop_u, r->prop_d, r->prop_s, r->prop_c})
    if (f < -1 || f >= nprops) return c->fail(P2_ERR_INVALID_ARG, "p2_contract_udsc: prop index out of range");
  if (!r->out) return c->fail(P2_ERR_INVALID_ARG, "null output");
  if (r->out_location != P2_DEVICE && r->out_location != P2_HOST)
    return c->fail(P2_ERR_INVALID_ARG, "bad out_location");
  if (r->mode != P2_PLAIN_FP64 && r->mode != P2_SPLIT_FP16) return c->fail(P2_ERR_INVALID_ARG, "bad mode");
  const bool split = r->mode == P2_SPLIT_FP16;
  p2_request base{};
  std::memcpy(base.source, r->source, sizeof(base.source));
  base.totalT = r->totalT;
  base.moms = r->moms;
  base.nmom = r->nmom;
  base.q2max = r->q2max;
  base.contractions = P2_NUCLEON_CG5;  // any valid set: only the window and momenta are used
  Plan pl;
  p2_status st = make_plan(c, base, pl);
  if (st != P2_OK) return st;
  const std::vector<int> todo = products_of(*r);
  for (int p : todo)
    for (int k = 0; k < 3; k++) {
      const p2_prop& pr = props[prop_of(*r, kUdscProduct[p][k])];
      if (!pr.data || pr.nt < 1 || pr.nt > c->T || pr.t_first < 0 || pr.t_first >= c->T)
        return c->fail(P2_ERR_INVALID_ARG, "p2_contract_udsc: bad propagator view");
      if ((pr.transform & ~0xFu) || ((pr.transform & 1u) && (pr.transform & 2u)))
        return c->fail(P2_ERR_INVALID_ARG, "p2_contract_udsc: bad transform bits");
      if (pr.precision != P2_FP64 && !(split && pr.precision == P2_FP32))
        return c->fail(P2_ERR_UNSUPPORTED, "p2_contract_udsc: FP32 propagators need the split form");
      if (pr.precision != props[prop_of(*r, kUdscProduct[todo[0]][0])].precision)
        return c->fail(P2_ERR_UNSUPPORTED, "p2_contract_udsc: all propagators must share a precision");
      if (pr.location != P2_DEVICE)
        return c->fail(P2_ERR_UNSUPPORTED, "p2_contract_udsc needs device-resident propagators");
    }
  if (c->host_only) return c->fail(P2_ERR_UNSUPPORTED, "host-only context");
  int nds = 0;
  for (int p : todo) nds += kUdscDsBegin[p + 1] - kUdscDsBegin[p];
  const size_t total = (size_t)nds * r->totalT * pl.nmom;
  if (todo.empty()) return P2_OK;
  if (!c->udsc) c->udsc = new p2_udsc_cache();
  p2_udsc_cache& U = *c->udsc;

  double* dres = r->out;
  if (r->out_location == P2_HOST) {
    P2_TRY(c, c->res.ensure(total * 16), "result alloc");
    P2_TRY(c, cudaMemsetAsync(c->res.p, 0, total * 16, c->stream), "result clear");
    dres = (double*)c->res.p;
  }
  const AxesPlan* ap = nullptr;  // the axis-by-axis projection, when the list qualifies
  // (an armed p2_debug_wait_timeout asks for the tensor-core projection)
  if (!(split && c->wait_test) && (st = axes_prepare(c, pl.moms, -1, &ap)) != P2_OK) return st;
  if (split && !axes_faster(c, pl.nmom, 4)) ap = nullptr;
  int nmtile = 0, nkstep = 0;
  if (split && !ap) {
    if (c->project_split_smem_max < project_split_smem_bytes(project_split_max_nt()))
      return c->fail(P2_ERR_UNSUPPORTED, "device shared memory per block too small for the tensor-core projection");
    if (!c->errflag.p) {
      P2_TRY(c, c->errflag.ensure(16), "error flag alloc");
      P2_TRY(c, cudaMemsetAsync(c->errflag.p, 0, 16, c->stream), "error flag clear");
    }
    if ((st = split_prepare_tables(c, pl, 0, nmtile, nkstep)) != P2_OK) return st;
  }
  // phase tables (origin 0; the scatter applies the source phase)
  if (!split && !ap && c->plain_moms_key != pl.moms) {
    c->plain_moms_key.clear();
    std::vector<double> tabh = phase_tables(c, pl.moms.data(), pl.nmom, -1, pl.Lmax);
    if ((st = upload_async(c, c->ptab, tabh.data(), tabh.size() * sizeof(double), "phase table")) != P2_OK)
      return st;
    if ((st = upload_async(c, c->moms, pl.moms.data(), pl.moms.size() * sizeof(int), "momenta")) != P2_OK)
      return st;
    c->plain_moms_key = pl.moms;
  }

  // groups of products
  const int T = c->T, tl0 = c->g.coords[3] * c->Ll[3];
  std::vector<UdscGroup> groups;
  auto slices_of = [&](const std::string& fl, UdscGroup& g) {
    for (int tau = 0; tau < r->totalT; tau++) {
      const int t = (r->source[3] + tau) % T;
      if (t < tl0 || t >= tl0 + c->Ll[3]) continue;
      UdscSlice s{};
      bool ok = true;
      for (size_t k = 0; k < fl.size(); k++) {
        const p2_prop& v = props[prop_of(*r, fl[k])];
        const int j = ((t - v.t_first) % T + T) % T;
        ok &= j < v.nt;
        s.off[k] = (long long)j * c->V3;
        s.xf[k] = prop_xf_code(v, t);
      }
      if (!ok) continue;
      g.taus.push_back(tau);
      g.sl.push_back(s);
    }
  };
  int ds_off = 0;
  std::vector<int> offs;
  for (int p : todo) {
    offs.push_back(ds_off);
    ds_off += kUdscDsBegin[p + 1] - kUdscDsBegin[p];
  }
  for (int pass = 0; pass < 2; pass++)  // products of a single flavour join a pair's group, so they come second
    for (size_t i = 0; i < todo.size(); i++) {
      const std::string f = kUdscProduct[todo[i]];
      UdscGroup g;
      for (char q : std::string("udsc"))
        if (f.find(q) != std::string::npos) g.flavours += q;
      if ((g.flavours.size() == 1) != (pass == 1)) continue;
      slices_of(g.flavours, g);
      if (g.taus.empty()) continue;
      UdscGroup* to = nullptr;
      for (UdscGroup& h : groups)
        if (!to && (int)h.prods.size() < kMaxProgs && h.taus == g.taus &&
            (h.flavours == g.flavours ||
             (pass == 1 && h.flavours.size() == 2 && h.flavours.find(g.flavours) != std::string::npos)))
          to = &h;
      if (!to) {
        groups.push_back(g);
        to = &groups.back();
      }
      to->prods.push_back(todo[i]);
      to->ds_off.push_back(offs[i]);
      to->K += kUdscDsBegin[todo[i] + 1] - kUdscDsBegin[todo[i]];
    }
  // one upload: the groups' slices, descriptors and, per component, how often
  // it carries each of the launch's first two scales (three flavours: their
  // summed scale once)
  std::vector<unsigned char> up;
  auto reserve = [&](size_t n) {
    const size_t o = up.size();
    up.resize(o + (n + 15) / 16 * 16, 0);
    return o;
  };
  for (UdscGroup& g : groups) {
    const size_t n = g.taus.size();
    g.o_sl = reserve(n * sizeof(UdscSlice));
    g.o_desc = reserve(n * sizeof(SliceDesc));
    g.o_kexp = reserve(2 * (size_t)g.K * sizeof(int));
    std::memcpy(&up[g.o_sl], g.sl.data(), n * sizeof(UdscSlice));
    SliceDesc* desc = (SliceDesc*)&up[g.o_desc];
    for (size_t i = 0; i < n; i++) {
      desc[i].out = dres;
      desc[i].tau = g.taus[i];
      desc[i].totalT = r->totalT;
      for (int d = 0; d < 3; d++) desc[i].x0[d] = r->source[d];
    }
    int* ke = (int*)&up[g.o_kexp];
    for (int p : g.prods) {
      const std::string f = kUdscProduct[p];
      for (int d = kUdscDsBegin[p]; d < kUdscDsBegin[p + 1]; d++, ke += 2) {
        if (g.flavours.size() == 3)
          ke[0] = 1;
        else
          for (size_t k = 0; k < g.flavours.size(); k++)
            ke[k] = (int)std::count(f.begin(), f.end(), g.flavours[k]);
      }
    }
  }
  if (!up.empty() && (st = upload_async(c, U.args, up.data(), up.size(), "udsc arguments")) != P2_OK) return st;

  // slices of a chunk; the scratch is sized for the largest group at once
  auto chunk_of = [&](const UdscGroup& g) { return chunk_slices(c, slice_bytes(c, ap, split, g.K, g.K, false), T); };
  size_t bytes = 0;
  for (const UdscGroup& g : groups)
    bytes = std::max(bytes, scratch_bytes(c, ap, split, std::min((size_t)chunk_of(g), g.taus.size()), g.K, g.K));
  P2_TRY(c, c->cbuf.ensure(bytes), "workspace alloc");

  for (const UdscGroup& g : groups) {
    const int nf = (int)g.flavours.size(), K = g.K, n_all = (int)g.taus.size();
    UdscArgs a{};
    for (int k = 0; k < nf; k++) {
      const p2_prop& v = props[prop_of(*r, g.flavours[k])];
      a.p[k] = v.data;
      a.vol[k] = c->V3 * v.nt;
    }
    const bool f32 = props[prop_of(*r, g.flavours[0])].precision == P2_FP32;
    a.V3 = (int)c->V3;
    a.K = K;
    a.nprog = (int)g.prods.size();
    std::vector<ScatterBlock> blocks;
    int k0 = 0;
    for (int i = 0; i < a.nprog; i++) {
      const int p = g.prods[i], nd = kUdscDsBegin[p + 1] - kUdscDsBegin[p];
      std::memcpy(a.prog[i].start, kUdscProgramStart[kUdscProgram[p]], sizeof(a.prog[i].start));
      a.prog[i].nd = nd;
      a.prog[i].k0 = k0;
      // a program's blocks count from its own first flavour
      size_t first = nf;
      for (char q : std::string(kUdscProduct[p])) first = std::min(first, g.flavours.find(q));
      a.prog[i].boff = 16 * (int)first;
      blocks.push_back(ScatterBlock{k0, 1, nd, 1, (long long)g.ds_off[i]});
      k0 += nd;
    }
    const int tc = chunk_of(g);
    for (int c0 = 0; c0 < n_all; c0 += tc) {
      const int n = std::min(tc, n_all - c0);
      const SliceDesc* dsl = (const SliceDesc*)((const unsigned char*)U.args.p + g.o_desc) + c0;
      const int* kexp = (const int*)((const unsigned char*)U.args.p + g.o_kexp);
      a.sl = (const UdscSlice*)((const unsigned char*)U.args.p + g.o_sl) + c0;
      a.ntau = n;
      a.out = c->cbuf.p;
      if (split) {
        P2_TRY(c, U.e3.ensure((size_t)n * 3 * sizeof(int)), "exponent alloc");
        P2_TRY(c, U.es.ensure((size_t)n * 2 * sizeof(int)), "exponent alloc");
        a.e3 = (int*)U.e3.p;
        a.es = (int*)U.es.p;
        if (!ap) {
          P2_TRY(c, c->cmaxb.ensure((size_t)n * K * sizeof(int)), "maxima alloc");
          P2_TRY(c, cudaMemsetAsync(c->cmaxb.p, 0, (size_t)n * K * sizeof(int), c->stream), "maxima clear");
          a.cmax = (int*)c->cmaxb.p;
        }
        ProfScope ps(c, "contract_udsc_f32");
        P2_TRY(c,
               f32 ? launch_udsc_split_t<float>(a, nf, c->nsm, c->stream)
                   : launch_udsc_split_t<double>(a, nf, c->nsm, c->stream),
               "udsc split contraction");
      } else {
        ProfScope ps(c, "contract_udsc_fp64");
        P2_TRY(c, launch_contract_udsc(a, nf, c->nsm, c->stream), "udsc contraction");
      }
      if (ap) {
        void* const s1 = (char*)c->cbuf.p + sums_offset(c, split, n, K);
        if ((st = axes_x(c, *ap, c->cbuf.p, split, (long long)K * c->V3, c->V3, n, K, K, s1)) != P2_OK)
          return st;
        AxesOut ao;
        ao.dsl = dsl;
        ao.blocks = &blocks;
        if (split) {
          ao.exps = a.es;
          ao.kexp = kexp;
        }
        if ((st = axes_yz(c, *ap, s1, split, n, K, ao)) != P2_OK) return st;
      } else if (split) {
        if ((st = split_project(c, pl, K, n, nmtile, nkstep, dsl, a.es, kexp, blocks)) != P2_OK) return st;
      } else if ((st = project_direct(c, pl, K, n, n, dsl, blocks)) != P2_OK) {
        return st;
      }
    }
  }
  if (r->out_location == P2_HOST) {
    P2_TRY(c, cudaMemcpyAsync(r->out, dres, total * 16, cudaMemcpyDeviceToHost, c->stream), "result download");
    P2_TRY(c, cudaStreamSynchronize(c->stream), "result download");
  }
  return P2_OK;
}

}  // extern "C"
