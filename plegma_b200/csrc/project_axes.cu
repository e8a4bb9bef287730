// Momentum projection one axis at a time.
//
// C(t, p, k) = sum_x c_k(x, t) exp(sign i p.(x - x0)) over a list of integer
// momenta (the reference's fourier_transform_3D sums every site with every
// momentum, lib/kernels/PLEGMA_kernel_utils.cuh:820-860).  The phase is a
// product of three one-dimensional phases, and a list |n|^2 <= q2 holds few
// distinct |n_x|, |n_y|, |n_z|, so the sum is taken over x first for each
// distinct |n_x|, then over y for each distinct (|n_x|, |n_y|), then over z:
//
//   S1[t][row = (z, y)][r][k]   = sum_x X_r(x) c_k(x, y, z, t)
//   S2[t][z][pair = (r, s)][k]  = sum_y Y_s(y) S1[t][z, y][r][k]
//   C(t, p, k) from sum_z Z_q(z) S2[t][z][pair][k], q in {cos, sin}
//
// X_r, Y_s, Z_q are cos(2 pi a x / L) and sin(2 pi a x / L), one or two rows
// per distinct a = min(n mod L, L - n mod L) (sin is absent for a = 0 and
// a = L/2), so that the eight momenta (+-a, +-b, +-c) share all their sums
// ("orbit"; the eight real-phase sums give them with signs and factors i).
// For the 123 momenta of |n|^2 <= 9 a site and component costs 7 real x
// complex products over x instead of 123 complex ones, and the later sums run
// on 7 / Lx of the data.
//
// Measured on B200, FP64, against the direct sum of project_fp64.cu (which
// larger lists keep): the plain form at 24^3 x 48 with 288 components and 123
// momenta 3.13 ms instead of 14.12 ms, with the sums over x inside the
// contraction (the projection was 10.8 ms of it), the transform of a 32-component
// field there 0.136 ms instead of 2.18 ms.  Error against 64 bits 1.7e-15
// instead of 4.0e-15 (fewer terms per sum).
// Split form, against the tensor-core projection (which larger lists, and
// short x axes of large lattices, keep): 8^3 x 16 with 288 components 84 us
// instead of 120, 24^3 x 48 light baryons 4.36 ms instead of 5.34, 64^3 x 128
// with K = 480 and 257 momenta 17.0 ms instead of 29.1 (both with the Delta's new
// contraction); error against 64 bits 1.7e-7 instead of 1e-6 (no split of the
// data into FP16 parts).  Without the fused contraction (contract_site.cuh) 48^3
// slices take what the tensor cores do (8 of them, nucleon and 16 x 16 mesons
// 2.48 and 2.49 ms): the position buffer's write and read bound both.
//
// Sums over x: FP64 for FP64 input; FP32 input in FP32 over groups of at most
// kSumGroup sites and in FP64 over these, one row of Lx sites by one thread, so
// a row's sum does not depend on the launch shape; over y in FP32 by groups of
// groups (a conversion to FP64 per group doubled its time: 402 us instead of 197
// at 48^3 x 24 slices with K = 288); over z in FP64.  All in a fixed order.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "ctx.h"
#include "launch_util.h"
#include "p2_common.cuh"

namespace p2 {
namespace {

// ---- sums over x of a position buffer ------------------------------------------
// A "line" is one row of Lx sites of one component; a warp takes 64 lines, two
// per lane, and streams them in chunks of kBytes = 128 bytes per line through
// its own shared memory with cp.async (two stages), so the global loads are
// coalesced 128-byte segments and a lane's reads of its line are free of bank
// conflicts (odd line stride).  Two lines per lane share each phase.  HBM
// bound: the buffer is read once and R1 / Lx of it written.
constexpr int kXWarps = 4;
constexpr int kLines = 64;

template <typename R>
struct XChunk {
  static constexpr int n = 128 / (2 * (int)sizeof(R));  // elements of a 128-byte chunk
  static constexpr int stride = n + 1;
  static constexpr int stage = kLines * stride;  // complex elements
};

template <typename R>
__device__ __forceinline__ void cp_line(Cx<R>* dst, const Cx<R>* src, bool ok) {
  if constexpr (sizeof(R) == 8)
    cp_async16(dst, src, ok ? 16 : 0);
  else
    cp_async8(dst, src, ok ? 8 : 0);
}

template <typename R, int R1>
__global__ void __launch_bounds__(32 * kXWarps, 3) k_axis_x(const AxisXArgs a) {
  using C = XChunk<R>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<R>* st = (Cx<R>*)smem_raw + (threadIdx.x >> 5) * 2 * C::stage;
  R* ph = (R*)((Cx<R>*)smem_raw + kXWarps * 2 * C::stage);  // [Lx][R1]
  for (int i = threadIdx.x; i < a.Lx * R1; i += blockDim.x) ph[i] = (R)a.xt[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const long long item = (long long)blockIdx.x * kXWarps + (threadIdx.x >> 5);
  const int kgroups = (a.K + a.KL - 1) / a.KL;
  const int rows_per = kLines / a.KL;
  const int rgroups = (a.rows + rows_per - 1) / rows_per;
  if (item >= (long long)kgroups * rgroups * a.ntau) return;
  // component groups vary slowest inside a slice, so that neighbouring warps read neighbouring rows
  const int rg = (int)(item % rgroups), kg = (int)((item / rgroups) % kgroups);
  const int tau = (int)(item / ((long long)rgroups * kgroups));
  const int lg = __ffs(a.KL) - 1;
  const Cx<R>* c = (const Cx<R>*)a.c + (long long)tau * a.sT;
  const int nchunk = (a.Lx + C::n - 1) / C::n;

  // this lane copies element e of the lines (lane / n) + 32 / n * i
  constexpr int kPer = 32 / C::n;
  const int e = lane % C::n, l0 = lane / C::n;
  auto issue = [&](int ch) {
    if (ch < nchunk) {
      Cx<R>* d = st + (ch & 1) * C::stage;
      const int x = ch * C::n + e;
#pragma unroll 8
      for (int i = 0; i < kLines / kPer; i++) {
        const int ln = l0 + kPer * i;
        const int k = kg * a.KL + (ln & (a.KL - 1)), row = rg * rows_per + (ln >> lg);
        const bool ok = x < a.Lx && k < a.K && row < a.rows;
        cp_line(d + ln * C::stride + e, ok ? c + (long long)k * a.sK + (long long)row * a.Lx + x : c, ok);
      }
    }
    cp_async_commit();
  };
  // FP32: acc the current group of kSumGroup sites, tot the groups before it
  constexpr bool kGroups = sizeof(R) == 4;
  static_assert(!kGroups || C::n % kSumGroup == 0, "a chunk holds whole groups");
  Cx<R> acc[2][R1];
  Cx<double> tot[2][kGroups ? R1 : 1];
#pragma unroll
  for (int j = 0; j < 2; j++) {
#pragma unroll
    for (int r = 0; r < R1; r++) acc[j][r] = czero<R>();
#pragma unroll
    for (int r = 0; r < (kGroups ? R1 : 1); r++) tot[j][r] = czero<double>();
  }
  auto add = [&](const Cx<R>* d, const R* p, int x) {
    const Cx<R> v0 = d[x], v1 = d[32 * C::stride + x];
#pragma unroll
    for (int r = 0; r < R1; r++) {
      const R f = p[x * R1 + r];
      acc[0][r].x = fma(f, v0.x, acc[0][r].x);
      acc[0][r].y = fma(f, v0.y, acc[0][r].y);
      acc[1][r].x = fma(f, v1.x, acc[1][r].x);
      acc[1][r].y = fma(f, v1.y, acc[1][r].y);
    }
  };
  issue(0);
  for (int ch = 0; ch < nchunk; ch++) {
    issue(ch + 1);
    cp_async_wait<1>();
    __syncwarp();
    const Cx<R>* d = st + (ch & 1) * C::stage + lane * C::stride;
    const R* p = ph + ch * C::n * R1;
    const int n = min(C::n, a.Lx - ch * C::n);
    if constexpr (kGroups) {
#pragma unroll 1
      for (int x0 = 0; x0 < n; x0 += kSumGroup) {
        const int x1 = min(n, x0 + kSumGroup);
#pragma unroll 4
        for (int x = x0; x < x1; x++) add(d, p, x);
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
          for (int r = 0; r < R1; r++) {
            tot[j][r].x += (double)acc[j][r].x;
            tot[j][r].y += (double)acc[j][r].y;
            acc[j][r] = czero<R>();
          }
      }
    } else {
#pragma unroll 4
      for (int x = 0; x < n; x++) add(d, p, x);
    }
    __syncwarp();  // the chunk is read: the stage may be refilled
  }
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const int ln = lane + 32 * j;
    const int k = kg * a.KL + (ln & (a.KL - 1)), row = rg * rows_per + (ln >> lg);
    if (k < a.K && row < a.rows) {
      Cx<R>* o = (Cx<R>*)a.s1 + (((long long)tau * a.rows + row) * R1) * a.Kst + k;
#pragma unroll
      for (int r = 0; r < R1; r++)
        o[(long long)r * a.Kst] = kGroups ? cx<R>((R)tot[j][kGroups ? r : 0].x, (R)tot[j][kGroups ? r : 0].y) : acc[j][r];
    }
  }
}

// ---- sums over y ----------------------------------------------------------------
// Warp r of a block takes x row r of (slice, z) for 32 or 64 components (KPL
// per lane): every value of S1 is read once and used for all the pairs of r,
// U rows y at a time (their loads are in flight together, and vector loads
// bring the phases of several y), zper values of z one after the other.  The
// body is instantiated for the number of pairs, so the rows with few of them
// spend nothing on the others.
template <int N, int KPL, int U>
__device__ __forceinline__ void axis_y_body(const AxisYArgs& a, const double* yt, int LyP, int r, int first) {
  typedef double R;
  const int lane = threadIdx.x & 31, tau = blockIdx.z, k0 = blockIdx.x * 32 * KPL + lane;
  const R* row[N];
#pragma unroll
  for (int j = 0; j < N; j++) row[j] = yt + a.ylist[first + j] * LyP;
  const long long rs = (long long)a.R1 * a.K;  // one row of S1
#pragma unroll 1
  for (int z = blockIdx.y * a.zper; z < min(a.Lz, (int)(blockIdx.y + 1) * a.zper); z++) {
    Cx<R> acc[N][KPL];
#pragma unroll
    for (int j = 0; j < N; j++)
#pragma unroll
      for (int q = 0; q < KPL; q++) acc[j][q] = czero<R>();
    const Cx<R>* s = (const Cx<R>*)a.s1 + ((long long)tau * a.Lz + z) * a.Ly * rs + (long long)r * a.K;
#pragma unroll 1
    for (int y0 = 0; y0 < a.Ly; y0 += U) {
      Cx<R> v[U][KPL];
#pragma unroll
      for (int i = 0; i < U; i++)
#pragma unroll
        for (int q = 0; q < KPL; q++)
          v[i][q] = y0 + i < a.Ly && k0 + 32 * q < a.K ? s[(y0 + i) * rs + k0 + 32 * q] : czero<R>();
#pragma unroll
      for (int j = 0; j < N; j++) {
        R f[U];  // zero beyond Ly
        constexpr int kVec = 16 / (int)sizeof(R);
#pragma unroll
        for (int i = 0; i < U; i += kVec)
          *reinterpret_cast<float4*>(f + i) = *reinterpret_cast<const float4*>(row[j] + y0 + i);
#pragma unroll
        for (int i = 0; i < U; i++)
#pragma unroll
          for (int q = 0; q < KPL; q++) {
            acc[j][q].x = fma(f[i], v[i][q].x, acc[j][q].x);
            acc[j][q].y = fma(f[i], v[i][q].y, acc[j][q].y);
          }
      }
    }
    Cx<R>* o = (Cx<R>*)a.s2 + (((long long)tau * a.Lz + z) * a.NP + first) * a.K;
#pragma unroll
    for (int j = 0; j < N; j++)
#pragma unroll
      for (int q = 0; q < KPL; q++)
        if (k0 + 32 * q < a.K) o[(long long)j * a.K + k0 + 32 * q] = acc[j][q];
  }
}

// FP32: a step's sums are added up over kSumGroups steps, and these in the result.
template <int N, int KPL, int U>
__device__ __forceinline__ void axis_y_body(const AxisYArgs& a, const float* yt, int LyP, int r, int first) {
  static_assert(U <= kSumGroup, "a running sum's steps");
  const int lane = threadIdx.x & 31, tau = blockIdx.z, k0 = blockIdx.x * 32 * KPL + lane;
  const float* row[N];
#pragma unroll
  for (int j = 0; j < N; j++) row[j] = yt + a.ylist[first + j] * LyP;
  const long long rs = (long long)a.R1 * a.K;  // one row of S1
#pragma unroll 1
  for (int z = blockIdx.y * a.zper; z < min(a.Lz, (int)(blockIdx.y + 1) * a.zper); z++) {
    const Cx<float>* s = (const Cx<float>*)a.s1 + ((long long)tau * a.Lz + z) * a.Ly * rs + (long long)r * a.K;
#pragma unroll 1
    for (int ys = 0; ys < a.Ly; ys += kSumGroups * U) {
      Cx<float> acc[N][KPL];
#pragma unroll
      for (int j = 0; j < N; j++)
#pragma unroll
        for (int q = 0; q < KPL; q++) acc[j][q] = czero<float>();
      const int ye = min(a.Ly, ys + kSumGroups * U);
#pragma unroll 1
      for (int y0 = ys; y0 < ye; y0 += U) {
        Cx<float> v[U][KPL];
#pragma unroll
        for (int i = 0; i < U; i++)
#pragma unroll
          for (int q = 0; q < KPL; q++)
            v[i][q] = y0 + i < a.Ly && k0 + 32 * q < a.K ? s[(y0 + i) * rs + k0 + 32 * q] : czero<float>();
#pragma unroll
        for (int j = 0; j < N; j++) {
          asm volatile("" ::: "memory");  // keeps the phases of later pairs from being moved up (registers)
          float f[U];                     // zero beyond Ly
#pragma unroll
          for (int i = 0; i < U; i += 4)
            *reinterpret_cast<float4*>(f + i) = *reinterpret_cast<const float4*>(row[j] + y0 + i);
#pragma unroll
          for (int q = 0; q < KPL; q++) {
            Cx<float> g = czero<float>();
#pragma unroll
            for (int i = 0; i < U; i++) {
              g.x = fma(f[i], v[i][q].x, g.x);
              g.y = fma(f[i], v[i][q].y, g.y);
            }
            acc[j][q] = acc[j][q] + g;
          }
        }
      }
      Cx<float>* o = (Cx<float>*)a.s2 + (((long long)tau * a.Lz + z) * a.NP + first) * a.K;
#pragma unroll
      for (int j = 0; j < N; j++)
#pragma unroll
        for (int q = 0; q < KPL; q++)
          if (k0 + 32 * q < a.K) {
            Cx<float>& d = o[(long long)j * a.K + k0 + 32 * q];
            d = ys ? d + acc[j][q] : acc[j][q];
          }
    }
  }
}

constexpr int kYUnroll = 8;

// W: most rows.  FP32: two blocks per SM; up to seven rows then have 128
// registers, which hold the sums (bounded for nine rows they spill: 207 us
// instead of 197 at 48^3 x 24 slices, K = 288).
template <typename R, int KPL, int W>
__global__ void __launch_bounds__(32 * W, sizeof(R) == 4 ? 2 : 0) k_axis_y(const __grid_constant__ AxisYArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int U = sizeof(R) * KPL == 16 ? kYUnroll / 2 : kYUnroll;
  R* yt = (R*)smem_raw;  // [RY][Ly rounded up]
  const int LyP = (a.Ly + kYUnroll - 1) / kYUnroll * kYUnroll;
  for (int i = threadIdx.x; i < a.RY * LyP; i += blockDim.x) {
    const int y = i % LyP;
    yt[i] = y < a.Ly ? (R)a.yt[(i / LyP) * a.Ly + y] : R(0);
  }
  __syncthreads();
  const int r = threadIdx.x >> 5;
  const int first = a.first[r], cnt = a.first[r + 1] - first;
  switch (cnt) {  // 0: a padding row
    case 1: axis_y_body<1, KPL, U>(a, yt, LyP, r, first); break;
    case 2: axis_y_body<2, KPL, U>(a, yt, LyP, r, first); break;
    case 3: axis_y_body<3, KPL, U>(a, yt, LyP, r, first); break;
    case 4: axis_y_body<4, KPL, U>(a, yt, LyP, r, first); break;
    case 5: axis_y_body<5, KPL, U>(a, yt, LyP, r, first); break;
    case 6: axis_y_body<6, KPL, U>(a, yt, LyP, r, first); break;
    case 7: axis_y_body<7, KPL, U>(a, yt, LyP, r, first); break;
    case 8: axis_y_body<8, KPL, U>(a, yt, LyP, r, first); break;
    case 9: axis_y_body<9, KPL, U>(a, yt, LyP, r, first); break;
  }
}

// ---- sums over z and the results --------------------------------------------------
// One block per (orbit, slice, 128 components): the eight real-phase sums of
// an orbit in FP64, its up to eight momenta, the un-scaling, the source phase
// and the result layout.
template <typename R>
__global__ void __launch_bounds__(128) k_axis_z(const AxisZArgs a) {
  const int ob = blockIdx.x, tl = blockIdx.y, k = blockIdx.z * 128 + threadIdx.x;
  if (k >= a.K) return;
  const int* od = a.orb + 8 * ob;  // pairs (cos cos, cos sin, sin cos, sin sin) of (x, y), z rows (cos, sin), momenta [m0, m1)
  int pr[4];
#pragma unroll
  for (int i = 0; i < 4; i++) pr[i] = od[i];
  const int zc = od[4], zs = od[5], m0 = od[6], m1 = od[7];
  Cx<double> A[4][2];
#pragma unroll
  for (int i = 0; i < 4; i++) A[i][0] = A[i][1] = czero<double>();
  const Cx<R>* s = (const Cx<R>*)a.s2 + (long long)tl * a.Lz * a.NP * a.K + k;
  const long long zstep = (long long)a.NP * a.K;
#pragma unroll 2
  for (int z = 0; z < a.Lz; z++) {
    const double fc = zc >= 0 ? a.zt[zc * a.Lz + z] : 0.0, fs = zs >= 0 ? a.zt[zs * a.Lz + z] : 0.0;
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (pr[i] >= 0) {
        const Cx<R> v = s[z * zstep + (long long)pr[i] * a.K];
        A[i][0].x = fma(fc, (double)v.x, A[i][0].x);
        A[i][0].y = fma(fc, (double)v.y, A[i][0].y);
        A[i][1].x = fma(fs, (double)v.x, A[i][1].x);
        A[i][1].y = fma(fs, (double)v.y, A[i][1].y);
      }
  }
  double f = 1.0;
  const SliceDesc* sd = a.sl ? a.sl + tl : nullptr;
  if (a.exps)
    f = ldexp(1.0, a.kexp[2 * k] * (a.exps[2 * tl] + sd->eh[0]) + a.kexp[2 * k + 1] * (a.exps[2 * tl + 1] + sd->eh[1]));
  long long base = 0;  // result element of momentum 0, and the step from one momentum to the next
  int step = 0;
  if (a.nblocks == 0) {
    base = (long long)(sd ? sd->tau : tl) * a.oT + (long long)k * a.oK;
    step = 1;
  }
  for (int b = 0; b < a.nblocks; b++) {
    const ScatterBlock& B = a.blk[b];
    const int rel = k - B.k0;
    if (rel >= 0 && rel < B.groups * B.datasets * B.comps) {
      const int gd = rel / B.comps;
      base = B.base * sd->totalT * a.nmom + ((long long)gd * sd->totalT + sd->tau) * a.nmom * B.comps + rel % B.comps;
      step = B.comps;
    }
  }
  Cx<double>* out = (Cx<double>*)(a.nblocks ? sd->out : a.out);
  const int kq = a.kphase ? a.kphase[k] : 0;
  for (int m = m0; m < m1; m++) {
    const int* md = a.omom + 8 * m;  // momentum index, signs of (x, y, z) times the transform's sign, n
    const double sx = md[1], sy = md[2], sz = md[3];
    // exp(i s.theta) = (cx + i sx Sx)(cy + i sy Sy)(cz + i sz Sz)
    Cx<double> v = A[0][0];
    v.x -= sx * sy * A[3][0].x + sz * (sx * A[2][1].x + sy * A[1][1].x);
    v.y -= sx * sy * A[3][0].y + sz * (sx * A[2][1].y + sy * A[1][1].y);
    // terms with one or three sines carry i and -i
    const double ix = sx * A[2][0].x + sy * A[1][0].x + sz * A[0][1].x - sx * sy * sz * A[3][1].x;
    const double iy = sx * A[2][0].y + sy * A[1][0].y + sz * A[0][1].y - sx * sy * sz * A[3][1].y;
    v = cx<double>((v.x - iy) * f, (v.y + ix) * f);
    if (a.nblocks) v = cmul(v, source_phase(md + 4, sd->x0, a.L));
    if (kq & 1) v = cx<double>(-v.y, v.x);
    if (kq & 2) v = cx<double>(-v.x, -v.y);
    out[base + (long long)md[0] * step] = v;
  }
}

template <typename R, int R1>
cudaError_t launch_x(const AxisXArgs& a, cudaStream_t s) {
  using C = XChunk<R>;
  const int smem = kXWarps * 2 * C::stage * 2 * (int)sizeof(R) + a.Lx * R1 * (int)sizeof(R);
  cudaError_t e = ensure_smem((const void*)k_axis_x<R, R1>, smem);
  if (e != cudaSuccess) return e;
  const long long rows_per = kLines / a.KL;
  const long long items = (a.rows + rows_per - 1) / rows_per * ((a.K + a.KL - 1) / a.KL) * a.ntau;
  k_axis_x<R, R1><<<(unsigned)((items + kXWarps - 1) / kXWarps), 32 * kXWarps, smem, s>>>(a);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launch_x_t(const AxisXArgs& a, cudaStream_t s) {
  switch (a.R1) {
    case 1: return launch_x<R, 1>(a, s);
    case 3: return launch_x<R, 3>(a, s);
    case 5: return launch_x<R, 5>(a, s);
    case 7: return launch_x<R, 7>(a, s);
    case 9: return launch_x<R, 9>(a, s);
  }
  return cudaErrorInvalidValue;
}

template <typename R, int KPL, int W>
cudaError_t launch_y(const AxisYArgs& a0, int nsm, cudaStream_t s) {
  AxisYArgs a = a0;
  // as many z per block as leave about eight blocks per SM: a block fills the phase table first
  const long long per_z = (long long)((a.K + 32 * KPL - 1) / (32 * KPL)) * a.ntau;
  a.zper = (int)std::max<long long>(1, std::min<long long>(a.Lz, per_z * a.Lz / (8 * nsm)));
  const int smem = a.RY * ((a.Ly + kYUnroll - 1) / kYUnroll * kYUnroll) * (int)sizeof(R);
  if (smem > 48 << 10) {
    cudaError_t e = ensure_smem((const void*)k_axis_y<R, KPL, W>, smem);
    if (e != cudaSuccess) return e;
  }
  const dim3 grid((a.K + 32 * KPL - 1) / (32 * KPL), (a.Lz + a.zper - 1) / a.zper, a.ntau);
  k_axis_y<R, KPL, W><<<grid, 32 * a.R1, smem, s>>>(a);
  return cudaGetLastError();
}

// The rows of one axis: for every distinct a its cos row and, unless a = 0 or
// a = L/2, its sin row.
struct AxisRows {
  std::vector<int> a, cos_row, sin_row;  // per distinct a
  std::vector<int> row_a, row_sin;       // per row
  int find(int v) const {
    for (size_t i = 0; i < a.size(); i++)
      if (a[i] == v) return (int)i;
    return -1;
  }
  int add(int v, int L) {
    int i = find(v);
    if (i >= 0) return i;
    i = (int)a.size();
    a.push_back(v);
    cos_row.push_back((int)row_a.size());
    row_a.push_back(v);
    row_sin.push_back(0);
    if (v != 0 && 2 * v != L) {
      sin_row.push_back((int)row_a.size());
      row_a.push_back(v);
      row_sin.push_back(1);
    } else {
      sin_row.push_back(-1);
    }
    return i;
  }
};

}  // namespace

cudaError_t launch_axis_x(const AxisXArgs& a0, int fp32, cudaStream_t s) {
  if (a0.ntau < 1 || a0.K < 1) return cudaSuccess;
  AxisXArgs a = a0;
  a.KL = 1;
  while (a.KL < 32 && a.KL < a.K) a.KL *= 2;
  return fp32 ? launch_x_t<float>(a, s) : launch_x_t<double>(a, s);
}

cudaError_t launch_axis_y(const AxisYArgs& a, int fp32, int kpl, int nsm, cudaStream_t s) {
  constexpr int W = kAxisMaxRows;
  if (!fp32) return kpl == 2 ? launch_y<double, 2, W>(a, nsm, s) : launch_y<double, 1, W>(a, nsm, s);
  if (a.R1 <= 7) return kpl == 2 ? launch_y<float, 2, 7>(a, nsm, s) : launch_y<float, 1, 7>(a, nsm, s);
  return kpl == 2 ? launch_y<float, 2, W>(a, nsm, s) : launch_y<float, 1, W>(a, nsm, s);
}

cudaError_t launch_axis_z(const AxisZArgs& a, int fp32, cudaStream_t s) {
  const dim3 grid(a.NO, a.ntau, (a.K + 127) / 128);
  if (fp32)
    k_axis_z<float><<<grid, 128, 0, s>>>(a);
  else
    k_axis_z<double><<<grid, 128, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace p2

namespace p2host {

// Whether a momentum list takes the axis-by-axis projection, and its tables
// on the device (kept per transform sign until the list changes).
// The list qualifies when no axis has more than kAxisMaxRows rows (|n| <= 4,
// every list up to |n|^2 <= 24).  The line is where the instantiations end, not
// where the direct projections win: with eleven rows (|n|^2 <= 25, 515 momenta) a
// build of these kernels took 2.4 ms at 24^3 x 24 slices in FP64, 288 components,
// where the direct sum takes 28.7, 4.3 ms against 7.1 of the tensor cores at 48^3 x
// 12, and 0.22 ms against 8.8 (FP64) and 0.71 for a field of 32 components.
p2_status axes_prepare(p2_ctx* c, const std::vector<int>& moms, int sign, const AxesPlan** out) {
  *out = nullptr;
  AxesPlan& ap = c->axes[sign > 0 ? 1 : 0];
  if (ap.key == moms) {
    if (ap.usable) *out = &ap;
    return P2_OK;
  }
  ap.key.clear();
  ap.usable = false;
  const int nmom = (int)moms.size() / 3;
  p2::AxisRows ax[3];
  std::vector<int> ia(3 * (size_t)nmom), sg(3 * (size_t)nmom);
  bool fits = true;
  for (int p = 0; p < nmom && fits; p++)
    for (int d = 0; d < 3; d++) {
      const int L = c->g.L[d];
      int m = moms[3 * p + d] % L;
      if (m < 0) m += L;
      const int a = std::min(m, L - m);
      ia[3 * p + d] = ax[d].add(a, L);
      sg[3 * p + d] = m == a ? 1 : -1;
      fits = fits && (int)ax[d].row_a.size() <= p2::kAxisMaxRows;
    }
  if (!fits || c->Ll[0] > 1024 || c->Ll[1] > 2048) {  // the phase tables fit in shared memory (73 and 148 KB)
    ap.key = moms;
    return P2_OK;
  }
  const int R1 = (int)ax[0].row_a.size() | 1;  // odd: the x sums are instantiated for 1, 3, 5, 7 and 9 rows
  const int RY = (int)ax[1].row_a.size(), RZ = (int)ax[2].row_a.size();
  // (x row, y row) pairs, ordered by x row
  std::vector<std::vector<int>> ylist(R1);
  auto use = [&](int r, int s) {
    if (r >= 0 && s >= 0 && std::find(ylist[r].begin(), ylist[r].end(), s) == ylist[r].end()) ylist[r].push_back(s);
  };
  for (int p = 0; p < nmom; p++)
    for (int i = 0; i < 2; i++)
      for (int j = 0; j < 2; j++)
        use(i ? ax[0].sin_row[ia[3 * p]] : ax[0].cos_row[ia[3 * p]],
            j ? ax[1].sin_row[ia[3 * p + 1]] : ax[1].cos_row[ia[3 * p + 1]]);
  std::vector<int> first(R1 + 1, 0), yl;
  for (int r = 0; r < R1; r++) {
    first[r] = (int)yl.size();
    yl.insert(yl.end(), ylist[r].begin(), ylist[r].end());
  }
  first[R1] = (int)yl.size();
  auto pair_of = [&](int r, int s) {
    if (r < 0 || s < 0) return -1;
    return first[r] + (int)(std::find(ylist[r].begin(), ylist[r].end(), s) - ylist[r].begin());
  };
  // orbits and their momenta, in first-occurrence order
  std::vector<int> orb, omom;
  std::vector<std::vector<int>> members;
  std::vector<int> okey;
  for (int p = 0; p < nmom; p++) {
    const int key = (ia[3 * p] * 64 + ia[3 * p + 1]) * 64 + ia[3 * p + 2];
    size_t o = std::find(okey.begin(), okey.end(), key) - okey.begin();
    if (o == okey.size()) {
      okey.push_back(key);
      members.emplace_back();
    }
    members[o].push_back(p);
  }
  for (const auto& mem : members) {
    const int p0 = mem[0];
    const int xc = ax[0].cos_row[ia[3 * p0]], xs = ax[0].sin_row[ia[3 * p0]];
    const int yc = ax[1].cos_row[ia[3 * p0 + 1]], ysn = ax[1].sin_row[ia[3 * p0 + 1]];
    for (int v : {pair_of(xc, yc), pair_of(xc, ysn), pair_of(xs, yc), pair_of(xs, ysn),
                  ax[2].cos_row[ia[3 * p0 + 2]], ax[2].sin_row[ia[3 * p0 + 2]], (int)omom.size() / 8,
                  (int)(omom.size() / 8 + mem.size())})
      orb.push_back(v);
    for (int p : mem) {
      omom.push_back(p);
      for (int d = 0; d < 3; d++) omom.push_back(sign * sg[3 * p + d]);
      for (int d = 0; d < 3; d++) omom.push_back(moms[3 * p + d]);
      omom.push_back(0);
    }
  }
  // phase tables in global coordinates, a x reduced mod L in integers
  std::vector<double> tab;
  auto value = [&](int d, int a, int is_sin, int xl) {
    const long long L = c->g.L[d], xg = xl + (long long)c->g.coords[d] * c->Ll[d];
    const double ph = 2.0 * M_PI * (double)((a * xg) % L) / (double)L;
    return is_sin ? std::sin(ph) : std::cos(ph);
  };
  for (int x = 0; x < c->Ll[0]; x++)
    for (int r = 0; r < R1; r++)
      tab.push_back(r < (int)ax[0].row_a.size() ? value(0, ax[0].row_a[r], ax[0].row_sin[r], x) : 0.0);
  const size_t oy = tab.size();
  for (int r = 0; r < RY; r++)
    for (int y = 0; y < c->Ll[1]; y++) tab.push_back(value(1, ax[1].row_a[r], ax[1].row_sin[r], y));
  const size_t oz = tab.size();
  for (int r = 0; r < RZ; r++)
    for (int z = 0; z < c->Ll[2]; z++) tab.push_back(value(2, ax[2].row_a[r], ax[2].row_sin[r], z));
  std::vector<int> idx(orb);
  const size_t om = idx.size();
  idx.insert(idx.end(), omom.begin(), omom.end());
  p2_status st;
  std::vector<unsigned char> up(tab.size() * sizeof(double) + idx.size() * sizeof(int));
  std::memcpy(up.data(), tab.data(), tab.size() * sizeof(double));
  std::memcpy(up.data() + tab.size() * sizeof(double), idx.data(), idx.size() * sizeof(int));
  if ((st = upload_async(c, ap.tab, up.data(), up.size(), "axis tables")) != P2_OK) return st;
  ap.R1 = R1;
  ap.RY = RY;
  ap.NP = (int)yl.size();
  ap.NO = (int)members.size();
  ap.nmom = nmom;
  ap.xth.assign(tab.begin(), tab.begin() + oy);
  ap.xt = (const double*)ap.tab.p;
  ap.yt = ap.xt + oy;
  ap.zt = ap.xt + oz;
  ap.first = first;
  ap.ylist = yl;
  ap.orb = (const int*)(ap.xt + tab.size());
  ap.omom = ap.orb + om;
  ap.usable = true;
  ap.key = moms;
  *out = &ap;
  return P2_OK;
}

size_t axes_s1_bytes(const p2_ctx* c, const AxesPlan& ap, int fp32, size_t n, size_t K) {
  return (n * c->Ll[1] * c->Ll[2] * ap.R1 * K * (fp32 ? 8 : 16) + 255) / 256 * 256;
}
size_t axes_ws_bytes(const p2_ctx* c, const AxesPlan& ap, int fp32, size_t n, size_t K) {
  return axes_s1_bytes(c, ap, fp32, n, K) + n * c->Ll[2] * ap.NP * K * (fp32 ? 8 : 16);
}

// Sums over x of n slices of K components of a position buffer into the
// first K of the Kst components of s1.
p2_status axes_x(p2_ctx* c, const AxesPlan& ap, const void* field, int fp32, long long sT, long long sK, int n, int K,
                 int Kst, void* s1) {
  p2::AxisXArgs a{};
  a.c = field;
  a.Kst = Kst;
  a.sT = sT;
  a.sK = sK;
  a.ntau = n;
  a.K = K;
  a.rows = c->Ll[1] * c->Ll[2];
  a.Lx = c->Ll[0];
  a.R1 = ap.R1;
  a.xt = ap.xt;
  a.s1 = s1;
  ProfScope ps(c, "project_axis_x");
  P2_TRY(c, p2::launch_axis_x(a, fp32, c->stream), "projection over x");
  return P2_OK;
}

// The Delta (from the second nucleon interpolator too: they share no work),
// and the nucleon with the 16 x 16 mesons unless other blocks of their pass
// are requested; the rest goes through a position buffer.  The Delta alone
// gains from it beside such blocks (24^3 x 48 light baryons 4.77 -> 4.34 ms, odd
// plain lattice 2.54 -> 2.39 ms), the nucleon would read its propagators a
// second time.  Lists and lattices whose x phases exceed the parameters keep
// the position buffer, and so does the nucleon alone in the split form on
// lattices of 200000 sites or more: most of a fused tile's time is spent on what
// the mesons share (with, without the fusion, us: 48^3 x 96 1564, 1334; 24^3 x 48
// 645, 600; 25 x 16 x 29 x 30 666, 555; but 16^3 x 32 173, 181; 8^3 x 16 60, 69).
unsigned fused_bits(const p2_ctx* c, const AxesPlan* ap, unsigned what, int split) {
  constexpr unsigned kDelta = P2_DELTA_ISO12 | P2_DELTA_ISO32, kMes = P2_NUCLEON_CG5 | P2_MESON_G16;
  constexpr unsigned kPass2 = kDelta | P2_NUCLEON_NTOR | P2_NUCLEON_RTON | P2_NUCLEON_RTOR;
  if (!ap || c->Ll[0] * (ap->R1 <= 3 ? 4 : ap->R1 <= 7 ? 8 : 12) > p2::kRowsMaxPhases) return 0;
  if (split && c->Ll[0] > p2::kRowsMaxSplit) return 0;
  unsigned mes = what & ~(kPass2 | kMes) ? 0u : what & kMes;
  if (split && mes == P2_NUCLEON_CG5 && c->V3 * c->Ll[3] >= 200000) mes = 0;
  return (what & kDelta) | mes;
}

// On a short x axis the sums over x leave about as much as they read, and the
// tensor-core projection is the faster one where its rows fit one tile of 128
// and the lattice is not so small that launches decide (nucleon and 16 x 16
// mesons, us, sums and tensor cores: 7 x 10 x 10 x 24 164 and 178, 7 x 20 x 20 x 16
// 158 and 153, 6 x 40 x 40 x 16 365 and 320; without an x axis to sum over, 1 x 32 x
// 32 x 16 200 and 152).  `shortest` is the first Lx where the sums win.  Measured at Lx x 48 x 40, 8 slices, 123 momenta, us, sums
// and tensor cores: nucleon and 16 x 16 mesons, fused, Lx = 4 359 and 327, 6 429
// and 363, 8 465 and 446, 16 737 and 774; 16 x 16 mesons alone 6 317 and 288, 8
// 334 and 351; 34 mesons, not fused, 8 301 and 275, 16 468 and 450; nucleon, not
// fused, 8 281 and 268, 16 449 and 446; u, d table-driven 3 425 and 409, 4 552 and 544.
bool axes_faster(const p2_ctx* c, int nmom, int shortest) {
  return c->V3 * c->Ll[3] < (c->Ll[0] > 1 ? 100000 : 10000) || nmom > 128 || c->Ll[0] >= shortest;
}

p2_status axes_x_blocks(p2_ctx* c, const AxesPlan& ap, unsigned what, unsigned rest, const void* cbuf, int fp32, int n,
                        void* s1) {
  const size_t esz = fp32 ? 8 : 16;
  const int K = components_of(what), Kr = components_of(rest);
  // runs of neighbouring blocks of `rest`, [k0, k1) in `what`, from component q0 of the buffer
  int k0 = 0, k1 = 0, q0 = 0;
  for (size_t i = 0; i <= sizeof(kBlocks) / sizeof(kBlocks[0]); i++) {
    const bool end = i == sizeof(kBlocks) / sizeof(kBlocks[0]);
    if (!end && !(what & kBlocks[i].bit)) continue;
    const int comps = end ? 0 : kBlocks[i].groups * kBlocks[i].datasets * kBlocks[i].comps;
    if (!end && (rest & kBlocks[i].bit)) {
      k1 += comps;
      continue;
    }
    if (k1 > k0) {
      p2_status st = axes_x(c, ap, (const char*)cbuf + (size_t)q0 * c->V3 * esz, fp32, (long long)Kr * c->V3, c->V3, n,
                            k1 - k0, K, (char*)s1 + (size_t)k0 * esz);
      if (st != P2_OK) return st;
      q0 += k1 - k0;
    }
    k0 = k1 = k1 + comps;
  }
  return P2_OK;
}

// Sums over y and z of S1 (n slices, K components), then the results: with
// blocks into the slices' results dsl, otherwise into out[tau * oT + k * oK + p].
p2_status axes_yz(p2_ctx* c, const AxesPlan& ap, const void* s1, int fp32, int n, int K, const AxesOut& o) {
  const int Lz = c->Ll[2];
  void* const s2 = (char*)s1 + axes_s1_bytes(c, ap, fp32, n, K);
  p2::AxisYArgs y{};
  y.s1 = s1;
  y.s2 = s2;
  y.ntau = n;
  y.K = K;
  y.Ly = c->Ll[1];
  y.Lz = Lz;
  y.R1 = ap.R1;
  y.RY = ap.RY;
  y.NP = ap.NP;
  y.yt = ap.yt;
  std::copy(ap.first.begin(), ap.first.end(), y.first);
  std::copy(ap.ylist.begin(), ap.ylist.end(), y.ylist);
  // two components per lane share each phase; one where that leaves too few blocks to fill the SMs
  // (FP64: the registers of two halve the warps in flight)
  std::vector<std::vector<int>> cands{{1}, {2}};
  if (fp32 && (long long)n * Lz * ((K + 63) / 64) >= 2LL * c->nsm) std::swap(cands[0], cands[1]);
  char key[160];
  std::snprintf(key, sizeof(key), "%s axes y=%d z=%d rows=%d pairs=%d K=%d n=%d",
                fp32 ? "project_split" : "project_fp64", y.Ly, Lz, ap.R1, ap.NP, K, n);
  std::vector<int> pick;
  P2_TRY(c,
         tune_choose(c->tuner.get(), key, cands, c->stream, !c->capturing,
                     [&](const std::vector<int>& v) { return p2::launch_axis_y(y, fp32, v[0], c->nsm, c->stream); }, pick),
         "projection tuning");
  {
    ProfScope ps(c, "project_axis_y");
    P2_TRY(c, p2::launch_axis_y(y, fp32, pick[0], c->nsm, c->stream), "projection over y");
  }
  p2::AxisZArgs z{};
  z.s2 = s2;
  z.ntau = n;
  z.K = K;
  z.Lz = Lz;
  z.NP = ap.NP;
  z.NO = ap.NO;
  z.nmom = ap.nmom;
  z.zt = ap.zt;
  z.orb = ap.orb;
  z.omom = ap.omom;
  z.sl = o.dsl;
  for (int d = 0; d < 3; d++) z.L[d] = c->g.L[d];
  z.exps = o.exps;
  z.kexp = o.kexp;
  z.kphase = o.kphase;
  const size_t nb = o.blocks ? o.blocks->size() : 0;
  if (nb > (size_t)p2::kMaxBlocks) return c->fail(P2_ERR_INVALID_ARG, "too many result blocks");
  z.nblocks = (int)nb;
  for (size_t b = 0; b < nb; b++) z.blk[b] = (*o.blocks)[b];
  z.out = o.out;
  z.oT = o.oT;
  z.oK = o.oK;
  ProfScope ps(c, "project_axis_z");
  P2_TRY(c, p2::launch_axis_z(z, fp32, c->stream), "projection over z");
  return P2_OK;
}

}  // namespace p2host
