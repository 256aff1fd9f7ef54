// FP32 pointwise kernels of the FFNO3D forward: lift, input gates, the 2-layer channel MLPs with fused residual
// prologues and GroupNorm-statistics epilogues, the branch-gate/fuse chain and the projection + level-fraction head.
// Every kernel is persistent over 64-voxel tiles (grid-stride), so the GroupNorm partials it writes have one row per
// CTA and a fixed summation order.
#include <math.h>

#include "common.cuh"
#include "gemm_f32.cuh"

using namespace ffno;

namespace {

int g_num_sms = 0;

int num_sms() {
  if (!g_num_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 152;
  }
  return g_num_sms;
}

__host__ __device__ __forceinline__ long ntiles_of(long V) { return (V + BM - 1) / BM; }

int grid_for(long V, int per_sm) {
  long t = ntiles_of(V);
  long g = (long)num_sms() * per_sm;
  return (int)(t < g ? (t > 0 ? t : 1) : g);
}

// CTAs an SM of the statistics chains (k_mlp2, k_fuse): three of 80 registers a thread, two where the accumulators of a
// 2C = 192 column GEMM need up to 128.
__host__ __device__ constexpr int tile_ctas(int C) { return C <= 64 ? 3 : 2; }

template <typename K>
bool set_smem(K kernel, size_t bytes) {
  return ffno::smem_cap_ok(kernel, bytes);
}

// ------------------------------------------------------------------------------------------------ depth weights
// A CTA holds DW_COLS neighbouring columns (coalesced rows), DW_SEGS threads share each column's levels, and the column
// sum is the fixed-order sum of the segments' sums. Bound by latency: with one thread a column, each of its D levels waited for
// memory twice. 101 x 45 x 75: 37 -> 5 us.
constexpr int DW_COLS = 32, DW_SEGS = 16;

__global__ void __launch_bounds__(DW_COLS* DW_SEGS) k_depth_weights(const float* __restrict__ z, int D, long HW,
                                                                    float* __restrict__ w) {
  griddep_sync();
  __shared__ float part[DW_SEGS][DW_COLS];
  const int tx = threadIdx.x % DW_COLS, sg = threadIdx.x / DW_COLS;
  const long col = (long)blockIdx.x * DW_COLS + tx;
  const bool ok = col < HW;
  if (D == 1) {
    if (ok && sg == 0) w[col] = 1.f;
    return;
  }
  // share of level d: half the distances to its neighbours
  auto share = [&](int d) {
    const float zd = __ldg(z + (long)d * HW + col);
    const float lo = d > 0 ? 0.5f * fabsf(zd - __ldg(z + (long)(d - 1) * HW + col)) : 0.f;
    const float hi = d + 1 < D ? 0.5f * fabsf(__ldg(z + (long)(d + 1) * HW + col) - zd) : 0.f;
    return lo + hi;
  };
  float s = 0.f;
  if (ok) {
#pragma unroll 4
    for (int d = sg; d < D; d += DW_SEGS) s += share(d);
  }
  part[sg][tx] = s;
  __syncthreads();
  if (!ok) return;
  s = 0.f;
#pragma unroll
  for (int i = 0; i < DW_SEGS; ++i) s += part[i][tx];
  const float mean = fmaxf(s / (float)D, 1e-12f);
#pragma unroll 4
  for (int d = sg; d < D; d += DW_SEGS) w[(long)d * HW + col] = share(d) / mean;
}

// ------------------------------------------------------------------------------------------------ column info
__global__ void k_column_info(const float* __restrict__ z, int D, long HW, unsigned int* __restrict__ flags) {
  griddep_sync();
  // flags[0]: 1 while every column equals column 0 (each shifted by its own minimum); flags[1]: float bits of the
  // largest span (non-negative floats order as unsigned ints)
  const long col = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (col >= HW) return;
  float mn = z[col], mx = z[col], mn0 = z[0];
  for (int d = 1; d < D; ++d) {
    const float v = z[(long)d * HW + col];
    mn = fminf(mn, v);
    mx = fmaxf(mx, v);
    mn0 = fminf(mn0, z[(long)d * HW]);
  }
  bool same = true;
  for (int d = 0; d < D && same; ++d) same = (z[(long)d * HW + col] - mn) == (z[(long)d * HW] - mn0);
  if (!same) atomicAnd(flags, 0u);
  atomicMax(flags + 1, __float_as_uint(mx - mn));
}

__global__ void k_column_info_init(unsigned int* flags) {
  griddep_sync();
  flags[0] = 1u;
  flags[1] = 0u;
}

__global__ void k_column_info_final(unsigned int* flags) {
  griddep_sync();
  float* out = reinterpret_cast<float*>(flags);
  const unsigned int s = flags[0];
  out[0] = s ? 1.f : 0.f;  // flags[1] already holds the span's float bits
}

// ------------------------------------------------------------------------------------------------ lift
// x_in arrives channels-first: a tile's rows of each input channel are 64 consecutive floats. The thread mapping is the tile
// GEMM's (4 voxels x C / 16 channels, 16-byte stores, 4-barrier statistics); bound by the store of pre. 4.2 M voxels,
// C = 64: 1.34 -> 0.53 ms.
template <int C>
__global__ void __launch_bounds__(NT, 3) k_lift(const float* __restrict__ xin, int cin, long V,
                                                const float* __restrict__ wl, const float* __restrict__ dw,
                                                float* __restrict__ pre, double* __restrict__ partials, int cpg,
                                                int groups, int al) {
  griddep_sync();
  __shared__ __align__(16) float xs[2][8][BM];
  __shared__ __align__(16) float ws[8][C];
  __shared__ g32::TileStats<C> st;
  using Cl = g32::Cols<C, 1>;
  const int tx = g32::tile_tx(), ty = g32::tile_ty();
  ShiftAcc acc_g;
  const long nt = ntiles_of(V);
  for (int e = threadIdx.x; e < cin * C; e += NT) ws[e / C][e % C] = __ldg(wl + e);
  // the next tile's inputs wait in registers (at most 2 of the 8 x 64 values a thread) while this one is processed
  float nx[2];
  auto fetch = [&](long t) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int e = threadIdx.x + i * NT, k = e / BM, r = e % BM;
      const long v = t * BM + r;
      nx[i] = k < cin && t < nt && v < V ? __ldg(xin + (long)k * V + v) : 0.f;
    }
  };
  fetch(blockIdx.x);
  int buf = 0;
  for (long t = blockIdx.x; t < nt; t += gridDim.x, buf ^= 1) {
    const long v0 = t * BM;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int e = threadIdx.x + i * NT;
      xs[buf][e / BM][e % BM] = nx[i];
    }
    __syncthreads();
    fetch(t + gridDim.x);
    float acc[C / 16][4], wr[4];
#pragma unroll
    for (int j = 0; j < C / 16; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
    for (int k = 0; k < cin; ++k) {
      const float4 q = *reinterpret_cast<const float4*>(&xs[buf][k][4 * ty]);
      const float x[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int j = 0; j < C / 16; ++j) {
        const float w = ws[k][Cl::col(tx, j)];
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = fmaf(x[e], w, acc[j][e]);
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const long v = v0 + 4 * ty + e;
      wr[e] = v < V ? __ldg(dw + v) : 0.f;
    }
    g32::store_rows<C>(pre, nullptr, v0, V, acc, al);
    g32::tile_stats<C>(acc, wr, cpg, groups, st, acc_g);
  }
  g32::write_tile_partial(partials, gridDim.x, groups, acc_g);
}

// ------------------------------------------------------------------------------------------------ GN finalize
// One CTA per group, each thread a few partials: the group's mean is the weighted mean of the partials' means, and its
// M2 the sum of the partials' M2 and of w (mean_p - mean)^2, so the loops hold no division (a serial Chan merge has two
// dependent FP64 divisions per partial). Bound by latency: two passes over at most a few partials a thread, two
// block-wide sums in a fixed tree (deterministic), one FP64 division. The groups take a CTA each because the FP64 rate of
// one SM (about two operations a cycle) would serialise eight groups of 304 partials; they spread over the SMs where the
// device places them, and above width 64 the launch keeps them on different ones (ffno_gn_finalize has the figures).
// 304 partials, 8 groups, C = 64: 22.0 us a launch in the form before (one CTA, a warp per group, Chan merges), 6.6 us in
// this one (a chain of three block sums, a division and a square root).
constexpr int FIN_NT = 128;

__device__ __forceinline__ double block_sum(double v, double* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < FIN_NT / 32; ++w) s += red[w];
  return s;
}

__global__ void __launch_bounds__(FIN_NT) k_gn_finalize(const double* __restrict__ partials, int nparts, int C,
                                                        int groups, const float* __restrict__ gamma,
                                                        const float* __restrict__ beta, float eps,
                                                        float* __restrict__ coefs, double* __restrict__ gstats) {
  griddep_sync();
  __shared__ double red[3][FIN_NT / 32];
  const int g = blockIdx.x, tid = threadIdx.x;
  double w = 0.0, wm = 0.0;
  for (int p = tid; p < nparts; p += FIN_NT) {
    const double* q = partials + ((long)p * groups + g) * 3;
    if (!(q[0] <= 0.0)) {   // a NaN weight counts
      w += q[0];
      wm += q[0] * q[1];
    }
  }
  const double wt = block_sum(w, red[0]);
  const double ms = block_sum(wm, red[1]);
  const double mean = wt == 0.0 ? 0.0 : ms / wt;
  double m2 = 0.0;
  for (int p = tid; p < nparts; p += FIN_NT) {
    const double* q = partials + ((long)p * groups + g) * 3;
    if (!(q[0] <= 0.0)) {
      const double d = q[1] - mean;
      m2 += q[2] + q[0] * d * d;
    }
  }
  m2 = block_sum(m2, red[2]);
  const double var = wt > 0.0 ? m2 / wt : 0.0;
  const double rstd = 1.0 / sqrt(var + (double)eps);
  if (tid == 0 && gstats) {
    gstats[3 * g] = mean;
    gstats[3 * g + 1] = rstd;
    gstats[3 * g + 2] = wt;
  }
  const int cpg = C / groups;
  for (int i = tid; i < cpg; i += FIN_NT) {
    const int c = g * cpg + i;
    coefs[c] = (float)mean;
    coefs[C + c] = (float)((double)gamma[c] * rstd);
    coefs[2 * C + c] = beta[c];
  }
}

// ------------------------------------------------------------------------------------------------ elementwise
// y = GN(pre) from the finalized coefficients, 4 channels a thread (float4), two float4 in flight per round; the
// channel index from a 32-bit modulo (n / 4 < 2^31 is checked by the launchers).
__device__ __forceinline__ float4 gn4(float4 p, const float* __restrict__ cf, int C, int c, int al = 1) {
  const float4 m = g32::ldq(cf + c, true, al);
  const float4 sc = g32::ldq(cf + C + c, true, al);
  const float4 b = g32::ldq(cf + 2 * C + c, true, al);
  return make_float4((p.x - m.x) * sc.x + b.x, (p.y - m.y) * sc.y + b.y, (p.z - m.z) * sc.z + b.z,
                     (p.w - m.w) * sc.w + b.w);
}

__global__ void k_gn_act(const float* __restrict__ pre, const float* __restrict__ coefs, unsigned n4, int C, int act,
                         float* __restrict__ out) {
  griddep_sync();
  const unsigned C4 = (unsigned)C / 4, stride = gridDim.x * blockDim.x;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += 2 * stride) {
    const unsigned i2 = i + stride;
    const float4 p0 = __ldg(reinterpret_cast<const float4*>(pre) + i);
    const float4 p1 = i2 < n4 ? __ldg(reinterpret_cast<const float4*>(pre) + i2) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 y = gn4(p0, coefs, C, (int)(i % C4) * 4);
    if (act) y = make_float4(gelu(y.x), gelu(y.y), gelu(y.z), gelu(y.w));
    reinterpret_cast<float4*>(out)[i] = y;
    if (i2 < n4) {
      y = gn4(p1, coefs, C, (int)(i2 % C4) * 4);
      if (act) y = make_float4(gelu(y.x), gelu(y.y), gelu(y.z), gelu(y.w));
      reinterpret_cast<float4*>(out)[i2] = y;
    }
  }
}

__global__ void k_resid_out(const float* __restrict__ x2, const float* __restrict__ pre,
                            const float* __restrict__ coefs, float res, unsigned n4, int C, float* __restrict__ out) {
  griddep_sync();
  const unsigned C4 = (unsigned)C / 4, stride = gridDim.x * blockDim.x;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += 2 * stride) {
    const unsigned i2 = i + stride;
    const bool two = i2 < n4;
    const float4 p0 = __ldg(reinterpret_cast<const float4*>(pre) + i);
    const float4 a0 = __ldg(reinterpret_cast<const float4*>(x2) + i);
    const float4 p1 = two ? __ldg(reinterpret_cast<const float4*>(pre) + i2) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 a1 = two ? __ldg(reinterpret_cast<const float4*>(x2) + i2) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 y = gn4(p0, coefs, C, (int)(i % C4) * 4);
    reinterpret_cast<float4*>(out)[i] =
        make_float4(fmaf(res, y.x, a0.x), fmaf(res, y.y, a0.y), fmaf(res, y.z, a0.z), fmaf(res, y.w, a0.w));
    if (two) {
      y = gn4(p1, coefs, C, (int)(i2 % C4) * 4);
      reinterpret_cast<float4*>(out)[i2] =
          make_float4(fmaf(res, y.x, a1.x), fmaf(res, y.y, a1.y), fmaf(res, y.z, a1.z), fmaf(res, y.w, a1.w));
    }
  }
}

// ------------------------------------------------------------------------------------------------ input gate
// 4.2 M voxels, C = 64: 4.65 -> 2.12 ms (32 TFLOP/s), four CTAs an SM.
template <int C>
__global__ void __launch_bounds__(NT, C <= 64 ? 4 : 2) k_gate(const float* __restrict__ x, long V, const float* __restrict__ w1,
                                                const float* __restrict__ w2, const float* __restrict__ zp,
                                                const float* __restrict__ z, float* __restrict__ out, int al) {
  griddep_sync();
  extern __shared__ __align__(16) float sm[];
  float* xs = sm;             // [C][64]
  float* hs = xs + C * BM;    // [C][64]
  g32::Ring ring(hs + C * BM, g32::KC * C, al);
  using Cl = g32::Cols<C, 1>;
  const int tx = g32::tile_tx(), ty = g32::tile_ty();
  const long nt = ntiles_of(V);
  for (long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long v0 = t * BM;
    __syncthreads();
    ring.pre<C>(w1, C);
    g32::load_tile<C>(xs, 0, x, v0, V, al);
    float acc[C / 16][4];
    g32::gemm<C, C>(xs, 0, w1, C, ring, acc);
    ring.pre<C>(w2, C);
#pragma unroll
    for (int j = 0; j < C / 16; ++j) {
      float h[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) h[e] = gelu(acc[j][e]);
      g32::put4(hs, Cl::col(tx, j), h);
    }
    g32::gemm<C, C>(hs, 0, w2, C, ring, acc);
    float zv[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const long v = v0 + 4 * ty + e;
      zv[e] = zp && v < V ? __ldg(z + v) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < C / 16; ++j) {
      const int c = Cl::col(tx, j);
      float xv[4];
      g32::get4(xs, c, xv);
      const float zc = zp ? __ldg(zp + c) : 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float o = xv[e] * sigmoid(acc[j][e]);
        acc[j][e] = zp ? o + zc * zv[e] : o;
      }
    }
    g32::store_rows<C>(out, nullptr, v0, V, acc, al);
  }
}

// ------------------------------------------------------------------------------------------------ 2-layer MLP
// The hidden layer overwrites the input tile's region (2C channels), so a tile takes 2C x 64 floats plus the weight
// ring: 48 KB at C = 64. Bound by the operand reads from shared memory (4 x 8 outputs a thread). 4.2 M
// voxels, C = 64: 7.1 -> 4.0 ms (34 TFLOP/s); 296 k voxels, C = 96: 861 -> 577 us.
template <int C>
constexpr size_t mlp2_smem() {
  return (2 * C * BM + 2 * g32::KC * 2 * C) * sizeof(float);
}

template <int C, int MODE>
__global__ void __launch_bounds__(NT, tile_ctas(C)) k_mlp2(const float* __restrict__ in, const float* __restrict__ prev_pre,
                                                const float* __restrict__ pc, float res, float* __restrict__ xout,
                                                long V, const float* __restrict__ w1, const float* __restrict__ w2,
                                                const float* __restrict__ dw, float* __restrict__ pre,
                                                double* __restrict__ partials, int nparts, int cpg, int groups, int al) {
  griddep_sync();
  extern __shared__ __align__(16) float sm[];
  __shared__ g32::TileStats<C> st;
  float* as = sm;   // [C][64] input, then [2C][64] hidden
  g32::Ring ring(as + 2 * C * BM, g32::KC * 2 * C, al);
  using Ch = g32::Cols<2 * C, 1>;
  const int tx = g32::tile_tx(), ty = g32::tile_ty();
  ShiftAcc acc_g;
  const long nt = ntiles_of(V);
  for (long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long v0 = t * BM;
    __syncthreads();
    ring.pre<2 * C>(w1, 2 * C);
    g32::each_quad<C>(v0, V, [&](int r, int c, long o, bool ok) {
      float4 a = g32::ldq(in + o, ok, al);
      if (MODE != 0 && ok) {
        float4 y = gn4(g32::ldq(prev_pre + o, ok, al), pc, C, c, al);
        if (MODE == 1) y = make_float4(gelu(y.x), gelu(y.y), gelu(y.z), gelu(y.w));
        a = make_float4(a.x + res * y.x, a.y + res * y.y, a.z + res * y.z, a.w + res * y.w);
        g32::stq(xout + o, a, al);
      }
      g32::put_quad(as, r, c, a);
    });
    {
      float h[2 * C / 16][4];
      g32::gemm<C, 2 * C>(as, 0, w1, 2 * C, ring, h);
      ring.pre<C>(w2, C);
      __syncthreads();   // every read of the input tile is done
#pragma unroll
      for (int j = 0; j < 2 * C / 16; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) h[j][e] = gelu(h[j][e]);
        g32::put4(as, Ch::col(tx, j), h[j]);
      }
    }
    float acc[C / 16][4], wr[4];
    g32::gemm<2 * C, C>(as, 0, w2, C, ring, acc);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const long v = v0 + 4 * ty + e;
      wr[e] = v < V ? __ldg(dw + v) : 0.f;
    }
    g32::store_rows<C>(pre, nullptr, v0, V, acc, al);
    g32::tile_stats<C>(acc, wr, cpg, groups, st, acc_g);
  }
  g32::write_tile_partial(partials, nparts, groups, acc_g);
}

// ------------------------------------------------------------------------------------------------ gate + fuse
// One region of 3C channels: [x | spec | vert], then the gate hidden layer over x, the gated branches in place, and the
// fuse hidden layer over the gated branches (their residual half-sum waits in registers): 64 KB at C = 64. 4.2 M voxels,
// C = 64: 24.1 -> 10.5 ms (36 TFLOP/s); 296 k voxels, C = 96: 3.90 -> 1.49 ms.
template <int C>
constexpr size_t fuse_smem() {
  return (3 * C * BM + 2 * g32::KC * 2 * C) * sizeof(float);
}

template <int C>
__global__ void __launch_bounds__(NT, tile_ctas(C)) k_fuse(const float* __restrict__ x, const float* __restrict__ sp,
                                                const float* __restrict__ sc, const float* __restrict__ vp,
                                                const float* __restrict__ vc, long V, const float* __restrict__ wg1,
                                                const float* __restrict__ wg2, const float* __restrict__ bg2,
                                                const float* __restrict__ wf1, const float* __restrict__ wf2,
                                                const float* __restrict__ dw, float* __restrict__ pre,
                                                double* __restrict__ partials, int nparts, int cpg, int groups, int al) {
  griddep_sync();
  extern __shared__ __align__(16) float sm[];
  __shared__ g32::TileStats<C> st;
  float* as = sm;
  g32::Ring ring(as + 3 * C * BM, g32::KC * 2 * C, al);
  using C1 = g32::Cols<C, 1>;
  using C2 = g32::Cols<2 * C, 2>;   // the thread owns channel c of both branches
  using Ch = g32::Cols<2 * C, 1>;
  const int tx = g32::tile_tx(), ty = g32::tile_ty();
  ShiftAcc acc_g;
  const long nt = ntiles_of(V);
  for (long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long v0 = t * BM;
    __syncthreads();
    ring.pre<C>(wg1, C);
    g32::each_quad<C>(v0, V, [&](int r, int c, long o, bool ok) {
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f), q = s;
      if (ok) {
        s = gn4(g32::ldq(sp + o, ok, al), sc, C, c, al);
        q = gn4(g32::ldq(vp + o, ok, al), vc, C, c, al);
        s = make_float4(gelu(s.x), gelu(s.y), gelu(s.z), gelu(s.w));
        q = make_float4(gelu(q.x), gelu(q.y), gelu(q.z), gelu(q.w));
      }
      g32::put_quad(as, r, c, g32::ldq(x + o, ok, al));
      g32::put_quad(as, r, C + c, s);
      g32::put_quad(as, r, 2 * C + c, q);
    });
    {
      float h[C / 16][4];
      g32::gemm<3 * C, C>(as, 0, wg1, C, ring, h);
      ring.pre<2 * C>(wg2, 2 * C);
      __syncthreads();   // every read of x is done
#pragma unroll
      for (int j = 0; j < C / 16; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) h[j][e] = gelu(h[j][e]);
        g32::put4(as, C1::col(tx, j), h[j]);
      }
    }
    float half[C / 16][4];
    {
      float g[2 * C / 16][4];
      g32::gemm<C, 2 * C, 2>(as, 0, wg2, 2 * C, ring, g);
      ring.pre<2 * C>(wf1, 2 * C);
      // the gates multiply spec and vert in place: gate channel n belongs to region channel C + n
#pragma unroll
      for (int j = 0; j < 2 * C / 16; ++j) {
        const int n = C2::col(tx, j);
        const float b = __ldg(bg2 + n);
        float a[4];
        g32::get4(as, C + n, a);
#pragma unroll
        for (int e = 0; e < 4; ++e) g[j][e] = a[e] * sigmoid(g[j][e] + b);
        g32::put4(as, C + n, g[j]);
      }
#pragma unroll
      for (int j = 0; j < C / 16; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) half[j][e] = 0.5f * (g[j][e] + g[j + C / 16][e]);
    }
    {
      float h[2 * C / 16][4];
      g32::gemm<2 * C, 2 * C>(as, C, wf1, 2 * C, ring, h);
      ring.pre<C>(wf2, C);
      __syncthreads();   // every read of the gated branches is done
#pragma unroll
      for (int j = 0; j < 2 * C / 16; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) h[j][e] = gelu(h[j][e]);
        g32::put4(as, Ch::col(tx, j), h[j]);
      }
    }
    float acc[C / 16][4], wr[4];
    g32::gemm<2 * C, C>(as, 0, wf2, C, ring, acc);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const long v = v0 + 4 * ty + e;
      wr[e] = v < V ? __ldg(dw + v) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < C / 16; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[j][e] += half[j][e];
    g32::store_rows<C>(pre, nullptr, v0, V, acc, al);
    g32::tile_stats<C>(acc, wr, cpg, groups, st, acc_g);
  }
  g32::write_tile_partial(partials, nparts, groups, acc_g);
}

// ------------------------------------------------------------------------------------------------ head

// The chain's two GEMMs as in the MLPs, then one thread a voxel for the level-fraction head, bound by its FP64 (log-softmax
// and LTE weights in double). 4.2 M voxels, C = 64, 12 levels: 8.5 -> 7.3 ms; 296 k voxels, C = 96: 1.11 -> 0.53 ms.
// kLte = false: FFNO3D._run_head alone (models/ffno_model.py:790-798), the head channels into head_out, no LTE head.
template <int C, int NHP, typename T, bool kLte = true>
__global__ void __launch_bounds__(NT, 2) k_head(const float* __restrict__ x, const float* __restrict__ xin, long V,
                                             const float* __restrict__ p1, const float* __restrict__ p2,
                                             const float* __restrict__ b2, int nh,
                                             const __grid_constant__ HeadParams hp, float* __restrict__ out,
                                             float* __restrict__ head_out, int al) {
  griddep_sync();
  extern __shared__ __align__(16) float sm[];
  __shared__ double etab[EXP_TAB];
  constexpr int LO = NHP + 1;
  if (kLte) fill_exp_table(etab);
  float* as = sm;                    // [C][64] input, then [2C][64] hidden
  float* os = as + 2 * C * BM;       // [64][NHP + 1] head channels
  g32::Ring ring(os + BM * LO, g32::KC * 2 * C, al);
  using Ch = g32::Cols<2 * C, 1>;
  using Co = g32::Cols<NHP, 1>;
  const int tx = g32::tile_tx(), ty = g32::tile_ty();
  const long nt = ntiles_of(V);
  for (long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long v0 = t * BM;
    __syncthreads();
    ring.pre<2 * C>(p1, 2 * C);
    g32::load_tile<C>(as, 0, x, v0, V, al);
    {
      float h[2 * C / 16][4];
      g32::gemm<C, 2 * C>(as, 0, p1, 2 * C, ring, h);
      ring.pre<NHP>(p2, NHP);
      __syncthreads();   // every read of the input tile is done
#pragma unroll
      for (int j = 0; j < 2 * C / 16; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) h[j][e] = gelu(h[j][e]);
        g32::put4(as, Ch::col(tx, j), h[j]);
      }
    }
    {
      float acc[NHP / 16][4];
      g32::gemm<2 * C, NHP>(as, 0, p2, NHP, ring, acc);
#pragma unroll
      for (int j = 0; j < NHP / 16; ++j) {
        const int n = Co::col(tx, j);
        const float b = __ldg(b2 + n);
#pragma unroll
        for (int e = 0; e < 4; ++e) os[(4 * ty + e) * LO + n] = acc[j][e] + b;
      }
    }
    __syncthreads();
    if (threadIdx.x < BM) {
      const int r = threadIdx.x;
      const long v = v0 + r;
      if (v < V) {
        const float* o = os + r * LO;
        if (head_out)
          for (int c = 0; c < nh; ++c) head_out[(long)c * V + v] = o[c];
        if constexpr (kLte) head_voxel_fwd<T>(hp, o, head_inputs(hp, xin, V, v), out, V, v, etab);
      }
    }
  }
}

// FFNO3D.head_output on head channels that are already computed (models/ffno_model.py:730-749): one thread per voxel,
// the head channels read channels-first (consecutive voxels of one channel plane per warp: coalesced), the levels
// written channels-first. Bound by HBM: (nh + 3 + levels) * 4 bytes a voxel.
template <typename T>
__global__ void __launch_bounds__(256) k_head_output(const float* __restrict__ head, const float* __restrict__ xin,
                                                     long V, int nh, const __grid_constant__ HeadParams hp,
                                                     float* __restrict__ out) {
  griddep_sync();
  __shared__ double etab[EXP_TAB];
  fill_exp_table(etab);
  __syncthreads();
  float o[FFNO_MAX_LEVELS + FFNO_MAX_SPECIES];
  for (long v = blockIdx.x * (long)blockDim.x + threadIdx.x; v < V; v += (long)gridDim.x * blockDim.x) {
    for (int c = 0; c < nh; ++c) o[c] = __ldg(head + (long)c * V + v);
    head_voxel_fwd<T>(hp, o, head_inputs(hp, xin, V, v), out, V, v, etab);
  }
}

bool width_ok(int C) { return C == 16 || C == 32 || C == 64 || C == 96; }

}  // namespace

// ====================================================================================================== C ABI
extern "C" {

const char* ffno_version(void) { return "ffnoml_gb300 0.1 (sm_103a)"; }

int ffno_stats_parts(long V) { return grid_for(V, 3); }

int ffno_depth_weights(const float* z, int D, long HW, float* w, ffno_stream_t stream) {
  if (!z || !w || D < 1 || HW < 1) return FFNO_EINVAL;
  ffno::launch(k_depth_weights, (unsigned)((HW + DW_COLS - 1) / DW_COLS), DW_COLS * DW_SEGS, 0, (cudaStream_t)stream, z, D, HW, w);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_column_info(const float* z, int D, long HW, float* out, ffno_stream_t stream) {
  if (!z || !out || D < 1 || HW < 1) return FFNO_EINVAL;
  unsigned int* flags = reinterpret_cast<unsigned int*>(out);
  ffno::launch(k_column_info_init, 1, 1, 0, (cudaStream_t)stream, flags);
  ffno::launch(k_column_info, (unsigned)((HW + 255) / 256), 256, 0, (cudaStream_t)stream, z, D, HW, flags);
  ffno::launch(k_column_info_final, 1, 1, 0, (cudaStream_t)stream, flags);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_lift_fwd(const float* x_in, int cin, long V, int C, const float* w_lift, const float* dw, float* pre,
                  double* partials, int nparts, int groups, ffno_stream_t stream) {
  if (!x_in || !w_lift || !dw || !pre || !partials) return FFNO_EINVAL;
  if (!width_ok(C) || cin < 1 || cin > 8 || V < 1 || groups < 1 || groups > GMAX || C % groups) return FFNO_EINVAL;
  if (nparts != ffno_stats_parts(V)) return FFNO_EINVAL;
  const int al = g32::aligned(pre);
  cudaStream_t s = (cudaStream_t)stream;
  const int cpg = C / groups;
  switch (C) {
#define L(CC) case CC: ffno::launch(k_lift<CC>, nparts, NT, 0, s, x_in, cin, V, w_lift, dw, pre, partials, cpg, groups, al); break;
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_gn_finalize(const double* partials, int nparts, int C, int groups, const float* gamma, const float* beta,
                     float eps, float* coefs, double* gstats, ffno_stream_t stream) {
  if (!partials || !gamma || !beta || !coefs) return FFNO_EINVAL;
  if (nparts < 1 || C < 1 || groups < 1 || groups > GMAX || C % groups) return FFNO_EINVAL;
  // Above width 64: more than half of an SM's shared memory, unused. The CTAs are FP64-bound, and placed together on the
  // SM that frees up first they took up to 25 us at width 96 instead of 9 (a forward of 296 k voxels 8.16 -> 8.07 ms).
  // Narrower models lose by it (the SMs' shared memory is set up anew around each launch): width 32, 65 k voxels,
  // 2.15 -> 2.21 ms.
  const size_t apart = C > 64 ? 116 * 1024 : 0;
  if (!ffno::smem_cap_ok(k_gn_finalize, apart)) return FFNO_ELAUNCH;
  ffno::launch(k_gn_finalize, groups, FIN_NT, apart, (cudaStream_t)stream, partials, nparts, C, groups, gamma, beta, eps, coefs,
                                                             gstats);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

bool elementwise_ok(long V, int C, const void* a, const void* b, const void* c) {
  return V >= 1 && C >= 4 && C % 4 == 0 && V * (long)C / 4 < 0x7fffffffL &&
         ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) % 16) == 0;
}

int elementwise_blocks(long n4) {
  const long want = (n4 + 511) / 512, cap = (long)num_sms() * 8;
  return (int)(want < cap ? (want > 0 ? want : 1) : cap);
}

int ffno_gn_act(const float* pre, const float* coefs, long V, int C, int act, float* out, ffno_stream_t stream) {
  if (!pre || !coefs || !out || !elementwise_ok(V, C, pre, coefs, out)) return FFNO_EINVAL;
  const long n4 = V * C / 4;
  ffno::launch(k_gn_act, elementwise_blocks(n4), 256, 0, (cudaStream_t)stream, pre, coefs, (unsigned)n4, C, act, out);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_resid_out(const float* x2, const float* pre, const float* coefs, float res, long V, int C, float* out,
                   ffno_stream_t stream) {
  if (!x2 || !pre || !coefs || !out || !elementwise_ok(V, C, x2, pre, out) ||
      reinterpret_cast<uintptr_t>(coefs) % 16)
    return FFNO_EINVAL;
  const long n4 = V * C / 4;
  ffno::launch(k_resid_out, elementwise_blocks(n4), 256, 0, (cudaStream_t)stream, x2, pre, coefs, res, (unsigned)n4, C, out);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_gate_fwd(const float* x, long V, int C, const float* w1, const float* w2, const float* zp, const float* z,
                  float* out, ffno_stream_t stream) {
  if (!x || !w1 || !w2 || !out || !width_ok(C) || V < 1 || (zp && !z)) return FFNO_EINVAL;
  cudaStream_t s = (cudaStream_t)stream;
  const size_t smem = (2 * BM * C + 2 * g32::KC * C) * sizeof(float);
  const int al = g32::aligned(x, w1, w2, out);
  switch (C) {
#define L(CC)                                                                   \
  case CC:                                                                      \
    if (!set_smem(k_gate<CC>, smem)) return FFNO_ELAUNCH;                       \
    ffno::launch(k_gate<CC>, grid_for(V, CC <= 64 ? 4 : 2), NT, smem, s, x, V, w1, w2, zp, z, out, al); \
    break;
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_mlp2_fwd(int mode, const float* in, const float* prev_pre, const float* prev_coefs, float res, float* xout,
                  long V, int C, const float* w1, const float* w2, const float* dw, float* pre, double* partials,
                  int nparts, int groups, ffno_stream_t stream) {
  if (!in || !w1 || !w2 || !dw || !pre || !partials) return FFNO_EINVAL;
  if (!width_ok(C) || V < 1 || mode < 0 || mode > 2 || groups < 1 || groups > GMAX || C % groups) return FFNO_EINVAL;
  if (mode && (!prev_pre || !prev_coefs || !xout)) return FFNO_EINVAL;
  if (nparts != ffno_stats_parts(V)) return FFNO_EINVAL;
  const int al = g32::aligned(in, w1, w2, pre) && (!mode || g32::aligned(prev_pre, prev_coefs, xout));
  cudaStream_t s = (cudaStream_t)stream;
  const int cpg = C / groups;
  switch (C) {
#define L(CC)                                                                                          \
  case CC: {                                                                                           \
    const size_t smem = mlp2_smem<CC>();                                                               \
    const int grid = grid_for(V, tile_ctas(CC));                                                       \
    if (mode == 0) {                                                                                   \
      if (!set_smem(k_mlp2<CC, 0>, smem)) return FFNO_ELAUNCH;                                         \
      ffno::launch(k_mlp2<CC, 0>, grid, NT, smem, s, in, prev_pre, prev_coefs, res, xout, V, w1, w2, dw, pre,    \
                                            partials, nparts, cpg, groups, al);                       \
    } else if (mode == 1) {                                                                            \
      if (!set_smem(k_mlp2<CC, 1>, smem)) return FFNO_ELAUNCH;                                         \
      ffno::launch(k_mlp2<CC, 1>, grid, NT, smem, s, in, prev_pre, prev_coefs, res, xout, V, w1, w2, dw, pre,    \
                                            partials, nparts, cpg, groups, al);                       \
    } else {                                                                                           \
      if (!set_smem(k_mlp2<CC, 2>, smem)) return FFNO_ELAUNCH;                                         \
      ffno::launch(k_mlp2<CC, 2>, grid, NT, smem, s, in, prev_pre, prev_coefs, res, xout, V, w1, w2, dw, pre,    \
                                            partials, nparts, cpg, groups, al);                       \
    }                                                                                                  \
    break;                                                                                             \
  }
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_fuse_fwd(const float* x, const float* spec_pre, const float* spec_coefs, const float* vert_pre,
                  const float* vert_coefs, long V, int C, const float* wg1, const float* wg2, const float* bg2,
                  const float* wf1, const float* wf2, const float* dw, float* pre, double* partials, int nparts,
                  int groups, ffno_stream_t stream) {
  if (!x || !spec_pre || !spec_coefs || !vert_pre || !vert_coefs || !wg1 || !wg2 || !bg2 || !wf1 || !wf2 || !dw ||
      !pre || !partials)
    return FFNO_EINVAL;
  if (!width_ok(C) || V < 1 || groups < 1 || groups > GMAX || C % groups) return FFNO_EINVAL;
  if (nparts != ffno_stats_parts(V)) return FFNO_EINVAL;
  const int al = g32::aligned(x, spec_pre, spec_coefs, vert_pre, vert_coefs, wg1, wg2, wf1, wf2, pre);
  cudaStream_t s = (cudaStream_t)stream;
  const int cpg = C / groups;
  switch (C) {
#define L(CC)                                                                                                \
  case CC: {                                                                                                 \
    const size_t smem = fuse_smem<CC>();                                                                     \
    const int grid = grid_for(V, tile_ctas(CC));                                                             \
    if (!set_smem(k_fuse<CC>, smem)) return FFNO_ELAUNCH;                                                    \
    ffno::launch(k_fuse<CC>, grid, NT, smem, s, x, spec_pre, spec_coefs, vert_pre, vert_coefs, V, wg1, wg2, bg2, wf1,   \
                                      wf2, dw, pre, partials, nparts, cpg, groups, al);                      \
    break;                                                                                                   \
  }
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_head_fwd(const float* x, const float* x_in, long V, int C, const float* p1, const float* p2, const float* b2,
                  int nh, int nhp, const ffno_head_params* params, float* out, float* head_out,
                  ffno_stream_t stream) {
  if (!x || !x_in || !p1 || !p2 || !b2 || !out) return FFNO_EINVAL;
  if (!width_ok(C) || V < 1 || !params || (nhp != 16 && nhp != 32) || nh > nhp) return FFNO_EINVAL;
  if (params->nspecies < 1 || params->nspecies > FFNO_MAX_SPECIES) return FFNO_EINVAL;
  int tot = 0;
  for (int s = 0; s < params->nspecies; ++s) tot += params->levels[s] + 1;
  if (tot != nh) return FFNO_EINVAL;
  const int al = g32::aligned(x, p1, p2);
  cudaStream_t s = (cudaStream_t)stream;
  switch (C) {
#define L(CC, NN)                                                                                       \
  if (C == CC && nhp == NN) {                                                                           \
    const size_t smem = (2 * CC * BM + BM * (NN + 1) + 2 * g32::KC * 2 * CC) * sizeof(float);            \
    if (params->math32) {                                                                               \
      if (!set_smem(k_head<CC, NN, float>, smem)) return FFNO_ELAUNCH;                                  \
      ffno::launch(k_head<CC, NN, float>, grid_for(V, 2), NT, smem, s, x, x_in, V, p1, p2, b2, nh, *params, out, head_out, al); \
    } else {                                                                                            \
      if (!set_smem(k_head<CC, NN, double>, smem)) return FFNO_ELAUNCH;                                 \
      ffno::launch(k_head<CC, NN, double>, grid_for(V, 2), NT, smem, s, x, x_in, V, p1, p2, b2, nh, *params, out, head_out, al); \
    }                                                                                                   \
  }
    default:
      L(16, 16) L(16, 32) L(32, 16) L(32, 32) L(64, 16) L(64, 32) L(96, 16) L(96, 32)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_proj_fwd(const float* x, long V, int C, const float* p1, const float* p2, const float* b2, int nh, int nhp,
                  float* head, ffno_stream_t stream) {
  if (!x || !p1 || !p2 || !b2 || !head) return FFNO_EINVAL;
  if (!width_ok(C) || V < 1 || (nhp != 16 && nhp != 32) || nh < 1 || nh > nhp) return FFNO_EINVAL;
  const int al = g32::aligned(x, p1, p2);
  cudaStream_t s = (cudaStream_t)stream;
  ffno_head_params none{};
  switch (C) {
#define L(CC, NN)                                                                                       \
  if (C == CC && nhp == NN) {                                                                           \
    const size_t smem = (2 * CC * BM + BM * (NN + 1) + 2 * g32::KC * 2 * CC) * sizeof(float);            \
    if (!set_smem(k_head<CC, NN, float, false>, smem)) return FFNO_ELAUNCH;                             \
    ffno::launch(k_head<CC, NN, float, false>, grid_for(V, 2), NT, smem, s, x, nullptr, V, p1, p2, b2, nh, none,  \
                                                                  nullptr, head, al);                       \
  }
    default:
      L(16, 16) L(16, 32) L(32, 16) L(32, 32) L(64, 16) L(64, 32) L(96, 16) L(96, 32)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_head_output(const float* head, const float* x_in, long V, int nh, const ffno_head_params* params,
                     float* out, ffno_stream_t stream) {
  if (!head || !x_in || !out || !params) return FFNO_EINVAL;
  if (V < 1 || params->nspecies < 1 || params->nspecies > FFNO_MAX_SPECIES || params->in_channels > 8)
    return FFNO_EINVAL;
  int tot = 0, lv = 0;
  for (int s = 0; s < params->nspecies; ++s) {
    if (params->levels[s] < 1) return FFNO_EINVAL;
    tot += params->levels[s] + 1;
    lv += params->levels[s];
  }
  if (tot != nh || lv > FFNO_MAX_LEVELS) return FFNO_EINVAL;
  cudaStream_t s = (cudaStream_t)stream;
  const long want = (V + 255) / 256, cap = 8L * num_sms();   // 8 CTAs of 256 threads per SM, grid-stride
  const long blocks = want < cap ? want : cap;
  if (params->math32)
    ffno::launch(k_head_output<float>, (unsigned)blocks, 256, 0, s, head, x_in, V, nh, *params, out);
  else
    ffno::launch(k_head_output<double>, (unsigned)blocks, 256, 0, s, head, x_in, V, nh, *params, out);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

}  // extern "C"
