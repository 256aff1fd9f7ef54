// FP32 kernels of the FFNO3D input VJP (the hand-written replacement of torch.autograd through FFNO3D.forward,
// models/ffno_model.py:536-553, 730-798). Every chain kernel recomputes its tile's forward activations from the
// block's saved inputs instead of storing them.
#include <math.h>

#include <mutex>

#include "common.cuh"
#include "gemm_f32.cuh"
#include "tc.cuh"

using namespace ffno;

namespace {

__host__ __device__ __forceinline__ long ntiles(long V, int rows) { return (V + rows - 1) / rows; }

int g_sms = 0;
int sms() {
  if (!g_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_sms <= 0) g_sms = 152;
  }
  return g_sms;
}

int grid_of(long V, int rows, int per_sm) {
  const long t = ntiles(V, rows);
  const long g = (long)sms() * per_sm;
  return (int)(t < g ? (t > 0 ? t : 1) : g);
}

template <typename K>
bool smem_attr(K kernel, size_t bytes) {
  return ffno::smem_cap_ok(kernel, bytes);
}

bool width_ok(int C) { return C == 16 || C == 32 || C == 64 || C == 96; }

__device__ __forceinline__ float upstream(int mode, float u, float r, float y) {
  // gradient w.r.t. the GroupNorm output y given the upstream u: r u (mode 0), r u gelu'(y) (mode 1: GELU after GN,
  // erf-based), or r u gelu'(y) with the tensor-core kernels' activation (mode 2: the split-BF16 path, whose forward
  // applies that GELU after these GroupNorms)
  if (mode == 2) return r * u * gelu_grad_tc(y);
  return mode ? r * u * gelu_grad(y) : r * u;
}

// ------------------------------------------------------------------------------------------------ GN backward
// Lane layout of the two GroupNorm-backward kernels: each voxel's C channels are held VW at a time by LPV consecutive
// lanes (C = 96: VW = 4 and 24 lanes of a warp); a warp covers VPW voxels per step. The application uses VW = 8 (one
// 32-byte request a lane) for C <= 64; the statistics keep VW = 4, whose per-slot double accumulators would
// otherwise take more registers than two CTAs of an SM have.
template <int C, int W>
struct GnLanes {
  static constexpr int VW = C <= 64 ? W : 4;
  static constexpr int LPV = C / VW;
  static constexpr int VPW = LPV <= 32 ? 32 / LPV : 1;
};

template <int VW>
__device__ __forceinline__ void ldv(const float* p, float (&o)[VW]) {
  if constexpr (VW == 8) {
    ffno::tc::ld8(p, o);
  } else {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p));
    o[0] = a.x, o[1] = a.y, o[2] = a.z, o[3] = a.w;
  }
}
template <int VW>
__device__ __forceinline__ void stv(float* p, const float (&v)[VW]) {
  if constexpr (VW == 8) {
    ffno::tc::st8(p, v);
  } else {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
}

// Per-group constants of one GroupNorm, as floats in shared memory: mean, rstd, 1/T, S1, S2, var*rstd^2.
struct GnConst {
  float mean[GMAX], rstd[GMAX], invT[GMAX], s1[GMAX], s2[GMAX], vr2[GMAX];
};

__device__ __forceinline__ void load_gn_const(GnConst& k, const double* gst, const double* sums, int groups,
                                              float eps) {
  if (threadIdx.x < groups) {
    const int g = threadIdx.x;
    const double rs = gst[3 * g + 1];
    k.mean[g] = (float)gst[3 * g];
    k.rstd[g] = (float)rs;
    k.invT[g] = (float)(1.0 / gst[3 * g + 2]);
    k.s1[g] = sums ? (float)sums[2 * g] : 0.f;
    k.s2[g] = sums ? (float)sums[2 * g + 1] : 0.f;
    k.vr2[g] = (float)(1.0 - (double)eps * rs * rs);
  }
  __syncthreads();
}

// Per group: S1 = sum ghat, S2 = sum ghat xhat, ghat = dL/dy * gamma, xhat = (pre - mean) rstd, as per-CTA partials.
template <int C>
__global__ void __launch_bounds__(256) k_gn_bwd_stats(int mode, const float* __restrict__ u, float r,
                                                      const float* __restrict__ pre, const float* __restrict__ gamma,
                                                      const float* __restrict__ beta,
                                                      const double* __restrict__ gst, long V,
                                                      double* __restrict__ partials, int nparts, int cpg, int groups) {
  griddep_sync();
  using Ln = GnLanes<C, 4>;
  __shared__ GnConst k;
  load_gn_const(k, gst, nullptr, groups, 0.f);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane / Ln::LPV, q = lane % Ln::LPV;
  const bool active = sub < Ln::VPW;
  constexpr int VW = Ln::VW;
  const int c = VW * q;
  float gm[VW], bt[VW];
  int grp[VW];
#pragma unroll
  for (int j = 0; j < VW; ++j) {
    gm[j] = active ? __ldg(gamma + c + j) : 0.f;
    bt[j] = active ? __ldg(beta + c + j) : 0.f;
    grp[j] = (c + j) / cpg;
  }
  double d1[VW], d2[VW];   // per element slot (groups of slot j fixed per thread)
  float f1[VW], f2[VW];
#pragma unroll
  for (int j = 0; j < VW; ++j) d1[j] = d2[j] = 0.0, f1[j] = f2[j] = 0.f;
  const long step = (long)gridDim.x * 8 * Ln::VPW;
  // UN voxels a thread are loaded before any is used (128 bytes in flight); float partials go to double every 4
  // rounds
  constexpr int UN = 16 / VW;
  int n = 0;
  for (long v0 = ((long)blockIdx.x * 8 + warp) * Ln::VPW + sub; active && v0 < V; v0 += UN * step) {
    float pu[UN][VW], pp[UN][VW];
#pragma unroll
    for (int e = 0; e < UN; ++e) {
      const long v = v0 + e * step;
      if (v < V) {
        ldv<VW>(u + v * C + c, pu[e]);
        ldv<VW>(pre + v * C + c, pp[e]);
      } else {
#pragma unroll
        for (int j = 0; j < VW; ++j) pu[e][j] = pp[e][j] = 0.f;
      }
    }
#pragma unroll
    for (int e = 0; e < UN; ++e) {
      if (v0 + e * step >= V) break;
#pragma unroll
      for (int j = 0; j < VW; ++j) {
        const int g = grp[j];
        const float xh = (pp[e][j] - k.mean[g]) * k.rstd[g];
        const float gh = upstream(mode, pu[e][j], r, xh * gm[j] + bt[j]) * gm[j];
        f1[j] += gh;
        f2[j] += gh * xh;
      }
    }
    if (++n == 16 / UN) {
#pragma unroll
      for (int j = 0; j < VW; ++j) {
        d1[j] += f1[j];
        d2[j] += f2[j];
        f1[j] = f2[j] = 0.f;
      }
      n = 0;
    }
  }
#pragma unroll
  for (int j = 0; j < VW; ++j) {
    d1[j] += f1[j];
    d2[j] += f2[j];
  }
  stats_partial_rows<C, VW>(d1, d2, active, q, cpg, groups, nparts, partials);
}

// upstream() of two channels: (r u) * act'(y), the activation known at compile time
template <int MODE>
__device__ __forceinline__ uint64_t upstream2(float u0, float u1, float r, uint64_t y) {
  float a0 = r * u0, a1 = r * u1, y0, y1;
  upk2(y, y0, y1);
  if constexpr (MODE == 1) a0 *= gelu_grad(y0), a1 *= gelu_grad(y1);
  if constexpr (MODE == 2) mul_gelu_grad_tc2(y0, y1, a0, a1);
  return pk2(a0, a1);
}

// Lanes of the eight-group kernels: a lane's VW channels lie in NG groups of CPG channels (every CPG is even, so a pair
// of channels never straddles two), whose constants stay in registers.
template <int C>
struct Gn8 : GnLanes<C, 8> {
  static constexpr int VW = GnLanes<C, 8>::VW, CPG = C / GMAX, NG = VW > CPG ? VW / CPG : 1;
  static_assert(C % GMAX == 0 && CPG % 2 == 0 && (VW % CPG == 0 || CPG % VW == 0), "groups");
};

// The statistics for eight groups: a lane reads 32 bytes of a row and tensor per request (16 at C = 96) and keeps packed
// partials per group, with the activation fixed at compile time. Bound by instruction issue more than by HBM: two
// channels an instruction and no branch on the mode inside the loop. Mean of a VJP's calls: 2.4 M voxels, C = 64 (1.2 GB):
// 216 -> 206 us; 1.0 M, C = 96 (0.8 GB): 205 -> 178 us.
// Same partials layout and fixed reduction order as k_gn_bwd_stats.
template <int C, int MODE>
__global__ void __launch_bounds__(256, 2) k_gn_bwd_stats8(const float* __restrict__ u, float r,
                                                       const float* __restrict__ pre, const float* __restrict__ gamma,
                                                       const float* __restrict__ beta,
                                                       const double* __restrict__ gst, long V,
                                                       double* __restrict__ partials, int nparts) {
  griddep_sync();
  using Ln = Gn8<C>;
  constexpr int VW = Ln::VW, CPG = Ln::CPG, NG = Ln::NG;
  constexpr bool POW2 = (Ln::LPV & (Ln::LPV - 1)) == 0;
  __shared__ GnConst k;
  __shared__ double red[8][POW2 ? GMAX : 32][2];
  load_gn_const(k, gst, nullptr, GMAX, 0.f);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane / Ln::LPV, q = lane % Ln::LPV;
  const bool active = sub < Ln::VPW;   // C = 96: 24 lanes of a warp
  const int c = VW * q, g0 = c / CPG;
  uint64_t gm[VW / 2], bt[VW / 2], nmean[NG], rstd[NG];
#pragma unroll
  for (int j = 0; j < VW / 2; ++j) {
    gm[j] = active ? pk2(__ldg(gamma + c + 2 * j), __ldg(gamma + c + 2 * j + 1)) : 0;
    bt[j] = active ? pk2(__ldg(beta + c + 2 * j), __ldg(beta + c + 2 * j + 1)) : 0;
  }
#pragma unroll
  for (int l = 0; l < NG; ++l) {
    nmean[l] = pk2(-k.mean[g0 + l], -k.mean[g0 + l]);
    rstd[l] = pk2(k.rstd[g0 + l], k.rstd[g0 + l]);
  }
  const uint64_t one = pk2(1.f, 1.f);
  double d1[NG], d2[NG];
  uint64_t f1[NG], f2[NG];
#pragma unroll
  for (int l = 0; l < NG; ++l) d1[l] = d2[l] = 0.0, f1[l] = f2[l] = 0;
  auto fold = [&] {
#pragma unroll
    for (int l = 0; l < NG; ++l) {
      float a, b;
      upk2(f1[l], a, b);
      d1[l] += a + b;
      upk2(f2[l], a, b);
      d2[l] += a + b;
      f1[l] = f2[l] = 0;
    }
  };
  const long step = (long)gridDim.x * 8 * Ln::VPW;
  constexpr int UN = 16 / VW;   // voxels a thread loaded before any is used: 128 bytes in flight
  int n = 0;
  for (long v0 = ((long)blockIdx.x * 8 + warp) * Ln::VPW + sub; active && v0 < V; v0 += UN * step) {
    float pu[UN][VW], pp[UN][VW];
#pragma unroll
    for (int e = 0; e < UN; ++e) {
      const long v = v0 + e * step;
      if (v < V) {
        ldv<VW>(u + v * C + c, pu[e]);
        ldv<VW>(pre + v * C + c, pp[e]);
      } else {
#pragma unroll
        for (int j = 0; j < VW; ++j) pu[e][j] = pp[e][j] = 0.f;
      }
    }
#pragma unroll
    for (int e = 0; e < UN; ++e) {
      if (v0 + e * step >= V) break;
#pragma unroll
      for (int j = 0; j < VW / 2; ++j) {
        const int l = NG == 1 ? 0 : 2 * j / CPG;
        const uint64_t xh = mul2(fma2(pk2(pp[e][2 * j], pp[e][2 * j + 1]), one, nmean[l]), rstd[l]);
        const uint64_t gh = mul2(upstream2<MODE>(pu[e][2 * j], pu[e][2 * j + 1], r, fma2(xh, gm[j], bt[j])), gm[j]);
        f1[l] = fma2(gh, one, f1[l]);
        f2[l] = fma2(gh, xh, f2[l]);
      }
    }
    if (++n == 16 / UN) {   // float partials go to double every 16 voxels, as in k_gn_bwd_stats
      fold();
      n = 0;
    }
  }
  fold();
  // sum over the lanes of a group in a warp, then over the warps, in a fixed order
  if constexpr (POW2) {
#pragma unroll
    for (int l = 0; l < NG; ++l) {
#pragma unroll
      for (int o = 16; o >= Ln::LPV; o >>= 1) {
        d1[l] += __shfl_xor_sync(0xffffffffu, d1[l], o);
        d2[l] += __shfl_xor_sync(0xffffffffu, d2[l], o);
      }
      if (sub == 0) {
        red[warp][g0 + l][0] = d1[l];
        red[warp][g0 + l][1] = d2[l];
      }
    }
  } else {
    red[warp][lane][0] = d1[0];
    red[warp][lane][1] = d2[0];
  }
  __syncthreads();
  if (threadIdx.x < 2 * GMAX) {
    const int g = threadIdx.x >> 1, i = threadIdx.x & 1;
    double a = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      if constexpr (POW2) {
        a += red[w][g][i];
      } else {
#pragma unroll
        for (int m = 0; m < CPG / VW; ++m) a += red[w][g * (CPG / VW) + m][i];
      }
    }
    partials[((long)blockIdx.x * GMAX + g) * 2 + i] = a;
    for (long p = blockIdx.x + gridDim.x; p < nparts; p += gridDim.x) partials[(p * GMAX + g) * 2 + i] = 0.0;
  }
}

__global__ void k_gn_bwd_final(const double* __restrict__ partials, int nparts, int groups, double* __restrict__ sums) {
  griddep_sync();
  // one warp per group: strided partial sums per lane, then a fixed shuffle tree (deterministic)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int g = warp; g < groups; g += nw) {
    double s1 = 0.0, s2 = 0.0;
    for (int p = lane; p < nparts; p += 32) {
      s1 += partials[((long)p * groups + g) * 2];
      s2 += partials[((long)p * groups + g) * 2 + 1];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      s1 += __shfl_down_sync(0xffffffffu, s1, off);
      s2 += __shfl_down_sync(0xffffffffu, s2, off);
    }
    if (lane == 0) {
      sums[2 * g] = s1;
      sums[2 * g + 1] = s2;
    }
  }
}

// pre_bar = rstd (ghat - (w / T)(S1 + xhat S2)); w_bar[v] += sum_c (1/T)(-S1 xhat - S2 (xhat^2 - var rstd^2) / 2).
template <int C>
__global__ void __launch_bounds__(256, 4) k_gn_bwd_apply(int mode, const float* __restrict__ u, float r,
                                                      const float* __restrict__ pre, const float* __restrict__ gamma,
                                                      const float* __restrict__ beta,
                                                      const double* __restrict__ gst, const double* __restrict__ sums,
                                                      const float* __restrict__ dw, long V,
                                                      float* __restrict__ pre_bar, float* __restrict__ w_bar, int cpg,
                                                      int groups, float eps) {
  griddep_sync();
  using Ln = GnLanes<C, 8>;
  __shared__ GnConst k;
  load_gn_const(k, gst, sums, groups, eps);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane / Ln::LPV, q = lane % Ln::LPV;
  const bool active = sub < Ln::VPW;
  constexpr int VW = Ln::VW;
  const int c = VW * q;
  float gm[VW], bt[VW];
  int grp[VW];
#pragma unroll
  for (int j = 0; j < VW; ++j) {
    gm[j] = active ? __ldg(gamma + c + j) : 0.f;
    bt[j] = active ? __ldg(beta + c + j) : 0.f;
    grp[j] = (c + j) / cpg;
  }
  const long step = (long)gridDim.x * 8 * Ln::VPW;
  const long first = ((long)blockIdx.x * 8 + warp) * Ln::VPW;
  for (long vb = first; vb < V; vb += step) {   // warp-uniform loop
    const long v = vb + sub;
    const bool ok = active && v < V;
    float wc = 0.f;
    if (ok) {
      const float wv = __ldg(dw + v);
      float uu[VW], xx[VW], o[VW];
      ldv<VW>(u + v * C + c, uu);
      ldv<VW>(pre + v * C + c, xx);
#pragma unroll
      for (int j = 0; j < VW; ++j) {
        const int g = grp[j];
        const float xh = (xx[j] - k.mean[g]) * k.rstd[g];
        const float gh = upstream(mode, uu[j], r, xh * gm[j] + bt[j]) * gm[j];
        o[j] = k.rstd[g] * (gh - wv * k.invT[g] * (k.s1[g] + xh * k.s2[g]));
        wc += k.invT[g] * (-k.s1[g] * xh - 0.5f * k.s2[g] * (xh * xh - k.vr2[g]));
      }
      stv<VW>(pre_bar + v * C + c, o);
    }
    // sum over the LPV lanes of this voxel (segments of a power-of-two LPV, or the whole warp for C = 96)
    if (Ln::LPV >= 32 || (Ln::LPV & (Ln::LPV - 1))) {
#pragma unroll
      for (int off = 16; off; off >>= 1) wc += __shfl_xor_sync(0xffffffffu, wc, off);
    } else {
#pragma unroll
      for (int off = Ln::LPV / 2; off; off >>= 1) wc += __shfl_xor_sync(0xffffffffu, wc, off);
    }
    if (ok && q == 0) w_bar[v] += wc;
  }
}

// The same for eight groups: the lane's group constants in registers (the general kernel reads six of them from shared
// memory for every channel) and two channels an instruction. Mean of a VJP's calls: 2.4 M voxels, C = 64 (1.8 GB): 325 ->
// 309 us; 1.0 M, C = 96 (1.2 GB): 340 -> 319 us.
template <int C, int MODE>
__global__ void __launch_bounds__(256, C <= 32 ? 3 : 4) k_gn_bwd_apply8(const float* __restrict__ u, float r,
                                                          const float* __restrict__ pre,
                                                          const float* __restrict__ gamma,
                                                          const float* __restrict__ beta,
                                                          const double* __restrict__ gst,
                                                          const double* __restrict__ sums,
                                                          const float* __restrict__ dw, long V,
                                                          float* __restrict__ pre_bar, float* __restrict__ w_bar,
                                                          float eps) {
  griddep_sync();
  using Ln = Gn8<C>;
  constexpr int VW = Ln::VW, CPG = Ln::CPG, NG = Ln::NG;
  __shared__ GnConst k;
  load_gn_const(k, gst, sums, GMAX, eps);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane / Ln::LPV, q = lane % Ln::LPV;
  const bool active = sub < Ln::VPW;
  const int c = VW * q, g0 = active ? c / CPG : 0;
  uint64_t gm[VW / 2], bt[VW / 2];
  float nmean[NG], rstd[NG], p1[NG], p2[NG], nvr2[NG];   // p = (1/T) (S1, S2)
#pragma unroll
  for (int j = 0; j < VW / 2; ++j) {
    gm[j] = active ? pk2(__ldg(gamma + c + 2 * j), __ldg(gamma + c + 2 * j + 1)) : 0;
    bt[j] = active ? pk2(__ldg(beta + c + 2 * j), __ldg(beta + c + 2 * j + 1)) : 0;
  }
#pragma unroll
  for (int l = 0; l < NG; ++l) {
    const int g = g0 + l;
    nmean[l] = -k.mean[g];
    rstd[l] = k.rstd[g];
    p1[l] = k.invT[g] * k.s1[g];
    p2[l] = k.invT[g] * k.s2[g];
    nvr2[l] = -k.vr2[g];
  }
  auto both = [](float x) { return pk2(x, x); };
  const long step = (long)gridDim.x * 8 * Ln::VPW;
  for (long vb = ((long)blockIdx.x * 8 + warp) * Ln::VPW; vb < V; vb += step) {   // warp-uniform loop
    const long v = vb + sub;
    const bool ok = active && v < V;
    float wc = 0.f;
    if (ok) {
      const float wv = __ldg(dw + v);
      float uu[VW], xx[VW], o[VW];
      ldv<VW>(u + v * C + c, uu);
      ldv<VW>(pre + v * C + c, xx);
      uint64_t w2 = 0;
#pragma unroll
      for (int j = 0; j < VW / 2; ++j) {
        const int l = NG == 1 ? 0 : 2 * j / CPG;
        const uint64_t xh = mul2(fma2(pk2(xx[2 * j], xx[2 * j + 1]), both(1.f), both(nmean[l])), both(rstd[l]));
        const uint64_t gh = mul2(upstream2<MODE>(uu[2 * j], uu[2 * j + 1], r, fma2(xh, gm[j], bt[j])), gm[j]);
        const uint64_t t = fma2(xh, both(p2[l]), both(p1[l]));
        upk2(mul2(both(rstd[l]), fma2(both(-wv), t, gh)), o[2 * j], o[2 * j + 1]);
        w2 = fma2(both(-p1[l]), xh, w2);
        w2 = fma2(both(-0.5f * p2[l]), fma2(xh, xh, both(nvr2[l])), w2);
      }
      upk2(w2, wc, uu[0]);
      wc += uu[0];
      stv<VW>(pre_bar + v * C + c, o);
    }
    // sum over the LPV lanes of this voxel (segments of a power-of-two LPV, or the whole warp for C = 96)
#pragma unroll
    for (int off = (Ln::LPV & (Ln::LPV - 1)) ? 16 : Ln::LPV / 2; off; off >>= 1)
      wc += __shfl_xor_sync(0xffffffffu, wc, off);
    if (ok && q == 0) w_bar[v] += wc;
  }
}

// ------------------------------------------------------------------------------------------------ MLP backward
// pre = gelu(a W1) W2; given pre_bar: a_bar = base + ((pre_bar W2^T) * gelu'(a W1)) W1^T. The hidden gradient overwrites
// the two input tiles (2C channels). 524 k voxels, C = 64: 1.21 -> 0.70 ms (37 TFLOP/s).
template <int C>
__global__ void __launch_bounds__(NT, 2) k_mlp2_bwd(const float* __restrict__ a, const float* __restrict__ pb,
                                                    const float* __restrict__ base, long V,
                                                    const float* __restrict__ w1, const float* __restrict__ w2t,
                                                    const float* __restrict__ w1t, float* __restrict__ abar, int al) {
  griddep_sync();
  extern __shared__ __align__(16) float sm[];
  float* as = sm;   // [C][64] a, [C][64] pre_bar, then [2C][64] the hidden gradient
  g32::Ring ring(as + 2 * C * BM, g32::KC * 2 * C, al);
  using Ch = g32::Cols<2 * C, 1>;
  const int tx = g32::tile_tx();
  const long nt = ntiles(V, BM);
  for (long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long v0 = t * BM;
    __syncthreads();
    ring.pre<2 * C>(w1, 2 * C);
    g32::load_tile<C>(as, 0, a, v0, V, al);
    g32::load_tile<C>(as, C, pb, v0, V, al);
    {
      float hp[2 * C / 16][4], gb[2 * C / 16][4];
      g32::gemm<C, 2 * C>(as, 0, w1, 2 * C, ring, hp);
      ring.pre<2 * C>(w2t, 2 * C);
#pragma unroll
      for (int j = 0; j < 2 * C / 16; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) hp[j][e] = gelu_grad(hp[j][e]);
      g32::gemm<C, 2 * C>(as, C, w2t, 2 * C, ring, gb);
      ring.pre<C>(w1t, C);
      __syncthreads();   // every read of the input tiles is done
#pragma unroll
      for (int j = 0; j < 2 * C / 16; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) gb[j][e] *= hp[j][e];
        g32::put4(as, Ch::col(tx, j), gb[j]);
      }
    }
    float acc[C / 16][4];
    g32::gemm<2 * C, C>(as, 0, w1t, C, ring, acc);
    g32::store_rows<C>(abar, base, v0, V, acc, al);
  }
}

// ------------------------------------------------------------------------------------------------ fuse backward
// Recomputes the gate/fuse chain of the tile and back-propagates fused_pre_bar (= pb) to x, spec and vert
// (FFNOBlock3dBalanced._fuse_branches, models/ffno_model.py:524-534). Three regions: X [C] holds x, then the gate hidden
// layer, pb, the gate hidden gradient; SV [2C] holds spec | vert, then their gated gradients; T [2C] holds each GEMM's
// operand in between. 80 KB and the 16 KB ring at C = 64: two CTAs an SM. 524 k voxels, C = 64: 5.51 -> 2.34 ms.
template <int C>
constexpr size_t fuse_bwd_smem() {
  return (5 * C * BM + 2 * g32::KC * 2 * C) * sizeof(float);
}

template <int C>
__global__ void __launch_bounds__(NT, C <= 64 ? 2 : 1) k_fuse_bwd(
    const float* __restrict__ x, const float* __restrict__ sp, const float* __restrict__ sc,
    const float* __restrict__ vp, const float* __restrict__ vc, const float* __restrict__ pb,
    const float* __restrict__ base, long V, const float* __restrict__ wg1, const float* __restrict__ wg2,
    const float* __restrict__ bg2, const float* __restrict__ wf1, const float* __restrict__ wf2t,
    const float* __restrict__ wf1t, const float* __restrict__ wg2t, const float* __restrict__ wg1t,
    float* __restrict__ xbar, float* __restrict__ sbar, float* __restrict__ vbar, int al) {
  griddep_sync();
  extern __shared__ __align__(16) float sm[];
  float* X = sm;                 // channels 0 .. C - 1 of the region [x | spec | vert]
  float* T = X + 3 * C * BM;
  g32::Ring ring(T + 2 * C * BM, g32::KC * 2 * C, al);
  constexpr int N1 = C / 16, N2 = 2 * C / 16;
  using C1 = g32::Cols<C, 1>;
  using C2 = g32::Cols<2 * C, 2>;   // the thread owns channel c of both branches
  using Ch = g32::Cols<2 * C, 1>;
  const int tx = g32::tile_tx();
  const long nt = ntiles(V, BM);
  for (long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long v0 = t * BM;
    __syncthreads();
    ring.pre<C>(wg1, C);
    g32::each_quad<C>(v0, V, [&](int r, int c, long o, bool ok) {
      const float4 ps = g32::ldq(sp + o, ok, al), pv = g32::ldq(vp + o, ok, al);
      const float as[4] = {ps.x, ps.y, ps.z, ps.w}, av[4] = {pv.x, pv.y, pv.z, pv.w};
      g32::put_quad(X, r, c, g32::ldq(x + o, ok, al));
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        X[g32::at(r, C + c + i)] =
            ok ? gelu((as[i] - __ldg(sc + c + i)) * __ldg(sc + C + c + i) + __ldg(sc + 2 * C + c + i)) : 0.f;
        X[g32::at(r, 2 * C + c + i)] =
            ok ? gelu((av[i] - __ldg(vc + c + i)) * __ldg(vc + C + c + i) + __ldg(vc + 2 * C + c + i)) : 0.f;
      }
    });
    // 1. branch-gate hidden layer: its gelu' stays in registers, its gelu replaces x
    float h1[N1][4];
    g32::gemm<3 * C, C>(X, 0, wg1, C, ring, h1);
    ring.pre<2 * C>(wg2, 2 * C);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < N1; ++j) {
      float h[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        h[e] = gelu(h1[j][e]);
        h1[j][e] = gelu_grad(h1[j][e]);
      }
      g32::put4(X, C1::col(tx, j), h);
    }
    // 2. gates (registers) and the mixed branches [spec g_s, vert g_v] -> T
    float g[N2][4];
    g32::gemm<C, 2 * C, 2>(X, 0, wg2, 2 * C, ring, g);
    ring.pre<2 * C>(wf1, 2 * C);
#pragma unroll
    for (int j = 0; j < N2; ++j) {
      const int n = C2::col(tx, j);
      const float b = __ldg(bg2 + n);
      float a[4];
      g32::get4(X, C + n, a);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        g[j][e] = sigmoid(g[j][e] + b);
        a[e] *= g[j][e];
      }
      g32::put4(T, n, a);
    }
    // 3. fuse hidden pre-activation (registers, as gelu'); pb into X
    float hf[N2][4];
    g32::gemm<2 * C, 2 * C>(T, 0, wf1, 2 * C, ring, hf);
    ring.pre<2 * C>(wf2t, 2 * C);
    g32::load_tile<C>(X, 0, pb, v0, V, al);   // the gate GEMM's reads of X ended before the last GEMM's barriers
#pragma unroll
    for (int j = 0; j < N2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) hf[j][e] = gelu_grad(hf[j][e]);
    // 4. fuse hidden gradient -> T
    {
      float acc[N2][4];
      g32::gemm<C, 2 * C>(X, 0, wf2t, 2 * C, ring, acc);
      ring.pre<2 * C>(wf1t, 2 * C);
#pragma unroll
      for (int j = 0; j < N2; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] *= hf[j][e];
        g32::put4(T, Ch::col(tx, j), acc[j]);   // T's readers (step 3) passed this GEMM's barriers
      }
    }
    // 5. B_bar = T Wf1^T + 0.5 [pb, pb]: the branch gradients replace spec | vert, the gate pre-activation gradient -> T
    {
      float acc[N2][4];
      g32::gemm<2 * C, 2 * C, 2>(T, 0, wf1t, 2 * C, ring, acc);
      ring.pre<C>(wg2t, C);
      __syncthreads();
#pragma unroll
      for (int j = 0; j < N2; ++j) {
        const int n = C2::col(tx, j);
        float a[4], f[4], d[4];
        g32::get4(X, C + n, a);
        g32::get4(X, C2::col(tx, j % N1), f);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float bb = acc[j][e] + 0.5f * f[e];
          d[e] = bb * a[e] * g[j][e] * (1.f - g[j][e]);
          a[e] = bb * g[j][e];
        }
        g32::put4(X, C + n, a);
        g32::put4(T, n, d);
      }
    }
    // 6. branch-gate hidden gradient -> X
    {
      float acc[N1][4];
      g32::gemm<2 * C, C>(T, 0, wg2t, C, ring, acc);
      ring.pre<C>(wg1t, 3 * C);
#pragma unroll
      for (int j = 0; j < N1; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] *= h1[j][e];
        g32::put4(X, C1::col(tx, j), acc[j]);   // pb's readers (step 5) passed this GEMM's barriers
      }
    }
    // 7. A_bar = X Wg1^T: x, spec, vert gradients
#pragma unroll 1
    for (int part = 0; part < 3; ++part) {
      float acc[N1][4];
      g32::gemm<C, C>(X, 0, wg1t + part * C, 3 * C, ring, acc);
      if (part < 2) ring.pre<C>(wg1t + (part + 1) * C, 3 * C);
      if (part) {
#pragma unroll
        for (int j = 0; j < N1; ++j) {
          float b[4];
          g32::get4(X, part * C + C1::col(tx, j), b);
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[j][e] += b[e];
        }
      }
      g32::store_rows<C>(part == 0 ? xbar : part == 1 ? sbar : vbar, part == 0 ? base : nullptr, v0, V, acc, al);
    }
  }
}

// ------------------------------------------------------------------------------------------------ gate backward
// x_bar = base + sum over the two branches of d/dx [x * sigmoid(gelu(x G1) G2)] applied to that branch's gradient;
// z_bar += sum_c xv_bar * zp (the z_proj term of the vertical branch, models/ffno_model.py:265). 524 k voxels, C = 64:
// 2.86 -> 1.02 ms.
template <int C>
__global__ void __launch_bounds__(NT, 3) k_gate_bwd(const float* __restrict__ x, const float* __restrict__ xsb,
                                                 const float* __restrict__ xvb, const float* __restrict__ base,
                                                 long V, const float* __restrict__ s1, const float* __restrict__ s2,
                                                 const float* __restrict__ s2t, const float* __restrict__ s1t,
                                                 const float* __restrict__ v1, const float* __restrict__ v2,
                                                 const float* __restrict__ v2t, const float* __restrict__ v1t,
                                                 const float* __restrict__ zp, float* __restrict__ xbar,
                                                 float* __restrict__ zbar, int al) {
  griddep_sync();
  extern __shared__ __align__(16) float sm[];
  float* SX = sm;               // [C][64] x
  float* SB = SX + C * BM;      // [C][64] the branch's gradient
  float* ST = SB + C * BM;      // [C][64] GEMM operand
  g32::Ring ring(ST + C * BM, g32::KC * C, al);
  using Cl = g32::Cols<C, 1>;
  constexpr int N = C / 16;
  const int tx = g32::tile_tx();
  const long nt = ntiles(V, BM);
  for (long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long v0 = t * BM;
    float xb[N][4];
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) xb[j][e] = 0.f;
    __syncthreads();
    ring.pre<C>(s1, C);
    g32::load_tile<C>(SX, 0, x, v0, V, al);
#pragma unroll 1
    for (int br = 0; br < 2; ++br) {
      const float* gbar = br ? xvb : xsb;
      const float* g1 = br ? v1 : s1;
      const float* g2 = br ? v2 : s2;
      const float* g2t = br ? v2t : s2t;
      const float* g1t = br ? v1t : s1t;
      g32::load_tile<C>(SB, 0, gbar, v0, V, al);   // its readers of the branch before passed later barriers
      float h[N][4], acc[N][4];
      g32::gemm<C, C>(SX, 0, g1, C, ring, h);
      ring.pre<C>(g2, C);
#pragma unroll
      for (int j = 0; j < N; ++j) {
        float a[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          a[e] = gelu(h[j][e]);
          h[j][e] = gelu_grad(h[j][e]);
        }
        g32::put4(ST, Cl::col(tx, j), a);   // ST's readers (the branch before) passed the last GEMM's barriers
      }
      g32::gemm<C, C>(ST, 0, g2, C, ring, acc);
      ring.pre<C>(g2t, C);
      __syncthreads();
#pragma unroll
      for (int j = 0; j < N; ++j) {
        float b[4], xv[4], d[4];
        g32::get4(SB, Cl::col(tx, j), b);
        g32::get4(SX, Cl::col(tx, j), xv);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float g = sigmoid(acc[j][e]);
          xb[j][e] += b[e] * g;
          d[e] = b[e] * xv[e] * g * (1.f - g);
        }
        g32::put4(ST, Cl::col(tx, j), d);
      }
      g32::gemm<C, C>(ST, 0, g2t, C, ring, acc);
      ring.pre<C>(g1t, C);
      __syncthreads();
#pragma unroll
      for (int j = 0; j < N; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] *= h[j][e];
        g32::put4(ST, Cl::col(tx, j), acc[j]);
      }
      g32::gemm<C, C>(ST, 0, g1t, C, ring, acc);
      if (br == 0) ring.pre<C>(v1, C);
#pragma unroll
      for (int j = 0; j < N; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) xb[j][e] += acc[j][e];
      if (br == 1 && zp) {
        // z_bar[v] += sum_c xv_bar[v][c] zp[c]: 4 lanes a voxel
        const int r = threadIdx.x >> 2, q = threadIdx.x & 3;
        float a = 0.f;
        for (int c = q; c < C; c += 4) a = fmaf(SB[g32::at(r, c)], __ldg(zp + c), a);
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        a += __shfl_xor_sync(0xffffffffu, a, 2);
        if (q == 0 && v0 + r < V) zbar[v0 + r] += a;
      }
    }
    g32::store_rows<C>(xbar, base, v0, V, xb, al);
  }
}

// ------------------------------------------------------------------------------------------------ lift backward
// x_in_bar[k][v] += sum_c pre_bar[v][c] w_lift[k][c]. The grid fills the SMs (seven or eight CTAs of 17-25 KB each): with
// half of that, CTAs placed early piled up on half of the SMs (2.4 M voxels, C = 64: 588 us; full: 300).
template <int C>
__global__ void __launch_bounds__(NT) k_lift_bwd(const float* __restrict__ pb, int cin, long V,
                                                 const float* __restrict__ wl, float* __restrict__ xib) {
  griddep_sync();
  __shared__ float ps[BM][C + 1];
  const long nt = ntiles(V, BM);
  for (long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long v0 = t * BM;
    __syncthreads();
    load_rows<C>(&ps[0][0], C + 1, pb, v0, V);
    __syncthreads();
    for (int e = threadIdx.x; e < cin * BM; e += NT) {
      const int k = e / BM, r = e % BM;
      const long v = v0 + r;
      if (v >= V) continue;
      float s = 0.f;
      for (int c = 0; c < C; ++c) s = fmaf(ps[r][c], __ldg(wl + k * C + c), s);
      xib[(long)k * V + v] += s;
    }
  }
}

// ------------------------------------------------------------------------------------------------ head backward

// kLte = false: the VJP of FFNO3D._run_head alone (models/ffno_model.py:790-798); ybar is then the gradient of the
// nh head channels [nh][V] and xin / xinbar are not used.
template <int C, int NHP, typename T, bool kLte = true>
__global__ void __launch_bounds__(NT, 2) k_head_bwd(const float* __restrict__ x, const float* __restrict__ xin,
                                                 const float* __restrict__ ybar, long V, const float* __restrict__ p1,
                                                 const float* __restrict__ p2, const float* __restrict__ b2,
                                                 const float* __restrict__ p2t, const float* __restrict__ p1t,
                                                 const __grid_constant__ HeadParams hp, int nh,
                                                 float* __restrict__ xbar, float* __restrict__ xinbar, int al) {
  griddep_sync();
  extern __shared__ __align__(16) float sm[];
  __shared__ double etab[EXP_TAB];
  constexpr int LO = NHP + 1, N2 = 2 * C / 16;
  if (kLte) fill_exp_table(etab);
  float* SA = sm;                    // [C][64] input, then [2C][64] hidden, then its gradient
  float* SG = SA + 2 * C * BM;       // [NHP][64] gradient of the head channels
  float* SO = SG + NHP * BM;         // [64][NHP + 1] head channels, then their gradient
  g32::Ring ring(SO + BM * LO, g32::KC * 2 * C, al);
  using Ch = g32::Cols<2 * C, 1>;
  using Co = g32::Cols<NHP, 1>;
  const int tx = g32::tile_tx(), ty = g32::tile_ty();
  const long nt = ntiles(V, BM);
  for (long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long v0 = t * BM;
    __syncthreads();
    ring.pre<2 * C>(p1, 2 * C);
    g32::load_tile<C>(SA, 0, x, v0, V, al);
    float h[N2][4];   // gelu' of the hidden pre-activation
    g32::gemm<C, 2 * C>(SA, 0, p1, 2 * C, ring, h);
    ring.pre<NHP>(p2, NHP);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < N2; ++j) {
      float a[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        a[e] = gelu(h[j][e]);
        h[j][e] = gelu_grad(h[j][e]);
      }
      g32::put4(SA, Ch::col(tx, j), a);
    }
    {
      float acc[NHP / 16][4];
      g32::gemm<2 * C, NHP>(SA, 0, p2, NHP, ring, acc);
      ring.pre<2 * C>(p2t, 2 * C);
#pragma unroll
      for (int j = 0; j < NHP / 16; ++j) {
        const int n = Co::col(tx, j);
        const float b = __ldg(b2 + n);
#pragma unroll
        for (int e = 0; e < 4; ++e) SO[(4 * ty + e) * LO + n] = acc[j][e] + b;
      }
    }
    __syncthreads();
    if (threadIdx.x < BM) {
      const int r = threadIdx.x;
      const long v = v0 + r;
      float* o = SO + r * LO;
      if (v < V) {
        if constexpr (kLte) {
          head_voxel_bwd<T>(hp, o, NHP, head_inputs(hp, xin, V, v), ybar, V, v, xinbar, etab);
        } else {
          for (int c = 0; c < NHP; ++c) o[c] = c < nh ? __ldg(ybar + (long)c * V + v) : 0.f;
        }
      }
      for (int c = 0; c < NHP; ++c) SG[g32::at(r, c)] = v < V ? o[c] : 0.f;
    }
    {
      float acc[N2][4];
      g32::gemm<NHP, 2 * C>(SG, 0, p2t, 2 * C, ring, acc);
      ring.pre<C>(p1t, C);
#pragma unroll
      for (int j = 0; j < N2; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] *= h[j][e];
        g32::put4(SA, Ch::col(tx, j), acc[j]);   // the hidden layer's readers passed later barriers
      }
    }
    {
      float acc[C / 16][4];
      g32::gemm<2 * C, C>(SA, 0, p1t, C, ring, acc);
      g32::store_rows<C>(xbar, nullptr, v0, V, acc, al);
    }
  }
}

// VJP of FFNO3D.head_output on precomputed head channels: one thread per voxel; head_bar [nh][V] and x_in_bar
// [cin][V] are written (the T, ne and rho channels carry the LTE and total terms, the others are zero).
template <typename T>
__global__ void __launch_bounds__(256) k_head_output_bwd(const float* __restrict__ head, const float* __restrict__ xin,
                                                         const float* __restrict__ ybar, long V, int nh,
                                                         const __grid_constant__ HeadParams hp,
                                                         float* __restrict__ hbar, float* __restrict__ xinbar) {
  griddep_sync();
  __shared__ double etab[EXP_TAB];
  fill_exp_table(etab);
  __syncthreads();
  float o[FFNO_MAX_LEVELS + FFNO_MAX_SPECIES];
  for (long v = blockIdx.x * (long)blockDim.x + threadIdx.x; v < V; v += (long)gridDim.x * blockDim.x) {
    for (int c = 0; c < nh; ++c) o[c] = __ldg(head + (long)c * V + v);
    head_voxel_bwd<T>(hp, o, nh, head_inputs(hp, xin, V, v), ybar, V, v, xinbar, etab);
    for (int c = 0; c < nh; ++c) hbar[(long)c * V + v] = o[c];
  }
}

// ------------------------------------------------------------------------------------------------ depth weights
// w = t / max(mean_d t, 1e-12), t_d = |z_{d+1} - z_d| / 2 + |z_d - z_{d-1}| / 2 (models/ffno_model.py:28-34, 67-74)
// A CTA holds DB_COLS neighbouring columns, DB_SEGS threads share each column's levels; the two column sums are fixed-order
// sums of the segments' sums, then every level's gradient is independent. One thread a column left each level waiting
// for memory (four walks). 101 x 45 x 75: 93 -> 9 us.
constexpr int DB_COLS = 32, DB_SEGS = 16;

__global__ void __launch_bounds__(DB_COLS* DB_SEGS) k_depth_weights_bwd(const float* __restrict__ z,
                                                                        const float* __restrict__ wb, int D, long HW,
                                                                        float* __restrict__ zb) {
  griddep_sync();
  __shared__ float part[2][DB_SEGS][DB_COLS];
  const int tx = threadIdx.x % DB_COLS, sg = threadIdx.x / DB_COLS;
  const long col = (long)blockIdx.x * DB_COLS + tx;
  const bool ok = col < HW;
  if (D == 1) return;
  auto Z = [&](int d) { return __ldg(z + (long)d * HW + col); };
  auto T = [&](int d) {
    float t = 0.f;
    if (d + 1 < D) t += 0.5f * fabsf(Z(d + 1) - Z(d));
    if (d > 0) t += 0.5f * fabsf(Z(d) - Z(d - 1));
    return t;
  };
  float sum = 0.f, corr = 0.f;
  if (ok) {
#pragma unroll 2
    for (int d = sg; d < D; d += DB_SEGS) {
      const float t = T(d);
      sum += t;
      corr += __ldg(wb + (long)d * HW + col) * t;
    }
  }
  part[0][sg][tx] = sum;
  part[1][sg][tx] = corr;
  __syncthreads();
  if (!ok) return;
  sum = corr = 0.f;
#pragma unroll
  for (int i = 0; i < DB_SEGS; ++i) {
    sum += part[0][i][tx];
    corr += part[1][i][tx];
  }
  const float mraw = sum / (float)D;
  const bool clamped = mraw < 1e-12f;
  const float m = clamped ? 1e-12f : mraw;
  // d/dt_d: wb_d / m - [m not clamped] (sum_j wb_j t_j / m^2) / D
  corr = clamped ? 0.f : corr / (m * m * (float)D);
  // segment s_d = z_{d+1} - z_d feeds t_d and t_{d+1} with weight sign(s_d) / 2
  auto seg = [&](int d) {
    const float s = Z(d + 1) - Z(d);
    const float sgn = (s > 0.f) ? 1.f : ((s < 0.f) ? -1.f : 0.f);
    const float tb0 = __ldg(wb + (long)d * HW + col) / m - corr;
    const float tb1 = __ldg(wb + (long)(d + 1) * HW + col) / m - corr;
    return 0.5f * sgn * (tb0 + tb1);
  };
#pragma unroll 2
  for (int d = sg; d < D; d += DB_SEGS) {
    float g = zb[(long)d * HW + col];
    if (d > 0) g += seg(d - 1);
    if (d + 1 < D) g -= seg(d);
    zb[(long)d * HW + col] = g;
  }
}

// ------------------------------------------------------------------------------------------------ A B^T split-K
// part[split][i][j] = sum_{n in split's range} A[i][n] B[j][n]; CTA tile 64 x 64.
__global__ void __launch_bounds__(NT) k_outer(const float* __restrict__ A, long lda, int Ma,
                                              const float* __restrict__ B, long ldb, int Mb, long N, long chunk,
                                              int ti, int tj, float* __restrict__ part) {
  griddep_sync();
  // 64 x 64 output tile, k in chunks of 64 read as float4 (16 threads per row: 256 contiguous bytes)
  __shared__ float as[64][65];
  __shared__ float bs[64][65];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  long bid = blockIdx.x;
  const int bi = (int)(bid % ti);
  bid /= ti;
  const int bj = (int)(bid % tj);
  const long split = bid / tj;
  const long n0 = split * chunk;
  const long n1 = (n0 + chunk < N) ? n0 + chunk : N;
  float acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.f;
  for (long k0 = n0; k0 < n1; k0 += 64) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = threadIdx.x + u * NT;
      const int r = e >> 4, c = (e & 15) * 4;
      const long n = k0 + c;
      const int i = bi * 64 + r, j = bj * 64 + r;
      float4 va = make_float4(0.f, 0.f, 0.f, 0.f), vb = va;
      if (n + 3 < n1) {
        if (i < Ma) va = __ldg(reinterpret_cast<const float4*>(A + (long)i * lda + n));
        if (j < Mb) vb = __ldg(reinterpret_cast<const float4*>(B + (long)j * ldb + n));
      } else {
        float ta[4] = {0.f, 0.f, 0.f, 0.f}, tb[4] = {0.f, 0.f, 0.f, 0.f};
        for (int q = 0; q < 4; ++q)
          if (n + q < n1) {
            if (i < Ma) ta[q] = __ldg(A + (long)i * lda + n + q);
            if (j < Mb) tb[q] = __ldg(B + (long)j * ldb + n + q);
          }
        va = make_float4(ta[0], ta[1], ta[2], ta[3]);
        vb = make_float4(tb[0], tb[1], tb[2], tb[3]);
      }
      as[r][c] = va.x;
      as[r][c + 1] = va.y;
      as[r][c + 2] = va.z;
      as[r][c + 3] = va.w;
      bs[r][c] = vb.x;
      bs[r][c + 1] = vb.y;
      bs[r][c + 2] = vb.z;
      bs[r][c + 3] = vb.w;
    }
    __syncthreads();
#pragma unroll 16
    for (int k = 0; k < 64; ++k) {
      float a[4], b[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        a[q] = as[ty + 16 * q][k];
        b[q] = bs[tx + 16 * q][k];
      }
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[p][q] = fmaf(a[p], b[q], acc[p][q]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int i = bi * 64 + ty + 16 * p;
    if (i >= Ma) continue;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int j = bj * 64 + tx + 16 * q;
      if (j < Mb) part[(split * Ma + i) * (long)Mb + j] = acc[p][q];
    }
  }
}

// Sum of the splits' partial products in FP64, OR_SEGS threads an element (each every OR_SEGS-th split), in a fixed order:
// one thread an element walked up to 304 splits, each a load's latency. 8448 elements, 304 splits: 40 -> 11.6 us.
constexpr int OR_EL = 32, OR_SEGS = 8;

__global__ void __launch_bounds__(OR_EL* OR_SEGS) k_outer_reduce(const float* __restrict__ part, long nsplit, long n,
                                                                 double* __restrict__ out, int accumulate) {
  griddep_sync();
  __shared__ double red[OR_SEGS][OR_EL];
  const int tx = threadIdx.x % OR_EL, sg = threadIdx.x / OR_EL;
  const long e = (long)blockIdx.x * OR_EL + tx;
  double s = 0.0;
  if (e < n) {
#pragma unroll 4
    for (long p = sg; p < nsplit; p += OR_SEGS) s += (double)__ldg(part + p * n + e);
  }
  red[sg][tx] = s;
  __syncthreads();
  if (sg || e >= n) return;
#pragma unroll
  for (int i = 1; i < OR_SEGS; ++i) s += red[i][tx];
  out[e] = accumulate ? out[e] + s : s;
}

}  // namespace

// ====================================================================================================== C ABI
extern "C" {

int ffno_gn_bwd_stats(int mode, const float* u, float r, const float* pre, const float* gamma, const float* beta,
                      const double* gstats, long V, int C, int groups, double* partials, int nparts,
                      ffno_stream_t stream) {
  if (!u || !pre || !gamma || !beta || !gstats || !partials) return FFNO_EINVAL;
  if (mode < 0 || mode > 2) return FFNO_EINVAL;
  if (!width_ok(C) || V < 1 || groups < 1 || groups > GMAX || C % groups || nparts < 1) return FFNO_EINVAL;
  cudaStream_t s = (cudaStream_t)stream;
  const int cpg = C / groups;
  const bool early = ffno::early_launch(V, C);
  const int grid = nparts < 2 * sms() ? nparts : 2 * sms();   // the CTAs an SM holds (97-124 registers a thread)
  // eight groups (the model's): 32-byte lanes for C <= 64, 16-byte lanes for C = 96; anything else takes the general
  // kernel, whose loads need 16 bytes
  if (groups == GMAX && (reinterpret_cast<uintptr_t>(u) | reinterpret_cast<uintptr_t>(pre)) % (C <= 64 ? 32 : 16) == 0) {
    switch (4 * C + mode) {
#define L1(CC, M) \
  case 4 * CC + M: ffno::launch_if(early, k_gn_bwd_stats8<CC, M>, grid, 256, 0, s, u, r, pre, gamma, beta, gstats, V, partials, nparts); break;
#define L(CC) L1(CC, 0) L1(CC, 1) L1(CC, 2)
      L(16) L(32) L(64) L(96)
#undef L
#undef L1
    }
    FFNO_CHECK_LAUNCH();
    return FFNO_OK;
  }
  switch (C) {
#define L(CC) case CC: ffno::launch(k_gn_bwd_stats<CC>, grid, 256, 0, s, mode, u, r, pre, gamma, beta, gstats, V, partials, nparts, cpg, groups); break;
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_gn_bwd_final(const double* partials, int nparts, int groups, double* sums, ffno_stream_t stream) {
  if (!partials || !sums || nparts < 1 || groups < 1 || groups > GMAX) return FFNO_EINVAL;
  ffno::launch(k_gn_bwd_final, 1, 512, 0, (cudaStream_t)stream, partials, nparts, groups, sums);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_gn_bwd_apply(int mode, const float* u, float r, const float* pre, const float* gamma, const float* beta,
                      const double* gstats, const double* sums, const float* dw, long V, int C, int groups, float eps,
                      float* pre_bar, float* w_bar, ffno_stream_t stream) {
  if (!u || !pre || !gamma || !beta || !gstats || !dw || !pre_bar || !w_bar) return FFNO_EINVAL;
  if (mode < 0 || mode > 2) return FFNO_EINVAL;
  if (!width_ok(C) || V < 1 || groups < 1 || groups > GMAX || C % groups) return FFNO_EINVAL;
  // a lane moves 32 bytes of a row per request for C <= 64, 16 bytes for C = 96
  const uintptr_t al = C <= 64 ? 32 : 16;
  if ((reinterpret_cast<uintptr_t>(u) | reinterpret_cast<uintptr_t>(pre) | reinterpret_cast<uintptr_t>(pre_bar)) % al)
    return FFNO_EINVAL;
  cudaStream_t s = (cudaStream_t)stream;
  const int cpg = C / groups;
  if (groups == GMAX) {
    const bool early = ffno::early_launch(V, C);
    const int blocks = grid_of(V, 8 * 8, C <= 32 ? 3 : 4);   // the CTAs an SM holds
    switch (4 * C + mode) {
#define L1(CC, M)                                                                                                  \
  case 4 * CC + M:                                                                                                 \
    ffno::launch_if(early, k_gn_bwd_apply8<CC, M>, blocks, 256, 0, s, u, r, pre, gamma, beta, gstats, sums, dw, V, pre_bar, w_bar, \
                 eps);                                                                                             \
    break;
#define L(CC) L1(CC, 0) L1(CC, 1) L1(CC, 2)
      L(16) L(32) L(64) L(96)
#undef L
#undef L1
    }
    FFNO_CHECK_LAUNCH();
    return FFNO_OK;
  }
  const int blocks = grid_of(V, 8 * 8, 4);
  switch (C) {
#define L(CC) case CC: ffno::launch(k_gn_bwd_apply<CC>, blocks, 256, 0, s, mode, u, r, pre, gamma, beta, gstats, sums, dw, V, pre_bar, w_bar, cpg, groups, eps); break;
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_mlp2_bwd(const float* a, const float* pre_bar, const float* base, long V, int C, const float* w1,
                  const float* w2t, const float* w1t, float* a_bar, ffno_stream_t stream) {
  if (!a || !pre_bar || !w1 || !w2t || !w1t || !a_bar || !width_ok(C) || V < 1) return FFNO_EINVAL;
  const int al = g32::aligned(a, pre_bar, base, w1, w2t, w1t, a_bar);
  cudaStream_t s = (cudaStream_t)stream;
  switch (C) {
#define L(CC)                                                                                   \
  case CC: {                                                                                    \
    const size_t smem = (2 * CC * BM + 2 * g32::KC * 2 * CC) * sizeof(float);                   \
    if (!smem_attr(k_mlp2_bwd<CC>, smem)) return FFNO_ELAUNCH;                                  \
    ffno::launch(k_mlp2_bwd<CC>, grid_of(V, BM, 2), NT, smem, s, a, pre_bar, base, V, w1, w2t, w1t, a_bar, al); \
    break;                                                                                      \
  }
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_fuse_bwd(const float* x, const float* spec_pre, const float* spec_coefs, const float* vert_pre,
                  const float* vert_coefs, const float* fused_pre_bar, const float* base, long V, int C,
                  const float* wg1, const float* wg2, const float* bg2, const float* wf1, const float* wf2t,
                  const float* wf1t, const float* wg2t, const float* wg1t, float* x_bar, float* spec_bar,
                  float* vert_bar, ffno_stream_t stream) {
  if (!x || !spec_pre || !spec_coefs || !vert_pre || !vert_coefs || !fused_pre_bar || !wg1 || !wg2 || !bg2 || !wf1 ||
      !wf2t || !wf1t || !wg2t || !wg1t || !x_bar || !spec_bar || !vert_bar)
    return FFNO_EINVAL;
  if (!width_ok(C) || V < 1) return FFNO_EINVAL;
  const int al = g32::aligned(x, spec_pre, vert_pre, fused_pre_bar, base, wg1, wg2, wf1, wf2t, wf1t, wg2t, wg1t, x_bar,
                              spec_bar, vert_bar);
  cudaStream_t s = (cudaStream_t)stream;
  switch (C) {
#define L(CC)                                                                                               \
  case CC: {                                                                                                \
    const size_t smem = fuse_bwd_smem<CC>();                                                                \
    if (!smem_attr(k_fuse_bwd<CC>, smem)) return FFNO_ELAUNCH;                                              \
    ffno::launch(k_fuse_bwd<CC>, grid_of(V, BM, CC <= 64 ? 2 : 1), NT, smem, s, x, spec_pre, spec_coefs, vert_pre,     \
                                                                      vert_coefs, fused_pre_bar, base, V,   \
                                                                      wg1, wg2, bg2, wf1, wf2t, wf1t, wg2t, \
                                                                      wg1t, x_bar, spec_bar, vert_bar, al); \
    break;                                                                                                  \
  }
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_gate_bwd(const float* x, const float* xs_bar, const float* xv_bar, const float* base, long V, int C,
                  const float* s_w1, const float* s_w2, const float* s_w2t, const float* s_w1t, const float* v_w1,
                  const float* v_w2, const float* v_w2t, const float* v_w1t, const float* zp, float* x_bar,
                  float* z_bar, ffno_stream_t stream) {
  if (!x || !xs_bar || !xv_bar || !s_w1 || !s_w2 || !s_w2t || !s_w1t || !v_w1 || !v_w2 || !v_w2t || !v_w1t || !x_bar)
    return FFNO_EINVAL;
  if (!width_ok(C) || V < 1 || (zp && !z_bar)) return FFNO_EINVAL;
  const int al = g32::aligned(x, xs_bar, xv_bar, base, s_w1, s_w2, s_w2t, s_w1t, v_w1, v_w2, v_w2t, v_w1t, x_bar);
  cudaStream_t s = (cudaStream_t)stream;
  switch (C) {
#define L(CC)                                                                                              \
  case CC: {                                                                                               \
    const size_t smem = (3 * CC * BM + 2 * g32::KC * CC) * sizeof(float);                                  \
    if (!smem_attr(k_gate_bwd<CC>, smem)) return FFNO_ELAUNCH;                                             \
    ffno::launch(k_gate_bwd<CC>, grid_of(V, BM, 3), NT, smem, s, x, xs_bar, xv_bar, base, V, s_w1, s_w2, s_w2t, s_w1t, \
                                                       v_w1, v_w2, v_w2t, v_w1t, zp, x_bar, z_bar, al);     \
    break;                                                                                                 \
  }
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_lift_bwd(const float* pre_bar, int cin, long V, int C, const float* w_lift, float* x_in_bar,
                  ffno_stream_t stream) {
  if (!pre_bar || !w_lift || !x_in_bar || !width_ok(C) || V < 1 || cin < 1 || cin > 8) return FFNO_EINVAL;
  cudaStream_t s = (cudaStream_t)stream;
  switch (C) {
#define L(CC) case CC: ffno::launch(k_lift_bwd<CC>, grid_of(V, BM, CC <= 64 ? 8 : 7), NT, 0, s, pre_bar, cin, V, w_lift, x_in_bar); break;
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_head_bwd(const float* x, const float* x_in, const float* y_bar, long V, int C, const float* p1,
                  const float* p2, const float* b2, const float* p2t, const float* p1t, int nhp,
                  const ffno_head_params* params, float* x_bar, float* x_in_bar, ffno_stream_t stream) {
  if (!x || !x_in || !y_bar || !p1 || !p2 || !b2 || !p2t || !p1t || !x_bar || !x_in_bar) return FFNO_EINVAL;
  if (!width_ok(C) || V < 1 || !params || (nhp != 16 && nhp != 32)) return FFNO_EINVAL;
  if (params->nspecies < 1 || params->nspecies > FFNO_MAX_SPECIES || params->in_channels > 8) return FFNO_EINVAL;
  const int al = g32::aligned(x, p1, p2, p2t, p1t, x_bar);
  cudaStream_t s = (cudaStream_t)stream;
  switch (C) {
#define L(CC, NN)                                                                                        \
  if (C == CC && nhp == NN) {                                                                            \
    const size_t smem = (2 * CC * BM + NN * BM + BM * (NN + 1) + 2 * g32::KC * 2 * CC) * sizeof(float);  \
    if (params->math32) {                                                                               \
      if (!smem_attr(k_head_bwd<CC, NN, float>, smem)) return FFNO_ELAUNCH;                             \
      ffno::launch(k_head_bwd<CC, NN, float>, grid_of(V, BM, 2), NT, smem, s, x, x_in, y_bar, V, p1, p2, b2, p2t, p1t, \
                                                                    *params, NN, x_bar, x_in_bar, al);      \
    } else {                                                                                            \
      if (!smem_attr(k_head_bwd<CC, NN, double>, smem)) return FFNO_ELAUNCH;                            \
      ffno::launch(k_head_bwd<CC, NN, double>, grid_of(V, BM, 2), NT, smem, s, x, x_in, y_bar, V, p1, p2, b2, p2t, p1t, \
                                                                     *params, NN, x_bar, x_in_bar, al);     \
    }                                                                                                   \
  }
    default:
      L(16, 16) L(16, 32) L(32, 16) L(32, 32) L(64, 16) L(64, 32) L(96, 16) L(96, 32)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_depth_weights_bwd(const float* z, const float* w_bar, int D, long HW, float* z_bar, ffno_stream_t stream) {
  if (!z || !w_bar || !z_bar || D < 1 || HW < 1) return FFNO_EINVAL;
  ffno::launch(k_depth_weights_bwd, (unsigned)((HW + DB_COLS - 1) / DB_COLS), DB_COLS * DB_SEGS, 0, (cudaStream_t)stream, 
      z, w_bar, D, HW, z_bar);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_outer_parts(int Ma, int Mb, long N) {
  const long tiles = (long)((Ma + 63) / 64) * ((Mb + 63) / 64);
  long nsplit = (4L * sms() + tiles - 1) / tiles;
  const long maxs = (N + 1023) / 1024;
  if (nsplit > maxs) nsplit = maxs;
  if (nsplit < 1) nsplit = 1;
  return (int)nsplit;
}

int ffno_outer(const float* A, long lda, int Ma, const float* B, long ldb, int Mb, long N, float* part, int nsplit,
               double* out, int accumulate, ffno_stream_t stream) {
  if (!A || !B || !part || !out || Ma < 1 || Mb < 1 || N < 1 || nsplit < 1) return FFNO_EINVAL;
  const int ti = (Ma + 63) / 64, tj = (Mb + 63) / 64;
  if (lda % 4 || ldb % 4 || (reinterpret_cast<uintptr_t>(A) % 16) || (reinterpret_cast<uintptr_t>(B) % 16))
    return FFNO_EINVAL;   // float4 loads
  long chunk = (N + nsplit - 1) / nsplit;
  chunk = (chunk + 63) / 64 * 64;
  cudaStream_t s = (cudaStream_t)stream;
  ffno::launch(k_outer, (unsigned)((long)ti * tj * nsplit), NT, 0, s, A, lda, Ma, B, ldb, Mb, N, chunk, ti, tj, part);
  const long n = (long)Ma * Mb;
  ffno::launch_if(false, k_outer_reduce, (unsigned)((n + OR_EL - 1) / OR_EL), OR_EL * OR_SEGS, 0, s, part, nsplit, n, out, accumulate);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

// ---------------------------------------------------------------------------------------------- no-allocation variant
// ffno_outer_noalloc: the same product as ffno_outer for hosts that cannot hand this library a scratch buffer on every
// call. A process that binds the C ABI from its own runtime (a Julia, Go or Java host whose device memory belongs to
// that runtime's own pool allocator, or a service that must not grow its footprint after start-up) often has no way to
// call cudaMalloc for us, and the split-K partial sums need somewhere to live. They live here instead: a fixed array in
// the library's own device memory, present on every GPU that loads the library until the process exits.
}  // extern "C"

namespace {

constexpr long kOuterScratchFloats = 4L << 20;  // 16 MiB: Ma * Mb * nsplit partial sums at most
__device__ __align__(256) float g_outer_scratch[kOuterScratchFloats];

std::mutex g_outer_scratch_mutex;
float* g_outer_scratch_ptr[256] = {};  // device address of g_outer_scratch per device ordinal, set on first use

}  // namespace

extern "C" {

int ffno_outer_noalloc(const float* A, long lda, int Ma, const float* B, long ldb, int Mb, long N, double* out,
                       int accumulate, ffno_stream_t stream) {
  if (!A || !B || !out || Ma < 1 || Mb < 1 || N < 1) return FFNO_EINVAL;
  const long n = (long)Ma * Mb;
  if (n > kOuterScratchFloats) return FFNO_ETOOBIG;
  if (lda % 4 || ldb % 4 || (reinterpret_cast<uintptr_t>(A) % 16) || (reinterpret_cast<uintptr_t>(B) % 16))
    return FFNO_EINVAL;   // k_outer reads float4
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) return FFNO_EINVAL;
  float* scratch = nullptr;
  {
    // The host-side name g_outer_scratch is not a device address: ask the runtime for it once per device, with that
    // device current.
    std::lock_guard<std::mutex> lock(g_outer_scratch_mutex);
    if (!g_outer_scratch_ptr[dev]) {
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_outer_scratch) != cudaSuccess || !p) return FFNO_ELAUNCH;
      g_outer_scratch_ptr[dev] = static_cast<float*>(p);
    }
    scratch = g_outer_scratch_ptr[dev];
  }
  long nsplit = ffno_outer_parts(Ma, Mb, N);
  if (nsplit > kOuterScratchFloats / n) nsplit = kOuterScratchFloats / n;
  const int ti = (Ma + 63) / 64, tj = (Mb + 63) / 64;
  long chunk = (N + nsplit - 1) / nsplit;
  chunk = (chunk + 63) / 64 * 64;
  cudaStream_t s = (cudaStream_t)stream;
  // every partial sum the reduction reads is written first by k_outer: nothing in the scratch has to start at zero
  ffno::launch(k_outer, (unsigned)((long)ti * tj * nsplit), NT, 0, s, A, lda, Ma, B, ldb, Mb, N, chunk, ti, tj, scratch);
  ffno::launch_if(false, k_outer_reduce, (unsigned)((n + OR_EL - 1) / OR_EL), OR_EL * OR_SEGS, 0, s, scratch, nsplit, n, out, accumulate);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_proj_bwd(const float* x, const float* head_bar, long V, int C, const float* p1, const float* p2,
                  const float* b2, const float* p2t, const float* p1t, int nh, int nhp, float* x_bar,
                  ffno_stream_t stream) {
  if (!x || !head_bar || !p1 || !p2 || !b2 || !p2t || !p1t || !x_bar) return FFNO_EINVAL;
  if (!width_ok(C) || V < 1 || (nhp != 16 && nhp != 32) || nh < 1 || nh > nhp) return FFNO_EINVAL;
  const int al = g32::aligned(x, p1, p2, p2t, p1t, x_bar);
  cudaStream_t s = (cudaStream_t)stream;
  ffno_head_params none{};
  switch (C) {
#define L(CC, NN)                                                                                        \
  if (C == CC && nhp == NN) {                                                                            \
    const size_t smem = (2 * CC * BM + NN * BM + BM * (NN + 1) + 2 * g32::KC * 2 * CC) * sizeof(float);  \
    if (!smem_attr(k_head_bwd<CC, NN, float, false>, smem)) return FFNO_ELAUNCH;                         \
    ffno::launch(k_head_bwd<CC, NN, float, false>, grid_of(V, BM, 2), NT, smem, s, x, nullptr, head_bar, V, p1, p2, b2, \
                                                                         p2t, p1t, none, nh, x_bar, nullptr, al); \
  }
    default:
      L(16, 16) L(16, 32) L(32, 16) L(32, 32) L(64, 16) L(64, 32) L(96, 16) L(96, 32)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_head_output_bwd(const float* head, const float* x_in, const float* y_bar, long V, int nh,
                         const ffno_head_params* params, float* head_bar, float* x_in_bar, ffno_stream_t stream) {
  if (!head || !x_in || !y_bar || !params || !head_bar || !x_in_bar) return FFNO_EINVAL;
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
  const long want = (V + 255) / 256, cap = 8L * sms();   // 8 CTAs of 256 threads per SM, grid-stride
  const long blocks = want < cap ? want : cap;
  if (params->math32)
    ffno::launch(k_head_output_bwd<float>, (unsigned)blocks, 256, 0, s, head, x_in, y_bar, V, nh, *params, head_bar, x_in_bar);
  else
    ffno::launch(k_head_output_bwd<double>, (unsigned)blocks, 256, 0, s, head, x_in, y_bar, V, nh, *params, head_bar,
                                                               x_in_bar);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

}  // extern "C"
