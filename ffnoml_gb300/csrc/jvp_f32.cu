// FP32 kernels of the FFNO3D forward-mode derivative (JVP): the tangent of every stage of FFNO3D.forward
// (models/ffno_model.py:524-553, 730-832) along an input tangent, evaluated next to the primal stage it linearises
// (what jvp_local gets from dual tensors carried through the network, ffno_fsdp_runtime.py:350-372). The linear stages
// (the lift convolution, the DFT contractions, the spectral mixing) reuse the forward kernels on the tangent; these are
// the nonlinear ones. The heights are fixed (the depth weights, the height tables and the z_proj term carry no
// tangent).
#include <math.h>

#include "common.cuh"
#include "gemm_f32.cuh"

using namespace ffno;

namespace {

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

int grid_rows(long V, int rows, int per_sm) {
  const long t = (V + rows - 1) / rows;
  const long g = (long)sms() * per_sm;
  return (int)(t < g ? (t > 0 ? t : 1) : g);
}

template <typename K>
bool smem_attr(K kernel, size_t bytes) {
  return ffno::smem_cap_ok(kernel, bytes);
}

bool width_ok(int C) { return C == 16 || C == 32 || C == 64 || C == 96; }

// ------------------------------------------------------------------------------------------------ GroupNorm JVP
// y = gamma (x - mu) r + beta over a group with depth weights w (T = sum of w over the group's elements):
// y' = gamma r (x' - S1 / T - xhat S2 / T), S1 = sum w x', S2 = sum w xhat x' (xhat = (x - mu) r).
// Statistics: per-CTA partial sums [nparts][groups][2] in a fixed order (the layout of ffno_gn_bwd_final).
template <int C>
__global__ void __launch_bounds__(256) k_gn_jvp_stats(const float* __restrict__ pre, const float* __restrict__ ud,
                                                      const double* __restrict__ gst, const float* __restrict__ dw,
                                                      long V, double* __restrict__ partials, int cpg, int groups) {
  griddep_sync();
  constexpr int LPV = C / 4;                       // lanes per voxel (float4 each)
  constexpr int VPW = LPV <= 32 ? 32 / LPV : 1;    // voxels per warp step
  __shared__ float mean[GMAX], rstd[GMAX];
  if (threadIdx.x < groups) {
    mean[threadIdx.x] = (float)gst[3 * threadIdx.x];
    rstd[threadIdx.x] = (float)gst[3 * threadIdx.x + 1];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane / LPV, q = lane % LPV;
  const bool active = sub < VPW;
  const int c = 4 * q;
  int grp[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) grp[j] = (c + j) / cpg;
  double d1[4] = {0, 0, 0, 0}, d2[4] = {0, 0, 0, 0};
  float f1[4] = {0, 0, 0, 0}, f2[4] = {0, 0, 0, 0};
  int n = 0;
  const long step = (long)gridDim.x * 8 * VPW;
  for (long v = ((long)blockIdx.x * 8 + warp) * VPW + sub; active && v < V; v += step) {
    const float w = __ldg(dw + v);
    const float4 pu = __ldg(reinterpret_cast<const float4*>(ud + v * C + c));
    const float4 pp = __ldg(reinterpret_cast<const float4*>(pre + v * C + c));
    const float uu[4] = {pu.x, pu.y, pu.z, pu.w}, xx[4] = {pp.x, pp.y, pp.z, pp.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int g = grp[j];
      const float xh = (xx[j] - mean[g]) * rstd[g];
      f1[j] = fmaf(w, uu[j], f1[j]);
      f2[j] = fmaf(w * xh, uu[j], f2[j]);
    }
    if (++n == 16) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        d1[j] += f1[j];
        d2[j] += f2[j];
        f1[j] = f2[j] = 0.f;
      }
      n = 0;
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    d1[j] += f1[j];
    d2[j] += f2[j];
  }
  stats_partial_rows<C, 4>(d1, d2, active, q, cpg, groups, gridDim.x, partials);
}

// out = base + res * y' (base may be null; act 1: y' times gelu'(y), a GELU after the GroupNorm)
template <int C>
__global__ void k_gn_jvp_apply(const float* __restrict__ pre, const float* __restrict__ ud,
                               const float* __restrict__ gamma, const float* __restrict__ beta,
                               const double* __restrict__ gst, const double* __restrict__ sums, int act,
                               const float* __restrict__ base, float res, long V, float* __restrict__ out, int cpg,
                               int groups) {
  griddep_sync();
  __shared__ float mean[GMAX], rstd[GMAX], s1[GMAX], s2[GMAX];
  if (threadIdx.x < groups) {
    const int g = threadIdx.x;
    const double it = 1.0 / gst[3 * g + 2];
    mean[g] = (float)gst[3 * g];
    rstd[g] = (float)gst[3 * g + 1];
    s1[g] = (float)(sums[2 * g] * it);
    s2[g] = (float)(sums[2 * g + 1] * it);
  }
  __syncthreads();
  const long n4 = V * (C / 4);
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n4; e += (long)gridDim.x * blockDim.x) {
    const long v = e / (C / 4);
    const int c = (int)(e % (C / 4)) * 4;
    const float4 pp = __ldg(reinterpret_cast<const float4*>(pre + v * C + c));
    const float4 pu = __ldg(reinterpret_cast<const float4*>(ud + v * C + c));
    const float xx[4] = {pp.x, pp.y, pp.z, pp.w}, uu[4] = {pu.x, pu.y, pu.z, pu.w};
    float o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int g = (c + j) / cpg;
      const float gm = __ldg(gamma + c + j);
      const float xh = (xx[j] - mean[g]) * rstd[g];
      float yd = gm * rstd[g] * (uu[j] - s1[g] - xh * s2[g]);
      if (act) yd *= gelu_grad(fmaf(gm, xh, __ldg(beta + c + j)));
      o[j] = res * yd;
    }
    if (base) {
      const float4 b4 = __ldg(reinterpret_cast<const float4*>(base + v * C + c));
      o[0] += b4.x;
      o[1] += b4.y;
      o[2] += b4.z;
      o[3] += b4.w;
    }
    *reinterpret_cast<float4*>(out + v * C + c) = make_float4(o[0], o[1], o[2], o[3]);
  }
}

// ------------------------------------------------------------------------------------------------ chains
// Tiles of BM voxels on the tile GEMM of gemm_f32.cuh; the primal and its tangent share each weight chunk (NA = 2).

// Input gate: out = x sigmoid(g), g = gelu(x G1) G2 (+ zp z, constant in x): out' = x' s + x s (1 - s) g',
// g' = (gelu'(x G1) x' G1) G2. 147 k voxels, C = 64: 269 -> 136 us.
template <int C>
__global__ void __launch_bounds__(NT, C <= 64 ? 3 : 2) k_gate_jvp(const float* __restrict__ x, const float* __restrict__ xd, long V,
                                                    const float* __restrict__ w1, const float* __restrict__ w2,
                                                    float* __restrict__ outd, int al) {
  griddep_sync();
  extern __shared__ __align__(16) float sm[];
  float* xs = sm;               // [2C][64]: x, x'
  float* hs = xs + 2 * C * BM;  // [2C][64]: the hidden layer and its tangent
  g32::Ring ring(hs + 2 * C * BM, g32::KC * C, al);
  using Cl = g32::Cols<C, 1>;
  const int tx = g32::tile_tx();
  const long nt = (V + BM - 1) / BM;
  for (long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long v0 = t * BM;
    __syncthreads();
    ring.pre<C>(w1, C);
    g32::load_tile<C>(xs, 0, x, v0, V, al);
    g32::load_tile<C>(xs + C * BM, 0, xd, v0, V, al);
    float a[2][C / 16][4];
    g32::gemm_n<C, C, 1, 2>(xs, C * BM, 0, w1, C, ring, a);
    ring.pre<C>(w2, C);
#pragma unroll
    for (int j = 0; j < C / 16; ++j) {
      const int c = Cl::col(tx, j);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        a[1][j][e] *= gelu_grad(a[0][j][e]);
        a[0][j][e] = gelu(a[0][j][e]);
      }
      g32::put4(hs, c, a[0][j]);
      g32::put4(hs + C * BM, c, a[1][j]);
    }
    g32::gemm_n<C, C, 1, 2>(hs, C * BM, 0, w2, C, ring, a);
#pragma unroll
    for (int j = 0; j < C / 16; ++j) {
      const int c = Cl::col(tx, j);
      float xv[4], xt[4];
      g32::get4(xs, c, xv);
      g32::get4(xs + C * BM, c, xt);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float s = sigmoid(a[0][j][e]);
        a[0][j][e] = xt[e] * s + xv[e] * s * (1.f - s) * a[1][j][e];
      }
    }
    g32::store_rows<C>(outd, nullptr, v0, V, a[0], al);
  }
}

// Two-layer MLP C -> 2C -> C: pre' = (gelu'(a W1) a' W1) W2. 147 k voxels, C = 64: 305 -> 190 us.
template <int C>
__global__ void __launch_bounds__(NT, 2) k_mlp2_jvp(const float* __restrict__ a, const float* __restrict__ ad, long V,
                                                    const float* __restrict__ w1, const float* __restrict__ w2,
                                                    float* __restrict__ outd, int al) {
  griddep_sync();
  extern __shared__ __align__(16) float sm[];
  float* as = sm;   // [C][64] a, [C][64] a', then [2C][64] the hidden tangent
  g32::Ring ring(as + 2 * C * BM, g32::KC * 2 * C, al);
  using Ch = g32::Cols<2 * C, 1>;
  const int tx = g32::tile_tx();
  const long nt = (V + BM - 1) / BM;
  for (long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long v0 = t * BM;
    __syncthreads();
    ring.pre<2 * C>(w1, 2 * C);
    g32::load_tile<C>(as, 0, a, v0, V, al);
    g32::load_tile<C>(as + C * BM, 0, ad, v0, V, al);
    {
      float h[2][2 * C / 16][4];
      g32::gemm_n<C, 2 * C, 1, 2>(as, C * BM, 0, w1, 2 * C, ring, h);
      ring.pre<C>(w2, C);
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 2 * C / 16; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) h[1][j][e] *= gelu_grad(h[0][j][e]);
        g32::put4(as, Ch::col(tx, j), h[1][j]);
      }
    }
    float o[C / 16][4];
    g32::gemm<2 * C, C>(as, 0, w2, C, ring, o);
    g32::store_rows<C>(outd, nullptr, v0, V, o, al);
  }
}

// Gate + fuse (_fuse_branches): A = [x, s, v] with s = gelu(GN(spec_pre)), v likewise (sd, vd: their tangents);
// gates = sigmoid(gelu(A Wg1) Wg2 + b); B = [s gs, v gv]; fused = gelu(B Wf1) Wf2 + (B_s + B_v) / 2 -> fused'. One
// region [A | A'] of 6C channels that each stage overwrites: the gate hidden layer over x, B over [s, v], the fuse hidden
// tangent over B. 147 k voxels, C = 64: 1587 -> 618 us.
template <int C>
constexpr size_t fuse_jvp_smem() {
  return (6 * C * BM + 2 * g32::KC * 2 * C) * sizeof(float);
}

template <int C>
__global__ void __launch_bounds__(NT, C <= 64 ? 2 : 1) k_fuse_jvp(const float* __restrict__ x, const float* __restrict__ xd,
                                                    const float* __restrict__ sp, const float* __restrict__ sc,
                                                    const float* __restrict__ vp, const float* __restrict__ vc,
                                                    const float* __restrict__ sd, const float* __restrict__ vd, long V,
                                                    const float* __restrict__ wg1, const float* __restrict__ wg2,
                                                    const float* __restrict__ bg2, const float* __restrict__ wf1,
                                                    const float* __restrict__ wf2, float* __restrict__ outd, int al) {
  griddep_sync();
  extern __shared__ __align__(16) float sm[];
  constexpr int TAN = 3 * C * BM, N1 = C / 16, N2 = 2 * C / 16;   // TAN: offset of the tangent's region
  float* A = sm;
  float* Ad = sm + TAN;
  g32::Ring ring(sm + 2 * TAN, g32::KC * 2 * C, al);
  using C1 = g32::Cols<C, 1>;
  using C2 = g32::Cols<2 * C, 2>;
  using Ch = g32::Cols<2 * C, 1>;
  const int tx = g32::tile_tx();
  const long nt = (V + BM - 1) / BM;
  for (long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long v0 = t * BM;
    __syncthreads();
    ring.pre<C>(wg1, C);
    g32::each_quad<C>(v0, V, [&](int r, int c, long o, bool ok) {
      const float4 ps = g32::ldq(sp + o, ok, al), pv = g32::ldq(vp + o, ok, al);
      const float as[4] = {ps.x, ps.y, ps.z, ps.w}, av[4] = {pv.x, pv.y, pv.z, pv.w};
      g32::put_quad(A, r, c, g32::ldq(x + o, ok, al));
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        A[g32::at(r, C + c + i)] =
            ok ? gelu((as[i] - __ldg(sc + c + i)) * __ldg(sc + C + c + i) + __ldg(sc + 2 * C + c + i)) : 0.f;
        A[g32::at(r, 2 * C + c + i)] =
            ok ? gelu((av[i] - __ldg(vc + c + i)) * __ldg(vc + C + c + i) + __ldg(vc + 2 * C + c + i)) : 0.f;
      }
      g32::put_quad(Ad, r, c, g32::ldq(xd + o, ok, al));
      g32::put_quad(Ad, r, C + c, g32::ldq(sd + o, ok, al));
      g32::put_quad(Ad, r, 2 * C + c, g32::ldq(vd + o, ok, al));
    });
    {
      float h[2][N1][4];
      g32::gemm_n<3 * C, C, 1, 2>(A, TAN, 0, wg1, C, ring, h);
      ring.pre<2 * C>(wg2, 2 * C);
      __syncthreads();
#pragma unroll
      for (int j = 0; j < N1; ++j) {
        const int c = C1::col(tx, j);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          h[1][j][e] *= gelu_grad(h[0][j][e]);
          h[0][j][e] = gelu(h[0][j][e]);
        }
        g32::put4(A, c, h[0][j]);
        g32::put4(Ad, c, h[1][j]);
      }
    }
    float half[N1][4];
    {
      float q[2][N2][4];
      g32::gemm_n<C, 2 * C, 2, 2>(A, TAN, 0, wg2, 2 * C, ring, q);
      ring.pre<2 * C>(wf1, 2 * C);
#pragma unroll
      for (int j = 0; j < N2; ++j) {
        const int n = C2::col(tx, j);
        const float b = __ldg(bg2 + n);
        float s[4], st[4];
        g32::get4(A, C + n, s);
        g32::get4(Ad, C + n, st);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float g = sigmoid(q[0][j][e] + b);
          const float gd = g * (1.f - g) * q[1][j][e];
          q[1][j][e] = st[e] * g + s[e] * gd;
          q[0][j][e] = s[e] * g;
        }
        g32::put4(A, C + n, q[0][j]);
        g32::put4(Ad, C + n, q[1][j]);
      }
#pragma unroll
      for (int j = 0; j < N1; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) half[j][e] = 0.5f * (q[1][j][e] + q[1][j + N1][e]);
    }
    {
      float h[2][N2][4];
      g32::gemm_n<2 * C, 2 * C, 1, 2>(A, TAN, C, wf1, 2 * C, ring, h);
      ring.pre<C>(wf2, C);
      __syncthreads();
#pragma unroll
      for (int j = 0; j < N2; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) h[1][j][e] *= gelu_grad(h[0][j][e]);
        g32::put4(A, Ch::col(tx, j), h[1][j]);
      }
    }
    float o[N1][4];
    g32::gemm<2 * C, C>(A, 0, wf2, C, ring, o);
#pragma unroll
    for (int j = 0; j < N1; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[j][e] += half[j][e];
    g32::store_rows<C>(outd, nullptr, v0, V, o, al);
  }
}

// ------------------------------------------------------------------------------------------------ head
// Tangent of head_output (models/ffno_model.py:730-749) along the last block's tangent x' and the input tangent
// x_in': h' = (gelu'(x P1) x' P1) P2; per species, d log10 n_i = d log10 rho + sech^2(h_tot / b) h_tot'
// + (l_i' - sum_j p_j l_j') / ln 10 with l = h + lte (p = softmax(l)); lte' follows MULTI3D's LTE weights through
// log10 T and log10 ne (models/ffno_model.py:131-141).
template <int C, int NHP>
__global__ void __launch_bounds__(NT, C <= 64 ? 2 : 1) k_head_jvp(const float* __restrict__ x, const float* __restrict__ xd,
                                                 const float* __restrict__ xin, const float* __restrict__ xind, long V,
                                                 const float* __restrict__ p1, const float* __restrict__ p2,
                                                 const float* __restrict__ b2, HeadParams hp,
                                                 float* __restrict__ outd, int al) {
  griddep_sync();
  extern __shared__ __align__(16) float sm[];
  __shared__ double etab[EXP_TAB];
  constexpr int LO = NHP + 1, TAN = 2 * C * BM;
  fill_exp_table(etab);
  float* as = sm;                 // [C][64] input, then [2C][64] hidden; their tangents TAN floats on
  float* os = as + 2 * TAN;       // [64][NHP + 1] head channels, then their tangents
  float* ods = os + BM * LO;
  g32::Ring ring(ods + BM * LO, g32::KC * 2 * C, al);
  using Ch = g32::Cols<2 * C, 1>;
  using Co = g32::Cols<NHP, 1>;
  const int tx = g32::tile_tx(), ty = g32::tile_ty();
  const long nt = (V + BM - 1) / BM;
  for (long t = blockIdx.x; t < nt; t += gridDim.x) {
    const long v0 = t * BM;
    __syncthreads();
    ring.pre<2 * C>(p1, 2 * C);
    g32::load_tile<C>(as, 0, x, v0, V, al);
    g32::load_tile<C>(as + TAN, 0, xd, v0, V, al);
    {
      float h[2][2 * C / 16][4];
      g32::gemm_n<C, 2 * C, 1, 2>(as, TAN, 0, p1, 2 * C, ring, h);
      ring.pre<NHP>(p2, NHP);
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 2 * C / 16; ++j) {
        const int c = Ch::col(tx, j);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          h[1][j][e] *= gelu_grad(h[0][j][e]);
          h[0][j][e] = gelu(h[0][j][e]);
        }
        g32::put4(as, c, h[0][j]);
        g32::put4(as + TAN, c, h[1][j]);
      }
    }
    {
      float o[2][NHP / 16][4];
      g32::gemm_n<2 * C, NHP, 1, 2>(as, TAN, 0, p2, NHP, ring, o);
#pragma unroll
      for (int j = 0; j < NHP / 16; ++j) {
        const int n = Co::col(tx, j);
        const float b = __ldg(b2 + n);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          os[(4 * ty + e) * LO + n] = o[0][j][e] + b;
          ods[(4 * ty + e) * LO + n] = o[1][j][e];
        }
      }
    }
    __syncthreads();
    if (threadIdx.x < BM) {
      const int r = threadIdx.x;
      const long v = v0 + r;
      if (v < V) {
        const float* o = os + r * LO;
        const float* od = ods + r * LO;
        const int tc = hp.temperature_channel, ec = hp.ne_channel, rc = hp.rho_channel;
        const HeadInputs in = head_inputs(hp, xin, V, v);
        const HeadMath<double> hm{etab, head_fast(hp, o, head_channels(hp), in)};
        const Lte<double> le(hp, in, hm);
        const double dlt = (double)__ldg(xind + (long)tc * V + v) * (double)hp.std_x[tc];
        const double dlne = (double)__ldg(xind + (long)ec * V + v) * (double)hp.std_x[ec];
        const double dlrho = (double)__ldg(xind + (long)rc * V + v) * (double)hp.std_x[rc];
        int hc = 0, lvl = 0;
        for (int s = 0; s < hp.nspecies; ++s) {
          const int L = hp.levels[s];
          double logit[FFNO_MAX_LEVELS], dl[FFNO_MAX_LEVELS];
          double mx = -1e300;
          for (int i = 0; i < L; ++i) {
            const int g = lvl + i;
            const double lte = le.weight(hp, g);
            // d lte / d log10 T and d lte / d log10 ne (through t, the Debye term dxi ~ sqrt(ne / t) and conl)
            const double dT = kLN10 * (le.ek_t * (hp.ev[g] - 1.5 * le.dxi * hp.ndxi[g]) + 1.5 * hp.dion[g]);
            const double dN = kLN10 * (0.5 * le.ek_t * hp.ndxi[g] * le.dxi - hp.dion[g]);
            logit[i] = (double)o[hc + i] + lte;
            dl[i] = (double)od[hc + i] + dT * dlt + dN * dlne;
            mx = fmax(mx, logit[i]);
          }
          double se = 0.0, md = 0.0;
          for (int i = 0; i < L; ++i) {
            const double ex = hm.exp_(logit[i] - mx);
            se += ex;
            md += ex * dl[i];
          }
          md *= hm.inv_(se);
          const double th = hm.tanh_((double)o[hc + L] * hm.inv_((double)hp.total_bound));
          const double dtot = (1.0 - th * th) * (double)od[hc + L];
          for (int i = 0; i < L; ++i) {
            const int g = lvl + i;
            const double d = dlrho + dtot + (dl[i] - md) * kINV_LN10;
            outd[(long)g * V + v] = (float)(d * hm.inv_((double)hp.std_y[g]));
          }
          hc += L + 1;
          lvl += L;
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ service units
// Input tangent in the service's SI units (T [K], v [m/s], log10 ne, log10 rho) -> tangent of the normalised model
// inputs (log10 T, v / 1e3, ..., then (x - mean) / std; ffno_fsdp_runtime.py:48-58, 274-280). flags |= 1 on NaN/Inf.
__global__ void k_si_input_tangent(const float* __restrict__ feat, const float* __restrict__ td, long V,
                                   const float* __restrict__ std_x, float* __restrict__ xd, int* __restrict__ flags) {
  griddep_sync();
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < 6 * V; e += (long)gridDim.x * blockDim.x) {
    const int c = (int)(e / V);
    const float t = td[e];
    if (!isfinite(t)) atomicOr(flags, 1);
    float m;
    if (c == 0)
      m = t / (feat[e] * (float)kLN10);
    else if (c < 4)
      m = t / 1.0e3f;
    else
      m = t;
    xd[e] = m / std_x[c];
  }
}

// Model-output tangent (normalised log10 n, [L][V]) -> population tangent (nz, nx, ny, L) in m^-3: n = 10^clamp(y std
// + mean, +-37), n' = n ln 10 std y' inside the clamp, 0 outside (linear_populations, ffno_fsdp_runtime.py:76-78).
// flags |= 8 on a non-finite tangent.
__global__ void k_si_population_tangent(const float* __restrict__ y, const float* __restrict__ yd, long V, int L,
                                        const float* __restrict__ mean_y, const float* __restrict__ std_y,
                                        float* __restrict__ out, int* __restrict__ flags) {
  griddep_sync();
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < (long)L * V; e += (long)gridDim.x * blockDim.x) {
    const long v = e / L;
    const int l = (int)(e % L);
    const float pl = y[(long)l * V + v] * std_y[l] + mean_y[l];
    float d = 0.f;
    if (pl >= -37.f && pl <= 37.f) d = exp10f(pl) * (float)kLN10 * std_y[l] * yd[(long)l * V + v];
    if (!isfinite(d)) atomicOr(flags, 8);
    out[e] = d;
  }
}

}  // namespace

// ====================================================================================================== C ABI
extern "C" {

int ffno_gn_jvp_stats(const float* pre, const float* pre_dot, const double* gstats, const float* dw, long V, int C,
                      int groups, double* partials, int nparts, ffno_stream_t stream) {
  if (!pre || !pre_dot || !gstats || !dw || !partials || !width_ok(C) || V < 1 || groups < 1 || groups > GMAX ||
      C % groups || nparts < 1)
    return FFNO_EINVAL;
  cudaStream_t s = (cudaStream_t)stream;
  const int cpg = C / groups;
  switch (C) {
#define L(CC) case CC: ffno::launch(k_gn_jvp_stats<CC>, nparts, 256, 0, s, pre, pre_dot, gstats, dw, V, partials, cpg, groups); break;
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_gn_jvp_apply(const float* pre, const float* pre_dot, const float* gamma, const float* beta,
                      const double* gstats, const double* sums, int act, const float* base, float res, long V, int C,
                      int groups, float* out, ffno_stream_t stream) {
  if (!pre || !pre_dot || !gamma || !beta || !gstats || !sums || !out || !width_ok(C) || V < 1 || groups < 1 ||
      groups > GMAX || C % groups || act < 0 || act > 1)
    return FFNO_EINVAL;
  cudaStream_t s = (cudaStream_t)stream;
  const int cpg = C / groups;
  const long n4 = V * (C / 4);
  const int blocks = (int)((n4 + 255) / 256 < 8L * sms() ? (n4 + 255) / 256 : 8L * sms());
  switch (C) {
#define L(CC) case CC: ffno::launch(k_gn_jvp_apply<CC>, blocks, 256, 0, s, pre, pre_dot, gamma, beta, gstats, sums, act, base, res, V, out, cpg, groups); break;
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_gate_jvp(const float* x, const float* x_dot, long V, int C, const float* w1, const float* w2, float* out_dot,
                  ffno_stream_t stream) {
  if (!x || !x_dot || !w1 || !w2 || !out_dot || !width_ok(C) || V < 1) return FFNO_EINVAL;
  const int al = g32::aligned(x, x_dot, w1, w2, out_dot);
  cudaStream_t s = (cudaStream_t)stream;
  switch (C) {
#define L(CC)                                                                                 \
  case CC: {                                                                                  \
    const size_t smem = (4 * CC * BM + 2 * g32::KC * CC) * sizeof(float);                     \
    if (!smem_attr(k_gate_jvp<CC>, smem)) return FFNO_ELAUNCH;                                \
    ffno::launch(k_gate_jvp<CC>, grid_rows(V, BM, CC <= 64 ? 3 : 2), NT, smem, s, x, x_dot, V, w1, w2, out_dot, al); \
    break;                                                                                    \
  }
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_mlp2_jvp(const float* a, const float* a_dot, long V, int C, const float* w1, const float* w2, float* out_dot,
                  ffno_stream_t stream) {
  if (!a || !a_dot || !w1 || !w2 || !out_dot || !width_ok(C) || V < 1) return FFNO_EINVAL;
  const int al = g32::aligned(a, a_dot, w1, w2, out_dot);
  cudaStream_t s = (cudaStream_t)stream;
  switch (C) {
#define L(CC)                                                                                   \
  case CC: {                                                                                    \
    const size_t smem = (2 * CC * BM + 2 * g32::KC * 2 * CC) * sizeof(float);                   \
    if (!smem_attr(k_mlp2_jvp<CC>, smem)) return FFNO_ELAUNCH;                                  \
    ffno::launch(k_mlp2_jvp<CC>, grid_rows(V, BM, 2), NT, smem, s, a, a_dot, V, w1, w2, out_dot, al);      \
    break;                                                                                      \
  }
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_fuse_jvp(const float* x, const float* x_dot, const float* spec_pre, const float* spec_coefs,
                  const float* vert_pre, const float* vert_coefs, const float* spec_dot, const float* vert_dot, long V,
                  int C, const float* wg1, const float* wg2, const float* bg2, const float* wf1, const float* wf2,
                  float* fused_dot, ffno_stream_t stream) {
  if (!x || !x_dot || !spec_pre || !spec_coefs || !vert_pre || !vert_coefs || !spec_dot || !vert_dot || !wg1 ||
      !wg2 || !bg2 || !wf1 || !wf2 || !fused_dot || !width_ok(C) || V < 1)
    return FFNO_EINVAL;
  const int al = g32::aligned(x, x_dot, spec_pre, vert_pre, spec_dot, vert_dot, wg1, wg2, wf1, wf2, fused_dot);
  cudaStream_t s = (cudaStream_t)stream;
  switch (C) {
#define L(CC)                                                                                                 \
  case CC: {                                                                                                  \
    const size_t smem = fuse_jvp_smem<CC>();                                                                  \
    if (!smem_attr(k_fuse_jvp<CC>, smem)) return FFNO_ELAUNCH;                                                \
    ffno::launch(k_fuse_jvp<CC>, grid_rows(V, BM, CC <= 64 ? 2 : 1), NT, smem, s, x, x_dot, spec_pre, spec_coefs,        \
                                                                        vert_pre, vert_coefs, spec_dot,       \
                                                                        vert_dot, V, wg1, wg2, bg2, wf1, wf2, \
                                                                        fused_dot, al);                       \
    break;                                                                                                    \
  }
    L(16) L(32) L(64) L(96)
#undef L
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_head_jvp(const float* x, const float* x_dot, const float* x_in, const float* x_in_dot, long V, int C,
                  const float* p1, const float* p2, const float* b2, int nhp, const ffno_head_params* params,
                  float* out_dot, ffno_stream_t stream) {
  if (!x || !x_dot || !x_in || !x_in_dot || !p1 || !p2 || !b2 || !params || !out_dot || !width_ok(C) || V < 1)
    return FFNO_EINVAL;
  const int al = g32::aligned(x, x_dot, p1, p2);
  cudaStream_t s = (cudaStream_t)stream;
  switch (C * 1000 + nhp) {
#define L(CC, NN)                                                                                                  \
  case CC * 1000 + NN: {                                                                                           \
    const size_t smem = (4 * CC * BM + 2 * BM * (NN + 1) + 2 * g32::KC * 2 * CC) * sizeof(float);                  \
    if (!smem_attr(k_head_jvp<CC, NN>, smem)) return FFNO_ELAUNCH;                                                \
    ffno::launch(k_head_jvp<CC, NN>, grid_rows(V, BM, CC <= 64 ? 2 : 1), NT, smem, s, x, x_dot, x_in, x_in_dot, V, p1, p2, b2,    \
                                                                            *params, out_dot, al);                     \
    break;                                                                                                         \
  }
    L(16, 16) L(16, 32) L(32, 16) L(32, 32) L(64, 16) L(64, 32) L(96, 16) L(96, 32)
#undef L
    default:
      return FFNO_EINVAL;
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_si_input_tangent(const float* features, const float* tangent, long V, const float* std_x, float* x_dot,
                          int* flags, ffno_stream_t stream) {
  if (!features || !tangent || !std_x || !x_dot || !flags || V < 1) return FFNO_EINVAL;
  const long n = 6 * V;
  const int blocks = (int)((n + 255) / 256 < 8L * sms() ? (n + 255) / 256 : 8L * sms());
  ffno::launch(k_si_input_tangent, blocks, 256, 0, (cudaStream_t)stream, features, tangent, V, std_x, x_dot, flags);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_si_population_tangent(const float* y, const float* y_dot, long V, int L, const float* mean_y,
                               const float* std_y, float* out, int* flags, ffno_stream_t stream) {
  if (!y || !y_dot || !mean_y || !std_y || !out || !flags || V < 1 || L < 1) return FFNO_EINVAL;
  const long n = (long)L * V;
  const int blocks = (int)((n + 255) / 256 < 8L * sms() ? (n + 255) / 256 : 8L * sms());
  ffno::launch(k_si_population_tangent, blocks, 256, 0, (cudaStream_t)stream, y, y_dot, V, L, mean_y, std_y, out, flags);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

}  // extern "C"
