// FP32 kernels of the two spectral operators: the batched transform GEMM that carries every DFT of the path as a
// contraction with a precomputed real table (rfft/irfft along W, complex DFT along H, the Filon height transform and
// its inverse), and the per-frequency complex channel mixing.
#include "common.cuh"
#include "gemm_f32.cuh"

using namespace ffno;

namespace {

// out[b][m][n] (+)= sum_k T[m][k] in[b][k][n], k ascending. CTA tile: 16 MR table rows x 128 data columns (64 with a
// table per batch element), 256 threads; a thread owns MR rows x NR columns, so a k step is MR / 4 + NR / 4 16-byte
// shared reads for MR NR FMAs (8 x 8: 64 FMAs per 4 reads). Bound by the FP32 pipe for the long contractions and by HBM
// for the short ones.
//  - Columns run over (batch, n) as one index, so that a tile is full at any N (the W transforms have N = C = 16-96); a
//    quad of 4 columns stays inside a batch because N % 4 == 0, and a thread keeps the same quads for every k.
//  - MR is the smallest that covers M in the fewest tiles of at most 144 rows (xform_rows): a 128-point real DFT has
//    130 rows, which take one tile of 9 x 16 instead of three tiles of 64.
//  - Chunks of 16 k arrive by cp.async into two stages, one barrier a chunk: the data 16 bytes at a time, the table
//    (transposed on the way) 4 bytes at a time.
//  - VEC = false: any N, strides and alignment (4-byte loads, 64 x 64 tiles).
// 4.2 M voxels, C = 64 (256 x 128 x 128), one forward's six transforms: 26.1 -> 10.1 ms; the H transforms run at
// 73 TFLOP/s.
constexpr int XK = 16;

__device__ __forceinline__ void cp16(void* dst, const void* src, bool ok) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  const int n = ok ? 16 : 0;   // the rest is zero
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

__device__ __forceinline__ void cp4(void* dst, const void* src, bool ok) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  const int n = ok ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

template <int MR>
struct XRows {   // rows of thread row ty in a 16 MR-row tile: quads of 4 consecutive rows, then single rows
  static constexpr int QA = MR / 4, RA = MR % 4, TM = 16 * MR, LD = TM + 4;
  __device__ static __forceinline__ int row(int ty, int i) {
    return i < 4 * QA ? (i / 4) * 64 + 4 * ty + i % 4 : 64 * QA + 16 * (i - 4 * QA) + ty;
  }
};

template <int MR, int NR, bool VEC>
__global__ void __launch_bounds__(NT, MR * NR > 32 ? 2 : 3) k_xform(const float* __restrict__ T, const float* __restrict__ in,
                                                 float* __restrict__ out, ffno_xform_desc d, long ntn, long ntm,
                                                 int accumulate, long t_b, long ncols) {
  griddep_sync();
  using R = XRows<MR>;
  constexpr int TN = 16 * NR, TPT = (R::TM * XK + NT - 1) / NT;   // table elements a thread moves per chunk
  __shared__ __align__(16) float ts[2][XK][R::LD];
  __shared__ __align__(16) float is[2][XK][TN];
  const int tid = threadIdx.x;
  const int ty = ((tid >> 6) << 2) + ((tid & 31) >> 3), tx = (((tid >> 5) & 1) << 3) + (tid & 7);
  // m tiles vary fastest, so the CTAs that share one slab of `in` run together and read it from L2
  long bid = blockIdx.x;
  const int m0 = (int)(bid % ntm) * R::TM;
  bid /= ntm;
  const long c0 = (bid % ntn) * TN;        // first column of the tile
  const long bt = bid / ntn;               // batch element with its own table (t_b != 0), else 0
  T += bt * t_b;
  // column c -> (batch, n); the batch's input and output offsets
  auto in_col = [&](long c, bool& ok) {
    const long b = t_b ? bt : c / d.N, n = t_b ? c : c % d.N;
    ok = c < ncols;
    return (b / d.nb2) * d.in_b1 + (b % d.nb2) * d.in_b2 + n;
  };
  auto in_row = [&](int k) {
    return k < d.in_split ? (long)k * d.in_lo
                          : (long)(k / d.in_split) * d.in_hi + (long)(k % d.in_split) * d.in_lo;
  };
  constexpr int QN = TN / 4, RPP = NT / QN;   // quads a row, k rows per pass of the CTA
  const int lq = tid % QN, lr = tid / QN;
  bool lok;
  const float* lsrc = in + in_col(c0 + 4 * lq, lok);
  if (!lok) lsrc = in;
  auto load_in = [&](int st, int k0) {
    if constexpr (VEC) {
#pragma unroll
      for (int p = 0; p < XK / RPP; ++p) {
        const int r = lr + p * RPP, k = k0 + r;
        const bool ok = lok && k < d.K;
        cp16(&is[st][r][4 * lq], ok ? lsrc + in_row(k) : in, ok);
      }
    } else {
      for (int e = tid; e < XK * TN; e += NT) {
        const int r = e / TN, c = e % TN, k = k0 + r;
        bool ok;
        const long o = in_col(c0 + c, ok);
        is[st][r][c] = ok && k < d.K ? __ldg(in + o + in_row(k)) : 0.f;
      }
    }
  };
  auto load_t = [&](int st, int k0) {
#pragma unroll
    for (int p = 0; p < TPT; ++p) {
      const int e = tid + p * NT, m = m0 + e / XK, k = k0 + e % XK;
      const bool ok = m < d.M && k < d.K;
      if (e < R::TM * XK) cp4(&ts[st][e % XK][e / XK], ok ? T + (long)m * d.K + k : T, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  uint64_t acc2[MR][NR / 2];   // two neighbouring columns per FMA (f32x2)
#pragma unroll
  for (int i = 0; i < MR; ++i)
#pragma unroll
    for (int j = 0; j < NR / 2; ++j) acc2[i][j] = 0;
  load_in(0, 0);
  load_t(0, 0);
  const int nch = (d.K + XK - 1) / XK;
#pragma unroll 1
  for (int c = 0; c < nch; ++c) {
    const int st = c & 1;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();   // chunk c is in, and every read of the other stage is done
    if (c + 1 < nch) {
      load_in(st ^ 1, (c + 1) * XK);
      load_t(st ^ 1, (c + 1) * XK);
    }
#pragma unroll
    for (int k = 0; k < XK; ++k) {
      float a[MR], b[NR];
#pragma unroll
      for (int q = 0; q < R::QA; ++q) {
        const float4 v = *reinterpret_cast<const float4*>(&ts[st][k][64 * q + 4 * ty]);
        a[4 * q] = v.x, a[4 * q + 1] = v.y, a[4 * q + 2] = v.z, a[4 * q + 3] = v.w;
      }
#pragma unroll
      for (int q = 0; q < R::RA; ++q) a[4 * R::QA + q] = ts[st][k][64 * R::QA + 16 * q + ty];
#pragma unroll
      for (int q = 0; q < NR / 4; ++q) {
        const float4 v = *reinterpret_cast<const float4*>(&is[st][k][64 * q + 4 * tx]);
        b[4 * q] = v.x, b[4 * q + 1] = v.y, b[4 * q + 2] = v.z, b[4 * q + 3] = v.w;
      }
#pragma unroll
      for (int i = 0; i < MR; ++i) {
        const uint64_t aa = pk2(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < NR / 2; ++j) acc2[i][j] = fma2(aa, pk2(b[2 * j], b[2 * j + 1]), acc2[i][j]);
      }
    }
  }
  float acc[MR][NR];
#pragma unroll
  for (int i = 0; i < MR; ++i)
#pragma unroll
    for (int j = 0; j < NR / 2; ++j) upk2(acc2[i][j], acc[i][2 * j], acc[i][2 * j + 1]);
#pragma unroll
  for (int q = 0; q < NR / 4; ++q) {
    const long cq = c0 + 64 * q + 4 * tx;
    if constexpr (VEC) {
      if (cq >= ncols) continue;
      const long b = t_b ? bt : cq / d.N, n = t_b ? cq : cq % d.N;
      float* ob = out + (b / d.nb2) * d.out_b1 + (b % d.nb2) * d.out_b2 + n;
#pragma unroll
      for (int i = 0; i < MR; ++i) {
        const int m = m0 + R::row(ty, i);
        if (m >= d.M) continue;
        float* o = ob + (long)(m / d.out_split) * d.out_hi + (long)(m % d.out_split) * d.out_lo;
        float4 v = make_float4(acc[i][4 * q], acc[i][4 * q + 1], acc[i][4 * q + 2], acc[i][4 * q + 3]);
        if (accumulate) {
          const float4 p = *reinterpret_cast<const float4*>(o);
          v = make_float4(p.x + v.x, p.y + v.y, p.z + v.z, p.w + v.w);
        }
        *reinterpret_cast<float4*>(o) = v;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (cq + j >= ncols) continue;
        const long b = t_b ? bt : (cq + j) / d.N, n = t_b ? cq + j : (cq + j) % d.N;
        float* ob = out + (b / d.nb2) * d.out_b1 + (b % d.nb2) * d.out_b2 + n;
#pragma unroll
        for (int i = 0; i < MR; ++i) {
          const int m = m0 + R::row(ty, i);
          if (m >= d.M) continue;
          float* o = ob + (long)(m / d.out_split) * d.out_hi + (long)(m % d.out_split) * d.out_lo;
          *o = accumulate ? *o + acc[i][4 * q + j] : acc[i][4 * q + j];
        }
      }
    }
  }
}

// Rows per thread: M in the fewest tiles of at most 9 x 16 rows, then the fewest rows that cover it.
int xform_rows(int M) {
  const int tiles = (M + 143) / 144;
  const int mr = (M + 16 * tiles - 1) / (16 * tiles);
  return mr < 2 ? 2 : mr == 7 ? 8 : mr;
}

template <int MR, int NR, bool VEC>
int launch_xform(const float* T, const float* in, float* out, const ffno_xform_desc& d, int accumulate, long t_b,
                 cudaStream_t s) {
  const long ncols = t_b ? d.N : d.N * d.nb;
  const long ntn = (ncols + 16 * NR - 1) / (16 * NR), ntm = (d.M + 16 * MR - 1) / (16 * MR);
  const long blocks = ntn * ntm * (t_b ? d.nb : 1);
  if (blocks > 0x7fffffffL) return FFNO_EINVAL;
  ffno::launch(k_xform<MR, NR, VEC>, (unsigned)blocks, NT, 0, s, T, in, out, d, ntn, ntm, accumulate, t_b, ncols);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int xform(const float* T, long t_b, const float* in, float* out, const ffno_xform_desc& d, int accumulate,
          cudaStream_t s) {
  if (d.nb < 1 || d.nb2 < 1 || d.K < 1 || d.M < 1 || d.N < 1 || d.in_split < 1 || d.out_split < 1)
    return FFNO_EINVAL;
  // 16-byte accesses: every column quad starts on 16 bytes in each row of each batch element
  const bool vec = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) % 16) == 0 &&
                   (d.N | d.in_b1 | d.in_b2 | d.in_hi | d.in_lo | d.out_b1 | d.out_b2 | d.out_hi | d.out_lo) % 4 == 0;
  if (!vec) return launch_xform<4, 4, false>(T, in, out, d, accumulate, t_b, s);
  if (t_b) {   // a table per batch element: N = C columns each
    switch (xform_rows(d.M)) {
      case 2: return launch_xform<2, 4, true>(T, in, out, d, accumulate, t_b, s);
      case 3: return launch_xform<3, 4, true>(T, in, out, d, accumulate, t_b, s);
      case 4: return launch_xform<4, 4, true>(T, in, out, d, accumulate, t_b, s);
      case 5: return launch_xform<5, 4, true>(T, in, out, d, accumulate, t_b, s);
      case 6: return launch_xform<6, 4, true>(T, in, out, d, accumulate, t_b, s);
      case 8: return launch_xform<8, 4, true>(T, in, out, d, accumulate, t_b, s);
      default: return launch_xform<9, 4, true>(T, in, out, d, accumulate, t_b, s);
    }
  }
  switch (xform_rows(d.M)) {
    case 2: return launch_xform<2, 8, true>(T, in, out, d, accumulate, 0, s);
    case 3: return launch_xform<3, 8, true>(T, in, out, d, accumulate, 0, s);
    case 4: return launch_xform<4, 8, true>(T, in, out, d, accumulate, 0, s);
    case 5: return launch_xform<5, 8, true>(T, in, out, d, accumulate, 0, s);
    case 6: return launch_xform<6, 8, true>(T, in, out, d, accumulate, 0, s);
    case 8: return launch_xform<8, 8, true>(T, in, out, d, accumulate, 0, s);
    default: return launch_xform<9, 8, true>(T, in, out, d, accumulate, 0, s);
  }
}

// Per-frequency mixing, CTA = 64 rows b of one frequency f: the region holds [re | im] of each row (2C channels,
// k-major), a thread owns channel o of both parts of its 4 rows. The projections V_f x (rank columns for each part) and
// their product with U_f run on the same operands, 4 rows a read. 4.2 M voxels, C = 64, plane and height mixing of a
// block: 5.89 -> 2.41 ms.
template <int C>
constexpr size_t mix_smem() {
  return (2 * C * BM + 2 * g32::KC * 2 * C + 2 * 16 * C + 32 * BM) * sizeof(float);
}

template <int C>
__global__ void __launch_bounds__(NT, C <= 32 ? 3 : 2) k_mix(const float* __restrict__ in, float* __restrict__ out, long F, long nb,
                                               long sf, long sb, long s_im, const float* __restrict__ wbig,
                                               const float* __restrict__ g, const float* __restrict__ U,
                                               const float* __restrict__ Vm, int rank, int al) {
  griddep_sync();
  extern __shared__ __align__(16) float sm[];
  float* xs = sm;                               // [2C][64]
  g32::Ring ring(xs + 2 * C * BM, g32::KC * 2 * C, al);
  float* us = xs + 2 * C * BM + 2 * g32::KC * 2 * C;   // [rank][C]
  float* vs = us + 16 * C;                      // [C][rank]
  float* ts = vs + 16 * C;                      // [2 rank][64]: V_f x, re then im
  using Cl = g32::Cols<2 * C, 2>;
  const int tx = g32::tile_tx(), ty = g32::tile_ty();
  const long nbt = (nb + BM - 1) / BM;
  const long f = blockIdx.x / nbt;
  const long b0 = (blockIdx.x % nbt) * BM;
  if (f >= F) return;
  const float* fin = in + f * sf;
  ring.pre<2 * C>(wbig, 2 * C);
  g32::each_quad<C>(0, BM, [&](int r, int c, long, bool) {
    const bool ok = b0 + r < nb;
    const float* p = fin + (b0 + r) * sb + c;
    const float4 re = g32::ldq(p, ok, al), im = g32::ldq(p + s_im, ok, al);
    g32::put_quad(xs, r, c, re);
    g32::put_quad(xs, r, C + c, im);
  });
  for (int e = threadIdx.x; e < C * rank; e += NT) {
    us[(e % rank) * C + e / rank] = __ldg(U + f * C * rank + e);
    vs[(e % C) * rank + e / C] = __ldg(Vm + f * C * rank + e);
  }
  float acc[2 * C / 16][4];
  g32::gemm<2 * C, 2 * C, 2>(xs, 0, wbig, 2 * C, ring, acc);
  const float gr = __ldg(g + 2 * f), gi = __ldg(g + 2 * f + 1);
#pragma unroll
  for (int j = 0; j < C / 16; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float ar = acc[j][e], ai = acc[j + C / 16][e];
      acc[j][e] = ar * gr - ai * gi;
      acc[j + C / 16][e] = ar * gi + ai * gr;
    }
  if (rank) {
    // t[q][row] = sum_i V[r][i] x[part C + i][row], q = part rank + r
    for (int q = tx; q < 2 * rank; q += 16) {
      const int part = q / rank;
      float t[4] = {0.f, 0.f, 0.f, 0.f};
      const float* vr = vs + q % rank;
#pragma unroll 8
      for (int i = 0; i < C; ++i) {
        float x[4];
        g32::get4(xs, part * C + i, x);
        const float v = vr[i * rank];
#pragma unroll
        for (int e = 0; e < 4; ++e) t[e] = fmaf(v, x[e], t[e]);
      }
      *reinterpret_cast<float4*>(ts + q * BM + 4 * ty) = make_float4(t[0], t[1], t[2], t[3]);
    }
    __syncthreads();
    float lo[2 * C / 16][4];
#pragma unroll
    for (int j = 0; j < 2 * C / 16; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) lo[j][e] = 0.f;
    for (int r = 0; r < rank; ++r) {
      const float4 re = *reinterpret_cast<const float4*>(ts + r * BM + 4 * ty);
      const float4 im = *reinterpret_cast<const float4*>(ts + (rank + r) * BM + 4 * ty);
      const float tr[4] = {re.x, re.y, re.z, re.w}, ti[4] = {im.x, im.y, im.z, im.w};
#pragma unroll
      for (int j = 0; j < C / 16; ++j) {
        const float u = us[r * C + Cl::col(tx, j)];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          lo[j][e] = fmaf(u, tr[e], lo[j][e]);
          lo[j + C / 16][e] = fmaf(u, ti[e], lo[j + C / 16][e]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 2 * C / 16; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[j][e] += lo[j][e];
  }
  constexpr int CV = Cl::CV;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const long b = b0 + 4 * ty + e;
    if (b >= nb) continue;
    float* fo = out + f * sf + b * sb;
#pragma unroll
    for (int j = 0; j < 2 * C / 16; j += CV) {
      const int o = Cl::col(tx, j);
      float* p = o < C ? fo + o : fo + s_im + (o - C);
      float v[CV];
#pragma unroll
      for (int i = 0; i < CV; ++i) v[i] = acc[j + i][e];
      g32::st_run<CV>(p, v, al);
    }
  }
}

}  // namespace

extern "C" {

int ffno_xform(const float* T, const float* in, float* out, const ffno_xform_desc* desc, int accumulate,
               ffno_stream_t stream) {
  if (!T || !in || !out || !desc) return FFNO_EINVAL;
  return xform(T, 0, in, out, *desc, accumulate, (cudaStream_t)stream);
}

int ffno_xform_pt(const float* T, long t_b, const float* in, float* out, const ffno_xform_desc* desc, int accumulate,
                  ffno_stream_t stream) {
  if (!T || !in || !out || !desc || t_b < 0) return FFNO_EINVAL;
  return xform(T, t_b, in, out, *desc, accumulate, (cudaStream_t)stream);
}

// out[col][i][j] (+)= sum_c A[i*rs + col*C + c] * B[j*rs + col*C + c], one CTA per column: the per-column
// height-table gradients. Output tiles of 64 rows of A x 64 rows of B: both row blocks staged in shared memory
// (coalesced row loads, rows padded to C + 1 floats), 4 x 4 outputs a thread summed over the C channels in FP32, then
// added to the FP64 output (which accumulates the blocks of a VJP).
constexpr int OT = 64;

__global__ void __launch_bounds__(256) k_col_outer(const float* __restrict__ A, int Ra, const float* __restrict__ B,
                                                   int Rb, long ncol, int C, long rs, double* __restrict__ out,
                                                   int accumulate) {
  griddep_sync();
  extern __shared__ float osm[];
  const int LD = C + 1;
  float* as = osm;             // [OT][C + 1]
  float* bs = osm + OT * LD;   // [OT][C + 1]
  const long col = blockIdx.x;
  if (col >= ncol) return;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  for (int i0 = 0; i0 < Ra; i0 += OT) {
    for (int j0 = 0; j0 < Rb; j0 += OT) {
      __syncthreads();   // the previous tile's reads are done
      for (int e = threadIdx.x; e < OT * C; e += blockDim.x) {
        const int r = e / C, c = e % C;
        as[r * LD + c] = i0 + r < Ra ? __ldg(A + (long)(i0 + r) * rs + col * C + c) : 0.f;
        bs[r * LD + c] = j0 + r < Rb ? __ldg(B + (long)(j0 + r) * rs + col * C + c) : 0.f;
      }
      __syncthreads();
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
      for (int c = 0; c < C; ++c) {
        float a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = as[(ty + 16 * i) * LD + c];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = bs[(tx + 16 * j) * LD + c];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int ii = i0 + ty + 16 * i;
        if (ii >= Ra) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int jj = j0 + tx + 16 * j;
          if (jj >= Rb) continue;
          double* o = out + (col * Ra + ii) * (long)Rb + jj;
          *o = accumulate ? *o + (double)acc[i][j] : (double)acc[i][j];
        }
      }
    }
  }
}

int ffno_col_outer(const float* A, int Ra, const float* B, int Rb, long ncol, int C, long row_stride, double* out,
                   int accumulate, ffno_stream_t stream) {
  if (!A || !B || !out || Ra < 1 || Rb < 1 || ncol < 1 || C < 1 || C > 512 || ncol > 0x7fffffffL) return FFNO_EINVAL;
  const size_t smem = (size_t)2 * OT * (C + 1) * sizeof(float);
  if (!ffno::smem_cap_ok(k_col_outer, smem)) return FFNO_ELAUNCH;
  ffno::launch(k_col_outer, (unsigned)ncol, 256, smem, (cudaStream_t)stream, A, Ra, B, Rb, ncol, C, row_stride, out,
                                                                  accumulate);
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

int ffno_spectral_mix(const float* in, float* out, long F, long nb, long sf, long sb, long s_im, int C,
                      const float* wbig, const float* g, const float* U, const float* Vm, int rank,
                      ffno_stream_t stream) {
  if (!in || !out || !wbig || !g || F < 1 || nb < 1 || rank < 0 || rank > 16) return FFNO_EINVAL;
  if (rank && (!U || !Vm)) return FFNO_EINVAL;
  const long nbt = (nb + BM - 1) / BM;
  const long blocks = F * nbt;
  if (blocks > 0x7fffffffL) return FFNO_EINVAL;
  // 16-byte accesses where every row and the weights start on 16 bytes
  const int al = (sf | sb | s_im) % 4 == 0 && g32::aligned(in, out, wbig);
  cudaStream_t s = (cudaStream_t)stream;
  switch (C) {
#define L(CC)                                                                                              \
  case CC: {                                                                                               \
    const size_t smem = mix_smem<CC>();                                                                    \
    if (!ffno::smem_cap_ok(k_mix<CC>, smem)) return FFNO_ELAUNCH;                                          \
    ffno::launch(k_mix<CC>, (unsigned)blocks, NT, smem, s, in, out, F, nb, sf, sb, s_im, wbig, g, U, Vm, rank, al);  \
    break;                                                                                                 \
  }
    L(16) L(32) L(64) L(96)
#undef L
    default:
      return FFNO_EINVAL;
  }
  FFNO_CHECK_LAUNCH();
  return FFNO_OK;
}

}  // extern "C"
