// FP32 tile GEMM of the channel chains (gates, MLPs, fusion, head, their VJPs and JVPs, the spectral mixing): tiles of
// 64 voxels by N output channels per CTA of 256 threads, operands in shared memory, FP32 FMAs in ascending k.
//
// What bounds it: the FP32 pipe (71 TFLOP/s measured for an outer-product loop in registers) once the operands arrive
// in few enough instructions (f32x2: two FMAs an instruction). A thread owns 4 consecutive voxels and N / 16 output channels, so one k step is one
// 16-byte read of the activations, one 8- or 16-byte read of the weights per 2-4 channels and 4 N / 16 FMAs: shared
// memory moves 4-5 wavefronts per 32-48 FMAs of a warp. (The form before read every operand as one 4-byte word, the
// weights from global memory: 12 loads per 32 FMAs, bound by the load unit at about 20 TFLOP/s.)
//
//  - Activations sit in k-major regions [k][64 voxels], where a thread's 4 voxels are one 16-byte chunk. Chunk j of row
//    k is stored at j ^ ((k / 4) % 8), so that the epilogues (8 lanes hold 8 groups of 4 consecutive channels) and the
//    row loads (8 channel quads x 4 voxels per warp) write without bank conflicts.
//  - Weights [K][N] stream from L2 through a two-stage ring of 16 k rows by cp.async; the caller issues the first
//    chunk (Ring::pre) before the elementwise work that precedes the GEMM, so its latency hides behind that work.
//  - Warp w covers 16 voxels (w / 2) x half of the channel groups (w % 2): 4 voxel quads x 8 channel groups.
#pragma once
#include "common.cuh"

namespace ffno {
namespace g32 {

constexpr int KC = 16;   // k rows of one weight chunk

__device__ __forceinline__ int tile_ty() { return ((threadIdx.x >> 6) << 2) + ((threadIdx.x & 31) >> 3); }
__device__ __forceinline__ int tile_tx() { return (((threadIdx.x >> 5) & 1) << 3) + (threadIdx.x & 7); }

// float offset of voxel row r of channel k in a k-major region
__device__ __forceinline__ int at(int r, int k) { return k * BM + ((((r >> 2) ^ ((k >> 2) & 7)) << 2) | (r & 3)); }
// float offset of the voxel quad 4 q .. 4 q + 3 of channel k (a 16-byte chunk)
__device__ __forceinline__ int at4(int q, int k) { return k * BM + ((q ^ ((k >> 2) & 7)) << 2); }

// The channels of thread column tx in an N-channel output cut into G equal groups (G = 2 where the same thread has to
// own channel c of both halves): runs of CV consecutive channels, interleaved over the 16 thread columns.
template <int N, int G>
struct Cols {
  static constexpr int NC = N / 16, NG = NC / G;
  static constexpr int CV = NG % 4 == 0 ? 4 : NG % 2 == 0 ? 2 : 1;
  static_assert(N % (16 * G) == 0, "16 thread columns per group");
  __device__ static __forceinline__ int col(int tx, int j) {
    const int g = j / NG, i = j % NG;
    return g * (N / G) + (i / CV) * (16 * CV) + tx * CV + i % CV;
  }
};

// Two-stage ring of weight chunks [KC][N] in shared memory (2 KC N floats for the widest GEMM of the kernel).
struct Ring {
  float* buf;
  int floats, st;   // floats per stage; the stage the next chunk goes to
  int al;           // the weights start on 16 bytes (else 4-byte copies)
  __device__ __forceinline__ Ring(float* b, int f, int a) : buf(b), floats(f), st(0), al(a) {}
  template <int N>
  __device__ __forceinline__ void issue(const float* __restrict__ w, int ldw) {
    constexpr int Q = N / 4;
    const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(buf + st * floats));
    if (al) {
#pragma unroll
      for (int u = threadIdx.x; u < KC * Q; u += NT) {
        const int k = u / Q, q = u % Q;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 4 * (k * N + 4 * q)),
                     "l"(w + (long)k * ldw + 4 * q)
                     : "memory");
      }
    } else {
#pragma unroll 1
      for (int u = threadIdx.x; u < KC * N; u += NT)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * u), "l"(w + (long)(u / N) * ldw + u % N)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // The first chunk of the next GEMM. The stage it goes to was last read before the last barrier of the GEMM before.
  template <int N>
  __device__ __forceinline__ void pre(const float* __restrict__ w, int ldw) { issue<N>(w, ldw); }
};

template <int CV>
__device__ __forceinline__ void ldw(const float* p, float* o) {
  if constexpr (CV == 4) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    o[0] = v.x, o[1] = v.y, o[2] = v.z, o[3] = v.w;
  } else if constexpr (CV == 2) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    o[0] = v.x, o[1] = v.y;
  } else {
    o[0] = *p;
  }
}

// acc[j][e] = sum_k A[k0 + k][voxel 4 ty + e] W[k][col(tx, j)], k < K ascending, for A in the k-major region `as` (NA
// operands at as, as + stride_a, ... share the weights). The first chunk of W has been issued by ring.pre<N>; the first
// barrier in here also publishes what the caller wrote to the region.
template <int K, int N, int G, int NA>
__device__ __forceinline__ void gemm_n(const float* __restrict__ as, int stride_a, int k0, const float* __restrict__ w,
                                       int ldw_, Ring& ring, float (&acc)[NA][N / 16][4]) {
  using Cl = Cols<N, G>;
  static_assert(K % KC == 0, "whole chunks");
  const int tx = tile_tx(), ty = tile_ty();
  // two neighbouring channels of a run per FMA where the run has two (f32x2: half the issue slots, the same products and
  // sums): NP accumulators of PW channels
  constexpr int PW = Cl::CV > 1 ? 2 : 1, NP = Cl::NC / PW;
  uint64_t acc2[PW == 2 ? NA : 1][PW == 2 ? NP : 1][4];
#pragma unroll
  for (int a = 0; a < NA; ++a)
#pragma unroll
    for (int j = 0; j < NP; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if constexpr (PW == 2)
          acc2[a][j][e] = 0;
        else
          acc[a][j][e] = 0.f;
      }
#pragma unroll 1
  for (int c = 0; c < K / KC; ++c) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const float* ws = ring.buf + ring.st * ring.floats + tx * Cl::CV;
    ring.st ^= 1;
    if (c + 1 < K / KC) ring.issue<N>(w + (long)(c + 1) * KC * ldw_, ldw_);
    const int kb = k0 + c * KC, sw = (kb >> 2) & 7;
    const float* ab = as + kb * BM;
#pragma unroll
    for (int k = 0; k < KC; ++k) {
      float b[Cl::NC];
#pragma unroll
      for (int j = 0; j < Cl::NC; j += Cl::CV)
        ldw<Cl::CV>(ws + k * N + (j / Cl::NG) * (N / G) + (j % Cl::NG) * 16, b + j);
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        const float4 v = *reinterpret_cast<const float4*>(ab + a * stride_a + k * BM + ((ty ^ sw ^ (k >> 2)) << 2));
        const float x[4] = {v.x, v.y, v.z, v.w};
        if constexpr (PW == 2) {
          uint64_t xx[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) xx[e] = pk2(x[e], x[e]);
#pragma unroll
          for (int j = 0; j < NP; ++j) {
            const uint64_t bb = pk2(b[2 * j], b[2 * j + 1]);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc2[a][j][e] = fma2(xx[e], bb, acc2[a][j][e]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < Cl::NC; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[a][j][e] = fmaf(x[e], b[j], acc[a][j][e]);
        }
      }
    }
  }
  if constexpr (PW == 2) {
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
      for (int j = 0; j < NP; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) upk2(acc2[a][j][e], acc[a][2 * j][e], acc[a][2 * j + 1][e]);
  }
}

template <int K, int N, int G = 1>
__device__ __forceinline__ void gemm(const float* __restrict__ as, int k0, const float* __restrict__ w, int ldw_,
                                     Ring& ring, float (&acc)[N / 16][4]) {
  gemm_n<K, N, G, 1>(as, 0, k0, w, ldw_, ring, reinterpret_cast<float (&)[1][N / 16][4]>(acc));
}

// Channel k of the thread's voxel quad in a region.
__device__ __forceinline__ void put4(float* s, int k, const float (&v)[4]) {
  *reinterpret_cast<float4*>(s + at4(tile_ty(), k)) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void get4(const float* s, int k, float (&v)[4]) {
  const float4 q = *reinterpret_cast<const float4*>(s + at4(tile_ty(), k));
  v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
}

// Visit the 64 x C tile at voxel v0 as quads of 4 channels: f(row, channel, global offset, inside). A warp covers 4 rows
// x 8 quads (128 contiguous bytes a row), 8 x 4 at C = 16, the order in which stores to a region have no conflicts.
template <int C, typename F>
__device__ __forceinline__ void each_quad(long v0, long V, F f) {
  constexpr int Q = C / 4, QW = Q < 8 ? Q : 8, RW = 32 / QW;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int u = threadIdx.x >> 5; u < (BM / RW) * (Q / QW); u += NT / 32) {
    const int r = (u / (Q / QW)) * RW + lane / QW, q = (u % (Q / QW)) * QW + lane % QW;
    f(r, 4 * q, (v0 + r) * C + 4 * q, v0 + r < V);
  }
}

// Whether every pointer starts on 16 bytes: the kernels' `al` argument, which picks 16-byte or 4-byte accesses.
template <typename... P>
inline int aligned(const P*... p) {
  return ((... | reinterpret_cast<uintptr_t>(p)) % 16) == 0;
}

__device__ __forceinline__ float4 ldq(const float* p, bool ok, int al) {
  if (!ok) return make_float4(0.f, 0.f, 0.f, 0.f);
  if (al) return __ldg(reinterpret_cast<const float4*>(p));
  return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}
__device__ __forceinline__ void stq(float* p, float4 v, int al) {
  if (al) {
    *reinterpret_cast<float4*>(p) = v;
  } else {
    p[0] = v.x, p[1] = v.y, p[2] = v.z, p[3] = v.w;
  }
}
__device__ __forceinline__ void put_quad(float* s, int r, int c, float4 v) {
  s[at(r, c)] = v.x;
  s[at(r, c + 1)] = v.y;
  s[at(r, c + 2)] = v.z;
  s[at(r, c + 3)] = v.w;
}

// Rows v0 .. v0 + 63 of g [V][C] into channels k0 .. k0 + C - 1 of a region; rows at or past V are zero.
template <int C>
__device__ __forceinline__ void load_tile(float* s, int k0, const float* __restrict__ g, long v0, long V, int al) {
  each_quad<C>(v0, V, [&](int r, int c, long o, bool ok) { put_quad(s, r, k0 + c, ldq(g + o, ok, al)); });
}

// Store the thread's CV consecutive channels of one voxel (v: the values of channels j .. j + CV - 1).
template <int CV>
__device__ __forceinline__ void st_run(float* p, const float* v, int al) {
  if (CV == 1 || !al) {
#pragma unroll
    for (int i = 0; i < CV; ++i) p[i] = v[i];
  } else if constexpr (CV == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else if constexpr (CV == 2) {
    *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  }
}
template <int CV>
__device__ __forceinline__ void ld_run(const float* p, float* v, int al) {
  if (CV == 1 || !al) {
#pragma unroll
    for (int i = 0; i < CV; ++i) v[i] = __ldg(p + i);
  } else if constexpr (CV == 4) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  } else if constexpr (CV == 2) {
    const float2 q = __ldg(reinterpret_cast<const float2*>(p));
    v[0] = q.x, v[1] = q.y;
  }
}

// out[v][c] = val (+ base[v][c]) for the thread's voxels and channels of a C-channel output (base may be null).
template <int C, int NACC>
__device__ __forceinline__ void store_rows(float* __restrict__ out, const float* __restrict__ base, long v0, long V,
                                           const float (&acc)[NACC][4], int al) {
  using Cl = Cols<C, 1>;
  const int tx = tile_tx(), ty = tile_ty();
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const long v = v0 + 4 * ty + e;
    if (v >= V) continue;
#pragma unroll
    for (int j = 0; j < Cl::NC; j += Cl::CV) {
      const long o = v * C + Cl::col(tx, j);
      float t[Cl::CV];
#pragma unroll
      for (int i = 0; i < Cl::CV; ++i) t[i] = acc[j + i][e];
      if (base) {
        float b[Cl::CV];
        ld_run<Cl::CV>(base + o, b, al);
#pragma unroll
        for (int i = 0; i < Cl::CV; ++i) t[i] += b[i];
      }
      st_run<Cl::CV>(out + o, t, al);
    }
  }
}

// Scratch of tile_stats: column sums per 16-voxel warp row, group means, the tile's weight.
template <int C>
struct TileStats {
  float part[4][C];
  float gmean[GMAX];
  float wpart[4];
};

// Depth-weighted statistics of one tile of C channels (the thread's accumulators acc, weights wr of its 4 voxels, zero
// past the cube) merged into the thread's group acc_g (thread 32 g holds group g). Two passes within the tile, fixed
// order; 4 barriers.
template <int C>
__device__ __forceinline__ void tile_stats(const float (&acc)[C / 16][4], const float (&wr)[4], int cpg, int groups,
                                           TileStats<C>& st, ShiftAcc& acc_g) {
  using Cl = Cols<C, 1>;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tx = tile_tx();
  auto columns = [&](auto value) {
#pragma unroll
    for (int j = 0; j < Cl::NC; ++j) {
      float s = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) s += value(j, e);
      s += __shfl_xor_sync(0xffffffffu, s, 8);
      s += __shfl_xor_sync(0xffffffffu, s, 16);
      if (lane < 8) st.part[warp >> 1][Cl::col(tx, j)] = s;
    }
  };
  auto group_sum = [&]() {   // warp g: the sum over group g's columns and the four warp rows
    float s = 0.f;
    for (int i = lane; i < 4 * cpg; i += 32) s += st.part[i / cpg][warp * cpg + i % cpg];
#pragma unroll
    for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    return s;
  };
  float sw = wr[0] + wr[1] + wr[2] + wr[3];
  sw += __shfl_xor_sync(0xffffffffu, sw, 8);
  sw += __shfl_xor_sync(0xffffffffu, sw, 16);
  if (lane == 0 && !(warp & 1)) st.wpart[warp >> 1] = sw;
  columns([&](int j, int e) { return wr[e] * acc[j][e]; });
  __syncthreads();
  const float wsum = (st.wpart[0] + st.wpart[1]) + (st.wpart[2] + st.wpart[3]);
  const float wt = wsum * cpg;
  if (warp < groups) {
    const float s = group_sum();
    if (lane == 0) st.gmean[warp] = wt > 0.f ? s / wt : 0.f;
  }
  __syncthreads();
  columns([&](int j, int e) {
    const float d = acc[j][e] - st.gmean[Cl::col(tx, j) / cpg];
    return wr[e] * d * d;
  });
  __syncthreads();
  if (warp < groups) {
    const float s = group_sum();
    if (lane == 0) acc_g.add(wt, st.gmean[warp], s);
  }
  __syncthreads();
}

// Partials row of this CTA, from thread 32 g's accumulators of group g; the rows past the grid (nparts is the most CTAs
// any of these kernels runs) hold no weight.
__device__ __forceinline__ void write_tile_partial(double* partials, int nparts, int groups, const ShiftAcc& acc_g) {
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  if (lane == 0 && g < groups) {
    const GroupAcc a = acc_g.get();
    double* p = partials + ((long)blockIdx.x * groups + g) * 3;
    p[0] = a.w;
    p[1] = a.mean;
    p[2] = a.m2;
    for (long r = blockIdx.x + gridDim.x; r < nparts; r += gridDim.x) {
      p = partials + (r * groups + g) * 3;
      p[0] = p[1] = p[2] = 0.0;
    }
  }
}

}  // namespace g32
}  // namespace ffno
