// Learned warm start: per-vertex features, the MLP that predicts each step's
// correction from the inertia guess, and the kernels that train it.
//
// Model (per solved vertex): 22 inputs -> 64 (SiLU) -> 64 (SiLU) -> 3.
// The output is the converged-minus-inertia displacement of the step divided
// by h s, with h the vertex's length scale and s the RMS of its
// displacement-type features (below): dividing by s makes the regression
// scale-free, so a network trained on large motions is equally accurate,
// relatively, on small ones.  Parameters (fp32, this order):
//   W1[64][22] b1[64] W2[64][64] b2[64] W3[3][64] b3[3]
// The network acts on normalised inputs and predicts normalised targets;
// inference (vbd_ws_tc.cu, tensor cores) applies the fp32 normalisation (mean
// and 1/std of every input, std and mean of every target) around bf16
// weights and activations with fp32 accumulation.  Training is fp32.
//
// Displacement-type features, divided by h and then by s = RMS of the 18:
//   0-2   inertia displacement of the coming step, v dt + g dt^2
//   3-5   previous-step displacement, v dt
//   6-8   1-ring mean of the neighbours' previous-step displacement minus the
//         vertex's own (neighbours counted once per incident tet)
//   9-11  1-ring mean of the neighbours' displacement from rest minus the
//         vertex's own (a discrete Laplacian of the displacement)
//   12-14 previous step's correction u - ut_prev (0 without history)
//   15-17 g dt^2
// Scale-free features:
//   18    log10(E dt^2 / (rho h^2)), the stiffness-to-inertia ratio
//   19    Poisson's ratio
//   20    valence / 20
//   21    log10(s)
// Row layout: 24 floats per vertex, 22 = s, 23 = 1 for a solved vertex.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "vbd_device.cuh"
#include "vbd_internal.h"
#include "vbd_warmstart.h"

namespace vbd {

__device__ __forceinline__ float silu(float a) { return a / (1.0f + expf(-a)); }

// ---------------------------------------------------------------------------
// Features: one warp per chunk, TPV lanes per vertex walk its slots.  The
// neighbour sums read a packed fp32 copy of every vertex's displacement and
// velocity (24 B instead of two 32 B double4 per neighbour visit, written
// once per step by ws_pack_kernel); the vertex's own values stay in the
// state precision.  fp32 differences of neighbouring displacements are far
// more accurate than the bf16 the network's inputs are rounded to.
// ---------------------------------------------------------------------------
template <typename SReal>
__global__ void ws_pack_kernel(DevMesh m, float4* __restrict__ pa, float2* __restrict__ pb) {
  using S4 = real4<SReal>;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m.n_vertices) return;
  const S4 u = reinterpret_cast<const S4*>(m.u)[i];
  const S4 v = reinterpret_cast<const S4*>(m.vel)[i];
  pa[i] = make_float4(float(u.x), float(u.y), float(u.z), float(v.x));
  pb[i] = make_float2(float(v.y), float(v.z));
}

template <typename SReal, int TPV, int FMT>
__global__ void __launch_bounds__(256) ws_features_kernel(DevMesh m, int n_chunks, float dt,
                                                          float gx, float gy, float gz,
                                                          float log_dt2, int history,
                                                          const float4* __restrict__ pa,
                                                          const float2* __restrict__ pb,
                                                          float* __restrict__ feat) {
  using S4 = real4<SReal>;
  const int lane = threadIdx.x & 31;
  const int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (q >= n_chunks) return;  // whole warp
  const int2 own = m.chunk_owner[q];
  const ColorInfo ci = m.color[own.x];
  const int vbase = m.env[own.y].vbase;
  constexpr int CPW = 32 / TPV;
  const int vi = lane / TPV, sub = lane % TPV;
  const int gv = ci.vbegin + (q - ci.chunk_begin) * CPW + vi;
  const bool valid = gv < ci.vend;
  const S4* U = reinterpret_cast<const S4*>(m.u);
  const S4* VEL = reinterpret_cast<const S4*>(m.vel);
  const ChunkInfo ch = m.chunk[q];
  // the chunk's slot indices up to the prefetch depth first, as the sweep does
  using RS = RawSlot<FMT>;
  constexpr int PF = Prefetch<TPV>::steps;
  const size_t base = (size_t)ch.block * 32 + lane;
  typename RS::type sl[PF];
#pragma unroll
  for (int s = 0; s < PF; ++s)
    if (s < ch.steps) sl[s] = RS::load(m, base + (size_t)s * 32);
  int k = 0;
  S4 uo, vo;
  uo.x = uo.y = uo.z = uo.w = SReal(0);
  vo = uo;
  if (valid) {
    k = m.valence[gv];
    uo = U[gv];
    vo = VEL[gv];
  }
  float su[3] = {0.f, 0.f, 0.f}, sv[3] = {0.f, 0.f, 0.f};
  const float ux = float(uo.x), uy = float(uo.y), uz = float(uo.z);
  const float vx = float(vo.x), vy = float(vo.y), vz = float(vo.z);
  auto visit = [&](const int4& id) {
    const int nb[3] = {id.x, id.y, id.z};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const float4 a = __ldg(pa + vbase + nb[j]);
      const float2 b = __ldg(pb + vbase + nb[j]);
      su[0] += a.x - ux;
      su[1] += a.y - uy;
      su[2] += a.z - uz;
      sv[0] += a.w - vx;
      sv[1] += b.x - vy;
      sv[2] += b.y - vz;
    }
  };
#pragma unroll
  for (int s = 0; s < PF; ++s)
    if (s < ch.steps && s * TPV + sub < k) visit(RS::unpack(sl[s]));
  for (int s = PF; s < ch.steps; ++s)
    if (s * TPV + sub < k) visit(load_slot<FMT>(m, base + (size_t)s * 32));
#pragma unroll
  for (int off = TPV / 2; off > 0; off >>= 1) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      su[i] += __shfl_xor_sync(0xffffffffu, su[i], off);
      sv[i] += __shfl_xor_sync(0xffffffffu, sv[i], off);
    }
  }
  if (!valid) return;
  // every lane of the vertex holds the sums now; each computes the row and
  // stores its share of the six 16-byte pieces
  const float4 ws = m.wstat[gv];
  const float ih = 1.0f / ws.x;
  const float icnt = 1.0f / float(3 * k);
  const S4 tp = reinterpret_cast<const S4*>(m.ut)[gv];  // the previous step's inertia target
  const float dt2 = dt * dt;
  const float g2[3] = {gx * dt2, gy * dt2, gz * dt2};
  const float v[3] = {vx, vy, vz};
  // the correction u - ut_prev is a difference of nearby values: take it in
  // the state precision before rounding
  const float up[3] = {float(uo.x - tp.x), float(uo.y - tp.y), float(uo.z - tp.z)};
  float r[kWsRow];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    r[i] = (v[i] * dt + g2[i]) * ih;
    r[3 + i] = v[i] * dt * ih;
    r[6 + i] = sv[i] * icnt * dt * ih;
    r[9 + i] = su[i] * icnt * ih;
    r[12 + i] = history ? up[i] * ih : 0.0f;
    r[15 + i] = g2[i] * ih;
  }
  float ss = 0.0f;
#pragma unroll
  for (int i = 0; i < 18; ++i) ss += r[i] * r[i];
  const float sc = sqrtf(ss * (1.0f / 18.0f)) + 1e-30f;
  const float isc = 1.0f / sc;
#pragma unroll
  for (int i = 0; i < 18; ++i) r[i] *= isc;
  r[18] = ws.y + log_dt2;
  r[19] = ws.z;
  r[20] = ws.w;
  r[21] = log10f(sc);
  r[22] = sc;
  r[23] = 1.0f;
  float4* f = reinterpret_cast<float4*>(feat + (size_t)gv * kWsRow);
#pragma unroll
  for (int j = 0; j < kWsRow / 4; ++j)
    if (j % TPV == sub) f[j] = make_float4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
}

// Training target after a step: (u - ut) / (h s) for solved vertices.
template <typename SReal>
__global__ void ws_targets_kernel(DevMesh m, const float* __restrict__ feat,
                                  float* __restrict__ target) {
  using S4 = real4<SReal>;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m.n_vertices) return;
  const S4 u = reinterpret_cast<const S4*>(m.u)[i];
  const S4 t = reinterpret_cast<const S4*>(m.ut)[i];
  const bool solved = feat[(size_t)i * kWsRow + 23] > 0.0f;
  const double ih = solved ? 1.0 / (double(m.wstat[i].x) * feat[(size_t)i * kWsRow + 22]) : 0.0;
  target[3 * (size_t)i] = solved ? float(double(u.x - t.x) * ih) : 0.0f;
  target[3 * (size_t)i + 1] = solved ? float(double(u.y - t.y) * ih) : 0.0f;
  target[3 * (size_t)i + 2] = solved ? float(double(u.z - t.z) * ih) : 0.0f;
}

// ---------------------------------------------------------------------------
// Forward pass (fp32), for evaluation: X [n][24] -> out [n][3].
//
// A block of 128 threads takes tiles of 16 x SPT samples and forms both hidden
// layers as register-tiled products: thread (ty, tx) holds SPT samples x 8 units
// (tx * 4 + 0..3 and 32 + tx * 4 + 0..3: eight threads then read consecutive
// 16-byte pieces of a weight row), two samples to a packed fp32x2 fused
// multiply-add.  Activations stay in shared memory, sample index fastest; the
// third layer is summed over the eight threads of a sample by shuffles.  What
// bounds it is the fp32 pipe (5,824 multiply-adds a sample) and the two SiLU
// layers' exponentials; with one thread per sample every four multiply-adds took
// a shared-memory load of weights.  262,147 samples on B200: 172 -> 107 us (16 samples
// a thread: 170, two blocks per SM do not hide the latencies; IEEE instead of
// approximate division in SiLU: 127, with the error against 64 bits 2.0e-7 instead of
// 2.1e-7 of the result, and 2.4e-7 before).
// ---------------------------------------------------------------------------
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

constexpr int kFwdThreads = 128;
// shared-memory map (floats): W1^T [22][64], W2^T [64][64], b1, b2, W3, b3, then the
// tile's activations [64][16 SPT], the 16-byte pieces of row r exchanged by
// (r / 4) % 8 (fw_at): eight threads that store four rows each then hit different
// banks, as do the eight that load a row.
constexpr int kFwW1T = 0;
constexpr int kFwW2T = kFwW1T + kWsIn * kWsHidden;
constexpr int kFwB1 = kFwW2T + kWsHidden * kWsHidden;
constexpr int kFwB2 = kFwB1 + kWsHidden;
constexpr int kFwW3 = kFwB2 + kWsHidden;
constexpr int kFwB3 = kFwW3 + kWsOut * kWsHidden;
constexpr int kFwAct = (kFwB3 + kWsOut + 3) / 4 * 4;
template <int SPT>
constexpr size_t kFwSmem = sizeof(float) * (kFwAct + kWsHidden * 16 * SPT);
template <int SPT>
__device__ __forceinline__ int fw_at(int row, int s) {
  return row * 16 * SPT + (s ^ ((row >> 2 & 7) << 2));
}

template <int SPT>
__global__ void __launch_bounds__(kFwdThreads, 4) mlp_forward_kernel(const float* __restrict__ X,
                                                                  int n,
                                                                  const float* __restrict__ P,
                                                                  float* __restrict__ out) {
  extern __shared__ __align__(16) float fw[];
  constexpr int TILE = 16 * SPT, SP = SPT / 2;
  const int t = threadIdx.x, tx = t & 7, ty = t >> 3;
  // all of a thread's weights in flight at once: 1 to 2 us of a launch
#pragma unroll
  for (int i = t; i < kWsIn * kWsHidden; i += kFwdThreads)
    fw[kFwW1T + i] = P[kWsW1 + i % kWsHidden * kWsIn + i / kWsHidden];
#pragma unroll 16
  for (int i = t; i < kWsHidden * kWsHidden; i += kFwdThreads)
    fw[kFwW2T + i] = P[kWsW2 + i % kWsHidden * kWsHidden + i / kWsHidden];
  for (int i = t; i < kWsHidden; i += kFwdThreads) {
    fw[kFwB1 + i] = P[kWsB1 + i];
    fw[kFwB2 + i] = P[kWsB2 + i];
  }
  for (int i = t; i < kWsOut * kWsHidden; i += kFwdThreads) fw[kFwW3 + i] = P[kWsW3 + i];
  if (t < kWsOut) fw[kFwB3 + t] = P[kWsB3 + t];
  float* act = fw + kFwAct;
  const bool aligned = (reinterpret_cast<size_t>(X) & 15) == 0;
  const int tiles = (n + TILE - 1) / TILE;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int s0 = tile * TILE;
    __syncthreads();  // the weights are in place; the previous tile's activations are used up
    for (int i = t; i < TILE * (kWsRow / 4); i += kFwdThreads) {
      const int s = i % TILE, q = i / TILE;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (s0 + s < n) {
        const float* x = X + (size_t)(s0 + s) * kWsRow + 4 * q;
        v = aligned ? __ldg(reinterpret_cast<const float4*>(x)) : make_float4(x[0], x[1], x[2], x[3]);
      }
      act[fw_at<SPT>(4 * q, s)] = v.x;
      act[fw_at<SPT>(4 * q + 1, s)] = v.y;
      act[fw_at<SPT>(4 * q + 2, s)] = v.z;
      act[fw_at<SPT>(4 * q + 3, s)] = v.w;
    }
    __syncthreads();
    f32x2 acc[SP][8];
    auto layer = [&](const float* W, const float* bias, int K) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float b = bias[(j >> 2) * 32 + tx * 4 + (j & 3)];
#pragma unroll
        for (int p = 0; p < SP; ++p) acc[p][j] = pack2(b, b);
      }
#pragma unroll 2
      for (int k = 0; k < K; ++k) {
        const float4 w0 = *reinterpret_cast<const float4*>(W + k * kWsHidden + tx * 4);
        const float4 w1 = *reinterpret_cast<const float4*>(W + k * kWsHidden + 32 + tx * 4);
        const f32x2 w[8] = {pack2(w0.x, w0.x), pack2(w0.y, w0.y), pack2(w0.z, w0.z),
                            pack2(w0.w, w0.w), pack2(w1.x, w1.x), pack2(w1.y, w1.y),
                            pack2(w1.z, w1.z), pack2(w1.w, w1.w)};
#pragma unroll
        for (int p = 0; p < SP; p += 2) {
          const ulonglong2 a =
              *reinterpret_cast<const ulonglong2*>(act + fw_at<SPT>(k, ty * SPT + 2 * p));
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            acc[p][j] = fma2(a.x, w[j], acc[p][j]);
            acc[p + 1][j] = fma2(a.y, w[j], acc[p + 1][j]);
          }
        }
      }
#pragma unroll
      for (int p = 0; p < SP; ++p)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 v = unpack2(acc[p][j]);
          acc[p][j] = pack2(__fdividef(v.x, 1.0f + expf(-v.x)), __fdividef(v.y, 1.0f + expf(-v.y)));
        }
    };
    layer(fw + kFwW1T, fw + kFwB1, kWsIn);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int p = 0; p < SP; ++p)
        *reinterpret_cast<f32x2*>(
            act + fw_at<SPT>((j >> 2) * 32 + tx * 4 + (j & 3), ty * SPT + 2 * p)) = acc[p][j];
    __syncthreads();
    layer(fw + kFwW2T, fw + kFwB2, kWsHidden);
#pragma unroll
    for (int k = 0; k < kWsOut; ++k) {
      float w[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        w[j] = fw[kFwW3 + k * kWsHidden + (j >> 2) * 32 + tx * 4 + (j & 3)];
#pragma unroll
      for (int p = 0; p < SP; ++p) {
        float2 o = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 v = unpack2(acc[p][j]);
          o.x += w[j] * v.x;
          o.y += w[j] * v.y;
        }
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) {
          o.x += __shfl_xor_sync(0xffffffffu, o.x, off);
          o.y += __shfl_xor_sync(0xffffffffu, o.y, off);
        }
        const int s = s0 + ty * SPT + 2 * p;
        if (tx == p % 8) {  // spread the stores over the eight threads
          if (s < n) out[(size_t)s * kWsOut + k] = o.x + fw[kFwB3 + k];
          if (s + 1 < n) out[(size_t)(s + 1) * kWsOut + k] = o.y + fw[kFwB3 + k];
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Training step, fused per tile of kTrainTile samples (one block): forward
// with the activations kept in shared memory, the loss gradient, backward to
// the pre-activation deltas, and the tile's partial weight gradients -- each
// parameter's sum over the tile's samples, in sample order.  A second kernel adds
// the tiles' partials in tile order, so the gradient is the same on every run (no
// atomics).
//
// All matrices lie sample-fastest in shared memory.  The hidden layers and the
// layer-1 deltas are register-tiled products of 4 units x 2 samples a thread,
// the weight gradients of 4 x 4 (layer 2) and 2 x 3 (layer 1) parameters a
// thread, four samples to a 16-byte load: with one result a thread every
// multiply-add loaded both operands from shared memory, half a million of them per
// tile.  Every sum keeps its order, so loss, gradient and parameters have the bits
// they had.  A 4,096-row minibatch (gradient and Adam) on B200: 54 -> 39 us with the
// torch calls around it (tile kernel 35 -> 20); the launches are half of what is left.
// ---------------------------------------------------------------------------
constexpr int kTrainTile = 32;
constexpr int kTrainThreads = 256;
constexpr int kTrainPartial = kWsParams + 1;  // + the tile's sum of squared errors
constexpr int kTsPitch = kTrainTile + 4;
// shared-memory map (floats)
constexpr int kTsW1T = 0;                                 // W1^T [22][64]
constexpr int kTsW2T = kTsW1T + kWsIn * kWsHidden;        // W2^T [64][64]
constexpr int kTsW2 = kTsW2T + kWsHidden * kWsHidden;     // W2 [64][64]
constexpr int kTsB1 = kTsW2 + kWsHidden * kWsHidden;
constexpr int kTsB2 = kTsB1 + kWsHidden;
constexpr int kTsW3 = kTsB2 + kWsHidden;                  // W3 [3][64]
constexpr int kTsX = kTsW3 + kWsOut * kWsHidden;          // X^T [24][tile], rows 22, 23 zero
constexpr int kTsS1 = kTsX + 24 * kTsPitch;               // silu(A1) [64][tile]
constexpr int kTsG1 = kTsS1 + kWsHidden * kTsPitch;       // silu'(A1)
constexpr int kTsS2 = kTsG1 + kWsHidden * kTsPitch;       // silu(A2)
constexpr int kTsG2 = kTsS2 + kWsHidden * kTsPitch;       // silu'(A2)
constexpr int kTsD1 = kTsG2 + kWsHidden * kTsPitch;       // dL/dA1
constexpr int kTsD2 = kTsD1 + kWsHidden * kTsPitch;       // dL/dA2
constexpr int kTsOut = kTsD2 + kWsHidden * kTsPitch;      // dL/dout [3][tile]
constexpr int kTsSse = kTsOut + kWsOut * kTsPitch;        // per-warp squared errors
constexpr int kTsB3 = kTsSse + kTrainThreads / 32;
constexpr int kTsY = kTsB3 + 4;                           // targets [tile][3]
constexpr int kTsFloats = kTsY + kTrainTile * kWsOut;
constexpr size_t kTrainSmem = sizeof(float) * kTsFloats;
static_assert(kTsX % 4 == 0 && kTsPitch % 4 == 0, "16-byte rows");

// 4 units x 2 samples of W^T a (W^T: [K][64], a: [K][tile]), added to acc.
__device__ __forceinline__ void train_product(const float* WT, const float* a, int K, int tx,
                                              int ty, f32x2 (&acc)[4]) {
#pragma unroll 8
  for (int k = 0; k < K; ++k) {
    const float4 w = *reinterpret_cast<const float4*>(WT + k * kWsHidden + 4 * tx);
    const f32x2 v = *reinterpret_cast<const f32x2*>(a + k * kTsPitch + 2 * ty);
    acc[0] = fma2(v, pack2(w.x, w.x), acc[0]);
    acc[1] = fma2(v, pack2(w.y, w.y), acc[1]);
    acc[2] = fma2(v, pack2(w.z, w.z), acc[2]);
    acc[3] = fma2(v, pack2(w.w, w.w), acc[3]);
  }
}

// Sums over the tile's samples, in order, of A[row][s] B[col][s] for NA x NB rows.
template <int NA, int NB>
__device__ __forceinline__ void train_gradient(const float* A, int sa, const float* B, int sb,
                                               float (&r)[NA][NB]) {
#pragma unroll
  for (int i = 0; i < NA; ++i)
#pragma unroll
    for (int j = 0; j < NB; ++j) r[i][j] = 0.0f;
#pragma unroll 2
  for (int s = 0; s < kTrainTile; s += 4) {
    float4 a[NA], b[NB];
#pragma unroll
    for (int i = 0; i < NA; ++i) a[i] = *reinterpret_cast<const float4*>(A + i * sa * kTsPitch + s);
#pragma unroll
    for (int j = 0; j < NB; ++j) b[j] = *reinterpret_cast<const float4*>(B + j * sb * kTsPitch + s);
#pragma unroll
    for (int i = 0; i < NA; ++i)
#pragma unroll
      for (int j = 0; j < NB; ++j)
        r[i][j] = fmaf(a[i].w, b[j].w,
                       fmaf(a[i].z, b[j].z, fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, r[i][j]))));
  }
}

__global__ void __launch_bounds__(kTrainThreads) mlp_train_tile_kernel(
    const float* __restrict__ X, const float* __restrict__ Y, const int* __restrict__ idx,
    int batch, const float* __restrict__ P, float* __restrict__ out) {
  extern __shared__ __align__(16) float ts[];
  cudaTriggerProgrammaticLaunchCompletion();  // the reduction's blocks may take their places
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int s0 = blockIdx.x * kTrainTile;
  const int ns = min(kTrainTile, batch - s0);
  for (int i = t; i < kTrainTile * 24; i += kTrainThreads) {
    const int s = i / 24, k = i % 24;
    float v = 0.0f;
    if (s < ns && k < kWsIn) {
      const int r = idx ? idx[s0 + s] : s0 + s;
      v = X[(size_t)r * kWsRow + k];
    }
    ts[kTsX + k * kTsPitch + s] = v;
  }
  // consecutive threads write consecutive words of the transposes (their strided
  // reads of the parameters hit L1)
#pragma unroll
  for (int i = t; i < kWsHidden * kWsIn; i += kTrainThreads)
    ts[kTsW1T + i] = P[kWsW1 + i % kWsHidden * kWsIn + i / kWsHidden];
#pragma unroll 8
  for (int i = t; i < kWsHidden * kWsHidden; i += kTrainThreads) ts[kTsW2 + i] = P[kWsW2 + i];
#pragma unroll 8
  for (int i = t; i < kWsHidden * kWsHidden; i += kTrainThreads)
    ts[kTsW2T + i] = P[kWsW2 + i % kWsHidden * kWsHidden + i / kWsHidden];
  if (t < kWsHidden) {
    ts[kTsB1 + t] = P[kWsB1 + t];
    ts[kTsB2 + t] = P[kWsB2 + t];
  }
  if (t < kWsOut * kWsHidden) ts[kTsW3 + t] = P[kWsW3 + t];
  if (t < kWsOut) ts[kTsB3 + t] = P[kWsB3 + t];
  if (t < kTrainTile * kWsOut && t / kWsOut < ns) {
    const int r = idx ? idx[s0 + t / kWsOut] : s0 + t / kWsOut;
    ts[kTsY + t] = Y[(size_t)r * kWsOut + t % kWsOut];
  }
  __syncthreads();
  // 4 units (4 tx ..) x 2 samples (2 ty ..) a thread
  const int tx = t & 15, ty = t >> 4;
  auto hidden = [&](const float* WT, const float* bias, const float* a, int K, float* S,
                    float* G) {
    f32x2 acc[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] = pack2(bias[4 * tx + j], bias[4 * tx + j]);
    train_product(WT, a, K, tx, ty, acc);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 v = unpack2(acc[j]);
      const float e0 = 1.0f + expf(-v.x), e1 = 1.0f + expf(-v.y);
      const float g0 = 1.0f / e0, g1 = 1.0f / e1;
      const int at = (4 * tx + j) * kTsPitch + 2 * ty;
      *reinterpret_cast<float2*>(S + at) = make_float2(v.x / e0, v.y / e1);
      *reinterpret_cast<float2*>(G + at) =
          make_float2(g0 * (1.0f + v.x * (1.0f - g0)), g1 * (1.0f + v.y * (1.0f - g1)));
    }
  };
  hidden(ts + kTsW1T, ts + kTsB1, ts + kTsX, kWsIn, ts + kTsS1, ts + kTsG1);
  __syncthreads();
  hidden(ts + kTsW2T, ts + kTsB2, ts + kTsS1, kWsHidden, ts + kTsS2, ts + kTsG2);
  __syncthreads();
  // layer 3 and the loss gradient: one warp per (sample, output), two hidden
  // units per lane and a shuffle reduction
  float sse = 0.0f;
#pragma unroll 4
  for (int o = warp; o < kTrainTile * kWsOut; o += kTrainThreads / 32) {
    const int s = o / kWsOut, k = o % kWsOut;
    float a = fmaf(ts[kTsW3 + k * kWsHidden + lane], ts[kTsS2 + lane * kTsPitch + s],
                   ts[kTsW3 + k * kWsHidden + lane + 32] * ts[kTsS2 + (lane + 32) * kTsPitch + s]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
    float g = 0.0f;
    if (s < ns) {
      const float d = a + ts[kTsB3 + k] - ts[kTsY + o];
      g = 2.0f * d / (kWsOut * batch);
      sse = fmaf(d, d, sse);
    }
    if (lane == 0) ts[kTsOut + k * kTsPitch + s] = g;
  }
  if (lane == 0) ts[kTsSse + warp] = sse;
  __syncthreads();
  // backward: layer-2 deltas, then layer-1 deltas
  {
    const float2 o0 = *reinterpret_cast<const float2*>(ts + kTsOut + 2 * ty);
    const float2 o1 = *reinterpret_cast<const float2*>(ts + kTsOut + kTsPitch + 2 * ty);
    const float2 o2 = *reinterpret_cast<const float2*>(ts + kTsOut + 2 * kTsPitch + 2 * ty);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int u = 4 * tx + j, at = u * kTsPitch + 2 * ty;
      const float w0 = ts[kTsW3 + u], w1 = ts[kTsW3 + kWsHidden + u],
                  w2 = ts[kTsW3 + 2 * kWsHidden + u];
      const float2 g = *reinterpret_cast<const float2*>(ts + kTsG2 + at);
      *reinterpret_cast<float2*>(ts + kTsD2 + at) =
          make_float2(fmaf(w2, o2.x, fmaf(w1, o1.x, w0 * o0.x)) * g.x,
                      fmaf(w2, o2.y, fmaf(w1, o1.y, w0 * o0.y)) * g.y);
    }
  }
  __syncthreads();
  {
    f32x2 acc[4] = {0ull, 0ull, 0ull, 0ull};
    train_product(ts + kTsW2, ts + kTsD2, kWsHidden, tx, ty, acc);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int at = (4 * tx + j) * kTsPitch + 2 * ty;
      const float2 v = unpack2(acc[j]), g = *reinterpret_cast<const float2*>(ts + kTsG1 + at);
      *reinterpret_cast<float2*>(ts + kTsD1 + at) = make_float2(v.x * g.x, v.y * g.y);
    }
  }
  // the tile's weight gradients (padding samples have zero deltas).  Layer 2
  // and 3 and the output bias need no layer-1 delta.
  float* dst = out + (size_t)blockIdx.x * kTrainPartial;
  {
    // units tx, tx + 16, .. of the row and ty, ty + 16, .. of the column: the
    // 16-byte loads of eight threads then fall into different banks
    float r[4][4];
    train_gradient<4, 4>(ts + kTsD2 + ty * kTsPitch, 16, ts + kTsS1 + tx * kTsPitch, 16, r);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) dst[kWsW2 + (ty + 16 * i) * kWsHidden + tx + 16 * j] = r[i][j];
  }
  auto row_sum = [&](const float* row) {
    float a = 0.0f;
#pragma unroll
    for (int s = 0; s < kTrainTile; s += 4) {
      const float4 v = *reinterpret_cast<const float4*>(row + s);
      a = (((a + v.x) + v.y) + v.z) + v.w;
    }
    return a;
  };
  if (t < kWsOut * kWsHidden) {  // W3[k][j] += dout[k][s] S2[j][s]
    float r[1][1];
    train_gradient<1, 1>(ts + kTsOut + (t / kWsHidden) * kTsPitch, 1,
                         ts + kTsS2 + (t % kWsHidden) * kTsPitch, 1, r);
    dst[kWsW3 + t] = r[0][0];
  } else {  // b2[j]: the last 64 threads
    dst[kWsB2 + t - kWsOut * kWsHidden] = row_sum(ts + kTsD2 + (t - kWsOut * kWsHidden) * kTsPitch);
  }
  __syncthreads();
  {  // W1[j][i] += D1[j][s] X[i][s]: rows u, u + 32 and columns c, c + 8, c + 16
    const int u = t >> 3, c = t & 7;
    float r[2][3];
    train_gradient<2, 3>(ts + kTsD1 + u * kTsPitch, 32, ts + kTsX + c * kTsPitch, 8, r);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (c + 8 * j < kWsIn) dst[kWsW1 + (u + 32 * i) * kWsIn + c + 8 * j] = r[i][j];
  }
  if (t < kWsHidden) dst[kWsB1 + t] = row_sum(ts + kTsD1 + t * kTsPitch);
  if (t >= 64 && t < 64 + kWsOut) dst[kWsB3 + t - 64] = row_sum(ts + kTsOut + (t - 64) * kTsPitch);
  if (t == 128) {
    float v = 0.0f;
    for (int w = 0; w < kTrainThreads / 32; ++w) v += ts[kTsSse + w];
    dst[kWsParams] = v;
  }
}

// Sum of the tiles' partial gradients in tile order (and of their squared
// errors into *loss): a parameter a thread, 32 tiles' partials in flight.
constexpr int kReduceThreads = 64;
__global__ void __launch_bounds__(kReduceThreads)
    mlp_reduce_tiles_kernel(const float* __restrict__ part, int tiles, float* __restrict__ grad,
                            double* __restrict__ loss) {
  const int p = blockIdx.x * kReduceThreads + threadIdx.x;
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();  // every tile's partials are written
  if (p > kWsParams) return;
  if (p == kWsParams) {
    if (loss) {
      double v = 0.0;
#pragma unroll 32
      for (int b = 0; b < tiles; ++b) v += double(part[(size_t)b * kTrainPartial + p]);
      *loss += v;
    }
    return;
  }
  float acc = 0.0f;
#pragma unroll 32
  for (int b = 0; b < tiles; ++b) acc += part[(size_t)b * kTrainPartial + p];
  grad[p] = acc;
}

__global__ void adam_kernel(float* __restrict__ P, const float* __restrict__ G,
                            float* __restrict__ M, float* __restrict__ V, int n, float lr,
                            float beta1, float beta2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  cudaGridDependencySynchronize();  // the gradient is written
  if (i >= n) return;
  const float g = G[i];
  const float m = beta1 * M[i] + (1.0f - beta1) * g;
  const float v = beta2 * V[i] + (1.0f - beta2) * g * g;
  M[i] = m;
  V[i] = v;
  P[i] -= lr * (m / c1) / (sqrtf(v / c2) + eps);
}

__global__ void to_bf16_kernel(const float* __restrict__ P, __nv_bfloat16* __restrict__ out,
                               int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = __float2bfloat16(P[i]);
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
namespace {
struct FeatLaunch {
  const DevMesh& m;
  int n_chunks;
  double dt, gx, gy, gz;
  int history;
  float* pack;
  float* feat;
  cudaStream_t s;
  template <typename Real, typename SReal, int TPV, int MAT, int FMT>
  cudaError_t run() {
    const int blocks = (n_chunks + 7) / 8;
    if (blocks == 0) return cudaSuccess;
    float4* pa = reinterpret_cast<float4*>(pack);
    float2* pb = reinterpret_cast<float2*>(pack + 4 * (size_t)m.n_vertices);
    ws_pack_kernel<SReal><<<(m.n_vertices + 255) / 256, 256, 0, s>>>(m, pa, pb);
    ws_features_kernel<SReal, TPV, FMT><<<blocks, 256, 0, s>>>(
        m, n_chunks, float(dt), float(gx), float(gy), float(gz), float(2.0 * log10(dt)), history,
        pa, pb, feat);
    return cudaGetLastError();
  }
};
inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }
}  // namespace

cudaError_t launch_ws_features(int prec, int tpv, const DevMesh& m, int n_chunks, double dt,
                               const double* g, int history, float* pack, float* feat,
                               cudaStream_t s) {
  FeatLaunch f{m, n_chunks, dt, g[0], g[1], g[2], history, pack, feat, s};
  // the features depend on the state precision only; material is irrelevant
  return dispatch(prec, kSNH, m.fmt, tpv, f);
}

cudaError_t launch_ws_targets(bool state64, const DevMesh& m, const float* feat, float* target,
                              cudaStream_t s) {
  const int n = m.n_vertices;
  if (n <= 0) return cudaSuccess;
  if (state64)
    ws_targets_kernel<double><<<nblk(n, 256), 256, 0, s>>>(m, feat, target);
  else
    ws_targets_kernel<float><<<nblk(n, 256), 256, 0, s>>>(m, feat, target);
  return cudaGetLastError();
}

cudaError_t launch_to_bf16(const float* P, void* out, int n, cudaStream_t s) {
  to_bf16_kernel<<<nblk(n, 256), 256, 0, s>>>(P, static_cast<__nv_bfloat16*>(out), n);
  return cudaGetLastError();
}

// Launches a kernel that waits for the one before it in the stream itself
// (cudaGridDependencySynchronize): its blocks take their places while that one
// still runs, so a launch of a few us does not wait for the launch before it (a
// 4096-row minibatch and its Adam update: 39 -> 37 us on B200).
template <class... P, class... A>
cudaError_t launch_early(void (*kernel)(P...), int blocks, int threads, cudaStream_t s, A... args) {
  cudaLaunchAttribute early{};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.stream = s;
  cfg.attrs = &early;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  return e != cudaSuccess ? e : cudaGetLastError();
}

size_t mlp_train_scratch_floats(int batch) {
  return (size_t)nblk(batch, kTrainTile) * kTrainPartial;
}

cudaError_t launch_mlp_train_batch(const float* X, const float* Y, const int* idx, int batch,
                                   const float* P, float* grad, float* scratch, double* loss,
                                   cudaStream_t s) {
  static bool attr_set = false;  // per process; the attribute is per function
  if (!attr_set) {
    const cudaError_t e = cudaFuncSetAttribute(
        mlp_train_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  const int tiles = nblk(batch, kTrainTile);
  mlp_train_tile_kernel<<<tiles, kTrainThreads, kTrainSmem, s>>>(X, Y, idx, batch, P, scratch);
  return launch_early(mlp_reduce_tiles_kernel, nblk(kTrainPartial, kReduceThreads), kReduceThreads,
                      s, scratch, tiles, grad, loss);
}

namespace {
template <int SPT>
cudaError_t forward_tiles(const float* X, int n, const float* P, float* out, int sms,
                          cudaStream_t s) {
  // the attributes are per device; each thread sets them for itself
  static thread_local int configured_device = -1, per_sm = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured_device != dev) {
    cudaError_t e = cudaFuncSetAttribute(mlp_forward_kernel<SPT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kFwSmem<SPT>);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mlp_forward_kernel<SPT>,
                                                        kFwdThreads, kFwSmem<SPT>);
    if (e != cudaSuccess) return e;
    configured_device = dev;
  }
  const int blocks = std::min(nblk(n, 16 * SPT), std::max(1, per_sm * sms));
  mlp_forward_kernel<SPT><<<blocks, kFwdThreads, kFwSmem<SPT>, s>>>(X, n, P, out);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_mlp_forward(const float* X, int n, const float* P, float* out,
                               cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  static thread_local int known_device = -1, sms = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (known_device != dev) {
    const cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    known_device = dev;
  }
  // 128-sample tiles reuse the weights more; below one wave of them (two a SM), 64-sample
  // tiles fill the device better
  return n >= sms * 2 * 128 ? forward_tiles<8>(X, n, P, out, sms, s)
                            : forward_tiles<4>(X, n, P, out, sms, s);
}

cudaError_t launch_adam(float* P, const float* G, float* M, float* V, int n, float lr,
                        float beta1, float beta2, float eps, int t, cudaStream_t s) {
  const float c1 = 1.0f - powf(beta1, (float)t), c2 = 1.0f - powf(beta2, (float)t);
  return launch_early(adam_kernel, nblk(n, 256), 256, s, P, G, M, V, n, lr, beta1, beta2, eps, c1,
                      c2);
}

}  // namespace vbd
