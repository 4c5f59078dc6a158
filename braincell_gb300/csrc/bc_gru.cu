// Training kernels of the subtree-surrogate GRU: forward over a window of a
// batch of sequences (storing the activations), backward through time with the
// weight gradients accumulated in the same pass, Adam, and the BF16 packing of
// the recurrent weights.  One CTA owns an M tile of 16 sequences for the whole
// window; warp w owns hidden units [8w, 8w + 8) in the elementwise parts.
//
// Loss: mean over the window's (sequence, step) entries of (y - y_target)^2.
// Truncated BPTT: the hidden state is carried from window to window, the
// gradient is not.
#include <cuda_runtime.h>

#include <cmath>

#include "../../include/braincell_gb300.h"
#include "bc_gru.cuh"
#include "bc_internal.h"

namespace bc {
namespace {

constexpr int kRows = 16;      // sequences per CTA
constexpr int kWarps = 8;      // kGruH / 8
constexpr int kThreads = kWarps * 32;
constexpr int kGPad = kGru3H + 8;       // bf16 row stride of dG [row][n]
constexpr int kRPad = kRows + 8;        // bf16 row stride of dG^T [n][row] and h^T [k][row]
constexpr int kDPad = kGruH + 4;        // fp32 row stride of dh [row][k]
// Row stride (floats) of the per-CTA gradient rows of the backward: kGruNParam
// rounded up to a multiple of 4, so that every row starts on a 16-byte boundary
// (the recurrent block is stored as float2 pairs).
constexpr int kPartialStride = (kGruNParam + 3) & ~3;

struct FwdArgs {
  const float* params;
  const uint32_t* wext;
  const float* x;
  const float* y;
  int64_t t_total;
  const int32_t* seq;
  int32_t batch;
  int64_t t0;
  int32_t T;
  float* h;
  float* acts;  // [5][batch][T][H] or null
  float* yout;  // [batch][T] or null
  double* loss;
  bool vec;     // x on a 16-byte, h and acts on an 8-byte boundary
};

struct BwdArgs {
  const float* params;
  const uint32_t* wht;
  const float* x;
  const float* y;
  int64_t t_total;
  const int32_t* seq;
  int32_t batch;
  int64_t t0;
  int32_t T;
  const float* acts;
  const float* yout;
  float gscale;
  float* partial;  // [gridDim.x][kPartialStride]: this CTA's gradient, every entry written
  bool vec;        // x on a 16-byte, acts on an 8-byte boundary
};

__device__ __forceinline__ size_t act_index(int k, int batch, int T, int b, int t, int j) {
  return ((size_t(k) * batch + b) * T + t) * kGruH + j;
}

// Inputs and targets come through shared memory, kChunk steps at a time, the next
// chunk's copies (cp.async) in flight while a chunk runs.
constexpr int kChunk = 32;
constexpr int kHBf = kGruH + 8;  // bf16 row stride of the hidden tile (conflict-free ldmatrix)

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
template <int kBytes>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
  if constexpr (kBytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst)), "l"(src), "n"(kBytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kLeft>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(kLeft) : "memory");
}

// Two floats at p, which is 8-byte aligned when vec.
__device__ __forceinline__ float2 load2(const float* p, bool vec) {
  return vec ? *reinterpret_cast<const float2*>(p) : make_float2(p[0], p[1]);
}
__device__ __forceinline__ void store2(float* p, float x, float y, bool vec) {
  if (vec) {
    *reinterpret_cast<float2*>(p) = make_float2(x, y);
  } else {
    p[0] = x;
    p[1] = y;
  }
}

struct StepInputs {
  float4 x[2][kChunk][kRows];
  float y[2][kChunk][kRows];
};

// Starts the copies of steps [t, t + kChunk) (those inside [0, T)) into buffer `buf`.
__device__ __forceinline__ void stage_inputs(StepInputs& in, int buf, const float* x, const float* y, bool vec,
                                             int64_t t_total, const int32_t* seq, int batch, int b_base, int64_t t0, int t,
                                             int T) {
  for (int i = threadIdx.x; i < kChunk * kRows; i += kThreads) {
    const int r = i / kChunk, k = i % kChunk;  // consecutive threads: consecutive steps of a row
    if (b_base + r >= batch || t + k < 0 || t + k >= T) continue;
    const int64_t at = int64_t(seq[b_base + r]) * t_total + t0 + t + k;
    if (vec) {
      cp_async<16>(&in.x[buf][k][r], x + at * kGruX);
    } else {
      for (int c = 0; c < kGruX; ++c) cp_async<4>(reinterpret_cast<float*>(&in.x[buf][k][r]) + c, x + at * kGruX + c);
    }
    if (y) cp_async<4>(&in.y[buf][k][r], y + at);
  }
  cp_async_commit();
}

// The step is a chain (product, gates, exchange of h through shared memory), so its time
// is latency.  A warp keeps its 32 B-fragment words in registers for the whole window
// and each thread its own four h in FP32; only the BF16 tile is exchanged, read with
// ldmatrix.  With the weights re-read every step, h re-rounded by every warp and the
// inputs and targets loaded where they are used, a step of 16 sequences took 2.0 us, now
// 1.07.
__global__ void __launch_bounds__(kThreads) gru_fwd_kernel(FwdArgs a) {
  __shared__ __align__(16) __nv_bfloat16 hs[2][kRows][kHBf];
  __shared__ float ypart[2][kWarps][kRows];
  __shared__ __align__(16) StepInputs in;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int g = lane >> 2, tq = lane & 3;
  const int b_base = blockIdx.x * kRows;
  const float bo = a.params[kGruOffBo];
  const int j0 = 8 * w + 2 * tq;
  const float wo[2] = {a.params[kGruOffWo + j0], a.params[kGruOffWo + j0 + 1]};

  for (int buf = 0; buf < 2; ++buf)  // rows without a sequence and steps past the window read 0
    for (int i = threadIdx.x; i < kChunk * kRows; i += kThreads) {
      (&in.x[buf][0][0])[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      (&in.y[buf][0][0])[i] = 0.f;
    }
  __syncthreads();
  stage_inputs(in, 0, a.x, a.y, a.vec, a.t_total, a.seq, a.batch, b_base, a.t0, 0, a.T);

  // B fragments of this warp's units: blocks r, z, hn (5 k steps), nx (the x step)
  uint32_t wb[kGruFragSlots][2];
#pragma unroll
  for (int slot = 0; slot < kGruFragSlots; ++slot) {
    const int q = slot < 15 ? slot / 5 : 3, kk = slot < 15 ? slot % 5 : 4;
    const uint32_t* p = a.wext + size_t(q * kGruH + w * 8 + g) * (kGruK / 2) + kk * 8 + tq;
    wb[slot][0] = p[0];
    wb[slot][1] = p[4];
  }
  float h[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int b = b_base + (e < 2 ? g : g + 8);
    h[e] = b < a.batch ? a.h[size_t(b) * kGruH + j0 + (e & 1)] : 0.0f;
  }
  *reinterpret_cast<uint32_t*>(&hs[0][g][j0]) = pack_bf16(h[0], h[1]);
  *reinterpret_cast<uint32_t*>(&hs[0][g + 8][j0]) = pack_bf16(h[2], h[3]);
  const bool v0 = b_base + g < a.batch, v1 = b_base + g + 8 < a.batch;
  double loss = 0.0;
  cp_async_wait<0>();
  __syncthreads();

  // ldmatrix x4: lanes 0-7, 8-15, 16-23, 24-31 address the rows of the four 8x8 parts
  const int lr = (lane & 7) + (lane & 8), lc = (lane & 16) >> 1;
  for (int t = 0; t < a.T; ++t) {
    const int cur = t & 1, nxt = cur ^ 1;
    const int buf = (t / kChunk) & 1, ck = t % kChunk;
    if (ck == 0 && t + kChunk < a.T)
      stage_inputs(in, buf ^ 1, a.x, a.y, a.vec, a.t_total, a.seq, a.batch, b_base, a.t0, t + kChunk, a.T);
    uint32_t ah[4][4], ax[4];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                   : "=r"(ah[kk][0]), "=r"(ah[kk][1]), "=r"(ah[kk][2]), "=r"(ah[kk][3])
                   : "r"(smem_addr(&hs[cur][lr][kk * 16 + lc]))
                   : "memory");
    const float4 xa = in.x[buf][ck][g], xb = in.x[buf][ck][g + 8];
    const float x0[kGruX] = {xa.x, xa.y, xa.z, xa.w}, x1[kGruX] = {xb.x, xb.y, xb.z, xb.w};
    xblock_frag(x0, x1, tq, ax);
    float acc[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[q][0] = acc[q][1] = acc[q][2] = acc[q][3] = 0.0f;
#pragma unroll
    for (int kk = 0; kk < 5; ++kk)
#pragma unroll
      for (int q = 0; q < 3; ++q)
        mma_bf16_16816(acc[q], kk < 4 ? ah[kk] : ax, wb[5 * q + kk][0], wb[5 * q + kk][1]);
    mma_bf16_16816(acc[3], ax, wb[15][0], wb[15][1]);
    GruGate G[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) G[e] = gru_gate(acc[0][e], acc[1][e], acc[2][e], acc[3][e], h[e]);
    *reinterpret_cast<uint32_t*>(&hs[nxt][g][j0]) = pack_bf16(G[0].h_new, G[1].h_new);
    *reinterpret_cast<uint32_t*>(&hs[nxt][g + 8][j0]) = pack_bf16(G[2].h_new, G[3].h_new);
    float ys0 = 0.0f, ys1 = 0.0f;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      ys0 += wo[e] * G[e].h_new;
      ys1 += wo[e] * G[2 + e].h_new;
    }
    ys0 += __shfl_xor_sync(0xffffffffu, ys0, 1);
    ys0 += __shfl_xor_sync(0xffffffffu, ys0, 2);
    ys1 += __shfl_xor_sync(0xffffffffu, ys1, 1);
    ys1 += __shfl_xor_sync(0xffffffffu, ys1, 2);
    if (tq == 0) {
      ypart[cur][w][g] = ys0;
      ypart[cur][w][g + 8] = ys1;
    }
    const bool turn = w == (t & (kWarps - 1));  // the warps take turns at the outputs
    const float target = turn ? in.y[buf][ck][lane & (kRows - 1)] : 0.0f;
    if (ck == kChunk - 1) cp_async_wait<0>();  // the next chunk, started kChunk steps ago
    __syncthreads();
    // after the barrier, off the other warps' path: the activations and the outputs
    if (a.acts) {
#pragma unroll
      for (int r = 0; r < 2; ++r)
        if (r == 0 ? v0 : v1) {
          const int b = b_base + g + 8 * r;
          const GruGate &A = G[2 * r], &B = G[2 * r + 1];
          float* p = a.acts + act_index(0, a.batch, a.T, b, t, j0);
          const size_t s = size_t(a.batch) * a.T * kGruH;
          store2(p, h[2 * r], h[2 * r + 1], a.vec);
          store2(p + s, A.r, B.r, a.vec);
          store2(p + 2 * s, A.z, B.z, a.vec);
          store2(p + 3 * s, A.n, B.n, a.vec);
          store2(p + 4 * s, A.hn, B.hn, a.vec);
        }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) h[e] = G[e].h_new;
    if (turn && lane < kRows) {
      const int b = b_base + lane;
      if (b < a.batch) {
        float y = bo;
#pragma unroll
        for (int q = 0; q < kWarps; ++q) y += ypart[cur][q][lane];
        if (a.yout) a.yout[size_t(b) * a.T + t] = y;
        if (a.y) {
          const double err = double(y) - double(target);
          loss += err * err;
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r)
    if (r == 0 ? v0 : v1)
      store2(a.h + size_t(b_base + g + 8 * r) * kGruH + j0, h[2 * r], h[2 * r + 1], a.vec);
  if (a.loss && lane < kRows && loss != 0.0) atomicAdd(a.loss, loss);
}

struct BwdShared {
  __nv_bfloat16 dGT[2][kGru3H][kRPad];
  __nv_bfloat16 HT[2][kGruH][kRPad];
  float dHs[2][kRows][kDPad];
  StepInputs in;
  float yo[2][kChunk][kRows];
};

// The same measures backwards: the transposed recurrent weights stay in registers, the
// activations are loaded one step ahead, inputs and errors come through shared memory,
// and the weight-gradient products fill the latency of the dh chain.  The sums and their
// order are those of the step-by-step form.  A batch of 512 sequences over 400 steps
// went from 1,911 to 572 us (the forward from 806 to 428 us).
__global__ void __launch_bounds__(kThreads) gru_bwd_kernel(BwdArgs a) {
  __shared__ __align__(16) __nv_bfloat16 dG[2][kRows][kGPad];
  extern __shared__ __align__(16) unsigned char dyn[];  // BwdShared
  auto& dGT = reinterpret_cast<BwdShared*>(dyn)->dGT;
  auto& HT = reinterpret_cast<BwdShared*>(dyn)->HT;
  auto& dHs = reinterpret_cast<BwdShared*>(dyn)->dHs;
  StepInputs& in = reinterpret_cast<BwdShared*>(dyn)->in;
  auto& yo = reinterpret_cast<BwdShared*>(dyn)->yo;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int g = lane >> 2, tq = lane & 3;
  const int b_base = blockIdx.x * kRows;
  const int r0 = g, r1 = g + 8;
  const int b0 = b_base + r0, b1 = b_base + r1;
  const bool v0 = b0 < a.batch, v1 = b1 < a.batch;
  const int j0 = 8 * w + 2 * tq;
  const float wo[2] = {a.params[kGruOffWo + j0], a.params[kGruOffWo + j0 + 1]};

  for (int buf = 0; buf < 2; ++buf)
    for (int i = threadIdx.x; i < kChunk * kRows; i += kThreads) {
      (&in.x[buf][0][0])[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      (&in.y[buf][0][0])[i] = 0.f;
      (&yo[buf][0][0])[i] = 0.f;
    }
  __syncthreads();
  auto stage = [&](int chunk) {
    const int buf = chunk & 1;
    for (int i = threadIdx.x; i < kChunk * kRows; i += kThreads) {
      const int r = i / kChunk, t = chunk * kChunk + i % kChunk;
      if (b_base + r < a.batch && t < a.T) cp_async<4>(&yo[buf][i % kChunk][r], a.yout + size_t(b_base + r) * a.T + t);
    }
    stage_inputs(in, buf, a.x, a.y, a.vec, a.t_total, a.seq, a.batch, b_base, a.t0, chunk * kChunk, a.T);
  };
  stage((a.T - 1) / kChunk);

  float carry[4] = {0.0f, 0.0f, 0.0f, 0.0f};     // dL/dh' of this step from later steps
  float gwx[3][2][kGruX], gbx[3][2], gbh[3][2], gwo[2];
#pragma unroll
  for (int q = 0; q < 3; ++q)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      gbx[q][u] = gbh[q][u] = 0.0f;
#pragma unroll
      for (int i = 0; i < kGruX; ++i) gwx[q][u][i] = 0.0f;
    }
  gwo[0] = gwo[1] = 0.0f;
  float gbo = 0.0f;
  float accw[12][4];
#pragma unroll
  for (int i = 0; i < 12; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) accw[i][e] = 0.0f;
  const int mt = w >> 1, nt = w & 1;  // this warp's tile of the dh^T = Wh^T dG^T product
  const int kr0 = mt * 16 + g, kr1 = kr0 + 8;
  uint32_t wt[kGru3H / 16][4];  // Wh^T rows kr0, kr1
#pragma unroll
  for (int kk = 0; kk < kGru3H / 16; ++kk) {
    wt[kk][0] = a.wht[kr0 * (kGru3H / 2) + kk * 8 + tq];
    wt[kk][1] = a.wht[kr1 * (kGru3H / 2) + kk * 8 + tq];
    wt[kk][2] = a.wht[kr0 * (kGru3H / 2) + kk * 8 + 4 + tq];
    wt[kk][3] = a.wht[kr1 * (kGru3H / 2) + kk * 8 + 4 + tq];
  }
  // activations h, r, z, n, hn of (row, units j0, j0 + 1), one step ahead
  float2 act[2][5];
  auto load_acts = [&](int t) {
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int k = 0; k < 5; ++k)
        act[r][k] = (r == 0 ? v0 : v1) && t >= 0
                        ? load2(a.acts + act_index(k, a.batch, a.T, r == 0 ? b0 : b1, t, j0), a.vec)
                        : make_float2(0.f, 0.f);
  };
  load_acts(a.T - 1);
  cp_async_wait<0>();
  __syncthreads();

  for (int t = a.T - 1; t >= 0; --t) {
    const int cur = t & 1;
    const int buf = (t / kChunk) & 1, ck = t % kChunk;
    if (t >= kChunk && (ck == kChunk - 1 || t == a.T - 1)) stage(t / kChunk - 1);
    const float4 xa = in.x[buf][ck][r0], xb = in.x[buf][ck][r1];
    const float x0[kGruX] = {xa.x, xa.y, xa.z, xa.w}, x1[kGruX] = {xb.x, xb.y, xb.z, xb.w};
    const float dy0 = v0 ? a.gscale * (yo[buf][ck][r0] - in.y[buf][ck][r0]) : 0.0f;
    const float dy1 = v1 ? a.gscale * (yo[buf][ck][r1] - in.y[buf][ck][r1]) : 0.0f;
    float dh_dir[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int row = e < 2 ? r0 : r1;
      const int u = e & 1;
      const int j = j0 + u;
      const float2* A = act[e >> 1];
      const float h_old = u ? A[0].y : A[0].x, r = u ? A[1].y : A[1].x, z = u ? A[2].y : A[2].x, n = u ? A[3].y : A[3].x,
                  hn = u ? A[4].y : A[4].x;
      const float dy = e < 2 ? dy0 : dy1;
      const float h_new = (1.0f - z) * n + z * h_old;
      const float dh = carry[e] + dy * wo[u];
      const float dn = dh * (1.0f - z);
      const float dz = dh * (h_old - n);
      dh_dir[e] = dh * z;
      const float dan = dn * (1.0f - n * n);
      const float dr = dan * hn;
      const float dar = dr * r * (1.0f - r);
      const float daz = dz * z * (1.0f - z);
      const float dhn = dan * r;
      const float* xr = e < 2 ? x0 : x1;
#pragma unroll
      for (int i = 0; i < kGruX; ++i) {
        gwx[0][u][i] += dar * xr[i];
        gwx[1][u][i] += daz * xr[i];
        gwx[2][u][i] += dan * xr[i];
      }
      gbx[0][u] += dar;
      gbx[1][u] += daz;
      gbx[2][u] += dan;
      gbh[0][u] += dar;
      gbh[1][u] += daz;
      gbh[2][u] += dhn;
      gwo[u] += dy * h_new;
      const __nv_bfloat16 qr = __float2bfloat16_rn(dar), qz = __float2bfloat16_rn(daz),
                          qn = __float2bfloat16_rn(dhn);
      dG[cur][row][j] = qr;
      dG[cur][row][kGruH + j] = qz;
      dG[cur][row][2 * kGruH + j] = qn;
      dGT[cur][j][row] = qr;
      dGT[cur][kGruH + j][row] = qz;
      dGT[cur][2 * kGruH + j][row] = qn;
      HT[cur][j][row] = __float2bfloat16_rn(h_old);
    }
    if (w == 0 && tq == 0) gbo += dy0 + dy1;
    load_acts(t - 1);
    __syncthreads();
    // dh^T[k][row] = sum_n Wh^T[k][n] dG[row][n]: M = k (16 per tile), N = rows, K = 3H, one dependent chain;
    // between its products, dWh[n][k] += sum_row dG[row][n] h~[row][k]: M = n, N = k, K = 16 rows
    float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int i = 0; i < 12; ++i) {
      const uint32_t bb0 = *reinterpret_cast<const uint32_t*>(&dG[cur][nt * 8 + g][i * 16 + 2 * tq]);
      const uint32_t bb1 = *reinterpret_cast<const uint32_t*>(&dG[cur][nt * 8 + g][i * 16 + 2 * tq + 8]);
      mma_bf16_16816(c, wt[i], bb0, bb1);
      const int q = 12 * w + i;
      const int mi = q >> 3, ni = q & 7;
      const uint32_t af[4] = {*reinterpret_cast<const uint32_t*>(&dGT[cur][mi * 16 + g][2 * tq]),
                              *reinterpret_cast<const uint32_t*>(&dGT[cur][mi * 16 + g + 8][2 * tq]),
                              *reinterpret_cast<const uint32_t*>(&dGT[cur][mi * 16 + g][2 * tq + 8]),
                              *reinterpret_cast<const uint32_t*>(&dGT[cur][mi * 16 + g + 8][2 * tq + 8])};
      const uint32_t hb0 = *reinterpret_cast<const uint32_t*>(&HT[cur][ni * 8 + g][2 * tq]);
      const uint32_t hb1 = *reinterpret_cast<const uint32_t*>(&HT[cur][ni * 8 + g][2 * tq + 8]);
      mma_bf16_16816(accw[i], af, hb0, hb1);
    }
    {
      const int rr = nt * 8 + 2 * tq;
      dHs[cur][rr][kr0] = c[0];
      dHs[cur][rr + 1][kr0] = c[1];
      dHs[cur][rr][kr1] = c[2];
      dHs[cur][rr + 1][kr1] = c[3];
    }
    if (ck == 0) cp_async_wait<0>();  // the chunk below, started a chunk ago
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int row = e < 2 ? r0 : r1;
      carry[e] = dh_dir[e] + dHs[cur][row][j0 + (e & 1)];
    }
  }
  // This CTA's gradient goes to its own row of the partial buffer, each entry
  // written by exactly one lane; bc_gru_backward then sums the rows in CTA order,
  // so the gradient is the same bit for bit on every run.
  float* G = a.partial + size_t(blockIdx.x) * kPartialStride;
#pragma unroll
  for (int i = 0; i < 12; ++i) {
    const int q = 12 * w + i;
    const int mi = q >> 3, ni = q & 7;
    const int n0 = mi * 16 + g, k0 = ni * 8 + 2 * tq;
    *reinterpret_cast<float2*>(&G[kGruOffWh + n0 * kGruH + k0]) = make_float2(accw[i][0], accw[i][1]);
    *reinterpret_cast<float2*>(&G[kGruOffWh + (n0 + 8) * kGruH + k0]) = make_float2(accw[i][2], accw[i][3]);
  }
  // the per-unit sums: reduce over the 8 lanes that share a unit (same tq)
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int j = 8 * w + 2 * tq + u;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
#pragma unroll
      for (int i = 0; i < kGruX; ++i) {
        float v = gwx[q][u][i];
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        if (g == 0) G[kGruOffWx + (q * kGruH + j) * kGruX + i] = v;
      }
      float vb = gbx[q][u], vh = gbh[q][u];
      vb += __shfl_xor_sync(0xffffffffu, vb, 4);
      vb += __shfl_xor_sync(0xffffffffu, vb, 8);
      vb += __shfl_xor_sync(0xffffffffu, vb, 16);
      vh += __shfl_xor_sync(0xffffffffu, vh, 4);
      vh += __shfl_xor_sync(0xffffffffu, vh, 8);
      vh += __shfl_xor_sync(0xffffffffu, vh, 16);
      if (g == 0) {
        G[kGruOffBx + q * kGruH + j] = vb;
        G[kGruOffBh + q * kGruH + j] = vh;
      }
    }
    float vo = gwo[u];
    vo += __shfl_xor_sync(0xffffffffu, vo, 4);
    vo += __shfl_xor_sync(0xffffffffu, vo, 8);
    vo += __shfl_xor_sync(0xffffffffu, vo, 16);
    if (g == 0) G[kGruOffWo + j] = vo;
  }
  if (w == 0) {
    float vb = tq == 0 ? gbo : 0.0f;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) vb += __shfl_xor_sync(0xffffffffu, vb, s);
    if (lane == 0) G[kGruOffBo] = vb;
  }
}

// grads[i] += sum over the CTAs c = 0, 1, ... of partial[c][i], in that order.
__global__ void gru_grad_reduce_kernel(const float* partial, int n_cta, float* grads) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kGruNParam; i += gridDim.x * blockDim.x) {
    float s = 0.0f;
    for (int c = 0; c < n_cta; ++c) s += partial[size_t(c) * kPartialStride + i];
    grads[i] += s;
  }
}

// Adam on the FP32 master vector; the gradient is cleared for the next window.
__global__ void gru_adam_kernel(float* p, float* gr, float* m, float* v, int n, float lr, float b1, float b2, float eps,
                                float c1, float c2, float clip_scale) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = gr[i] * clip_scale;
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
    gr[i] = 0.0f;
  }
}

__global__ void gru_sqnorm_kernel(const float* gr, int n, float* out) {
  float s = 0.0f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) s += gr[i] * gr[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

// Extended weight matrix (BF16 pairs, [4H][K], rows r, z, hn, nx; see
// bc_gru.cuh) and the transposed recurrent block Wh^T [H][3H] for the backward.
__device__ __forceinline__ float wext_value(const float* p, int n, int k) {
  const int q = n / kGruH, u = n % kGruH;
  if (k < kGruH) return q < 3 ? p[kGruOffWh + (q * kGruH + u) * kGruH + k] : 0.0f;
  const int c = k - kGruH;
  const int xrow = q == 0 ? u : q == 1 ? kGruH + u : 2 * kGruH + u;  // Wx row of this block
  if (c < 2 * kGruX) return q == 2 ? 0.0f : bf16_round(p[kGruOffWx + xrow * kGruX + (c % kGruX)]);
  if (c < 2 * kGruX + 2) {
    const float bsum = q == 0   ? p[kGruOffBx + u] + p[kGruOffBh + u]
                       : q == 1 ? p[kGruOffBx + kGruH + u] + p[kGruOffBh + kGruH + u]
                       : q == 2 ? p[kGruOffBh + 2 * kGruH + u]
                                : p[kGruOffBx + 2 * kGruH + u];
    const float hi = bf16_round(bsum);
    return c == 2 * kGruX ? hi : bsum - hi;
  }
  return 0.0f;
}

__global__ void gru_pack_kernel(const float* p, uint32_t* wext, uint32_t* wht) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kGruRows * kGruK / 2; i += gridDim.x * blockDim.x) {
    const int n = i / (kGruK / 2), k = 2 * (i % (kGruK / 2));
    wext[i] = pack_bf16(wext_value(p, n, k), wext_value(p, n, k + 1));
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kGru3H * kGruH / 2; i += gridDim.x * blockDim.x) {
    const int kt = i / (kGru3H / 2), nt = 2 * (i % (kGru3H / 2));
    wht[i] = pack_bf16(p[kGruOffWh + nt * kGruH + kt], p[kGruOffWh + (nt + 1) * kGruH + kt]);
  }
}

bc_status launch_status(cudaError_t e, const char* what) {
  if (e != cudaSuccess) return fail(BC_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  return BC_OK;
}

}  // namespace
}  // namespace bc

using namespace bc;

extern "C" {

int32_t bc_gru_nparam(void) { return kGruNParam; }

bc_status bc_gru_pack(const float* params, uint32_t* wext, uint32_t* wht, void* stream) {
  if (!params || !wext || !wht) return fail(BC_ERR_INVALID, "bc_gru_pack: null buffer");
  gru_pack_kernel<<<40, 256, 0, static_cast<cudaStream_t>(stream)>>>(params, wext, wht);
  return launch_status(cudaGetLastError(), "gru_pack_kernel");
}

bc_status bc_gru_forward(const float* params, const uint32_t* wext, const float* x, const float* y, int64_t t_total,
                         const int32_t* seq, int32_t batch, int64_t t0, int32_t T, float* h, float* acts, float* yout,
                         double* loss, void* stream) {
  if (!params || !wext || !x || !seq || !h) return fail(BC_ERR_INVALID, "bc_gru_forward: null buffer");
  if (batch <= 0 || T <= 0 || t0 < 0 || t0 + T > t_total)
    return fail(BC_ERR_INVALID, "bc_gru_forward: window outside the sequences");
  if (acts && !yout) return fail(BC_ERR_INVALID, "bc_gru_forward: acts need yout");
  const bool vec = reinterpret_cast<uintptr_t>(x) % 16 == 0 && reinterpret_cast<uintptr_t>(h) % 8 == 0 &&
                   reinterpret_cast<uintptr_t>(acts) % 8 == 0;
  FwdArgs a{params, wext, x, y, t_total, seq, batch, t0, T, h, acts, yout, loss, vec};
  gru_fwd_kernel<<<(batch + kRows - 1) / kRows, kThreads, 0, static_cast<cudaStream_t>(stream)>>>(a);
  return launch_status(cudaGetLastError(), "gru_fwd_kernel");
}

int64_t bc_gru_backward_workspace(int32_t batch) {
  return batch > 0 ? int64_t((batch + kRows - 1) / kRows) * kPartialStride : 0;
}

bc_status bc_gru_backward(const float* params, const uint32_t* wht, const float* x, const float* y, int64_t t_total,
                          const int32_t* seq, int32_t batch, int64_t t0, int32_t T, const float* acts,
                          const float* yout, float gscale, float* grads, float* workspace, void* stream) {
  if (!params || !wht || !x || !y || !seq || !acts || !yout || !grads || !workspace)
    return fail(BC_ERR_INVALID, "bc_gru_backward: null buffer");
  if (batch <= 0 || T <= 0 || t0 < 0 || t0 + T > t_total)
    return fail(BC_ERR_INVALID, "bc_gru_backward: window outside the sequences");
  if (reinterpret_cast<uintptr_t>(workspace) % 16 != 0)
    return fail(BC_ERR_INVALID, "bc_gru_backward: workspace must be 16-byte aligned");
  const int n_cta = (batch + kRows - 1) / kRows;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool vec = reinterpret_cast<uintptr_t>(x) % 16 == 0 && reinterpret_cast<uintptr_t>(acts) % 8 == 0;
  BwdArgs a{params, wht, x, y, t_total, seq, batch, t0, T, acts, yout, gscale, workspace, vec};
  bc_status s = launch_status(
      cudaFuncSetAttribute(gru_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(BwdShared))),
      "gru_bwd_kernel");
  if (s != BC_OK) return s;
  gru_bwd_kernel<<<n_cta, kThreads, sizeof(BwdShared), st>>>(a);
  s = launch_status(cudaGetLastError(), "gru_bwd_kernel");
  if (s != BC_OK) return s;
  gru_grad_reduce_kernel<<<(kGruNParam + 255) / 256, 256, 0, st>>>(workspace, n_cta, grads);
  return launch_status(cudaGetLastError(), "gru_grad_reduce_kernel");
}

bc_status bc_gru_grad_sqnorm(const float* grads, float* out, void* stream) {
  if (!grads || !out) return fail(BC_ERR_INVALID, "bc_gru_grad_sqnorm: null buffer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(out, 0, sizeof(float), s);
  if (e != cudaSuccess) return launch_status(e, "cudaMemsetAsync");
  gru_sqnorm_kernel<<<8, 256, 0, s>>>(grads, kGruNParam, out);
  return launch_status(cudaGetLastError(), "gru_sqnorm_kernel");
}

bc_status bc_gru_adam(float* params, float* grads, float* m, float* v, int64_t step, float lr, float beta1,
                      float beta2, float eps, float clip_scale, void* stream) {
  if (!params || !grads || !m || !v) return fail(BC_ERR_INVALID, "bc_gru_adam: null buffer");
  if (step < 1) return fail(BC_ERR_INVALID, "bc_gru_adam: step counts from 1");
  const float c1 = float(1.0 / (1.0 - std::pow(double(beta1), double(step))));
  const float c2 = float(1.0 / (1.0 - std::pow(double(beta2), double(step))));
  gru_adam_kernel<<<(kGruNParam + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      params, grads, m, v, kGruNParam, lr, beta1, beta2, eps, c1, c2, clip_scale);
  return launch_status(cudaGetLastError(), "gru_adam_kernel");
}

}  // extern "C"
