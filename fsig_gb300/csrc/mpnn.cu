// Order-scoring network kernels: features, forward, backward, weight
// gradients and Adam, all hand-written; matrix products on the tensor cores
// with mma.sync m16n8k16 (BF16 operands, FP32 accumulation), four warps per
// query graph (at most 32 vertices = two 16-row tiles), each warp 16 of the 64
// output columns.  (The products are 32 x 64 x 64: far below a tcgen05 tile of
// 128 rows.)
//
//   h0 = relu(x W_in + b_in)                        x: 8 features, padded to 16
//   h_{l+1} = relu(h_l W_s[l] + (D^-1 A h_l) W_n[l] + b[l]),  l = 0, 1, 2
//   score = h3 . w_out + b_out
//
// Rows of absent vertices (index >= n) are kept at zero.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "match.h"
#include "mpnn.h"

namespace fsig {
namespace {

constexpr int kWBf = kPB;  // BF16 weight copy covers [0, kPB): W_in, b_in (unused), W_s, W_n
constexpr int kGraphThreads = 128;  // threads of one graph
constexpr int kGraphsPerBlock = 2;  // graphs at a time, sharing the block's weights
// Row strides in shared memory, padded so that the 8 rows of an ldmatrix (or of
// a fragment's epilogue) fall into different banks.
constexpr int kLd = kHid + 8, kLdX = kFeatPad + 8, kLdF = kHid + 8;

__device__ __forceinline__ uint16_t f2bf(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float bf2f(uint16_t x) { return __bfloat162float(__ushort_as_bfloat16(x)); }

__device__ __forceinline__ void mma_bf16(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Four 8 x 8 BF16 matrices; lane l gives the address of row l % 8 of matrix l / 8.
template <bool kTrans>
__device__ __forceinline__ void ldmatrix4(uint32_t r[4], const uint16_t* p) {
  const uint32_t a = uint32_t(__cvta_generic_to_shared(p));
  if constexpr (kTrans)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}

// acc (rows 0..31, columns n0..n0+15 of C, m16n8k16 fragments) += A B, with A
// [32][K] at row stride lda, and B [K][64] (kTransB: [64][K], i.e. B^T) at row
// stride kLd.  K ascending in steps of 16.
template <int K, bool kTransB>
__device__ __forceinline__ void gemm_cols(const uint16_t* A, int lda, const uint16_t* B, int n0, float acc[2][2][4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int kk = 0; kk < K; kk += 16) {
    uint32_t a[2][4], b[4];
#pragma unroll
    for (int mt = 0; mt < 2; mt++) ldmatrix4<false>(a[mt], A + (mt * 16 + (lane & 15)) * lda + kk + (lane >> 4) * 8);
    if constexpr (kTransB)
      ldmatrix4<false>(b, B + (n0 + (lane & 7) + (lane >> 4) * 8) * kLd + kk + ((lane >> 3) & 1) * 8);
    else
      ldmatrix4<true>(b, B + (kk + (lane & 15)) * kLd + n0 + (lane >> 4) * 8);
#pragma unroll
    for (int nt = 0; nt < 2; nt++) {
      mma_bf16(acc[0][nt], a[0], b[2 * nt], b[2 * nt + 1]);
      mma_bf16(acc[1][nt], a[1], b[2 * nt], b[2 * nt + 1]);
    }
  }
}

__device__ __forceinline__ void zero_acc(float acc[2][2][4]) {
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int k = 0; k < 4; k++) acc[i][j][k] = 0.f;
}

// Visits every accumulator element as (row, col, value).
template <class F>
__device__ __forceinline__ void for_acc(float acc[2][2][4], int n0, F f) {
  const int lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
#pragma unroll
  for (int mt = 0; mt < 2; mt++)
#pragma unroll
    for (int nt = 0; nt < 2; nt++)
#pragma unroll
      for (int j = 0; j < 4; j++)
        f(mt * 16 + g + (j >= 2 ? 8 : 0), n0 + nt * 8 + 2 * c + (j & 1), acc[mt][nt][j]);
}

struct BlockW {
  uint16_t win[kFeatPad * kLd];
  uint16_t ws[kLayers][kHid * kLd];
  uint16_t wn[kLayers][kHid * kLd];
};

struct GraphBuf {
  uint16_t x[32 * kLdX];
  uint16_t h[kLayers + 1][32 * kLd];
  uint16_t m[kLayers][32 * kLd];
  uint32_t nbr[32];
  float invdeg[32];
};

struct GraphBufTrain : GraphBuf {
  uint16_t dz[32 * kLd];
  float dh[32 * kLdF];
  float q[32 * kLdF];
  float ds[32];
};

// Per-node record of what the weight-gradient kernel needs (BF16).
constexpr int kActX = 0, kActH = kFeatPad, kActM = kActH + kLayers * kHid, kActDz = kActM + kLayers * kHid,
              kActW = kActDz + (kLayers + 1) * kHid;
static_assert(kActW % 8 == 0 && kActH % 8 == 0 && kPWs % 8 == 0 && kPWn % 8 == 0 && kLd % 8 == 0,
              "rows are copied 16 bytes at a time");

// rows x 64 BF16 from a dense array in global memory to row stride kLd, 16
// bytes a thread.
__device__ __forceinline__ void load_weights(uint16_t* dst, const uint16_t* __restrict__ src, int rows) {
  for (int i = threadIdx.x; i < rows * (kHid / 8); i += blockDim.x)
    *reinterpret_cast<uint4*>(dst + (i >> 3) * kLd + (i & 7) * 8) =
        __ldg(reinterpret_cast<const uint4*>(src) + i);
}

// A group of kGraphThreads threads per graph.  Train: also the loss, the bias
// and output gradients, and per-node activations and pre-activation gradients
// for the weight gradients.  Bound by latency: a chain of small products with a
// barrier after each.  (One warp per graph, its operands gathered element by
// element with 8-way bank conflicts and the weights copied two bytes at a time,
// took 158 us for the training step of 256 graphs; this takes 41 us.)
template <bool kTrain>
__global__ void __launch_bounds__(kGraphThreads * kGraphsPerBlock) mpnn_graph_kernel(
    const uint16_t* __restrict__ wbf, const float* __restrict__ master, uint32_t num_graphs,
    const uint32_t* __restrict__ goff, const float* __restrict__ feat, const uint32_t* __restrict__ nbr,
    float* __restrict__ scores, const float* __restrict__ target, float inv_count, float* __restrict__ grad,
    float* __restrict__ loss, uint16_t* __restrict__ acts) {
  using Buf = typename std::conditional<kTrain, GraphBufTrain, GraphBuf>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  BlockW& W = *reinterpret_cast<BlockW*>(smem);
  const int group = threadIdx.x / kGraphThreads, tid = threadIdx.x % kGraphThreads;
  Buf& B = reinterpret_cast<Buf*>(smem + sizeof(BlockW))[group];
  load_weights(W.win, wbf + kPWin, kFeatPad);
  load_weights(W.ws[0], wbf + kPWs, kLayers * kHid);
  load_weights(W.wn[0], wbf + kPWn, kLayers * kHid);
  __syncthreads();
  auto sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(kGraphThreads) : "memory"); };
  const int lane = tid & 31, warp = tid >> 5, n0 = warp * 16;
  const float* b_in = master + kPBin;
  const float* b_l = master + kPB;
  const float* w_out = master + kPWout;
  const float b_out = master[kPBout];
  float acc[2][2][4];
  for (uint32_t q = blockIdx.x + group * gridDim.x; q < num_graphs; q += gridDim.x * kGraphsPerBlock) {
    const uint32_t g0 = goff[q];
    const int n = int(goff[q + 1] - g0);
    sync();  // the previous graph's buffers are read
    // inputs
    for (int i = tid; i < 32 * kFeatPad; i += kGraphThreads) {
      const int r = i / kFeatPad, c = i % kFeatPad;
      B.x[r * kLdX + c] = (r < n && c < kFeat) ? f2bf(feat[uint64_t(g0 + r) * kFeat + c]) : uint16_t(0);
    }
    if (tid < 32) {
      const uint32_t mine = tid < n ? nbr[g0 + tid] : 0u;
      B.nbr[tid] = mine;
      B.invdeg[tid] = mine ? 1.f / float(__popc(mine)) : 0.f;
    }
    sync();
    // input layer
    zero_acc(acc);
    gemm_cols<kFeatPad, false>(B.x, kLdX, W.win, n0, acc);
    for_acc(acc, n0, [&](int r, int c, float v) { B.h[0][r * kLd + c] = r < n ? f2bf(fmaxf(v + b_in[c], 0.f)) : 0; });
    sync();
    for (int l = 0; l < kLayers; l++) {
      // mean over neighbours, eight rows per warp, two columns per lane
      for (int r = warp * 8; r < warp * 8 + 8; r++) {
        float s0 = 0.f, s1 = 0.f;
        uint32_t m = B.nbr[r];
        while (m) {
          const int j = __ffs(m) - 1;
          m &= m - 1;
          const uint32_t v = *reinterpret_cast<const uint32_t*>(&B.h[l][j * kLd + 2 * lane]);
          s0 += bf2f(uint16_t(v));
          s1 += bf2f(uint16_t(v >> 16));
        }
        const float id = B.invdeg[r];
        *reinterpret_cast<uint32_t*>(&B.m[l][r * kLd + 2 * lane]) =
            uint32_t(f2bf(s0 * id)) | (uint32_t(f2bf(s1 * id)) << 16);
      }
      sync();
      zero_acc(acc);
      gemm_cols<kHid, false>(B.h[l], kLd, W.ws[l], n0, acc);
      gemm_cols<kHid, false>(B.m[l], kLd, W.wn[l], n0, acc);
      const float* bl = b_l + l * kHid;
      for_acc(acc, n0, [&](int r, int c, float v) {
        B.h[l + 1][r * kLd + c] = r < n ? f2bf(fmaxf(v + bl[c], 0.f)) : 0;
      });
      sync();
    }
    // scores: row tid
    if (warp == 0) {
      float s = 0.f;
      if (lane < n) {
        s = b_out;
        for (int c = 0; c < kHid; c++) s += bf2f(B.h[kLayers][lane * kLd + c]) * w_out[c];
        scores[g0 + lane] = s;
      }
      if constexpr (kTrain) {
        const float ds = lane < n ? 2.f * inv_count * (s - target[g0 + lane]) : 0.f;
        const float lsum = warp_sum(lane < n ? (s - target[g0 + lane]) * (s - target[g0 + lane]) * inv_count : 0.f);
        const float dsum = warp_sum(ds);
        B.ds[lane] = ds;
        if (lane == 0) {
          atomicAdd(loss, lsum);
          atomicAdd(grad + kPBout, dsum);
        }
      }
    }
    if constexpr (kTrain) {
      sync();
      // ---- backward ----
      // d w_out[c] = sum_r h3[r][c] ds_r ; d h3[r][c] = ds_r w_out[c]
      const int col = tid & (kHid - 1), half = tid / kHid;  // a column, and every other row
      {
        float gw = 0.f;
        const float wo = w_out[col];
        for (int r = half; r < 32; r += 2) {
          const float dr = B.ds[r];
          if (r < n) gw += bf2f(B.h[kLayers][r * kLd + col]) * dr;
          B.dh[r * kLdF + col] = dr * wo;
        }
        atomicAdd(grad + kPWout + col, gw);
      }
      sync();
      for (int l = kLayers - 1; l >= -1; l--) {
        // dz = dh * relu'(h_{l+1}); bias gradient
        const uint16_t* hl1 = B.h[l + 1];
        float db = 0.f;
        for (int r = half; r < 32; r += 2) {
          const float z = (r < n && bf2f(hl1[r * kLd + col]) > 0.f) ? B.dh[r * kLdF + col] : 0.f;
          B.dz[r * kLd + col] = f2bf(z);
          db += z;
        }
        atomicAdd(grad + (l >= 0 ? kPB + l * kHid : kPBin) + col, db);
        sync();
        // save per-node records for the weight gradients, 16 bytes a thread
        for (int i = tid; i < n * 8; i += kGraphThreads) {
          const int r = i >> 3, c = (i & 7) * 8;
          uint16_t* rec = acts + uint64_t(g0 + r) * kActW;
          auto save = [&](int to, const uint16_t* from) {
            *reinterpret_cast<uint4*>(rec + to + c) = *reinterpret_cast<const uint4*>(from + r * kLd + c);
          };
          save(kActDz + (l + 1) * kHid, B.dz);
          if (l >= 0) {
            save(kActH + l * kHid, B.h[l]);
            save(kActM + l * kHid, B.m[l]);
          } else if (c < kFeatPad) {
            *reinterpret_cast<uint4*>(rec + kActX + c) = *reinterpret_cast<const uint4*>(B.x + r * kLdX + c);
          }
        }
        if (l < 0) break;
        // dh_l = dz W_s^T + A_norm^T (dz W_n^T)
        zero_acc(acc);
        gemm_cols<kHid, true>(B.dz, kLd, W.wn[l], n0, acc);
        for_acc(acc, n0, [&](int r, int c, float v) { B.q[r * kLdF + c] = v * B.invdeg[r]; });
        zero_acc(acc);
        gemm_cols<kHid, true>(B.dz, kLd, W.ws[l], n0, acc);
        sync();
        for_acc(acc, n0, [&](int r, int c, float v) {
          // (A_norm^T Q)[r] = sum over i with r in nbr(i) of Q[i] / deg_i (already scaled)
          float t = v;
          uint32_t m = B.nbr[r];  // symmetric adjacency: i in nbr(r) <=> r in nbr(i)
          while (m) {
            const int i = __ffs(m) - 1;
            m &= m - 1;
            t += B.q[i * kLdF + c];
          }
          B.dh[r * kLdF + c] = r < n ? t : 0.f;
        });
        sync();
      }
    }
  }
}

// Weight gradients: for matrix id (0: W_in, 1..3: W_s, 4..6: W_n),
// G[i][c] = sum over nodes of A_node[i] * dZ_node[c]; blocks of kWgradNodes
// nodes, staged in shared memory, one warp per 16 output rows.  Bound by the
// records' reads from L2 and the atomics of the partial sums.  (512 nodes a
// block, one warp per 32 rows gathering two bytes at a time, ran 63 blocks and
// took 169 us for 4,600 nodes; this takes 11.5 us.)
constexpr int kWgradNodes = 128;
__global__ void __launch_bounds__(128) mpnn_wgrad_kernel(const uint16_t* __restrict__ acts, uint32_t nodes,
                                                         float* __restrict__ grad) {
  __shared__ __align__(16) uint16_t sa[kWgradNodes * kLd], sz[kWgradNodes * kLd];
  const int mat = blockIdx.y;
  const int rows = mat == 0 ? kFeatPad : kHid;
  int asrc, dzsrc, gdst;
  if (mat == 0) { asrc = kActX; dzsrc = kActDz; gdst = kPWin; }
  else if (mat <= kLayers) { asrc = kActH + (mat - 1) * kHid; dzsrc = kActDz + mat * kHid; gdst = kPWs + (mat - 1) * kHid * kHid; }
  else { asrc = kActM + (mat - 1 - kLayers) * kHid; dzsrc = kActDz + (mat - kLayers) * kHid; gdst = kPWn + (mat - 1 - kLayers) * kHid * kHid; }
  const uint32_t begin = blockIdx.x * kWgradNodes;
  const uint4 none = make_uint4(0, 0, 0, 0);
  for (int i = threadIdx.x; i < kWgradNodes * 8; i += blockDim.x) {
    const int k = i >> 3, c = (i & 7) * 8;
    const uint16_t* rec = acts + uint64_t(begin + k) * kActW;
    const bool in = begin + k < nodes;
    *reinterpret_cast<uint4*>(sz + k * kLd + c) = in ? *reinterpret_cast<const uint4*>(rec + dzsrc + c) : none;
    if (c < rows) *reinterpret_cast<uint4*>(sa + k * kLd + c) = in ? *reinterpret_cast<const uint4*>(rec + asrc + c) : none;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, m0 = (threadIdx.x >> 5) * 16;
  if (m0 >= rows) return;
  float acc[8][4] = {};
#pragma unroll 2
  for (int kk = 0; kk < kWgradNodes; kk += 16) {
    uint32_t a[4];
    ldmatrix4<true>(a, sa + (kk + (lane & 7) + (lane >> 4) * 8) * kLd + m0 + ((lane >> 3) & 1) * 8);
#pragma unroll
    for (int nt = 0; nt < 8; nt += 2) {
      uint32_t b[4];
      ldmatrix4<true>(b, sz + (kk + (lane & 15)) * kLd + nt * 8 + (lane >> 4) * 8);
      mma_bf16(acc[nt], a, b[0], b[1]);
      mma_bf16(acc[nt + 1], a, b[2], b[3]);
    }
  }
  const int g = lane >> 2, c = lane & 3;
#pragma unroll
  for (int nt = 0; nt < 8; nt++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float v = acc[nt][j];
      if (v != 0.f) atomicAdd(grad + gdst + (m0 + g + (j >= 2 ? 8 : 0)) * kHid + nt * 8 + 2 * c + (j & 1), v);
    }
}

__global__ void mpnn_adam_kernel(float* p, const float* g, float* m1, float* m2, uint16_t* wbf, int n, float lr,
                                 float b1, float b2, float eps, float c1, float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float a = b1 * m1[i] + (1.f - b1) * gi;
    const float b = b2 * m2[i] + (1.f - b2) * gi * gi;
    m1[i] = a;
    m2[i] = b;
    const float v = p[i] - lr * (a / c1) / (sqrtf(b / c2) + eps);
    p[i] = v;
    if (i < kWBf) wbf[i] = f2bf(v);
  }
}

__global__ void mpnn_to_bf16_kernel(const float* p, uint16_t* wbf, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) wbf[i] = f2bf(p[i]);
}

// Features (see fsig_mpnn_features in include/fsig.h); thread per query vertex.
__global__ void mpnn_features_kernel(const QVert* __restrict__ qv, uint32_t G, const uint32_t* __restrict__ qoff,
                                     uint32_t Q, const uint32_t* __restrict__ counts,
                                     const uint32_t* __restrict__ orders, const uint32_t* __restrict__ base,
                                     int32_t L, float* __restrict__ feat, uint32_t* __restrict__ nbr) {
  for (uint32_t gi = blockIdx.x * blockDim.x + threadIdx.x; gi < G; gi += gridDim.x * blockDim.x) {
    const QVert& x = qv[gi];
    uint32_t lo = 0, hi = Q;  // query of gi: last q with qoff[q] <= gi
    while (hi - lo > 1) {
      const uint32_t mid = midpoint(lo, hi);
      if (qoff[mid] <= gi) lo = mid; else hi = mid;
    }
    const uint32_t g0 = qoff[lo], n = qoff[lo + 1] - g0;
    const uint32_t deg = __popc(x.adj), cnt = counts[gi];
    const uint32_t cls = (x.label >= 0 && x.label < L) ? base[x.label + 1] - base[x.label] : 0u;
    uint32_t sigbits = 0;
    for (int i = 1; i < kSigWords; i++) sigbits += __popc(x.sig[i]);
    float nsum = 0.f;
    for (uint32_t w = 0; w < n; w++)
      if ((x.adj >> w) & 1u) nsum += plog2(counts[g0 + w]);
    uint32_t pos = 0;  // position of this vertex in the heuristic order
    const uint32_t u = gi - g0;
    for (uint32_t i = 0; i < n; i++)
      if (orders[uint64_t(lo) * kMaxQ + i] == u) pos = i;
    float* f = feat + uint64_t(gi) * kFeat;
    f[0] = n > 1 ? float(pos) / float(n - 1) : 0.f;
    f[1] = float(deg) / 8.f;
    f[2] = plog2(cnt) / 20.f;
    f[3] = plog2(cls) / 20.f;
    f[4] = cls ? float(cnt) / float(cls) : 0.f;
    f[5] = float(sigbits) / 16.f;
    f[6] = float(n) / 32.f;
    f[7] = deg ? nsum / float(20u * deg) : 0.f;
    nbr[gi] = x.adj;
  }
}

size_t graph_kernel_smem(bool train) {
  return sizeof(BlockW) + kGraphsPerBlock * (train ? sizeof(GraphBufTrain) : sizeof(GraphBuf));
}

int launch_graph_kernel(Engine& e, bool train, uint32_t num_graphs, const uint32_t* d_goff, const float* d_feat,
                        const uint32_t* d_nbr, float* d_scores, const float* d_target, float inv_count,
                        float* d_loss, uint16_t* d_acts) {
  MpnnState& M = *e.mpnn;
  if (!num_graphs) return FSIG_OK;
  const size_t smem = graph_kernel_smem(train);
  const unsigned threads = kGraphThreads * kGraphsPerBlock;
  // one block an SM (shared memory); few graphs go to a block each
  const unsigned grid = std::min<unsigned>(num_graphs, unsigned(e.num_sms));
  int rc = mpnn_configure(e);
  if (rc) return rc;
  if (train) {
    mpnn_graph_kernel<true><<<grid, threads, smem, e.stream>>>(
        M.wbf, M.master, num_graphs, d_goff, d_feat, d_nbr, d_scores, d_target, inv_count, M.grad, d_loss, d_acts);
  } else {
    mpnn_graph_kernel<false><<<grid, threads, smem, e.stream>>>(
        M.wbf, M.master, num_graphs, d_goff, d_feat, d_nbr, d_scores, nullptr, 0.f, nullptr, nullptr, nullptr);
  }
  FSIG_CUDA_TRY(cudaGetLastError());
  return FSIG_OK;
}

}  // namespace

int mpnn_configure(Engine& e) {
  if (e.mpnn_configured) return FSIG_OK;
  FSIG_CUDA_TRY(cudaFuncSetAttribute(mpnn_graph_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     int(graph_kernel_smem(true))));
  FSIG_CUDA_TRY(cudaFuncSetAttribute(mpnn_graph_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     int(graph_kernel_smem(false))));
  e.mpnn_configured = true;
  return FSIG_OK;
}

int mpnn_init(Engine& e) {
  if (e.mpnn) return FSIG_OK;
  auto* M = new MpnnState();
  const size_t pb = sizeof(float) * kParams;
  // One-time state outside the arena (the arena is reset when a graph loads).
  if (cudaMalloc(&M->master, pb) != cudaSuccess || cudaMalloc(&M->grad, pb + sizeof(float)) != cudaSuccess ||
      cudaMalloc(&M->m1, pb) != cudaSuccess || cudaMalloc(&M->m2, pb) != cudaSuccess ||
      cudaMalloc(&M->wbf, sizeof(uint16_t) * kWBf) != cudaSuccess) {
    cudaFree(M->master);
    cudaFree(M->grad);
    cudaFree(M->m1);
    cudaFree(M->m2);
    cudaFree(M->wbf);
    delete M;
    return fail(FSIG_EADMISSION, "cannot reserve the order network's state");
  }
  e.mpnn = M;
  FSIG_CUDA_TRY(cudaMemsetAsync(M->master, 0, pb, e.stream));
  FSIG_CUDA_TRY(cudaMemsetAsync(M->grad, 0, pb, e.stream));
  FSIG_CUDA_TRY(cudaMemsetAsync(M->m1, 0, pb, e.stream));
  FSIG_CUDA_TRY(cudaMemsetAsync(M->m2, 0, pb, e.stream));
  FSIG_CUDA_TRY(cudaMemsetAsync(M->wbf, 0, sizeof(uint16_t) * kWBf, e.stream));
  return FSIG_OK;
}

void mpnn_free(Engine& e) {
  if (!e.mpnn) return;
  cudaFree(e.mpnn->master);
  cudaFree(e.mpnn->grad);
  cudaFree(e.mpnn->m1);
  cudaFree(e.mpnn->m2);
  cudaFree(e.mpnn->wbf);
  delete e.mpnn;
  e.mpnn = nullptr;
}

int mpnn_set_params(Engine& e, const float* params) {
  int rc = mpnn_init(e);
  if (rc) return rc;
  MpnnState& M = *e.mpnn;
  FSIG_CUDA_TRY(cudaMemcpyAsync(M.master, params, sizeof(float) * kParams, cudaMemcpyHostToDevice, e.stream));
  FSIG_CUDA_TRY(cudaMemsetAsync(M.m1, 0, sizeof(float) * kParams, e.stream));
  FSIG_CUDA_TRY(cudaMemsetAsync(M.m2, 0, sizeof(float) * kParams, e.stream));
  mpnn_to_bf16_kernel<<<64, 256, 0, e.stream>>>(M.master, M.wbf, kWBf);
  FSIG_CUDA_TRY(cudaGetLastError());
  FSIG_CUDA_TRY(cudaStreamSynchronize(e.stream));
  M.step = 0;
  M.loaded = true;
  return FSIG_OK;
}

int mpnn_get_params(Engine& e, float* params) {
  if (!e.mpnn || !e.mpnn->loaded) return fail(FSIG_EINVAL, "no order network loaded");
  FSIG_CUDA_TRY(cudaMemcpyAsync(params, e.mpnn->master, sizeof(float) * kParams, cudaMemcpyDeviceToHost, e.stream));
  FSIG_CUDA_TRY(cudaStreamSynchronize(e.stream));
  return FSIG_OK;
}

int mpnn_features_device(Engine& e, const QVert* d_qv, uint32_t G, const uint32_t* d_qoff, uint32_t Q,
                         const uint32_t* d_counts, const uint32_t* d_orders, float* d_feat, uint32_t* d_nbr) {
  if (!e.has_graph) return fail(FSIG_ENOGRAPH, "no data graph loaded");
  if (!G) return FSIG_OK;
  mpnn_features_kernel<<<std::min<uint32_t>((G + 127) / 128, e.num_sms * 8), 128, 0, e.stream>>>(
      d_qv, G, d_qoff, Q, d_counts, d_orders, e.g.base, e.g.L, d_feat, d_nbr);
  FSIG_CUDA_TRY(cudaGetLastError());
  return FSIG_OK;
}

int mpnn_forward_device(Engine& e, uint32_t num_graphs, const uint32_t* d_goff, const float* d_feat,
                        const uint32_t* d_nbr, float* d_scores) {
  if (!e.mpnn || !e.mpnn->loaded) return fail(FSIG_EINVAL, "no order network loaded");
  return launch_graph_kernel(e, false, num_graphs, d_goff, d_feat, d_nbr, d_scores, nullptr, 0.f, nullptr, nullptr);
}

// Host-array entry used by the C ABI: scores, and with targets one training
// step (loss, gradients, Adam update when lr > 0).
int mpnn_run(Engine& e, uint32_t num_graphs, const uint32_t* goff, const float* feat, const uint32_t* nbr,
             const float* target, float lr, float* scores, float* loss, float* grads_out) {
  if (!e.mpnn || !e.mpnn->loaded) return fail(FSIG_EINVAL, "no order network loaded");
  MpnnState& M = *e.mpnn;
  cudaStream_t s = e.stream;
  for (uint32_t q = 0; q < num_graphs; q++)
    if (goff[q + 1] < goff[q] || goff[q + 1] - goff[q] > 32) return fail(FSIG_EINVAL, "graphs have 0..32 vertices");
  const uint32_t nodes = goff[num_graphs];
  const uint64_t mark = e.arena.mark();
  // inputs and outputs in one block each, copied at once through the staging area
  Block in, res;
  const uint64_t at_goff = in.add(sizeof(uint32_t) * (uint64_t(num_graphs) + 1)),
                 at_feat = in.add(sizeof(float) * uint64_t(nodes) * kFeat), at_nbr = in.add(sizeof(uint32_t) * nodes),
                 at_target = in.add(target ? sizeof(float) * nodes : 0);
  const uint64_t at_scores = scores ? res.add(sizeof(float) * nodes) : 0;
  const uint64_t out_bytes = target ? sizeof(float) * (kParams + 1) : res.bytes;  // a step's gradients and loss are in M.grad
  int rc = reserve_pinned(e, in.bytes + std::max<uint64_t>(out_bytes, 1));
  if (rc) return rc;
  in.host = static_cast<uint8_t*>(e.pinned);
  res.host = in.host + in.bytes;
  in.dev = e.arena.take<uint8_t>(in.bytes);
  float* d_scores = e.arena.take<float>(std::max<uint32_t>(nodes, 1));
  uint16_t* d_acts = target ? e.arena.take<uint16_t>(std::max<uint64_t>(uint64_t(nodes) * kActW, 1)) : nullptr;
  if (!in.dev || !d_scores || (target && !d_acts)) {
    e.arena.release(mark);
    return fail(FSIG_EADMISSION, "order-network batch does not fit the arena");
  }
  in.fill(at_goff, goff, sizeof(uint32_t) * (uint64_t(num_graphs) + 1));
  in.fill(at_feat, feat, sizeof(float) * uint64_t(nodes) * kFeat);
  in.fill(at_nbr, nbr, sizeof(uint32_t) * nodes);
  if (target) in.fill(at_target, target, sizeof(float) * nodes);
  FSIG_CUDA_TRY(cudaMemcpyAsync(in.dev, in.host, in.bytes, cudaMemcpyHostToDevice, s));
  uint32_t *d_goff = in.d<uint32_t>(at_goff), *d_nbr = in.d<uint32_t>(at_nbr);
  float *d_feat = in.d<float>(at_feat), *d_target = in.d<float>(at_target), *d_loss = M.grad + kParams;
  if (!target) {
    rc = launch_graph_kernel(e, false, num_graphs, d_goff, d_feat, d_nbr, d_scores, nullptr, 0.f, nullptr, nullptr);
  } else {
    FSIG_CUDA_TRY(cudaMemsetAsync(M.grad, 0, sizeof(float) * (kParams + 1), s));
    rc = launch_graph_kernel(e, true, num_graphs, d_goff, d_feat, d_nbr, d_scores, d_target,
                             nodes ? 1.f / float(nodes) : 0.f, d_loss, d_acts);
    if (!rc && nodes) {
      dim3 grid((nodes + kWgradNodes - 1) / kWgradNodes, 1 + 2 * kLayers);
      mpnn_wgrad_kernel<<<grid, 128, 0, s>>>(d_acts, nodes, M.grad);
      FSIG_CUDA_TRY(cudaGetLastError());
    }
    if (!rc && lr > 0.f) {
      M.step++;
      const float b1 = 0.9f, b2 = 0.999f;
      const float c1 = 1.f - std::pow(b1, float(M.step)), c2 = 1.f - std::pow(b2, float(M.step));
      mpnn_adam_kernel<<<64, 256, 0, s>>>(M.master, M.grad, M.m1, M.m2, M.wbf, kParams, lr, b1, b2, 1e-8f, c1, c2);
      FSIG_CUDA_TRY(cudaGetLastError());
    }
  }
  if (rc) {
    cudaStreamSynchronize(s);  // the queued copy reads the staging area
    e.arena.release(mark);
    return rc;
  }
  if (scores && nodes)
    FSIG_CUDA_TRY(cudaMemcpyAsync(res.host + at_scores, d_scores, sizeof(float) * nodes, cudaMemcpyDeviceToHost, s));
  if (target && (loss || grads_out))
    FSIG_CUDA_TRY(cudaMemcpyAsync(res.host, M.grad, sizeof(float) * (kParams + 1), cudaMemcpyDeviceToHost, s));
  FSIG_CUDA_TRY(cudaStreamSynchronize(s));
  if (scores && nodes) std::memcpy(scores, res.host + at_scores, sizeof(float) * nodes);
  if (target && grads_out) std::memcpy(grads_out, res.host, sizeof(float) * kParams);
  if (target && loss) std::memcpy(loss, res.host + sizeof(float) * kParams, sizeof(float));
  e.arena.release(mark);
  return FSIG_OK;
}

}  // namespace fsig
