// CUDA-core kernels of the compressed-KV path: the fused read that rebuilds K / V tiles in shared memory
// (fp32 with a positional restore or narrow heads, and bf16 with the rounding points of the tensor-core
// path, which the test-suite uses to cross-check it), plain attention, the online C-means' updates,
// rotations and camera transforms of explicit rows.
#include "nkv_internal.h"

namespace nkv {
namespace {

constexpr int BM = 64, BN = 64, BK = 16, PAD = 4;
constexpr int THREADS = 256;

// acc[4][4] += A[64 x K] * B[64 x K]^T for the calling block's tile.
// loadA(m, k) / loadB(n, k) return the operand element (0 outside bounds).
// As / Bs: BK * (64 + PAD) floats each.
template <class FA, class FB>
__device__ __forceinline__ void gemm_tile(float (&acc)[4][4], int K, FA loadA, FB loadB,
                                          float* As, float* Bs) {
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      int idx = tid + i * THREADS;
      int m = idx / BK, kk = idx % BK;
      int k = k0 + kk;
      As[kk * (BM + PAD) + m] = k < K ? loadA(m, k) : 0.f;
      Bs[kk * (BN + PAD) + m] = k < K ? loadB(m, k) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk * (BM + PAD) + ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk * (BN + PAD) + tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
}

// ----------------------------------------------------------------- attention
// One block = 64 queries of one head; K/V tiles of 64 tokens are either read
// from memory (CODEC = false) or rebuilt from the compressed history into
// shared memory (CODEC = true).  Online softmax in fp32.
struct AttnArgs {
  const void* q; int dtype; int64_t q_stride_token, q_stride_head;
  int Q, heads, N; float scale;
  nkv_history hk, hv;
  const void* wk; const float* bias_k; const void* wv; const float* bias_v;
  const void* k_plain; const void* v_plain; int64_t kv_stride_token, kv_stride_head;
  void* out; float* lse;
  nkv_rope rope;   // cos_sin == nullptr: no positional restore
  nkv_camera cam_k, cam_v;   // matrices == nullptr: no camera transform
};

template <int DK, int DV, bool CODEC>
__global__ void __launch_bounds__(THREADS)
attn_kernel(AttnArgs a) {
  extern __shared__ float smem[];
  float* Qs = smem;                 // [DK][64]
  float* Ks = Qs + DK * 64;         // [DK][64]
  float* Vs = Ks + DK * 64;         // [64][DV]
  float* Ps = Vs + 64 * DV;         // [64][64]
  float* As = Ps + 64 * 64;         // staging for the decode GEMM
  float* Bs = As + BK * (BM + PAD);
  __shared__ int crow_k[64], crow_v[64];
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int q0 = blockIdx.x * 64, head = blockIdx.y;
  const bool bf16 = a.dtype == NKV_BF16;
  for (int idx = tid; idx < 64 * DK; idx += THREADS) {
    int i = idx / DK, d = idx % DK;
    float v = 0.f;
    if (q0 + i < a.Q)
      v = load_float(a.q, a.dtype, static_cast<size_t>(q0 + i) * a.q_stride_token +
                                       static_cast<size_t>(head) * a.q_stride_head + d);
    Qs[d * 64 + i] = v;
  }
  constexpr int OC = DV / 16;
  float o[4][OC] = {};
  float m_run[4], l_run[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) { m_run[i] = -INFINITY; l_run[i] = 0.f; }

  for (int t0 = 0; t0 < a.N; t0 += 64) {
    __syncthreads();  // previous tile fully consumed (also orders the Qs fill)
    if (CODEC) {
      if (tid < 64) {
        int t = t0 + tid;
        crow_k[tid] = t < a.N ? center_row_of(a.hk, t) : 0;
        crow_v[tid] = t < a.N ? center_row_of(a.hv, t) : 0;
      }
      __syncthreads();
      // K and V tiles: [64 tok x D] = latent [64 x r] * W_head [D x r]^T, 64 columns at a time
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        const nkv_history& h = which == 0 ? a.hk : a.hv;
        const void* w = which == 0 ? a.wk : a.wv;
        const float* bias = which == 0 ? a.bias_k : a.bias_v;
        const int* crow = which == 0 ? crow_k : crow_v;
        const int D = which == 0 ? DK : DV;
        const uint16_t* centers = static_cast<const uint16_t*>(h.centers);
        for (int n0 = 0; n0 < D; n0 += 64) {
          float acc[4][4] = {};
          auto loadA = [&](int m, int k) {
            int t = t0 + m;
            if (t >= a.N) return 0.f;
            float v = latent_value(h, t, k);
            return bf16 ? round_to_bf16(v) : v;
          };
          auto loadB = [&](int nn, int k) {
            int c = n0 + nn;
            return c < D ? load_float(w, a.dtype,
                                      (static_cast<size_t>(head) * D + c) * h.rank + k) : 0.f;
          };
          gemm_tile(acc, h.rank, loadA, loadB, As, Bs);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            int m = ty * 4 + i;
            float vals[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              int c = n0 + tx * 4 + j;
              float v = 0.f;
              if (c < D && t0 + m < a.N) {
                float center = bf16_bits_to_float(
                    centers[static_cast<size_t>(crow[m]) * h.center_width +
                            static_cast<size_t>(head) * D + c]);
                float b = bias[head * D + c];
                if (bf16) {
                  v = round_to_bf16(__fadd_rn(acc[i][j], b));
                  v = round_to_bf16(__fadd_rn(v, center));
                } else {
                  v = __fadd_rn(__fadd_rn(acc[i][j], b), center);
                }
              }
              vals[j] = v;
            }
            if (which == 0 && a.rope.cos_sin != nullptr && t0 + m < a.N) {
              // rotate the adjacent pairs (c, c+1) by the token's frame / row / column
              const int half = D / 2, th = a.rope.table_half, third = th / 3;
              const int band_a = th - 2 * third, band_b = band_a + third;
              const int pos = max(a.rope.positions[t0 + m], 0);
              int frame = pos, prow = pos, pcol = pos;   // frame_seqlen 0: one table row per token
              if (a.rope.frame_seqlen > 0) {
                frame = pos / a.rope.frame_seqlen;
                const int spatial = pos - frame * a.rope.frame_seqlen;
                prow = spatial / a.rope.width;
                pcol = spatial - prow * a.rope.width;
              }
#pragma unroll
              for (int pr = 0; pr < 2; ++pr) {
                const int pl = (n0 + tx * 4) / 2 + pr;
                if (pl >= half) continue;
                const int pg = a.rope.pair_index ? a.rope.pair_index[head * half + pl] : pl;
                int coord = pg < band_a ? frame : (pg < band_b ? prow : pcol);
                coord = min(coord, a.rope.table_rows - 1);
                const float2 cs = reinterpret_cast<const float2*>(a.rope.cos_sin)[static_cast<size_t>(coord) * th + pg];
                const float x0 = vals[2 * pr], x1 = vals[2 * pr + 1];
                float y0 = fmaf(x0, cs.x, -(x1 * cs.y)), y1 = fmaf(x0, cs.y, x1 * cs.x);
                vals[2 * pr] = bf16 ? round_to_bf16(y0) : y0;
                vals[2 * pr + 1] = bf16 ? round_to_bf16(y1) : y1;
              }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              int c = n0 + tx * 4 + j;
              if (c >= D) continue;
              if (which == 0) Ks[c * 64 + m] = vals[j]; else Vs[m * DV + c] = vals[j];
            }
          }
        }
      }
    } else {
      for (int idx = tid; idx < 64 * DK; idx += THREADS) {
        int j = idx / DK, d = idx % DK;
        float v = 0.f;
        if (t0 + j < a.N)
          v = load_float(a.k_plain, a.dtype, static_cast<size_t>(t0 + j) * a.kv_stride_token +
                                                 static_cast<size_t>(head) * a.kv_stride_head + d);
        Ks[d * 64 + j] = v;
      }
      for (int idx = tid; idx < 64 * DV; idx += THREADS) {
        int j = idx / DV, d = idx % DV;
        float v = 0.f;
        if (t0 + j < a.N)
          v = load_float(a.v_plain, a.dtype, static_cast<size_t>(t0 + j) * a.kv_stride_token +
                                                 static_cast<size_t>(head) * a.kv_stride_head + d);
        Vs[j * DV + d] = v;
      }
    }
    if (CODEC && (a.cam_k.matrices != nullptr || a.cam_v.matrices != nullptr)) {
      // camera transform of the finished tiles: thread = one (token, 8-wide block)
      __syncthreads();
      for (int which = 0; which < 2; ++which) {
        const nkv_camera& cam = which == 0 ? a.cam_k : a.cam_v;
        if (cam.matrices == nullptr) continue;
        const int D = which == 0 ? DK : DV;
        for (int idx = tid; idx < 64 * (D / 8); idx += THREADS) {
          const int m = idx % 64, g = idx / 64;
          if (t0 + m >= a.N) continue;
          const int frame = min((t0 + m) / cam.tokens_per_frame, cam.frames - 1);
          const float* mat = cam.matrices + (static_cast<size_t>(frame) * 4 + (cam.cam_index[head * (D / 8) + g] & 3)) * 16;
          float x[8], y[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) x[k] = which == 0 ? Ks[(g * 8 + k) * 64 + m] : Vs[m * DV + g * 8 + k];
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              float acc = 0.f;
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float mij = bf16 ? round_to_bf16(mat[i * 4 + j]) : mat[i * 4 + j];
                acc = fmaf(mij, x[2 * j + r], acc);
              }
              y[2 * i + r] = bf16 ? round_to_bf16(acc) : acc;
            }
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            if (which == 0) Ks[(g * 8 + k) * 64 + m] = y[k]; else Vs[m * DV + g * 8 + k] = y[k];
          }
        }
      }
    }
    __syncthreads();
    // S = Q K^T
    float s[4][4] = {};
#pragma unroll 8
    for (int d = 0; d < DK; ++d) {
      float qa[4], kb[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) qa[i] = Qs[d * 64 + ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) kb[j] = Ks[d * 64 + tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = fmaf(qa[i], kb[j], s[i][j]);
    }
    float alpha[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = (t0 + tx * 4 + j < a.N) ? s[i][j] * a.scale : -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int off = 8; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      float m_new = fmaxf(m_run[i], mx);  // finite: every processed tile has a valid token
      alpha[i] = expf(m_run[i] - m_new);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float p = expf(s[i][j] - m_new);
        Ps[(ty * 4 + i) * 64 + tx * 4 + j] = p;
        sum += p;
      }
#pragma unroll
      for (int off = 8; off >= 1; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
      l_run[i] = l_run[i] * alpha[i] + sum;
      m_run[i] = m_new;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < OC; ++c) o[i][c] *= alpha[i];
#pragma unroll 4
    for (int t = 0; t < 64; ++t) {
      float p[4], vv[OC];
#pragma unroll
      for (int i = 0; i < 4; ++i) p[i] = Ps[(ty * 4 + i) * 64 + t];
#pragma unroll
      for (int c = 0; c < OC; ++c) vv[c] = Vs[t * DV + tx + 16 * c];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < OC; ++c) o[i][c] = fmaf(p[i], vv[c], o[i][c]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int qi = q0 + ty * 4 + i;
    if (qi >= a.Q) continue;
    float inv = l_run[i] > 0.f ? 1.0f / l_run[i] : 0.f;
    size_t row = static_cast<size_t>(qi) * a.heads + head;
#pragma unroll
    for (int c = 0; c < OC; ++c)
      store_float(a.out, a.dtype, row * DV + tx + 16 * c, o[i][c] * inv);
    if (tx == 0) a.lse[row] = l_run[i] > 0.f ? m_run[i] + logf(l_run[i]) : -INFINITY;
  }
}

template <int DK, int DV, bool CODEC>
int launch_attn(const AttnArgs& a, cudaStream_t stream) {
  size_t smem = sizeof(float) * (2 * DK * 64 + 64 * DV + 64 * 64 + 2 * BK * (BM + PAD));
  auto kernel = attn_kernel<DK, DV, CODEC>;
  NKV_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(smem)));
  dim3 grid(ceil_div(a.Q, 64), a.heads);
  kernel<<<grid, THREADS, smem, stream>>>(a);
  NKV_LAUNCH_CHECK("attn_kernel");
  return NKV_OK;
}

// -------------------------------------------------------------------- k-means
// One centre value as the assignment on the tensor cores takes it: three bf16 planes side by side along a row of
// [C, 3 J] (v = hi + mid + lo exactly, up to the last bit of the third).
__device__ __forceinline__ void split_planes(float v, uint16_t& hi, uint16_t& mid, uint16_t& lo) {
  hi = float_to_bf16_bits(v);
  const float r1 = __fsub_rn(v, bf16_bits_to_float(hi));
  mid = float_to_bf16_bits(r1);
  lo = float_to_bf16_bits(__fsub_rn(r1, bf16_bits_to_float(mid)));
}

__global__ void gather_init_kernel(const void* x, int x_dtype, int J, const int32_t* init_rows,
                                   float* centers, uint16_t* planes) {
  const int c = blockIdx.x, j = blockIdx.y * blockDim.x + threadIdx.x;
  if (j >= J) return;
  const float v = load_float(x, x_dtype, static_cast<size_t>(init_rows[c]) * J + j);
  centers[static_cast<size_t>(c) * J + j] = v;
  if (planes != nullptr) {
    uint16_t* out = planes + static_cast<size_t>(c) * 3 * J + j;
    split_planes(v, out[0], out[J], out[2 * J]);
  }
}

// The update: block (c, column block) sets centre c to the mean of the rows labelled c, summed in increasing token
// order (one fp32 addition per row, the order a sequential scatter-add takes) so that the result does not depend on
// the launch shape.  An empty cluster keeps its centre.  The new centre leaves as the next assignment's planes
// (`planes`) or as the stored centre (`stored`) too.
constexpr int UPDATE_SPAN = 8192;                       // labels taken at a time

// The tokens of [s0, s0 + len) labelled c, in order, into `list`; gives their number.  A warp looks at a run of labels,
// 128 at a time in whole lines (four per lane), keeps the matches as bits, and writes its tokens behind those of the
// warps before it.
template <int THREADS_>
__device__ __forceinline__ int list_members(const int32_t* labels, int s0, int len, int c, uint16_t* list, int* warp_total) {
  constexpr int WARPS_ = THREADS_ / 32;
  static_assert(UPDATE_SPAN / WARPS_ <= 16 * 128, "a lane keeps 16 times four matches");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rounds = (len + WARPS_ * 128 - 1) / (WARPS_ * 128), first = warp * rounds * 128 + lane * 4;
  const bool vector = (reinterpret_cast<uintptr_t>(labels) & 15) == 0;
  uint64_t match = 0;
#pragma unroll 4
  for (int r = 0; r < rounds; ++r) {
    const int at = first + r * 128;
    uint32_t m = 0;
    if (vector && at + 4 <= len) {
      const int4 l = __ldg(reinterpret_cast<const int4*>(labels + s0 + at));
      m = (l.x == c ? 1u : 0u) | (l.y == c ? 2u : 0u) | (l.z == c ? 4u : 0u) | (l.w == c ? 8u : 0u);
    } else {
      for (int i = 0; i < 4; ++i)
        if (at + i < len && __ldg(labels + s0 + at + i) == c) m |= 1u << i;
    }
    match |= static_cast<uint64_t>(m) << (4 * r);
  }
  const int mine = __reduce_add_sync(0xffffffffu, __popcll(match));
  __syncthreads();                                        // the previous list has been consumed
  if (lane == 0) warp_total[warp] = mine;
  __syncthreads();
  int base = 0, total = 0;
#pragma unroll
  for (int w = 0; w < WARPS_; ++w) {
    if (w < warp) base += warp_total[w];
    total += warp_total[w];
  }
  for (int r = 0; r < rounds; ++r) {
    const uint32_t m = static_cast<uint32_t>(match >> (4 * r)) & 15u;
    int before = 0, all = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint32_t votes = __ballot_sync(0xffffffffu, (m >> e) & 1u);
      before += __popc(votes & ((1u << lane) - 1u));
      all += __popc(votes);
    }
    int at = base + before;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if ((m >> e) & 1u) list[at++] = static_cast<uint16_t>(first + r * 128 + e);
    base += all;
  }
  __syncthreads();
  return total;
}

template <int COLS>
__device__ __forceinline__ void store_centre(const float (&sum)[COLS], int count, int c, int j, int J, float* centers,
                                             uint16_t* planes, uint16_t* stored) {
  float* centre = centers + static_cast<size_t>(c) * J + j;
  uint16_t* plane = planes == nullptr ? nullptr : planes + static_cast<size_t>(c) * 3 * J + j;
#pragma unroll
  for (int q = 0; q < COLS; ++q) {
    float v = 0.f;
    if (count > 0) {
      v = __fdiv_rn(sum[q], static_cast<float>(count));
      centre[q] = v;
      if (plane != nullptr) split_planes(v, plane[q], plane[J + q], plane[2 * J + q]);
    } else if (stored != nullptr) {
      v = centre[q];
    }
    if (stored != nullptr) stored[static_cast<size_t>(c) * J + j + q] = float_to_bf16_bits(v);
  }
}

// bf16 rows, four columns per thread.  Bound: the chain of row loads of the largest cluster -- start rows
// drawn from one true cluster leave others to be shared, so a cluster can hold several times the mean.  The members'
// pieces run through a ring in shared memory that every thread fills for itself: registers filled in
// turn share a handful of scoreboards, and waiting for one waits for the ones filled after it.
// us per call, 64 centres, 4,680 x 5,120 / 880 x 3,072 / 8,000 x 1,536: 41 / 9 / 52 with two columns per thread, 32 row
// loads at a time and a thread's labels side by side (32 lines per load of a warp); 35 / 9 / 42 with this ring in groups
// of four rows and labels in whole lines; 22 / 6 / 25 with groups of eight whose places come in one load.
// Threads past the last column copy nothing: copies of column 0 in their place cost 20,000 x 128 to 16 centres 214 us
// instead of 73, more than two columns per thread (132).  fp32 rows go two columns per thread: a ring for them
// holds 16 rows of 16 bytes a thread and was slower at every size (3,000 x 1,536 to 16 centres 21 us against 16, 9,500
// x 128 73 against 34).
constexpr int RING_THREADS = 128, RING_GROUP = 8, RING_GROUPS = 3;
__global__ void __launch_bounds__(RING_THREADS)
kmeans_update_ring_kernel(const uint16_t* x, int S, int J, const int32_t* labels, float* centers, uint16_t* planes,
                          uint16_t* stored) {
  constexpr int PIECE = 8;
  __shared__ __align__(16) uint16_t list[UPDATE_SPAN];
  __shared__ int warp_total[RING_THREADS / 32];
  __shared__ __align__(16) uint8_t ring[RING_GROUPS * RING_GROUP][RING_THREADS * PIECE];
  const int c = blockIdx.x, j = (blockIdx.y * RING_THREADS + threadIdx.x) * 4;
  const bool in = j < J;
  const uint8_t* column = reinterpret_cast<const uint8_t*>(x + (in ? j : 0));
  const uint32_t pitch = static_cast<uint32_t>(J) * 2;
  const uint32_t my_ring = static_cast<uint32_t>(__cvta_generic_to_shared(&ring[0][threadIdx.x * PIECE]));
  float sum[4] = {};
  int count = 0;
  for (int s0 = 0; s0 < S; s0 += UPDATE_SPAN) {
    const int total = list_members<RING_THREADS>(labels, s0, min(UPDATE_SPAN, S - s0), c, list, warp_total);
    count += total;
    if (!in) continue;
    auto copy = [&](uint32_t dst, uint32_t member) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(column + static_cast<uint64_t>(member) * pitch)
                   : "memory");
    };
    auto fetch = [&](int first, int slot) {       // members first .. first + RING_GROUP - 1, a group always
      const uint32_t dst = my_ring + slot * RING_GROUP * RING_THREADS * PIECE;
      if (first + RING_GROUP <= total) {
        const uint4 four = *reinterpret_cast<const uint4*>(list + first);
        const uint32_t pair[4] = {four.x, four.y, four.z, four.w};
#pragma unroll
        for (int k = 0; k < RING_GROUP; ++k)
          copy(dst + k * RING_THREADS * PIECE, s0 + ((k & 1) ? pair[k >> 1] >> 16 : pair[k >> 1] & 0xFFFFu));
      } else {
        for (int k = 0; first + k < total; ++k) copy(dst + k * RING_THREADS * PIECE, s0 + list[first + k]);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto add = [&](const uint8_t* piece) {
      const uint2 w = *reinterpret_cast<const uint2*>(piece);
      sum[0] = __fadd_rn(sum[0], __uint_as_float(w.x << 16));
      sum[1] = __fadd_rn(sum[1], __uint_as_float(w.x & 0xFFFF0000u));
      sum[2] = __fadd_rn(sum[2], __uint_as_float(w.y << 16));
      sum[3] = __fadd_rn(sum[3], __uint_as_float(w.y & 0xFFFF0000u));
    };
#pragma unroll
    for (int g = 0; g < RING_GROUPS; ++g) fetch(g * RING_GROUP, g);
    int slot = 0;
    for (int i = 0; i < total; i += RING_GROUP) {
      asm volatile("cp.async.wait_group %0;" ::"n"(RING_GROUPS - 1) : "memory");
      const uint8_t* piece = &ring[slot * RING_GROUP][threadIdx.x * PIECE];
      if (i + RING_GROUP <= total) {
#pragma unroll
        for (int k = 0; k < RING_GROUP; ++k) add(piece + k * RING_THREADS * PIECE);
      } else {
        for (int k = 0; i + k < total; ++k) add(piece + k * RING_THREADS * PIECE);
      }
      fetch(i + RING_GROUPS * RING_GROUP, slot);
      if (++slot == RING_GROUPS) slot = 0;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  if (in) store_centre(sum, count, c, j, J, centers, planes, stored);
}

// Other rows: two columns per thread (rows of even length on their own multiple), or one column of any type, 32 row
// loads at a time.
struct PairBf16 {
  static constexpr int COLS = 2;
  uint32_t w;
  __device__ __forceinline__ void load(const void* base, int, size_t i) {
    w = __ldg(reinterpret_cast<const uint32_t*>(static_cast<const uint16_t*>(base) + i));
  }
  __device__ __forceinline__ float value(int k) const { return __uint_as_float(k ? w & 0xFFFF0000u : w << 16); }
};
struct PairF32 {
  static constexpr int COLS = 2;
  float2 v;
  __device__ __forceinline__ void load(const void* base, int, size_t i) {
    v = __ldg(reinterpret_cast<const float2*>(static_cast<const float*>(base) + i));
  }
  __device__ __forceinline__ float value(int k) const { return k ? v.y : v.x; }
};
struct Single {
  static constexpr int COLS = 1;
  float v;
  __device__ __forceinline__ void load(const void* base, int dtype, size_t i) { v = load_float(base, dtype, i); }
  __device__ __forceinline__ float value(int) const { return v; }
};

constexpr int UPDATE_FLIGHT = 32;                       // row loads in flight per thread
template <class Columns>
__global__ void __launch_bounds__(256)
kmeans_update_kernel(const void* x, int x_dtype, int S, int J, const int32_t* labels,
                     float* centers, uint16_t* planes, uint16_t* stored) {
  __shared__ uint16_t list[UPDATE_SPAN];
  __shared__ int warp_total[8];
  constexpr int COLS = Columns::COLS;
  const int c = blockIdx.x, j = (blockIdx.y * 256 + threadIdx.x) * COLS;
  float sum[COLS] = {};
  int count = 0;
  for (int s0 = 0; s0 < S; s0 += UPDATE_SPAN) {
    const int total = list_members<256>(labels, s0, min(UPDATE_SPAN, S - s0), c, list, warp_total);
    count += total;
    if (j < J) {
      for (int i = 0; i < total; i += UPDATE_FLIGHT) {
        Columns v[UPDATE_FLIGHT];
#pragma unroll
        for (int k = 0; k < UPDATE_FLIGHT; ++k)
          if (i + k < total) v[k].load(x, x_dtype, static_cast<size_t>(s0 + list[i + k]) * J + j);
#pragma unroll
        for (int k = 0; k < UPDATE_FLIGHT; ++k)
          if (i + k < total) {
#pragma unroll
            for (int q = 0; q < COLS; ++q) sum[q] = __fadd_rn(sum[q], v[k].value(q));
          }
      }
    }
  }
  if (j < J) store_centre(sum, count, c, j, J, centers, planes, stored);
}

__global__ void kmeans_store_kernel(const float* centers, const int32_t* labels, int S, size_t CJ,
                                    uint16_t* centers_bf16, void* ids, int id_bytes) {
  size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < CJ) centers_bf16[i] = float_to_bf16_bits(centers[i]);
  if (i < static_cast<size_t>(S)) {
    if (id_bytes == 1) static_cast<uint8_t*>(ids)[i] = static_cast<uint8_t>(labels[i]);
    else static_cast<uint16_t*>(ids)[i] = static_cast<uint16_t>(labels[i]);
  }
}

}  // namespace

int simt_attn(const void* q, int dtype, int64_t q_stride_token, int64_t q_stride_head, int Q,
              int heads, int dk, int dv, const nkv_history* hist_k, const nkv_history* hist_v,
              const void* wk, const float* bias_k, const void* wv, const float* bias_v,
              const void* k_plain, const void* v_plain, int64_t kv_stride_token,
              int64_t kv_stride_head, int N, float scale, void* out, float* lse,
              cudaStream_t stream, const nkv_rope* rope, const nkv_camera* cam_k,
              const nkv_camera* cam_v) {
  if (Q == 0 || heads == 0) return NKV_OK;
  AttnArgs a{};
  if (rope != nullptr) a.rope = *rope;
  if (cam_k != nullptr) a.cam_k = *cam_k;
  if (cam_v != nullptr) a.cam_v = *cam_v;
  a.q = q; a.dtype = dtype; a.q_stride_token = q_stride_token; a.q_stride_head = q_stride_head;
  a.Q = Q; a.heads = heads; a.N = N; a.scale = scale;
  const bool codec = hist_k != nullptr;
  if (codec) { a.hk = *hist_k; a.hv = *hist_v; }
  a.wk = wk; a.bias_k = bias_k; a.wv = wv; a.bias_v = bias_v;
  a.k_plain = k_plain; a.v_plain = v_plain;
  a.kv_stride_token = kv_stride_token; a.kv_stride_head = kv_stride_head;
  a.out = out; a.lse = lse;
#define NKV_ATTN_CASE(DK_, DV_)                                            \
  if (dk == DK_ && dv == DV_)                                              \
    return codec ? launch_attn<DK_, DV_, true>(a, stream) : launch_attn<DK_, DV_, false>(a, stream);
  NKV_ATTN_CASE(128, 128)
  NKV_ATTN_CASE(64, 64)
  NKV_ATTN_CASE(32, 32)
  NKV_ATTN_CASE(16, 16)
#undef NKV_ATTN_CASE
  return fail(NKV_ERR_UNSUPPORTED, "attention head widths dk=%d dv=%d (built: 16, 32, 64, 128 with dk == dv)", dk, dv);
}

// camera transform of explicit rows: thread = one (row, head, 8-wide block)
__global__ void __launch_bounds__(256)
camera_rows_kernel(const void* x, int dtype, long long stride_row, long long stride_head, int S,
                   int heads, int d, nkv_camera cam, void* out) {
  const int blocks = d / 8;
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= static_cast<long long>(S) * heads * blocks) return;
  const int g = static_cast<int>(idx % blocks);
  const int head = static_cast<int>((idx / blocks) % heads);
  const int row = static_cast<int>(idx / (static_cast<long long>(blocks) * heads));
  const int frame = min(row / cam.tokens_per_frame, cam.frames - 1);
  const float* mat = cam.matrices + (static_cast<size_t>(frame) * 4 + (cam.cam_index[head * blocks + g] & 3)) * 16;
  const bool bf16 = dtype == NKV_BF16;
  const size_t src = static_cast<size_t>(row) * stride_row + static_cast<size_t>(head) * stride_head + g * 8;
  const size_t dst = (static_cast<size_t>(row) * heads + head) * d + g * 8;
  float v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = load_float(x, dtype, src + k);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float acc = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        acc = fmaf(bf16 ? round_to_bf16(mat[i * 4 + j]) : mat[i * 4 + j], v[2 * j + r], acc);
      store_float(out, dtype, dst + 2 * i + r, acc);
    }
}

int camera_rows(const void* x, int dtype, int64_t stride_row, int64_t stride_head, int S, int heads,
                int d, const nkv_camera& camera, void* out, cudaStream_t stream) {
  const long long total = static_cast<long long>(S) * heads * (d / 8);
  if (total == 0) return NKV_OK;
  camera_rows_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, stream>>>(
      x, dtype, stride_row, stride_head, S, heads, d, camera, out);
  NKV_LAUNCH_CHECK("camera_rows_kernel");
  return NKV_OK;
}

// rotation of explicit rows: thread = four adjacent pairs (8 elements) of one (row, head)
__global__ void __launch_bounds__(256)
rope_rows_kernel(const void* x, int dtype, long long stride_row, long long stride_head, int S,
                 int heads, int d, nkv_rope rope, void* out, int vector) {
  const int half = d / 2, quads = half / 4 + (half % 4 ? 1 : 0);
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= static_cast<long long>(S) * heads * quads) return;
  const int pl0 = static_cast<int>(idx % quads) * 4;
  const int head = static_cast<int>((idx / quads) % heads);
  const int row = static_cast<int>(idx / (static_cast<long long>(quads) * heads));
  const int th = rope.table_half, third = th / 3, band_a = th - 2 * third, band_b = band_a + third;
  const int pos = max(rope.positions[row], 0);
  int frame = pos, prow = pos, pcol = pos;   // frame_seqlen 0: one table row per token
  if (rope.frame_seqlen > 0) {
    frame = pos / rope.frame_seqlen;
    const int spatial = pos - frame * rope.frame_seqlen;
    prow = spatial / rope.width;
    pcol = spatial - prow * rope.width;
  }
  const size_t src = static_cast<size_t>(row) * stride_row + static_cast<size_t>(head) * stride_head + 2 * pl0;
  const size_t dst = (static_cast<size_t>(row) * heads + head) * d + 2 * pl0;
  float v[8];
  const int count = min(4, half - pl0);
  if (vector && dtype == NKV_BF16) {
    const uint4 raw = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(x) + src);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[2 * k] = __uint_as_float(w[k] << 16);
      v[2 * k + 1] = __uint_as_float(w[k] & 0xFFFF0000u);
    }
  } else {
    for (int k = 0; k < 2 * count; ++k) v[k] = load_float(x, dtype, src + k);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k >= count) break;
    const int pl = pl0 + k;
    const int pg = rope.pair_index ? rope.pair_index[head * half + pl] : pl;
    int coord = pg < band_a ? frame : (pg < band_b ? prow : pcol);
    coord = min(coord, rope.table_rows - 1);
    const float2 cs = reinterpret_cast<const float2*>(rope.cos_sin)[static_cast<size_t>(coord) * th + pg];
    const float x0 = v[2 * k], x1 = v[2 * k + 1];
    v[2 * k] = fmaf(x0, cs.x, -(x1 * cs.y));
    v[2 * k + 1] = fmaf(x0, cs.y, x1 * cs.x);
  }
  if (vector && dtype == NKV_BF16) {
    uint4 packed;
    packed.x = float_to_bf16_bits(v[0]) | (static_cast<uint32_t>(float_to_bf16_bits(v[1])) << 16);
    packed.y = float_to_bf16_bits(v[2]) | (static_cast<uint32_t>(float_to_bf16_bits(v[3])) << 16);
    packed.z = float_to_bf16_bits(v[4]) | (static_cast<uint32_t>(float_to_bf16_bits(v[5])) << 16);
    packed.w = float_to_bf16_bits(v[6]) | (static_cast<uint32_t>(float_to_bf16_bits(v[7])) << 16);
    *reinterpret_cast<uint4*>(static_cast<uint16_t*>(out) + dst) = packed;
  } else {
    for (int k = 0; k < 2 * count; ++k) store_float(out, dtype, dst + k, v[k]);
  }
}

// The same for bf16 rows whose heads share their rotation (no pair index) and start on 16 bytes: a thread keeps the four
// entries of its pairs and takes ROPE_HEADS heads, all loads ahead of the arithmetic.  Bound: memory; with one
// thread per head and piece the coordinates, divisions and table loads were the time.  4,680 x 40 x 128: 48 us, now 26.
constexpr int ROPE_HEADS = 8;
__global__ void __launch_bounds__(256)
rope_rows_heads_kernel(const uint16_t* x, long long stride_row, long long stride_head, int S, int heads, int d,
                       nkv_rope rope, uint16_t* out) {
  const int quads = d / 8, index = blockIdx.x * 256 + threadIdx.x;
  const int row = index / quads, pl0 = (index - row * quads) * 4;
  if (row >= S) return;
  const int th = rope.table_half, third = th / 3, band_a = th - 2 * third, band_b = band_a + third;
  const int pos = max(__ldg(rope.positions + row), 0);
  int frame = pos, prow = pos, pcol = pos;   // frame_seqlen 0: one table row per token
  if (rope.frame_seqlen > 0) {
    frame = pos / rope.frame_seqlen;
    const int spatial = pos - frame * rope.frame_seqlen;
    prow = spatial / rope.width;
    pcol = spatial - prow * rope.width;
  }
  float2 cs[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int pg = pl0 + k;
    const int coord = min(pg < band_a ? frame : (pg < band_b ? prow : pcol), rope.table_rows - 1);
    cs[k] = __ldg(reinterpret_cast<const float2*>(rope.cos_sin) + static_cast<size_t>(coord) * th + pg);
  }
  const int first = blockIdx.y * ROPE_HEADS;
  const uint16_t* src = x + static_cast<size_t>(row) * stride_row + static_cast<size_t>(first) * stride_head + 2 * pl0;
  uint16_t* dst = out + (static_cast<size_t>(row) * heads + first) * d + 2 * pl0;
  uint4 raw[ROPE_HEADS];
#pragma unroll
  for (int h = 0; h < ROPE_HEADS; ++h)
    if (first + h < heads) raw[h] = __ldg(reinterpret_cast<const uint4*>(src + h * stride_head));
#pragma unroll
  for (int h = 0; h < ROPE_HEADS; ++h) {
    if (first + h >= heads) break;
    const uint32_t w[4] = {raw[h].x, raw[h].y, raw[h].z, raw[h].w};
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float x0 = __uint_as_float(w[k] << 16), x1 = __uint_as_float(w[k] & 0xFFFF0000u);
      const __nv_bfloat162 both = __floats2bfloat162_rn(fmaf(x0, cs[k].x, -(x1 * cs[k].y)), fmaf(x0, cs[k].y, x1 * cs[k].x));
      o[k] = *reinterpret_cast<const uint32_t*>(&both);
    }
    *reinterpret_cast<uint4*>(dst + static_cast<size_t>(h) * d) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

int rope_rows(const void* x, int dtype, int64_t stride_row, int64_t stride_head, int S, int heads,
              int d, const nkv_rope& rope, void* out, cudaStream_t stream) {
  const int half = d / 2, quads = half / 4 + (half % 4 ? 1 : 0);
  const long long total = static_cast<long long>(S) * heads * quads;
  if (total == 0) return NKV_OK;
  // 16-byte path: whole groups of 8 elements, every row and head start 16-byte aligned
  const int vector = d % 8 == 0 && stride_row % 8 == 0 && stride_head % 8 == 0 &&
                     ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  if (vector && dtype == NKV_BF16 && rope.pair_index == nullptr && (reinterpret_cast<uintptr_t>(rope.cos_sin) & 7) == 0 &&
      static_cast<long long>(S) * quads < (1ll << 31) - 256) {
    rope_rows_heads_kernel<<<dim3(ceil_div(S * quads, 256), ceil_div(heads, ROPE_HEADS)), 256, 0, stream>>>(
        static_cast<const uint16_t*>(x), stride_row, stride_head, S, heads, d, rope, static_cast<uint16_t*>(out));
    NKV_LAUNCH_CHECK("rope_rows_heads_kernel");
    return NKV_OK;
  }
  rope_rows_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, stream>>>(
      x, dtype, stride_row, stride_head, S, heads, d, rope, out, vector);
  NKV_LAUNCH_CHECK("rope_rows_kernel");
  return NKV_OK;
}

int kmeans_gather_init(const void* x, int x_dtype, int J, int C, const int32_t* init_rows,
                       float* centers, uint16_t* planes, cudaStream_t stream) {
  gather_init_kernel<<<dim3(C, ceil_div(J, 256)), 256, 0, stream>>>(x, x_dtype, J, init_rows, centers, planes);
  NKV_LAUNCH_CHECK("gather_init_kernel");
  return NKV_OK;
}

int kmeans_update(const void* x, int x_dtype, int S, int J, int C, const int32_t* labels,
                  float* centers, uint16_t* planes, uint16_t* stored, cudaStream_t stream) {
  // four columns per thread for bf16 rows that start on a multiple of that many, two for the others and for fp32; every
  // other form (fp16 rows among them) one column, converted by load_float
  const bool bf16 = x_dtype == NKV_BF16, f32 = x_dtype == NKV_F32;
  auto fits = [&](int columns) { return J % columns == 0 && reinterpret_cast<uintptr_t>(x) % (columns * (f32 ? 4 : 2)) == 0; };
  if (bf16 && fits(4)) {
    kmeans_update_ring_kernel<<<dim3(C, ceil_div(J, 4 * RING_THREADS)), RING_THREADS, 0, stream>>>(
        static_cast<const uint16_t*>(x), S, J, labels, centers, planes, stored);
  } else {
    const bool pairs = (bf16 || f32) && fits(2);
    const dim3 grid(C, ceil_div(J, pairs ? 512 : 256));
    auto kernel = !pairs ? kmeans_update_kernel<Single> : (f32 ? kmeans_update_kernel<PairF32> : kmeans_update_kernel<PairBf16>);
    kernel<<<grid, 256, 0, stream>>>(x, x_dtype, S, J, labels, centers, planes, stored);
  }
  NKV_LAUNCH_CHECK("kmeans_update_kernel");
  return NKV_OK;
}

int kmeans_store(const float* centers, const int32_t* labels, int S, int J, int C,
                 void* centers_bf16, void* ids, int id_bytes, cudaStream_t stream) {
  size_t CJ = static_cast<size_t>(C) * J;
  size_t total = CJ > static_cast<size_t>(S) ? CJ : static_cast<size_t>(S);
  kmeans_store_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, stream>>>(
      centers, labels, S, CJ, static_cast<uint16_t*>(centers_bf16), ids, id_bytes);
  NKV_LAUNCH_CHECK("kmeans_store_kernel");
  return NKV_OK;
}

}  // namespace nkv
