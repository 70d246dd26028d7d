// Rows of a compressed history rebuilt on tcgen05 tensor cores, one or two tensors per launch:
//   row[t] = bf16(bf16(latent[t] decoder^T + bias) + centre[t]),  latent[t] = bf16(code * scale),
// plus the positional restore (rotation, camera transform) where the caller asks for it.
//
// The product is [n tokens x rank] x [J x rank]^T.  A cluster of two CTAs owns a tile of 256 tokens
// (128 per CTA) and computes 256 columns of J at a time with cta_group::2 MMAs: the tile's codes are
// expanded ONCE into bf16 latents that stay in shared memory for all of its columns (160 KB at rank
// 640), and only decoder rows are streamed (TMA, each CTA of a pair loads half of the 256 rows, so a
// pair reads every decoder byte once per 256 tokens: 64 bytes per clock and SM at the full MMA rate;
// one CTA on its own would need 128, which the L2 does not deliver to 148 SMs).  Two accumulators of
// 256 columns in TMEM: the epilogue of a tile runs under the MMAs of the next one.
//
// Work is the list of (tensor, 256-token tile, 256-column tile) in that order; every cluster takes a
// contiguous run of equal length, so the last wave is never emptier than one tile and a run expands
// two or three token tiles.  No wait crosses clusters.  A wait that gives up leaves its site in the status
// word and in the block's word of `failed` (which the attention behind a decode reads), and the rows that
// were not finished become NaN.
//
// Bound: the epilogue's chain of latencies per 32 columns (accumulator read, staging, store; without it the
// same launch takes 145 us), then the decoder stream into three 16 KB stages, all that 160 KB of latents
// leave at rank 640.  28,080 rows x 5,120 columns at rank 640: 191 us = 964 TFLOP/s; 255 with cluster-scope
// waits and releases on every hand-off, bias and centres loaded where they are used, and the centres
// staged; the CUDA-core kernel that served bf16 operators before took 8.9 ms.
//
// Warps 0-7: expansion and epilogue (warp w serves TMEM lanes 32 (w & 3) .. and column half w >> 2),
// warp 8 lane 0: TMA, warp 9 of the even CTA: MMA.
#include "nkv_internal.h"
#include "nkv_tc.cuh"
#include "nkv_tc_dequant.cuh"

namespace nkv {
namespace {

using namespace tc;

constexpr int TM = 128;                     // tokens per CTA (256 per cluster)
constexpr int TN = 256;                     // columns per accumulator
constexpr int COMPUTE_WARPS = 8;
constexpr int THREADS = COMPUTE_WARPS * 32 + 64;
constexpr int CHUNK_BYTES = TM * 128;       // [128 rows x 64 bf16], 128-byte swizzle
constexpr int MAX_CHUNKS = 10;              // rank <= 640
constexpr int MAX_STAGES = 8;
constexpr int META = 1024;
constexpr int SCRATCH = COMPUTE_WARPS * 2048;
constexpr size_t SMEM_LIMIT = 232448;

constexpr int A_GROUP = 5;                  // latent chunks handed over together
enum Bar { FULL = 0, FREE = 8, A_FULL = 16, ACC_FULL = 18, ACC_FREE = 20, NUM_BARS = 22 };

struct Tensor {
  nkv_history h;
  const float* bias;
  const int32_t* rows;        // listed rows, or NULL: rows 0 .. n
  uint16_t* out;              // element (row, head, column): row * row_stride + head * head_stride + column
  long long row_stride, head_stride;
  nkv_rope rope;              // cos_sin == NULL: none
  nkv_camera cam;             // matrices == NULL: none
};

struct Params {
  Tensor t[2];
  int tensors, n, J, D, nchunks, ngroups, group, w_perm, round_bias, nstages;
  int rope_pairs;             // rotation tables may be read two pairs (16 bytes) at a time
  int m_tiles, n_tiles, total;
  int32_t* status;
  int32_t* failed;            // one word per block, written by every launch: 0, or the site of a wait that gave up; NULL: none
  long long wait_budget;      // SM cycles per wait
  int starve;                 // self-test: no decoder row is loaded, so that the waits for them run out
};

__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y,
                                                 uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar_cluster_addr)
      : "memory");
}

__device__ __forceinline__ void tmem_alloc_pair(uint32_t* slot_in_smem, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(slot_in_smem)), "r"(columns) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t columns) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns)
               : "memory");
}
// D[256 x N over the pair] (+)= A B^T; each CTA holds its 128 rows of A and half of B's rows
__device__ __forceinline__ void mma_bf16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                              uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(static_cast<uint32_t>(accumulate))
      : "memory");
}
// one arrival on the barrier at this offset in both CTAs of the pair once the MMAs issued so far are done
__device__ __forceinline__ void mma_commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64"
      " [%0], %1;" ::"r"(smem_u32(bar)), "h"(static_cast<uint16_t>(3))
      : "memory");
}

__device__ __forceinline__ uint4 add_bf16x8(uint4 a, const uint4& b) {
  uint32_t* x = &a.x;
  const uint32_t* y = &b.x;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 sum = __hadd2(*reinterpret_cast<const __nv_bfloat162*>(x + i),
                                       *reinterpret_cast<const __nv_bfloat162*>(y + i));
    x[i] = *reinterpret_cast<const uint32_t*>(&sum);
  }
  return a;
}

// a run of column tiles of one token tile
struct Run { int tensor, m, nt0, count; };
__device__ __forceinline__ Run run_at(const Params& p, int w, int w_end) {
  Run r;
  const int seg = w / p.n_tiles;
  r.nt0 = w - seg * p.n_tiles;
  r.count = min(p.n_tiles - r.nt0, w_end - w);
  r.tensor = seg / p.m_tiles;
  r.m = seg - r.tensor * p.m_tiles;
  return r;
}

// Arrival that hands back tensor memory whose loads have completed: nothing written is published by it, so
// it does not wait for the stores under way (a releasing arrival would: a tile's rows to L2, every tile).
__device__ __forceinline__ void arrive_relaxed(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}

// history row of row `row` of this CTA's tile, or -1 past the end of the list
__device__ __forceinline__ int token_at(const Params& p, const Run& r, uint32_t cta, int row) {
  const int m = (r.m * 2 + static_cast<int>(cta)) * TM + row;
  if (m >= p.n) return -1;
  const Tensor& t = p.t[r.tensor];
  const int tok = t.rows != nullptr ? __ldg(t.rows + m) : m;
  return tok < 0 || tok >= t.h.tokens ? -1 : tok;
}

// After a wait gave up: NaN in this thread's row and column half of the tiles [w, w_end) it did not finish, so
// that nothing unwritten looks like a result.
__device__ __noinline__ void fill_unfinished(const Params& p, int w, int w_end, uint32_t cta, int row, int wg) {
  const uint32_t nan2 = 0x7FC07FC0u;
  for (; w < w_end; ++w) {
    const Run r = run_at(p, w, w_end);
    if (token_at(p, r, cta, row) < 0) continue;
    const Tensor& t = p.t[r.tensor];
    const int m = (r.m * 2 + static_cast<int>(cta)) * TM + row, first = r.nt0 * TN + wg * 128;
    for (int col = first; col < min(first + 128, p.J); col += 8) {
      const int head = col / p.D;
      *reinterpret_cast<uint4*>(t.out + static_cast<size_t>(m) * t.row_stride + head * t.head_stride + (col - head * p.D)) =
          make_uint4(nan2, nan2, nan2, nan2);
    }
  }
}

template <bool ROPE, bool CAM>
__global__ void __launch_bounds__(THREADS, 1)
decode_gemm_kernel(const __grid_constant__ CUtensorMap map_0, const __grid_constant__ CUtensorMap map_1,
                   const __grid_constant__ Params p) {
  constexpr bool POS = ROPE || CAM;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + NUM_BARS * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + NUM_BARS * 8 + 4);
  uint8_t* a_tiles = smem + META;
  uint8_t* b_tiles = a_tiles + p.nchunks * CHUNK_BYTES;
  uint8_t* scratch = b_tiles + p.nstages * CHUNK_BYTES;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t cta = cluster_ctarank();
  const int clusters = gridDim.x >> 1, cluster = blockIdx.x >> 1;
  const int w_begin = static_cast<int>(static_cast<long long>(p.total) * cluster / clusters);
  const int w_end = static_cast<int>(static_cast<long long>(p.total) * (cluster + 1) / clusters);
  const int nst = p.nstages, nchunks = p.nchunks;

  if (tid == 0) {
    for (int s = 0; s < MAX_STAGES; ++s) {
      mbar_init(&bars[FULL + s], 1);
      mbar_init(&bars[FREE + s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars[A_FULL + b], 2 * COMPUTE_WARPS);
      mbar_init(&bars[ACC_FULL + b], 1);
      mbar_init(&bars[ACC_FREE + b], 2 * COMPUTE_WARPS);
    }
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 9) tmem_alloc_pair(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();      // the peer's barriers exist before anyone arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 8) {
    // ---------------------------------------------------------------- TMA: decoder rows
    if (lane == 0) {
      prefetch_tensormap(&map_0);
      if (p.tensors > 1) prefetch_tensormap(&map_1);
      const uint32_t full_even = map_to_cta(smem_u32(&bars[FULL]), 0);
      bool ok = true;
      int s = 0, phase = 0;
      bool wrapped = false;        // the ring has been filled once: stages must be handed back first
      for (int w = p.starve ? w_end : w_begin; w < w_end && ok;) {
        const Run r = run_at(p, w, w_end);
        const CUtensorMap* map = r.tensor ? &map_1 : &map_0;
        for (int k = 0; k < r.count && ok; ++k) {
          const int y = (r.nt0 + k) * TN + static_cast<int>(cta) * TM;
          for (int c = 0; c < nchunks; ++c) {
            if (wrapped) ok = mbar_wait(&bars[FREE + s], phase ^ 1, abort_flag, 700 + s, p.wait_budget);
            if (!ok) break;
            // both halves land on the even CTA's barrier, whose MMA warp reads them
            if (cta == 0) mbar_arrive_expect_tx(&bars[FULL + s], 2 * CHUNK_BYTES);
            tma_load_2d_pair(b_tiles + s * CHUNK_BYTES, map, c * 64, y, full_even + s * 8);
            if (++s == nst) { s = 0; phase ^= 1; wrapped = true; }
          }
        }
        w += r.count;
      }
      if (!ok) {   // let copies already in flight land before the CTA goes away
        const long long start = clock64();
        while (clock64() - start < (1ll << 21)) {}
      }
    }
    __syncwarp();
  } else if (warp == 9) {
    if (cta == 0) {
      // -------------------------------------------------------------- MMA issuer of the pair
      const bool leader = elect_one();
      const uint32_t idesc = make_idesc_bf16(2 * TM, TN);
      const uint32_t a_base = smem_u32(a_tiles), b_base = smem_u32(b_tiles);
      bool ok = true;
      int s = 0, phase = 0, tile = 0, seg = 0;   // the ring's place is counted: no division per stage
      for (int w = w_begin; w < w_end && ok; ++seg) {
        const Run r = run_at(p, w, w_end);
        for (int k = 0; k < r.count && ok; ++k, ++tile) {
          const int b = tile & 1, use = tile >> 1;
          if (use >= 1) ok = wait_all(&bars[ACC_FREE + b], (use - 1) & 1, abort_flag, 710 + b, p.wait_budget);
          const uint32_t acc = tmem_base + b * TN;
          for (int c = 0; c < nchunks && ok; ++c) {
            if (k == 0 && c % A_GROUP == 0)
              ok = wait_all_cluster(&bars[A_FULL + c / A_GROUP], seg & 1, abort_flag, 720 + c, p.wait_budget);
            ok = ok && wait_all(&bars[FULL + s], phase, abort_flag, 730 + s, p.wait_budget);
            if (!ok) break;
            tc_fence_after();
            const uint64_t a_desc = make_smem_desc_sw128(a_base + c * CHUNK_BYTES);
            const uint64_t b_desc = make_smem_desc_sw128(b_base + s * CHUNK_BYTES);
            if (leader) {
              mma_bf16_pair(acc, a_desc, b_desc, idesc, c > 0);
              mma_bf16_pair(acc, a_desc + 2, b_desc + 2, idesc, true);
              mma_bf16_pair(acc, a_desc + 4, b_desc + 4, idesc, true);
              mma_bf16_pair(acc, a_desc + 6, b_desc + 6, idesc, true);
              mma_commit_pair(&bars[FREE + s]);
            }
            __syncwarp();
            if (++s == nst) { s = 0; phase ^= 1; }
          }
          if (ok && leader) mma_commit_pair(&bars[ACC_FULL + b]);
          __syncwarp();
        }
        w += r.count;
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ expansion and epilogue
    const int row = tid & 127, wg = tid >> 7, wrow0 = 32 * (warp & 3);
    const uint32_t lane_sel = static_cast<uint32_t>(wrow0) << 16;
    uint8_t* stage = scratch + warp * 2048;
    bool ok = true;
    int tile = 0;                       // tiles whose epilogue is done or pending, in order
    // this thread's codes of its token, 16 bytes of every chunk, with their scales
    struct Codes { uint4 word[MAX_CHUNKS]; uint16_t scale[MAX_CHUNKS]; };
    auto fetch_codes = [&](const Run& r, int tok, Codes& in) {
      const nkv_history& h = p.t[r.tensor].h;
      const uint8_t* codes = h.codes + static_cast<size_t>(tok < 0 ? 0 : tok) * (h.rank >> 1) + wg * 16;
      const uint16_t* scales = static_cast<const uint16_t*>(h.scales) + static_cast<size_t>(tok < 0 ? 0 : tok) * p.ngroups;
#pragma unroll
      for (int c = 0; c < MAX_CHUNKS; ++c) {
        in.word[c] = make_uint4(0, 0, 0, 0);
        in.scale[c] = 0;
        if (c < nchunks && tok >= 0) {
          in.word[c] = __ldg(reinterpret_cast<const uint4*>(codes + c * 32));
          in.scale[c] = __ldg(scales + (p.ngroups == 1 ? 0 : (c * 64 + wg * 32) / p.group));
        }
      }
    };
    auto expand = [&](const Run& r, const Codes& in) {
      const int scale_dtype = p.t[r.tensor].h.scale_dtype;
#pragma unroll
      for (int c = 0; c < MAX_CHUNKS; ++c) {
        if (c >= nchunks) break;
        const uint32_t words[4] = {in.word[c].x, in.word[c].y, in.word[c].z, in.word[c].w};
        uint8_t* dst = a_tiles + c * CHUNK_BYTES;
        const uint32_t pair = static_cast<uint32_t>(in.scale[c]) * 0x00010001u;
        const __nv_bfloat162 scale2 = *reinterpret_cast<const __nv_bfloat162*>(&pair);
        const float sc = scale_to_float(in.scale[c], scale_dtype);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          uint4 v;
          if (scale_dtype == NKV_BF16) v = p.w_perm ? dequant8_bf16_perm(words[k], scale2) : dequant8_bf16(words[k], scale2);
          else v = p.w_perm ? dequant8_perm(words[k], sc) : dequant8(words[k], sc);
          *reinterpret_cast<uint4*>(dst + sw128_offset(row, wg * 32 + k * 8)) = v;
        }
        if (c % A_GROUP == A_GROUP - 1 || c == nchunks - 1) {
          fence_proxy_async();             // the pair's MMAs read this through the async proxy
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&bars[A_FULL + c / A_GROUP]), 0));
        }
      }
    };
    // columns [n0 + 128 wg, +128) of this warp's 32 rows, 32 columns at a time
    auto epilogue = [&](const Run& r, int nt, int tok, int crow) {
      const Tensor& t = p.t[r.tensor];
      const int b = tile & 1, use = tile >> 1;
      const int m0 = (r.m * 2 + static_cast<int>(cta)) * TM + wrow0;
      const int rounds = min(4, max(0, (p.J - nt * TN - wg * 128) / 32));
      // centre rows: 4 lanes read the 16-byte pieces of one row, 8 rows per load instruction.  Centres and
      // bias of a round are requested a round ahead (the first ones ahead of the accumulator wait): next to
      // 220 KB of shared memory the first-level cache holds neither.
      int crow_of[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) crow_of[i] = __shfl_sync(0xffffffffu, tok < 0 ? -1 : crow, i * 8 + lane / 4);
      auto load_centers = [&](int sub, uint4 (&dst)[4]) {
        const uint16_t* cbase = static_cast<const uint16_t*>(t.h.centers) + nt * TN + wg * 128 + sub * 32 + (lane & 3) * 8;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          dst[i] = make_uint4(0, 0, 0, 0);
          if (sub < rounds && crow_of[i] >= 0)
            dst[i] = __ldg(reinterpret_cast<const uint4*>(cbase + static_cast<size_t>(crow_of[i]) * t.h.center_width));
        }
      };
      // bias of a round's 32 columns (the same for every lane)
      auto load_bias = [&](int sub, float4 (&dst)[8]) {
        if (sub >= rounds) return;
        const float4* src = reinterpret_cast<const float4*>(t.bias + nt * TN + wg * 128 + sub * 32);
#pragma unroll
        for (int j = 0; j < 8; ++j) dst[j] = __ldg(src + j);
      };
      uint4 cen[4];
      float4 bias[POS ? 1 : 8];
      float bias_lane[POS ? 4 : 1];
      load_centers(0, cen);
      if constexpr (POS) {
        // the registers hold rotation entries instead: a lane keeps one column of every round, rounded once, and the
        // lanes share theirs through the staging area
#pragma unroll
        for (int sub = 0; sub < 4; ++sub) {
          bias_lane[sub] = sub < rounds ? __ldg(t.bias + nt * TN + wg * 128 + sub * 32 + lane) : 0.f;
          if (p.round_bias) bias_lane[sub] = round_to_bf16(bias_lane[sub]);
        }
      } else {
        load_bias(0, bias);
      }
      // positional restore: table rows and frame of the four tokens this lane stores a piece of
      const bool rotate = ROPE && t.rope.cos_sin != nullptr;
      const bool transform = CAM && t.cam.matrices != nullptr;
      const int band_a = t.rope.table_half - 2 * (t.rope.table_half / 3);
      const int band_b = band_a + t.rope.table_half / 3;
      int coord_t[4], coord_h[4], coord_w[4], frame_of[4];
      if (rotate) {
        const int pos = tok >= 0 ? max(__ldg(t.rope.positions + tok), 0) : 0;
        const int last = t.rope.table_rows - 1;
        int ct = min(pos, last), ch = ct, cw = ct;   // frame_seqlen 0: one table row per token
        if (t.rope.frame_seqlen > 0) {
          const int frame = pos / t.rope.frame_seqlen, spatial = pos - frame * t.rope.frame_seqlen;
          const int prow = spatial / t.rope.width;
          ct = min(frame, last);
          ch = min(prow, last);
          cw = min(spatial - prow * t.rope.width, last);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          coord_t[i] = __shfl_sync(0xffffffffu, ct, i * 8 + lane / 4) * t.rope.table_half;
          coord_h[i] = __shfl_sync(0xffffffffu, ch, i * 8 + lane / 4) * t.rope.table_half;
          coord_w[i] = __shfl_sync(0xffffffffu, cw, i * 8 + lane / 4) * t.rope.table_half;
        }
      }
      if (transform) {
        const int frame = min(max(tok, 0) / t.cam.tokens_per_frame, t.cam.frames - 1);
#pragma unroll
        for (int i = 0; i < 4; ++i) frame_of[i] = __shfl_sync(0xffffffffu, frame, i * 8 + lane / 4);
      }

      // The restore works on the 16-byte pieces a lane stores -- four pairs, or one camera block, of one
      // token -- because four lanes then read 128 contiguous bytes of a token's table row; a lane that
      // kept a whole row of the accumulator would gather from 32 rows at a time.  26,917 rotated tokens x
      // 5,120 columns, rank 640 (K and V): 570 us; 655 with the entries requested in the round that uses them and every
      // lane loading and rounding a round's 32 bias columns; 1,328 with the gather per row as well.
      auto load_rotation = [&](int head, int dcol, float2* rot) {
        const int local = dcol / 2 + (lane & 3) * 4;
        const float2* table = reinterpret_cast<const float2*>(t.rope.cos_sin);
#pragma unroll
        for (int w = 0; w < 4; w += 2) {
          int pg[2] = {local + w, local + w + 1};
          if (t.rope.pair_index != nullptr) {
            pg[0] = __ldg(t.rope.pair_index + head * (p.D / 2) + pg[0]);
            pg[1] = __ldg(t.rope.pair_index + head * (p.D / 2) + pg[1]);
          }
          // both pairs of one band, adjacent and 16-byte aligned: one load
          const bool together = p.rope_pairs != 0 && pg[1] == pg[0] + 1 && (pg[0] & 1) == 0 && pg[1] != band_a && pg[1] != band_b;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int row0 = pg[0] < band_a ? coord_t[i] : (pg[0] < band_b ? coord_h[i] : coord_w[i]);
            if (together) {
              const float4 both = __ldg(reinterpret_cast<const float4*>(table + row0 + pg[0]));
              rot[i * 4 + w] = make_float2(both.x, both.y);
              rot[i * 4 + w + 1] = make_float2(both.z, both.w);
            } else {
              const int row1 = pg[1] < band_a ? coord_t[i] : (pg[1] < band_b ? coord_h[i] : coord_w[i]);
              rot[i * 4 + w] = __ldg(table + row0 + pg[0]);
              rot[i * 4 + w + 1] = __ldg(table + row1 + pg[1]);
            }
          }
        }
      };
      auto restore = [&](int i, int head, int dcol, const float2* rot, uint4& v) {
        uint32_t word[4] = {v.x, v.y, v.z, v.w};
        if (rotate) {
#pragma unroll
          for (int w = 0; w < 4; ++w) {   // a pair of the rebuilt bf16 key is one complex number
            const float k0 = __uint_as_float(word[w] << 16), k1 = __uint_as_float(word[w] & 0xFFFF0000u);
            const float2 cs = rot[i * 4 + w];
            word[w] = pack_bf16x2(fmaf(k0, cs.x, -(k1 * cs.y)), fmaf(k0, cs.y, k1 * cs.x));
          }
        }
        if (transform) {   // the four two-element slots of the block, mixed by the frame's matrix
          const int which = __ldg(t.cam.cam_index + head * (p.D / 8) + dcol / 8 + (lane & 3)) & 3;
          const float4* m = reinterpret_cast<const float4*>(t.cam.matrices + static_cast<size_t>(frame_of[i]) * 64 + which * 16);
          float block[8];
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            block[2 * w] = __uint_as_float(word[w] << 16);
            block[2 * w + 1] = __uint_as_float(word[w] & 0xFFFF0000u);
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float4 mi = __ldg(m + k);
            const float c0 = round_to_bf16(mi.x), c1 = round_to_bf16(mi.y);
            const float c2 = round_to_bf16(mi.z), c3 = round_to_bf16(mi.w);
            word[k] = pack_bf16x2(fmaf(c3, block[6], fmaf(c2, block[4], fmaf(c1, block[2], c0 * block[0]))),
                                  fmaf(c3, block[7], fmaf(c2, block[5], fmaf(c1, block[3], c0 * block[1]))));
          }
        }
        v = make_uint4(word[0], word[1], word[2], word[3]);
      };
      // rotation entries of the pieces this lane stores, requested behind the round before like the centres
      float2 rot[ROPE ? 16 : 1];
      auto fetch_rotation = [&](int sub) {
        if (!rotate || sub >= rounds) return;
        const int col0 = nt * TN + wg * 128 + sub * 32, head = col0 / p.D;
        load_rotation(head, col0 - head * p.D, rot);
      };
      fetch_rotation(0);
      ok = wait_all(&bars[ACC_FULL + b], use & 1, abort_flag, 740 + b, p.wait_budget);
      if (!ok) return;
      tc_fence_after();
      auto round = [&](int sub) {
        const int col0 = nt * TN + wg * 128 + sub * 32;
        const int head = col0 / p.D, dcol = col0 - head * p.D;
        uint32_t acc_raw[32];
        tmem_ld32_issue(tmem_base + lane_sel + b * TN + wg * 128 + sub * 32, acc_raw);
        uint32_t packed[16];
        if constexpr (POS) {
          reinterpret_cast<float*>(stage)[lane] = sub == 0 ? bias_lane[0] : (sub == 1 ? bias_lane[1] : (sub == 2 ? bias_lane[2] : bias_lane[3]));
          __syncwarp();
          ulonglong2 add[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) add[j] = reinterpret_cast<const ulonglong2*>(stage)[j];
          tmem_ld32_wait(acc_raw);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            float lo, hi;
            split_f32(add_f32x2(pair_bits(acc_raw[2 * j], acc_raw[2 * j + 1]), (j & 1) ? add[j >> 1].y : add[j >> 1].x), lo, hi);
            packed[j] = pack_bf16x2(lo, hi);
          }
          __syncwarp();        // the bias has been read
        } else {
          tmem_ld32_wait(acc_raw);
#pragma unroll
          for (int j4 = 0; j4 < 4; ++j4) {
            const float4 lo = bias[2 * j4], hi = bias[2 * j4 + 1];
            float add[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            if (p.round_bias) {
#pragma unroll
              for (int j = 0; j < 8; ++j) add[j] = round_to_bf16(add[j]);
            }
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              const int j = j4 * 8 + w * 2;
              packed[j4 * 4 + w] = pack_bf16x2(__uint_as_float(acc_raw[j]) + add[2 * w],
                                               __uint_as_float(acc_raw[j + 1]) + add[2 * w + 1]);
            }
          }
        }
        if constexpr (!POS) load_bias(sub + 1, bias);
        // Through the warp's staging area, so that four lanes hold 64 contiguous bytes of a row: they add
        // the centre (the second bf16 rounding: the packed addition of two bf16 numbers rounds their exact
        // sum once), restore positions and store.  Two rows fill the banks: the swizzle follows the row pair.
#pragma unroll
        for (int j = 0; j < 4; ++j)
          *reinterpret_cast<uint4*>(stage + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) =
              make_uint4(packed[j * 4], packed[j * 4 + 1], packed[j * 4 + 2], packed[j * 4 + 3]);
        __syncwarp();
        uint16_t* dst = t.out + head * t.head_stride + dcol + (lane & 3) * 8;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int rloc = i * 8 + lane / 4, piece = lane & 3;
          uint4 v = *reinterpret_cast<const uint4*>(stage + rloc * 64 + ((piece ^ ((rloc >> 1) & 3)) << 4));
          v = add_bf16x8(v, cen[i]);
          if (POS) restore(i, head, dcol, rot, v);
          if (crow_of[i] >= 0) *reinterpret_cast<uint4*>(dst + static_cast<size_t>(m0 + rloc) * t.row_stride) = v;
        }
        load_centers(sub + 1, cen);
        fetch_rotation(sub + 1);
        __syncwarp();
      };
#pragma unroll 1
      for (int sub = 0; sub < rounds; ++sub) round(sub);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_relaxed(map_to_cta(smem_u32(&bars[ACC_FREE + b]), 0));
      ++tile;
    };

    Run run{}, next{};
    int tok = -1, crow = 0, next_tok = -1, next_crow = 0;
    for (int w = w_begin; w <= w_end && ok; ++w) {
      const bool starts = w < w_end && (w == w_begin || w % p.n_tiles == 0);
      if (starts) {
        next = run_at(p, w, w_end);
        next_tok = token_at(p, next, cta, row);   // this lane's row of the tile
        next_crow = next_tok < 0 ? 0 : center_row_of(p.t[next.tensor].h, next_tok);
        Codes codes;
        fetch_codes(next, next_tok, codes);
        // the latents in shared memory are free once the previous run's last tile is complete; the new
        // ones go in before that tile's epilogue, so that the MMAs of this run start under it
        if (w > w_begin) ok = wait_all(&bars[ACC_FULL + (tile & 1)], (tile >> 1) & 1, abort_flag, 750, p.wait_budget);
        if (!ok) break;
        expand(next, codes);
      }
      if (w > w_begin) epilogue(run, (w - 1) % p.n_tiles, tok, crow);
      if (starts) { run = next; tok = next_tok; crow = next_crow; }
    }
    if (!ok) fill_unfinished(p, w_begin + tile, w_end, cta, row, wg);
  }
  tc_fence_before();
  __syncthreads();
  // neither CTA leaves while the other may still arrive on its barriers or read its operands
  cluster_sync_all();
  if (warp == 9) tmem_dealloc_pair(tmem_base, 512);
  if (tid == 0) {
    if (p.failed != nullptr) p.failed[blockIdx.x] = *abort_flag;
    if (*abort_flag && p.status) atomicCAS(p.status, 0, *abort_flag);
  }
}

int tiles_of(int count, int n, int J) { return count * ceil_div(n, 2 * TM) * ceil_div(J, TN); }

size_t smem_bytes(int nchunks, int stages) {
  return 1024 + META + static_cast<size_t>(nchunks + stages) * CHUNK_BYTES + SCRATCH;
}

}  // namespace

bool tc_decode_supported(const nkv_history& h, int J) {
  return h.rank % 64 == 0 && h.rank <= 64 * MAX_CHUNKS && J % 64 == 0 && h.center_width % 8 == 0 &&
         (h.group == 32 || h.group % 64 == 0) && h.rank % h.group == 0 &&
         ((reinterpret_cast<uintptr_t>(h.codes) | reinterpret_cast<uintptr_t>(h.centers)) & 15) == 0;
}

int tc_decode_blocks(int count, int n, int J, int sms) {
  const int total = tiles_of(count, n, J);
  return 2 * (total < sms / 2 ? total : sms / 2);
}

int tc_decode(const DecodeTensor* tensors, int count, int n, int J, int D, bool w_perm, bool round_bias,
              int32_t* status, int32_t* failed, int sms, long long selftest_budget, cudaStream_t stream) {
  if (n == 0) return NKV_OK;
  Params p{};
  CUtensorMap maps[2];
  bool rotated = false, transformed = false;
  for (int i = 0; i < count; ++i) {
    const DecodeTensor& src = tensors[i];
    Tensor& t = p.t[i];
    t.h = *src.hist;
    t.bias = src.bias;
    t.rows = src.rows;
    t.out = static_cast<uint16_t*>(src.out);
    t.row_stride = src.row_stride;
    t.head_stride = src.head_stride;
    if (src.rope != nullptr) {
      t.rope = *src.rope;
      p.rope_pairs = t.rope.table_half % 2 == 0 && (reinterpret_cast<uintptr_t>(t.rope.cos_sin) & 15) == 0;
      rotated = true;
    }
    if (src.camera != nullptr) { t.cam = *src.camera; transformed = true; }
    uint64_t dims[2] = {static_cast<uint64_t>(t.h.rank), static_cast<uint64_t>(J)};
    uint64_t strides[1] = {static_cast<uint64_t>(t.h.rank) * 2};
    uint32_t box[2] = {64, TM};
    int rc = encode_tensor_map(&maps[i], 2, src.decoder, 2, dims, strides, box, 128);
    if (rc != NKV_OK) return rc;
  }
  if (count == 1) maps[1] = maps[0];
  const nkv_history& h = p.t[0].h;
  p.tensors = count;
  p.n = n; p.J = J; p.D = D;
  p.nchunks = h.rank / 64;
  p.group = h.group;
  p.ngroups = h.rank / h.group;
  p.w_perm = w_perm ? 1 : 0;
  p.round_bias = round_bias ? 1 : 0;
  p.nstages = MAX_STAGES;
  while (p.nstages > 2 && smem_bytes(p.nchunks, p.nstages) > SMEM_LIMIT) --p.nstages;
  const size_t smem = smem_bytes(p.nchunks, p.nstages);
  p.m_tiles = ceil_div(n, 2 * TM);
  p.n_tiles = ceil_div(J, TN);
  p.total = tiles_of(count, n, J);
  p.status = status;
  p.failed = failed;
  p.starve = selftest_budget > 0 ? 1 : 0;
  p.wait_budget = selftest_budget > 0 ? selftest_budget : WAIT_BUDGET_CYCLES;
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(tc_decode_blocks(count, n, J, sms));
  config.blockDim = dim3(THREADS);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  config.attrs = &attr;
  config.numAttrs = 1;
  auto kernel = transformed ? decode_gemm_kernel<true, true>      // a NULL table switches the rotation off
                : (rotated ? decode_gemm_kernel<true, false> : decode_gemm_kernel<false, false>);
  NKV_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  NKV_CUDA(cudaLaunchKernelEx(&config, kernel, maps[0], maps[1], p));
  return NKV_OK;
}

}  // namespace nkv
