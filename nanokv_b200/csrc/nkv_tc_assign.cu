// Nearest-centre assignment on tcgen05: [S x J] x [C x J]^T tiles with fp32 accumulators in TMEM, squared norms of
// both operands summed from the tiles while they lie in shared memory, and an epilogue that evaluates
// (||x||^2 + ||c||^2) - 2 x.c in fp32 and keeps the first minimum.
//
// Given centres are bf16.  The C-means' fp32 means come as three bf16 planes side by side along K (hi, mid, lo:
// every product is exact in the fp32 accumulator); the token rows are walked once per plane, and the warps that sum
// norms square the fp32 rows themselves while the second and third plane are multiplied.  K is never cut, every sum
// runs in the order of K, and every tile starts at a multiple of eight tokens (a row's place modulo eight is part of
// its norm's order): what is stored does not depend on how a call is tiled, nor on where a history is cut into calls
// as long as the calls start at multiples of eight tokens of it.
//
// A thread block owns `rows` tokens and C / parts centres; the `parts` blocks of one token tile are a cluster,
// whose first block collects the others' minima through its shared memory; the parts share out the norms of the
// tile's tokens.  Where one block takes more than 256 centres, two tiles are a cluster and share out the centres' norms.  The MMA always spans 128 rows: rows
// past the tile's are whatever lies behind it in shared memory, and their sums are read by nobody.
//
// Bound: the K loop of a tile.  MMAs on one accumulator follow one another at 86 cycles whatever their width (measured:
// 345 cycles per 64 columns of K up to 96 centres, 512 at 256), so 3,072 columns take 9 us, three planes of them 26,
// and only the operands and the norms can be kept from adding to that.  Hence
//   * tiles of 64 rows and less and parts of the centres for short calls, which otherwise leave most SMs idle;
//   * stages of up to four 64-column chunks: the thread that fills a stage needs some 330 cycles for it;
//   * norms without bank conflicts (a lane starts at another of its half-row's four pieces and puts the four sums
//     back in order before they are added), two chains per packed multiply-add, shared within the cluster;
//   * two accumulators of one block take turns.
// us, before (one block per tile of 64 rows, 64-column stages) and now: 1,560 x 3,072 to 256 centres 59, 17; 12,480 x
// 5,120 to 512 165, 100; three planes of 64 centres, 880 x 3,072 49, 26; 4,680 x 5,120 80, 52.
//
// Warps 0-7: norms and epilogue, warp 8 lane 0: TMA, warp 9: MMA.
#include "nkv_internal.h"
#include "nkv_tc.cuh"

namespace nkv {

int pick_rows(int S, int column_parts);

namespace {

using namespace tc;

constexpr int TM = 128;
constexpr int COMPUTE_THREADS = 256;
constexpr int WARPS = COMPUTE_THREADS / 32;
constexpr int THREADS = COMPUTE_THREADS + 64;
constexpr int MAX_STAGES = 8;
constexpr int MAX_PARTS = 8;
constexpr int MAX_KC = 4;                  // 64-column chunks of a stage
constexpr int MAX_CENTRES = 512;
constexpr int MAX_ITEMS = 5;               // half-rows whose squares a thread sums: (2 * 128 + 2 * 512) / 256
enum Bar { FULL = 0, FREE = 8, NORMS_FREE = 16, ACC_DONE = 24, SIDE_READY = 25, CAND_READY = 26, PEER_READY = 27,
           NUM_BARS = 28 };

struct Meta {
  uint64_t bars[NUM_BARS];
  uint32_t tmem_slot;
  int abort_flag;
  alignas(16) float norm_x[TM];
  float norm_c[MAX_CENTRES];   // squared norms of the tile's tokens and of the block's centres
  alignas(16) float cand_d[TM];
  int cand_i[TM];
  float peer_d[MAX_PARTS][TM];
  int peer_i[MAX_PARTS][TM];
};

struct Params {
  int S, C, rows, rows_pad, NB, NACC, parts;
  int team;                                // blocks of a cluster: the parts of a tile, or two tiles
  int nstages, steps, norm_steps;          // stages of KC chunks in all, and of the first plane
  int tmem_columns;
  void* ids_out; int id_bytes;
  int32_t* labels_out;                     // optional 32-bit copy of the ids (the C-means update reads it)
  const float* centers;                    // fp32 centres (their planes are the operand), or NULL: bf16 centres
  int J;
};

// sums of the eight squares of two pieces, each one chain of fused multiply-adds in the order of its elements
__device__ __forceinline__ void sumsq8_pair(const uint4& u, const uint4& v, float& su, float& sv) {
  const uint32_t a[4] = {u.x, u.y, u.z, u.w}, b[4] = {v.x, v.y, v.z, v.w};
  uint64_t sum = 0ull;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint64_t even = pair_f32(__uint_as_float(a[i] << 16), __uint_as_float(b[i] << 16));
    const uint64_t odd = pair_f32(__uint_as_float(a[i] & 0xFFFF0000u), __uint_as_float(b[i] & 0xFFFF0000u));
    sum = fma_f32x2(even, even, sum);
    sum = fma_f32x2(odd, odd, sum);
  }
  split_f32(sum, su, sv);
}

// Squared norm of an fp32 row of J columns (a multiple of 64), by one warp (lane 0 has it): partial sum t of 256 runs
// over the columns t, t + 256, ... in turn, and the partial sums are added in halves, 128 and 128, 64 and 64 and so on.
// A lane keeps the partial sums 4 lane .. 4 lane + 3 of either half.
__device__ __forceinline__ float row_norm(const float* row, int J, int lane) {
  float part[2][4] = {};
  auto square = [&](int half, const float4& v) {
    part[half][0] = fmaf(v.x, v.x, part[half][0]);
    part[half][1] = fmaf(v.y, v.y, part[half][1]);
    part[half][2] = fmaf(v.z, v.z, part[half][2]);
    part[half][3] = fmaf(v.w, v.w, part[half][3]);
  };
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int k = 4 * lane; k < J; k += 256) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(row + k));
    const float4 b = k + 128 < J ? __ldg(reinterpret_cast<const float4*>(row + k + 128)) : zero;
    square(0, a);
    square(1, b);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float sum = part[0][e] + part[1][e];
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, off);
    part[0][e] = sum;
  }
  return (part[0][0] + part[0][2]) + (part[0][1] + part[0][3]);
}

template <int KC>
__global__ void __launch_bounds__(THREADS, 1)
assign_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                   const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  Meta& meta = *reinterpret_cast<Meta*>(smem_raw);
  uint8_t* ring = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + sizeof(Meta) + 1023) & ~static_cast<uintptr_t>(1023));
  const int a_tile = p.rows_pad * 128, b_tile = p.NACC * p.NB * 128;     // one 64-column chunk
  const int a_bytes = KC * a_tile, stage_bytes = a_bytes + KC * b_tile;
  const int nst = p.nstages;
  uint64_t* bars = meta.bars;
  volatile int* abort_flag = &meta.abort_flag;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int part = blockIdx.x % p.parts;
  const int m0 = (blockIdx.x / p.parts) * p.rows, m_end = min(p.S, m0 + p.rows);
  const int columns = p.NACC * p.NB, n_base = part * columns;

  if (tid == 0) {
    for (int s = 0; s < MAX_STAGES; ++s) {
      mbar_init(&bars[FULL + s], 1);
      mbar_init(&bars[FREE + s], 1);
      mbar_init(&bars[NORMS_FREE + s], WARPS);
    }
    mbar_init(&bars[ACC_DONE], 1);
    mbar_init(&bars[SIDE_READY], WARPS * p.team);
    mbar_init(&bars[CAND_READY], TM);
    mbar_init(&bars[PEER_READY], TM * (p.parts > 1 ? p.parts - 1 : 1));
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 9) tmem_alloc(&meta.tmem_slot, p.tmem_columns);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = meta.tmem_slot;
  // the blocks of a cluster write into each other's shared memory: nobody may do so before the barriers exist
  if (p.team > 1) cluster_arrive();
  bool ok = true, joined = false;

  if (warp == 8) {
    if (lane == 0) {
      prefetch_tensormap(&map_a);
      prefetch_tensormap(&map_b);
      Ring at;
      int a_step = 0;
      for (int i = 0; i < p.steps && ok; ++i, at.advance(nst)) {
        const int s = at.stage;
        if (i >= nst) {
          ok = mbar_wait(&bars[FREE + s], at.phase ^ 1, abort_flag, 400 + s);
          if (ok && i - nst < p.norm_steps) ok = mbar_wait(&bars[NORMS_FREE + s], at.phase ^ 1, abort_flag, 408 + s);
        }
        if (!ok) break;
        uint8_t* stage = ring + s * stage_bytes;
        mbar_arrive_expect_tx(&bars[FULL + s], stage_bytes);
        tma_load_3d(stage, &map_a, 0, m0, a_step * KC, &bars[FULL + s]);
        // accumulators of up to 256 columns: chunk by chunk within a stage, one after the other
        for (int a = 0; a < p.NACC; ++a)
          tma_load_3d(stage + a_bytes + a * KC * p.NB * 128, &map_b, 0, n_base + a * p.NB, i * KC, &bars[FULL + s]);
        if (++a_step == p.norm_steps) a_step = 0;
      }
      if (!ok) {   // copies in flight land before the block goes away
        const long long start = clock64();
        while (clock64() - start < (1ll << 21)) {}
      }
    }
    __syncwarp();
  } else if (warp == 9) {
    const bool leader = elect_one();
    const uint32_t idesc = make_idesc_bf16(TM, p.NB);
    const uint32_t ring_base = smem_u32(ring);
    Ring at;
    for (int i = 0; i < p.steps && ok; ++i, at.advance(nst)) {
      const int s = at.stage;
      ok = wait_all(&bars[FULL + s], at.phase, abort_flag, 416 + s);
      if (!ok) break;
      tc_fence_after();
      const uint32_t stage = ring_base + s * stage_bytes;
      if (leader) {
        // an accumulator's MMAs follow one another at 86 cycles at the least; two accumulators take turns
#pragma unroll
        for (int q = 0; q < KC; ++q) {
          const uint64_t a_desc = make_smem_desc_sw128(stage + q * a_tile);
          const uint64_t b_desc = make_smem_desc_sw128(stage + a_bytes + q * p.NB * 128);
          const uint64_t b_next = make_smem_desc_sw128(stage + a_bytes + (KC + q) * p.NB * 128);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            mma_bf16(tmem_base, a_desc + 2 * k, b_desc + 2 * k, idesc, (i | q | k) != 0);
            if (p.NACC == 2) mma_bf16(tmem_base + 256, a_desc + 2 * k, b_next + 2 * k, idesc, (i | q | k) != 0);
          }
        }
        mma_commit(&bars[FREE + s]);
      }
      __syncwarp();
    }
    if (ok && leader) mma_commit(&bars[ACC_DONE]);
    __syncwarp();
  } else {
    const int row = tid & 127, wg = tid >> 7;
    const uint32_t lane_sel = static_cast<uint32_t>(32 * (warp & 3)) << 16;
    // ---- squared norms from the resident tiles: half-rows of 32 columns, tokens first, then centres.  The order
    // of a half-row's sums (four pieces of eight columns, in the order they have in the swizzled tile) is part of
    // what the stored ids were made with: a row's place modulo 8 in its tile decides it, so every
    // tile starts at a multiple of 8 tokens.
    // The blocks of a cluster share the work: the parts of a tile its tokens, two tiles their centres.
    const uint32_t me = p.team > 1 ? cluster_ctarank() : 0;
    const int x_share = p.parts > 1 ? (p.rows_pad + p.parts - 1) / p.parts : p.rows_pad, x_first = p.parts > 1 ? part * x_share : 0;
    const int c_share = p.centers != nullptr ? 0 : (p.parts == 1 ? columns / p.team : columns);
    const int c_first = p.parts == 1 ? static_cast<int>(me) * c_share : 0;
    const int x_items = 2 * max(0, min(x_share, p.rows_pad - x_first)), items = x_items + 2 * c_share;
    for (int c = columns + tid; c < MAX_CENTRES; c += COMPUTE_THREADS) meta.norm_c[c] = INFINITY;   // infinitely far
    const int rot = (tid >> 1) & 3;
    uint32_t at_stage[MAX_ITEMS];         // an item's place in a stage's first chunk; the further chunks follow a tile apart
#pragma unroll
    for (int k = 0; k < MAX_ITEMS; ++k) {
      const int item = tid + k * COMPUTE_THREADS;
      at_stage[k] = (x_first + (item >> 1)) * 128 + (item & 1) * 64;
      if (item >= x_items) {
        const int c = c_first + ((item - x_items) >> 1), a = c >= p.NB ? 1 : 0;
        at_stage[k] = a_bytes + (a * KC * p.NB + c - a * p.NB) * 128 + (item & 1) * 64;
      }
    }
    float sums[MAX_ITEMS] = {};
    Ring at;
    for (int i = 0; i < p.norm_steps && ok; ++i, at.advance(nst)) {
      const int s = at.stage;
      ok = wait_all(&bars[FULL + s], at.phase, abort_flag, 424 + s);
      if (!ok) break;
      const uint8_t* stage = ring + s * stage_bytes;
#pragma unroll
      for (int k = 0; k < MAX_ITEMS; ++k) {
        const int item = tid + k * COMPUTE_THREADS;
        if (item < items) {
          const uint8_t* src = stage + at_stage[k];
          const int pitch = item < x_items ? a_tile : p.NB * 128;
          float t[KC][4];
#pragma unroll
          for (int q = 0; q < KC; ++q) {
            const uint4* piece = reinterpret_cast<const uint4*>(src + q * pitch);
            const uint4 p0 = piece[rot], p1 = piece[(rot + 1) & 3], p2 = piece[(rot + 2) & 3], p3 = piece[(rot + 3) & 3];
            sumsq8_pair(p0, p1, t[q][0], t[q][1]);
            sumsq8_pair(p2, p3, t[q][2], t[q][3]);
          }
#pragma unroll
          for (int q = 0; q < KC; ++q) {   // back in order, then one after the other
            const bool one = rot & 1, two = rot & 2;
            const float a = one ? t[q][3] : t[q][0], b = one ? t[q][0] : t[q][1];
            const float c = one ? t[q][1] : t[q][2], d = one ? t[q][2] : t[q][3];
            sums[k] += two ? c : a;
            sums[k] += two ? d : b;
            sums[k] += two ? a : c;
            sums[k] += two ? b : d;
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[NORMS_FREE + s]);
    }
    if (p.centers != nullptr && ok)
      for (int c = warp; c < columns; c += WARPS) {
        const float norm = row_norm(p.centers + static_cast<size_t>(n_base + c) * p.J, p.J, lane);
        if (lane == 0) meta.norm_c[c] = norm;
      }
    if (p.team > 1) cluster_wait();
    joined = true;
    if (ok) {
#pragma unroll
      for (int k = 0; k < MAX_ITEMS; ++k) {
        const int item = tid + k * COMPUTE_THREADS;
        const float both = sums[k] + __shfl_xor_sync(0xffffffffu, sums[k], 1);    // the two half-rows
        if (item < items && (item & 1) == 0) {
          const bool token = item < x_items;
          float* at_norm = token ? &meta.norm_x[x_first + (item >> 1)] : &meta.norm_c[c_first + ((item - x_items) >> 1)];
          if (p.team > 1 && token == (p.parts > 1)) {      // what the cluster shares
            for (int peer = 0; peer < p.team; ++peer) st_cluster_b32(map_to_cta(smem_u32(at_norm), peer), __float_as_uint(both));
          } else {
            *at_norm = both;
          }
        }
      }
      __syncwarp();
      if (p.team > 1) {
        if (lane < p.team) mbar_arrive_cluster(map_to_cta(smem_u32(&bars[SIDE_READY]), lane));
      } else if (lane == 0) {
        mbar_arrive(&bars[SIDE_READY]);
      }
      ok = wait_all_cluster(&bars[SIDE_READY], 0, abort_flag, 432) && wait_all(&bars[ACC_DONE], 0, abort_flag, 433);
    }
    // ---- distances: the two warpgroups take half of the columns each
    if (ok) {
      tc_fence_after();
      const float xn = row < p.rows_pad ? meta.norm_x[row] : 0.f;
      const int chunks = (columns + 31) / 32, middle = (chunks + 1) / 2;
      const int first = wg == 0 ? 0 : middle, last = wg == 0 ? middle : chunks;
      float best = INFINITY;
      int best_i = 0;      // a row without a finite distance: centre 0, never an id past C
#pragma unroll 1
      for (int cc = first; cc < last; ++cc) {
        const int col = cc * 32, acc = col / p.NB;
        float v[32];
        tmem_ld32(tmem_base + lane_sel + acc * 256 + (col - acc * p.NB), v);
#pragma unroll
        for (int j4 = 0; j4 < 8; ++j4) {
          const float4 cn4 = *reinterpret_cast<const float4*>(&meta.norm_c[col + j4 * 4]);
          const float cn[4] = {cn4.x, cn4.y, cn4.z, cn4.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float dist = __fsub_rn(__fadd_rn(xn, cn[j]), __fmul_rn(2.0f, v[j4 * 4 + j]));
            if (dist < best) { best = dist; best_i = n_base + col + j4 * 4 + j; }
          }
        }
      }
      if (wg == 1) {
        meta.cand_d[row] = best;
        meta.cand_i[row] = best_i;
        mbar_arrive(&bars[CAND_READY]);
      } else {
        ok = wait_all(&bars[CAND_READY], 0, abort_flag, 434);
        if (ok) {
          if (meta.cand_d[row] < best) { best = meta.cand_d[row]; best_i = meta.cand_i[row]; }
          if (part > 0) {
            st_cluster_b32(map_to_cta(smem_u32(&meta.peer_d[part][row]), 0), __float_as_uint(best));
            st_cluster_b32(map_to_cta(smem_u32(&meta.peer_i[part][row]), 0), static_cast<uint32_t>(best_i));
            mbar_arrive_cluster(map_to_cta(smem_u32(&bars[PEER_READY]), 0));
          } else {
            if (p.parts > 1) ok = wait_all_cluster(&bars[PEER_READY], 0, abort_flag, 435);
            if (ok) {
              for (int peer = 1; peer < p.parts; ++peer)
                if (meta.peer_d[peer][row] < best) { best = meta.peer_d[peer][row]; best_i = meta.peer_i[peer][row]; }
              const int t = m0 + row;
              if (row < p.rows && t < m_end) {
                if (p.ids_out != nullptr) {
                  if (p.id_bytes == 1) static_cast<uint8_t*>(p.ids_out)[t] = static_cast<uint8_t>(best_i);
                  else static_cast<uint16_t*>(p.ids_out)[t] = static_cast<uint16_t>(best_i);
                }
                if (p.labels_out != nullptr) p.labels_out[t] = best_i;
              }
            }
          }
        }
      }
    }
  }
  if (p.team > 1 && !joined) cluster_wait();
  tc_fence_before();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem_base, p.tmem_columns);
  // nobody leaves while another may still write into its shared memory
  if (p.team > 1) cluster_sync_all();
}

constexpr size_t SMEM_LIMIT = 232448;

// Shared memory of a ring: the MMA reads 128 rows from where the last token tile starts, which may reach past it.
size_t smem_bytes(int rows_pad, int columns, int kc, int stages) {
  const size_t stage = static_cast<size_t>(kc) * (rows_pad + columns) * 128;
  const size_t end = stages * stage, last_a = (stages - 1) * stage + static_cast<size_t>(kc - 1) * rows_pad * 128;
  const size_t reach = last_a + TM * 128;
  return sizeof(Meta) + 1024 + (reach > end ? reach : end);
}

struct Cut { int rows, parts, kc, stages; };

// Tokens per tile and parts of the centres.  Estimate in SM cycles: a 64-column chunk takes its bytes from L2 at 48
// per clock, at least 130 cycles of hand-offs; a block has about 6,000 cycles of prologue and epilogue.  Calls that
// one round of 64-row tiles covers take tiles of 16, 32 or 64 rows, longer ones the rows that fill whole rounds, up
// to the next multiple of eight (a row's place modulo eight decides the order of its norm's sum, see the kernel).  Measured against
// the alternatives, us: 4,680 x 5,120, 64 centres, 64 rows x 2 parts 22, 64 x 1 24, 32 x 1 25; 256 centres, 64 x 2 34,
// 64 x 1 51; 1,560 x 5,120, 512 centres, 64 x 4 32, 64 x 8 45, 64 x 2 50.
Cut plan_assign(int S, int C, int a_chunks, int planes) {
  const int sms = sm_count();
  const int whole = (pick_rows(S, 1) + 7) / 8 * 8;
  Cut best{whole, 1, 1, 2};
  double best_cost = -1;
  for (int rows = whole; rows >= 16; rows /= 2) {
    for (int parts = 1; parts <= MAX_PARTS; ++parts) {
      const int columns = C / parts;
      if (C % parts || columns % 16 || (columns > 256 && columns % 64) || columns > 512) continue;
      const int room = parts > 4 ? sms - 20 : (parts > 2 ? sms - 4 : sms);
      const long long blocks = static_cast<long long>(ceil_div(S, rows)) * parts;
      const double bytes = ((rows + 7) / 8 * 8 + columns) * 128.0;
      const double chunk = bytes / 48 > 130 ? bytes / 48 : 130;
      const double cost = static_cast<double>((blocks + room - 1) / room) *
                          (chunk * a_chunks * planes + 6000);
      if (best_cost < 0 || cost < best_cost) {
        best_cost = cost;
        best = Cut{rows, parts, 1, 2};
      }
    }
    if (whole != 64) break;
  }
  return best;
}

int launch_assign(const void* x, const void* centers, int S, int J, int C, int planes, Params& p, cudaStream_t stream) {
  Cut cut = plan_assign(S, C, J / 64, planes);
  const int columns = C / cut.parts, rows_pad = (cut.rows + 7) / 8 * 8;
  // large stages: a stage costs the thread that fills it some 330 cycles, whatever it holds
  for (cut.kc = MAX_KC; cut.kc > 1; cut.kc /= 2)
    if ((J / 64) % cut.kc == 0 && smem_bytes(rows_pad, columns, cut.kc, 2) <= SMEM_LIMIT) break;
  for (cut.stages = MAX_STAGES; cut.stages > 2; --cut.stages)
    if (smem_bytes(rows_pad, columns, cut.kc, cut.stages) <= SMEM_LIMIT) break;
  const size_t smem = smem_bytes(rows_pad, columns, cut.kc, cut.stages);
  NKV_REQUIRE(smem <= SMEM_LIMIT, NKV_ERR_UNSUPPORTED, "assign: %zu bytes of shared memory", smem);
  p.S = S; p.J = J; p.C = C;
  p.rows = cut.rows; p.rows_pad = rows_pad; p.parts = cut.parts;
  const int tiles = ceil_div(S, p.rows);
  // two tiles share the norms of many centres (bf16 ones: the fp32 ones' are known)
  const bool two = cut.parts == 1 && planes == 1 && C > 256 && tiles > 1;
  p.team = two ? 2 : cut.parts;
  p.NACC = columns > 256 ? 2 : 1;
  p.NB = columns / p.NACC;
  p.nstages = cut.stages;
  p.norm_steps = J / 64 / cut.kc;
  p.steps = planes * p.norm_steps;
  p.tmem_columns = p.NACC == 2 ? 512 : (p.NB > 128 ? 256 : (p.NB > 64 ? 128 : (p.NB > 32 ? 64 : 32)));
  CUtensorMap map_a, map_b;
  const uint64_t row_bytes = static_cast<uint64_t>(J) * 2;
  {
    const uint64_t dims[3] = {64, static_cast<uint64_t>(S), static_cast<uint64_t>(J / 64)};
    const uint64_t strides[2] = {row_bytes, 128};
    const uint32_t box[3] = {64, static_cast<uint32_t>(rows_pad), static_cast<uint32_t>(cut.kc)};
    int rc = encode_tensor_map(&map_a, 2, x, 3, dims, strides, box, 128);
    if (rc != NKV_OK) return rc;
  }
  {
    const uint64_t dims[3] = {64, static_cast<uint64_t>(C), static_cast<uint64_t>(planes * (J / 64))};
    const uint64_t strides[2] = {planes * row_bytes, 128};
    const uint32_t box[3] = {64, static_cast<uint32_t>(p.NB), static_cast<uint32_t>(cut.kc)};
    int rc = encode_tensor_map(&map_b, 2, centers, 3, dims, strides, box, 128);
    if (rc != NKV_OK) return rc;
  }
  auto kernel = cut.kc == 4 ? assign_gemm_kernel<4> : (cut.kc == 2 ? assign_gemm_kernel<2> : assign_gemm_kernel<1>);
  NKV_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(static_cast<unsigned>(two ? (tiles + 1) / 2 * 2 : tiles * p.parts));
  config.blockDim = dim3(THREADS);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = p.team;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  config.attrs = &attr;
  config.numAttrs = 1;
  NKV_CUDA(cudaLaunchKernelEx(&config, kernel, map_a, map_b, p));
  return NKV_OK;
}

}  // namespace

bool tc_assign_supported(int J, int C) {
  if (J % 64 || C % 16 || C > 512) return false;
  return C <= 256 || C % 64 == 0;
}

int tc_assign(const void* x_bf16, const void* centers_bf16, int S, int J, int C, void* ids,
              int id_bytes, cudaStream_t stream) {
  if (S == 0) return NKV_OK;
  Params p{};
  p.ids_out = ids; p.id_bytes = id_bytes;
  return launch_assign(x_bf16, centers_bf16, S, J, C, 1, p, stream);
}

// Nearest centre against fp32 centres on the tensor cores: every bf16 x bf16 product is exact in the
// fp32 accumulator, and the three planes restore the centres' 24 mantissa bits, so the distances
// carry fp32 accuracy (the accumulation order is the tensor core's).  Writes 32-bit labels, and ids where asked.
int tc_assign_f32(const void* x_bf16, const float* centers_f32, const uint16_t* planes, int S, int J, int C,
                  int32_t* labels, void* ids, int id_bytes, cudaStream_t stream) {
  if (S == 0) return NKV_OK;
  Params p{};
  p.labels_out = labels;
  p.ids_out = ids; p.id_bytes = id_bytes;
  p.centers = centers_f32;
  return launch_assign(x_bf16, planes, S, J, C, 3, p, stream);
}

}  // namespace nkv
