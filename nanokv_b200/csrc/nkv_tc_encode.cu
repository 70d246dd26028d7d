// Encoder projection on tcgen05: coefficients = bf16((x - centre[id]) - mean) encoder^T, fp32 accumulators in TMEM,
// and the INT4 quantiser behind it.
//
// x and the encoder's rows come by TMA into a ring of stages along K = J; the compute warps turn x into the residual in
// its place (the swizzled operand layout), the centres' pieces fetched into registers some stages ahead.  K is never
// cut: every sum runs in the order of K whatever the call's length, so that a row gets the same codes and scale in a
// chunk of any size.
//   project            rounds the coefficients to bf16 and writes them.
//   project + quantise keeps them in TMEM and writes packed codes and scales to their place in the history.  With one
//                      scale per token the column parts of a token tile (a cluster of up to eight) swap the maxima of
//                      their columns through each other's shared memory; with one per 32 coefficients a thread holds
//                      whole groups.
//
// Bound: short calls the length of the K loop (a 64-column chunk costs 500 to 550 cycles: MMAs on one accumulator follow one
// another at 86 cycles, forming the residual takes the load / store and conversion units about as long) and 10 us
// of prologue and epilogue; long calls what a block takes from L2 (2.0 GB at about 14 TB/s for 12,480 x 5,120 x 640).
// What counted, us for 1,560 x 3,072 x 384 / 4,680 x 5,120 x 640 / 12,480 x 5,120 x 640: 38 / 72 / 171 with x loaded by the
// residual warps, the mean from L2, values quantised one by one; 32 / 72 / 192 with x by TMA and the mean in shared memory
// read once per row (eight conflicting lines each: more than all else the residual reads); 27 / 67 / 162 read once
// per chunk, in whole lines; 25 / 61 / 146 with packed quantising and without the rows that are nobody's in it.
// Tried: the residual of a tile formed once and written to all its parts' shared memory 47 / 148 / 316 (every
// stage waits for the slowest remote store); centres by TMA gathers of four rows 56 / 97 / 238 (about 100 cycles each); 16
// residual warps 31 / 71 / 199; started ahead of the assignment's end (programmatic launch): no difference.
// Warps 0-7: residual and epilogue, warp 8 lane 0: TMA, warp 9: MMA.
#include <atomic>

#include "nkv_internal.h"
#include "nkv_tc.cuh"

namespace nkv {

int pick_rows(int S, int column_parts);

namespace {

using namespace tc;

constexpr int TM = 128;
constexpr int COMPUTE_THREADS = 256;
constexpr int GROUPS = COMPUTE_THREADS / TM;   // warpgroups: a TMEM lane is served by one thread of each
constexpr int WARPS = COMPUTE_THREADS / 32;
constexpr int THREADS = COMPUTE_THREADS + 64;
constexpr int MAX_STAGES = 8;
constexpr int MAX_PARTS = 8;            // thread blocks of one token tile that form a cluster
constexpr int MAX_MEAN = 8192;          // widest row whose mean is kept in shared memory
enum Bar { FULL = 0, FORMED = 8, FREE = 16, B_FULL = 24, ACC_DONE = 32, SIDE_READY = 33, PEER_READY = 34, NUM_BARS = 35 };

struct Meta {
  uint64_t bars[NUM_BARS];
  uint32_t tmem_slot;
  int abort_flag;
  float row_max[GROUPS][TM];
  float peer_max[MAX_PARTS][TM];
};

struct Params {
  int S, J, rows, rows_pad, NB, NACC, n_total;          // n_total = r
  int parts, kc;            // column parts of a tile; 64-column chunks of a stage
  int nstages, units;       // stages of the ring; SPLIT: stages of token rows, and units of encoder rows
  int nchunks, tmem_columns, mean_bytes;                // mean_bytes 0: the mean is read where it lies
  const uint16_t* centers; const void* ids; int id_bytes;
  const float* mean; uint16_t* coeff;
  // project + quantise: codes u8 [S, r/2] and scales [S, r/group] at the history's token offset
  uint8_t* codes; void* scales; float eps; int in_bf16; int scale_dtype; int group32;
};

__device__ __forceinline__ float scale_of(float amax, const Params& p) {
  return p.in_bf16 ? round_to_bf16(__fdiv_rn(fmaxf(amax, round_to_bf16(p.eps)), 7.0f))
                   : __fdiv_rn(fmaxf(amax, p.eps), 7.0f);
}

// 32 coefficients of this thread's token, rounded to bf16 (two per word)
__device__ __forceinline__ void round_chunk(const float (&v)[32], uint32_t (&w)[16]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) w[i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
}

// largest magnitude of the 32, as bf16 bits in both halves (a NaN or an infinity gives 0x7F80 or more)
__device__ __forceinline__ uint32_t max_bits(const uint32_t (&w)[16]) {
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) m = __vmaxu2(m, w[i] & 0x7FFF7FFFu);
  const uint32_t swapped = __byte_perm(m, m, 0x1032);
  return __vmaxu2(m, swapped);
}
constexpr uint32_t NOT_FINITE = 0x7F807F80u;

// the same with NaNs left out, for rows that are not finite
__device__ __forceinline__ float max_of_numbers(const uint32_t (&w)[16]) {
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i)
    amax = fmaxf(fmaxf(amax, fabsf(__uint_as_float(w[i] << 16))), fabsf(__uint_as_float(w[i] & 0xFFFF0000u)));
  return amax;
}
__device__ __forceinline__ float max_magnitude(const uint32_t (&w)[16], uint32_t& worst) {
  const uint32_t bits = max_bits(w);
  worst = __vmaxu2(worst, bits);
  return bits >= NOT_FINITE ? max_of_numbers(w) : __uint_as_float(bits << 16);
}

// value by value, with every rounding and clamp spelled out: NaN gives code 0.  By value: an array whose address
// leaves the caller would live in local memory there, on the path that finite rows take too.
__device__ __noinline__ uint32_t quant_word_any(uint4 v, float scale, float inv, bool in_bf16) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t out = 0;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float z = __uint_as_float((e & 1) ? w[e >> 1] & 0xFFFF0000u : w[e >> 1] << 16);
    const int code = in_bf16 ? quant_code<true>(z, scale, inv) : quant_code<false>(z, scale, inv);
    out |= static_cast<uint32_t>(code) << (4 * e);
  }
  return out;
}

// packed codes of 32 coefficients; `finite`: none of them is a NaN or an infinity.  A scale below 2^-128 (a caller's
// small eps) has no finite reciprocal, and quant_word takes every quotient through it.
__device__ __forceinline__ uint4 pack_codes(const uint32_t (&w)[16], float scale, bool in_bf16, bool finite) {
  const float inv = __frcp_rn(scale);
  finite = finite && inv < INFINITY;
  uint32_t words[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t part[4] = {w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]};
    words[i] = !finite ? quant_word_any(make_uint4(part[0], part[1], part[2], part[3]), scale, inv, in_bf16)
                       : (in_bf16 ? quant_word<true>(part, scale, inv) : quant_word<false>(part, scale, inv));
  }
  return make_uint4(words[0], words[1], words[2], words[3]);
}

// SLOTS: rows of a stage's residual of which a thread forms 16 bytes, their centres fetched DEPTH stages ahead.
// SPLIT: token rows and encoder rows have rings of their own, the encoder's in units of one accumulator's columns, each
// free as soon as its MMAs are done.  For tiles so wide that two whole stages is all that fits: with two, a stage is
// loaded, formed and multiplied with only one other under way.  us, two whole stages / SPLIT: 12,480 x 2,048 x 512 43 / 35,
// 12,480 x 3,072 x 1,024 122 / 98, 9,500 x 5,120 x 512 109 / 76.  With three whole stages and more one barrier for both
// operands is as fast or faster (20,000 x 2,048 x 256 47, SPLIT 49; 4,680 x 5,120 x 640 59, SPLIT 62).
template <bool QUANT, bool SPLIT, int SLOTS, int DEPTH>
__global__ void __launch_bounds__(THREADS, 1)
project_gemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  Meta& meta = *reinterpret_cast<Meta*>(smem_raw);
  float* mean_smem = reinterpret_cast<float*>(smem_raw + (sizeof(Meta) + 15) / 16 * 16);
  uint8_t* ring = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(mean_smem) + p.mean_bytes + 1023) & ~static_cast<uintptr_t>(1023));
  const int a_tile = p.rows_pad * 128, b_tile = p.NB * 128;       // one 64-column chunk; of one accumulator
  const int kc = p.kc, a_bytes = kc * a_tile, stage_bytes = SPLIT ? a_bytes : a_bytes + kc * p.NACC * b_tile;
  uint8_t* units = ring + p.nstages * a_bytes;                    // SPLIT: the encoder's ring
  const int unit_bytes = kc * b_tile;
  const int nst = p.nstages, nchunks = p.nchunks, steps = (nchunks + kc - 1) / kc;
  uint64_t* bars = meta.bars;
  volatile int* abort_flag = &meta.abort_flag;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int part = blockIdx.x % p.parts;                   // place in the tile's cluster
  const int m0 = (blockIdx.x / p.parts) * p.rows, m_end = min(p.S, m0 + p.rows);
  const int columns = p.NACC * p.NB, n_base = part * columns;

  if (tid == 0) {
    for (int s = 0; s < MAX_STAGES; ++s) {
      mbar_init(&bars[FULL + s], 1);
      mbar_init(&bars[FORMED + s], WARPS);
      mbar_init(&bars[FREE + s], 1);                       // SPLIT: of a unit
      mbar_init(&bars[B_FULL + s], 1);
    }
    mbar_init(&bars[ACC_DONE], 1);
    mbar_init(&bars[SIDE_READY], COMPUTE_THREADS);
    mbar_init(&bars[PEER_READY], TM * (p.parts > 1 ? p.parts - 1 : 1));
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == WARPS + 1) tmem_alloc(&meta.tmem_slot, p.tmem_columns);
  // The slots of a compute thread: rows of one of the stage's chunks, eight threads (16 bytes each) to the 128-byte piece
  // of a row.  Their ids and the mean come while the barriers and tensor memory are set up.
  const int per_chunk = COMPUTE_THREADS / kc, chunk_of = tid / per_chunk, piece = tid & 7;
  const int first_row = (tid % per_chunk) >> 3, row_step = per_chunk >> 3;
  int ids[SLOTS];
#pragma unroll
  for (int j = 0; j < SLOTS; ++j) {
    const int r = first_row + row_step * j, t = m0 + r;
    ids[j] = tid < COMPUTE_THREADS && r < p.rows && t < m_end ? load_id(p.ids, p.id_bytes, t) : 0;
  }
  // the eight columns of a piece as two halves 128 bytes apart: a quarter of a warp reads whole lines
  for (int i = tid; i < p.mean_bytes / 16; i += THREADS)
    reinterpret_cast<float4*>(mean_smem)[(i & ~15) + (i & 1) * 8 + ((i & 15) >> 1)] = __ldg(reinterpret_cast<const float4*>(p.mean) + i);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = meta.tmem_slot;
  // the column parts of one token tile write into each other's shared memory: nobody may do so before
  // the peers' barriers exist
  const bool joined = QUANT && !p.group32 && p.parts > 1;
  if (joined) cluster_arrive();
  bool ok = true, met = false;

  if (warp == WARPS) {
    if (lane == 0) {
      prefetch_tensormap(&map_x);
      prefetch_tensormap(&map_b);
      Ring at;
      if constexpr (SPLIT) {
        // chunks past the row's end arrive as zeros and are not used
        const int all = steps * p.NACC;
        int rows = 0, loaded = 0, row_place = 0, place = 0, column = 0, chunk = 0;
        auto load_rows = [&] {
          mbar_arrive_expect_tx(&bars[FULL + row_place], a_bytes);
          tma_load_3d(ring + row_place * a_bytes, &map_x, 0, m0, rows++ * kc, &bars[FULL + row_place]);
          if (++row_place == nst) row_place = 0;
        };
        auto load_unit = [&] {
          mbar_arrive_expect_tx(&bars[B_FULL + place], unit_bytes);
          tma_load_3d(units + place * unit_bytes, &map_b, 0, n_base + column, chunk, &bars[B_FULL + place]);
          ++loaded;
          if (++place == p.units) place = 0;
          column += p.NB;
          if (column == columns) { column = 0; chunk += kc; }
        };
        while (rows < min(nst, steps) || loaded < min(p.units, all)) {
          if (rows < min(nst, steps)) load_rows();
          if (loaded < min(p.units, all)) load_unit();
        }
        // a unit's MMAs done free its place, those of a stage's last unit the token rows' too
        int acc = 0;
        for (; ok && (rows < steps || loaded < all); at.advance(p.units)) {
          ok = mbar_wait(&bars[FREE + at.stage], at.phase, abort_flag, 400 + at.stage);
          if (!ok) break;
          if (++acc == p.NACC) {
            acc = 0;
            if (rows < steps) load_rows();
          }
          if (loaded < all) load_unit();
        }
      }
      for (int i = 0; !SPLIT && i < steps && ok; ++i, at.advance(nst)) {
        const int s = at.stage;
        if (i >= nst) ok = mbar_wait(&bars[FREE + s], at.phase ^ 1, abort_flag, 400 + s);
        if (!ok) break;
        uint8_t* stage = ring + s * stage_bytes;
        mbar_arrive_expect_tx(&bars[FULL + s], stage_bytes);   // chunks past the row's end arrive as zeros and are not used
        tma_load_3d(stage, &map_x, 0, m0, i * kc, &bars[FULL + s]);
        for (int a = 0; a < p.NACC; ++a)
          tma_load_3d(stage + a_bytes + a * kc * b_tile, &map_b, 0, n_base + a * p.NB, i * kc, &bars[FULL + s]);
      }
      if (!ok) {   // copies in flight land before the block goes away
        const long long start = clock64();
        while (clock64() - start < (1ll << 21)) {}
      }
    }
    __syncwarp();
  } else if (warp == WARPS + 1) {
    // The whole warp walks the uniform control flow; one elected lane issues.
    const bool leader = elect_one();
    const uint32_t idesc = make_idesc_bf16(TM, p.NB);
    const uint32_t ring_base = smem_u32(ring);
    if constexpr (SPLIT) {
      const uint32_t unit_base = smem_u32(units);
      Ring at, at_unit;
      for (int i = 0; i < steps && ok; ++i, at.advance(nst)) {
        ok = wait_all(&bars[FORMED + at.stage], at.phase, abort_flag, 410 + at.stage);
        const uint32_t rows = ring_base + at.stage * a_bytes;
        const int last = min(kc, nchunks - i * kc);
        for (int a = 0; a < p.NACC && ok; ++a, at_unit.advance(p.units)) {
          ok = wait_all(&bars[B_FULL + at_unit.stage], at_unit.phase, abort_flag, 420 + at_unit.stage);
          if (!ok) break;
          tc_fence_after();
          const uint32_t unit = unit_base + at_unit.stage * unit_bytes;
          if (leader) {
            for (int q = 0; q < last; ++q) {
              const uint64_t a_desc = make_smem_desc_sw128(rows + q * a_tile);
              const uint64_t b_desc = make_smem_desc_sw128(unit + q * b_tile);
#pragma unroll
              for (int k = 0; k < 4; ++k) mma_bf16(tmem_base + a * 256, a_desc + 2 * k, b_desc + 2 * k, idesc, (i | q | k) != 0);
            }
            mma_commit(&bars[FREE + at_unit.stage]);
          }
          __syncwarp();
        }
      }
    }
    Ring at;
    for (int i = 0; !SPLIT && i < steps && ok; ++i, at.advance(nst)) {
      const int s = at.stage;
      ok = wait_all(&bars[FORMED + s], at.phase, abort_flag, 410 + s);
      if (!ok) break;
      tc_fence_after();
      const uint32_t stage = ring_base + s * stage_bytes;
      const int last = min(kc, nchunks - i * kc);
      if (leader) {
        // an accumulator's MMAs follow one another at 86 cycles at the least; two accumulators take turns
        for (int q = 0; q < last; ++q) {
          const uint64_t a_desc = make_smem_desc_sw128(stage + q * a_tile);
          const uint64_t b_desc = make_smem_desc_sw128(stage + a_bytes + q * b_tile);
          const uint64_t b_next = make_smem_desc_sw128(stage + a_bytes + (kc + q) * b_tile);
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
    // ---- residual operand: bf16((x - centre[id]) - mean), in the place of x.  Loads carry no conditions: a row that
    // is not the tile's takes centre 0, a chunk past the row's end the last one, and what comes of them is not used.
    const uint16_t* crow[SLOTS];
    uint32_t place[SLOTS];
    bool stored[SLOTS];
#pragma unroll
    for (int j = 0; j < SLOTS; ++j) {
      const int r = first_row + row_step * j;
      stored[j] = r < p.rows_pad;
      place[j] = chunk_of * a_tile + (stored[j] ? r : 0) * 128 + ((piece ^ (r & 7)) << 4);
      crow[j] = p.centers + static_cast<size_t>(ids[j]) * p.J + piece * 8;
    }
    uint4 cq[DEPTH][SLOTS];
    auto fetch = [&](int buf, int i) {
      const int j0 = min((i * kc + chunk_of) * 64, p.J - 64);
#pragma unroll
      for (int j = 0; j < SLOTS; ++j) cq[buf][j] = __ldg(reinterpret_cast<const uint4*>(crow[j] + j0));
    };
#pragma unroll
    for (int b = 0; b < DEPTH; ++b) fetch(b, b);
    const uint64_t minus_one = pair_f32(-1.f, -1.f);
    Ring at;
    auto step = [&](int buf, int i) {
      const int s = at.stage;
      ok = wait_all(&bars[FULL + s], at.phase, abort_flag, 440 + s);
      if (!ok) return;
      uint8_t* stage = ring + s * stage_bytes;
      uint4 xv[SLOTS];
#pragma unroll
      for (int j = 0; j < SLOTS; ++j) xv[j] = *reinterpret_cast<const uint4*>(stage + place[j]);
      const int j0 = min((i * kc + chunk_of) * 64, p.J - 64);
      ulonglong2 m01, m23;
      if (p.mean_bytes > 0) {
        m01 = *reinterpret_cast<const ulonglong2*>(mean_smem + j0 + piece * 4);
        m23 = *reinterpret_cast<const ulonglong2*>(mean_smem + j0 + 32 + piece * 4);
      } else {
        m01 = __ldg(reinterpret_cast<const ulonglong2*>(p.mean + j0 + piece * 8));
        m23 = __ldg(reinterpret_cast<const ulonglong2*>(p.mean + j0 + piece * 8 + 4));
      }
      const uint64_t m2[4] = {m01.x, m01.y, m23.x, m23.y};
#pragma unroll
      for (int j = 0; j < SLOTS; ++j) {
        const uint32_t xw[4] = {xv[j].x, xv[j].y, xv[j].z, xv[j].w};
        const uint32_t cw[4] = {cq[buf][j].x, cq[buf][j].y, cq[buf][j].z, cq[buf][j].w};
        uint32_t out[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          // (x - c) - m in fp32, each difference rounded once: a + (-1) b is a - b
          const uint64_t x2 = pair_bits(xw[w] << 16, xw[w] & 0xFFFF0000u), c2 = pair_bits(cw[w] << 16, cw[w] & 0xFFFF0000u);
          float lo, hi;
          split_f32(fma_f32x2(m2[w], minus_one, fma_f32x2(c2, minus_one, x2)), lo, hi);
          out[w] = pack_bf16x2(lo, hi);
        }
        if (stored[j]) *reinterpret_cast<uint4*>(stage + place[j]) = make_uint4(out[0], out[1], out[2], out[3]);
      }
      fetch(buf, i + DEPTH);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[FORMED + s]);
      at.advance(nst);
    };
#pragma unroll 1
    for (int i = 0; i < steps && ok; i += DEPTH) {
#pragma unroll
      for (int b = 0; b < DEPTH; ++b)
        if (i + b < steps && ok) step(b, i + b);
    }
    if (ok) ok = wait_all(&bars[ACC_DONE], 0, abort_flag, 450);
    const int tok = m0 + row;
    const bool mine = row < p.rows && tok < m_end;
    const int column_chunks = __any_sync(0xffffffffu, mine) ? columns / 32 : 0;
    auto chunk = [&](int cc, uint32_t (&w)[16]) {
      const int col = cc * 32, acc = col / p.NB;
      float v[32];
      tmem_ld32(tmem_base + lane_sel + acc * 256 + (col - acc * p.NB), v);
      round_chunk(v, w);
#pragma unroll
      for (int i = 0; i < 16; ++i) w[i] = mine ? w[i] : 0u;     // rows that are nobody's hold anything
      return n_base + col;
    };
    if (ok) tc_fence_after();
    if (ok && QUANT && p.group32) {
      // ---- one scale per 32 coefficients: a thread's chunk is a group
#pragma unroll 1
      for (int cc = wg; cc < column_chunks; cc += GROUPS) {
        uint32_t w[16], worst = 0;
        const int col = chunk(cc, w);
        const float scale = scale_of(max_magnitude(w, worst), p);
        const uint4 words = pack_codes(w, scale, p.in_bf16, worst < NOT_FINITE);
        if (mine) {
          *reinterpret_cast<uint4*>(p.codes + static_cast<size_t>(tok) * (p.n_total >> 1) + (col >> 1)) = words;
          store_float(p.scales, p.scale_dtype, static_cast<size_t>(tok) * (p.n_total / 32) + col / 32, scale);
        }
      }
    } else if (ok && QUANT) {
      // ---- one scale per token.  Pass 1: |max| of the bf16-rounded coefficients of this thread's column chunks;
      // the two warpgroups, then the column parts' CTAs, combine.
      float amax = 0.f;
      uint32_t worst = 0;
#pragma unroll 1
      for (int cc = wg; cc < column_chunks; cc += GROUPS) {
        uint32_t w[16];
        chunk(cc, w);
        amax = fmaxf(amax, max_magnitude(w, worst));
      }
      meta.row_max[wg][row] = amax;
      mbar_arrive(&bars[SIDE_READY]);
      ok = wait_all(&bars[SIDE_READY], 0, abort_flag, 451);
      if (ok) {
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) amax = fmaxf(amax, meta.row_max[g][row]);
        if (joined) {
          cluster_wait();
          met = true;
          if (wg == 0) {
            for (int peer = 0; peer < p.parts; ++peer) {
              if (peer == part) continue;
              st_cluster_b32(map_to_cta(smem_u32(&meta.peer_max[part][row]), peer), __float_as_uint(amax));
              mbar_arrive_cluster(map_to_cta(smem_u32(&bars[PEER_READY]), peer));
            }
          }
          ok = wait_all_cluster(&bars[PEER_READY], 0, abort_flag, 452);
          if (ok)
            for (int peer = 0; peer < p.parts; ++peer)
              if (peer != part) amax = fmaxf(amax, meta.peer_max[peer][row]);
        }
      }
      if (ok) {
        const float scale = scale_of(amax, p);
#pragma unroll 1
        for (int cc = wg; cc < column_chunks; cc += GROUPS) {
          uint32_t w[16];
          const int col = chunk(cc, w);
          const uint4 words = pack_codes(w, scale, p.in_bf16, worst < NOT_FINITE);
          if (mine) *reinterpret_cast<uint4*>(p.codes + static_cast<size_t>(tok) * (p.n_total >> 1) + (col >> 1)) = words;
        }
        if (wg == 0 && part == 0 && mine) store_float(p.scales, p.scale_dtype, tok, scale);
      }
    } else if (ok) {
#pragma unroll 1
      for (int cc = wg; cc < column_chunks; cc += GROUPS) {
        uint32_t w[16];
        const int col = chunk(cc, w);
        if (mine) {
          uint4* dst = reinterpret_cast<uint4*>(p.coeff + static_cast<size_t>(tok) * p.n_total + col);
#pragma unroll
          for (int i = 0; i < 4; ++i) dst[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
        }
      }
    }
  }
  if (joined && !met) cluster_wait();
  tc_fence_before();
  __syncthreads();
  if (warp == WARPS + 1) tmem_dealloc(tmem_base, p.tmem_columns);
  // no CTA of a tile leaves while another may still write into its shared memory
  if (joined) cluster_sync_all();
}

// split n_total columns into grid.y CTAs x NACC accumulators x NB columns
bool plan_columns(int n_total, int* gy, int* nacc, int* nb) {
  for (int g = 1; g <= 16; ++g) {
    if (n_total % g) continue;
    int nc = n_total / g;
    if (nc <= 256 && nc % 32 == 0) { *gy = g; *nacc = 1; *nb = nc; return true; }
    if (nc <= 512 && nc % 64 == 0) { *gy = g; *nacc = 2; *nb = nc / 2; return true; }
  }
  return false;
}

constexpr size_t SMEM_LIMIT = 232448;

size_t mean_bytes(int J) { return J <= MAX_MEAN ? static_cast<size_t>(J) * 4 : 0; }

// the MMA reads 128 rows from where the last token tile starts, which may reach past the ring
size_t smem_bytes(int J, int rows_pad, int columns, int kc, int stages) {
  const size_t stage = static_cast<size_t>(kc) * (rows_pad + columns) * 128;
  const size_t end = stages * stage, last_a = (stages - 1) * stage + static_cast<size_t>(kc - 1) * rows_pad * 128;
  const size_t reach = last_a + TM * 128;
  return sizeof(Meta) + 16 + mean_bytes(J) + 1024 + (reach > end ? reach : end);
}
// the same for rings of their own
size_t split_bytes(int J, int rows_pad, int nb, int kc, int stages, int units) {
  const size_t tile = static_cast<size_t>(rows_pad) * 128, tiles = static_cast<size_t>(stages) * kc;
  const size_t end = tiles * tile + static_cast<size_t>(units) * kc * nb * 128, reach = (tiles - 1) * tile + TM * 128;
  return sizeof(Meta) + 16 + mean_bytes(J) + 1024 + (reach > end ? reach : end);
}

// Tokens per tile, column parts and chunks of a stage.  The estimate counts SM cycles.  A 64-column chunk costs the
// longer of its bytes from L2 (encoder rows, x and centre rows) at 45 per clock and its MMAs (four in a chain of 86
// cycles each at the least).  Clusters of more than four fill 128 of the 148 SMs, of three or four 144.
struct Cut { int rows, parts, kc, stages; };

Cut plan_project(int S, int J, int r, int first_parts, bool cluster) {
  const int sms = sm_count(), chunks = J / 64;
  Cut best{0, 0, 0, 0};
  double best_cost = -1;
  const int candidates[5] = {pick_rows(S, first_parts), 128, 96, 64, 32};
  for (int rows : candidates)
    for (int h = first_parts; h <= (cluster ? MAX_PARTS : 16); ++h) {
      const int cols = r / h, nacc = cols > 256 ? 2 : 1;
      if (r % h || cols > 512 || cols % (nacc == 2 ? 64 : 32)) continue;
      const int rows_pad = (rows + 7) / 8 * 8;
      Cut cut{rows, h, rows_pad <= 32 ? 4 : (rows_pad <= 64 ? 2 : 1), MAX_STAGES};
      while (cut.kc > 1 && smem_bytes(J, rows_pad, cols, cut.kc, 3) > SMEM_LIMIT) cut.kc /= 2;
      while (cut.stages > 2 && smem_bytes(J, rows_pad, cols, cut.kc, cut.stages) > SMEM_LIMIT) --cut.stages;
      const int room = !cluster ? sms : h > 4 ? sms - 20 : (h > 2 ? sms - 4 : sms);
      const double bytes = (rows * 256.0 + cols * 128.0) / 45;
      const double mma = nacc == 2 ? (4.0 * cols / 2 > 390 ? 4.0 * cols / 2 : 390) : (2.0 * cols > 340 + cols / 4 ? 2.0 * cols : 340 + cols / 4);
      const double chunk = bytes > mma ? bytes : mma;
      const double cost = static_cast<double>((static_cast<long long>(ceil_div(S, rows)) * h + room - 1) / room) *
                          (chunk * chunks + 18000 + cols * 20);
      if (best_cost < 0 || cost < best_cost) {
        best_cost = cost;
        best = cut;
      }
    }
  return best;
}

template <bool QUANT, bool SPLIT, int SLOTS, int DEPTH>
int launch_slots(const CUtensorMap (&maps)[2], const Params& p, size_t smem, cudaStream_t stream) {
  auto kernel = project_gemm_kernel<QUANT, SPLIT, SLOTS, DEPTH>;
  NKV_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(static_cast<unsigned>(ceil_div(p.S, p.rows)) * p.parts);
  config.blockDim = dim3(THREADS);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = QUANT && !p.group32 ? p.parts : 1;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  config.attrs = &attr;
  config.numAttrs = 1;
  NKV_CUDA(cudaLaunchKernelEx(&config, kernel, maps[0], maps[1], p));
  return NKV_OK;
}

template <bool QUANT>
int launch_project(const void* x, const void* centers, const void* encoder, Params& p, cudaStream_t stream) {
  NKV_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(centers) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(p.mean) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(QUANT ? static_cast<const void*>(p.codes) : p.coeff) & 15) == 0 &&
                  (!QUANT || (p.n_total / 2) % 16 == 0),
              NKV_ERR_INVALID, "projection operands must be 16-byte aligned");
  int gy, nacc, nb;
  NKV_REQUIRE(plan_columns(p.n_total, &gy, &nacc, &nb), NKV_ERR_UNSUPPORTED, "projection rank %d cannot be tiled", p.n_total);
  NKV_REQUIRE(!QUANT || p.group32 || gy <= 2, NKV_ERR_UNSUPPORTED,
              "fused projection: rank %d cannot be tiled over at most two column parts", p.n_total);
  const Cut cut = plan_project(p.S, p.J, p.n_total, gy, QUANT && !p.group32);
  p.rows = cut.rows; p.parts = cut.parts; p.kc = cut.kc; p.nstages = cut.stages;
  p.rows_pad = (p.rows + 7) / 8 * 8;
  const int columns = p.n_total / p.parts;
  p.NACC = columns > 256 ? 2 : 1;
  p.NB = columns / p.NACC;
  p.tmem_columns = p.NACC == 2 ? 512 : (p.NB > 128 ? 256 : (p.NB > 64 ? 128 : (p.NB > 32 ? 64 : 32)));
  p.nchunks = p.J / 64;
  p.mean_bytes = static_cast<int>(mean_bytes(p.J));
  p.centers = static_cast<const uint16_t*>(centers);
  // two accumulators with room for two whole stages only (512 columns): as many units as fit beside their token rows,
  // five or four, and token rows in the rest
  const bool split = p.NACC == 2 && p.nstages == 2;
  size_t smem = smem_bytes(p.J, p.rows_pad, columns, p.kc, p.nstages);
  if (split) {
    auto bytes = [&](int stages, int units) { return split_bytes(p.J, p.rows_pad, p.NB, p.kc, stages, units); };
    p.units = MAX_STAGES;
    while (p.units > 4 && bytes((p.units + 1) / 2, p.units) > SMEM_LIMIT) --p.units;
    p.nstages = MAX_STAGES;
    while (p.nstages > 2 && bytes(p.nstages, p.units) > SMEM_LIMIT) --p.nstages;
    smem = bytes(p.nstages, p.units);
  }
  NKV_REQUIRE(smem <= SMEM_LIMIT, NKV_ERR_UNSUPPORTED, "projection: %zu bytes of shared memory", smem);
  CUtensorMap maps[2];     // rows, encoder
  const uint64_t chunk_strides[2] = {static_cast<uint64_t>(p.J) * 2, 128};
  {
    const uint64_t dims[3] = {64, static_cast<uint64_t>(p.S), static_cast<uint64_t>(p.nchunks)};
    const uint32_t box[3] = {64, static_cast<uint32_t>(p.rows_pad), static_cast<uint32_t>(p.kc)};
    const int rc = encode_tensor_map(&maps[0], 2, x, 3, dims, chunk_strides, box, 128);
    if (rc != NKV_OK) return rc;
  }
  {
    const uint64_t dims[3] = {64, static_cast<uint64_t>(p.n_total), static_cast<uint64_t>(p.nchunks)};
    const uint32_t box[3] = {64, static_cast<uint32_t>(p.NB), static_cast<uint32_t>(p.kc)};
    const int rc = encode_tensor_map(&maps[1], 2, encoder, 3, dims, chunk_strides, box, 128);
    if (rc != NKV_OK) return rc;
  }
  const int slots = ceil_div(p.rows_pad, COMPUTE_THREADS / 8 / p.kc);
  auto launch = slots <= 1   ? (split ? launch_slots<QUANT, true, 1, 6> : launch_slots<QUANT, false, 1, 6>)
                : slots <= 2 ? (split ? launch_slots<QUANT, true, 2, 4> : launch_slots<QUANT, false, 2, 4>)
                             : (split ? launch_slots<QUANT, true, 4, 3> : launch_slots<QUANT, false, 4, 3>);
  return launch(maps, p, smem, stream);
}

}  // namespace

bool tc_project_supported(int J, int r) {
  int gy, nacc, nb;
  return J % 64 == 0 && plan_columns(r, &gy, &nacc, &nb);
}

// SM count of the current device, cached per device ordinal
int sm_count() {
  static std::atomic<int> cached[64];
  int device = 0, sms = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) device = -1;
  if (device >= 0) sms = cached[device].load(std::memory_order_relaxed);
  if (sms == 0) {
    if (device < 0 ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0)
      sms = 148;
    if (device >= 0) cached[device].store(sms, std::memory_order_relaxed);
  }
  return sms;
}

// Tokens per CTA (<= TM): the MMA always spans TM rows, but the operand build, the loads and the
// epilogue scale with the rows a CTA owns, so the token tiles are sized to fill whole rounds of the
// SMs instead of leaving the last round mostly empty (12,480 tokens: 147 CTAs of 85 rows instead
// of 98 of 128).  Not below 64 rows: every CTA streams the whole B operand from L2.
int pick_rows(int S, int column_parts) {
  const int sms = sm_count();
  const long long units = static_cast<long long>(ceil_div(S, TM)) * column_parts;
  const long long waves = (units + sms - 1) / sms;
  const long long tiles = waves * sms / column_parts;
  long long rows = (S + tiles - 1) / (tiles > 0 ? tiles : 1);
  rows = rows < 64 ? 64 : (rows > TM ? TM : rows);
  return static_cast<int>(rows);
}

int tc_project(const void* x_bf16, const void* centers_bf16, const void* ids, int id_bytes,
               const float* mean, const void* encoder_bf16, int S, int J, int r, void* coeff,
               cudaStream_t stream) {
  if (S == 0) return NKV_OK;
  Params p{};
  p.S = S; p.J = J; p.n_total = r;
  p.ids = ids; p.id_bytes = id_bytes; p.mean = mean;
  p.coeff = static_cast<uint16_t*>(coeff);
  return launch_project<false>(x_bf16, centers_bf16, encoder_bf16, p, stream);
}

bool tc_project_quant_supported(int J, int r, int group) {
  int gy, nacc, nb;
  if (!tc_project_supported(J, r) || !plan_columns(r, &gy, &nacc, &nb)) return false;
  return group == r ? r % 64 == 0 && gy <= 2 : group == 32;
}

int tc_project_quant(const void* x_bf16, const void* centers_bf16, const void* ids, int id_bytes,
                     const float* mean, const void* encoder_bf16, int S, int J, int r, int group, float eps,
                     int quant_mode, int scale_dtype, uint8_t* codes, void* scales, cudaStream_t stream) {
  if (S == 0) return NKV_OK;
  Params p{};
  p.S = S; p.J = J; p.n_total = r;
  p.ids = ids; p.id_bytes = id_bytes; p.mean = mean;
  p.codes = codes; p.scales = scales; p.eps = eps;
  p.in_bf16 = quant_mode == NKV_QUANT_IN_BF16 ? 1 : 0;
  p.scale_dtype = scale_dtype;
  p.group32 = group != r ? 1 : 0;
  return launch_project<true>(x_bf16, centers_bf16, encoder_bf16, p, stream);
}

}  // namespace nkv
