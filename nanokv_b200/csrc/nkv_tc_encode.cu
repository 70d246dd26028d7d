// Encoder projection on tcgen05: [128 tokens x K=J] x [N x K]^T tiles with fp32 accumulators in TMEM,
// K streamed 64 columns at a time through a shared-memory ring of up to eight stages.
//   project: A = bf16((x - centre[id]) - mean), formed by the compute warps in
//            the swizzled operand layout; B = encoder rows (TMA); the epilogue
//            rounds once to bf16.
//   project + quantise: the same GEMM, but the epilogue keeps the coefficients in TMEM, takes the
//            token's absolute maximum over the whole rank row (the up to eight column parts of a token
//            tile form a cluster and swap the maxima of their columns through each other's shared
//            memory), quantises to INT4, packs two codes per byte and writes codes and scale to
//            their place in the history: the bf16 coefficients never travel to HBM.
// A CTA covers up to 512 output columns as 1 or 2 accumulators of NB <= 256.
// Calls of a few thousand tokens have too few token tiles for 148 SMs, and a tile's time is the length
// of its K loop (J / 64 stages of operand latency).  Such calls of the projection take more column parts
// per tile (plan_split).  K itself is never cut: every sum runs in the order of K whatever the call's
// length, so that a row gets the same id, codes and scale in a chunk of any size.
// Warps 0-7 compute, warp 8 lane 0 issues TMA, warp 9 lane 0 issues MMA.
#include <atomic>

#include "nkv_internal.h"
#include "nkv_tc.cuh"

namespace nkv {

int pick_rows(int S, int column_parts);

namespace {

using namespace tc;

constexpr int TM = 128;
constexpr int COMPUTE_THREADS = 256;
constexpr int THREADS = COMPUTE_THREADS + 64;
constexpr int A_BYTES = 128 * 128;

constexpr int MAX_STAGES = 8;
enum Bar { TMA_FULL = 0, A_FULL = 8, STAGE_FREE = 16, ACC_DONE = 24, SIDE_READY = 25, CAND_READY = 26,
           PEER_READY = 27, NUM_BARS = 28 };
enum Mode { PROJECT = 0, PROJECT_QUANT = 2 };
constexpr int META_HEAD = 256;      // barriers, TMEM slot, abort flag
constexpr int WARPS = COMPUTE_THREADS / 32;
constexpr int MAX_PARTS = 8;        // thread blocks of one token tile that form a cluster

struct Params {
  int S, J, NB, NACC, n_total;      // n_total = r (project) or C (assign)
  int nstages;                      // depth of the shared-memory operand ring (2..MAX_STAGES)
  int rows;                         // tokens of a tile (<= TM)
  // project
  const uint16_t* x; const uint16_t* centers; const void* ids; int id_bytes;
  const float* mean; uint16_t* coeff;
  // project + quantise: codes u8 [S, r/2] and scales [S] at the history's token offset
  uint8_t* codes; void* scales; float eps; int in_bf16; int scale_dtype; int column_parts;
};

template <int MODE>
__global__ void __launch_bounds__(THREADS, 1)
encode_gemm_kernel(const __grid_constant__ CUtensorMap map_a,
                   const __grid_constant__ CUtensorMap map_b, Params p) {
  constexpr bool QUANT = MODE == PROJECT_QUANT;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int b_bytes = p.NB * 128;                       // one accumulator's B tile
  const int stage_bytes = A_BYTES + p.NACC * b_bytes;
  const int nst = p.nstages;
  uint8_t* meta = smem + nst * stage_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(meta);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(meta + NUM_BARS * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(meta + NUM_BARS * 8 + 4);
  float* xn_part = reinterpret_cast<float*>(meta + META_HEAD);    // [256]
  float* peer_max = xn_part + 512;                                // project + quantise: [MAX_PARTS][128]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int part = blockIdx.x % p.column_parts;         // place in the tile's cluster
  const int m0 = (blockIdx.x / p.column_parts) * p.rows;   // this tile's tokens: [m0, m_end)
  const int m_end = min(p.S, m0 + p.rows);
  const int n_base = part * p.NACC * p.NB;
  const int nchunks = p.J / 64;

  if (tid == 0) {
    for (int s = 0; s < MAX_STAGES; ++s) {
      mbar_init(&bars[TMA_FULL + s], 1);
      mbar_init(&bars[A_FULL + s], WARPS);
      mbar_init(&bars[STAGE_FREE + s], 1);
    }
    mbar_init(&bars[ACC_DONE], 1);
    mbar_init(&bars[SIDE_READY], COMPUTE_THREADS);
    mbar_init(&bars[CAND_READY], 128);
    mbar_init(&bars[PEER_READY], 128 * (p.column_parts > 1 ? p.column_parts - 1 : 1));
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 9) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // the column parts of one token tile write into each other's shared memory: nobody may do so before
  // the peers' barriers exist
  const bool joined = QUANT && p.column_parts > 1;
  if (joined) cluster_sync_all();
  bool ok = true;

  if (warp == 8) {
    if (lane == 0) {
      prefetch_tensormap(&map_b);
      Ring at;
      for (int c = 0; c < nchunks && ok; ++c, at.advance(nst)) {
        const int s = at.stage;
        if (c >= nst) ok = mbar_wait(&bars[STAGE_FREE + s], at.phase ^ 1, abort_flag, 400 + s);
        if (!ok) break;
        uint8_t* stage = smem + s * stage_bytes;
        mbar_arrive_expect_tx(&bars[TMA_FULL + s], p.NACC * b_bytes);
        for (int a = 0; a < p.NACC; ++a)
          tma_load_2d(stage + A_BYTES + a * b_bytes, &map_b, c * 64, n_base + a * p.NB,
                      &bars[TMA_FULL + s]);
      }
      if (!ok) {
        const long long start = clock64();
        while (clock64() - start < (1ll << 21)) {}
      }
    }
    __syncwarp();
  } else if (warp == 9) {
    // The whole warp walks the uniform control flow; one elected lane issues.
    const bool leader = elect_one();
    const uint32_t idesc = make_idesc_bf16(128, p.NB);
    const uint32_t smem_base = smem_u32(smem);
    Ring at;
    for (int c = 0; c < nchunks && ok; ++c, at.advance(nst)) {
      const int s = at.stage;
      ok = wait_all(&bars[TMA_FULL + s], at.phase, abort_flag, 410 + s);
      if (ok) ok = wait_all(&bars[A_FULL + s], at.phase, abort_flag, 412 + s);
      if (!ok) break;
      tc_fence_after();
      const uint32_t stage = smem_base + s * stage_bytes;
      const uint64_t a_desc = make_smem_desc_sw128(stage);
      for (int a = 0; a < p.NACC; ++a) {
        const uint64_t b_desc = make_smem_desc_sw128(stage + A_BYTES + a * b_bytes);
        if (leader) {
          mma_bf16(tmem_base + a * 256, a_desc, b_desc, idesc, c > 0);
          mma_bf16(tmem_base + a * 256, a_desc + 2, b_desc + 2, idesc, true);
          mma_bf16(tmem_base + a * 256, a_desc + 4, b_desc + 4, idesc, true);
          mma_bf16(tmem_base + a * 256, a_desc + 6, b_desc + 6, idesc, true);
        }
      }
      if (leader) mma_commit(&bars[STAGE_FREE + s]);
      __syncwarp();
    }
    if (ok && leader) mma_commit(&bars[ACC_DONE]);
    __syncwarp();
  } else {
    const int row = tid & 127, wg = tid >> 7;
    const uint32_t lane_sel = static_cast<uint32_t>(32 * (warp & 3)) << 16;
    // eight threads share a 128-byte row chunk (16 bytes each), a thread serves rows r0 + 32 i: loads and
    // the swizzled stores touch whole lines
    const int r0 = tid >> 3, piece = tid & 7;
    {
      // ---- residual operand: bf16((x - centre[id]) - mean), 8 columns of four rows per thread and
      // chunk; the operands of two chunks are in flight while one is formed
      const uint16_t* xrow[4];
      const uint16_t* crow[4];
      bool in[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = r0 + 32 * j, t = m0 + r;
        in[j] = r < p.rows && t < m_end;
        xrow[j] = p.x + static_cast<size_t>(in[j] ? t : 0) * p.J + piece * 8;
        crow[j] = p.centers + static_cast<size_t>(in[j] ? load_id(p.ids, p.id_bytes, t) : 0) * p.J + piece * 8;
      }
      uint4 xq[2][4], cq[2][4];
      float4 mq[2][2];
      auto fetch = [&](int buf, int i) {
        if (i >= nchunks) return;
        const int j0 = i * 64;
        mq[buf][0] = __ldg(reinterpret_cast<const float4*>(p.mean + j0 + piece * 8));
        mq[buf][1] = __ldg(reinterpret_cast<const float4*>(p.mean + j0 + piece * 8) + 1);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (in[j]) {
            xq[buf][j] = __ldg(reinterpret_cast<const uint4*>(xrow[j] + j0));
            cq[buf][j] = __ldg(reinterpret_cast<const uint4*>(crow[j] + j0));
          }
      };
      Ring at;
      auto step = [&](int buf, int i) {
        const int s = at.stage;
        const float mv[8] = {mq[buf][0].x, mq[buf][0].y, mq[buf][0].z, mq[buf][0].w,
                             mq[buf][1].x, mq[buf][1].y, mq[buf][1].z, mq[buf][1].w};
        uint4 out[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          out[j] = make_uint4(0, 0, 0, 0);
          if (in[j]) {
            const uint32_t xw[4] = {xq[buf][j].x, xq[buf][j].y, xq[buf][j].z, xq[buf][j].w};
            const uint32_t cw[4] = {cq[buf][j].x, cq[buf][j].y, cq[buf][j].z, cq[buf][j].w};
            uint32_t* o = &out[j].x;
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              const float lo = __fsub_rn(__fsub_rn(__uint_as_float(xw[w] << 16), __uint_as_float(cw[w] << 16)), mv[2 * w]);
              const float hi = __fsub_rn(__fsub_rn(__uint_as_float(xw[w] & 0xFFFF0000u),
                                                   __uint_as_float(cw[w] & 0xFFFF0000u)), mv[2 * w + 1]);
              o[w] = pack_bf16x2(lo, hi);
            }
          }
        }
        fetch(buf, i + 2);
        if (i >= nst) ok = wait_all(&bars[STAGE_FREE + s], at.phase ^ 1, abort_flag, 440 + s);
        if (!ok) return;
        at.advance(nst);
        uint8_t* stage = smem + s * stage_bytes + r0 * 128 + ((piece ^ (r0 & 7)) << 4);
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(stage + j * 32 * 128) = out[j];
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[A_FULL + s]);
      };
      fetch(0, 0);
      fetch(1, 1);
      for (int i = 0; i < nchunks && ok; i += 2) {
        step(0, i);
        if (i + 1 < nchunks && ok) step(1, i + 1);
      }
      if (ok) ok = wait_all(&bars[ACC_DONE], 0, abort_flag, 450);
      if (ok && QUANT) {
        // ---- quantise + pack from TMEM.  Pass 1: |max| of the bf16-rounded coefficients of this
        // thread's column chunks; the two warpgroups, then the column parts' CTAs, combine.
        tc_fence_after();
        const int nc = p.NACC * p.NB;
        const int tok = m0 + row;
        float amax = 0.f;
#pragma unroll 1
        for (int cc = wg; cc < nc / 32; cc += 2) {
          const int col = cc * 32, acc = col / p.NB;
          float v[32];
          tmem_ld32(tmem_base + lane_sel + acc * 256 + (col - acc * p.NB), v);
#pragma unroll
          for (int j = 0; j < 32; ++j) amax = fmaxf(amax, fabsf(round_to_bf16(v[j])));
        }
        xn_part[wg * 128 + row] = amax;
        mbar_arrive(&bars[SIDE_READY]);
        ok = wait_all(&bars[SIDE_READY], 0, abort_flag, 451);
        if (ok) {
          amax = fmaxf(xn_part[row], xn_part[128 + row]);
          if (joined) {
            if (wg == 0) {
              for (int peer = 0; peer < p.column_parts; ++peer) {
                if (peer == part) continue;
                st_cluster_b32(map_to_cta(smem_u32(&peer_max[part * 128 + row]), peer), __float_as_uint(amax));
                mbar_arrive_cluster(map_to_cta(smem_u32(&bars[PEER_READY]), peer));
              }
            }
            ok = wait_all_cluster(&bars[PEER_READY], 0, abort_flag, 452);
            if (ok)
              for (int peer = 0; peer < p.column_parts; ++peer)
                if (peer != part) amax = fmaxf(amax, peer_max[peer * 128 + row]);
          }
        }
        if (ok) {
          float scale;
          if (p.in_bf16) scale = round_to_bf16(__fdiv_rn(fmaxf(amax, round_to_bf16(p.eps)), 7.0f));
          else scale = __fdiv_rn(fmaxf(amax, p.eps), 7.0f);
          const float inv = __frcp_rn(scale);
#pragma unroll 1
          for (int cc = wg; cc < nc / 32; cc += 2) {
            const int col = cc * 32, acc = col / p.NB;
            float v[32];
            tmem_ld32(tmem_base + lane_sel + acc * 256 + (col - acc * p.NB), v);
            uint32_t words[4];
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              uint32_t out = 0;
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const float z0 = round_to_bf16(v[w * 8 + 2 * k]), z1 = round_to_bf16(v[w * 8 + 2 * k + 1]);
                const int c0 = p.in_bf16 ? quant_code<true>(z0, scale, inv) : quant_code<false>(z0, scale, inv);
                const int c1 = p.in_bf16 ? quant_code<true>(z1, scale, inv) : quant_code<false>(z1, scale, inv);
                out |= static_cast<uint32_t>(c0 | (c1 << 4)) << (8 * k);
              }
              words[w] = out;
            }
            if (tok < m_end)
              *reinterpret_cast<uint4*>(p.codes + static_cast<size_t>(tok) * (p.n_total >> 1) +
                                        ((n_base + col) >> 1)) = make_uint4(words[0], words[1], words[2], words[3]);
          }
          if (wg == 0 && part == 0 && tok < m_end) store_float(p.scales, p.scale_dtype, tok, scale);
        }
      } else if (ok) {
        tc_fence_after();
        const int nc = p.NACC * p.NB;
        const int tok = m0 + row;
#pragma unroll 1
        for (int cc = wg; cc < nc / 32; cc += 2) {
          const int col = cc * 32, acc = col / p.NB;
          float v[32];
          tmem_ld32(tmem_base + lane_sel + acc * 256 + (col - acc * p.NB), v);
          if (tok < m_end) {
            uint16_t* dst = p.coeff + static_cast<size_t>(tok) * p.n_total + n_base + col;
#pragma unroll
            for (int j4 = 0; j4 < 4; ++j4) {
              uint4 w;
              w.x = pack_bf16x2(v[j4 * 8 + 0], v[j4 * 8 + 1]);
              w.y = pack_bf16x2(v[j4 * 8 + 2], v[j4 * 8 + 3]);
              w.z = pack_bf16x2(v[j4 * 8 + 4], v[j4 * 8 + 5]);
              w.w = pack_bf16x2(v[j4 * 8 + 6], v[j4 * 8 + 7]);
              *reinterpret_cast<uint4*>(dst + j4 * 8) = w;
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem_base, 512);
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

// n_norms: centres whose squared norms are kept (assign); 512 floats of them, or the parts' row maxima
size_t meta_bytes(int n_norms) {
  const size_t tail = 8 * static_cast<size_t>(n_norms);
  return META_HEAD + 4 * (256 + 128 + 128) + (tail > 4 * MAX_PARTS * 128 ? tail : 4 * MAX_PARTS * 128);
}

size_t ring_bytes(int nacc, int nb, int stages) { return stages * static_cast<size_t>(A_BYTES + nacc * nb * 128); }

size_t smem_bytes(int nacc, int nb, int n_total, int stages = 2) {
  return ring_bytes(nacc, nb, stages) + meta_bytes(n_total) + 1024;
}

constexpr size_t SMEM_LIMIT = 232448;

// How a GEMM of S tokens x `columns` over `chunks` stages is cut: tokens per tile and column parts.
// The estimate counts SM cycles: a stage costs the bytes it takes from L2 (token rows, centre rows, B) at
// 48 bytes per clock, at least 350 cycles of latency.  Column parts of the projection form clusters of up
// to eight, of which 128 of the 148 SMs hold whole ones at a time, of four about 144.
// Bound of short calls: 880 tokens x 3,072 columns x rank 384 in tiles of 128 whole rows keep 14 SMs busy for
// 48 stages of operand latency (107 us; 39 with six column parts); 4,680 x 5,120 x 640 71 (128 before the
// operands of two chunks were in flight); assignment to 64 fp32 centres 880 x 3,072 49 (70), 4,680 x 5,120 80
// (116).  Cutting K over a cluster as well was faster still for given centres (assignment of 1,560 x 3,072 to
// 256 centres 28 us against 60), but then the order of a row's fp32 sums, and now and then a code or an id,
// depends on the length of the call.
struct Split { int rows, column_parts; };

Split plan_split(int S, int chunks, int columns, int column_parts, bool residual) {
  const int sms = sm_count();
  Split best{pick_rows(S, column_parts), column_parts};
  auto stage_cost = [&](int rows, int cols) {
    const double bytes = rows * (residual ? 256.0 : 128.0) + cols * 128.0;
    return bytes / 48 > 350 ? bytes / 48 : 350.0;
  };
  auto rounds = [](long long ctas, int room) { return static_cast<double>((ctas + room - 1) / room); };
  double best_cost = rounds(static_cast<long long>(ceil_div(S, best.rows)) * column_parts, sms) *
                     (chunks * stage_cost(best.rows, columns / column_parts) + 3000);
  for (int rows = 64; rows <= TM; rows *= 2)
    for (int h = column_parts; h <= (residual ? MAX_PARTS : column_parts); ++h) {
      const int cols = columns / h;
      if (columns % h || cols > 512 || cols % (cols > 256 ? 64 : 32)) continue;
      const int room = h > 4 ? sms - 20 : (h > 2 ? sms - 4 : sms);
      const double cost = rounds(static_cast<long long>(ceil_div(S, rows)) * h, room) *
                          (chunks * stage_cost(rows, cols) + 3000 + 300 * h);
      if (cost < best_cost) {
        best_cost = cost;
        best = Split{rows, h};
      }
    }
  return best;
}

// accumulators of one CTA's columns
void set_columns(Params& p, int columns) {
  p.NACC = columns > 256 ? 2 : 1;
  p.NB = columns / p.NACC;
}

template <int MODE>
int launch_gemm(const CUtensorMap& map_a, const CUtensorMap& map_b, Params& p, int n_norms, const char* name,
                cudaStream_t stream) {
  p.nstages = MAX_STAGES;
  while (p.nstages > 2 && smem_bytes(p.NACC, p.NB, n_norms, p.nstages) > SMEM_LIMIT) --p.nstages;
  const size_t smem = smem_bytes(p.NACC, p.NB, n_norms, p.nstages);
  NKV_REQUIRE(smem <= SMEM_LIMIT, NKV_ERR_UNSUPPORTED, "%s needs %zu bytes of shared memory", name, smem);
  auto kernel = encode_gemm_kernel<MODE>;
  NKV_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(static_cast<unsigned>(ceil_div(p.S, p.rows)) * p.column_parts);
  config.blockDim = dim3(THREADS);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = MODE == PROJECT_QUANT ? p.column_parts : 1;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  config.attrs = &attr;
  config.numAttrs = 1;
  NKV_CUDA(cudaLaunchKernelEx(&config, kernel, map_a, map_b, p));
  return NKV_OK;
}

}  // namespace

bool tc_project_supported(int J, int r) {
  int gy, nacc, nb;
  return J % 64 == 0 && plan_columns(r, &gy, &nacc, &nb) &&
         smem_bytes(nacc, nb, 0) <= 232448;
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
  int gy;
  NKV_REQUIRE(plan_columns(r, &gy, &p.NACC, &p.NB), NKV_ERR_UNSUPPORTED,
              "projection rank %d cannot be tiled", r);
  const Split cut = plan_split(S, J / 64, r, gy, true);
  p.rows = cut.rows; p.column_parts = cut.column_parts;
  set_columns(p, r / p.column_parts);
  NKV_REQUIRE((reinterpret_cast<uintptr_t>(x_bf16) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(centers_bf16) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(mean) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(coeff) & 15) == 0,
              NKV_ERR_INVALID, "projection operands must be 16-byte aligned");
  p.S = S; p.J = J; p.n_total = r;
  p.x = static_cast<const uint16_t*>(x_bf16);
  p.centers = static_cast<const uint16_t*>(centers_bf16);
  p.ids = ids; p.id_bytes = id_bytes; p.mean = mean;
  p.coeff = static_cast<uint16_t*>(coeff);
  CUtensorMap map_b;
  uint64_t dims[2] = {static_cast<uint64_t>(J), static_cast<uint64_t>(r)};
  uint64_t strides[1] = {static_cast<uint64_t>(J) * 2};
  uint32_t box[2] = {64, static_cast<uint32_t>(p.NB)};
  int rc = encode_tensor_map(&map_b, 2, encoder_bf16, 2, dims, strides, box, 128);
  if (rc != NKV_OK) return rc;
  return launch_gemm<PROJECT>(map_b, map_b, p, 0, "encode_gemm_kernel<project>", stream);
}

bool tc_project_quant_supported(int J, int r, int group) {
  int gy, nacc, nb;
  return group == r && r % 64 == 0 && tc_project_supported(J, r) && plan_columns(r, &gy, &nacc, &nb) && gy <= 2;
}

int tc_project_quant(const void* x_bf16, const void* centers_bf16, const void* ids, int id_bytes,
                     const float* mean, const void* encoder_bf16, int S, int J, int r, float eps,
                     int quant_mode, int scale_dtype, uint8_t* codes, void* scales, cudaStream_t stream) {
  if (S == 0) return NKV_OK;
  Params p{};
  int gy;
  NKV_REQUIRE(plan_columns(r, &gy, &p.NACC, &p.NB) && gy <= 2, NKV_ERR_UNSUPPORTED,
              "fused projection: rank %d cannot be tiled over at most two column parts", r);
  const Split cut = plan_split(S, J / 64, r, gy, true);
  p.rows = cut.rows; p.column_parts = cut.column_parts;
  set_columns(p, r / p.column_parts);
  NKV_REQUIRE((reinterpret_cast<uintptr_t>(x_bf16) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(centers_bf16) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(mean) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(codes) & 15) == 0 && (r / 2) % 16 == 0,
              NKV_ERR_INVALID, "fused projection operands must be 16-byte aligned");
  p.S = S; p.J = J; p.n_total = r;
  p.x = static_cast<const uint16_t*>(x_bf16);
  p.centers = static_cast<const uint16_t*>(centers_bf16);
  p.ids = ids; p.id_bytes = id_bytes; p.mean = mean;
  p.codes = codes; p.scales = scales; p.eps = eps;
  p.in_bf16 = quant_mode == NKV_QUANT_IN_BF16 ? 1 : 0;
  p.scale_dtype = scale_dtype;
  CUtensorMap map_b;
  uint64_t dims[2] = {static_cast<uint64_t>(J), static_cast<uint64_t>(r)};
  uint64_t strides[1] = {static_cast<uint64_t>(J) * 2};
  uint32_t box[2] = {64, static_cast<uint32_t>(p.NB)};
  int rc = encode_tensor_map(&map_b, 2, encoder_bf16, 2, dims, strides, box, 128);
  if (rc != NKV_OK) return rc;
  return launch_gemm<PROJECT_QUANT>(map_b, map_b, p, 0, "encode_gemm_kernel<project + quantise>", stream);
}

}  // namespace nkv
