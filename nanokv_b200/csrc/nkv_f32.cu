// fp32 GEMMs and attention on the CUDA cores: nearest-centre assignment, residual projection, row decode
// and the attention of rebuilt rows.
//
// These carry the fp32 configuration (operators stored in fp32, where the reference runs true IEEE fp32
// GEMMs and tensor cores have no matching mode) and the C-means of fp32 rows.  With bf16 operands they
// reproduce the rounding points of the bf16 path, which the test-suite uses to cross-check the
// tensor-core kernels at full size.
//
// Assignment and projection: every sum is one chain of fused multiply-adds in the order of K, because what they give is
// stored -- ids, and codes that another order would move now and then.  assign_few_kernel and project_rows_kernel take
// aligned fp32 rows; gemm_ordered takes the rest, with packed multiply-adds and two steps' operands in registers.
// Row decode (gemm64): 64 x 64 of the product per block; its four groups of 64 threads take a quarter of K each,
// with operand tiles and barriers of their own, and add their sums in order at the end.
#include "nkv_internal.h"

namespace nkv {
namespace {

constexpr int TILE = 64, BK = 16, GROUPS = 4, GROUP_THREADS = 64, THREADS = GROUPS * GROUP_THREADS;
constexpr int PITCH = TILE + 4;                          // of a column of K in gemm64's operand tiles
constexpr int OPERAND = BK * PITCH;                      // floats of one operand tile
constexpr int SMEM_FLOATS = GROUPS * 2 * 2 * OPERAND;    // two buffers of two operands per group
static_assert(SMEM_FLOATS >= GROUPS * TILE * TILE, "the partial sums reuse the operand tiles");

// elements k .. k + 3 of a row (0 past K); `vector`: rows start on 16 (fp32) or 8 (16-bit) bytes, K % 4 == 0
__device__ __forceinline__ float4 load4(const void* base, int dtype, size_t row_start, int k, int K, bool vector) {
  if (vector && k + 4 <= K) {
    if (dtype == NKV_F32) return __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(base) + row_start + k));
    if (dtype == NKV_BF16) {
      const uint2 w = __ldg(reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(base) + row_start + k));
      return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xFFFF0000u),
                         __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xFFFF0000u));
    }
  }
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = k + i < K ? load_float(base, dtype, row_start + k + i) : 0.f;
  return make_float4(v[0], v[1], v[2], v[3]);
}

bool vector_rows(const void* base, int dtype, int K) {
  return K % 4 == 0 && (reinterpret_cast<uintptr_t>(base) & (dtype == NKV_F32 ? 15 : 7)) == 0;
}

// The block's 64 x 64 tile of A B^T over K: op.fetch(c) requests the operands' chunk c of BK columns for the thread's
// group, op.stage(as, bs) puts them into shared memory, column k of K at k * PITCH.  Afterwards the tile's sums lie in
// `sm` as GROUPS partial tiles; the caller's barrier comes before tile_sum.
template <class Operands>
__device__ __forceinline__ void gemm64(float* sm, int K, Operands& op) {
  const int g = threadIdx.x / GROUP_THREADS, t = threadIdx.x % GROUP_THREADS;
  const int tx = t & 7, ty = t >> 3;          // rows ty * 8 .. + 7, columns tx * 4 .. + 3 and 32 + tx * 4 .. + 3
  const int chunks = (K + BK - 1) / BK;
  const int first = chunks * g / GROUPS, last = chunks * (g + 1) / GROUPS;
  float* mine = sm + g * 4 * OPERAND;
  uint64_t acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  if (first < last) op.fetch(first);
#pragma unroll 1
  for (int c = first; c < last; ++c) {
    float* as = mine + (c & 1) * 2 * OPERAND;
    float* bs = as + OPERAND;
    op.stage(as, bs);
    asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "n"(GROUP_THREADS) : "memory");
    if (c + 1 < last) op.fetch(c + 1);
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      const float4 a0 = *reinterpret_cast<const float4*>(as + k * PITCH + ty * 8);
      const float4 a1 = *reinterpret_cast<const float4*>(as + k * PITCH + ty * 8 + 4);
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(bs + k * PITCH + tx * 4);
      const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(bs + k * PITCH + 32 + tx * 4);
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const uint64_t b[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint64_t a2 = pair_f32(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma_f32x2(a2, b[j], acc[i][j]);
      }
    }
  }
  __syncthreads();
  float* part = sm + g * TILE * TILE;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float* dst = part + (ty * 8 + i) * TILE + tx * 4;
    *reinterpret_cast<ulonglong2*>(dst) = make_ulonglong2(acc[i][0], acc[i][1]);
    *reinterpret_cast<ulonglong2*>(dst + 32) = make_ulonglong2(acc[i][2], acc[i][3]);
  }
}

// columns c .. c + 3 of a finished row: the groups' partial sums in the order of K
__device__ __forceinline__ float4 tile_sum(const float* sm, int row, int c) {
  float4 s = *reinterpret_cast<const float4*>(sm + row * TILE + c);
#pragma unroll
  for (int g = 1; g < GROUPS; ++g) {
    const float4 v = *reinterpret_cast<const float4*>(sm + (g * TILE + row) * TILE + c);
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  return s;
}

// ------------------------------------------------------- sums in the order of K
// TM x 64 of A B^T per block: thread (ty, tx) owns TM / 16 rows x 4 columns, each sum one chain over K.  A step takes
// 32 columns of K through one of two buffers; a.load(k) / b.load(k) give elements k .. k + 3 of row threadIdx.x % TM
// resp. % 64 as they come from memory, a.value / b.value what is multiplied: the operands of two steps are in flight
// while one is multiplied.  Bound: 4,096 multiply-adds per column of K and 64 x 64 tile, 32 cycles of an SM (a step of
// 1,024 cycles); reached is what shared memory gives to registers, 128 bytes a cycle, twice that time at pieces of
// 4 x 4.  us, 1,536 columns, assignment to 256 bf16 centres, now and with one step in flight whose loads stood in
// branches on type and range (a branch's result is merged into a register, which waits for the load: no step
// overlapped its loads): 2,048 tokens 262 (316), 9,000 322 (399).
constexpr int STEP = 32;
template <int TM>
constexpr int ORDERED_FLOATS = 2 * STEP * (TM + TILE);

// NORMS: threads 0 .. TM - 1 / 128 .. 191 also square row threadIdx.x of A / threadIdx.x - 128 of B, elements
// j, j + 4, j + 8 ... in chain j.
template <int TM, bool NORMS, class LA, class LB>
__device__ __forceinline__ void gemm_ordered(float* sm, int K, const LA& operand_a, const LB& operand_b,
                                             float (&sums)[TM / 16][4], float (&norm)[4]) {
  constexpr int ROWS = TM / 16, NA = TM * STEP / 4 / THREADS, NB = TILE * STEP / 4 / THREADS;
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  const int ra = t % TM, ka = t / TM * 4, rb = t % TILE, kb = t / TILE * 4;   // first piece loaded; the others further along K
  uint64_t acc[ROWS][2];
#pragma unroll
  for (int i = 0; i < ROWS; ++i) acc[i][0] = acc[i][1] = 0ull;
  decltype(operand_a.load(0)) va[2][NA];
  decltype(operand_b.load(0)) vb[2][NB];
  auto fetch = [&](int buffer, int k0) {
#pragma unroll
    for (int i = 0; i < NA; ++i) va[buffer][i] = operand_a.load(k0 + ka + i * (STEP / NA));
#pragma unroll
    for (int i = 0; i < NB; ++i) vb[buffer][i] = operand_b.load(k0 + kb + i * (STEP / NB));
  };
  auto step = [&](int buffer, int k0) {
    float* as = sm + buffer * STEP * (TM + TILE);
    float* bs = as + STEP * TM;
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      const float4 f = operand_a.value(va[buffer][i]);
      const float v[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) as[(ka + i * (STEP / NA) + j) * TM + ra] = v[j];
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const float4 f = operand_b.value(vb[buffer][i]);
      const float v[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) bs[(kb + i * (STEP / NB) + j) * TILE + rb] = v[j];
    }
    __syncthreads();      // one per step: whoever fills this buffer next is behind the barrier of the step between
    if (k0 + 2 * STEP < K) fetch(buffer, k0 + 2 * STEP);
#pragma unroll
    for (int k = 0; k < STEP; ++k) {
      float a[ROWS];
      if constexpr (ROWS == 4) {
        const float4 v = *reinterpret_cast<const float4*>(as + k * TM + ty * 4);
        a[0] = v.x; a[1] = v.y; a[2] = v.z; a[3] = v.w;
      } else {
        const float2 v = *reinterpret_cast<const float2*>(as + k * TM + ty * 2);
        a[0] = v.x; a[1] = v.y;
      }
      const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(bs + k * TILE + tx * 4);
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        const uint64_t a2 = pair_f32(a[i], a[i]);
        acc[i][0] = fma_f32x2(a2, b.x, acc[i][0]);
        acc[i][1] = fma_f32x2(a2, b.y, acc[i][1]);
      }
    }
    if (NORMS && (t < TM || (t >= 128 && t < 128 + TILE))) {
      const float* row = t < TM ? as + t : bs + (t - 128);
      const int pitch = t < TM ? TM : TILE;
#pragma unroll
      for (int k = 0; k < STEP; ++k) norm[k & 3] = fmaf(row[k * pitch], row[k * pitch], norm[k & 3]);
    }
  };
  fetch(0, 0);
  if (STEP < K) fetch(1, STEP);
#pragma unroll 1
  for (int k0 = 0; k0 < K; k0 += 2 * STEP) {
    step(0, k0);
    if (k0 + STEP < K) step(1, k0 + STEP);
  }
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    split_f32(acc[i][0], sums[i][0], sums[i][1]);
    split_f32(acc[i][1], sums[i][2], sums[i][3]);
  }
}

// A row of either operand.  ANY: any type and alignment, rows past the last one zero.  F32 / BF16: rows that are read as
// vectors, K a multiple of STEP, and no condition on a load -- one merges two values, and the merge waits for the load.
// Their rows past the last one are another row's (what comes of them is stored nowhere).
enum Form { ANY = 0, F32_ROWS = 1, BF16_ROWS = 2 };
template <Form FORM>
struct RowOperand {
  const void* base; int dtype; size_t row; int K; bool vector, in;
  __device__ __forceinline__ float4 load(int k) const {
    return in ? load4(base, dtype, row, k, K, vector) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __device__ __forceinline__ float4 value(const float4& v) const { return v; }
};
template <>
struct RowOperand<F32_ROWS> {
  const void* base; int dtype; size_t row; int K; bool vector, in;
  __device__ __forceinline__ float4 load(int k) const {
    return __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(base) + row + k));
  }
  __device__ __forceinline__ float4 value(const float4& v) const { return v; }
};
template <>
struct RowOperand<BF16_ROWS> {
  const void* base; int dtype; size_t row; int K; bool vector, in;
  __device__ __forceinline__ uint2 load(int k) const {
    return __ldg(reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(base) + row + k));
  }
  __device__ __forceinline__ float4 value(const uint2& w) const {
    return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xFFFF0000u), __uint_as_float(w.y << 16),
                       __uint_as_float(w.y & 0xFFFF0000u));
  }
};

// whether rows can be read as `form`
bool has_form(Form form, const void* base, int dtype, int K) {
  return form == ANY || (dtype == (form == F32_ROWS ? NKV_F32 : NKV_BF16) && K % STEP == 0 && vector_rows(base, dtype, K));
}

// ---------------------------------------------------------------- assignment
template <int TM, Form X, Form C_>
__global__ void __launch_bounds__(THREADS, 2)
assign_kernel(const void* x, int x_dtype, bool x_vec, const void* centers, int c_dtype, bool c_vec, int S, int J, int C,
              void* ids, int id_bytes, int32_t* labels32) {
  __shared__ __align__(16) float sm[ORDERED_FLOATS<TM>];
  __shared__ float xn[TM], cn[TILE];
  constexpr int ROWS = TM / 16;
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  const int m0 = blockIdx.x * TM;
  const bool in_a = m0 + t % TM < S;
  const size_t a_row = static_cast<size_t>(in_a ? m0 + t % TM : 0) * J;
  float best[ROWS];
  int best_i[ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; ++i) { best[i] = INFINITY; best_i[i] = 0; }
  for (int n0 = 0; n0 < C; n0 += TILE) {
    const bool in_b = n0 + t % TILE < C;
    const size_t b_row = static_cast<size_t>(in_b ? n0 + t % TILE : 0) * J;
    float dots[ROWS][4], norm[4] = {0.f, 0.f, 0.f, 0.f};
    __syncthreads();        // the previous tile's operands and norms have been read
    gemm_ordered<TM, true>(sm, J, RowOperand<X>{x, x_dtype, a_row, J, x_vec, in_a},
                           RowOperand<C_>{centers, c_dtype, b_row, J, c_vec, in_b}, dots, norm);
    const float square = (norm[0] + norm[1]) + (norm[2] + norm[3]);
    if (t < TM) xn[t] = square;
    else if (t >= 128 && t < 128 + TILE) cn[t - 128] = square;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      float d = INFINITY;
      int idx = 0x7fffffff;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = n0 + tx * 4 + j;
        if (c < C) {
          // (||x||^2 + ||c||^2) - 2 x.c, in that association, in fp32
          const float dist = __fsub_rn(__fadd_rn(xn[ty * ROWS + i], cn[tx * 4 + j]), __fmul_rn(2.0f, dots[i][j]));
          if (dist < d) { d = dist; idx = c; }
        }
      }
#pragma unroll
      for (int off = 1; off < 16; off <<= 1) {
        const float od = __shfl_xor_sync(0xffffffffu, d, off);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, off);
        if (od < d || (od == d && oi < idx)) { d = od; idx = oi; }
      }
      if (d < best[i]) { best[i] = d; best_i[i] = idx; }
    }
  }
  if (tx != 0) return;
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const int token = m0 + ty * ROWS + i;
    if (token >= S) continue;
    if (ids) {
      if (id_bytes == 1) static_cast<uint8_t*>(ids)[token] = static_cast<uint8_t>(best_i[i]);
      else static_cast<uint16_t*>(ids)[token] = static_cast<uint16_t>(best_i[i]);
    }
    if (labels32) labels32[token] = best_i[i];
  }
}

// Few centres: block = 16 rows of x against all TN of them (16, 32 or 64 columns, C used), so that 2,048 rows are 128
// blocks, and no column of a 64-wide tile is multiplied for nothing.  64 columns of K per stage come by cp.async as they
// lie in memory, six stages in flight; the multiplying warps (8 rows x 16 centres each, a thread 2 x 2) read four columns
// of a row at a time, and the norms are other warps' work.  Sums in the order of K and norms in four chains, as in
// gemm_ordered: the same ids.  Bound: what shared memory gives to registers, 128 bytes a cycle (64 columns of K, 16 bf16
// centres: 448 cycles, about half of the step's time).  us, 1,536 columns, 16 / 32 / 64 bf16 centres, now (gemm_ordered):
// 2,048 rows 14 / 18 / 28 (56 / 60 / 67), 9,000 rows 29 / 45 / 85 (71 / 75 / 84), 40,000 rows 107 / 166 / 345
// (330 / 350 / 385).
constexpr int FEW_ROWS = 16, FEW_STEP = 64, FEW_STAGES = 6;

template <int TN, Form C_>
struct Few {
  static constexpr int MULTIPLY_WARPS = TN / 8, NORM_WARPS = 1 + (TN + 31) / 32;   // x, centres
  static constexpr int THREADS = (MULTIPLY_WARPS + NORM_WARPS) * 32;
  static constexpr int X_PITCH = FEW_STEP + 4;                                          // floats
  static constexpr int C_PITCH = C_ == BF16_ROWS ? FEW_STEP * 2 + 16 : FEW_STEP * 4 + 16;      // bytes
  static constexpr int X_BYTES = FEW_ROWS * X_PITCH * 4, STAGE = X_BYTES + TN * C_PITCH;
  static __device__ __forceinline__ float4 centre(const uint8_t* row, int k) {
    if constexpr (C_ == BF16_ROWS) return RowOperand<BF16_ROWS>{}.value(*reinterpret_cast<const uint2*>(row + k * 2));
    else return *reinterpret_cast<const float4*>(row + k * 4);
  }
};

__device__ __forceinline__ void copy_async(void* smem, const void* global) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem))),
               "l"(global) : "memory");
}

template <int TN, Form C_>
__global__ void __launch_bounds__(Few<TN, C_>::THREADS)
assign_few_kernel(const float* x, const void* centers, int S, int J, int C, void* ids, int id_bytes, int32_t* labels32) {
  using F = Few<TN, C_>;
  extern __shared__ __align__(16) uint8_t stages[];
  __shared__ float norms[FEW_ROWS + TN];
  __shared__ float row_d[TN / 16][FEW_ROWS];
  __shared__ int row_i[TN / 16][FEW_ROWS];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int m0 = blockIdx.x * FEW_ROWS, steps = J / FEW_STEP;
  constexpr int C_SIZE = C_ == BF16_ROWS ? 2 : 4, C_PIECES = FEW_STEP * C_SIZE / 16, PIECES = FEW_ROWS * 16 + TN * C_PIECES;
  constexpr int LOADERS = F::NORM_WARPS * 32, LOADS = (PIECES + LOADERS - 1) / LOADERS;
  const uint8_t* from[LOADS];            // the loader's pieces of 16 bytes, where they come from and go to
  int to[LOADS];
  const int loader = t - F::MULTIPLY_WARPS * 32;
#pragma unroll
  for (int l = 0; l < LOADS; ++l) {      // rows past the last: another one (of centres not one row for all of them)
    const int i = loader + l * LOADERS, j = i - FEW_ROWS * 16;
    if (i < FEW_ROWS * 16) {
      from[l] = reinterpret_cast<const uint8_t*>(x + static_cast<size_t>(min(m0 + (i >> 4), S - 1)) * J) + (i & 15) * 16;
      to[l] = (i >> 4) * F::X_PITCH * 4 + (i & 15) * 16;
    } else {
      from[l] = static_cast<const uint8_t*>(centers) + static_cast<size_t>(j / C_PIECES % C) * J * C_SIZE + j % C_PIECES * 16;
      to[l] = F::X_BYTES + j / C_PIECES * F::C_PITCH + j % C_PIECES * 16;
    }
  }
  auto request = [&](int step) {
    if (step < steps) {
      uint8_t* at = stages + step % FEW_STAGES * F::STAGE;
#pragma unroll
      for (int l = 0; l < LOADS; ++l) {
        const bool rows_of_x = l * LOADERS + LOADERS <= FEW_ROWS * 16 || loader + l * LOADERS < FEW_ROWS * 16;
        if (PIECES % LOADERS == 0 || loader + l * LOADERS < PIECES)
          copy_async(at + to[l], from[l] + step * (FEW_STEP * (rows_of_x ? 4 : C_SIZE)));
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");      // an empty one past the last step keeps the count
  };
  const bool multiplies = warp < F::MULTIPLY_WARPS;
  const int row = (warp & 1) * 8 + (lane >> 3) * 2, column = (warp >> 1) * 16 + (lane & 7);    // and row + 1, column + 8
  // squared: a row of x by the first of the other warps, a centre by the rest (two types in one warp would merge loads)
  const bool of_x = warp == F::MULTIPLY_WARPS;
  const int squared = of_x ? lane : loader - 32;
  const bool squares = !multiplies && squared < (of_x ? FEW_ROWS : TN);
  float dot[2][2] = {}, norm[4] = {0.f, 0.f, 0.f, 0.f};
  if (!multiplies)
    for (int step = 0; step < FEW_STAGES - 1; ++step) request(step);
  for (int step = 0; step < steps; ++step) {
    if (!multiplies) asm volatile("cp.async.wait_group %0;" ::"n"(FEW_STAGES - 2) : "memory");
    __syncthreads();                      // all copies of this step; the stage before it has been read
    if (!multiplies) request(step + FEW_STAGES - 1);
    const uint8_t* at = stages + step % FEW_STAGES * F::STAGE;
    const float* xs = reinterpret_cast<const float*>(at);
    const uint8_t* cs = at + F::X_BYTES;
    if (multiplies) {
#pragma unroll
      for (int k = 0; k < FEW_STEP; k += 4) {
        const float4 a[2] = {*reinterpret_cast<const float4*>(xs + row * F::X_PITCH + k),
                             *reinterpret_cast<const float4*>(xs + (row + 1) * F::X_PITCH + k)};
        const float4 b[2] = {F::centre(cs + column * F::C_PITCH, k), F::centre(cs + (column + 8) * F::C_PITCH, k)};
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            dot[i][j] = fmaf(a[i].x, b[j].x, dot[i][j]);
            dot[i][j] = fmaf(a[i].y, b[j].y, dot[i][j]);
            dot[i][j] = fmaf(a[i].z, b[j].z, dot[i][j]);
            dot[i][j] = fmaf(a[i].w, b[j].w, dot[i][j]);
          }
      }
    } else if (squares) {
      auto square = [&](const float4& v) {
        norm[0] = fmaf(v.x, v.x, norm[0]);
        norm[1] = fmaf(v.y, v.y, norm[1]);
        norm[2] = fmaf(v.z, v.z, norm[2]);
        norm[3] = fmaf(v.w, v.w, norm[3]);
      };
      if (of_x) {
#pragma unroll 8
        for (int k = 0; k < FEW_STEP; k += 4) square(*reinterpret_cast<const float4*>(xs + squared * F::X_PITCH + k));
      } else {
#pragma unroll 8
        for (int k = 0; k < FEW_STEP; k += 4) square(F::centre(cs + squared * F::C_PITCH, k));
      }
    }
  }
  if (squares) norms[(of_x ? 0 : FEW_ROWS) + squared] = (norm[0] + norm[1]) + (norm[2] + norm[3]);
  __syncthreads();
  if (multiplies) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float d = INFINITY;
      int idx = 0x7fffffff;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int c = column + j * 8;
        // (||x||^2 + ||c||^2) - 2 x.c, in that association, in fp32
        const float dist = __fsub_rn(__fadd_rn(norms[row + i], norms[FEW_ROWS + c]), __fmul_rn(2.0f, dot[i][j]));
        if (c < C && dist < d) { d = dist; idx = c; }
      }
#pragma unroll
      for (int off = 1; off < 8; off <<= 1) {
        const float od = __shfl_xor_sync(0xffffffffu, d, off);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, off);
        if (od < d || (od == d && oi < idx)) { d = od; idx = oi; }
      }
      if ((lane & 7) == 0) { row_d[warp >> 1][row + i] = d; row_i[warp >> 1][row + i] = idx; }
    }
  }
  __syncthreads();
  if (t >= FEW_ROWS || m0 + t >= S) return;
  float best = INFINITY;                  // no distance below it (NaN, infinities): centre 0
  int best_i = 0;
#pragma unroll
  for (int g = 0; g < TN / 16; ++g)
    if (row_d[g][t] < best) { best = row_d[g][t]; best_i = row_i[g][t]; }
  if (ids) {
    if (id_bytes == 1) static_cast<uint8_t*>(ids)[m0 + t] = static_cast<uint8_t>(best_i);
    else static_cast<uint16_t*>(ids)[m0 + t] = static_cast<uint16_t>(best_i);
  }
  if (labels32) labels32[m0 + t] = best_i;
}

// ---------------------------------------------------------------- projection
__device__ __forceinline__ float4 residual_of(const float4& x, const float4& c, const float4& m) {
  return make_float4(__fsub_rn(__fsub_rn(x.x, c.x), m.x), __fsub_rn(__fsub_rn(x.y, c.y), m.y),
                     __fsub_rn(__fsub_rn(x.z, c.z), m.z), __fsub_rn(__fsub_rn(x.w, c.w), m.w));
}

template <bool BF16>
struct Residual {      // (x - centre) - mean, rounded to bf16 where the operators are
  RowOperand<ANY> x, centre, mean;
  struct Raw { float4 x, centre, mean; };
  __device__ __forceinline__ Raw load(int k) const { return Raw{x.load(k), centre.load(k), mean.load(k)}; }
  __device__ __forceinline__ float4 value(const Raw& raw) const {
    float4 res = residual_of(raw.x, raw.centre, raw.mean);
    if (BF16) res = make_float4(round_to_bf16(res.x), round_to_bf16(res.y), round_to_bf16(res.z), round_to_bf16(res.w));
    return res;
  }
};

template <bool BF16, int TM>
__global__ void __launch_bounds__(THREADS, 2)
project_kernel(const void* x, int x_dtype, bool x_vec, const uint16_t* centers, bool c_vec, const void* ids, int id_bytes,
               const float* mean, const void* encoder, bool e_vec, int S, int J, int r, void* coeff) {
  __shared__ __align__(16) float sm[ORDERED_FLOATS<TM>];
  constexpr int ROWS = TM / 16;
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  const int m0 = blockIdx.x * TM, n0 = blockIdx.y * TILE;
  const bool in_a = m0 + t % TM < S, in_b = n0 + t % TILE < r;
  const size_t a_row = static_cast<size_t>(in_a ? m0 + t % TM : 0) * J, b_row = static_cast<size_t>(in_b ? n0 + t % TILE : 0) * J;
  const size_t c_row = static_cast<size_t>(in_a ? load_id(ids, id_bytes, m0 + t % TM) : 0) * J;
  const Residual<BF16> residual{{x, x_dtype, a_row, J, x_vec, in_a}, {centers, NKV_BF16, c_row, J, c_vec, in_a},
                                {mean, NKV_F32, 0, J, e_vec, in_a}};
  float sums[ROWS][4], unused[4];
  gemm_ordered<TM, false>(sm, J, residual, RowOperand<ANY>{encoder, BF16 ? NKV_BF16 : NKV_F32, b_row, J, e_vec, in_b}, sums, unused);
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const int token = m0 + ty * ROWS + i;
    if (token >= S) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = n0 + tx * 4 + j;
      if (c < r) store_float(coeff, BF16 ? NKV_BF16 : NKV_F32, static_cast<size_t>(token) * r + c, sums[i][j]);
    }
  }
}

// fp32 rows, operators and mean as vectors: block = TM rows x 64 columns of the encoder, thread = TM / 8 x 4 sums, each one
// chain in the order of K as above.  Bound: what shared memory gives to registers, 128 bytes a cycle -- (TM / 8 + 4) * 4
// cycles per column of K, where gemm_ordered's 4 x 4 pieces take 64 for 64 rows -- and the lines that loads touch: eight
// threads read a line of a row of x here, one row per thread there.  Operand tiles lie as in memory, 32 columns of K and
// four words of padding a row, which the reads of eight rows need; a thread takes four columns of K at a time.  The
// encoder's come by cp.async, three steps ahead; x, centre and mean wait in registers, two steps ahead.  us, 1,536
// columns to 192, now (gemm_ordered): 300 tokens 25 (67), 2,048 44 (83), 4,096 77 (162), 20,000 300 (551).
constexpr int ROW_THREADS = 128, ROW_PITCH = STEP + 4, ROW_STAGES = 4;
template <int TM>
constexpr int ROW_SMEM = (ROW_STAGES * TILE + 2 * TM) * ROW_PITCH * 4;

template <int TM>
__global__ void __launch_bounds__(ROW_THREADS, 2)
project_rows_kernel(const float* x, const uint16_t* centers, const void* ids, int id_bytes, const float* mean,
                    const float* encoder, int S, int J, int r, float* coeff) {
  extern __shared__ float sm[];
  constexpr int PIECES = TM / 16, ROWS = TM / 8;
  const int t = threadIdx.x, m0 = blockIdx.x * TM, n0 = blockIdx.y * TILE, steps = J / STEP;
  const int piece = (t & 7) * 4, first = t >> 3;         // loads: columns piece .. + 3 of rows first, first + 16 ...
  const float* x_at[PIECES];
  const uint16_t* c_at[PIECES];
  const float* e_at[TILE / 16];
#pragma unroll
  for (int p = 0; p < PIECES; ++p) {                      // rows past the last: another one's, stored nowhere
    const int token = min(m0 + first + p * 16, S - 1);
    x_at[p] = x + static_cast<size_t>(token) * J + piece;
    c_at[p] = centers + static_cast<size_t>(load_id(ids, id_bytes, token)) * J + piece;
  }
#pragma unroll
  for (int p = 0; p < TILE / 16; ++p) {
    const int row = n0 + first + p * 16;
    e_at[p] = encoder + static_cast<size_t>(row < r ? row : row % r) * J + piece;
  }
  float4 xv[2][PIECES], mv[2];
  uint2 cv[2][PIECES];
  auto fetch = [&](int buffer, int step) {
    mv[buffer] = __ldg(reinterpret_cast<const float4*>(mean + step * STEP + piece));
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      xv[buffer][p] = __ldg(reinterpret_cast<const float4*>(x_at[p] + step * STEP));
      cv[buffer][p] = __ldg(reinterpret_cast<const uint2*>(c_at[p] + step * STEP));
    }
  };
  auto request = [&](int step) {
    if (step < steps) {
      float* at = sm + step % ROW_STAGES * TILE * ROW_PITCH + first * ROW_PITCH + piece;
#pragma unroll
      for (int p = 0; p < TILE / 16; ++p) copy_async(at + p * 16 * ROW_PITCH, e_at[p] + step * STEP);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");      // an empty one past the last step keeps the count
  };
  const int tx = t & 15, ty = t >> 4;                     // sums: rows ty + 8 i, columns tx + 16 j
  float sums[ROWS][4] = {};
  auto step = [&](int buffer, int s) {
    float* as = sm + (ROW_STAGES * TILE + buffer * TM) * ROW_PITCH;
    const float* bs = sm + s % ROW_STAGES * TILE * ROW_PITCH;
#pragma unroll
    for (int p = 0; p < PIECES; ++p)
      *reinterpret_cast<float4*>(as + (first + p * 16) * ROW_PITCH + piece) =
          residual_of(xv[buffer][p], RowOperand<BF16_ROWS>{}.value(cv[buffer][p]), mv[buffer]);
    asm volatile("cp.async.wait_group %0;" ::"n"(ROW_STAGES - 2) : "memory");
    __syncthreads();        // this step's tiles; what they lie on next time has been read behind the barrier before
    if (s + 2 < steps) fetch(buffer, s + 2);
    request(s + ROW_STAGES - 1);
#pragma unroll
    for (int k = 0; k < STEP; k += 4) {
      float4 a[ROWS], b[4];
#pragma unroll
      for (int i = 0; i < ROWS; ++i) a[i] = *reinterpret_cast<const float4*>(as + (ty + i * 8) * ROW_PITCH + k);
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(bs + (tx + j * 16) * ROW_PITCH + k);
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          sums[i][j] = fmaf(a[i].x, b[j].x, sums[i][j]);
          sums[i][j] = fmaf(a[i].y, b[j].y, sums[i][j]);
          sums[i][j] = fmaf(a[i].z, b[j].z, sums[i][j]);
          sums[i][j] = fmaf(a[i].w, b[j].w, sums[i][j]);
        }
    }
  };
  fetch(0, 0);
  if (1 < steps) fetch(1, 1);
  for (int s = 0; s < ROW_STAGES - 1; ++s) request(s);
#pragma unroll 1
  for (int s = 0; s < steps; s += 2) {
    step(0, s);
    if (s + 1 < steps) step(1, s + 1);
  }
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const int token = m0 + ty + i * 8;
    if (token >= S) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = n0 + tx + j * 16;
      if (c < r) coeff[static_cast<size_t>(token) * r + c] = sums[i][j];
    }
  }
}

// -------------------------------------------------------------------- decode
// Operands of gemm64: codes x scales of 64 tokens, 64 decoder rows.
struct DecodeSource {
  const nkv_history& h; int token; const void* decoder; int j0, J; bool d_vec;   // token: of row t, -1 for none
};

template <bool BF16>
struct AnyDecode {          // any type, group and alignment: thread t takes row t of either operand
  const DecodeSource& src;
  float4 a[4], b[4];
  __device__ __forceinline__ float4 latent(int k) const {
    const nkv_history& h = src.h;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (src.token >= 0 && h.group % 4 == 0 && k < h.rank) {      // four coefficients share a scale and two whole bytes
      const uint8_t* code = h.codes + static_cast<size_t>(src.token) * (h.rank >> 1) + (k >> 1);
      const int b0 = __ldg(code), b1 = __ldg(code + 1);
      const float scale = load_float(h.scales, h.scale_dtype,
                                     static_cast<size_t>(src.token) * (h.rank / h.group) + (h.group == h.rank ? 0 : k / h.group));
      v[0] = static_cast<float>((b0 & 15) - 7) * scale;
      v[1] = static_cast<float>((b0 >> 4) - 7) * scale;
      v[2] = static_cast<float>((b1 & 15) - 7) * scale;
      v[3] = static_cast<float>((b1 >> 4) - 7) * scale;
    } else if (src.token >= 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (k + i < h.rank) v[i] = latent_value(h, src.token, k + i);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (BF16) v[i] = round_to_bf16(v[i]);
    return make_float4(v[0], v[1], v[2], v[3]);
  }
  __device__ __forceinline__ void fetch(int c) {
    const int row = src.j0 + threadIdx.x % GROUP_THREADS, K = src.h.rank;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      a[j] = latent(c * BK + 4 * j);
      b[j] = row < src.J ? load4(src.decoder, BF16 ? NKV_BF16 : NKV_F32, static_cast<size_t>(row) * K, c * BK + 4 * j, K, src.d_vec)
                         : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  __device__ __forceinline__ void stage(float* as, float* bs) const {
    const int t = threadIdx.x % GROUP_THREADS;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float av[4] = {a[j].x, a[j].y, a[j].z, a[j].w}, bv[4] = {b[j].x, b[j].y, b[j].z, b[j].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        as[(4 * j + i) * PITCH + t] = av[i];
        bs[(4 * j + i) * PITCH + t] = bv[i];
      }
    }
  }
};

// fp32 decoder rows read as vectors, BK dividing rank and group, the codes of a chunk as one word of 8 bytes: thread t
// takes the codes and the scale of row t; of the decoder two threads take 32 bytes of a row, which PITCH puts into
// different banks.  No load has a condition on it, so a chunk's are in flight while the one before is multiplied.
// Bound: multiply-adds, 128 a cycle and SM, of which 45 to 58% is reached; AnyDecode is bound by its loads, each of
// which touches a line per lane.  us of a decode, VectorDecode / AnyDecode, x 1,536 columns of rank 192: 300 tokens
// 8.7 / 14.1, 2,048 37.6 / 64.0; x 3,072 columns of rank 384: 4,096 229 / 404.
struct VectorDecode {
  const uint2* codes; const uint16_t* scales; const float* rows; int K, group; bool one, f16;
  long long half;         // elements to the decoder row 32 further on
  uint2 a; uint16_t scale; float4 b[4];
  __device__ __forceinline__ explicit VectorDecode(const DecodeSource& src) {
    const int t = threadIdx.x % GROUP_THREADS, row = src.j0 + (t >> 1);     // rows and tokens past the last: the first
    const size_t token = src.token < 0 ? 0 : src.token;
    K = src.h.rank;
    group = src.h.group;
    one = group == K;
    f16 = src.h.scale_dtype == NKV_F16;
    codes = reinterpret_cast<const uint2*>(src.h.codes + token * (K >> 1));
    scales = static_cast<const uint16_t*>(src.h.scales) + token * (one ? 1 : K / group);
    const long long low = row < src.J ? row : 0, high = row + 32 < src.J ? row + 32 : 0;
    rows = static_cast<const float*>(src.decoder) + low * K + (t & 1) * 4;
    half = (high - low) * K;
  }
  __device__ __forceinline__ void fetch(int c) {
    a = __ldg(codes + c);
    scale = __ldg(scales + (one ? 0 : c * BK / group));
#pragma unroll
    for (int j = 0; j < 4; ++j)
      b[j] = __ldg(reinterpret_cast<const float4*>(rows + (c * BK + (j & 1) * 8 + (j >> 1) * half)));
  }
  __device__ __forceinline__ void stage(float* as, float* bs) const {
    const int t = threadIdx.x % GROUP_THREADS;
    const float s = f16 ? __half2float(__ushort_as_half(scale)) : bf16_bits_to_float(scale);
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      const int code = (k < 8 ? a.x : a.y) >> (4 * (k & 7)) & 15;
      as[k * PITCH + t] = static_cast<float>(code - 7) * s;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float v[4] = {b[j].x, b[j].y, b[j].z, b[j].w};
      const int row = (t >> 1) + (j >> 1) * 32, k = (j & 1) * 8 + (t & 1) * 4;
#pragma unroll
      for (int i = 0; i < 4; ++i) bs[(k + i) * PITCH + row] = v[i];
    }
  }
};

// decoder rows, bias and centre columns of `J` columns; out has rows of out_stride elements.  VECTOR: operands as
// VectorDecode takes them; mean, centres and out in pieces of four columns.
template <bool BF16, bool VECTOR>
__global__ void __launch_bounds__(THREADS, 2)
decode_rows_kernel(nkv_history h, const int32_t* rows_index, int n, const void* decoder, bool d_vec,
                   const float* mean, int J, void* out, int out_dtype, long long out_stride) {
  static_assert(!(BF16 && VECTOR), "the bf16 operators' decode of aligned rows is on the tensor cores");
  extern __shared__ float sm[];
  __shared__ int tok[TILE], crow[TILE];
  const int t = threadIdx.x % GROUP_THREADS;
  const int m0 = blockIdx.x * TILE, n0 = blockIdx.y * TILE;
  int token = -1;
  if (m0 + t < n) {
    token = rows_index ? rows_index[m0 + t] : m0 + t;
    if (token < 0 || token >= h.tokens) token = -1;
  }
  if (threadIdx.x < TILE) {
    tok[t] = token;
    crow[t] = token < 0 ? 0 : center_row_of(h, token);
  }
  const DecodeSource source{h, token, decoder, n0, J, d_vec};
  if constexpr (VECTOR) {
    VectorDecode operands(source);
    gemm64(sm, h.rank, operands);
  } else {
    AnyDecode<BF16> operands{source};
    gemm64(sm, h.rank, operands);
  }
  const uint16_t* centers = static_cast<const uint16_t*>(h.centers);
  constexpr int PASSES = TILE * TILE / 4 / THREADS;
  const int row0 = threadIdx.x >> 4, c0 = (threadIdx.x & 15) * 4;       // rows row0, row0 + 16 ...
  if constexpr (VECTOR) {
    const int col = n0 + c0 < J ? n0 + c0 : 0;
    uint2 centre[PASSES];
    const float4 m = __ldg(reinterpret_cast<const float4*>(mean + col));
    // tok and crow are another thread's: the barrier that gemm64 has in front of its partial sums lies between
#pragma unroll
    for (int i = 0; i < PASSES; ++i)
      centre[i] = __ldg(reinterpret_cast<const uint2*>(centers + static_cast<size_t>(crow[row0 + i * 16]) * h.center_width + col));
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PASSES; ++i) {
      const int row = row0 + i * 16;
      if (m0 + row >= n || tok[row] < 0 || n0 + c0 >= J) continue;
      const float4 s = tile_sum(sm, row, c0);
      const uint2 c = centre[i];
      *reinterpret_cast<float4*>(static_cast<float*>(out) + static_cast<size_t>(m0 + row) * out_stride + n0 + c0) =
          make_float4(__fadd_rn(__fadd_rn(s.x, m.x), __uint_as_float(c.x << 16)),
                      __fadd_rn(__fadd_rn(s.y, m.y), __uint_as_float(c.x & 0xFFFF0000u)),
                      __fadd_rn(__fadd_rn(s.z, m.z), __uint_as_float(c.y << 16)),
                      __fadd_rn(__fadd_rn(s.w, m.w), __uint_as_float(c.y & 0xFFFF0000u)));
    }
  } else {
    __syncthreads();
#pragma unroll 1
    for (int row = row0; row < TILE; row += 16) {
      if (m0 + row >= n || tok[row] < 0) continue;
      const float4 s = tile_sum(sm, row, c0);
      const float sums[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = n0 + c0 + i;
        if (c >= J) continue;
        const float center = bf16_bits_to_float(centers[static_cast<size_t>(crow[row]) * h.center_width + c]);
        float v;
        if (BF16) {
          v = round_to_bf16(__fadd_rn(sums[i], round_to_bf16(mean[c])));
          v = round_to_bf16(__fadd_rn(v, center));
        } else {
          v = __fadd_rn(__fadd_rn(sums[i], mean[c]), center);
        }
        store_float(out, out_dtype, static_cast<size_t>(m0 + row) * out_stride + c, v);
      }
    }
  }
}

// ----------------------------------------------------------------- attention
// Block = 64 queries of one head over one run of history tokens, 64 at a time: K and V tiles in shared
// memory, online softmax in fp32, two blocks per SM.  A thread owns 8 x 4 scores and 8 queries x D / 16
// columns of O.  K of the next tile arrives while the weights meet V, and V while the scores are made.
// Bound: what shared memory gives to registers, 128 bytes a cycle: 48 cycles per column of K and 64 (heads of 64: 48) per
// token of V, against 32 and 64 (32) of multiply-adds; pieces of 4 x 4 took 64 and 96.  us of a read with rank 32, now /
// with 4 x 4: 2,048 tokens, 12 heads of 128 and 256 queries 127 / 146, 4,096 tokens and 512 queries 382 / 452; heads of
// 64, 2,048 tokens and 256 queries 76 / 85.
struct RowAttn {
  const float* q; const float* k; const float* v;
  long long q_stride_token, q_stride_head, kv_stride_token, kv_stride_head;
  int Q, heads, N, tokens_per_split, out_heads;
  float scale;
  float* out; float* lse;      // partial z at z * Q * out_heads rows
};

constexpr int ATTN_THREADS = 128;

template <int D>
__global__ void __launch_bounds__(ATTN_THREADS, 2)
attn_rows_f32_kernel(RowAttn a) {
  extern __shared__ __align__(16) float smem[];
  float* Qs = smem;                  // [64][D], as in memory but for the order of a row's pieces of four
  float* Ks = Qs + 64 * D;           // [64][D], the same
  float* Vs = Ks + 64 * D;           // [64][D]
  float* Ps = Vs + 64 * D;           // [64 tokens][64 queries], pieces of four queries in another order too
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;       // queries ty * 8 .. + 7, tokens tx * 4 .. + 3
  const int q0 = blockIdx.x * 64, head = blockIdx.y, z = blockIdx.z;
  const int t_begin = z * a.tokens_per_split, t_end = min(a.N, t_begin + a.tokens_per_split);
  // piece p of row r lies at p ^ (r / 4 % 8): eight threads read one piece of rows four apart from different banks
  auto copy_tile = [&](float* tile, const float* base, long long stride, int row0, int rows, bool permuted) {
#pragma unroll
    for (int n = 0; n < 64 * (D / 4) / ATTN_THREADS; ++n) {
      const int idx = tid + n * ATTN_THREADS, i = idx / (D / 4), piece = idx % (D / 4);
      const int row = min(row0 + i, rows - 1), bytes = row0 + i < rows ? 16 : 0;      // past the last: zeros
      const float* at = tile + i * D + (permuted ? piece ^ (i >> 2 & 7) : piece) * 4;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(at))),
                   "l"(base + static_cast<size_t>(row) * stride + piece * 4), "r"(bytes) : "memory");
    }
  };
  auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
  const float* k_head = a.k + static_cast<size_t>(head) * a.kv_stride_head;
  const float* v_head = a.v + static_cast<size_t>(head) * a.kv_stride_head;
  copy_tile(Qs, a.q + static_cast<size_t>(head) * a.q_stride_head, a.q_stride_token, q0, a.Q, true);
  copy_tile(Ks, k_head, a.kv_stride_token, t_begin, t_end, true);
  commit();
  constexpr int OC = D / 64;         // pieces of four O columns per thread: c * 64 + tx * 4
  float o[8][OC][4] = {};
  float m_run[8], l_run[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    m_run[i] = -INFINITY;
    l_run[i] = 0.f;
  }
#pragma unroll 1
  for (int t0 = t_begin; t0 < t_end; t0 += 64) {
    copy_tile(Vs, v_head, a.kv_stride_token, t0, t_end, false);
    commit();
    asm volatile("cp.async.wait_group 1;" ::: "memory");        // K, and Q
    __syncthreads();
    float s[8][4] = {};
#pragma unroll 4
    for (int piece = 0; piece < D / 4; ++piece) {
      float4 q[8], k[4];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        q[i] = *reinterpret_cast<const float4*>(Qs + (ty * 8 + i) * D + (piece ^ ((ty * 2 + i / 4) & 7)) * 4);
#pragma unroll
      for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const float4*>(Ks + (tx * 4 + j) * D + (piece ^ (tx & 7)) * 4);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s[i][j] = fmaf(q[i].x, k[j].x, s[i][j]);
          s[i][j] = fmaf(q[i].y, k[j].y, s[i][j]);
          s[i][j] = fmaf(q[i].z, k[j].z, s[i][j]);
          s[i][j] = fmaf(q[i].w, k[j].w, s[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = t0 + tx * 4 + j < t_end ? s[i][j] * a.scale : -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int off = 8; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      const float m_new = fmaxf(m_run[i], mx);   // finite: every processed tile has a valid token
      const float alpha = expf(m_run[i] - m_new);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = expf(s[i][j] - m_new);
        sum += s[i][j];
      }
#pragma unroll
      for (int off = 8; off >= 1; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
      l_run[i] = l_run[i] * alpha + sum;
      m_run[i] = m_new;
#pragma unroll
      for (int c = 0; c < OC; ++c)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][c][e] = fmaf(o[i][c][e], alpha, 0.f);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int half = 0; half < 2; ++half)
        *reinterpret_cast<float4*>(Ps + (tx * 4 + j) * 64 + ((ty * 2 + half) ^ (tx & 7)) * 4) =
            make_float4(s[half * 4][j], s[half * 4 + 1][j], s[half * 4 + 2][j], s[half * 4 + 3][j]);
    asm volatile("cp.async.wait_group 0;" ::: "memory");        // V
    __syncthreads();                 // and everyone has read K
    if (t0 + 64 < t_end) copy_tile(Ks, k_head, a.kv_stride_token, t0 + 64, t_end, true);
    commit();
#pragma unroll 4
    for (int t = 0; t < 64; ++t) {
      const float4 p0 = *reinterpret_cast<const float4*>(Ps + t * 64 + ((ty * 2) ^ (t >> 2 & 7)) * 4);
      const float4 p1 = *reinterpret_cast<const float4*>(Ps + t * 64 + ((ty * 2 + 1) ^ (t >> 2 & 7)) * 4);
      const float p[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
#pragma unroll
      for (int c = 0; c < OC; ++c) {
        const float4 v = *reinterpret_cast<const float4*>(Vs + t * D + c * 64 + tx * 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          o[i][c][0] = fmaf(p[i], v.x, o[i][c][0]);
          o[i][c][1] = fmaf(p[i], v.y, o[i][c][1]);
          o[i][c][2] = fmaf(p[i], v.z, o[i][c][2]);
          o[i][c][3] = fmaf(p[i], v.w, o[i][c][3]);
        }
      }
    }
    __syncthreads();                 // V and the weights have been read
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int qi = q0 + ty * 8 + i;
    if (qi >= a.Q) continue;
    const float inv = l_run[i] > 0.f ? 1.0f / l_run[i] : 0.f;
    const size_t row = (static_cast<size_t>(z) * a.Q + qi) * a.out_heads + head;
#pragma unroll
    for (int c = 0; c < OC; ++c)
      *reinterpret_cast<float4*>(a.out + row * D + c * 64 + tx * 4) =
          make_float4(o[i][c][0] * inv, o[i][c][1] * inv, o[i][c][2] * inv, o[i][c][3] * inv);
    if (tx == 0) a.lse[row] = l_run[i] > 0.f ? m_run[i] + logf(l_run[i]) : -INFINITY;
  }
}

// Merge of the history splits: thread = (row, 4 columns).  Weights against the largest LSE, one logarithm: the
// pairwise fold of lse_merge rounds the LSE once per part (3,102 tokens in 16 parts: 4.9e-7 rms from float64,
// where one part has 3.2e-7).
__global__ void __launch_bounds__(256)
merge_splits_kernel(const float* part_out, const float* part_lse, int splits, long long rows, int d, float* out,
                    float* lse_out) {
  const int per_row = d / 4;
  const long long idx = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
  if (idx >= rows * per_row) return;
  const long long row = idx / per_row;
  const int col = static_cast<int>(idx - row * per_row) * 4;
  float top = -INFINITY;
  bool nan = false;
  for (int z = 0; z < splits; ++z) {
    const float l = part_lse[z * rows + row];
    nan = nan || l != l;
    top = fmaxf(top, l);
  }
  const float origin = isfinite(top) ? top : 0.f;   // all of them -inf: weights of zero
  float acc[4] = {0.f, 0.f, 0.f, 0.f}, weight = 0.f;
  for (int z = 0; z < splits; ++z) {
    const float w = expf(part_lse[z * rows + row] - origin);
    const float4 v = *reinterpret_cast<const float4*>(part_out + (z * rows + row) * d + col);
    weight += w;
    acc[0] = fmaf(w, v.x, acc[0]); acc[1] = fmaf(w, v.y, acc[1]);
    acc[2] = fmaf(w, v.z, acc[2]); acc[3] = fmaf(w, v.w, acc[3]);
  }
  const float inv = weight == 0.f ? 1.f : 1.0f / weight;
  *reinterpret_cast<float4*>(out + row * d + col) = make_float4(acc[0] * inv, acc[1] * inv, acc[2] * inv, acc[3] * inv);
  if (col == 0) lse_out[row] = nan ? __int_as_float(0x7fc00000) : origin + logf(weight);
}

template <class K>
int allow_smem(K kernel) {
  NKV_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_FLOATS * 4));
  return NKV_OK;
}

}  // namespace

// Rows of a tile in gemm_ordered: 32 while that still gives every block an SM of its own, else 64.  A tile of
// half the rows takes four fifths of the time (K = 1,536: 66 against 82 us), so two on one SM would lose.
static int ordered_rows(int S, int column_tiles) {
  return static_cast<long long>(ceil_div(S, 32)) * column_tiles <= sm_count() ? 32 : 64;
}

template <int TN>
static int assign_few(const float* x, const void* centers, int c_dtype, int S, int J, int C, void* ids, int id_bytes,
                      int32_t* labels32, cudaStream_t stream) {
  const bool bf16 = c_dtype == NKV_BF16;
  auto kernel = bf16 ? assign_few_kernel<TN, BF16_ROWS> : assign_few_kernel<TN, F32_ROWS>;
  const int smem = FEW_STAGES * (bf16 ? Few<TN, BF16_ROWS>::STAGE : Few<TN, F32_ROWS>::STAGE);
  NKV_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  kernel<<<ceil_div(S, FEW_ROWS), Few<TN, BF16_ROWS>::THREADS, smem, stream>>>(x, centers, S, J, C, ids, id_bytes, labels32);
  NKV_LAUNCH_CHECK("assign_few_kernel");
  return NKV_OK;
}

int simt_assign(const void* x, int x_dtype, const void* centers, int c_dtype, int S, int J,
                int C, void* ids, int id_bytes, int32_t* labels32, cudaStream_t stream) {
  if (S == 0) return NKV_OK;
  const bool x_rows = has_form(F32_ROWS, x, x_dtype, J);
  // 33 to 64 centres in fp32 are twice the bytes of bf16 through shared memory: beyond two blocks per SM gemm_ordered's
  // tile, whose values are reused more, is ahead (4,096 rows 65 / 69 us, 9,000 rows 129 / 84)
  const bool few = C >= 1 && (C <= 32 || (C <= 64 && (c_dtype == NKV_BF16 || ceil_div(S, FEW_ROWS) <= 2 * sm_count())));
  if (few && x_rows && J % FEW_STEP == 0 && (reinterpret_cast<uintptr_t>(centers) & 15) == 0) {
    const float* rows = static_cast<const float*>(x);
    return C <= 16   ? assign_few<16>(rows, centers, c_dtype, S, J, C, ids, id_bytes, labels32, stream)
           : C <= 32 ? assign_few<32>(rows, centers, c_dtype, S, J, C, ids, id_bytes, labels32, stream)
                     : assign_few<64>(rows, centers, c_dtype, S, J, C, ids, id_bytes, labels32, stream);
  }
  const int rows = ordered_rows(S, 1);
  auto kernel = x_rows && has_form(BF16_ROWS, centers, c_dtype, J)
                    ? (rows == 32 ? assign_kernel<32, F32_ROWS, BF16_ROWS> : assign_kernel<64, F32_ROWS, BF16_ROWS>)
                : x_rows && has_form(F32_ROWS, centers, c_dtype, J)
                    ? (rows == 32 ? assign_kernel<32, F32_ROWS, F32_ROWS> : assign_kernel<64, F32_ROWS, F32_ROWS>)
                    : (rows == 32 ? assign_kernel<32, ANY, ANY> : assign_kernel<64, ANY, ANY>);
  kernel<<<ceil_div(S, rows), THREADS, 0, stream>>>(
      x, x_dtype, vector_rows(x, x_dtype, J), centers, c_dtype, vector_rows(centers, c_dtype, J), S, J, C, ids,
      id_bytes, labels32);
  NKV_LAUNCH_CHECK("assign_kernel");
  return NKV_OK;
}

template <int TM>
static int project_rows(const float* x, const uint16_t* centers, const void* ids, int id_bytes, const float* mean,
                        const float* encoder, int S, int J, int r, float* coeff, cudaStream_t stream) {
  NKV_CUDA(cudaFuncSetAttribute(project_rows_kernel<TM>, cudaFuncAttributeMaxDynamicSharedMemorySize, ROW_SMEM<TM>));
  project_rows_kernel<TM><<<dim3(ceil_div(S, TM), ceil_div(r, TILE)), ROW_THREADS, ROW_SMEM<TM>, stream>>>(
      x, centers, ids, id_bytes, mean, encoder, S, J, r, coeff);
  NKV_LAUNCH_CHECK("project_rows_kernel");
  return NKV_OK;
}

// Rows of a tile of project_rows_kernel: the least blocks on the fullest SM times what one takes (TM / 8 + 4 reads of
// shared memory; one block alone, K = 1,536: 16 rows 25 us, 32 rows 34, 48 rows 44); of equal ones the largest, which
// reads the encoder least often.  64 rows take 220 registers and 91 us, more than two blocks of 48 (77).
static int project_tile(int S, int r) {
  int best = 48;
  long long least = 0;
  for (int rows = 48; rows >= 16; rows -= 16) {
    const long long blocks = static_cast<long long>(ceil_div(S, rows)) * ceil_div(r, TILE);
    const long long cost = (blocks + sm_count() - 1) / sm_count() * (rows / 8 + 4);
    if (rows == 48 || cost < least) { best = rows; least = cost; }
  }
  return best;
}

int simt_project(const void* x, int x_dtype, const void* centers_bf16, const void* ids,
                 int id_bytes, const float* mean, const void* encoder, int enc_dtype, int S,
                 int J, int r, void* coeff, cudaStream_t stream) {
  if (S == 0) return NKV_OK;
  if (has_form(F32_ROWS, x, x_dtype, J) && has_form(BF16_ROWS, centers_bf16, NKV_BF16, J) &&
      has_form(F32_ROWS, encoder, enc_dtype, J) && has_form(F32_ROWS, mean, NKV_F32, J)) {
    const int tile = project_tile(S, r);
    auto run = tile == 16 ? project_rows<16> : tile == 32 ? project_rows<32> : project_rows<48>;
    return run(static_cast<const float*>(x), static_cast<const uint16_t*>(centers_bf16), ids, id_bytes, mean,
               static_cast<const float*>(encoder), S, J, r, static_cast<float*>(coeff), stream);
  }
  const int rows = ordered_rows(S, ceil_div(r, TILE));
  const dim3 grid(ceil_div(S, rows), ceil_div(r, TILE));
  const bool e_vec = vector_rows(encoder, enc_dtype, J) && vector_rows(mean, NKV_F32, J);
  auto kernel = enc_dtype == NKV_BF16 ? (rows == 32 ? project_kernel<true, 32> : project_kernel<true, 64>)
                                      : (rows == 32 ? project_kernel<false, 32> : project_kernel<false, 64>);
  kernel<<<grid, THREADS, 0, stream>>>(
      x, x_dtype, vector_rows(x, x_dtype, J), static_cast<const uint16_t*>(centers_bf16),
      vector_rows(centers_bf16, NKV_BF16, J), ids, id_bytes, mean, encoder, e_vec, S, J, r, coeff);
  NKV_LAUNCH_CHECK("project_kernel");
  return NKV_OK;
}

int simt_decode_rows(const nkv_history& hist, const int32_t* rows_index, int n,
                     const void* decoder, int dec_dtype, const float* mean, int J, void* out,
                     int out_dtype, int64_t out_stride, cudaStream_t stream) {
  if (n == 0) return NKV_OK;
  const dim3 grid(ceil_div(n, TILE), ceil_div(J, TILE));
  const auto aligned = [](const void* at, int bytes) { return reinterpret_cast<uintptr_t>(at) % bytes == 0; };
  const bool vector = dec_dtype == NKV_F32 && out_dtype == NKV_F32 && hist.tokens > 0 && hist.rank % BK == 0 &&
                      hist.group % BK == 0 && J % 4 == 0 && out_stride % 4 == 0 && hist.center_width % 4 == 0 &&
                      aligned(decoder, 16) && aligned(mean, 16) && aligned(out, 16) && aligned(hist.codes, 8) &&
                      aligned(hist.scales, 2) && aligned(hist.centers, 8);
  auto kernel = dec_dtype == NKV_BF16 ? decode_rows_kernel<true, false>
                : vector ? decode_rows_kernel<false, true> : decode_rows_kernel<false, false>;
  int rc = allow_smem(kernel);
  if (rc != NKV_OK) return rc;
  kernel<<<grid, THREADS, SMEM_FLOATS * 4, stream>>>(hist, rows_index, n, decoder,
                                                     vector_rows(decoder, dec_dtype, hist.rank), mean, J, out, out_dtype,
                                                     out_stride);
  NKV_LAUNCH_CHECK("decode_rows_kernel");
  return NKV_OK;
}

// ---- the fp32 read: rows of a batch of heads rebuilt into scratch, then attended over history splits ----
namespace {

struct F32Plan { int batch_heads, splits, tokens_per_split; };

constexpr size_t ROW_BATCH_BYTES = 512u << 20;

// Splits: about two blocks per SM, at least two 64-token tiles each.
F32Plan plan_f32(int Q, int heads, int d, int tokens, bool rebuild) {
  F32Plan plan{};
  const size_t head_bytes = static_cast<size_t>(tokens) * d * 8;
  int batches = 1;
  while (rebuild && batches < heads && head_bytes * ceil_div(heads, batches) > ROW_BATCH_BYTES) ++batches;
  plan.batch_heads = ceil_div(heads, batches);
  const int tiles = ceil_div(tokens, 64);
  const long long blocks = static_cast<long long>(ceil_div(Q, 64)) * plan.batch_heads;
  long long splits = (2ll * sm_count() + blocks / 2) / blocks;
  if (splits > tiles / 2) splits = tiles / 2;
  if (splits > 16) splits = 16;
  if (splits < 1) splits = 1;
  const int per = ceil_div(tiles, static_cast<int>(splits));
  plan.splits = ceil_div(tiles, per);
  plan.tokens_per_split = per * 64;
  return plan;
}

size_t partial_bytes(const F32Plan& plan, int Q, int heads, int d) {
  return plan.splits > 1 ? static_cast<size_t>(plan.splits) * Q * heads * (static_cast<size_t>(d) + 4) * 4 : 0;
}

template <int D>
int launch_rows(const RowAttn& a, int heads, int splits, cudaStream_t stream) {
  const size_t smem = sizeof(float) * (3 * D * 64 + 64 * 64);
  NKV_CUDA(cudaFuncSetAttribute(attn_rows_f32_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  attn_rows_f32_kernel<D><<<dim3(ceil_div(a.Q, 64), heads, splits), ATTN_THREADS, smem, stream>>>(a);
  NKV_LAUNCH_CHECK("attn_rows_f32_kernel");
  return NKV_OK;
}

}  // namespace

bool f32_attn_by_rows(int dk, int dv) { return dk == dv && (dk == 64 || dk == 128); }

size_t f32_attn_rows_workspace_bytes(int Q, int heads, int d, int tokens) {
  if (Q <= 0 || heads <= 0 || tokens <= 0) return 0;
  const F32Plan plan = plan_f32(Q, heads, d, tokens, true);
  return partial_bytes(plan, Q, heads, d) + static_cast<size_t>(tokens) * plan.batch_heads * d * 8 + 512;
}

int f32_attn_by_rows_run(const float* q, int64_t q_stride_token, int64_t q_stride_head, int Q, int heads, int d,
                         const nkv_history* hist_k, const nkv_history* hist_v, const float* wk, const float* bias_k,
                         const float* wv, const float* bias_v, float scale, float* out, float* lse, void* workspace,
                         cudaStream_t stream) {
  if (Q == 0 || heads == 0) return NKV_OK;
  const int N = hist_k->tokens, rank = hist_k->rank;
  const F32Plan plan = plan_f32(Q, heads, d, N, true);
  uint8_t* space = static_cast<uint8_t*>(workspace);
  space += (256 - (reinterpret_cast<uintptr_t>(space) & 255)) & 255;
  const size_t rows = static_cast<size_t>(Q) * heads;
  float* part_out = plan.splits > 1 ? reinterpret_cast<float*>(space) : out;
  float* part_lse = plan.splits > 1 ? part_out + plan.splits * rows * d : lse;
  float* rows_k = reinterpret_cast<float*>(space + (partial_bytes(plan, Q, heads, d) + 255) / 256 * 256);
  float* rows_v = rows_k + static_cast<size_t>(N) * plan.batch_heads * d;
  for (int h0 = 0; h0 < heads; h0 += plan.batch_heads) {
    const int hb = heads - h0 < plan.batch_heads ? heads - h0 : plan.batch_heads;
    const size_t col0 = static_cast<size_t>(h0) * d;
    const int J = hb * d;
    nkv_history hk = *hist_k, hv = *hist_v;
    hk.centers = static_cast<const uint16_t*>(hk.centers) + col0;
    hv.centers = static_cast<const uint16_t*>(hv.centers) + col0;
    int rc = simt_decode_rows(hk, nullptr, N, wk + col0 * rank, NKV_F32, bias_k + col0, J, rows_k, NKV_F32, J, stream);
    if (rc == NKV_OK)
      rc = simt_decode_rows(hv, nullptr, N, wv + col0 * rank, NKV_F32, bias_v + col0, J, rows_v, NKV_F32, J, stream);
    if (rc != NKV_OK) return rc;
    RowAttn a{};
    a.q = q + h0 * q_stride_head; a.q_stride_token = q_stride_token; a.q_stride_head = q_stride_head;
    a.k = rows_k; a.v = rows_v; a.kv_stride_token = J; a.kv_stride_head = d;
    a.Q = Q; a.heads = hb; a.out_heads = heads; a.N = N; a.tokens_per_split = plan.tokens_per_split; a.scale = scale;
    a.out = part_out + col0; a.lse = part_lse + h0;
    rc = d == 128 ? launch_rows<128>(a, hb, plan.splits, stream) : launch_rows<64>(a, hb, plan.splits, stream);
    if (rc != NKV_OK) return rc;
  }
  if (plan.splits == 1) return NKV_OK;
  merge_splits_kernel<<<static_cast<unsigned>((rows * (d / 4) + 255) / 256), 256, 0, stream>>>(
      part_out, part_lse, plan.splits, static_cast<long long>(rows), d, out, lse);
  NKV_LAUNCH_CHECK("merge_splits_kernel");
  return NKV_OK;
}

}  // namespace nkv
