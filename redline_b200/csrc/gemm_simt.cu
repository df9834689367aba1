// y[M, N] = x[M, K] . W[N, K]^T with float accumulation on the CUDA cores.
//
// This is the matrix product of the true 32-bit path (float operands, FFMA only,
// no tensor-core or TF32 mode), and the fallback for any mix of float / bfloat16
// operands (a weight stored in 32-bit next to bfloat16 activations, float logits
// from bfloat16 operands at small sizes).  Any M, N, K.
//
// Every output is summed in one order, whichever kernel computes it and whatever else is in the batch: K is cut
// into four quarters (of a multiple of four entries), a quarter's even and odd k run as two chains in ascending k
// (the two halves of a packed fma.rn.f32x2, each rounded like a plain fma), even + odd is the quarter's sum, and the
// quarters are added in order.  So a row's bits do not depend on how many other rows there are.  Places past the end
// are zeros in both operands and leave a sum as it is.
//
// Two kernels.  Few rows are bound by the weights' way from DRAM, and want many thread blocks with deep copy
// rings; many rows are bound by the FFMA pipe and want 8 x 8 outputs a thread, so that 16 shared-memory loads feed
// 256 multiply-adds.
// Measured on a B200 (float32; one launch over weights that are not in L2; in brackets the kernel of 64 x 64 tiles, 4 x 4
// outputs a thread and one chain over all of K that stood here before):
//   rows   N 3072 K 2048    N 2048 K 2048    N 16384 K 2048   N 2048 K 8192    N 128256 K 2048
//      1    8.1 us (152)     7.1 us (152)     31 us (232)      27 us (615)      183 us (1182; 5.7 TB/s)
//      4   12.1   (153)     10.3   (153)      38   (233)       30   (610)       221   (1191)
//     16   25     (152)     21     (153)      66   (237)       76   (623)       434   (1227)
//     64   49     (155)     32     (155)     148   (255)      126   (617)      1013   (1372)
//    210  117     (288)     74     (243)     479   (690)      280   (587)
//    512  218     (389)    146     (356)    1015  (1367)      555  (1119; 31 TFLOP/s)
// Their error against float64 is a third of the one chain's (2.9e-7 against 8e-7 at K = 2048).
#include <atomic>
#include <type_traits>

#include "common.cuh"

namespace rl {

constexpr int kQuarters = 4;

__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float even_plus_odd(unsigned long long acc) {
  return __uint_as_float(static_cast<uint32_t>(acc)) + __uint_as_float(static_cast<uint32_t>(acc >> 32));
}
// 16 bytes to shared memory; zeros where `in` is false (src is then any valid address).
__device__ __forceinline__ void copy16(void* dst, const void* src, bool in) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  const int n = in ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
// The same with 4 or 8 bytes (aligned to as many).
template <int BYTES>
__device__ __forceinline__ void copy_piece(void* dst, const void* src, bool in) {
  if constexpr (BYTES == 16) {
    copy16(dst, src, in);
  } else {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    const int n = in ? BYTES : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(BYTES), "r"(n) : "memory");
  }
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait_group() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__host__ __device__ inline int quarter_len(int K) { return ((K + kQuarters - 1) / kQuarters + 3) & ~3; }

// ---------------------------------------------------------------- few rows
//
// MG groups of 64 threads = 16 row groups x 4 quarters; a thread owns NPT weight rows of one quarter for MR rows of
// x, every group other rows of x.  A stage brings 32 k of every quarter; segments are 36 floats apart, so that eight
// neighbouring lanes' 16-byte reads fall into different banks.  N = 2048 gives 128 blocks (NPT = 1), which is what
// fills the chip at the smallest products; the ring keeps about 50 KB on their way per SM.
// Bound: the weights' bytes up to 2 rows; above, shared-memory reads (NPT + MR per NPT * MR * 4 multiply-adds), which
// want more warps than two, hence the groups.
constexpr int kSkK = 32, kSkPitch = kSkK + 4;

template <int MR, int NPT, int MG, int STAGES>
__global__ void __launch_bounds__(64 * MG)
simt_few_kernel(const float* __restrict__ w, const float* x, float* y, int M, int N, int K, int ldx, int ldy) {
  pdl_launch();
  constexpr int kThreads = 64 * MG;
  constexpr int NB = 16 * NPT;                     // weight rows of a block
  constexpr int kWSegs = NB * kQuarters, kXSegs = MR * MG * kQuarters;
  constexpr int kStageFloats = (kWSegs + kXSegs) * kSkPitch;
  extern __shared__ __align__(16) float sm[];
  const int t = threadIdx.x;
  const int n0 = blockIdx.x * NB, m0 = blockIdx.y * (MR * MG);
  const int ql = quarter_len(K);
  const int steps = (ql + kSkK - 1) / kSkK;

  auto ask_w = [&](int s) {
    float* st = sm + (s % STAGES) * kStageFloats;
#pragma unroll
    for (int j = 0; j < (kWSegs * 8 + kThreads - 1) / kThreads; ++j) {
      const int c = j * kThreads + t, seg = c >> 3, piece = c & 7;
      if (kWSegs * 8 % kThreads != 0 && seg >= kWSegs) break;
      const int n = n0 + seg / kQuarters, q = seg % kQuarters;
      const int off = s * kSkK + piece * 4, k = q * ql + off;
      const bool in = n < N && off < ql && k < K;
      copy16(st + seg * kSkPitch + piece * 4, in ? w + static_cast<size_t>(n) * K + k : w, in);
    }
  };
  auto ask_x = [&](int s) {
    float* st = sm + (s % STAGES) * kStageFloats + kWSegs * kSkPitch;
    for (int c = t; c < kXSegs * 8; c += kThreads) {
      const int seg = c >> 3, piece = c & 7;
      const int m = m0 + seg / kQuarters, q = seg % kQuarters;
      const int off = s * kSkK + piece * 4, k = q * ql + off;
      const bool in = m < M && off < ql && k < K;
      copy16(st + seg * kSkPitch + piece * 4, in ? x + static_cast<size_t>(m) * ldx + k : x, in);
    }
  };
  // the weights are nobody's output: the ring is filled before the wait on the kernel before
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s)
    if (s < steps) ask_w(s);
  pdl_wait();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < steps) ask_x(s);
    commit();                                      // (the weights asked for above belong to the first group)
  }
  const int q = t % kQuarters, g = (t / kQuarters) % 16, mg = t / 64;  // lanes: four quarters of eight row groups
  unsigned long long acc[NPT][MR];
#pragma unroll
  for (int i = 0; i < NPT; ++i)
#pragma unroll
    for (int m = 0; m < MR; ++m) acc[i][m] = 0ull;

  for (int s = 0; s < steps; ++s) {
    wait_group<STAGES - 2>();
    __syncthreads();
    if (s + STAGES - 1 < steps) {
      ask_w(s + STAGES - 1);
      ask_x(s + STAGES - 1);
    }
    commit();
    const float* st = sm + (s % STAGES) * kStageFloats;
    const float* xs = st + (kWSegs + mg * MR * kQuarters + q) * kSkPitch;
#pragma unroll
    for (int p = 0; p < kSkK / 4; ++p) {
      ulonglong2 a[NPT];
#pragma unroll
      for (int i = 0; i < NPT; ++i)
        a[i] = *reinterpret_cast<const ulonglong2*>(st + ((i * 16 + g) * kQuarters + q) * kSkPitch + p * 4);
#pragma unroll
      for (int m = 0; m < MR; ++m) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(xs + m * kQuarters * kSkPitch + p * 4);
#pragma unroll
        for (int i = 0; i < NPT; ++i) {
          fma2(acc[i][m], a[i].x, b.x);
          fma2(acc[i][m], a[i].y, b.y);
        }
      }
    }
  }
  // four neighbouring lanes hold an output's quarters
#pragma unroll
  for (int i = 0; i < NPT; ++i) {
    const int n = n0 + i * 16 + g;
#pragma unroll
    for (int m = 0; m < MR; ++m) {
      const int row = m0 + mg * MR + m;
      const float v = even_plus_odd(acc[i][m]);
      float sum = __shfl_sync(0xffffffffu, v, 0, kQuarters);
#pragma unroll
      for (int p = 1; p < kQuarters; ++p) sum += __shfl_sync(0xffffffffu, v, p, kQuarters);
      if (q == m % kQuarters && n < N && row < M) y[static_cast<size_t>(row) * ldy + n] = sum;
    }
  }
}

// ---------------------------------------------------------------- many rows, and every other mix of types
//
// A block computes 64 x 64 outputs; its four groups of 64 threads take a quarter of K each, 8 x 8 outputs a thread.
// Shared memory holds rows as they are (16 k of a row, 20 floats apart: conflict-free 16-byte reads along k, and
// the pairs of a packed fma lie side by side; bfloat16 rows stay bfloat16 and are widened when they are read).  The
// quarters meet in shared memory at the end.  P: the entries of an asynchronous copy into the ring of four stages, 4
// where every four k of both operands start on a boundary of their size, else 1 for two float operands; 0: loads
// entry by entry (a bfloat16 entry is too small to copy).
// Mixed types took the loads of P = 0, one after the other, in every case at first: 224 to 270 us for one row, 330 to
// 416 for 64, 2,000 for 2,048 at N 2048 K 2048 (the kernel of 64 x 64 tiles before: 135 to 150, 143 to 159, 690); with
// copies 29 to 33, 72 to 75, 502 to 521; with the loads of P = 0 asked for together (K 2045, 2046) 55, 91 to 96, 566 to 594.
// Bound: the FFMA pipe and the shared-memory reads, one after the other (2,048 cycles each a stage; 31 of 74 TFLOP/s).
// Plain instead of packed multiply-adds, or 8 x 4 outputs a thread on twice the warps, come out the same.
// The last tile of rows is often short of 64 (two prompts of 100 tokens leave 8): it runs with as many eights of rows as
// it has, in steps of two, and a thread's reads for the next four k lie among the multiply-adds of the present ones.
// Two prompts of 90 to 120 tokens with 8 new tokens each, Llama 1B sizes: 30.5 -> 29.2 ms by the two together.
constexpr int kTile = 64, kTlK = 16, kTlPitch = kTlK + 4, kTlStages = 4;
constexpr int kTlN = 8;                                                 // outputs of a thread: 8 rows of x, kTlN of the weights
constexpr int kTlCols = kTile / kTlN, kTlGroup = 8 * kTlCols, kTlThreads = kQuarters * kTlGroup;
constexpr int kTlGroupFloats = 2 * kTile * kTlPitch;                     // x rows, then weight rows
constexpr int kTlStageFloats = kQuarters * kTlGroupFloats;
constexpr int kTlSmem = kTlStages * kTlStageFloats * 4;
static_assert(kTlStages * kTlStageFloats >= (kQuarters - 1) * kTile * kTile, "the quarters' sums fit the ring");

// Four neighbouring k of a row in shared memory, as the two pairs of a packed multiply-add.
__device__ __forceinline__ ulonglong2 four(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }
__device__ __forceinline__ ulonglong2 four(const bf16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  auto pair = [](uint32_t v) { return static_cast<unsigned long long>(v & 0xffff0000u) << 32 | (v << 16); };
  return make_ulonglong2(pair(u.x), pair(u.y));
}

template <typename TA, typename TW, typename TC, int P>
__global__ void __launch_bounds__(kTlThreads, 1)
simt_tile_kernel(const TA* x, const TW* __restrict__ w, TC* y, int M, int N, int K, int ldx, int ldy) {
  pdl_launch();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  const int m0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
  const int g = threadIdx.x / kTlGroup, t = threadIdx.x % kTlGroup;     // the quarter; the thread in its group
  const int ty = t % 8, tx = t / 8;
  const int ql = quarter_len(K);
  const int steps = (ql + kTlK - 1) / kTlK;

  auto ask = [&](int s) {
    float* st = sm + (s % kTlStages) * kTlStageFloats + g * kTlGroupFloats;
    TA* xs = reinterpret_cast<TA*>(st);
    TW* ws = reinterpret_cast<TW*>(st + kTile * kTlPitch);
    if constexpr (P > 0) {
      constexpr int kPieces = kTlK / P, kRowsApart = kTlGroup / kPieces;
      const int at = t % kPieces * P, off = s * kTlK + at, k = g * ql + off;
      const bool in = off < ql && k < K;
#pragma unroll
      for (int j = 0; j < kTile / kRowsApart; ++j) {
        const int row = j * kRowsApart + t / kPieces;
        const bool xin = in && m0 + row < M, win = in && n0 + row < N;
        copy_piece<P * sizeof(TA)>(xs + row * kTlPitch + at, xin ? x + static_cast<size_t>(m0 + row) * ldx + k : x, xin);
        copy_piece<P * sizeof(TW)>(ws + row * kTlPitch + at, win ? w + static_cast<size_t>(n0 + row) * K + k : w, win);
      }
    } else {
      // (a thread has one k of every fourth row; all its loads, from places inside the operands, are on their way
      // before the first is stored)
      constexpr int kRowsApart = kTlGroup / kTlK, kLoads = kTile / kRowsApart;
      const int off = s * kTlK + t % kTlK, k = g * ql + off, kc = min(k, K - 1);
      const bool in = off < ql && k < K;
      TA xv[kLoads];
      TW wv[kLoads];
#pragma unroll
      for (int j = 0; j < kLoads; ++j) {
        const int row = j * kRowsApart + t / kTlK;
        xv[j] = x[static_cast<size_t>(min(m0 + row, M - 1)) * ldx + kc];
        wv[j] = w[static_cast<size_t>(min(n0 + row, N - 1)) * K + kc];
      }
#pragma unroll
      for (int j = 0; j < kLoads; ++j) {
        const int row = j * kRowsApart + t / kTlK;
        xs[row * kTlPitch + t % kTlK] = in && m0 + row < M ? xv[j] : from_float<TA>(0.f);
        ws[row * kTlPitch + t % kTlK] = in && n0 + row < N ? wv[j] : from_float<TW>(0.f);
      }
    }
  };
#pragma unroll
  for (int s = 0; s < kTlStages - 1; ++s) {
    if (s < steps) ask(s);
    commit();
  }
  unsigned long long acc[8][kTlN];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < kTlN; ++j) acc[i][j] = 0ull;

  // MI: eights of rows of x that the tile has (the last tile of a product has often fewer than eight).  The operands
  // of the next four k, and of the next column, are read while the present ones are multiplied.
  auto multiply = [&](auto mi) {
    constexpr int MI = decltype(mi)::value;
    for (int s = 0; s < steps; ++s) {
      wait_group<kTlStages - 2>();
      __syncthreads();
      if (s + kTlStages - 1 < steps) ask(s + kTlStages - 1);
      commit();
      const float* st = sm + (s % kTlStages) * kTlStageFloats + g * kTlGroupFloats;
      const TA* xs = reinterpret_cast<const TA*>(st);
      const TW* ws = reinterpret_cast<const TW*>(st + kTile * kTlPitch);
      auto x4 = [&](int i, int p) { return four(xs + (i * 8 + ty) * kTlPitch + p * 4); };
      auto w4 = [&](int j, int p) { return four(ws + (j * kTlCols + tx) * kTlPitch + p * 4); };
      ulonglong2 a[2][MI], b[2];
#pragma unroll
      for (int i = 0; i < MI; ++i) a[0][i] = x4(i, 0);
      b[0] = w4(0, 0);
#pragma unroll
      for (int p = 0; p < kTlK / 4; ++p) {
#pragma unroll
        for (int j = 0; j < kTlN; ++j) {
          const ulonglong2 bj = b[j & 1];
          if (j + 1 < kTlN) b[(j + 1) & 1] = w4(j + 1, p);
          else if (p + 1 < kTlK / 4) b[(j + 1) & 1] = w4(0, p + 1);
          if (j < MI && p + 1 < kTlK / 4) a[(p + 1) & 1][j] = x4(j, p + 1);
#pragma unroll
          for (int i = 0; i < MI; ++i) fma2(acc[i][j], a[p & 1][i].x, bj.x);
#pragma unroll
          for (int i = 0; i < MI; ++i) fma2(acc[i][j], a[p & 1][i].y, bj.y);
        }
      }
    }
  };
  const int eights = (min(M - m0, kTile) + 7) / 8;
  if (eights > 6) multiply(std::integral_constant<int, 8>());
  else if (eights > 4) multiply(std::integral_constant<int, 6>());
  else if (eights > 2) multiply(std::integral_constant<int, 4>());
  else multiply(std::integral_constant<int, 2>());
  wait_group<0>();
  __syncthreads();                                   // the ring is free: the quarters' sums move in
  if (g > 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < kTlN; ++j) sm[((g - 1) * kTile + i * 8 + ty) * kTile + j * kTlCols + tx] = even_plus_odd(acc[i][j]);
  }
  __syncthreads();
  if (g > 0) return;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + i * 8 + ty;
#pragma unroll
    for (int j = 0; j < kTlN; ++j) {
      const int n = n0 + j * kTlCols + tx;
      float sum = even_plus_odd(acc[i][j]);
#pragma unroll
      for (int q = 1; q < kQuarters; ++q) sum += sm[((q - 1) * kTile + i * 8 + ty) * kTile + j * kTlCols + tx];
      if (m < M && n < N) y[static_cast<size_t>(m) * ldy + n] = from_float<TC>(sum);
    }
  }
}

template <auto kKernel>
int raise_smem(int bytes) {
  static std::atomic<bool> raised[64];                 // per device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess && (dev >= 64 || !raised[dev].load(std::memory_order_relaxed))) {
    e = cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && dev < 64) raised[dev].store(true, std::memory_order_relaxed);
  }
  return static_cast<int>(e);
}

template <typename TA, typename TW, typename TC, int P>
int launch_tile(const void* x, const void* w, void* y, int M, int N, int K, int ldx, int ldy, cudaStream_t stream) {
  if (const int e = raise_smem<simt_tile_kernel<TA, TW, TC, P>>(kTlSmem)) return e;
  dim3 grid((N + kTile - 1) / kTile, (M + kTile - 1) / kTile);
  launch_kernel(simt_tile_kernel<TA, TW, TC, P>, grid, dim3(kTlThreads), kTlSmem, stream, static_cast<const TA*>(x),
                static_cast<const TW*>(w), static_cast<TC*>(y), M, N, K, ldx, ldy);
  return static_cast<int>(cudaGetLastError());
}

// Whether every four k of both operands lie on a boundary of their size.
template <typename TA, typename TW>
bool in_fours(const void* x, const void* w, int K, int ldx) {
  return K % 4 == 0 && ldx % 4 == 0 && reinterpret_cast<uintptr_t>(x) % (4 * sizeof(TA)) == 0 &&
         reinterpret_cast<uintptr_t>(w) % (4 * sizeof(TW)) == 0;
}

template <typename TA, typename TW, typename TC>
int launch_tiles(const void* x, const void* w, void* y, int M, int N, int K, int ldx, int ldy, cudaStream_t stream) {
  if (in_fours<TA, TW>(x, w, K, ldx)) return launch_tile<TA, TW, TC, 4>(x, w, y, M, N, K, ldx, ldy, stream);
  constexpr int kRest = sizeof(TA) == 4 && sizeof(TW) == 4 ? 1 : 0;          // (the smallest asynchronous copy is 4 bytes)
  return launch_tile<TA, TW, TC, kRest>(x, w, y, M, N, K, ldx, ldy, stream);
}

template <int MR, int NPT, int MG, int STAGES>
int launch_few(const float* x, const float* w, float* y, int M, int N, int K, int ldx, int ldy, cudaStream_t stream) {
  constexpr int smem = STAGES * (16 * NPT + MR * MG) * kQuarters * kSkPitch * 4;
  if (const int e = raise_smem<simt_few_kernel<MR, NPT, MG, STAGES>>(smem)) return e;
  dim3 grid((N + 16 * NPT - 1) / (16 * NPT), (M + MR * MG - 1) / (MR * MG));
  launch_kernel(simt_few_kernel<MR, NPT, MG, STAGES>, grid, dim3(64 * MG), smem, stream, w, x, y, M, N, K, ldx, ldy);
  return static_cast<int>(cudaGetLastError());
}

// Up to 16 rows the weights' bytes bound the product: the kernel for few rows.  Above, that kernel (16 rows at a
// time, 57 multiply-adds a clock and SM by its shared-memory reads on every SM) is the faster one while the tiles of
// the other (96 or so a clock on as many SMs as it has tiles) leave a third of the chip without work.
bool few_rows(int M, int N) {
  const long long tiles = static_cast<long long>((M + kTile - 1) / kTile) * ((N + kTile - 1) / kTile);
  return M <= 16 || tiles < 96;
}

int launch_f32(const void* xv, const void* wv, void* yv, int M, int N, int K, int ldx, int ldy, cudaStream_t stream) {
  const long long chunks = (static_cast<long long>(M) + 15) / 16;
  if (!in_fours<float, float>(xv, wv, K, ldx) || !few_rows(M, N) || chunks > 65535)
    return launch_tiles<float, float, float>(xv, wv, yv, M, N, K, ldx, ldy, stream);
  const float *x = static_cast<const float*>(xv), *w = static_cast<const float*>(wv);
  float* y = static_cast<float*>(yv);
  if (M == 1) return launch_few<1, 1, 1, 6>(x, w, y, M, N, K, ldx, ldy, stream);
  if (M == 2) return launch_few<2, 1, 1, 6>(x, w, y, M, N, K, ldx, ldy, stream);
  if (M <= 4) return launch_few<2, 1, 2, 6>(x, w, y, M, N, K, ldx, ldy, stream);
  if (M <= 8) return launch_few<4, 1, 2, 5>(x, w, y, M, N, K, ldx, ldy, stream);
  return launch_few<4, 2, 4, 4>(x, w, y, M, N, K, ldx, ldy, stream);
}

}  // namespace rl

using namespace rl;

extern "C" {

// dtypes: 0 = float32, 1 = bfloat16.  ldx / ldy: row strides of x and y in elements.
int rl_gemm_tn_simt(const void* x, int x_dtype, const void* w, int w_dtype, void* y, int y_dtype,
                    int M, int N, int K, int ldx, int ldy, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  const int code = x_dtype * 4 + w_dtype * 2 + y_dtype;
  switch (code) {
    case 0: return launch_f32(x, w, y, M, N, K, ldx, ldy, stream);
    case 1: return launch_tiles<float, float, bf16>(x, w, y, M, N, K, ldx, ldy, stream);
    case 2: return launch_tiles<float, bf16, float>(x, w, y, M, N, K, ldx, ldy, stream);
    case 3: return launch_tiles<float, bf16, bf16>(x, w, y, M, N, K, ldx, ldy, stream);
    case 4: return launch_tiles<bf16, float, float>(x, w, y, M, N, K, ldx, ldy, stream);
    case 5: return launch_tiles<bf16, float, bf16>(x, w, y, M, N, K, ldx, ldy, stream);
    case 6: return launch_tiles<bf16, bf16, float>(x, w, y, M, N, K, ldx, ldy, stream);
    case 7: return launch_tiles<bf16, bf16, bf16>(x, w, y, M, N, K, ldx, ldy, stream);
  }
  return static_cast<int>(cudaErrorInvalidValue);
}

}  // extern "C"
