// Token sampling on the GPU: one CTA per row of float logits, or a cluster of eight where rows are drawn from a
// large vocabulary (sample_clusters).
//
//   temperature <= 0   greedy: the arg max, the smaller index on ties
//   temperature  > 0   temperature, then top-k (ties at the k-th value kept), then
//                      top-p over what top-k kept, then one draw by the Gumbel-max
//                      trick: argmax_i (l_i - max) / T - log(-log(u_i)), u_i from
//                      Philox4x32-10 keyed by the request's seed with the counter
//                      (token index, position of the token being drawn, stream),
//                      so a draw does not depend on what else is in the batch.
//
// The thresholds of top-k and top-p are found without a sort by four 8-bit radix
// passes over order-preserving integer keys of the logits, counting tokens (top-k)
// or probability mass (top-p).  Mass is summed as 40-bit fixed point in integer
// atomics, so the result does not depend on the order in which threads arrive.
//
// What is the reference's and what is this file's own: the threshold search follows the
// reference's radix selection pass for pass (src/cuda/kernels/sampling.cu:53-127, including
// its rule for a target that rounding left out of reach: keep all that remains), and the
// Philox round, its counter layout and the constant 0x52444C4E in the counter are the
// reference's (src/cuda/kernels/common.cuh:105-140), as they must be for a seed to draw the
// same token in both engines.  The fixed-point mass in integer atomics, the two-stage arg max
// over chunks of a row and the kernels' organisation are this file's.
#include <atomic>
#include <cfloat>

#include "common.cuh"

namespace rl {

constexpr int kSampleThreads = 1024;

__device__ __forceinline__ uint32_t order_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u >> 31) ? ~u : (u | 0x80000000u);
}

struct Best {
  float v;
  int i;
};
__device__ __forceinline__ Best better(Best a, Best b) {
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}
__device__ Best block_best(Best x, Best* scratch) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Best y;
    y.v = __shfl_xor_sync(0xffffffffu, x.v, o);
    y.i = __shfl_xor_sync(0xffffffffu, x.i, o);
    x = better(x, y);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) scratch[warp] = x;
  __syncthreads();
  Best r = lane < (blockDim.x >> 5) ? scratch[lane] : Best{-FLT_MAX, 0x7fffffff};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Best y;
    y.v = __shfl_xor_sync(0xffffffffu, r.v, o);
    y.i = __shfl_xor_sync(0xffffffffu, r.i, o);
    r = better(r, y);
  }
  return r;
}

__device__ __forceinline__ uint4 philox_4x32_10(uint4 c, uint2 k) {
  const uint32_t m0 = 0xD2511F53u, m1 = 0xCD9E8D57u;
  for (int round = 0; round < 10; ++round) {
    const uint32_t h0 = __umulhi(m0, c.x), l0 = m0 * c.x;
    const uint32_t h1 = __umulhi(m1, c.z), l1 = m1 * c.z;
    c = make_uint4(h1 ^ c.y ^ k.x, l1, h0 ^ c.w ^ k.y, l0);
    k.x += 0x9E3779B9u;
    k.y += 0xBB67AE85u;
  }
  return c;
}

// Uniform in the open interval (0, 1): 24 bits of the first Philox word, centred.
__device__ __forceinline__ float uniform_open01(uint32_t seed_lo, uint32_t seed_hi, uint32_t position,
                                                uint32_t stream, uint32_t index) {
  const uint4 r = philox_4x32_10(make_uint4(index, position, stream, 0x52444C4Eu),
                                 make_uint2(seed_lo, seed_hi));
  return (static_cast<float>(r.x >> 8) + 0.5f) * (1.0f / 16777216.0f);
}

struct SampleSmem {
  float fscratch[32];
  Best bscratch[32];
  unsigned long long hist[256];
  uint32_t prefix;
  unsigned long long remaining;
};

constexpr float kMassScale = 1099511627776.0f;  // 2^40

// Key of the k-th largest logit.
__device__ uint32_t select_top_k(const float* l, int vocab, int k, SampleSmem& sh) {
  uint32_t prefix = 0, mask = 0;
  unsigned long long want = static_cast<unsigned long long>(k);
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (int b = threadIdx.x; b < 256; b += blockDim.x) sh.hist[b] = 0ull;
    __syncthreads();
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
      const uint32_t key = order_key(l[i]);
      if ((key & mask) == prefix) atomicAdd(&sh.hist[(key >> shift) & 255u], 1ull);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long above = 0;
      int b = 255;
      for (; b > 0; --b) {
        if (above + sh.hist[b] >= want) break;
        above += sh.hist[b];
      }
      sh.prefix = prefix | (static_cast<uint32_t>(b) << shift);
      sh.remaining = want - above;
    }
    __syncthreads();
    prefix = sh.prefix;
    want = sh.remaining;
    mask |= 255u << shift;
  }
  return prefix;
}

// Largest key t such that the mass of {key >= t} among {key >= floor_key} reaches `target`
// (fixed point, scaled by 2^40 relative to the largest term).
__device__ uint32_t select_top_p(const float* l, int vocab, float mx, float inv_t, uint32_t floor_key,
                                 unsigned long long target, SampleSmem& sh) {
  uint32_t prefix = 0, mask = 0;
  unsigned long long want = target;
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (int b = threadIdx.x; b < 256; b += blockDim.x) sh.hist[b] = 0ull;
    __syncthreads();
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
      const uint32_t key = order_key(l[i]);
      if (key >= floor_key && (key & mask) == prefix) {
        const unsigned long long q =
            static_cast<unsigned long long>(expf((l[i] - mx) * inv_t) * kMassScale);
        atomicAdd(&sh.hist[(key >> shift) & 255u], q);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long above = 0;
      int chosen = -1, lowest = 0;
      for (int b = 255; b >= 0; --b) {
        const unsigned long long c = sh.hist[b];
        if (c == 0ull) continue;
        lowest = b;
        if (above + c >= want) {
          chosen = b;
          break;
        }
        above += c;
      }
      if (chosen < 0) {  // rounding left the target out of reach: keep all that remains
        chosen = lowest;
        sh.remaining = 0ull;
      } else {
        sh.remaining = want - above;
      }
      sh.prefix = prefix | (static_cast<uint32_t>(chosen) << shift);
    }
    __syncthreads();
    prefix = sh.prefix;
    want = sh.remaining;
    mask |= 255u << shift;
  }
  return prefix;
}

// First stage for greedy rows: the row is cut into pieces (kSampleChunks of them, or a quarter as many
// when the launch has many rows: CTAs of 2,000 values each are mostly start and end), one CTA each, which
// leave (max, arg max, sum of exp(l - max)) of their piece.  sample_kernel combines them.
constexpr int kSampleChunks = 64;

struct ChunkStat {
  float mx;
  int idx;
  float sumexp;
  float pad;
};

template <int kSampleHeld>
__global__ void __launch_bounds__(256)
sample_partial_kernel(const float* __restrict__ logits, int vocab, int ld, ChunkStat* __restrict__ stats, int chunks) {
  pdl_launch();
  pdl_wait();
  __shared__ Best bscratch[32];
  __shared__ float fscratch[32];
  const int row = blockIdx.x, chunk = blockIdx.y;
  const int per = (vocab + chunks - 1) / chunks;
  const int lo = chunk * per, hi = min(vocab, lo + per);
  const float* l = logits + static_cast<size_t>(row) * ld;
  // (the second stage reads kSampleChunks slots a row: those beyond this launch's pieces are marked empty)
  if (chunk == 0 && threadIdx.x < kSampleChunks - chunks)
    stats[row * kSampleChunks + chunks + threadIdx.x] = ChunkStat{-FLT_MAX, 0x7fffffff, 0.f, 0.f};
  // A thread's first kSampleHeld values stay in registers (all their loads are in flight together, and the
  // piece is read once); a piece longer than 256 * kSampleHeld goes on through memory.
  float v[kSampleHeld];
#pragma unroll
  for (int j = 0; j < kSampleHeld; ++j) {
    const int i = lo + threadIdx.x + j * 256;
    v[j] = i < hi ? l[i] : -FLT_MAX;
  }
  Best b{-FLT_MAX, 0x7fffffff};
#pragma unroll
  for (int j = 0; j < kSampleHeld; ++j) {
    const int i = lo + threadIdx.x + j * 256;
    if (i < hi) b = better(b, Best{v[j], i});
  }
  for (int i = lo + threadIdx.x + kSampleHeld * 256; i < hi; i += 256) b = better(b, Best{l[i], i});
  b = block_best(b, bscratch);
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < kSampleHeld; ++j) {
    const int i = lo + threadIdx.x + j * 256;
    if (i < hi) s += expf(v[j] - b.v);
  }
  for (int i = lo + threadIdx.x + kSampleHeld * 256; i < hi; i += 256) s += expf(l[i] - b.v);
  s = block_sum(s, fscratch);
  if (threadIdx.x == 0) stats[row * kSampleChunks + chunk] = ChunkStat{b.v, b.i, s, 0.f};
}

// A row's result (one thread).  A row of which no logit is above -inf (all -inf, or NaN) has no best token: it gets
// token 0 and the log-probability NaN, and nothing is read at the index that stands for "none".
__device__ __forceinline__ void write_draw(const float* l, int token, float lse, int row, int32_t* out_token,
                                           float* out_logprob) {
  const bool found = token != 0x7fffffff;
  out_token[row] = found ? token : 0;
  if (out_logprob) out_logprob[row] = found ? l[token] - lse : NAN;
}

// Greedy row with first-stage statistics, by one warp: combine the pieces (smaller index wins ties).
__device__ __forceinline__ void greedy_from_stats(const float* l, const ChunkStat* stats, int row,
                                                  int32_t* out_token, float* out_logprob) {
  Best b{-FLT_MAX, 0x7fffffff};
  for (int c = threadIdx.x; c < kSampleChunks; c += 32) {
    const ChunkStat st = stats[c];
    if (st.idx != 0x7fffffff) b = better(b, Best{st.mx, st.idx});
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Best y;
    y.v = __shfl_xor_sync(0xffffffffu, b.v, o);
    y.i = __shfl_xor_sync(0xffffffffu, b.i, o);
    b = better(b, y);
  }
  float sum = 0.f;
  for (int c = threadIdx.x; c < kSampleChunks; c += 32) {
    const ChunkStat st = stats[c];
    if (st.idx != 0x7fffffff) sum += st.sumexp * expf(st.mx - b.v);
  }
  sum = warp_sum(sum);
  if (threadIdx.x == 0) write_draw(l, b.i, b.v + logf(sum), row, out_token, out_logprob);
}

__global__ void __launch_bounds__(kSampleThreads)
sample_kernel(const float* __restrict__ logits, int vocab, int ld, const float* __restrict__ temperature,
              const int32_t* __restrict__ top_k, const float* __restrict__ top_p,
              const uint32_t* __restrict__ seed_lo, const uint32_t* __restrict__ seed_hi,
              const int32_t* __restrict__ position, uint32_t stream_id, int32_t* __restrict__ out_token,
              float* __restrict__ out_logprob, const ChunkStat* __restrict__ stats) {
  pdl_launch();
  pdl_wait();
  __shared__ SampleSmem sh;
  const int row = blockIdx.x;
  const float* l = logits + static_cast<size_t>(row) * ld;
  if (stats != nullptr && temperature[row] <= 0.f) {
    if (threadIdx.x < 32) greedy_from_stats(l, stats + row * kSampleChunks, row, out_token, out_logprob);
    return;
  }

  Best b{-FLT_MAX, 0x7fffffff};
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) b = better(b, Best{l[i], i});
  b = block_best(b, sh.bscratch);
  const float mx = b.v;
  float s = 0.f;
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) s += expf(l[i] - mx);
  s = block_sum(s, sh.fscratch);
  const float lse = mx + logf(s);

  int token = b.i;
  const float temp = temperature[row];
  if (temp > 0.f) {
    const float inv_t = 1.f / temp;
    uint32_t thr = 0;
    const int k = top_k[row];
    if (k > 0 && k < vocab) thr = select_top_k(l, vocab, k, sh);
    const float p = top_p[row];
    if (p < 1.f) {
      // total mass of what top-k kept, in the same fixed point
      unsigned long long part = 0;
      for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
        if (order_key(l[i]) >= thr)
          part += static_cast<unsigned long long>(expf((l[i] - mx) * inv_t) * kMassScale);
      }
      __syncthreads();
      if (threadIdx.x == 0) sh.remaining = 0ull;
      __syncthreads();
      atomicAdd(&sh.remaining, part);
      __syncthreads();
      const unsigned long long total = sh.remaining;
      __syncthreads();
      const unsigned long long target =
          static_cast<unsigned long long>(static_cast<double>(p) * static_cast<double>(total));
      const uint32_t thr_p = select_top_p(l, vocab, mx, inv_t, thr, target > 0 ? target : 1ull, sh);
      thr = max(thr, thr_p);
    }
    Best g{-FLT_MAX, 0x7fffffff};
    const uint32_t slo = seed_lo[row], shi = seed_hi[row];
    const uint32_t pos = static_cast<uint32_t>(position[row]);
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
      if (order_key(l[i]) < thr) continue;
      const float u = uniform_open01(slo, shi, pos, stream_id, static_cast<uint32_t>(i));
      g = better(g, Best{(l[i] - mx) * inv_t - logf(-logf(u)), i});
    }
    g = block_best(g, sh.bscratch);
    if (g.i != 0x7fffffff) token = g.i;
  }
  if (threadIdx.x == 0) write_draw(l, token, lse, row, out_token, out_logprob);
}

// ---------------------------------------------------------------- sampled rows of a large vocabulary
//
// The same draw with a cluster of kRowCtas CTAs per row, each with its share of the row in shared memory.  The draw
// takes ten passes over the row (arg max, sum, mass, four radix passes each of top-k and top-p, Gumbel); one CTA that
// read 513 KB for each of them from L2 took 344 us for rows of 128,256 logits (B200, 1 to 32 rows with top-p), this
// one 47 us at 21 rows together with the wait for the kernel before it.  Every pass here runs over 64 KB in shared memory, and the CTAs' counts or masses meet through distributed shared memory.
// All selections are over integers (counts, fixed-point mass) or maxima, so they are the same bits in any order: the
// tokens are those of sample_kernel.  Of a greedy row's cluster one warp works.
constexpr int kRowCtas = 8, kRowThreads = 512;
constexpr int kRowMaxBytes = 200 * 1024;

int row_share_bytes(int vocab) { return (((vocab + kRowCtas - 1) / kRowCtas + 3) & ~3) * 4; }

// Whether a launch gets clusters.  draws: 0 no row is drawn (all temperatures are 0), 1 rows are drawn from the whole
// vocabulary, 2 with top-k or top-p.  Clusters are eight times the CTAs, so few rows and long ones gain; us for one CTA
// per row / clusters, B200:
//               vocabulary 8,192                      16,384                       32,000               128,256
//   top-p       21 rows 184 / 65, 96 237 / 193,       64 355 / 167, 192 556 / 476, 256 965 / 880,       256 3,582 / 2,485,
//               192 348 / 376, 512 695 / 946          256 568 / 629                512 1,878 / 1,681    512 7,067 / 4,779
//   no filter   16 rows 16 / 15, 32 19 / 19,          32 27 / 21, 48 30 / 32,      64 51 / 46,          384 584 / 539,
//               64 32 / 34, 256 65 / 122              128 58 / 70                  96 56 / 66           512 763 / 714
//   greedy      8 rows 5.5 / 6.5, 256 48 / 53         8 5.5 / 6.5, 256 49 / 54     64 16.3 / 17.0       64 20.9 / 21.8
// Below 8,192 entries a pass of one CTA is short (4,096: 21 rows with top-p 126 us).
bool sample_clusters(int rows, int vocab, int draws) {
  if (draws <= 0 || vocab < 8192 || row_share_bytes(vocab) > kRowMaxBytes) return false;
  return rows <= vocab / (draws == 1 ? 340 : 80);
}

struct RowSmem {
  float fscratch[32];
  Best bscratch[32];
  Best best;                           // this CTA's answers, for the cluster
  float fsum;
  unsigned long long mass;
  unsigned long long hist[2][256];     // this CTA's bins (two sets in turn: one is cleared while peers may read the other)
  unsigned long long total[256];       // the cluster's
  uint32_t prefix;
  unsigned long long remaining;
};

__device__ __forceinline__ void cluster_meet() {
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t peer_address(const void* p, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(rank));
  return a;
}
__device__ __forceinline__ uint32_t peer_u32(const void* p, uint32_t rank) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(peer_address(p, rank)) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long peer_u64(const void* p, uint32_t rank) {
  unsigned long long v;
  asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(peer_address(p, rank)) : "memory");
  return v;
}

// The best of every CTA's `b` (which all threads of the CTA have).  `slot` is free again after the next meeting.
__device__ Best cluster_best(Best b, Best* slot) {
  if (threadIdx.x == 0) *slot = b;
  cluster_meet();
  Best r{-FLT_MAX, 0x7fffffff};
#pragma unroll
  for (int c = 0; c < kRowCtas; ++c)
    r = better(r, Best{__uint_as_float(peer_u32(&slot->v, c)), static_cast<int>(peer_u32(&slot->i, c))});
  return r;
}

// One radix selection over the cluster's rows: `add(i)` says what value i of this CTA's share adds to its bin (0: not
// counted).  Walks the bins from the top until `want` is reached.  kMass: bins without mass are passed over, and if
// rounding left the target out of reach the lowest one with mass is taken and all that remains kept; otherwise the
// lowest bin is taken unseen.
template <bool kMass, typename Add>
__device__ uint32_t cluster_select(const float* l, int count, unsigned long long want, Add add, RowSmem& sh) {
  uint32_t prefix = 0, mask = 0;
  int turn = 0;
  for (int b = threadIdx.x; b < 256; b += blockDim.x) sh.hist[0][b] = 0ull;
  __syncthreads();
  for (int shift = 24; shift >= 0; shift -= 8, turn ^= 1) {
    for (int i = threadIdx.x; i < count; i += blockDim.x) {
      const uint32_t key = order_key(l[i]);
      if ((key & mask) == prefix) {
        const unsigned long long q = add(l[i], key);
        if (q != 0ull) atomicAdd(&sh.hist[turn][(key >> shift) & 255u], q);
      }
    }
    cluster_meet();
    if (threadIdx.x < 256) {
      unsigned long long t = 0;
#pragma unroll
      for (int c = 0; c < kRowCtas; ++c) t += peer_u64(&sh.hist[turn][threadIdx.x], c);
      sh.total[threadIdx.x] = t;
      sh.hist[turn ^ 1][threadIdx.x] = 0ull;       // (read by peers before this meeting only)
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      // lane n has the bins 255 - 8 n .. 248 - 8 n, from the top
      const int top = 255 - 8 * static_cast<int>(threadIdx.x);
      unsigned long long own = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) own += sh.total[top - j];
      unsigned long long upto = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, upto, o);
        if (static_cast<int>(threadIdx.x) >= o) upto += y;
      }
      // (a mass of zero is wanted where rounding ended an earlier pass: the first bin with mass then)
      const unsigned long long least = kMass && want == 0ull ? 1ull : want;
      const unsigned reached = __ballot_sync(0xffffffffu, upto >= least);
      const unsigned filled = __ballot_sync(0xffffffffu, own != 0ull);
      if (reached != 0u) {
        if (static_cast<int>(threadIdx.x) == __ffs(reached) - 1) {
          unsigned long long above = upto - own;
          int b = top;
          for (; b > top - 7; --b) {
            if (above + sh.total[b] >= least) break;
            above += sh.total[b];
          }
          sh.prefix = prefix | (static_cast<uint32_t>(b) << shift);
          sh.remaining = want > above ? want - above : 0ull;
        }
      } else if (kMass) {
        if (filled == 0u ? threadIdx.x == 0 : static_cast<int>(threadIdx.x) == 31 - __clz(filled)) {
          int b = top - 7;
          while (b < top && sh.total[b] == 0ull) ++b;
          sh.prefix = prefix | (static_cast<uint32_t>(filled == 0u ? 0 : b) << shift);
          sh.remaining = 0ull;
        }
      } else if (threadIdx.x == 31) {
        sh.prefix = prefix;
        sh.remaining = want - (upto - sh.total[0]);
      }
    }
    __syncthreads();
    prefix = sh.prefix;
    want = sh.remaining;
    mask |= 255u << shift;
  }
  cluster_meet();                                  // (no peer reads these bins any more)
  return prefix;
}

__global__ void __launch_bounds__(kRowThreads)
sample_cluster_kernel(const float* __restrict__ logits, int vocab, int ld, const float* __restrict__ temperature,
                      const int32_t* __restrict__ top_k, const float* __restrict__ top_p,
                      const uint32_t* __restrict__ seed_lo, const uint32_t* __restrict__ seed_hi,
                      const int32_t* __restrict__ position, uint32_t stream_id, int32_t* __restrict__ out_token,
                      float* __restrict__ out_logprob, const ChunkStat* __restrict__ stats) {
  pdl_launch();
  pdl_wait();
  __shared__ RowSmem sh;
  extern __shared__ __align__(16) float share[];
  const int row = blockIdx.x / kRowCtas;
  const uint32_t rank = cluster_rank();
  const float* l = logits + static_cast<size_t>(row) * ld;
  const float temp = temperature[row];
  if (stats != nullptr && temp <= 0.f) {           // (the same for every CTA of the cluster)
    if (rank == 0 && threadIdx.x < 32) greedy_from_stats(l, stats + row * kSampleChunks, row, out_token, out_logprob);
    return;
  }
  const int per = ((vocab + kRowCtas - 1) / kRowCtas + 3) & ~3;
  const int lo = min(vocab, static_cast<int>(rank) * per), count = min(vocab - lo, per);
  if ((ld & 3) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0) {
    for (int i = threadIdx.x * 4; i + 4 <= count; i += blockDim.x * 4)
      *reinterpret_cast<float4*>(share + i) = *reinterpret_cast<const float4*>(l + lo + i);
    for (int i = (count & ~3) + threadIdx.x; i < count; i += blockDim.x) share[i] = l[lo + i];
  } else {
    for (int i = threadIdx.x; i < count; i += blockDim.x) share[i] = l[lo + i];
  }
  __syncthreads();
  Best b{-FLT_MAX, 0x7fffffff};
  for (int i = threadIdx.x; i < count; i += blockDim.x) b = better(b, Best{share[i], lo + i});
  b = cluster_best(block_best(b, sh.bscratch), &sh.best);
  const float mx = b.v;
  float s = 0.f;
  for (int i = threadIdx.x; i < count; i += blockDim.x) s += expf(share[i] - mx);
  s = block_sum(s, sh.fscratch);
  if (threadIdx.x == 0) sh.fsum = s;
  cluster_meet();
  s = 0.f;
#pragma unroll
  for (int c = 0; c < kRowCtas; ++c) s += __uint_as_float(peer_u32(&sh.fsum, c));
  const float lse = mx + logf(s);

  int token = b.i;
  if (temp > 0.f) {
    const float inv_t = 1.f / temp;
    uint32_t thr = 0;
    const int k = top_k[row];
    if (k > 0 && k < vocab)
      thr = cluster_select<false>(share, count, static_cast<unsigned long long>(k),
                                  [](float, uint32_t) { return 1ull; }, sh);
    const float p = top_p[row];
    if (p < 1.f) {
      // total mass of what top-k kept, in the same fixed point
      unsigned long long part = 0;
      for (int i = threadIdx.x; i < count; i += blockDim.x) {
        if (order_key(share[i]) >= thr)
          part += static_cast<unsigned long long>(expf((share[i] - mx) * inv_t) * kMassScale);
      }
      if (threadIdx.x == 0) sh.mass = 0ull;
      __syncthreads();
      if (part != 0ull) atomicAdd(&sh.mass, part);
      cluster_meet();
      unsigned long long total = 0;
#pragma unroll
      for (int c = 0; c < kRowCtas; ++c) total += peer_u64(&sh.mass, c);
      const unsigned long long target =
          static_cast<unsigned long long>(static_cast<double>(p) * static_cast<double>(total));
      const uint32_t floor_key = thr;
      const uint32_t thr_p = cluster_select<true>(
          share, count, target > 0 ? target : 1ull,
          [=](float v, uint32_t key) {
            return key >= floor_key ? static_cast<unsigned long long>(expf((v - mx) * inv_t) * kMassScale) : 0ull;
          },
          sh);
      thr = max(thr, thr_p);
    }
    Best g{-FLT_MAX, 0x7fffffff};
    const uint32_t slo = seed_lo[row], shi = seed_hi[row];
    const uint32_t pos = static_cast<uint32_t>(position[row]);
    for (int i = threadIdx.x; i < count; i += blockDim.x) {
      if (order_key(share[i]) < thr) continue;
      const float u = uniform_open01(slo, shi, pos, stream_id, static_cast<uint32_t>(lo + i));
      g = better(g, Best{(share[i] - mx) * inv_t - logf(-logf(u)), lo + i});
    }
    cluster_meet();                                // (sh.best has been read by every CTA)
    g = cluster_best(block_best(g, sh.bscratch), &sh.best);
    if (g.i != 0x7fffffff) token = g.i;
  }
  if (rank == 0 && threadIdx.x == 0) write_draw(l, token, lse, row, out_token, out_logprob);
  cluster_meet();                                  // (no CTA ends while a peer may read its shared memory)
}

// out[r] = log_softmax(logits[r, :])[target[r]]   (sampling.cu:288-300); NaN for a target outside the row.
// One pass: a thread keeps a running maximum and the sum scaled to it over eight values at a time, which are all on
// their way together (bound by the rows' bytes: 400 rows of 128,256 logits in 53 us, 3.9 TB/s; two passes a value
// at a time took 138 us for 64 rows).
__global__ void __launch_bounds__(512)
gather_logprob_kernel(const float* __restrict__ logits, int vocab, int ld,
                      const int32_t* __restrict__ target, float* __restrict__ out) {
  pdl_launch();
  pdl_wait();
  __shared__ float scratch[32];
  const float* l = logits + static_cast<size_t>(blockIdx.x) * ld;
  constexpr int kHeld = 8;
  float m = -FLT_MAX, s = 0.f;
  for (int base = 0; base < vocab; base += kHeld * 512) {
    float v[kHeld];
#pragma unroll
    for (int j = 0; j < kHeld; ++j) {
      const int i = base + j * 512 + threadIdx.x;
      v[j] = i < vocab ? l[i] : -INFINITY;
    }
    float top = m;
#pragma unroll
    for (int j = 0; j < kHeld; ++j) top = fmaxf(top, v[j]);
    s *= expf(m - top);
#pragma unroll
    for (int j = 0; j < kHeld; ++j) s += expf(v[j] - top);
    m = top;
  }
  const float mx = block_max(m, scratch);
  s = block_sum(s * expf(m - mx), scratch);
  if (threadIdx.x == 0) {
    const int t = target[blockIdx.x];
    out[blockIdx.x] = t >= 0 && t < vocab ? l[t] - (mx + logf(s)) : NAN;
  }
}

}  // namespace rl

using namespace rl;

extern "C" {

int rl_sample_chunks() { return kSampleChunks; }

// Whether rl_sample with these arguments launches clusters (see sample_clusters).
int rl_sample_clusters(int rows, int vocab, int draws) { return sample_clusters(rows, vocab, draws) ? 1 : 0; }

// scratch: optional [rows * rl_sample_chunks() * 4] floats.  With it, rows whose temperature is <= 0
// are served by a two-stage arg max that uses the whole GPU instead of one CTA per row.
// draws: what the rows ask for (see sample_clusters); it decides which kernel runs, not what a row gets.
int rl_sample(const float* logits, int rows, int vocab, int ld, const float* temperature,
              const int32_t* top_k, const float* top_p, const uint32_t* seed_lo,
              const uint32_t* seed_hi, const int32_t* position, unsigned stream_id,
              int32_t* out_token, float* out_logprob, float* scratch, int draws, cudaStream_t stream) {
  if (rows <= 0) return 0;
  ChunkStat* stats = reinterpret_cast<ChunkStat*>(scratch);
  if (stats != nullptr) {
    if (rows >= 16)
      launch_kernel(sample_partial_kernel<32>, dim3(rows, kSampleChunks / 4), dim3(256), 0, stream, logits, vocab, ld,
                    stats, kSampleChunks / 4);
    else
      launch_kernel(sample_partial_kernel<8>, dim3(rows, kSampleChunks), dim3(256), 0, stream, logits, vocab, ld,
                    stats, kSampleChunks);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  if (sample_clusters(rows, vocab, draws)) {
    static std::atomic<bool> raised[64];              // per device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev >= 64 || !raised[dev].load(std::memory_order_relaxed)) {
      e = cudaFuncSetAttribute(sample_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowMaxBytes);
      if (e != cudaSuccess) return static_cast<int>(e);
      if (dev < 64) raised[dev].store(true, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(rows * kRowCtas);
    cfg.blockDim = dim3(kRowThreads);
    cfg.dynamicSmemBytes = row_share_bytes(vocab);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kRowCtas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, sample_cluster_kernel, logits, vocab, ld, temperature, top_k, top_p,
                                             seed_lo, seed_hi, position, static_cast<uint32_t>(stream_id), out_token,
                                             out_logprob, static_cast<const ChunkStat*>(stats));
    return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
  }
  launch_kernel(sample_kernel, dim3(rows), dim3(kSampleThreads), 0, stream, logits, vocab, ld, temperature, top_k, top_p,
                                                     seed_lo, seed_hi, position, stream_id, out_token,
                                                     out_logprob, stats);
  RL_LAUNCH_END();
}

int rl_gather_logprob(const float* logits, int rows, int vocab, int ld, const int32_t* target,
                      float* out, cudaStream_t stream) {
  if (rows <= 0) return 0;
  launch_kernel(gather_logprob_kernel, dim3(rows), dim3(512), 0, stream, logits, vocab, ld, target, out);
  RL_LAUNCH_END();
}

}  // extern "C"
