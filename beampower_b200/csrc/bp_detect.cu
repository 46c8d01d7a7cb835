// Detection on the beam series, on the GPU: the reference tutorial's
// time-dependent threshold (notebooks/3_beampower.ipynb:497-579) and its
// peak picking -- scipy.signal.find_peaks(beam_max, distance=...) followed by
// the strict threshold test (notebooks/3_beampower.ipynb:618-626) -- with
// results identical to the NumPy / SciPy code.
//
// Exactness rests on three restatements:
//  * NumPy's float32 sum (inside mean and std) is a pairwise sum whose split
//    points depend on the length only, so every node is found from its path
//    from the root.  Leaves are summed in parallel, and nodes level by level,
//    each with the same rounded operations as NumPy's loop.
//  * NumPy's median is an order statistic (the mean of the two middle values
//    for even lengths); a radix select on the order-preserving integer image of
//    the floats finds it exactly.
//  * SciPy's distance rule is a greedy pass in decreasing height.  Its result
//    is also the fixed point of rounds in which every undecided peak with no
//    higher undecided peak within the distance is kept, and then every
//    undecided peak within the distance of a kept one is dropped.
#define BP_TEMPLATE_KERNELS_ONLY
#include <cmath>
#include <utility>

#include <cooperative_groups.h>
#include <cuda.h>

#include "bp_stats.cuh"

namespace {

// ---- NumPy's float32 pairwise summation --------------------------------------
// numpy/_core/src/umath/loops_utils.h.src, pairwise_sum: a run of n values
// sums as: n < 8, in order; n <= 128, eight strided partial sums r[0..7]
// combined as ((r0+r1)+(r2+r3))+((r4+r5)+(r6+r7)) and then the n % 8 tail in
// order; otherwise sum([0, n2)) + sum([n2, n)) with n2 = n/2 - (n/2) % 8.
// The reduction then adds that sum to its initial +0.0.
constexpr int kPwLeaf = 128;

__host__ __device__ inline int pw_left(int len) { return len / 2 - len / 2 % 8; }

float pw_host(const float* x, int len) {
  if (len < 8) {
    float r = 0.0f;
    for (int i = 0; i < len; ++i) r += x[i];
    return r;
  }
  if (len > kPwLeaf) {
    const int n2 = pw_left(len);
    return pw_host(x, n2) + pw_host(x + n2, len - n2);
  }
  float r[8];
  for (int k = 0; k < 8; ++k) r[k] = x[k];
  int i = 8;
  for (; i < len - len % 8; i += 8)
    for (int k = 0; k < 8; ++k) r[k] += x[i + k];
  float res = ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
  for (; i < len; ++i) res += x[i];
  return res;
}

// Depth of the deepest leaf (the right child is the longer one).
int pw_depth(int len) {
  int d = 0;
  for (; len > kPwLeaf; ++d) len -= pw_left(len);
  return d;
}

// The node at the end of a path of `bits` turns (the highest bit first; 1:
// right) from a node.  A path that goes on below a leaf is the leaf's when the
// rest of it turns left, else nothing's (len 0).
struct PwNode {
  int begin, len;
  __device__ PwNode down(int path, int bits) const {
    PwNode v = *this;
    for (int b = bits - 1; b >= 0; --b) {
      const bool right = (path >> b) & 1, leaf = v.len <= kPwLeaf;
      const int n2 = (int)((unsigned)v.len >> 1 & ~7u);  // pw_left
      v.begin += right && !leaf ? n2 : 0;
      v.len = leaf ? (right ? 0 : v.len) : right ? v.len - n2 : n2;
    }
    return v;
  }
};

// One step up the tree: a node without a right part is its left part.
__device__ __forceinline__ void pw_up(float& v, bool h, unsigned lanes, int o) {
  const float r = __shfl_down_sync(lanes, v, o);
  const int has = __shfl_down_sync(lanes, (int)h, o);
  if (has) v = __fadd_rn(v, r);
}

// A leaf's sum by eight lanes (`lane` of them, `group` their mask), one of its eight
// strided partial sums each; adding the partial sums by exchange is NumPy's order,
// since a rounded addition commutes.  get(i): value i.  All lanes of the group call it.
template <class Get>
__device__ __forceinline__ float pw_leaf(const PwNode& nd, int lane, unsigned group,
                                         const Get& get) {
  float r = 0.0f;
  if (nd.len >= 8) {
    // the lane's values and the leaf's tail, loaded before they are added
    const int rows = nd.len / 8, tail = nd.len % 8, lim = nd.begin + nd.len - tail;
    float v[kPwLeaf / 8], t[7];
#pragma unroll
    for (int i = 0; i < kPwLeaf / 8; ++i) v[i] = i < rows ? get(nd.begin + 8 * i + lane) : 0.0f;
#pragma unroll
    for (int i = 0; i < 7; ++i) t[i] = i < tail ? get(lim + i) : 0.0f;
    r = v[0];
#pragma unroll
    for (int i = 1; i < kPwLeaf / 8; ++i)
      if (i < rows) r = __fadd_rn(r, v[i]);
    r = __fadd_rn(r, __shfl_xor_sync(group, r, 1));
    r = __fadd_rn(r, __shfl_xor_sync(group, r, 2));
    r = __fadd_rn(r, __shfl_xor_sync(group, r, 4));
#pragma unroll
    for (int i = 0; i < 7; ++i)
      if (i < tail) r = __fadd_rn(r, t[i]);
  } else {
    for (int i = 0; i < nd.len; ++i) r = __fadd_rn(r, get(nd.begin + i));
  }
  return r;
}

// The sum of `count` (a power of two) paths' nodes at their common root: a warp
// for 32 of them at a time, in shared memory.
__device__ float pw_join(float* val, unsigned char* has, int count) {
  const int lane = threadIdx.x & 31;
  while (count > 1) {
    for (int i0 = 0; i0 < count; i0 += blockDim.x) {
      const int i = i0 + threadIdx.x;
      bool h = i < count && has[i];
      float v = h ? val[i] : 0.0f;
#pragma unroll
      for (int o = 1; o < 32; o *= 2) pw_up(v, h, kFull, o);
      __syncthreads();
      if (lane == 0 && i < count) {
        val[i / 32] = v;
        has[i / 32] = h;
      }
      __syncthreads();
    }
    count = (count + 31) / 32;
  }
  return val[0];
}

// Mean (mode 0) or population variance (mode 1, given the means; its root when
// `root`) of segments of `len` values that start every seg_stride values, as
// NumPy's mean / var store them.  Block (b, w) sums the 1 << lower paths below
// path b of the upper `upper` turns of segment w's tree, and the last of a
// segment's blocks joins their sums.
// What bounds it is latency: on 2.16 million samples a launch takes 13 us where
// a thread per leaf and a second launch for the inner nodes, level by level from
// tables in global memory, took 46.
constexpr int kPwThreads = 1024, kPwSlots = kPwThreads / 8;
__global__ void __launch_bounds__(kPwThreads)
pw_kernel(const float* __restrict__ x, long long seg_stride, int len, int n_seg, int mode,
          const float* __restrict__ centre, int upper, int lower, bool root,
          float* __restrict__ parts, int* __restrict__ tickets, float* __restrict__ out) {
  // a sum per warp and kPwSlots paths, or one per block; then their flags
  extern __shared__ float pw_val[];
  __shared__ PwNode nodes[kPwSlots];
  __shared__ bool last;
  const int slots = 1 << lower, blocks = 1 << upper;
  const int sums = max(slots / kPwSlots, 1) * (kPwThreads / 32);
  unsigned char* has = reinterpret_cast<unsigned char*>(pw_val + max(sums, blocks));
  const int tid = threadIdx.x, lane = tid & 7;
  const unsigned group = 0xFFu << (tid & 24);  // of the warp's lanes
  for (int w = blockIdx.y; w < n_seg; w += gridDim.y) {
    const float* base = x + (size_t)w * seg_stride;
    const float c = mode ? centre[w] : 0.0f;
    auto get = [&](int i) {
      const float v = base[i];
      if (!mode) return v;
      const float d = __fsub_rn(v, c);
      return __fmul_rn(d, d);
    };
    for (int s0 = 0; s0 < slots; s0 += kPwSlots) {
      if (tid < kPwSlots)
        nodes[tid] = s0 + tid < slots
                         ? PwNode{0, len}.down((int)(blockIdx.x << lower) + s0 + tid,
                                               upper + lower)
                         : PwNode{0, 0};
      __syncthreads();
      const PwNode nd = nodes[tid / 8];
      float r = pw_leaf(nd, lane, group, get);
      __syncwarp();
      const bool h = nd.len > 0;
      pw_up(r, h, kFull, 8);  // the warp's four leaves
      pw_up(r, h, kFull, 16);
      if ((tid & 31) == 0) {
        const int at = s0 / kPwSlots * (kPwThreads / 32) + tid / 32;
        pw_val[at] = r;
        has[at] = h;
      }
      __syncthreads();
    }
    float sum = pw_join(pw_val, has, sums);
    bool write = tid == 0;
    if (blocks > 1) {
      if (tid == 0) {
        parts[(size_t)w * blocks + blockIdx.x] = sum;
        __threadfence();
        last = atomicAdd(&tickets[w], 1) == blocks - 1;
      }
      __syncthreads();
      if (last) {
        __threadfence();
        for (int b = tid; b < blocks; b += kPwThreads) {
          pw_val[b] = __ldcg(parts + (size_t)w * blocks + b);
          has[b] = PwNode{0, len}.down(b, upper).len > 0;
        }
        __syncthreads();
        sum = pw_join(pw_val, has, blocks);
      }
      write = write && last;
    }
    if (write) {
      const float v = np_divide_count(__fadd_rn(0.0f, sum), len);
      out[w] = root ? __fsqrt_rn(v) : v;
    }
    __syncthreads();
  }
}

// The same for segments of at most 1 << kPwShort leaves: a block takes as many of them
// as its 64 groups of eight lanes have leaves for.  (With a block of pw_kernel for each,
// the threshold of 2.16 million samples over windows of 500 took 564 us and over windows
// of 7 took 22.4 ms; now 142 and 230, and 256 and 1,232 with a thread per leaf.)
constexpr int kPwShort = 6, kPwShortThreads = 8 << kPwShort;
__global__ void __launch_bounds__(kPwShortThreads)
pw_short_kernel(const float* __restrict__ x, long long seg_stride, int len, int n_seg, int mode,
                const float* __restrict__ centre, int depth, bool root,
                float* __restrict__ out) {
  __shared__ float val[kPwShortThreads / 32];
  __shared__ unsigned char has[kPwShortThreads / 32];
  const int tid = threadIdx.x, slot = tid / 8;
  const int each = 1 << (kPwShort - depth);  // segments of a block
  const int w = blockIdx.x * each + (slot >> depth);
  const bool live = w < n_seg;
  const float* base = x + (size_t)(live ? w : 0) * seg_stride;
  const float c = mode && live ? centre[w] : 0.0f;
  PwNode nd{0, live ? len : 0};
  if (live) nd = nd.down(slot & ((1 << depth) - 1), depth);
  float r = pw_leaf(nd, tid & 7, 0xFFu << (tid & 24), [&](int i) {
    const float v = base[i];
    if (!mode) return v;
    const float d = __fsub_rn(v, c);
    return __fmul_rn(d, d);
  });
  __syncwarp();
  const bool h = nd.len > 0;
  if (depth >= 1) pw_up(r, h, kFull, 8);  // the warp's four leaves
  if (depth >= 2) pw_up(r, h, kFull, 16);
  const int lane = tid & 31;
  bool write = (lane & ((8 << min(depth, 2)) - 1)) == 0;
  int mine = w;
  if (depth > 2) {  // then the warps
    if (lane == 0) {
      val[tid / 32] = r;
      has[tid / 32] = h;
    }
    __syncthreads();
    if (tid >= 32) return;
    const bool g = lane < kPwShortThreads / 32 && has[lane];
    r = g ? val[lane] : 0.0f;
    for (int o = 1; o < 1 << (depth - 2); o *= 2) pw_up(r, g, kFull, o);
    write = lane < kPwShortThreads / 32 && (lane & ((1 << (depth - 2)) - 1)) == 0;
    mine = blockIdx.x * each + (lane >> (depth - 2));
  }
  if (write && mine < n_seg) {
    const float v = np_divide_count(__fadd_rn(0.0f, r), len);
    out[mine] = root ? __fsqrt_rn(v) : v;
  }
}

// tickets: n_seg zeros, for this call alone.
int pw_mean(const float* x, long long seg_stride, int len, int n_seg, int mode,
            const float* centre, bool root, float* out, Scratch& sc, cudaStream_t st) {
  const int depth = pw_depth(len);
  if (depth <= kPwShort && n_seg > 1) {
    const int each = 1 << (kPwShort - depth);
    pw_short_kernel<<<(unsigned)(((long long)n_seg + each - 1) / each), kPwShortThreads, 0, st>>>(
        x, seg_stride, len, n_seg, mode, centre, depth, root, out);
    BP_LAUNCHED("pw_short_kernel");
    return BP_OK;
  }
  // 128 leaves per block, at most 256 blocks per segment, at most 4,096 leaves
  // per block: 2.16 million samples have 32,768
  const int lower = std::min(std::max(std::min(depth, 7), depth - 8), 12), upper = depth - lower;
  const size_t sums = std::max(std::max((1 << lower) / kPwSlots, 1) * (kPwThreads / 32), 1 << upper);
  const size_t smem = sums * (sizeof(float) + 1);
  float* parts = nullptr;
  int* tickets = nullptr;
  if (upper > 0) {
    BP_TRY(sc.get(&parts, (size_t)n_seg << upper));
    BP_TRY(sc.get(&tickets, n_seg));
    BP_CUDA(cudaMemsetAsync(tickets, 0, (size_t)n_seg * sizeof(int), st));
  }
  pw_kernel<<<dim3(1u << upper, (unsigned)std::min(n_seg, 65535)), kPwThreads, smem, st>>>(
      x, seg_stride, len, n_seg, mode, centre, upper, lower, root, parts, tickets, out);
  BP_LAUNCHED("pw_kernel");
  return BP_OK;
}

// ---- bit masks over the samples ------------------------------------------------
// One bit per sample and the number set per kMaskBlock samples.  A compaction
// then is a launch that sets the bits, one that scans the counts (a single
// block) and one that takes the set bits with their ranks.  (With flags and ranks
// as integers per sample, the compaction of 2.16 million samples moved 35 MB and
// took 35 us.)
constexpr int kMaskRows = 16, kMaskThreads = 256;
constexpr int kMaskBlock = kMaskThreads * kMaskRows;  // 32 samples per word, 16 words per warp

struct Mask {
  unsigned* bits;
  int* counts;  // per block; after scan_counts the set bits before it, and all of them
  int n_words, n_blocks;
};
int get_mask(Mask* m, int n, Scratch& sc) {
  m->n_words = (int)(((long long)n + 31) / 32);
  m->n_blocks = (int)(((long long)n + kMaskBlock - 1) / kMaskBlock);
  BP_TRY(sc.get(&m->bits, m->n_words));
  return sc.get(&m->counts, (size_t)m->n_blocks + 1);
}

// The block's bits and count: flag(i, v, r) for its samples, v their values in
// the thread's rows (loaded before any is looked at), v[r] the sample's.
template <class Flag>
__device__ void mask_set(const float* __restrict__ x, int n, const Mask& m, const Flag& flag) {
  __shared__ int total;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned base = (blockIdx.x * (kMaskThreads / 32) + warp) * 32u * kMaskRows;
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  float v[kMaskRows];
#pragma unroll
  for (int r = 0; r < kMaskRows; ++r) {
    const unsigned i = base + r * 32 + lane;
    v[r] = i < (unsigned)n ? x[i] : 0.0f;
  }
  unsigned word = 0;
#pragma unroll
  for (int r = 0; r < kMaskRows; ++r) {
    const unsigned i = base + r * 32 + lane;
    const bool f = flag(i, v, r);
    const unsigned b = __ballot_sync(kFull, i < (unsigned)n && f);
    if (lane == r) word = b;
  }
  const unsigned at = base / 32 + lane;
  if (lane < kMaskRows && at < (unsigned)m.n_words) m.bits[at] = word;
  const int c = __reduce_add_sync(kFull, __popc(word));
  if (lane == 0 && c) atomicAdd(&total, c);
  __syncthreads();
  if (threadIdx.x == 0) m.counts[blockIdx.x] = total;
}

// counts -> the counts before each block, and the total behind the last.
__global__ void __launch_bounds__(1024) scan_counts_kernel(int* __restrict__ counts, int n) {
  __shared__ int warp_sum[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int each = (n + 1023) / 1024;
  const int b = min(tid * each, n), e = min(b + each, n);
  int mine = 0;
  for (int i = b; i < e; ++i) mine += counts[i];
  int sum = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(kFull, sum, o);
    if (lane >= o) sum += v;
  }
  if (lane == 31) warp_sum[warp] = sum;
  __syncthreads();
  const int from = __reduce_add_sync(kFull, lane < warp ? warp_sum[lane] : 0);
  int run = from + sum - mine;
  for (int i = b; i < e; ++i) {
    const int c = counts[i];
    counts[i] = run;
    run += c;
  }
  if (tid == 1023) counts[n] = run;
}
int scan_counts(const Mask& m, cudaStream_t st) {
  scan_counts_kernel<<<1, 1024, 0, st>>>(m.counts, m.n_blocks);
  BP_LAUNCHED("scan_counts_kernel");
  return BP_OK;
}

// take(i, v, set, rank) for the block's samples: rank = set bits before i, v =
// load(i, set, rank), loaded for all of the thread's rows before any is taken.
template <class Load, class Take>
__device__ void mask_take(int n, const Mask& m, const Load& load, const Take& take) {
  __shared__ int warp_sum[kMaskThreads / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned low = (1u << lane) - 1u;
  const unsigned base = (blockIdx.x * (kMaskThreads / 32) + warp) * 32u * kMaskRows;
  const unsigned at = base / 32 + lane;
  const unsigned word = lane < kMaskRows && at < (unsigned)m.n_words ? m.bits[at] : 0u;
  int sum = __popc(word);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(kFull, sum, o);
    if (lane >= o) sum += u;
  }
  if (lane == 31) warp_sum[warp] = sum;
  __syncthreads();
  int from = m.counts[blockIdx.x] + sum - __popc(word);  // before the lane's word
#pragma unroll
  for (int u = 0; u < kMaskThreads / 32; ++u) from += u < warp ? warp_sum[u] : 0;
  float v[kMaskRows];
#pragma unroll
  for (int r = 0; r < kMaskRows; ++r) {
    const unsigned w = __shfl_sync(kFull, word, r);
    const int f = __shfl_sync(kFull, from, r);
    const unsigned i = base + r * 32 + lane;
    v[r] = i < (unsigned)n ? load((int)i, ((w >> lane) & 1u) != 0u, f + __popc(w & low)) : 0.0f;
  }
#pragma unroll
  for (int r = 0; r < kMaskRows; ++r) {
    const unsigned w = __shfl_sync(kFull, word, r);
    const int f = __shfl_sync(kFull, from, r);
    const unsigned i = base + r * 32 + lane;
    if (i < (unsigned)n) take((int)i, v[r], ((w >> lane) & 1u) != 0u, f + __popc(w & low));
  }
}

// ---- threshold kernels ---------------------------------------------------------
__global__ void __launch_bounds__(kMaskThreads)
zero_mask_kernel(const float* __restrict__ x, int n, Mask m) {
  mask_set(x, n, m, [](unsigned, const float (&v)[kMaskRows], int r) { return v[r] == 0.0f; });
}

// Non-zero samples, in order, into nz.
__global__ void __launch_bounds__(kMaskThreads)
gather_nonzero_kernel(const float* __restrict__ x, int n, Mask zeros, float* __restrict__ nz) {
  mask_take(
      n, zeros, [&](int i, bool, int) { return x[i]; },
      [&](int i, float v, bool zero, int rank) {
        if (!zero) nz[i - rank] = v;
      });
}

// SplitMix64 output function (Steele, Lea & Flood, OOPSLA 2014).
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// Standard normal draws: Box-Muller on two counter-based uniforms.
__global__ void normal_kernel(unsigned long long seed, int n, float* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t a = mix64(seed ^ mix64(2ull * (uint64_t)i));
  const uint64_t b = mix64(seed ^ mix64(2ull * (uint64_t)i + 1ull));
  const float u1 = ((float)(a >> 40) + 0.5f) * 0x1p-24f;  // (0, 1)
  const float u2 = (float)(b >> 40) * 0x1p-24f;           // [0, 1)
  out[i] = sqrtf(-2.0f * logf(u1)) * cospif(2.0f * u2);
}

// Zeros replaced by noise * deviation + centre (NumPy float32 multiply, add).
__global__ void __launch_bounds__(kMaskThreads)
fill_zeros_kernel(const float* __restrict__ x, int n, Mask zeros,
                  const float* __restrict__ noise, const float* __restrict__ centre0,
                  const float* __restrict__ dev0, float* __restrict__ out) {
  const float c = *centre0, d = *dev0;
  mask_take(
      n, zeros, [&](int i, bool zero, int rank) { return zero ? noise[rank] : x[i]; },
      [&](int i, float v, bool zero, int) {
        out[i] = zero ? __fadd_rn(__fmul_rn(v, d), c) : v;
      });
}

// NumPy's mean and deviation of nothing.
__global__ void no_stats_kernel(float* __restrict__ stats) {
  if (threadIdx.x < 2) stats[threadIdx.x] = __uint_as_float(0x7FC00000u);
}

// np.maximum on float32: NaN propagates, equal values give the second operand.
__device__ __forceinline__ float np_maximum(float a, float b) {
  return (a > b || isnan(a)) ? a : b;
}

// A window's threshold, centre + num_dev * deviation (rms: deviation =
// sqrt(variance)), and the maximum over its neighbours as the tutorial takes it:
// first with the window before, then of those with the window after.
struct WindowThreshold {
  const float *centre, *spread;
  int n_win, is_var;
  float num_dev;
  __device__ float at(int w) const {
    const float dev = is_var ? __fsqrt_rn(spread[w]) : spread[w];
    return __fadd_rn(centre[w], __fmul_rn(num_dev, dev));
  }
  __device__ float with_before(int w) const {
    return w >= 1 ? np_maximum(at(w - 1), at(w)) : at(w);
  }
  __device__ float with_both(int w) const {
    return w + 1 < n_win ? np_maximum(with_before(w), with_before(w + 1)) : with_before(w);
  }
};

// Per-sample threshold: windows' values at (half + j) / shift for the middle
// samples, the first / last middle value repeated at both ends.
__global__ void __launch_bounds__(256)
spread_threshold_kernel(WindowThreshold thr, int n, int window, int half, int shift,
                        float* __restrict__ out) {
  constexpr int U = 4;
  const unsigned i0 = blockIdx.x * 256u * U + threadIdx.x;
  const int n_mid = n - window;
  unsigned done = ~0u;
  float v = 0.0f;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const unsigned i = i0 + u * 256;
    if (i >= (unsigned)n) return;
    const int j = min(max((int)i - half, 0), n_mid - 1);
    const unsigned w = min((unsigned)(half + j) / (unsigned)shift, (unsigned)thr.n_win - 1u);
    if (w != done) v = thr.with_both((int)w);
    done = w;
    out[i] = v;
  }
}

// ---- peak kernels ----------------------------------------------------------
// Rising edges x[i-1] < x[i]: a peak at i when x[i+1] < x[i]; a plateau to
// measure when x[i+1] == x[i].
__global__ void __launch_bounds__(kMaskThreads)
local_max_kernel(const float* __restrict__ x, int n, Mask peaks, int* __restrict__ plateau,
                 int* __restrict__ n_plateau) {
  const int lane = threadIdx.x & 31;
  const unsigned base =
      (blockIdx.x * (kMaskThreads / 32) + (threadIdx.x >> 5)) * 32u * kMaskRows;
  // the samples before and after the warp's
  const float first = base >= 1 && base - 1 < (unsigned)n ? x[base - 1] : 0.0f;
  const unsigned end = base + 32 * kMaskRows;
  const float last = end < (unsigned)n ? x[end] : 0.0f;
  mask_set(x, n, peaks, [&](unsigned i, const float (&v)[kMaskRows], int r) {
    float before = __shfl_up_sync(kFull, v[r], 1), after = __shfl_down_sync(kFull, v[r], 1);
    const float row_before = r ? __shfl_sync(kFull, v[r ? r - 1 : 0], 31) : first;
    const float row_after =
        r + 1 < kMaskRows ? __shfl_sync(kFull, v[r + 1 < kMaskRows ? r + 1 : r], 0) : last;
    if (lane == 0) before = row_before;
    if (lane == 31) after = row_after;
    if (i < 1 || i >= (unsigned)n - 1 || !(before < v[r])) return false;
    if (after == v[r]) plateau[atomicAdd(n_plateau, 1)] = (int)i;
    return after < v[r];
  });
}

// A warp per plateau starting at i: its end j is the first index > i with
// x[j] != x[i], capped at n - 1; a peak at (i + j - 1) / 2 when x[j] < x[i].
__global__ void __launch_bounds__(256)
plateau_kernel(const float* __restrict__ x, int n, const int* __restrict__ plateau,
               const int* __restrict__ n_plateau, Mask peaks) {
  const int lane = threadIdx.x & 31, total = *n_plateau;
  const int warps = gridDim.x * (blockDim.x >> 5);
  for (int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < total; w += warps) {
    const int i = plateau[w];
    const float xi = x[i];
    for (long long base = (long long)i + 1;; base += 32) {
      const long long j = base + lane;
      const bool stop = j >= (long long)n - 1 || x[j] != xi;
      const unsigned b = __ballot_sync(kFull, stop);
      if (b) {
        long long e = base + __ffs(b) - 1;
        if (e > n - 1) e = n - 1;
        if (lane == 0 && x[e] < xi) {
          const int p = (int)((i + e - 1) / 2);
          atomicOr(&peaks.bits[p >> 5], 1u << (p & 31));
          atomicAdd(&peaks.counts[p / kMaskBlock], 1);
        }
        break;
      }
    }
  }
}

__global__ void __launch_bounds__(kMaskThreads)
positions_kernel(int n, Mask m, int* __restrict__ out) {
  mask_take(n, m, [](int, bool, int) { return 0.0f; }, [&](int i, float, bool set, int rank) {
    if (set) out[rank] = i;
  });
}

// SciPy's distance rule, one cooperative launch for all of its rounds.
struct Peak {
  int pos;
  float val;  // -infinity once it is dropped (a peak is above its neighbours)
};
struct Distance {
  const float* x;
  const int* pos;      // peaks, ascending
  const int* n_peaks;  // on the device
  int dist;
  const float* above;  // peaks that are not above it are left out of `out`; may be NULL
  Peak* peaks;
  int *list, *list2, *kept;  // per peak
  int* counters;             // 6
  Mask out;                  // the kept peaks
};

// A round: every undecided peak with no undecided one before it within the
// distance is kept, and then what is undecided within the distance of a kept one
// is dropped.  (Before it, in SciPy's order: higher, or as high and later -- a
// stable ascending sort read backwards.  No kept peak lies within the distance
// of an undecided one.)  A lane looks at the nearest kNear peaks on both sides of
// its own, which block sixteen peaks in seventeen; a warp then looks along for
// each that is left.
// What bounds it is the latency of the rounds: two grid barriers and a few
// dependent reads each.  On 2.16 million samples with 538,000 peaks it takes
// 86 us; a warp per peak, three launches and a read-back per round took 420.
constexpr int kNear = 8, kDistThreads = 1024;
__global__ void __launch_bounds__(kDistThreads) distance_kernel(Distance a) {
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  const int lane = threadIdx.x & 31;
  const int thread = blockIdx.x * blockDim.x + threadIdx.x, threads = gridDim.x * blockDim.x;
  const int warp = thread >> 5, warps = threads >> 5;
  const unsigned before_lane = (1u << lane) - 1u;
  const int m = *a.n_peaks;
  for (int j = thread; j < m; j += threads) a.peaks[j] = Peak{a.pos[j], a.x[a.pos[j]]};
  for (int w = thread; w < a.out.n_words; w += threads) a.out.bits[w] = 0u;
  for (int b = thread; b < a.out.n_blocks; b += threads) a.out.counts[b] = 0;
  if (thread < 6) a.counters[thread] = 0;
  grid.sync();
  // The peak, or where there is none one that is too far and blocks nothing.
  auto peak = [&](int k) {
    if (k < 0 || k >= m) return make_int2(k < 0 ? INT_MIN : INT_MAX, 0xFF800000);
    return *reinterpret_cast<const int2*>(a.peaks + k);
  };
  // A peak's window is lo < position < hi; no end lies beyond those of peak().
  auto window_lo = [&](int p) { return (int)max((long long)p - a.dist, (long long)INT_MIN); };
  auto window_hi = [&](int p) { return (int)min((long long)p + a.dist, (long long)INT_MAX); };
  int u = m;
  int *list = nullptr, *next = a.list, *spare = a.list2;
  for (int round = 0; u > 0 && round <= m; ++round) {
    int* n_kept = a.counters + round % 3;
    int* n_next = a.counters + 3 + round % 3;
    for (int t = warp; t < (u + 31) / 32; t += warps) {
      const int i = t * 32 + lane;
      const int j = i >= u ? -1 : list ? list[i] : i;
      const int2 mine = peak(j);
      const float vj = __int_as_float(mine.y);
      const bool open = vj > __int_as_float(0xFF800000);
      const int lo = window_lo(mine.x), hi = window_hi(mine.x);
      bool blocked = false, left = false, right = false;
      if (open) {
        int2 l[kNear], r[kNear];
#pragma unroll
        for (int d = 0; d < kNear; ++d) {
          l[d] = peak(j - 1 - d);
          r[d] = j < m - 1 - d ? peak(j + 1 + d) : make_int2(INT_MAX, 0xFF800000);
        }
#pragma unroll
        for (int d = 0; d < kNear; ++d) {
          blocked |= l[d].x > lo && __int_as_float(l[d].y) > vj;
          blocked |= r[d].x < hi && __int_as_float(r[d].y) >= vj;
        }
        left = !blocked && l[kNear - 1].x > lo;
        right = !blocked && r[kNear - 1].x < hi;
      }
      unsigned rest = __ballot_sync(kFull, left || right);
      while (rest) {
        const int src = __ffs(rest) - 1;
        rest &= rest - 1;
        const int jj = __shfl_sync(kFull, j, src);
        const float vv = __shfl_sync(kFull, vj, src);
        const int ll = __shfl_sync(kFull, lo, src), hh = __shfl_sync(kFull, hi, src);
        bool go_l = __shfl_sync(kFull, (int)left, src) != 0;
        bool go_r = __shfl_sync(kFull, (int)right, src) != 0;
        bool hit = false;
        for (int d = kNear + 1 + lane; (go_l || go_r) && !hit; d += 32) {
          const int2 l = go_l && d <= jj ? peak(jj - d) : make_int2(INT_MIN, 0xFF800000);
          const int2 r = go_r && d < m - jj ? peak(jj + d) : make_int2(INT_MAX, 0xFF800000);
          hit = __any_sync(kFull, (l.x > ll && __int_as_float(l.y) > vv) ||
                                      (r.x < hh && __int_as_float(r.y) >= vv));
          go_l = __all_sync(kFull, l.x > ll);
          go_r = __all_sync(kFull, r.x < hh);
        }
        if (lane == src) blocked = hit;
      }
      const unsigned keep = __ballot_sync(kFull, open && !blocked);
      const unsigned stay = __ballot_sync(kFull, open && blocked);
      int k0 = 0, s0 = 0;
      if (lane == 0) {
        if (keep) k0 = atomicAdd(n_kept, __popc(keep));
        if (stay) s0 = atomicAdd(n_next, __popc(stay));
      }
      k0 = __shfl_sync(kFull, k0, 0);
      s0 = __shfl_sync(kFull, s0, 0);
      if (open && !blocked) a.kept[k0 + __popc(keep & before_lane)] = j;
      if (open && blocked) next[s0 + __popc(stay & before_lane)] = j;
    }
    grid.sync();
    const int nk = *(volatile int*)n_kept;
    for (int t = warp; t < nk; t += warps) {
      const int j = a.kept[t], pj = a.peaks[j].pos;
      const int lo = window_lo(pj), hi = window_hi(pj);
      if (lane == 0 && (!a.above || a.x[pj] > a.above[pj])) {
        atomicOr(&a.out.bits[pj >> 5], 1u << (pj & 31));
        atomicAdd(&a.out.counts[pj / kMaskBlock], 1);
      }
      bool go_l = true, go_r = true;
      for (int d = 1 + lane; go_l || go_r; d += 32) {
        const bool l = go_l && d <= j && a.peaks[j - d].pos > lo;
        const bool r = go_r && d < m - j && a.peaks[j + d].pos < hi;
        if (l) a.peaks[j - d].val = __int_as_float(0xFF800000);
        if (r) a.peaks[j + d].val = __int_as_float(0xFF800000);
        go_l = __all_sync(kFull, l);
        go_r = __all_sync(kFull, r);
      }
    }
    // the counters of the next round: last read a round ago
    if (thread < 2) a.counters[3 * thread + (round + 1) % 3] = 0;
    grid.sync();
    u = *(volatile int*)n_next;
    list = next;
    next = spare;
    spare = list;
  }
}

__global__ void above_flags_kernel(const float* __restrict__ x, const float* __restrict__ thr,
                                   const int* __restrict__ peaks, int m, int* __restrict__ flags) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j > m) return;
  flags[j] = (j < m && x[peaks[j]] > thr[peaks[j]]) ? 1 : 0;
}

__global__ void scatter_detections_kernel(const int* __restrict__ flags,
                                          const int* __restrict__ rank,
                                          const int* __restrict__ peaks, int m,
                                          const float* __restrict__ x,
                                          const int32_t* __restrict__ argmax,
                                          int32_t* __restrict__ out_peaks,
                                          float* __restrict__ out_heights,
                                          int32_t* __restrict__ out_sources) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m || !flags[j]) return;
  const int r = rank[j], p = peaks[j];
  out_peaks[r] = p;
  if (out_heights) out_heights[r] = x[p];
  if (argmax && out_sources) out_sources[r] = argmax[p];
}

__global__ void __launch_bounds__(kMaskThreads)
mask_detections_kernel(int n, Mask m, const float* __restrict__ x,
                       const int32_t* __restrict__ argmax, int32_t* __restrict__ out_peaks,
                       float* __restrict__ out_heights, int32_t* __restrict__ out_sources) {
  mask_take(n, m, [](int, bool, int) { return 0.0f; }, [&](int i, float, bool set, int r) {
    if (!set) return;
    out_peaks[r] = i;
    if (out_heights) out_heights[r] = x[i];
    if (argmax && out_sources) out_sources[r] = argmax[i];
  });
}

// ---- host drivers -------------------------------------------------------------
// Peaks of x into d_peaks (device, ascending); their number into *m_out.
// ---- height and prominence conditions (SciPy's find_peaks options) ----------
// lo <= v_lo and v_hi <= hi in float64; a NaN scalar border is an open side,
// a per-sample border array (float64, read at the peak) compares as SciPy
// does (NaN fails).
__device__ __forceinline__ bool within(double v_lo, double v_hi, double lo, double hi,
                                       const double* lo_arr, const double* hi_arr, int p) {
  bool ok = true;
  if (lo_arr) ok = ok && (lo_arr[p] <= v_lo);
  else if (!isnan(lo)) ok = ok && (lo <= v_lo);
  if (hi_arr) ok = ok && (v_hi <= hi_arr[p]);
  else if (!isnan(hi)) ok = ok && (v_hi <= hi);
  return ok;
}

// SciPy's threshold condition: the peak's rise over each neighbour (float64),
// the smaller rise against the lower border, the larger against the upper.
// A peak's neighbours exist and are never NaN (both are below the peak).
__global__ void threshold_flags_kernel(const float* __restrict__ x, const int* __restrict__ pos,
                                       int m, double lo, double hi,
                                       const double* __restrict__ lo_arr,
                                       const double* __restrict__ hi_arr,
                                       int* __restrict__ flags) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j > m) return;
  int keep = 0;
  if (j < m) {
    const int p = pos[j];
    const double left = (double)x[p] - (double)x[p - 1];
    const double right = (double)x[p] - (double)x[p + 1];
    keep = within(fmin(left, right), fmax(left, right), lo, hi, lo_arr, hi_arr, p) ? 1 : 0;
  }
  flags[j] = keep;
}

__global__ void height_flags_kernel(const float* __restrict__ x, const int* __restrict__ pos,
                                    int m, double lo, double hi, const double* __restrict__ lo_arr,
                                    const double* __restrict__ hi_arr, int* __restrict__ flags) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j > m) return;
  int keep = 0;
  if (j < m) {
    const double v = (double)x[pos[j]];
    keep = within(v, v, lo, hi, lo_arr, hi_arr, pos[j]) ? 1 : 0;
  }
  flags[j] = keep;
}

// One warp per peak: from the peak, walk outwards while the signal is not
// above it (NaN stops the walk), at most `half` samples when half >= 0; the
// base of each side is its lowest sample (the one nearest the peak among
// equals), the prominence the peak minus the higher base, in float64.
__global__ void prominence_kernel(const float* __restrict__ x, int n, const int* __restrict__ pos,
                                  int m, long long half, double* __restrict__ prom,
                                  int* __restrict__ lbase, int* __restrict__ rbase) {
  const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= m) return;
  const int p = pos[gw];
  const float xp = x[p];
  const long long lo_end = half >= 0 ? max(0LL, (long long)p - half) : 0LL;
  const long long hi_end = half >= 0 ? min((long long)n - 1, (long long)p + half)
                                     : (long long)n - 1;
  float side_min[2];
  int side_base[2];
  for (int dir = 0; dir < 2; ++dir) {  // 0: left, 1: right
    float best = xp;
    int best_i = p;
    for (long long base = p;; base += dir ? 32 : -32) {
      const long long i = dir ? base + lane : base - lane;
      const bool inside = dir ? i <= hi_end : i >= lo_end;
      const float v = inside ? x[i] : 0.0f;
      const bool walk = inside && v <= xp;  // false past the window, above the peak, NaN
      const unsigned stop = __ballot_sync(kFull, !walk);
      const int n_walk = stop ? __ffs(stop) - 1 : 32;  // lanes before the first stop
      // lowest value among the walked lanes, nearest the peak among equals
      float cv = lane < n_walk ? v : INFINITY;
      int ci = lane < n_walk ? (int)i : INT_MAX;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(kFull, cv, o);
        const int oi = __shfl_xor_sync(kFull, ci, o);
        const bool nearer = dir ? oi < ci : (oi != INT_MAX && (ci == INT_MAX || oi > ci));
        if (ov < cv || (ov == cv && nearer)) {
          cv = ov;
          ci = oi;
        }
      }
      if (n_walk > 0 && cv < best) {  // a strictly lower sample further out
        best = cv;
        best_i = ci;
      }
      if (stop) break;
    }
    side_min[dir] = best;
    side_base[dir] = best_i;
  }
  if (lane == 0) {
    prom[gw] = (double)xp - (double)fmaxf(side_min[0], side_min[1]);
    lbase[gw] = side_base[0];
    rbase[gw] = side_base[1];
  }
}

__global__ void prominence_flags_kernel(const double* __restrict__ prom,
                                        const int* __restrict__ pos, int m, double lo, double hi,
                                        const double* __restrict__ lo_arr,
                                        const double* __restrict__ hi_arr,
                                        int* __restrict__ flags) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j > m) return;
  flags[j] = (j < m && within(prom[j], prom[j], lo, hi, lo_arr, hi_arr, pos[j])) ? 1 : 0;
}

__global__ void compact_peaks_kernel(const int* __restrict__ flags, const int* __restrict__ rank,
                                     int m, const int* __restrict__ pos,
                                     const double* __restrict__ prom, const int* __restrict__ lb,
                                     const int* __restrict__ rb, int* __restrict__ out_pos,
                                     double* __restrict__ out_prom, int* __restrict__ out_lb,
                                     int* __restrict__ out_rb) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m || !flags[j]) return;
  const int r = rank[j];
  out_pos[r] = pos[j];
  if (out_prom) out_prom[r] = prom[j];
  if (out_lb) out_lb[r] = lb[j];
  if (out_rb) out_rb[r] = rb[j];
}

// ---- host driver of the peak finder -----------------------------------------
struct PeakOut {
  int32_t* peaks;
  double* prominences;  // may be NULL
  int32_t* left_bases;  // may be NULL
  int32_t* right_bases; // may be NULL
};

// Keeps the entries of `pos` (m, device) whose flag is set, in order, into a
// new scratch array; returns their number
// and where it is on the device.
int keep_flagged(int* flags, int m, int** pos, Scratch& sc, cudaStream_t st, int* kept,
                 const int** d_kept) {
  int* rank = nullptr;
  int* out = nullptr;
  BP_TRY(sc.get(&rank, (size_t)m + 1));
  BP_TRY(scan_flags(flags, rank, m, sc, st));
  *d_kept = rank + m;
  BP_TRY(read_back(kept, rank + m, st));
  BP_TRY(sc.get(&out, std::max(*kept, 1)));
  compact_peaks_kernel<<<grid_for(m, 256), 256, 0, st>>>(flags, rank, m, *pos, nullptr, nullptr,
                                                         nullptr, out, nullptr, nullptr,
                                                         nullptr);
  BP_LAUNCHED("compact_peaks_kernel");
  *pos = out;
  return BP_OK;
}

// Local maxima of x (plateaus by their midpoint) as a mask with scanned counts.
int local_maxima(const float* x, int n, Mask* peaks, Scratch& sc, cudaStream_t st) {
  int *plateau = nullptr, *n_plateau = nullptr;
  BP_TRY(get_mask(peaks, n, sc));
  BP_TRY(sc.get(&plateau, (size_t)n / 2 + 1));  // a rising edge and an equal sample each
  BP_TRY(sc.get(&n_plateau, 1));
  BP_CUDA(cudaMemsetAsync(n_plateau, 0, sizeof(int), st));
  local_max_kernel<<<(unsigned)peaks->n_blocks, kMaskThreads, 0, st>>>(x, n, *peaks, plateau,
                                                                      n_plateau);
  BP_LAUNCHED("local_max_kernel");
  plateau_kernel<<<(unsigned)std::min(peaks->n_blocks, 148), 256, 0, st>>>(x, n, plateau,
                                                                           n_plateau, *peaks);
  BP_LAUNCHED("plateau_kernel");
  return scan_counts(*peaks, st);
}

// SMs that the blocks of a launch on `st` can have: the device's, or fewer where the
// stream or the current context has a share of them (a green context).
int stream_sms(cudaStream_t st, int* sms) {
  using GetStream = CUresult (*)(CUstream, CUgreenCtx*);
  using GetGreen = CUresult (*)(CUgreenCtx, CUdevResource*, CUdevResourceType);
  using GetCtx = CUresult (*)(CUcontext, CUdevResource*, CUdevResourceType);
  using Current = CUresult (*)(CUcontext*);
  // the driver's calls by name: the library does not link against it
  static const auto entry = [](const char* name) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion(name, &f, 12040, cudaEnableDefault, &q) != cudaSuccess) {
      cudaGetLastError();
      return (void*)nullptr;
    }
    return q == cudaDriverEntryPointSuccess ? f : nullptr;
  };
  static const auto stream_green = (GetStream)entry("cuStreamGetGreenCtx");
  static const auto green_share = (GetGreen)entry("cuGreenCtxGetDevResource");
  static const auto current = (Current)entry("cuCtxGetCurrent");
  static const auto ctx_share = (GetCtx)entry("cuCtxGetDevResource");
  int dev = 0;
  BP_CUDA(cudaGetDevice(&dev));
  BP_CUDA(cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev));
  CUdevResource r{};
  CUgreenCtx green = nullptr;
  CUcontext ctx = nullptr;
  if (stream_green && green_share && stream_green(st, &green) == CUDA_SUCCESS && green) {
    if (green_share(green, &r, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS)
      *sms = std::min(*sms, (int)r.sm.smCount);
  } else if (current && ctx_share && current(&ctx) == CUDA_SUCCESS && ctx) {
    if (ctx_share(ctx, &r, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS)
      *sms = std::min(*sms, (int)r.sm.smCount);
  }
  *sms = std::max(*sms, 1);
  return BP_OK;
}

// The distance rule on the peaks pos[0 .. *d_m - 1] (at most `cap`, on the
// device): the kept ones as a mask with scanned counts.
int distance_rule(const float* x, int n, const int* pos, const int* d_m, int cap, double distance,
                  const float* above, Mask* out, Scratch& sc, cudaStream_t st) {
  const double dc = std::ceil(distance);
  Distance a{};
  a.x = x;
  a.pos = pos;
  a.n_peaks = d_m;
  a.dist = dc > (double)n ? n + 1 : (int)dc;
  a.above = above;
  BP_TRY(sc.get(&a.peaks, cap));
  BP_TRY(sc.get(&a.list, cap));
  BP_TRY(sc.get(&a.list2, cap));
  BP_TRY(sc.get(&a.kept, cap));
  BP_TRY(sc.get(&a.counters, 6));
  BP_TRY(get_mask(&a.out, n, sc));
  // One block per SM: they are resident together, and a barrier of few blocks is the
  // quicker one.  Fewer blocks do the same work, so where some limit that was not
  // asked for (a share of the SMs held another way) refuses them, fewer are tried.
  int sms = 0;
  BP_TRY(stream_sms(st, &sms));
  unsigned grid = grid_for(cap, kDistThreads, sms);
  void* args[] = {&a};
  cudaError_t e = cudaSuccess;
  while (true) {
    e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(distance_kernel), dim3(grid),
                                    dim3(kDistThreads), args, 0, st);
    if (e != cudaErrorCooperativeLaunchTooLarge || grid == 1) break;
    cudaGetLastError();
    grid /= 2;
  }
  if (e != cudaSuccess) return cuda_fail(e, "launch distance_kernel");
  BP_LAUNCHED("distance_kernel");
  *out = a.out;
  return scan_counts(*out, st);
}

// Peaks of x in SciPy's order of conditions: local maxima (plateaus by their
// midpoint), height, threshold, distance, prominence.  Writes `*m_out` entries
// of `out`.
int find_peaks_impl(const float* x, int n, const bp_peak_options& o, const PeakOut& out,
                    int* m_out, Scratch& sc, cudaStream_t st) {
  *m_out = 0;
  if (n < 3) return BP_OK;
  Mask peaks{};
  int *pos = nullptr, *flags = nullptr;
  BP_TRY(local_maxima(x, n, &peaks, sc, st));
  int cap = n / 2 + 1;  // peaks, at most
  const int* d_m = peaks.counts + peaks.n_blocks;
  BP_TRY(sc.get(&pos, cap));
  positions_kernel<<<(unsigned)peaks.n_blocks, kMaskThreads, 0, st>>>(n, peaks, pos);
  BP_LAUNCHED("positions_kernel");
  int m = -1;  // not read back yet
  if (o.use_height || o.use_threshold || o.use_prominence) {
    BP_TRY(read_back(&m, d_m, st));
    BP_TRY(sc.get(&flags, (size_t)m + 1));
    cap = std::max(m, 1);
  }
  // height
  if (o.use_height && m > 0) {
    height_flags_kernel<<<grid_for((long long)m + 1, 256), 256, 0, st>>>(
        x, pos, m, o.height_min, o.height_max, o.d_height_min, o.d_height_max, flags);
    BP_LAUNCHED("height_flags_kernel");
    BP_TRY(keep_flagged(flags, m, &pos, sc, st, &m, &d_m));
  }
  // threshold
  if (o.use_threshold && m > 0) {
    threshold_flags_kernel<<<grid_for((long long)m + 1, 256), 256, 0, st>>>(
        x, pos, m, o.threshold_min, o.threshold_max, o.d_threshold_min, o.d_threshold_max,
        flags);
    BP_LAUNCHED("threshold_flags_kernel");
    BP_TRY(keep_flagged(flags, m, &pos, sc, st, &m, &d_m));
  }
  // greedy distance rule
  if (o.distance > 0.0 && m != 0) {
    Mask kept{};
    BP_TRY(distance_rule(x, n, pos, d_m, cap, o.distance, nullptr, &kept, sc, st));
    d_m = kept.counts + kept.n_blocks;
    positions_kernel<<<(unsigned)kept.n_blocks, kMaskThreads, 0, st>>>(n, kept, pos);
    BP_LAUNCHED("positions_kernel");
    m = -1;
  }
  if (m < 0) BP_TRY(read_back(&m, d_m, st));
  // prominence
  if (o.use_prominence && m > 0) {
    double* prom = nullptr;
    int *lb = nullptr, *rb = nullptr;
    BP_TRY(sc.get(&prom, m));
    BP_TRY(sc.get(&lb, m));
    BP_TRY(sc.get(&rb, m));
    const long long half = o.wlen > 1.0 ? (long long)std::ceil(o.wlen) / 2 : -1;
    prominence_kernel<<<grid_for((long long)m * 32, 256), 256, 0, st>>>(x, n, pos, m, half,
                                                                        prom, lb, rb);
    BP_LAUNCHED("prominence_kernel");
    prominence_flags_kernel<<<grid_for((long long)m + 1, 256), 256, 0, st>>>(
        prom, pos, m, o.prominence_min, o.prominence_max, o.d_prominence_min,
        o.d_prominence_max, flags);
    BP_LAUNCHED("prominence_flags_kernel");
    int* prank = nullptr;
    BP_TRY(sc.get(&prank, (size_t)m + 1));
    BP_TRY(scan_flags(flags, prank, m, sc, st));
    int k = 0;
    BP_TRY(read_back(&k, prank + m, st));
    compact_peaks_kernel<<<grid_for(m, 256), 256, 0, st>>>(flags, prank, m, pos, prom, lb, rb,
                                                           out.peaks, out.prominences,
                                                           out.left_bases, out.right_bases);
    BP_LAUNCHED("compact_peaks_kernel");
    *m_out = k;
    return BP_OK;
  }
  if (m > 0)
    BP_CUDA(cudaMemcpyAsync(out.peaks, pos, (size_t)m * sizeof(int32_t),
                            cudaMemcpyDeviceToDevice, st));
  *m_out = m;
  return BP_OK;
}

bp_peak_options distance_only(double distance) {
  bp_peak_options o{};
  o.distance = distance;
  o.height_min = o.height_max = NAN;
  o.threshold_min = o.threshold_max = NAN;
  o.prominence_min = o.prominence_max = NAN;
  return o;
}

int check_series(const void* p, size_t n, const char* what) {
  if (!p && n) return fail(BP_ERR_INVALID_ARGUMENT, "%s is NULL", what);
  if (n > (size_t)INT_MAX - 1) return fail(BP_ERR_UNSUPPORTED, "%s longer than 2^31 - 2", what);
  return BP_OK;
}

}  // namespace

extern "C" {

float bp_pairwise_sum_f32(const float* x, size_t n) {
  if (n == 0 || !x || n > (size_t)INT_MAX) return 0.0f;
  return 0.0f + pw_host(x, (int)n);
}

int bp_threshold_dev(const float* d_series, size_t n_samples, size_t sliding_window,
                     double overlap, int kind, float num_dev, const float* d_white_noise,
                     size_t n_white_noise, unsigned long long seed, float* d_threshold,
                     void* stream) {
  BP_NVTX("bp_threshold_dev");
  BP_TRY(check_series(d_series, n_samples, "series"));
  if (!d_threshold) return fail(BP_ERR_INVALID_ARGUMENT, "threshold output is NULL");
  if (kind != BP_THRESHOLD_RMS && kind != BP_THRESHOLD_MAD)
    return fail(BP_ERR_INVALID_ARGUMENT, "threshold kind must be rms (0) or mad (1)");
  if (sliding_window < 1 || n_samples <= sliding_window)
    return fail(BP_ERR_INVALID_ARGUMENT,
                "the series (%zu samples) must be longer than the sliding window (%zu)",
                n_samples, sliding_window);
  const double step = (1.0 - overlap) * (double)sliding_window;
  if (!(step >= 1.0) || step > (double)INT_MAX)
    return fail(BP_ERR_INVALID_ARGUMENT, "(1 - overlap) * sliding_window must be in [1, 2^31)");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int n = (int)n_samples, W = (int)sliding_window, half = W / 2;
  const int shift = (int)step;  // int() truncation, as in the notebook
  const int n_win = (n - W) / shift + 1;
  Scratch sc(st);
  Mask zeros{};
  float* stats0 = nullptr;
  BP_TRY(get_mask(&zeros, n, sc));
  BP_TRY(sc.get(&stats0, 2));  // default centre, deviation
  zero_mask_kernel<<<(unsigned)zeros.n_blocks, kMaskThreads, 0, st>>>(d_series, n, zeros);
  BP_LAUNCHED("zero_mask_kernel");
  BP_TRY(scan_counts(zeros, st));
  int n_zeros = 0;
  BP_TRY(read_back(&n_zeros, zeros.counts + zeros.n_blocks, st));
  if (d_white_noise && n_white_noise < (size_t)n_zeros)
    return fail(BP_ERR_INVALID_ARGUMENT, "white noise holds %zu values for %d zero samples",
                n_white_noise, n_zeros);
  const int m = n - n_zeros;
  // without a zero the series is its own non-zero samples, and stays as it is
  const float *nz = d_series, *filled = d_series;
  float *nz_mem = nullptr, *filled_mem = nullptr;
  if (n_zeros > 0) {
    BP_TRY(sc.get(&nz_mem, n));
    BP_TRY(sc.get(&filled_mem, n));
    gather_nonzero_kernel<<<(unsigned)zeros.n_blocks, kMaskThreads, 0, st>>>(d_series, n, zeros,
                                                                             nz_mem);
    BP_LAUNCHED("gather_nonzero_kernel");
    nz = nz_mem;
    filled = filled_mem;
  }
  // centre and deviation of the non-zero samples (NaN when there are none)
  if (kind == BP_THRESHOLD_RMS) {
    if (n_zeros == 0) {
      // nothing to fill
    } else if (m > 0) {
      BP_TRY(pw_mean(nz, 0, m, 1, 0, nullptr, false, stats0, sc, st));
      BP_TRY(pw_mean(nz, 0, m, 1, 1, stats0, true, stats0 + 1, sc, st));
    } else {
      no_stats_kernel<<<1, 32, 0, st>>>(stats0);
      BP_LAUNCHED("no_stats_kernel");
    }
  } else if (n_zeros > 0) {
    BP_TRY(np_median(nz, 0, m, 1, 0, nullptr, stats0, sc, st));
    BP_TRY(np_median(nz, 0, m, 1, 1, stats0, stats0 + 1, sc, st));
  }
  const float* noise = d_white_noise;
  if (n_zeros > 0 && !noise) {
    float* gen = nullptr;
    BP_TRY(sc.get(&gen, n_zeros));
    normal_kernel<<<grid_for(n_zeros, 256), 256, 0, st>>>(seed, n_zeros, gen);
    BP_LAUNCHED("normal_kernel");
    noise = gen;
  }
  if (n_zeros > 0) {
    fill_zeros_kernel<<<(unsigned)zeros.n_blocks, kMaskThreads, 0, st>>>(
        d_series, n, zeros, noise, stats0, stats0 + 1, filled_mem);
    BP_LAUNCHED("fill_zeros_kernel");
  }
  // per-window centre and spread
  float *centre = nullptr, *spread = nullptr;
  BP_TRY(sc.get(&centre, n_win));
  BP_TRY(sc.get(&spread, n_win));
  if (kind == BP_THRESHOLD_RMS) {
    BP_TRY(pw_mean(filled, shift, W, n_win, 0, nullptr, false, centre, sc, st));
    BP_TRY(pw_mean(filled, shift, W, n_win, 1, centre, false, spread, sc, st));
  } else {
    BP_TRY(np_median(filled, shift, W, n_win, 0, nullptr, centre, sc, st));
    BP_TRY(np_median(filled, shift, W, n_win, 1, centre, spread, sc, st));
  }
  const WindowThreshold thr{centre, spread, n_win, kind == BP_THRESHOLD_RMS ? 1 : 0, num_dev};
  spread_threshold_kernel<<<grid_for(n, 1024), 256, 0, st>>>(thr, n, W, half, shift,
                                                             d_threshold);
  BP_LAUNCHED("spread_threshold_kernel");
  return BP_OK;
}

int bp_find_peaks_dev(const float* d_x, size_t n_samples, double distance, int32_t* d_peaks,
                      size_t capacity, size_t* n_peaks, void* stream) {
  BP_NVTX("bp_find_peaks_dev");
  BP_TRY(check_series(d_x, n_samples, "series"));
  if (!n_peaks) return fail(BP_ERR_INVALID_ARGUMENT, "n_peaks is NULL");
  *n_peaks = 0;
  if (distance > 0.0 && distance < 1.0)
    return fail(BP_ERR_INVALID_ARGUMENT, "distance must be greater or equal to 1");
  if (capacity < n_samples / 2 || (!d_peaks && n_samples >= 3))
    return fail(BP_ERR_INVALID_ARGUMENT, "peak capacity must be at least n_samples / 2");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  Scratch sc(st);
  int m = 0;
  BP_TRY(find_peaks_impl(d_x, (int)n_samples, distance_only(distance),
                         PeakOut{d_peaks, nullptr, nullptr, nullptr}, &m, sc, st));
  BP_CUDA(cudaStreamSynchronize(st));
  *n_peaks = (size_t)m;
  return BP_OK;
}

int bp_find_peaks_opt_dev(const float* d_x, size_t n_samples, const bp_peak_options* opt,
                          int32_t* d_peaks, double* d_prominences, int32_t* d_left_bases,
                          int32_t* d_right_bases, size_t capacity, size_t* n_peaks,
                          void* stream) {
  BP_NVTX("bp_find_peaks_opt_dev");
  BP_TRY(check_series(d_x, n_samples, "series"));
  if (!n_peaks || !opt) return fail(BP_ERR_INVALID_ARGUMENT, "n_peaks / options is NULL");
  *n_peaks = 0;
  if (opt->distance > 0.0 && opt->distance < 1.0)
    return fail(BP_ERR_INVALID_ARGUMENT, "distance must be greater or equal to 1");
  if (opt->use_prominence && opt->wlen > 0.0 && std::ceil(opt->wlen) <= 1.0)
    return fail(BP_ERR_INVALID_ARGUMENT, "wlen must be larger than 1");
  if (capacity < n_samples / 2 || (!d_peaks && n_samples >= 3))
    return fail(BP_ERR_INVALID_ARGUMENT, "peak capacity must be at least n_samples / 2");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  Scratch sc(st);
  int m = 0;
  BP_TRY(find_peaks_impl(d_x, (int)n_samples, *opt,
                         PeakOut{d_peaks, d_prominences, d_left_bases, d_right_bases}, &m, sc,
                         st));
  BP_CUDA(cudaStreamSynchronize(st));
  *n_peaks = (size_t)m;
  return BP_OK;
}

int bp_detect_dev(const float* d_beam_max, const int32_t* d_argmax, const float* d_threshold,
                  size_t n_samples, double distance, int32_t* d_peaks, float* d_heights,
                  int32_t* d_sources, size_t capacity, size_t* n_detections, void* stream) {
  BP_NVTX("bp_detect_dev");
  BP_TRY(check_series(d_beam_max, n_samples, "beam_max"));
  BP_TRY(check_series(d_threshold, n_samples, "threshold"));
  if (!n_detections) return fail(BP_ERR_INVALID_ARGUMENT, "n_detections is NULL");
  *n_detections = 0;
  if (distance > 0.0 && distance < 1.0)
    return fail(BP_ERR_INVALID_ARGUMENT, "distance must be greater or equal to 1");
  if (capacity < n_samples / 2 || (!d_peaks && n_samples >= 3))
    return fail(BP_ERR_INVALID_ARGUMENT, "detection capacity must be at least n_samples / 2");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  Scratch sc(st);
  const int n = (int)n_samples;
  if (n < 3) return BP_OK;
  if (distance > 0.0) {
    Mask peaks{}, kept{};
    int *pos = nullptr, k = 0;
    BP_TRY(local_maxima(d_beam_max, n, &peaks, sc, st));
    BP_TRY(sc.get(&pos, (size_t)n / 2 + 1));
    positions_kernel<<<(unsigned)peaks.n_blocks, kMaskThreads, 0, st>>>(n, peaks, pos);
    BP_LAUNCHED("positions_kernel");
    BP_TRY(distance_rule(d_beam_max, n, pos, peaks.counts + peaks.n_blocks, n / 2 + 1, distance,
                         d_threshold, &kept, sc, st));
    mask_detections_kernel<<<(unsigned)kept.n_blocks, kMaskThreads, 0, st>>>(
        n, kept, d_beam_max, d_argmax, d_peaks, d_heights, d_sources);
    BP_LAUNCHED("mask_detections_kernel");
    BP_TRY(read_back(&k, kept.counts + kept.n_blocks, st));
    *n_detections = (size_t)k;
    return BP_OK;
  }
  int* peaks = nullptr;
  BP_TRY(sc.get(&peaks, n / 2 + 1));
  int m = 0;
  BP_TRY(find_peaks_impl(d_beam_max, n, distance_only(distance),
                         PeakOut{peaks, nullptr, nullptr, nullptr}, &m, sc, st));
  if (m == 0) return BP_OK;
  int *flags = nullptr, *rank = nullptr;
  BP_TRY(sc.get(&flags, (size_t)m + 1));
  BP_TRY(sc.get(&rank, (size_t)m + 1));
  above_flags_kernel<<<grid_for((long long)m + 1, 256), 256, 0, st>>>(d_beam_max, d_threshold,
                                                                      peaks, m, flags);
  BP_LAUNCHED("above_flags_kernel");
  BP_TRY(scan_flags(flags, rank, m, sc, st));
  int k = 0;
  BP_TRY(read_back(&k, rank + m, st));
  scatter_detections_kernel<<<grid_for(m, 256), 256, 0, st>>>(
      flags, rank, peaks, m, d_beam_max, d_argmax, d_peaks, d_heights, d_sources);
  BP_LAUNCHED("scatter_detections_kernel");
  BP_CUDA(cudaStreamSynchronize(st));
  *n_detections = (size_t)k;
  return BP_OK;
}

}  // extern "C"
