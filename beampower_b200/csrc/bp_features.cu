// Waveform features on the GPU: the reference tutorial's envelope transform
// (notebooks/3_beampower.ipynb:74-103, `envelope`): the modulus of the
// analytic signal (scipy.signal.hilbert), centred on its median and divided
// by its median absolute deviation (1 when that is 0), clipped above at 1e5.
//
// Per row of samples: a real-to-complex FFT (cuFFT), the Hilbert weights on
// the spectrum (1 at DC and, for even lengths, Nyquist; 2 on the positive
// frequencies; 0 on the negative ones) written as a full-length spectrum, an
// inverse complex FFT, and the modulus scaled by 1/N.  The median and the
// median absolute deviation are exact order statistics of that envelope, and
// the normalisation uses NumPy's float32 subtract and divide.
//
// What bounds it is HBM traffic, two thirds of it in the FFTs' passes.  On 180
// rows of 180,000 samples it takes 796 us; 1470 us with the row copied for
// the FFT, three histogram passes of a radix select for each statistic and one
// sample per thread in the passes between.  (The Hilbert transform alone, as one
// complex transform of half the length each way, takes 720 us and is as
// accurate, but its envelopes differ in the last bit, and with them the source
// of the beam's maximum where two sources are that close.)
#define BP_TEMPLATE_KERNELS_ONLY
#include <cmath>
#include <map>
#include <mutex>
#include <tuple>

#include <cufft.h>

#include "bp_stats.cuh"

namespace {

const char* cufft_name(cufftResult r) {
  switch (r) {
    case CUFFT_SUCCESS: return "success";
    case CUFFT_INVALID_PLAN: return "invalid plan";
    case CUFFT_ALLOC_FAILED: return "allocation failed";
    case CUFFT_INVALID_VALUE: return "invalid value";
    case CUFFT_INTERNAL_ERROR: return "internal error";
    case CUFFT_EXEC_FAILED: return "exec failed";
    case CUFFT_SETUP_FAILED: return "setup failed";
    case CUFFT_INVALID_SIZE: return "invalid size";
    default: return "error";
  }
}

#define BP_CUFFT(call)                                                              \
  do {                                                                              \
    cufftResult r_ = (call);                                                        \
    if (r_ != CUFFT_SUCCESS)                                                        \
      return fail(r_ == CUFFT_ALLOC_FAILED ? BP_ERR_OUT_OF_MEMORY : BP_ERR_CUDA,     \
                  "%s: cuFFT %s", #call, cufft_name(r_));                           \
  } while (0)

// Plans are costly to make: kept per (device, length, batch, kind) for the
// life of the process.  A plan holds one stream at a time, so setting its
// stream and enqueueing its transform happen under the cache's lock.  The
// lock orders the enqueues only: a plan's work area is shared by every stream
// that uses it, so transforms of one shape on different streams must not
// overlap on the GPU (stated in the header; the library's own callers use
// one stream per call).
struct PlanCache {
  std::mutex mu;
  std::map<std::tuple<int, int, int, int>, cufftHandle> plans;
};
PlanCache g_plans;

// Caller holds g_plans.mu.
int get_plan(int n, int batch, cufftType type, cufftHandle* out) {
  int dev = 0;
  BP_CUDA(cudaGetDevice(&dev));
  const auto key = std::make_tuple(dev, n, batch, (int)type);
  auto it = g_plans.plans.find(key);
  if (it != g_plans.plans.end()) {
    *out = it->second;
    return BP_OK;
  }
  cufftHandle h;
  BP_CUFFT(cufftCreate(&h));
  size_t work = 0;
  int len = n;
  const int in_dist = n, out_dist = type == CUFFT_R2C ? n / 2 + 1 : n;
  cufftResult r = cufftMakePlanMany(h, 1, &len, nullptr, 1, in_dist, nullptr, 1, out_dist, type,
                                    batch, &work);
  if (r != CUFFT_SUCCESS) {
    cufftDestroy(h);
    return fail(r == CUFFT_ALLOC_FAILED ? BP_ERR_OUT_OF_MEMORY : BP_ERR_CUDA,
                "cufftMakePlanMany(n=%d, batch=%d): %s", n, batch, cufft_name(r));
  }
  g_plans.plans.emplace(key, h);
  *out = h;
  return BP_OK;
}

int fft_forward_r2c(int n, int batch, const float* in, cufftComplex* out, cudaStream_t st) {
  std::lock_guard<std::mutex> lock(g_plans.mu);
  cufftHandle h;
  BP_TRY(get_plan(n, batch, CUFFT_R2C, &h));
  BP_CUFFT(cufftSetStream(h, st));
  BP_CUFFT(cufftExecR2C(h, const_cast<float*>(in), out));  // out of place: in is kept
  return BP_OK;
}

int fft_inverse_c2c(int n, int batch, cufftComplex* data, cudaStream_t st) {
  std::lock_guard<std::mutex> lock(g_plans.mu);
  cufftHandle h;
  BP_TRY(get_plan(n, batch, CUFFT_C2C, &h));
  BP_CUFFT(cufftSetStream(h, st));
  BP_CUFFT(cufftExecC2C(h, data, data, CUFFT_INVERSE));
  return BP_OK;
}

// Full-length analytic spectrum from the half spectrum of a real row
// (grid: x over the row's bins, kEachBin per thread, y over rows).
constexpr int kEachBin = 4;
__global__ void __launch_bounds__(256)
hilbert_weights_kernel(const cufftComplex* __restrict__ half, int n,
                       cufftComplex* __restrict__ full) {
  const size_t r = blockIdx.y;
  const int nh = n / 2 + 1;
  const int k0 = blockIdx.x * 256 * kEachBin + threadIdx.x;
  cufftComplex z[kEachBin];
#pragma unroll
  for (int u = 0; u < kEachBin; ++u) {
    const int k = k0 + u * 256;
    z[u] = k < nh ? half[r * nh + k] : make_cuFloatComplex(0.0f, 0.0f);
  }
#pragma unroll
  for (int u = 0; u < kEachBin; ++u) {
    const int k = k0 + u * 256;
    if (k >= n) break;
    const float w = k == 0 || 2 * k == n ? 1.0f : 2.0f;
    full[r * n + k] = k < nh ? make_cuFloatComplex(w * z[u].x, w * z[u].y) : z[u];
  }
}

__device__ __forceinline__ float envelope_of(cufftComplex z, float inv_n) {
  return hypotf(z.x * inv_n, z.y * inv_n);
}

// ---- medians of the rows -------------------------------------------------------
// A sample of kSample values of a row brackets its median: the sample's median
// lies within kSampleRanks of the right rank (4.5 standard deviations of the
// binomial) but for a few rows in a million.  The pass that makes the values
// anyway (the envelope, then the deviations) counts those below the bracket and
// at its ends and collects the 7% inside; one block per row selects among them.
// A row whose bracket misses (or whose inside does not fit) is selected by its
// block from the whole row, so the result is always the exact statistic.
// Three histogram passes per statistic, which this replaces, took 500 of 1470 us
// on 180 rows of 180,000 samples: shared-memory atomics at about one lane per
// clock, with the values of a row in few bins.
constexpr int kSample = 4096, kSampleRanks = 144;
constexpr int kSelThreads = 1024;

struct RowSelect {
  float lo, hi;  // the bracket: two values of the row
  unsigned below, at_lo, inside, at_hi;
  unsigned nan;
  unsigned pad;
};

// Shared memory of a selection.
constexpr int kSelBins = 2 * kSelThreads;
struct SelectShared {
  unsigned hist[kSelBins];
  uint32_t few[kSelThreads];
  unsigned warp_sum[32];
  unsigned n_few;
  uint32_t result;
};

// Keys are the bits of floats that are not negative, so ordered as they are.
// Histogram of the keys in [lo, hi] by (key - lo) >> shift.
template <class Key>
__device__ void select_histogram(const Key& key, int len, uint32_t lo, uint32_t hi, int shift,
                                 SelectShared& s) {
  const int tid = threadIdx.x;
  __syncthreads();
  s.hist[tid] = s.hist[tid + kSelThreads] = 0u;
  __syncthreads();
#pragma unroll 4
  for (int i = tid; i < len; i += kSelThreads) {
    const uint32_t k = key(i);
    if (k >= lo && k <= hi) atomicAdd(&s.hist[(k - lo) >> shift], 1u);
  }
  __syncthreads();
}

struct Place {
  unsigned bin, before, count;
};
// The histogram's bin that holds a rank, and what lies before it.
__device__ Place select_place(unsigned rank, SelectShared& s) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned a = s.hist[2 * tid], b = s.hist[2 * tid + 1];
  unsigned sum = a + b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned v = __shfl_up_sync(kFull, sum, o);
    if (lane >= o) sum += v;
  }
  if (lane == 31) s.warp_sum[warp] = sum;
  __syncthreads();
  const unsigned from = __reduce_add_sync(kFull, lane < warp ? s.warp_sum[lane] : 0u);
  const unsigned excl = from + sum - a - b;
  __syncthreads();
  if (rank >= excl && rank < excl + a + b) {
    const bool second = rank >= excl + a;
    s.warp_sum[0] = 2 * tid + (second ? 1 : 0);
    s.warp_sum[1] = excl + (second ? a : 0u);
    s.warp_sum[2] = second ? b : a;
  }
  __syncthreads();
  const Place p{s.warp_sum[0], s.warp_sum[1], s.warp_sum[2]};
  __syncthreads();
  return p;
}

__device__ __forceinline__ int select_shift(uint32_t lo, uint32_t hi) {
  return max(0, 32 - __clz((int)(hi - lo)) - 11);  // kSelBins bins
}

// The rank[0 .. Q - 1]-th smallest (0-based) of `len` keys, all of them in
// [lo, hi]: one histogram, and for each rank the keys of its bin, the one among
// them found by counting those before it when they are at most one per thread,
// else by another histogram of the bin.  All threads of the block call it.
template <int Q, class Key>
__device__ void select_keys(const Key& key, int len, const unsigned (&rank)[Q], uint32_t lo,
                            uint32_t hi, SelectShared& s, uint32_t (&out)[Q]) {
  const int tid = threadIdx.x;
  int shift = select_shift(lo, hi);
  select_histogram(key, len, lo, hi, shift, s);
  Place place[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) place[q] = select_place(rank[q], s);
#pragma unroll 1
  for (int q = 0; q < Q; ++q) {
    Place p = place[q];
    uint32_t l = lo, h = hi;
    unsigned r = rank[q];
    int sh = shift;
    while (true) {
      r -= p.before;
      l += p.bin << sh;
      h = l + ((1u << sh) - 1u);
      if (sh == 0 || p.count <= kSelThreads) break;
      sh = select_shift(l, h);
      select_histogram(key, len, l, h, sh, s);
      p = select_place(r, s);
    }
    if (sh == 0) {
      out[q] = l;
      continue;
    }
    if (tid == 0) s.n_few = 0u;
    __syncthreads();
#pragma unroll 4
    for (int i = tid; i < len; i += kSelThreads) {
      const uint32_t k = key(i);
      if (k >= l && k <= h) s.few[atomicAdd(&s.n_few, 1u)] = k;
    }
    __syncthreads();
    if (tid < (int)p.count) {
      const uint32_t mine = s.few[tid];
      unsigned less = 0, upto = 0;
      for (unsigned i = 0; i < p.count; ++i) {
        less += s.few[i] < mine;
        upto += s.few[i] <= mine;
      }
      if (r >= less && r < upto) s.result = mine;  // equal keys write the same
    }
    __syncthreads();
    out[q] = s.result;
    __syncthreads();
  }
}

// Both middle keys of `len` keys (one and the same for an odd len).
template <class Key>
__device__ uint2 middle_keys(const Key& key, int len, SelectShared& s) {
  const unsigned r[2] = {(unsigned)(len - 1) / 2, (unsigned)len / 2};
  uint32_t k[2];
  select_keys<2>(key, len, r, 0u, 0x7FFFFFFFu, s, k);
  return make_uint2(k[0], k[1]);
}

// NumPy's median of the middle keys.
__device__ __forceinline__ float middle_value(uint2 k, int len) {
  const float a = __uint_as_float(k.x), b = __uint_as_float(k.y);
  if (len % 2) return np_divide_count(__fadd_rn(0.0f, a), 1);
  return np_divide_count(__fadd_rn(0.0f, __fadd_rn(a, b)), 2);
}

// The row's place of sample j of kSample: one in each stride, not at a fixed
// phase of it.
__device__ __forceinline__ int sample_place(int j, int n) {
  const unsigned stride = (unsigned)(n / kSample);
  const unsigned h = (unsigned)j * 2654435761u;
  return (int)((long long)j * n / kSample) + (int)__umulhi(h, stride);
}

// The bracket of the median of `kSample` keys.
template <class Key>
__device__ void bracket(const Key& key, RowSelect* r, SelectShared& s) {
  const unsigned ranks[2] = {kSample / 2 - kSampleRanks, kSample / 2 + kSampleRanks};
  uint32_t k[2];
  select_keys<2>(key, kSample, ranks, 0u, 0x7FFFFFFFu, s, k);
  if (threadIdx.x == 0)
    *r = RowSelect{__uint_as_float(k[0]), __uint_as_float(k[1]), 0u, 0u, 0u, 0u, 0u, 0u};
}

// Block r: row r's sample of the envelope and its median's bracket.
__global__ void __launch_bounds__(kSelThreads, 2)
sample_kernel(const cufftComplex* __restrict__ z, int n, float inv_n, float* __restrict__ sample,
              RowSelect* __restrict__ rows) {
  __shared__ uint32_t v[kSample];
  __shared__ SelectShared sh;
  const size_t row = blockIdx.x;
  cufftComplex a[kSample / kSelThreads];
#pragma unroll
  for (int t = 0; t < kSample / kSelThreads; ++t)
    a[t] = z[row * n + sample_place(t * kSelThreads + threadIdx.x, n)];
#pragma unroll
  for (int t = 0; t < kSample / kSelThreads; ++t) {
    const int j = t * kSelThreads + threadIdx.x;
    const float e = envelope_of(a[t], inv_n);
    v[j] = __float_as_uint(e) & 0x7FFFFFFFu;  // (a NaN's sign)
    sample[row * kSample + j] = e;
  }
  bracket([&](int i) { return v[i]; }, rows + row, sh);
}

// A warp's values against its row's bracket: counts per lane, a list in shared
// memory.  Warps take kChunks chunks of the row, one after the other, loading the
// next before they look at the present one, and add their counts and lists to
// the row's by themselves.  (A list per block of 4,096 samples, with its two
// barriers and the wait for the row's counter, took 92 and 100 us for the two
// passes on 180 x 180,000 samples.)
struct RowCounter {
  static constexpr int kWarps = 8, kThreads = 32 * kWarps;
  static constexpr int kEach = 8, kChunk = 32 * kEach, kChunks = 8;
  static constexpr int kBlock = kWarps * kChunks * kChunk;
  static constexpr int kList = 3 * kChunk;
  struct Shared {
    float list[kWarps][kList];
  };
  float* list;
  RowSelect* row;
  float* out;
  unsigned capacity;
  float lo, hi;
  unsigned below = 0, at_lo = 0, at_hi = 0, nan = 0, n_list = 0;
  __device__ RowCounter(Shared& sh, RowSelect* rows, size_t r, float* lists, unsigned cap)
      : list(sh.list[threadIdx.x >> 5]),
        row(rows + r),
        out(lists + r * cap),
        capacity(cap),
        lo(row->lo),
        hi(row->hi) {}

  // A chunk's values; the first `use` of each lane's count (kEach but at the
  // row's end).  Every lane of the warp calls it.
  template <bool WHOLE>
  __device__ __forceinline__ void add(const float (&v)[kEach], int use) {
    const unsigned before = (1u << (threadIdx.x & 31)) - 1u;
    int seen = 0;  // below, inside and above: not the bracket's ends, not NaN
#pragma unroll
    for (int u = 0; u < kEach; ++u) {
      const bool live = WHOLE || u < use;
      const bool in = live && v[u] > lo && v[u] < hi;
      const bool less = live && v[u] < lo;
      const unsigned b = __ballot_sync(kFull, in);
      if (in) list[n_list + __popc(b & before)] = v[u];
      n_list += __popc(b);
      if (less) ++below;
      if (in || less || (live && v[u] > hi)) ++seen;
    }
    if (seen != (WHOLE ? kEach : use)) {
#pragma unroll
      for (int u = 0; u < kEach; ++u)
        if (WHOLE || u < use) {
          at_lo += v[u] == lo;
          at_hi += v[u] == hi && lo < hi;
          nan |= v[u] != v[u];
        }
    }
    __syncwarp();
    if (n_list > kList - kChunk) flush();
  }
  __device__ void flush() {
    const int lane = threadIdx.x & 31;
    unsigned to = 0;
    if (lane == 0 && n_list) to = atomicAdd(&row->inside, n_list);
    to = __shfl_sync(kFull, to, 0);
    for (unsigned i = lane; i < n_list; i += 32)
      if (to + i < capacity) out[to + i] = list[i];
    __syncwarp();
    n_list = 0;
  }
  __device__ void finish() {
    flush();
    below = __reduce_add_sync(kFull, below);
    at_lo = __reduce_add_sync(kFull, at_lo);
    at_hi = __reduce_add_sync(kFull, at_hi);
    nan = __any_sync(kFull, nan);
    if ((threadIdx.x & 31) == 0) {
      if (below) atomicAdd(&row->below, below);
      if (at_lo) atomicAdd(&row->at_lo, at_lo);
      if (at_hi) atomicAdd(&row->at_hi, at_hi);
      if (nan) atomicOr(&row->nan, 1u);
    }
  }
  // A chunk's first sample of this lane, and how many it has.
  static __device__ __forceinline__ int first(int chunk) {
    return blockIdx.x * kBlock + (chunk * kWarps + (int)(threadIdx.x >> 5)) * kChunk +
           (int)(threadIdx.x & 31);
  }
  static __device__ __forceinline__ int number(int i, int n) {
    return i >= n ? 0 : min(kEach, (n - i + 31) / 32);
  }
};

// Envelope of a row's kBlock samples (grid: x over the row, y over rows), with
// the counts of the median's bracket when COUNT.
template <bool COUNT>
__global__ void __launch_bounds__(RowCounter::kThreads)
envelope_kernel(const cufftComplex* __restrict__ z, int n, float inv_n, float* __restrict__ out,
                RowSelect* __restrict__ rows, float* __restrict__ lists, unsigned capacity) {
  using C = RowCounter;
  __shared__ C::Shared sh;
  const size_t row = blockIdx.y;
  z += row * n;
  out += row * n;
  auto run = [&](auto& count) {
    cufftComplex a[C::kEach];
    auto load = [&](int i) {
      if (i + 32 * C::kEach - 32 < n) {
#pragma unroll
        for (int u = 0; u < C::kEach; ++u) a[u] = z[i + 32 * u];
      } else {
#pragma unroll
        for (int u = 0; u < C::kEach; ++u)
          a[u] = i + 32 * u < n ? z[i + 32 * u] : make_cuFloatComplex(0.0f, 0.0f);
      }
    };
    load(C::first(0));
#pragma unroll 1
    for (int chunk = 0; chunk < C::kChunks; ++chunk) {
      const int i = C::first(chunk);
      if (i - (int)(threadIdx.x & 31) >= n) break;  // the whole warp
      float v[C::kEach];
#pragma unroll
      for (int u = 0; u < C::kEach; ++u) v[u] = envelope_of(a[u], inv_n);
      if (chunk + 1 < C::kChunks) load(C::first(chunk + 1));
      const int use = C::number(i, n);
      if (__all_sync(kFull, use == C::kEach)) {
#pragma unroll
        for (int u = 0; u < C::kEach; ++u) out[i + 32 * u] = v[u];
        if constexpr (COUNT) count.template add<true>(v, use);
      } else {
#pragma unroll
        for (int u = 0; u < C::kEach; ++u)
          if (u < use) out[i + 32 * u] = v[u];
        if constexpr (COUNT) count.template add<false>(v, use);
      }
    }
    if constexpr (COUNT) count.finish();
  };
  if constexpr (COUNT) {
    C count(sh, rows, row, lists, capacity);
    run(count);
  } else {
    int none = 0;
    run(none);
  }
}

// The counts of the bracket of the deviations from the median.
__global__ void __launch_bounds__(RowCounter::kThreads)
deviation_kernel(const float* __restrict__ env, int n, const float* __restrict__ med,
                 RowSelect* __restrict__ rows, float* __restrict__ lists, unsigned capacity) {
  using C = RowCounter;
  __shared__ C::Shared sh;
  const size_t row = blockIdx.y;
  env += row * n;
  const float c = med[row];
  C count(sh, rows, row, lists, capacity);
  float a[C::kEach];
  auto load = [&](int i) {
    if (i + 32 * C::kEach - 32 < n) {
#pragma unroll
      for (int u = 0; u < C::kEach; ++u) a[u] = env[i + 32 * u];
    } else {
#pragma unroll
      for (int u = 0; u < C::kEach; ++u) a[u] = i + 32 * u < n ? env[i + 32 * u] : 0.0f;
    }
  };
  load(C::first(0));
#pragma unroll 1
  for (int chunk = 0; chunk < C::kChunks; ++chunk) {
    const int i = C::first(chunk);
    if (i - (int)(threadIdx.x & 31) >= n) break;  // the whole warp
    float v[C::kEach];
#pragma unroll
    for (int u = 0; u < C::kEach; ++u) v[u] = fabsf(__fsub_rn(a[u], c));
    if (chunk + 1 < C::kChunks) load(C::first(chunk + 1));
    const int use = C::number(i, n);
    if (__all_sync(kFull, use == C::kEach)) count.add<true>(v, use);
    else count.add<false>(v, use);
  }
  count.finish();
}

// Block r: row r's median from the counts and the list.  SPREAD: of the
// deviations from `centre`; without it, also the bracket of those.
template <bool SPREAD>
__global__ void __launch_bounds__(kSelThreads, 2)
row_median_kernel(const float* __restrict__ env, int n, const float* __restrict__ lists,
                  unsigned capacity, const RowSelect* __restrict__ rows,
                  const float* __restrict__ centre, float* __restrict__ out,
                  const float* __restrict__ sample, RowSelect* __restrict__ spread_rows) {
  __shared__ SelectShared sh;
  const size_t row = blockIdx.x;
  const RowSelect r = rows[row];
  float m = __uint_as_float(0x7FC00000u);
  if (!r.nan) {
    const unsigned first = (unsigned)(n - 1) / 2, last = (unsigned)n / 2;
    const unsigned inside = r.below + r.at_lo, end = inside + r.inside;
    const uint32_t klo = __float_as_uint(r.lo), khi = __float_as_uint(r.hi);
    uint2 k;
    if (first >= r.below && last < end + r.at_hi && r.inside <= capacity) {
      k.x = first < inside ? klo : khi;
      k.y = last < inside ? klo : khi;
      const bool in_first = first >= inside && first < end;
      const bool in_last = last >= inside && last < end;
      if (in_first || in_last) {
        const float* list = lists + row * capacity;
        const unsigned ranks[2] = {(in_first ? first : last) - inside,
                                   (in_last ? last : first) - inside};
        uint32_t keys[2];
        select_keys<2>([&](int i) { return __float_as_uint(list[i]); }, (int)r.inside, ranks,
                       klo, khi, sh, keys);
        if (in_first) k.x = keys[0];
        if (in_last) k.y = keys[1];
      }
    } else {
      const float* e = env + row * n;
      if (SPREAD) {
        const float c = centre[row];
        k = middle_keys([&](int i) { return __float_as_uint(fabsf(__fsub_rn(e[i], c))); }, n,
                        sh);
      } else {
        k = middle_keys([&](int i) { return __float_as_uint(e[i]); }, n, sh);
      }
    }
    m = middle_value(k, n);
  }
  if (threadIdx.x == 0) out[row] = m;
  if (!SPREAD)
    bracket(
        [&](int i) {
          return __float_as_uint(fabsf(__fsub_rn(sample[row * kSample + i], m)));
        },
        spread_rows + row, sh);
}

// Block r: median and median absolute deviation of a row of at most kSample
// samples.
__global__ void __launch_bounds__(kSelThreads, 2)
short_row_kernel(const float* __restrict__ env, int n, float* __restrict__ med,
                 float* __restrict__ mad) {
  __shared__ float v[kSample];
  __shared__ SelectShared sh;
  const size_t row = blockIdx.x;
  bool nan = false;
  for (int i = threadIdx.x; i < n; i += kSelThreads) {
    v[i] = env[row * n + i];
    nan |= v[i] != v[i];
  }
  nan = __syncthreads_or(nan);
  float m = __uint_as_float(0x7FC00000u), d = m;
  if (!nan) {
    m = middle_value(middle_keys([&](int i) { return __float_as_uint(v[i]); }, n, sh), n);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kSelThreads) {
      v[i] = fabsf(__fsub_rn(v[i], m));
      nan |= v[i] != v[i];
    }
    nan = __syncthreads_or(nan);
    if (!nan)
      d = middle_value(middle_keys([&](int i) { return __float_as_uint(v[i]); }, n, sh), n);
  }
  if (threadIdx.x == 0) {
    med[row] = m;
    mad[row] = d;
  }
}

// NumPy's minimum against the clip value: NaN stays NaN.
__device__ __forceinline__ float clip_above(float x, float hi) {
  return (isnan(x) || x <= hi) ? x : hi;
}

// (env - median) / (mad, or 1 when it is 0), clipped above (grid: x over
// the row's samples, y over rows; in place).
__global__ void __launch_bounds__(256)
normalise_kernel(float* __restrict__ env, int n, const float* __restrict__ med,
                 const float* __restrict__ mad, float clip_max) {
  constexpr int U = 8;
  const int i0 = blockIdx.x * 256 * U + threadIdx.x;
  const size_t r = blockIdx.y;
  env += r * n;
  const float m = mad[r], c = med[r];
  const float scale = m == 0.0f ? 1.0f : m;
  float v[U];
#pragma unroll
  for (int u = 0; u < U; ++u) v[u] = i0 + u * 256 < n ? env[i0 + u * 256] : 0.0f;
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (i0 + u * 256 < n)
      env[i0 + u * 256] = clip_above(__fdiv_rn(__fsub_rn(v[u], c), scale), clip_max);
}

// Rows per pass so that the scratch buffers stay within a few GB.
int rows_per_pass(size_t n, size_t rows) {
  const size_t per_row = n * sizeof(float) * 5;
  const size_t budget = size_t(6) << 30;
  size_t r = std::max<size_t>(1, budget / std::max<size_t>(per_row, 1));
  return (int)std::min<size_t>(std::min<size_t>(r, rows), 65535);
}

// Rows whose medians go through a bracket: one block selects among 7% of a
// row, which for few long rows takes longer than the radix select's passes over
// all of the chip (one row of 2^21 samples: about 100 us against 50).
bool bracket_rows(int n, int rows) {
  return n > kSample && n <= (rows >= 16 ? 1 << 22 : 1 << 18);
}

int envelope_rows(const float* x, size_t rows, size_t n, float clip_max, float* out,
                  cudaStream_t st) {
  const int N = (int)n;
  if (N == 1) {  // the analytic signal of one sample is itself: feature 0
    BP_CUDA(cudaMemsetAsync(out, 0, rows * sizeof(float), st));
    return BP_OK;
  }
  const int chunk = rows_per_pass(n, rows);
  const float inv_n = 1.0f / (float)N;
  Scratch sc(st);
  float *re = nullptr, *med = nullptr, *mad = nullptr, *sample = nullptr, *lists = nullptr;
  cufftComplex *half = nullptr, *full = nullptr;
  RowSelect* sel = nullptr;
  const bool brackets = bracket_rows(N, chunk);
  const unsigned capacity = (unsigned)(N / 8);
  BP_TRY(sc.get(&half, (size_t)chunk * (n / 2 + 1)));
  BP_TRY(sc.get(&full, (size_t)chunk * n));
  BP_TRY(sc.get(&med, chunk));
  BP_TRY(sc.get(&mad, chunk));
  if (brackets) {
    BP_TRY(sc.get(&sample, (size_t)chunk * kSample));
    BP_TRY(sc.get(&lists, (size_t)chunk * capacity));
    BP_TRY(sc.get(&sel, 2 * (size_t)chunk));
  }
  for (size_t r0 = 0; r0 < rows; r0 += chunk) {
    const int b = (int)std::min<size_t>(chunk, rows - r0);
    const float* in = x + r0 * n;
    float* o = out + r0 * n;
    if (reinterpret_cast<uintptr_t>(in) % 256 != 0) {  // as an allocation's start is, for cuFFT
      if (!re) BP_TRY(sc.get(&re, (size_t)chunk * n));
      BP_CUDA(cudaMemcpyAsync(re, in, (size_t)b * n * sizeof(float), cudaMemcpyDeviceToDevice,
                              st));
      in = re;
    }
    BP_TRY(fft_forward_r2c(N, b, in, half, st));
    hilbert_weights_kernel<<<dim3((unsigned)((N + 256 * kEachBin - 1) / (256 * kEachBin)),
                                  (unsigned)b),
                             256, 0, st>>>(half, N, full);
    BP_LAUNCHED("hilbert_weights_kernel");
    BP_TRY(fft_inverse_c2c(N, b, full, st));
    const dim3 rows_grid((unsigned)((N + RowCounter::kBlock - 1) / RowCounter::kBlock),
                         (unsigned)b);
    if (brackets) {
      RowSelect *centre = sel, *spread = sel + chunk;
      sample_kernel<<<(unsigned)b, kSelThreads, 0, st>>>(full, N, inv_n, sample, centre);
      BP_LAUNCHED("sample_kernel");
      envelope_kernel<true><<<rows_grid, RowCounter::kThreads, 0, st>>>(
          full, N, inv_n, o, centre, lists, capacity);
      BP_LAUNCHED("envelope_kernel");
      row_median_kernel<false><<<(unsigned)b, kSelThreads, 0, st>>>(
          o, N, lists, capacity, centre, nullptr, med, sample, spread);
      BP_LAUNCHED("row_median_kernel");
      deviation_kernel<<<rows_grid, RowCounter::kThreads, 0, st>>>(o, N, med, spread,
                                                                            lists, capacity);
      BP_LAUNCHED("deviation_kernel");
      row_median_kernel<true><<<(unsigned)b, kSelThreads, 0, st>>>(
          o, N, lists, capacity, spread, med, mad, nullptr, nullptr);
      BP_LAUNCHED("row_median_kernel");
    } else {
      envelope_kernel<false><<<rows_grid, RowCounter::kThreads, 0, st>>>(full, N, inv_n, o,
                                                                         nullptr, nullptr, 0u);
      BP_LAUNCHED("envelope_kernel");
      if (N <= kSample) {
        short_row_kernel<<<(unsigned)b, kSelThreads, 0, st>>>(o, N, med, mad);
        BP_LAUNCHED("short_row_kernel");
      } else {
        BP_TRY(np_median(o, N, N, b, 0, nullptr, med, sc, st));
        BP_TRY(np_median(o, N, N, b, 1, med, mad, sc, st));
      }
    }
    normalise_kernel<<<dim3((unsigned)((N + 2047) / 2048), (unsigned)b), 256, 0, st>>>(
        o, N, med, mad, clip_max);
    BP_LAUNCHED("normalise_kernel");
  }
  return BP_OK;
}

}  // namespace

extern "C" {

int bp_envelope_dev(const float* d_x, size_t n_rows, size_t n_samples, float clip_max,
                    float* d_out, void* stream) {
  BP_NVTX("bp_envelope_dev");
  if (n_rows == 0 || n_samples == 0) return BP_OK;
  if (!d_x || !d_out) return fail(BP_ERR_INVALID_ARGUMENT, "NULL pointer");
  if (n_samples > (size_t)INT_MAX / 2)
    return fail(BP_ERR_UNSUPPORTED, "rows longer than 2^30 samples");
  return envelope_rows(d_x, n_rows, n_samples, clip_max, d_out,
                       reinterpret_cast<cudaStream_t>(stream));
}

}  // extern "C"

extern "C" {

int bp_prestack_envelope_dev(const float* d_waveforms, const float* d_weights_phases,
                             size_t n_samples, size_t n_stations, size_t n_channels,
                             size_t n_phases, float clip_max, int storage, size_t lpad,
                             size_t pitch, void* d_traces, float* d_scales, void* stream) {
  BP_NVTX("bp_prestack_envelope_dev");
  if (n_samples == 0 || n_stations == 0 || n_channels == 0) return BP_OK;
  if (!d_waveforms || !d_weights_phases || !d_traces)
    return fail(BP_ERR_INVALID_ARGUMENT, "NULL pointer");
  if (n_samples > (size_t)INT_MAX / 2)
    return fail(BP_ERR_UNSUPPORTED, "rows longer than 2^30 samples");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const size_t rows = n_stations * n_channels;
  float* features = nullptr;
  {
    Scratch sc(st);
    BP_TRY(sc.get(&features, rows * n_samples));
    BP_TRY(envelope_rows(d_waveforms, rows, n_samples, clip_max, features, st));
    BP_TRY(bp_prestack_dev(features, d_weights_phases, n_samples, n_stations, n_channels,
                           n_phases, storage, lpad, pitch, d_traces, d_scales, stream));
  }
  return BP_OK;
}

}  // extern "C"
