// Shift-and-stack through tensor memory (TMEM), sm_100a.
//
// The staged kernel of bp_kernels.cuh reads every beam term from shared
// memory, whose 128 B/clk/SM (32 FP32 words) bound it: 0.86 of that roof on
// the 400,000-source workload.  A delay is a shift, and a tcgen05.ld takes
// its first column from a register, so rows of consecutive samples kept in
// TMEM serve every source at its own shift: lane i's row holds the samples
// from 16 i on, and a load of 16 columns from column (delay - window start)
// gives lane i its 16 shifted samples.  TMEM reads do not pass through shared
// memory: a probe loop reads 136 words/clk/SM alone and 78 with the packed
// adds and the fills.  This kernel sums 47 terms/clk/SM (64,000 sources x 60
// stations x 2 phases x 18,000 samples: 10.1 ms; the staged shape 8 takes 17.9
// ms, 27 terms) and takes 446 instead of 742 ms on the 400,000-source
// workload.  It is bound by instruction issue (0.67 busy; of 243 instructions
// a warp takes per station, 64 are the adds), the adds' pipe is 0.49 busy.
//
// Block = 640 threads over one 64-source table tile and time tiles of 512
// samples (32 lanes x 16):
//   * 16 compute warps, 4 sources each: 64 accumulators per thread and one
//     load of 16 columns in flight per warp.  (2 sources x 32 samples halve the
//     loads but double the ring's traffic and the fills per source: 13.6 ms.)
//   * 4 producer warps, which take the fills in turn.  Bulk copies (TMA
//     engine) bring the delay window of a station and phase into a
//     shared-memory ring, and tcgen05.cp (32x128b, the same 32 rows into all
//     four lane quarters) moves it into TMEM without passing through
//     registers: (16 + span) / 4 copies per station and phase instead of 64 x
//     16 words read per lane.
//     (Filling TMEM from registers, by warps of its own or by the compute
//     warps, was measured at 26 and 15 terms/clk/SM: the instructions, not the
//     bytes, were in the way.)
// The windows are read from planes (planes_kernel): tcgen05.cp takes rows 16
// bytes apart, lanes are 64 bytes (16 FP32 samples) apart, so plane k holds
// the 16-byte chunks k, k + 4, k + 8, ... of a trace row one after the other.
// 16-bit storage keeps two planes of each of the copies 0 and 1 (pairs of
// samples from even and from odd samples on).
// TMEM holds 4, 2 or 1 fills by the widest window of the block's tile.  (Two
// fills of whole stations need fewer waits, but the round trip from the last
// read of a fill to the next one in its place showed: 10.7 ms.)
// Registers: 640 threads leave 96 each at launch; the producer warps give 64
// back and the compute warps run with 112.
//
// Arithmetic and order are the staged kernel's, term for term: FP32 bit for
// bit the reference's, 16-bit storage bit for bit the staged shapes'.
#pragma once

#include <algorithm>

#include "bp_kernels.cuh"

namespace bp {

// ---- tcgen05 wrappers ---------------------------------------------------------
// Loads of 16 or 8 columns into r[AT..].
template <int B>
__device__ __forceinline__ void tm_ld16(uint32_t taddr, uint32_t (&r)[B]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
template <int AT, int B>
__device__ __forceinline__ void tm_ld8(uint32_t taddr, uint32_t (&r)[B]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[AT]), "=r"(r[AT + 1]), "=r"(r[AT + 2]), "=r"(r[AT + 3]), "=r"(r[AT + 4]),
        "=r"(r[AT + 5]), "=r"(r[AT + 6]), "=r"(r[AT + 7])
      : "r"(taddr));
}
// 32 rows of 16 bytes from shared memory into 4 columns of all four lane
// quarters; asynchronous, completed by tm_commit's mbarrier.
__device__ __forceinline__ void tm_cp(uint32_t taddr, uint64_t desc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(desc)
               : "memory");
}
__device__ __forceinline__ void tm_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_addr(bar))
      : "memory");
}
// Shared-memory matrix descriptor of rows 16 bytes apart (no swizzle, groups
// of 8 rows 128 bytes apart); the low 14 bits count 16-byte units.
__device__ __forceinline__ uint64_t tm_desc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(128 >> 4) << 32) | (1ull << 46);
}
// One lane of the (converged) warp arrives.
__device__ __forceinline__ void mbar_arrive_elected(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 st;\n\t"
      "elect.sync _|p, 0xFFFFFFFF;\n\t"
      "@p mbarrier.arrive.release.cta.shared::cta.b64 st, [%0];\n\t}" ::"r"(bar)
      : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ bool mbar_try_wait_at(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(e));
  return e != 0;
}
__device__ __forceinline__ void tm_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tm_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tm_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Ties N loaded registers to the wait before their use: nothing that reads
// them may move above this point.
template <int N, int B>
__device__ __forceinline__ void tm_tie(uint32_t (&r)[B]) {
#pragma unroll
  for (int i = 0; i < N; i += 4)
    asm volatile("" : "+r"(r[i]), "+r"(r[i + 1]), "+r"(r[i + 2]), "+r"(r[i + 3]));
}

constexpr int kTmCols = 512;       // TMEM columns of an SM, all allocated
constexpr int kTmTile = 512;       // samples of a time tile: 32 lanes x 16
constexpr int kTmCompute = 16;     // compute warps
constexpr int kTmThreads = 640;    // + 4 producer warps
constexpr int kTmMaxStage = 4;     // ring stages of a producer warp
constexpr int kTmRedRow = 16 * 33; // keys of a quarter of the warps, padded
// Bytes of an element's record: 64 first columns (one per source), flags, a
// spare word, address of its station's weights, scale.
constexpr int kTmRecord = kTableTile * 4 + 16;
constexpr int kTmFixed = 384 + kTableTile * 16;  // barriers, flags, source records

// Samples of a 16-byte chunk.  A (station, phase) whose delay offsets, counted
// from a window start on a 16-sample boundary, run from `shift` (< 16) to
// `off`: the chunks before `shift` stay out; TMEM columns (FP32 one row of
// samples, 16-bit two rows of sample pairs), plane rows.
__host__ __device__ constexpr int tm_chunk(bool f32) { return f32 ? 4 : 8; }
__host__ __device__ inline int tm_row_cols(int shift, int off, bool f32) {
  const int skip = shift / tm_chunk(f32) * 4;
  return f32 ? (off + 16 - skip + 3) / 4 * 4 : (off / 2 + 8 - skip + 3) / 4 * 4;
}
__host__ __device__ inline int tm_cols(int shift, int off, bool f32) {
  return (f32 ? 1 : 2) * tm_row_cols(shift, off, f32);
}
__host__ __device__ inline int tm_rows(int off) { return 32 + (off + 15) / 16; }
// Rows of one plane of a trace row of `pitch` elements.
__host__ __device__ inline long long tm_plane_rows(long long pitch) { return pitch / 16 + 4; }

// TMEM slots of an item: 4, 2 or 1 fills of its widest window; fill n's first
// column is (n << shift) mod 512.
struct TmSlots {
  int n, shift;
  __host__ __device__ __forceinline__ TmSlots(int widest)
      : n(widest <= 128 ? 4 : widest <= 256 ? 2 : 1),
        shift(widest <= 128 ? 7 : widest <= 256 ? 8 : 9) {}
};

// Trace rows -> planes: 16-byte chunk c of row r (16-bit: of its copies 0 and
// 1) to plane c mod 4 (16-bit: copy * 2 + c mod 2); zeros past the row.
// r: FP32 the row; 16-bit row * 2 + copy.
constexpr int kPlanesBlock = 256;  // chunks
__host__ __device__ inline long long tm_planes_blocks(long long pitch, bool f32) {
  return (tm_plane_rows(pitch) * (f32 ? 4 : 2) + kPlanesBlock - 1) / kPlanesBlock;
}
template <bool F32>
__device__ __forceinline__ void plane_chunk(const uint4* __restrict__ traces, long long pitch,
                                            uint4* __restrict__ planes, long long r,
                                            long long c) {
  constexpr int CH = F32 ? 4 : 8, PL = F32 ? 4 : 2;  // samples of a chunk, planes of a copy
  const long long rows = tm_plane_rows(pitch);
  if (c >= rows * PL) return;
  const long long src = F32 ? r : (r >> 1) * kHalfCopies + (r & 1);
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (c * CH < pitch) v = traces[src * (pitch / CH) + c];
  planes[(r * PL + c % PL) * rows + c / PL] = v;
}

// One record; grid (tm_planes_blocks, rows x copies).
template <bool F32>
__global__ void __launch_bounds__(kPlanesBlock)
planes_kernel(const uint4* __restrict__ traces, long long pitch, uint4* __restrict__ planes) {
  plane_chunk<F32>(traces, pitch, planes, blockIdx.y,
                   (long long)blockIdx.x * kPlanesBlock + threadIdx.x);
}

// Every record of a batch in one launch: record r has the blocks prefix[r] ..
// prefix[r + 1] - 1.  (256 windows of 1,500 samples, 400 sources x 10 stations: with a
// launch per record the batch took 3.51 ms, 2.26 as a graph; now 2.44 and 1.76, and the
// staged kernel, which needs no planes, 2.42 and 1.79.)
template <bool F32>
__global__ void __launch_bounds__(kPlanesBlock)
batch_planes_kernel(const RecordView* __restrict__ records, int n_records,
                    const long long* __restrict__ prefix) {
  int lo = 0, hi = n_records - 1;
  const long long b = blockIdx.x;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (prefix[mid] <= b) lo = mid; else hi = mid - 1;
  }
  const RecordView& q = records[lo];
  const long long local = b - prefix[lo], each = tm_planes_blocks(q.pitch, F32);
  plane_chunk<F32>(static_cast<const uint4*>(q.traces), q.pitch,
                   reinterpret_cast<uint4*>(const_cast<unsigned char*>(q.planes)), local / each,
                   local % each * kPlanesBlock + threadIdx.x);
}

// Shared-memory carve-up, made on the host and read from the kernel's
// parameters (constant bank), so that no offset holds a register.
template <int P, bool MAXRED>
__host__ inline TmLayout tm_layout(int max_rows, int max_active, int n_stage) {
  TmLayout l{};
  size_t o = kTmFixed;
  l.n_stage = n_stage;
  l.plane_bytes = max_rows * 16;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o = align_up_sz(o + bytes, 16);
    return (uint32_t)at;
  };
  const size_t el = (size_t)max_active * P;
  // max: four rows of keys; whole response: 16 x 34 floats per warp
  l.red = take(MAXRED ? (size_t)4 * kTmRedRow * 8 : (size_t)kTmCompute * 16 * 34 * 4);
  l.records = take((el + 1) * kTmRecord);
  l.weights = take((size_t)max_active * kTableTile * 4);
  l.el_src = take(el * 8);
  l.el_info = take(el * 4);
  l.st_j = take((size_t)max_active * 4);
  o = align_up_sz(o, 128);
  l.ring = (uint32_t)o;
  o += (size_t)n_stage * 4 * 4 * l.plane_bytes;  // stages x warps x planes
  l.total = (uint32_t)std::min<size_t>(align_up_sz(o, 128), 0xFFFFFFFFu);
  return l;
}

template <int P, bool MAXRED, int STORAGE>
struct Tm {
  static constexpr bool F32 = STORAGE == BP_STORAGE_F32;
  static constexpr bool F16 = STORAGE == BP_STORAGE_F16;
  using M = typename MetaT<P>::type;
  static constexpr int KS = 4;            // sources per compute warp
  static constexpr int NB = F32 ? 16 : 8;  // registers of one load

  struct Smem {
    unsigned char* base;
    const TmLayout& l;
    template <class V>
    __device__ __forceinline__ V* at(uint32_t off) const {
      return reinterpret_cast<V*>(base + off);
    }
    // ring stage s of producer warp w
    __device__ __forceinline__ uint64_t* full(int w, int s) const {
      return at<uint64_t>(32 * w + 8 * s);
    }
    __device__ __forceinline__ uint64_t* empty(int w, int s) const {
      return at<uint64_t>(128 + 32 * w + 8 * s);
    }
    // fill n (w = n & 3): in TMEM, read by every compute warp
    __device__ __forceinline__ uint64_t* tfull(int w) const { return at<uint64_t>(256 + 8 * w); }
    __device__ __forceinline__ uint64_t* tempty(int w) const { return at<uint64_t>(288 + 8 * w); }
    __device__ __forceinline__ volatile int* abort_flag() const { return at<int>(320); }
    __device__ __forceinline__ int* n_act() const { return at<int>(324); }
    __device__ __forceinline__ uint32_t* tm_base() const { return at<uint32_t>(328); }
    // item: its widest fill, and whether some weight is neither 0 nor 1
    __device__ __forceinline__ int* widest() const { return at<int>(332); }
    __device__ __forceinline__ int* real() const { return at<int>(344); }
    __device__ __forceinline__ long long* plane_stride() const { return at<long long>(336); }
    __device__ __forceinline__ int4* cur_item() const { return at<int4>(352); }
    __device__ __forceinline__ int4* srci() const { return at<int4>(384); }
    // per element (active station i, phase p) e = i * P + p, or per station
    __device__ __forceinline__ unsigned char* red() const { return base + l.red; }
    __device__ __forceinline__ uint32_t* record(int e) const {
      return at<uint32_t>(l.records + e * kTmRecord);
    }
    __device__ __forceinline__ uint32_t* weights() const { return at<uint32_t>(l.weights); }
    __device__ __forceinline__ const unsigned char** el_src() const {
      return at<const unsigned char*>(l.el_src);
    }
    __device__ __forceinline__ uint32_t* el_info() const { return at<uint32_t>(l.el_info); }
    __device__ __forceinline__ int* st_j() const { return at<int>(l.st_j); }
    __device__ __forceinline__ unsigned char* ring() const { return base + l.ring; }
  };
  // el_info: bits 0..9 TMEM columns, 10..13 the window's shift, 16..31 plane rows.
  // record flags: bit w every weight of compute warp w is 1, bit 16 + w every
  // one 0; all bits set: behind the last element.
  __device__ static __forceinline__ int info_cols(uint32_t v) { return (int)(v & 0x3FFu); }
  __device__ static __forceinline__ int info_shift(uint32_t v) { return (int)(v >> 10 & 15u); }
  __device__ static __forceinline__ int info_rows(uint32_t v) { return (int)(v >> 16); }

  // All threads, once per block: barriers and the TMEM allocation.  One block
  // runs per SM (61,440 registers), so the allocation of every column waits
  // for no block of this kernel.
  __device__ static __forceinline__ void start(const Smem& sm) {
    if (threadIdx.x == 0) {
      for (int w = 0; w < 4; ++w)
        for (int s = 0; s < kTmMaxStage; ++s) {
          mbar_init(sm.full(w, s), 1);
          mbar_init(sm.empty(w, s), 1);
        }
      for (int w = 0; w < 4; ++w) {
        mbar_init(sm.tfull(w), 1);
        mbar_init(sm.tempty(w), kTmCompute);
      }
      *sm.abort_flag() = 0;
      fence_mbar_init();
    }
    if ((threadIdx.x >> 5) == kTmCompute) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                       smem_addr(sm.tm_base()))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tm_fence_before();
    __syncthreads();
    tm_fence_after();
  }

  // The producer warps, at the end (the compute warps fence and meet the barrier).
  __device__ static __forceinline__ void finish(const Smem& sm) {
    tm_fence_before();
    __syncthreads();
    tm_fence_after();
    if ((threadIdx.x >> 5) == kTmCompute)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(
          *sm.tm_base()));
  }

  // All threads, before an item: the tile's stations (those the record uses),
  // per source slot the samples it keeps, per element its planes and TMEM
  // columns, per (element, source) the first column of its load, per (station,
  // source) the weight.  Returns whether every factor w * scale is exact in
  // the 16-bit format.
  __device__ static __forceinline__ bool prologue(const Smem& sm, const TableView& tb,
                                                  const RecordView& rc, int tile, int tau0,
                                                  int tau1, int max_rows, int* status) {
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    if (warp == 0) {
      const int n_tab = tb.tile_hdr[tile].x;
      int n = 0;
      for (int j0 = 0; j0 < n_tab; j0 += 32) {
        const int j = j0 + lane;
        bool use = false;
        if (j < n_tab) {
          const int s = tb.st_s[(size_t)tile * tb.S + j];
          use = !rc.station_mask || ((rc.station_mask[s >> 5] >> (s & 31)) & 1u);
        }
        const unsigned bal = __ballot_sync(0xFFFFFFFFu, use);
        if (use) sm.st_j()[n + __popc(bal & ((1u << lane) - 1u))] = j;  // table slot
        n += __popc(bal);
      }
      if (lane == 0) {
        *sm.n_act() = n;
        *sm.widest() = 0;
        *sm.real() = 0;
        *sm.plane_stride() = tm_plane_rows(rc.pitch) * 16;
      }
    } else if (tid < 32 + kTableTile) {
      // {source, first, end, 0}: the record-local samples [first, end) the
      // out-of-bounds rule keeps (strict: every delay of the source inside the
      // record, the lower bound in global time); empty for an unused slot.
      // Clamped to +-2^30, beyond any sample index of a record.
      constexpr long long kFar = 1ll << 30;
      const int i = tid - 32;
      const size_t slot = (size_t)tile * kTableTile + i;
      int4 si = tb.src_info[slot];
      if (rc.srcmm) {
        const int2 mm = rc.srcmm[slot];
        si.y = mm.x;
        si.z = mm.y;
      }
      long long first = -kFar, end = kFar;
      if (si.x < 0 || (!rc.flexible && si.y > si.z)) {
        first = kFar;
        end = -kFar;
      } else if (!rc.flexible) {
        first = min(max(-rc.t_origin - (long long)si.y, -kFar), kFar);
        end = min(max((long long)rc.T - (long long)si.z, -kFar), kFar);
      }
      sm.srci()[i] = make_int4(si.x, (int)first, (int)end, 0);
    }
    __syncthreads();
    const int n_active = *sm.n_act();
    // a warp per station, two sources per lane
    const M* gm = reinterpret_cast<const M*>(tb.meta) + (size_t)tile * tb.S * kTableTile;
    int exact = 1;
    for (int i = warp; i < n_active; i += kTmThreads / 32) {
      const int j = sm.st_j()[i];
      const int s = tb.st_s[(size_t)tile * tb.S + j];
      const float scale = F32 ? 1.0f : rc.scales[s];
      int shift[P], row_cols[P];  // offsets counted from 16-sample boundaries
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const size_t g = ((size_t)tile * tb.S + j) * P + p;
        const long long x = (long long)rc.lpad + tb.st_lo[g];  // window start at time 0
        shift[p] = (int)(x & 15);
        const int off = tb.st_spread[g] + shift[p];
        row_cols[p] = tm_row_cols(shift[p], off, F32);
        int rows = tm_rows(off), cols = tm_cols(shift[p], off, F32);
        if (rows > max_rows || cols > kTmCols) {  // the host keeps such tables away
          if (lane == 0) atomicOr(status, kStatusBadWindow);
          rows = min(rows, max_rows);
          cols = min(cols, kTmCols);
        }
#if BP_DEBUG_CHECKS
        // every copy of the item's time tiles inside the planes
        if (x < 0 || (x >> 4) + tau0 * (kTmTile / 16) < 0 ||
            (x >> 4) + (tau1 - 1) * (kTmTile / 16) + rows > tm_plane_rows(rc.pitch)) {
          if (lane == 0) atomicOr(status, kStatusBadIndex);
          rows = 0;
        }
#endif
        if (lane == 0) {
          sm.el_src()[i * P + p] =
              rc.planes + ((long long)(s * P + p) * 4 * tm_plane_rows(rc.pitch) + (x >> 4)) * 16;
          sm.el_info()[i * P + p] =
              (uint32_t)cols | ((uint32_t)shift[p] << 10) | ((uint32_t)rows << 16);
          atomicMax(sm.widest(), cols);
        }
      }
      uint32_t ones = 0, none = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = 32 * h + lane;
        const M m = gm[(size_t)j * kTableTile + k];
        const float w = __uint_as_float(m.x);
#pragma unroll
        for (int p = 0; p < P; ++p) {
          const int o = w != 0.0f ? meta_off<P>(m, p) + shift[p] : 0;
          const int skip = shift[p] / tm_chunk(F32) * 4;  // columns left out
          sm.record(i * P + p)[k] =
              (uint32_t)(w == 0.0f ? 0
                         : F32     ? o - skip
                                   : (o & 1) * row_cols[p] + (o >> 1) - skip);
#if BP_DEBUG_CHECKS
          if (o > tb.st_spread[((size_t)tile * tb.S + j) * P + p] + shift[p])
            atomicOr(status, kStatusBadIndex);
#endif
        }
        sm.weights()[i * kTableTile + k] = m.x;
        if constexpr (!F32) {
          uint32_t pk;
          if (w != 0.0f && !pack_factor16<STORAGE>(w * scale, &pk)) exact = 0;
        }
        const uint32_t b1 = __ballot_sync(0xFFFFFFFFu, w == 1.0f);
        const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, w == 0.0f);
        if (F32 && lane == 0 && (b1 | b0) != 0xFFFFFFFFu) atomicOr(sm.real(), 1);
        // lanes 0..7: the 8 warps of these 32 sources
        const uint32_t n1 = (b1 >> (4 * (lane & 7))) & 15u, n0 = (b0 >> (4 * (lane & 7))) & 15u;
        ones |= (__ballot_sync(0xFFFFFFFFu, lane < 8 && n1 == 15u) & 0xFFu) << (8 * h);
        none |= (__ballot_sync(0xFFFFFFFFu, lane < 8 && n0 == 15u) & 0xFFu) << (8 * h);
      }
      if (lane < P) {
        uint32_t* r = sm.record(i * P + lane) + kTableTile;
        r[0] = ones | (none << 16);
        r[2] = smem_addr(sm.weights() + i * kTableTile);
        r[3] = __float_as_uint(scale);
      }
    }
    if (tid == 0) sm.record(n_active * P)[kTableTile] = 0xFFFFFFFFu;
    (void)tau0;
    (void)tau1;
    if constexpr (F32) {
      __syncthreads();
      return false;
    } else {
      const bool fast16 = __syncthreads_and(exact) != 0;
      if (fast16) {
        for (int x = tid; x < n_active * kTableTile; x += kTmThreads) {
          const float w = __uint_as_float(sm.weights()[x]);
          uint32_t pk = 0u;
          if (w != 0.0f) pack_factor16<STORAGE>(
                w * __uint_as_float(sm.record(x / kTableTile * P)[kTableTile + 3]), &pk);
          sm.weights()[x] = pk;
        }
        __syncthreads();
      }
      return fast16;
    }
  }

  // What a warp carries from item to item.  Fill n has producer warp and
  // barriers n & 3 (their parity n >> 2 & 1); the item's fills go through its
  // TMEM slots in turn.
  struct State {
    int n = 0;                // next fill
    int slot = 0, phase = 0;  // producer: next ring stage to read, its parity
#if BP_DEBUG_CHECKS
    int lose = -1;            // a fill that is not made, so that the waits for it run out
#endif
  };
  __device__ static __forceinline__ State state(const LaunchArgs& a, bool batch = false) {
    State st;
#if BP_DEBUG_CHECKS
    if (blockIdx.x == 0 || batch) st.lose = a.lose_fill - 1;
#endif
    (void)a;
    (void)batch;
    return st;
  }

  // After an abort: lets the copies already issued land, those from the ring into
  // TMEM (the last stage read; at the start of a barrier's life its odd phase counts
  // as over) and those into the ring.  A stage that holds none looks like one whose
  // copy is on its way, so it costs the limit.  (Counting the stages in produce()
  // costs that loop, which has 32 registers, a fifth of the kernel's speed: 52,311
  // sources x 37 stations x 15,001 samples 5.4 -> 6.7 ms.)
  __device__ static __forceinline__ void drain(const Smem& sm, int w, const State& st) {
    if (!*sm.abort_flag()) return;
    constexpr unsigned long long kLimitNs = 20000000ull;
    const bool wrap = st.slot == 0;
    mbar_wait_limit(sm.empty(w, (wrap ? sm.l.n_stage : st.slot) - 1),
                    wrap ? st.phase ^ 1 : st.phase, kLimitNs, nullptr);
    for (int s = 0; s < sm.l.n_stage; ++s)
      mbar_wait_limit(sm.full(w, s), s < st.slot ? st.phase ^ 1 : st.phase, kLimitNs, nullptr);
  }

  // ---- producer warps ---------------------------------------------------------
  // Warp w makes fills n = w, w + 4, ... (one station and phase each).  The
  // loop's values are kept warp-uniform (shuffles), so that the tcgen05.cp
  // operands come from uniform registers: with per-lane values one copy took 96
  // cycles to issue, with uniform ones about 15.
  __device__ static __forceinline__ void produce(const Smem& sm, int tau0, int tau1, int* status,
                                                 State& st) {
    const int w = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5) - kTmCompute, 0);
    const int lane = threadIdx.x & 31;
    const int n_el = *sm.n_act() * P;  // fills of a time tile
    const int total = (tau1 - tau0) * n_el;
    const int n_stage = sm.l.n_stage;
    const TmSlots slots(__shfl_sync(0xFFFFFFFFu, *sm.widest(), 0));
    const int first = (w - st.n) & 3;  // this warp's first fill of the item
    // next fill to issue copies for / to make: number in the item, element,
    // byte offset of its time tile (16 bytes of a plane to 16 samples)
    int ri = first, ei = first, r = first, e = first;
    long long it = (long long)tau0 * kTmTile;
    int islot = st.slot, iphase = st.phase;
    const uint32_t tm0 = *sm.tm_base();
    const uint32_t ring = smem_addr(sm.ring()) + w * n_stage * 4 * sm.l.plane_bytes;
    bool ok = true;
    auto issue_next = [&]() {
      if (ri >= total) return;
      while (ei >= n_el) {
        ei -= n_el;
        it += kTmTile;
      }
      ok = mbar_wait_spin(smem_addr(sm.empty(w, islot)), iphase ^ 1, sm.abort_flag(), status);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (!ok) return;
      const uint32_t bytes = (uint32_t)info_rows(sm.el_info()[ei]) * 16;
      if (lane == 0) mbar_arrive_expect_tx(sm.full(w, islot), 4 * bytes);
      __syncwarp();
      if (lane < 4 && (!BP_DEBUG_CHECKS || bytes))  // lane k: plane k
        bulk_g2s(sm.ring() + ((w * n_stage + islot) * 4 + lane) * sm.l.plane_bytes,
                 sm.el_src()[ei] + *sm.plane_stride() * lane + it, bytes, sm.full(w, islot));
      __syncwarp();
      if (++islot == n_stage) {
        islot = 0;
        iphase ^= 1;
      }
      ri += 4;
      ei += 4;
    };
#pragma unroll 1
    for (int k = max(1, n_stage - 1); k > 0 && ok; --k) issue_next();
#pragma unroll 1
    for (; r < total && ok; r += 4, e += 4) {
      while (e >= n_el) e -= n_el;
      const int n = __shfl_sync(0xFFFFFFFFu, st.n + r, 0);
      const uint32_t info = __shfl_sync(0xFFFFFFFFu, sm.el_info()[e], 0);
#if BP_DEBUG_CHECKS
      const bool lost = n == st.lose;
#else
      constexpr bool lost = false;
#endif
      const int cols = lost ? 0 : info_cols(info);
      ok = mbar_wait_spin(smem_addr(sm.full(w, st.slot)), st.phase, sm.abort_flag(), status);
      const int m = n - slots.n;  // the slot's last fill is read
      ok = ok && mbar_wait_spin(smem_addr(sm.tempty(m & 3)), (m >> 2) & 1, sm.abort_flag(),
                                status);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (!ok) break;
      tm_fence_after();
      const uint64_t d = tm_desc(ring + st.slot * 4 * sm.l.plane_bytes);
      const uint32_t du = (uint32_t)sm.l.plane_bytes / 16;  // a plane, in descriptor units
      const uint32_t t = tm0 + (((uint32_t)n << slots.shift) & (kTmCols - 1));
      // The window's chunks [j0, j1); FP32: chunk 4 c + k is row c of plane k;
      // 16-bit: of copy v, chunk 2 c + k is row c of plane 2 v + k.
      const int j0 = info_shift(info) / tm_chunk(F32);
      if (elect_one()) {
        if constexpr (F32) {
          const int j1 = j0 + cols / 4;
          const uint32_t tb = t - 4 * j0;
          int c = 0;
          if (j0 > 0) {  // some chunks of the first row are left out
#pragma unroll
            for (int k = 1; k < 4; ++k)
              if (k >= j0 && k < j1) tm_cp(tb + 4 * k, d + k * du);
            c = 1;
          }
#pragma unroll 1
          for (; 4 * c + 4 <= j1; ++c) {
            tm_cp(tb + 16 * c, d + c);
            tm_cp(tb + 16 * c + 4, d + c + du);
            tm_cp(tb + 16 * c + 8, d + c + 2 * du);
            tm_cp(tb + 16 * c + 12, d + c + 3 * du);
          }
#pragma unroll
          for (int k = 0; k < 3; ++k)
            if (4 * c + k < j1) tm_cp(tb + 16 * c + 4 * k, d + c + k * du);
        } else {
          const int j1 = j0 + cols / 8;
#pragma unroll
          for (int v = 0; v < 2; ++v) {
            const uint32_t tb = t + v * (cols / 2) - 4 * j0;
            const uint64_t dv = d + 2 * v * du;
            int c = 0;
            if (j0 > 0) {
              if (1 < j1) tm_cp(tb + 4, dv + du);
              c = 1;
            }
#pragma unroll 1
            for (; 2 * c + 2 <= j1; ++c) {
              tm_cp(tb + 8 * c, dv + c);
              tm_cp(tb + 8 * c + 4, dv + c + du);
            }
            if (2 * c < j1) tm_cp(tb + 8 * c, dv + c);
          }
        }
        if (!lost) tm_commit(sm.tfull(n & 3));
        tm_commit(sm.empty(w, st.slot));
      }
      __syncwarp();
      if (++st.slot == n_stage) {
        st.slot = 0;
        st.phase ^= 1;
      }
      issue_next();
    }
    st.n += total;
  }

  // ---- compute warps ----------------------------------------------------------
  // How a fill's FP32 terms are added: every weight is 1, every one is 0 or 1
  // (1 * u == u exactly: no multiply), or any.
  enum : int { kOnes, kBinary, kAny };
  template <int MODE>
  __device__ static __forceinline__ void add_term(float2 (&acc)[8], float w,
                                                  const uint32_t (&b)[NB]) {
    auto u = [&](int x) { return __uint_as_float(b[x]); };
    if (MODE != kOnes && w == 0.0f) return;  // warp-uniform
    if constexpr (MODE != kAny) {
#pragma unroll
      for (int x = 0; x < 8; ++x) acc[x] = add2_rn(acc[x], make_float2(u(2 * x), u(2 * x + 1)));
    } else {
      const float2 w2 = make_float2(w, w);  // rounded multiply, then rounded add
#pragma unroll
      for (int x = 0; x < 8; ++x)
        acc[x] = add2_rn(acc[x], mul2_rn(w2, make_float2(u(2 * x), u(2 * x + 1)), neg_zero()));
    }
  }

  // acc += c * v, the staged kernel's 16-bit arithmetic (v: FP16 the phases'
  // sum, BF16 one phase).  wt: the weight, or the packed factor.
  template <bool FAST16>
  __device__ static __forceinline__ void add_term16(float2 (&acc)[8], uint32_t wt, float scale,
                                                    const uint32_t (&v)[NB]) {
    if (FAST16 ? (wt == 0u) : (__uint_as_float(wt) == 0.0f)) return;  // warp-uniform
    const float c = FAST16 ? 0.0f : __uint_as_float(wt) * scale;
    const float2 c2 = make_float2(c, c);
    (void)c2;
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      if constexpr (F16) {
        if constexpr (FAST16) {
          fma2_f32_f16(acc[x], v[x], wt);
        } else {
          __half2 hh;
          memcpy(&hh, &v[x], 4);
          acc[x] = __ffma2_rn(c2, __half22float2(hh), acc[x]);
        }
      } else {
        if constexpr (FAST16) {
          fma2_f32_bf16(acc[x], v[x], wt);
        } else {
          const float2 u =
              make_float2(__uint_as_float(v[x] << 16), __uint_as_float(v[x] & 0xFFFF0000u));
          acc[x] = __ffma2_rn(c2, u, acc[x]);
        }
      }
    }
  }

  // Fill n, waited for (unless every lane has seen it complete: lanes may see it at
  // different tries, and the loads that follow are the whole warp's).
  __device__ static __forceinline__ void tm_take(const Smem& sm, int n, int* status,
                                                 bool seen = false) {
    if (!__all_sync(0xFFFFFFFFu, seen)) {
      mbar_wait_spin(smem_addr(sm.tfull(0)) + (n & 3) * 8, (n >> 2) & 1, sm.abort_flag(),
                     status);
      __syncwarp();
    }
    tm_fence_after();
  }
  // This warp is past its last load from fill n.
  __device__ static __forceinline__ void tm_give(const Smem& sm, int n) {
    tm_fence_before();
    __syncwarp();
    mbar_arrive_elected(smem_addr(sm.tempty(0)) + (n & 3) * 8);
  }
  __device__ static __forceinline__ void load(uint32_t t, uint32_t (&b)[NB]) {
    if constexpr (F32) tm_ld16(t, b);
    else tm_ld8<0>(t, b);
  }
  __device__ static __forceinline__ uint32_t part(const uint4& v, int k) {
    return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w;
  }

  // The fills as a compute warp goes through them: the next one's number, TMEM
  // address of column 0 of this warp's lanes, TmSlots::shift.
  struct Turn {
    int n;
    uint32_t t0;
    int shift;
    __device__ __forceinline__ uint32_t column() const {
      return t0 + (((uint32_t)n << shift) & (kTmCols - 1));
    }
  };

  // Sums the stations of the records from `ep` on (the address of this warp's
  // first columns in a record) as long as RUN fits their flags: kOnes all
  // weights 1 for this warp, kBinary and kAny some weight not 0 (kBinary: and
  // not all 1; so with 16-bit storage kAny).  FP32 and BF16; phases ascending.
  // Every warp of the block waits for the same fills, so what a warp waits for
  // at a fill's start is not hidden by the others: the next fill's flags, first
  // column and state are read during the last load of this one.  One load in
  // flight per warp: with two, the second buffer's registers were spilled.
  template <int RUN, bool FAST16>
  __device__ static __forceinline__ void sum_run(const Smem& sm, uint32_t& ep,
                                                 float2 (&acc)[KS][8], Turn& u, int* status) {
    const int warp = threadIdx.x >> 5;
    const uint32_t tail = (uint32_t)(kTableTile * 4 - warp * KS * 4);  // ep to flags
    auto suits = [&](uint32_t f) {
      f >>= warp;
      if (F32 && RUN == kOnes) return (f & 0x10001u) == 1u;
      if (F32 && RUN == kBinary) return (f & 0x10001u) == 0u;
      return (f & 0x10000u) == 0u;
    };
    uint32_t b[NB];
    uint32_t c = lds32(ep);
    uint32_t t = u.column();
    tm_take(sm, u.n, status);
    load(t + c, b);
#pragma unroll 1
    while (true) {
      uint32_t wp = 0;
      float scale = 1.0f;
      if (RUN != kOnes) wp = lds32(ep + tail + 8) + warp * (KS * 4);
      if (!F32) scale = __uint_as_float(lds32(ep + tail + 12));
      bool more = true, ready = false;
#pragma unroll
      for (int x = 0; x < KS * P; ++x) {
        const int k = x % KS, p = x / KS;
        uint32_t w = 0;
        if (RUN != kOnes) w = lds32(wp + k * 4);
        if (k + 1 < KS) {
          c = lds32(ep + p * kTmRecord + (k + 1) * 4);
        } else {
          // the next fill
          if (p + 1 == P) more = suits(lds32(ep + P * kTmRecord + tail));
          c = lds32(ep + (p + 1) * kTmRecord);
          ready = mbar_try_wait_at(smem_addr(sm.tfull(0)) + ((u.n + 1) & 3) * 8,
                                   ((u.n + 1) >> 2) & 1);
        }
        tm_wait_ld();
        tm_tie<NB>(b);
        if (k + 1 == KS) {
          tm_give(sm, u.n);
          ++u.n;
          t = u.column();
        }
        if constexpr (F32) add_term<RUN>(acc[k], __uint_as_float(w), b);
        else add_term16<FAST16>(acc[k], w, scale, b);
        if (k + 1 == KS) {
          if (p + 1 == P) {
            ep += P * kTmRecord;
            if (!more) return;
          }
          tm_take(sm, u.n, status, ready);
        }
        load(t + c, b);
      }
    }
  }

  // FP16: a station's phases are summed in FP16 first, then one FMA per sample.
  template <bool FAST16>
  __device__ static __forceinline__ void sum_phases16(const Smem& sm, uint32_t& ep,
                                                      float2 (&acc)[KS][8], Turn& u,
                                                      int* status) {
    const int warp = threadIdx.x >> 5;
    const uint32_t tail = (uint32_t)(kTableTile * 4 - warp * KS * 4);
    const uint32_t wp = lds32(ep + tail + 8) + warp * (KS * 4);
    const float scale = __uint_as_float(lds32(ep + tail + 12));
    uint32_t h[KS][NB];
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const uint32_t t = u.column();
      tm_take(sm, u.n, status);
#pragma unroll
      for (int k = 0; k < KS; ++k) {
        uint32_t b[NB];
        load(t + lds32(ep + 4 * k), b);
        tm_wait_ld();
        tm_tie<NB>(b);
        if (k == KS - 1) tm_give(sm, u.n);
#pragma unroll
        for (int x = 0; x < NB; ++x) h[k][x] = p == 0 ? b[x] : hadd2_rn(h[k][x], b[x]);
      }
      ++u.n;
      ep += kTmRecord;
    }
#pragma unroll
    for (int k = 0; k < KS; ++k) add_term16<FAST16>(acc[k], lds32(wp + 4 * k), scale, h[k]);
  }

  // Every station of a time tile into the accumulators.
  // MODE: FP32 kBinary or kAny; 16-bit: 1 when the weights are packed factors.
  template <int MODE>
  __device__ static __forceinline__ void sum_tile(const Smem& sm, float2 (&acc)[KS][8], Turn& u,
                                                  int* status) {
    const int warp = threadIdx.x >> 5;
    uint32_t ep = smem_addr(sm.record(0)) + warp * (KS * 4);
#pragma unroll 1
    while (true) {
      const uint32_t f =
          (lds32(ep + (uint32_t)(kTableTile * 4 - warp * KS * 4)) >> warp) & 0x10001u;
      if (f == 0x10001u) break;  // behind the last one
      if (f == 0x10000u) {       // no source of this warp uses the station
#pragma unroll 1
        for (int p = 0; p < P; ++p) {
          tm_take(sm, u.n, status);
          tm_give(sm, u.n);
          ++u.n;
          ep += kTmRecord;
        }
      } else if constexpr (F16) {
        sum_phases16<MODE == 1>(sm, ep, acc, u, status);
      } else if constexpr (F32 && MODE == kBinary) {
        if (f) sum_run<kOnes, false>(sm, ep, acc, u, status);
        else sum_run<kBinary, false>(sm, ep, acc, u, status);
      } else {
        sum_run<kAny, !F32 && MODE == 1>(sm, ep, acc, u, status);
      }
    }
  }

  // An item's time tiles.  One copy per kind of weights, so that each has the
  // registers to itself.
  __device__ static __forceinline__ void compute_item(const Smem& sm, const RecordView& rc,
                                                      int tau0, int tau1, bool fast16,
                                                      int* status, State& st) {
    constexpr int M0 = F32 ? kBinary : 0, M1 = F32 ? kAny : 1;
    if (F32 ? *sm.real() != 0 : fast16) compute<M1>(sm, rc, tau0, tau1, status, st);
    else compute<M0>(sm, rc, tau0, tau1, status, st);
  }

  template <int MODE>
  __device__ static __forceinline__ void compute(const Smem& sm, const RecordView& rc, int tau0,
                                                 int tau1, int* status, State& st) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const TmSlots slots(*sm.widest());
    Turn u;
    u.n = st.n;
    u.t0 = *sm.tm_base() + ((uint32_t)(32 * (warp & 3)) << 16);
    u.shift = slots.shift;
    const int src0 = warp * KS;
    const int4* my_src = sm.srci() + src0;
    const int own = 16 * lane;
    int past = 0;  // moves the loop beyond its end
#pragma unroll 1
    for (int tau = tau0; tau + past < tau1; ++tau) {
      const int t0 = tau * kTmTile;
      float2 acc[KS][8];  // pair x: samples own + 2x, + 1
#pragma unroll
      for (int k = 0; k < KS; ++k)
#pragma unroll
        for (int x = 0; x < 8; ++x) acc[k][x] = make_float2(0.0f, 0.0f);
      sum_tile<MODE>(sm, acc, u, status);

      // ---- epilogue of the time tile ----
      if constexpr (MAXRED) {
        // Per sample the best of this thread's 4 slots (ascending slots are
        // ascending sources: a strict `>` keeps the lowest index among equal
        // maxima; the -FLT_MAX seed makes NaN and -FLT_MAX lose).
        const int q = warp & 3, grp = warp >> 2;
        unsigned long long* row = reinterpret_cast<unsigned long long*>(sm.red()) + q * kTmRedRow;
        float bv[16];
        int bi[16];
        bool all_kept = true;  // warp-uniform: every slot keeps the whole tile
#pragma unroll
        for (int k = 0; k < KS; ++k)
          all_kept = all_kept && my_src[k].y <= t0 && t0 + kTmTile <= my_src[k].z;
#pragma unroll
        for (int x = 0; x < 16; ++x) {
          bv[x] = -FLT_MAX;
          bi[x] = -1;
        }
#pragma unroll
        for (int k = 0; k < KS; ++k) {
          const int4 si = my_src[k];
#pragma unroll
          for (int x = 0; x < 16; ++x) {
            const int t = t0 + own + x;
            const float v = (x & 1) ? acc[k][x >> 1].y : acc[k][x >> 1].x;
            if (v > bv[x] && (all_kept || (t >= si.y && t < si.z))) {
              bv[x] = v;
              bi[x] = si.x;
            }
          }
        }
        // four warps max into one row of keys one after the other
        uint32_t hi[16];
#pragma unroll
        for (int x = 0; x < 16; ++x) hi[x] = bi[x] >= 0 ? ordered_bits(bv[x]) : 0u;
#pragma unroll 1
        for (int g = 0; g < 4; ++g) {
          if (grp == g) {
#pragma unroll
            for (int x = 0; x < 16; ++x) {
              const uint32_t from = 0xFFFFFFFFu - (uint32_t)bi[x];
              unsigned long long key = hi[x] ? ((unsigned long long)hi[x] << 32) | from : 0ull;
              if (g > 0) {
                const unsigned long long old = row[x * 33 + lane];
                key = old > key ? old : key;
              }
              row[x * 33 + lane] = key;
            }
          }
          if (g < 3) named_barrier_sync(2 + q, 128);
        }
        // A warp whose wait ran out (which raised the abort flag) has summed what
        // was not there: none of them writes, and all of them end with this tile.
        // (Leaving the loop from here spills 39 registers of its body, and setting
        // its end costs the form with shares and one phase 12%.)
        const bool lost = named_barrier_or(1, kTmCompute * 32, *sm.abort_flag() != 0);
        if (lost) past = 1 << 30;
        {
          const unsigned long long* r0 = reinterpret_cast<const unsigned long long*>(sm.red()) +
                                         (tid & 15) * 33 + (tid >> 4);
          unsigned long long b = r0[0];
#pragma unroll
          for (int g = 1; g < 4; ++g) b = max(b, r0[g * kTmRedRow]);
          const int t = t0 + tid;
          if (!lost && b != 0ull && t >= rc.out0 && t < rc.out1)
            red_max_u64(&rc.keys[t - rc.out0], b);
        }
        named_barrier_sync(1, kTmCompute * 32);
      } else {
        // (a wait of this warp that ran out raised the abort flag)
        // (the two ways out: with one phase setting `past` costs the form with shares
        // 13%, with two and three the other one 10 to 40%)
        if (__any_sync(0xFFFFFFFFu, *sm.abort_flag() != 0)) {
          if constexpr (P == 1) break;
          past = 1 << 30;
        }
        // through this warp's buffer, so that the stores are coalesced
        float* buf = reinterpret_cast<float*>(sm.red()) + warp * (16 * 34);
#pragma unroll
        for (int k = 0; k < KS; ++k) {
          const int4 si = my_src[k];
          if (si.x < 0 || past) continue;  // warp-uniform
          float* out = rc.beam + (size_t)si.x * rc.ldb - rc.out0;
#pragma unroll
          for (int x = 0; x < 16; ++x)
            buf[x * 34 + lane] = (x & 1) ? acc[k][x >> 1].y : acc[k][x >> 1].x;
          __syncwarp();
          const int first = max(si.y, rc.out0), end = min(si.z, rc.out1);
#pragma unroll
          for (int y = 0; y < 16; ++y) {
            const int o = y * 32 + lane;
            const int t = t0 + o;
            if (t >= first && t < end) out[t] = buf[(o & 15) * 34 + (o >> 4)];
          }
          __syncwarp();
        }
      }
    }
    st.n = u.n;
  }
};

// Plain launch: one record, block = (table tile, chunk of time tiles),
// time-chunk major so that the blocks in flight share an L2-resident stretch
// of trace.  The two roles do not share code after their register split (the
// shared part would be held to the smaller share).
template <int P, bool MAXRED, int STORAGE>
__global__ void __launch_bounds__(kTmThreads, 1)
beam_tmem_kernel(const __grid_constant__ LaunchArgs a) {
  using T = Tm<P, MAXRED, STORAGE>;
  extern __shared__ __align__(128) unsigned char smem[];
  const typename T::Smem sm{smem, a.tm};
  T::start(sm);
  int tile = blockIdx.x % a.tab0.n_tiles;
  const int chunk = blockIdx.x / a.tab0.n_tiles;
  if (a.tile_order) tile = a.tile_order[tile];
  const int tau_end = (a.rec0.out1 + kTmTile - 1) / kTmTile;
  const int tau0 = a.rec0.out0 / kTmTile + chunk * a.tiles_per_chunk;
  const int tau1 = min(tau0 + a.tiles_per_chunk, tau_end);
  const bool fast16 = T::prologue(sm, a.tab0, a.rec0, tile, tau0, tau1, a.rowcap, a.status);
  typename T::State st = T::state(a);
  if ((threadIdx.x >> 5) < kTmCompute) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    T::compute_item(sm, a.rec0, tau0, tau1, fast16, a.status, st);
    tm_fence_before();
    __syncthreads();
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    T::produce(sm, tau0, tau1, a.status, st);
    T::drain(sm, (threadIdx.x >> 5) - kTmCompute, st);
    T::finish(sm);
  }
}

// Plain launch of few (table tile, time tile) pairs per SM: a block per SM, and
// each takes an equal share of the pairs, tile after tile.  No last wave that is
// partly filled, and one prologue and TMEM allocation for a tile's pairs (4,000
// sources, 20 stations, 6,000 samples, five pairs per SM: 157 us with a block per
// pair, 130 us with shares).  With many pairs blocks of a few are the better
// balance, since tiles differ in cost (52,311 sources, 37 stations, 15,001
// samples, 166 pairs per SM: 5.3 ms, and 6.8 ms with shares), and the loop over a
// share costs them registers (2% in beam_tmem_kernel).
struct TmItem {
  int tile, tau0, tau1;
};
// The block's item that starts `done` time tiles into its share; empty behind
// the last one.
__device__ __forceinline__ TmItem tm_item(const LaunchArgs& a, int done) {
  const int first = a.rec0.out0 / kTmTile;
  const int n_tau = (a.rec0.out1 + kTmTile - 1) / kTmTile - first;
  const long long pairs = (long long)a.tab0.n_tiles * n_tau;
  const long long j = pairs * blockIdx.x / gridDim.x + done;
  const long long end = pairs * (blockIdx.x + 1) / gridDim.x;
  const int i = (int)(j / n_tau), from = (int)(j - (long long)i * n_tau);
  const int tile = a.tile_order && j < end ? a.tile_order[i] : i;
  return TmItem{tile, first + from, first + from + (int)min(end - j, (long long)(n_tau - from))};
}

template <int P, bool MAXRED, int STORAGE>
__global__ void __launch_bounds__(kTmThreads, 1)
beam_tmem_share_kernel(const __grid_constant__ LaunchArgs a) {
  using T = Tm<P, MAXRED, STORAGE>;
  extern __shared__ __align__(128) unsigned char smem[];
  const typename T::Smem sm{smem, a.tm};
  T::start(sm);
  typename T::State st = T::state(a);
  int done = 0;
  TmItem it = tm_item(a, 0);
  bool fast16 = T::prologue(sm, a.tab0, a.rec0, it.tile, it.tau0, it.tau1, a.rowcap, a.status);
  // To the next item; false behind the last one.
  auto next = [&]() {
    done += it.tau1 - it.tau0;
    __syncthreads();
    it = tm_item(a, done);
    if (it.tau0 >= it.tau1 || *sm.abort_flag()) return false;
    fast16 = T::prologue(sm, a.tab0, a.rec0, it.tile, it.tau0, it.tau1, a.rowcap, a.status);
    return true;
  };
  if ((threadIdx.x >> 5) < kTmCompute) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    do {
      T::compute_item(sm, a.rec0, it.tau0, it.tau1, fast16, a.status, st);
    } while (next());
    tm_fence_before();
    __syncthreads();
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    do {
      T::produce(sm, it.tau0, it.tau1, a.status, st);
    } while (next());
    T::drain(sm, (threadIdx.x >> 5) - kTmCompute, st);
    T::finish(sm);
  }
}

// Persistent launch over a batch's work queue (see beam_batch_kernel).
template <int P, int STORAGE>
__global__ void __launch_bounds__(kTmThreads, 1)
beam_tmem_batch_kernel(const __grid_constant__ LaunchArgs a) {
  using T = Tm<P, true, STORAGE>;
  extern __shared__ __align__(128) unsigned char smem[];
  const typename T::Smem sm{smem, a.tm};
  T::start(sm);
  // The next item {record, table tile, first and end time tile}, record -1 at
  // the end of the queue.
  auto next_item = [&]() -> int4 {
    if (threadIdx.x == 0) {
      const long long i = (long long)atomicAdd(a.next_item, 1ull);
      int4 cur = make_int4(-1, 0, 0, 0);
      if (i < a.rec_prefix[a.n_records]) {
        // record r: rec_prefix[r] <= i < rec_prefix[r + 1]
        int lo = 0, hi = a.n_records - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (a.rec_prefix[mid] <= i) lo = mid; else hi = mid - 1;
        }
        const RecordView& r = a.records[lo];
        const int n_tiles = a.tables[r.table].n_tiles;
        const long long local = i - a.rec_prefix[lo];
        const int chunk = (int)(local / n_tiles);
        const int tile = (int)(local - (long long)chunk * n_tiles);
        const int tau_end = (r.out1 + kTmTile - 1) / kTmTile;
        const int tau0 = r.out0 / kTmTile + chunk * r.tpc;
        cur = make_int4(lo, tile, tau0, min(tau0 + r.tpc, tau_end));
      }
      *sm.cur_item() = cur;
    }
    __syncthreads();
    return *sm.cur_item();
  };
  typename T::State st = T::state(a, true);
  if ((threadIdx.x >> 5) < kTmCompute) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    while (true) {
      const int4 item = next_item();
      if (item.x < 0) break;
      // by reference: copies would hold registers through the inner loops
      const RecordView& rc = a.records[item.x];
      const bool fast16 = T::prologue(sm, a.tables[rc.table], rc, item.y, item.z, item.w,
                                      a.rowcap, a.status);
      T::compute_item(sm, rc, item.z, item.w, fast16, a.status, st);
      __syncthreads();
      if (*sm.abort_flag()) break;
    }
    tm_fence_before();
    __syncthreads();
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    while (true) {
      const int4 item = next_item();
      if (item.x < 0) break;
      const RecordView& rc = a.records[item.x];
      T::prologue(sm, a.tables[rc.table], rc, item.y, item.z, item.w, a.rowcap, a.status);
      T::produce(sm, item.z, item.w, a.status, st);
      __syncthreads();
      if (*sm.abort_flag()) break;
    }
    T::drain(sm, (threadIdx.x >> 5) - kTmCompute, st);
    T::finish(sm);
  }
}

}  // namespace bp
