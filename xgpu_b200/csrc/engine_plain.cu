// engine_plain.cu -- CUDA-core X-engine: 2x2 register tile, FP32 and dp4a.
//
// The B200 counterpart of xGPU's shared2x2 kernels (kernel.cuh:238-422 FP32,
// kernel.cuh:427-591 dp4a, compute macros shared_transfer_4.cuh:91-156 and
// shared_transfer_4_dp4a.cuh:99-164).  The arithmetic per thread is the same:
// each thread owns a 2x2 block of stations (rows i, i+1 x columns j, j+1) and
// all 4 polarisation products of each, i.e. 16 complex visibilities.
//   FP32: 32 float sums; per sample and visibility the two products of the
//         real (and of the imaginary) part are summed exactly and the sum is
//         added with one rounding, as xGPU's float engine does
//         (omp_xengine.c:24-28), so the sums equal its own bit for bit.  While
//         no sum can pass 2^24 those additions are exact and dp4a does them;
//         from there on 3 FP32 instructions per component, 96 per sample.
//   dp4a: 48 int32 accumulators (re, im1, im2 as in kernel.cuh:464-479,574),
//         64 dp4a per group of 4 samples.
// What changes is the data path.  xGPU fetches one sample at a time through
// textures and swizzled input; here a CTA of 128 threads covers a block of
// 16 x 32 stations of one channel (small CTAs balance the SMs: the FP32
// engine may not split time), stages 128-byte panels of the natural
// [t][f][s][p][c] input into shared memory with TMA (one thread issues each
// chunk's panels on an mbarrier, double buffered; stations past n and samples
// past the input are zero-filled), and converts them in shared memory -- to 4-sample
// words for dp4a (a 4x4 byte transpose with PRMT) or to floats -- in an order
// that makes the 128-bit shared loads of the compute loop conflict-free.
// One launch covers a whole time range (not one NTIME_PIPE chunk), and the
// sums are added to the integration buffer once, at the end.
#include <atomic>

#include "internal.h"
#include "tc_common.cuh"

namespace xgpu {
namespace plain {

// A CTA covers a block of 16 (rows) x 32 (columns) stations of one channel
// with 128 threads, 8 x 16, each a 2x2 station tile.  Small CTAs balance the
// SMs: at N=256, F=10 there are 720 of them, five resident per SM, all at
// once (32 x 32 blocks of 256 threads gave 360 CTAs, two or three per SM).
constexpr int kBlk = 32;        // stations per column block
constexpr int kRows = 16;       // stations per row block
constexpr int kThreads = (kRows / 2) * (kBlk / 2);   // 128
constexpr int kRowBytes = kBlk * 4;   // one sample of one panel: 32 stations x 2 pol x re/im

// Block k -> (row block r of 16 stations, column block c of 32), 2c <= r:
// row blocks 2m and 2m + 1 both have m + 1 column blocks at or left of the
// diagonal, so blocks m(m+1) .. (m+1)^2 - 1 are row 2m, (m+1)^2 ..
// (m+1)(m+2) - 1 row 2m + 1.
__device__ __forceinline__ void decode_block(int k, int &rb, int &cb) {
  int m = (int)((sqrtf(4.0f * (float)k + 1.0f) - 1.0f) * 0.5f);
  while (m * (m + 1) > k) --m;
  while ((m + 1) * (m + 2) <= k) ++m;
  if (k < (m + 1) * (m + 1)) {
    rb = 2 * m;
    cb = k - m * (m + 1);
  } else {
    rb = 2 * m + 1;
    cb = k - (m + 1) * (m + 1);
  }
}

// Station (0..31) held in slot q of a converted panel: thread column tx reads
// stations 2tx and 2tx+1 from slots tx and 16+tx, so that 16 threads read 256
// contiguous bytes.  The conversions fill slot q from lane q, so a warp's
// stores are 32 consecutive slots (no bank conflicts).
__device__ __forceinline__ int station_of_slot(int q) { return q < 16 ? 2 * q : 2 * (q - 16) + 1; }

// Station (0..15) in slot q of a converted row panel: thread row ty reads
// stations 2ty and 2ty+1 from slots ty and 8+ty.
__device__ __forceinline__ int row_station_of_slot(int q) { return q < 8 ? 2 * q : 2 * (q - 8) + 1; }

struct Params {
  CUtensorMap map;        // the input, boxes of 128 bytes x 64 samples (one dp4a chunk)
  CUtensorMap map_float;  // FP32 engine: the same in boxes of 32 samples (float phase)
  int n, f;
  int t0, tcount;
  long long nbaseline;
  void *state;
  int overwrite;
  int per;          // samples per time split (blockIdx.z); == tcount without splits
  int *err;         // receives kErrTimeoutPanel (may be null)
  int stall;        // test switch: issue no panel loads (the waits on them expire)
  int f0;           // first channel (blockIdx.y counts from it)
  int overlap;      // dp4a: may run beside the previous (adding) launch of the stream
  FloatPast past;   // FP32 engine
};

// A block went to the float phase; the block in the middle of each channel's says so to
// the host (fp32_pieces).
__device__ __forceinline__ void report_past(const FloatPast &past) {
  if (past.word && threadIdx.x == 0 && blockIdx.z == 0 && blockIdx.x == gridDim.x / 2)
    *(volatile int *)past.word = past.integration;
}

// Queue the TMA loads of samples [tb, tb+NT) of the row panel and the column
// panel into raw[0] / raw[1], completing on bar.  Called by one thread.  The
// row panel is the 32 stations from station 16 rb (its 16 row stations are
// the first half; stations past n are zero-filled), the column panel the
// column block's 32 stations.
template <int NT>
__device__ __forceinline__ void issue_panels(uint8_t (*raw)[NT * kRowBytes], uint32_t bar,
                                             const Params &p, const CUtensorMap &map, int f, int rb,
                                             int cb, int tb) {
  if (p.stall) return;
  tc::mbar_expect_tx(bar, 2 * NT * kRowBytes);
  tc::tma_load_3d(tc::smem_u32(raw[0]), &map, bar, rb * kRows * 4, f, tb);
  tc::tma_load_3d(tc::smem_u32(raw[1]), &map, bar, cb * kRowBytes, f, tb);
}

// A panel that never arrived (bounded wait expired): record it and leave
// without touching the integration buffer, after the other buffer's load (if
// one is in flight) has landed or its wait has expired too.
__device__ __forceinline__ void panel_timeout(const Params &p, uint32_t other_bar,
                                              uint32_t other_parity, bool other_in_flight) {
  if (threadIdx.x == 0) {
    if (p.err) tc::report_error(p.err, kErrTimeoutPanel);
    if (other_in_flight && !p.stall) tc::mbar_wait(other_bar, other_parity, nullptr);
  }
}

// ---------------------------------------------------------------- dp4a ----
constexpr int kTcD = 64;                        // samples per chunk
constexpr int kGroups = kTcD / 4;               // 4-sample groups per chunk
constexpr int kRawPanel = kTcD * kRowBytes;     // 8 KiB
constexpr int kWordPanel = kGroups * kBlk * 16; // 8 KiB: [group][slot][Xr,Xi,Yr,Yi]
constexpr int kWordPanelRows = kGroups * kRows * 16;   // 4 KiB: the row block's 16 stations

__device__ __forceinline__ int dp4a(int a, int b, int c) {
  int d;
  asm("dp4a.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// raw [sample][station][4 bytes] -> words [group][slot][4 words of 4 samples]
// for the `slots` stations of a panel (32, or the row panel's first 16).  power:
// adds the power of the two inputs of the station in the thread's slot
// (threadIdx.x % kSlots for every item of a thread).
template <int kSlots>
__device__ __forceinline__ void to_words(const uint8_t *raw, int4 *words, int *power = nullptr) {
  for (int u = threadIdx.x; u < kGroups * kSlots; u += kThreads) {
    const int g = u / kSlots, q = u % kSlots;
    const int s = kSlots == kBlk ? station_of_slot(q) : row_station_of_slot(q);
    const uint32_t *r = (const uint32_t *)(raw + (4 * g) * kRowBytes) + s;
    const uint32_t w0 = r[0], w1 = r[kRowBytes / 4], w2 = r[2 * kRowBytes / 4],
                   w3 = r[3 * kRowBytes / 4];
    const uint32_t lo01 = __byte_perm(w0, w1, 0x5140), hi01 = __byte_perm(w0, w1, 0x7362);
    const uint32_t lo23 = __byte_perm(w2, w3, 0x5140), hi23 = __byte_perm(w2, w3, 0x7362);
    int4 o;
    o.x = (int)__byte_perm(lo01, lo23, 0x5410);  // X re, samples 0..3
    o.y = (int)__byte_perm(lo01, lo23, 0x7632);  // X im
    o.z = (int)__byte_perm(hi01, hi23, 0x5410);  // Y re
    o.w = (int)__byte_perm(hi01, hi23, 0x7632);  // Y im
    words[g * kSlots + q] = o;
    if (power) {
      power[0] = dp4a(o.x, o.x, dp4a(o.y, o.y, power[0]));
      power[1] = dp4a(o.z, o.z, dp4a(o.w, o.w, power[1]));
    }
  }
}

// One converted chunk into the thread's 2x2 tile: re, and the two halves of im
// (im = i1 - i2) kept apart, as -128 has no int8 negation.  Unrolled whole: a
// dp4a takes two issue slots, and each instruction beside the 64 of a group adds
// to them; with the loop's index and address arithmetic gone and the operand
// loads ahead, N=256, F=10, T=1024 goes from 110 us per call in chains to 101 (by
// 8), 94 (whole).
__device__ __forceinline__ void dp4a_chunk(const int4 *wrow, const int4 *wcol, int ty, int tx,
                                           int (&re)[2][2][2][2], int (&i1)[2][2][2][2],
                                           int (&i2)[2][2][2][2]) {
#pragma unroll
  for (int g = 0; g < kGroups; ++g) {
    int4 r[2], c[2];
    r[0] = wrow[g * kRows + ty];
    r[1] = wrow[g * kRows + 8 + ty];
    c[0] = wcol[g * kBlk + tx];
    c[1] = wcol[g * kBlk + 16 + tx];
    // Four sweeps over the 16 visibilities of the 2x2 tile, so that the two
    // dp4a of one real part are 48 instructions apart, not back to back.
#pragma unroll
    for (int sweep = 0; sweep < 4; ++sweep)
#pragma unroll
      for (int rs = 0; rs < 2; ++rs)
#pragma unroll
        for (int cs = 0; cs < 2; ++cs) {
          const int ar[2] = {r[rs].x, r[rs].z}, ai[2] = {r[rs].y, r[rs].w};
          const int br[2] = {c[cs].x, c[cs].z}, bi[2] = {c[cs].y, c[cs].w};
#pragma unroll
          for (int p1 = 0; p1 < 2; ++p1)
#pragma unroll
            for (int p2 = 0; p2 < 2; ++p2) {
              if (sweep == 0) re[rs][cs][p1][p2] = dp4a(ar[p1], br[p2], re[rs][cs][p1][p2]);
              if (sweep == 1) i1[rs][cs][p1][p2] = dp4a(ai[p1], br[p2], i1[rs][cs][p1][p2]);
              if (sweep == 2) i2[rs][cs][p1][p2] = dp4a(ar[p1], bi[p2], i2[rs][cs][p1][p2]);
              if (sweep == 3) re[rs][cs][p1][p2] = dp4a(ai[p1], bi[p2], re[rs][cs][p1][p2]);
            }
        }
  }
}

// Epilogue staging (in the panels' memory): 8 block rows of 32 baselines x
// 4 products x {re, im} int64, thread tx's two baselines (128 bytes) at
// tx * kEpiSeg in its row, 16 bytes apart from the next thread's, so that the
// eight lanes of each 16-byte store phase write eight different bank groups.
constexpr int kEpiSeg = 144;
constexpr int kEpiRow = 16 * kEpiSeg;

// Dynamic shared memory of the dp4a kernel: raw panels [2 buffers][row,
// column], the converted row and column words, two mbarriers, and room to
// align the panels to 128 bytes (TMA destinations): 45.2 KB, five CTAs per
// SM (96 registers a thread, the most that five allow; the unrolled tile loop stores 136
// bytes beyond them and loads 88, and four CTAs an SM without that take 95.4 us at
// N=256, F=10, T=1024 in chains against 94.4).
constexpr int kSmemDp4a = 2 * 2 * kRawPanel + kWordPanelRows + kWordPanel + 16 + 128;
static_assert(5 * (kSmemDp4a + 1024) <= 228 * 1024, "five dp4a CTAs per SM");
static_assert((kRows / 2) * kEpiRow <= 2 * 2 * kRawPanel, "epilogue staging fits the panels");

__global__ void __launch_bounds__(kThreads, 5) xengine_dp4a_kernel(const __grid_constant__ Params p) {
  extern __shared__ __align__(128) uint8_t dsm_raw[];
  uint8_t *dsm = (uint8_t *)(((uintptr_t)dsm_raw + 127) & ~(uintptr_t)127);
  auto raw = (uint8_t(*)[2][kRawPanel])dsm;
  int4 *wrow = (int4 *)(dsm + 2 * 2 * kRawPanel);   // row words, 16 slots
  int4 *wcol = wrow + kGroups * kRows;               // column words, 32 slots
  uint64_t *bars = (uint64_t *)(wcol + kGroups * kBlk);

  const int f = p.f0 + (int)blockIdx.y;
  int rb, cb;   // row block of 16 stations, column block of 32
  decode_block(blockIdx.x, rb, cb);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;   // ty 0..7
  // Time split blockIdx.z covers samples [tbeg, tend) of the call's range.
  const int tbeg = p.t0 + (int)blockIdx.z * p.per;
  const int tend = min(p.t0 + p.tcount, tbeg + p.per);
  const int nchunks = (tend - tbeg + kTcD - 1) / kTcD;

  int re[2][2][2][2], i1[2][2][2][2], i2[2][2][2][2];   // [rs][cs][p1][p2]
#pragma unroll
  for (int a = 0; a < 16; ++a) {
    (&re[0][0][0][0])[a] = 0;
    (&i1[0][0][0][0])[a] = 0;
    (&i2[0][0][0][0])[a] = 0;
  }

  // Programmatic launch (as the tensor-core kernels): unless this launch only
  // adds into sums that the previous launch of the stream also only adds
  // into, nothing below reads or writes global memory before that launch has
  // finished; an overlapping launch waits for it at the end instead, so it
  // never completes first.  Either way the next launch may start now.
  if (!p.overlap) tc::pdl_wait();
  tc::pdl_trigger();
  const uint32_t bar0 = tc::smem_u32(&bars[0]);
  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&p.map) : "memory");
    tc::mbar_init(bar0, 1);
    tc::mbar_init(bar0 + 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    issue_panels<kTcD>(raw[0], bar0, p, p.map, f, rb, cb, tbeg);
  }
  __syncthreads();

  for (int ch = 0; ch < nchunks; ++ch) {
    const int buf = ch & 1;
    // Chunk ch+1 goes into the other buffer, free since the end of chunk ch-1.
    if (threadIdx.x == 0 && ch + 1 < nchunks)
      issue_panels<kTcD>(raw[buf ^ 1], bar0 + 8 * (buf ^ 1), p, p.map, f, rb, cb,
                         tbeg + (ch + 1) * kTcD);
    const bool got = tc::mbar_wait(bar0 + 8 * buf, (ch >> 1) & 1, nullptr);
    if (__syncthreads_or(!got)) {
      panel_timeout(p, bar0 + 8 * (buf ^ 1), ((ch + 1) >> 1) & 1, ch + 1 < nchunks);
      if (p.overlap) tc::pdl_wait();
      return;
    }
    to_words<kRows>(raw[buf][0], wrow);
    to_words<kBlk>(raw[buf][1], wcol);
    __syncthreads();
    dp4a_chunk(wrow, wcol, ty, tx, re, i1, i2);
    __syncthreads();
  }

  // Sums out, half of the block's rows at a time (rs = 0: even rows, 1: odd
  // rows): the threads stage them in shared memory (the panels are free) in
  // the buffer's order, and each of the four warps then adds two of the eight
  // staged rows with 32
  // consecutive words per instruction -- 256 contiguous bytes, where adding
  // straight from the threads' 2x2 tiles scatters every instruction over 32
  // lines (measured: the epilogue took 20 of 135 us at N=256, F=10, T=1024).
  // Time splits of one block add exactly, in any order, as does an adding
  // call; a storing call without splits stores.
  int64_t *state = (int64_t *)p.state;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool store = p.overwrite && gridDim.z == 1;
#pragma unroll
  for (int rs = 0; rs < 2; ++rs) {
    uint8_t *seg = dsm + ty * kEpiRow + tx * kEpiSeg;
#pragma unroll
    for (int cs = 0; cs < 2; ++cs)
#pragma unroll
      for (int p1 = 0; p1 < 2; ++p1)
#pragma unroll
        for (int p2 = 0; p2 < 2; ++p2) {
          const long long vr = re[rs][cs][p1][p2];
          const long long vi = (long long)i1[rs][cs][p1][p2] - (long long)i2[rs][cs][p1][p2];
          *(longlong2 *)(seg + (cs * 4 + p1 * 2 + p2) * 16) = make_longlong2(vr, vi);
        }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = warp + 4 * h;              // staged row: station i of the block
      const int i = rb * kRows + 2 * r + rs;
      if (i < p.n) {
        // the row's baselines (i, cb*32 .. cb*32+31) are 256 consecutive
        // words of the buffer; on the diagonal only columns j <= i count
        int64_t *row = state + ((long long)f * p.nbaseline + (long long)i * (i + 1) / 2 +
                                cb * kBlk) * 8;
        const int jmax = i - cb * kBlk;
#pragma unroll
        for (int it = 0; it < 8; ++it) {
          const int w = it * 32 + lane;         // word w: baseline w / 8 of the row
          if ((w >> 3) <= jmax) {
            const long long v =
                *(const long long *)(dsm + r * kEpiRow + (w >> 4) * kEpiSeg + (w & 15) * 8);
            if (store) row[w] = v;
            else atomicAdd((unsigned long long *)(row + w), (unsigned long long)v);
          }
        }
      }
    }
    __syncthreads();
  }
  if (p.overlap) tc::pdl_wait();
}

// ---------------------------------------------------------------- FP32 ----
// xGPU's float sums (omp_xengine.c:24-28) in two phases, with the same bits.
// A sample adds to each component an integer of at most 2^15 in magnitude, so
// while a float sum stays within 2^24 every one of its additions is exact, and
// any exact arithmetic gives the same value.
//  * Exact phase: chunks of 64 samples through the dp4a tile loop, into int32
//    sums that start from the buffer's.  Before a chunk the block checks that
//    none of its sums can leave [-2^24, 2^24] within it.
//  * Float phase, from the first chunk for which that check fails on: the
//    samples' exact product sums added one by one, in time order, with one
//    rounding each.
// Gaussian samples of sigma 16 stay in the exact phase for 32000 samples (an
// autocorrelation adds 512 a sample; the blocks off the diagonal stay much
// longer).  dp4a does 4 samples' products for two issue slots of the pipe that
// takes 4 x 3 float operations otherwise: N=64, F=10, T=1024 from 117 us per
// call to 33, N=256 from 354 to 110.  The float phase works on both
// column polarisations at once with packed float pairs: the float pipe's rate
// is the same, but half the instructions leave issue slots for the operand
// loads (sums past 2^24 throughout, N=64: 113 to 101 us; N=256: 354 to 285).
constexpr int kTcF = 32;                         // samples per chunk of the float phase
constexpr int kRawPanelF = kTcF * kRowBytes;     // 4 KiB
constexpr int kFloatPanel = kTcF * kBlk;         // float4 entries: [sample][slot]
constexpr int kFloatPanelRows = kTcF * kRows;    // the row block's 16 stations
constexpr int kExactLimit = 1 << 24;             // float sums up to here are exact
constexpr int kExactChunk = kTcD << 15;          // most that a chunk adds to a sum

// Two floats in one register pair: sm_100's packed float instructions round
// each half as the scalar ones do.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 halves(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// raw [sample][station][4 bytes] -> [sample][slot] {X re, Y re, X im, Y im}: the
// two column polarisations of each part side by side.
__device__ __forceinline__ void to_floats(const uint8_t *raw, float4 *fl) {
  for (int u = threadIdx.x; u < kTcF * kBlk; u += kThreads) {
    const int t = u / kBlk, q = u % kBlk, s = station_of_slot(q);
    const char4 b = *(const char4 *)(raw + t * kRowBytes + s * 4);
    fl[t * kBlk + q] = make_float4((float)b.x, (float)b.z, (float)b.y, (float)b.w);
  }
}

// The row panel, {X re, X im, Y re, Y im}: the first 16 stations of a 32-station
// panel.
__device__ __forceinline__ void to_floats_rows(const uint8_t *raw, float4 *fl) {
  for (int u = threadIdx.x; u < kTcF * kRows; u += kThreads) {
    const int t = u / kRows, q = u % kRows, s = row_station_of_slot(q);
    const char4 b = *(const char4 *)(raw + t * kRowBytes + s * 4);
    fl[t * kRows + q] = make_float4((float)b.x, (float)b.y, (float)b.z, (float)b.w);
  }
}

// Dynamic shared memory of the FP32 kernel: the dp4a kernel's panels and words,
// or the float phase's raw panels [2 buffers][row, column] and converted row
// and column panels in the same place; then four mbarriers (two a phase), what
// the CTAs of a split call tell one another, and room to align the panels to
// 128 bytes.
constexpr int kPanelsFp32 = 2 * 2 * kRawPanel + kWordPanelRows + kWordPanel;
constexpr int kBarriersFp32 = 4;
static_assert(2 * 2 * kRawPanelF + (kFloatPanelRows + kFloatPanel) * 16 <= kPanelsFp32,
              "the float phase's panels take the exact phase's place");

// i1 - i2 where only the difference is known to fit 32 bits (each half may have
// wrapped).
__device__ __forceinline__ int difference(int i1, int i2) { return (int)((unsigned)i1 - (unsigned)i2); }

constexpr int kSmemFp32 = kPanelsFp32 + 8 * kBarriersFp32 + 40 + 128;
static_assert(8 * kThreads * 16 <= 2 * 2 * kRawPanel, "the pieces' sums fit the panels");
static_assert(5 * (kSmemFp32 + 128 + 1024) <= 228 * 1024, "five FP32 CTAs per SM");

// The thread's 2x2 stations x 4 products as eight parts e = (rs, cs, p1) of
// {re, im} x p2.  buffer_slot: part e of the tile at stations i0, j0.
__device__ __forceinline__ float4 *buffer_slot(const Params &p, int f, int i0, int j0, int e) {
  const long long i = i0 + (e >> 2), j = j0 + ((e >> 1) & 1);
  return (float4 *)((float *)p.state + ((long long)f * p.nbaseline + i * (i + 1) / 2 + j) * 8) +
         (e & 1);
}

// Whether the buffer has part e (a baseline of the array, on or below the
// diagonal).
__device__ __forceinline__ bool in_buffer(const Params &p, int i0, int j0, int e) {
  const int i = i0 + (e >> 2), j = j0 + ((e >> 1) & 1);
  return i < p.n && j <= i;
}

// The sums that the call continues: the buffer's, or zeros after a clear.
__device__ __forceinline__ float4 buffer_part(const Params &p, int f, int i0, int j0, int e) {
  return !p.overwrite && in_buffer(p, i0, j0, e) ? *buffer_slot(p, f, i0, j0, e)
                                                 : make_float4(0.f, 0.f, 0.f, 0.f);
}

__device__ __forceinline__ float largest(float4 v) {
  return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
}

// The float phase: samples tbeg .. t0 + tcount - 1, one by one, into parts
// e0 .. e0 + kParts - 1 (e0 a multiple of kParts).  barf: two initialised
// mbarriers.  False: a panel never came (the error word is set).
template <int kParts>
__device__ __forceinline__ bool float_phase(const Params &p, uint8_t *dsm, uint32_t barf, int f,
                                            int rb, int cb, int tbeg, int e0,
                                            float4 (&sum)[kParts]) {
  constexpr int kR = kParts == 8 ? 2 : 1;   // row stations, column stations and row
  constexpr int kC = kParts >= 4 ? 2 : 1;   // polarisations among the parts
  constexpr int kP = kParts >= 2 ? 2 : 1;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  auto raw = (uint8_t(*)[2][kRawPanelF])dsm;
  float4 *flr = (float4 *)(dsm + 2 * 2 * kRawPanelF);   // row panel, 16 slots
  float4 *flc = flr + kFloatPanelRows;                   // column panel, 32 slots
  const float4 *row = flr + (kR == 2 ? 0 : e0 >> 2) * 8 + ty;
  const float4 *col = flc + (kC == 2 ? 0 : (e0 >> 1) & 1) * 16 + tx;
  const bool y = kP == 1 && (e0 & 1);
  const int nchunks = (p.t0 + p.tcount - tbeg + kTcF - 1) / kTcF;
  f32x2 xr[kParts], xi[kParts];   // real and imaginary sums of both column polarisations
#pragma unroll
  for (int k = 0; k < kParts; ++k) {
    xr[k] = pair(sum[k].x, sum[k].z);
    xi[k] = pair(sum[k].y, sum[k].w);
  }
  if (threadIdx.x == 0) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    issue_panels<kTcF>(raw[0], barf, p, p.map_float, f, rb, cb, tbeg);
  }
  for (int ch = 0; ch < nchunks; ++ch) {
    const int buf = ch & 1;
    // Chunk ch+1 goes into the other buffer, free since the end of chunk ch-1.
    if (threadIdx.x == 0 && ch + 1 < nchunks)
      issue_panels<kTcF>(raw[buf ^ 1], barf + 8 * (buf ^ 1), p, p.map_float, f, rb, cb,
                         tbeg + (ch + 1) * kTcF);
    const bool got = tc::mbar_wait(barf + 8 * buf, (ch >> 1) & 1, nullptr);
    if (__syncthreads_or(!got)) {
      panel_timeout(p, barf + 8 * (buf ^ 1), ((ch + 1) >> 1) & 1, ch + 1 < nchunks);
      return false;
    }
    to_floats_rows(raw[buf][0], flr);
    to_floats(raw[buf][1], flc);
    __syncthreads();
#pragma unroll 4
    for (int t = 0; t < kTcF; ++t) {
      float4 r[kR];
      f32x2 br[kC], bi[kC], nbi[kC];   // both polarisations of a column station, and -bi
#pragma unroll
      for (int q = 0; q < kR; ++q) r[q] = row[t * kRows + 8 * q];
#pragma unroll
      for (int q = 0; q < kC; ++q) {
        const float4 c = col[t * kBlk + 16 * q];
        br[q] = pair(c.x, c.y);
        bi[q] = pair(c.z, c.w);
        nbi[q] = pair(-c.z, -c.w);
      }
#pragma unroll
      for (int k = 0; k < kParts; ++k) {
        const int rs = k / (kC * kP), cs = k / kP % kC;
        const bool p1 = kP == 2 ? k % 2 == 1 : y;
        const float re = p1 ? r[rs].z : r[rs].x, im = p1 ? r[rs].w : r[rs].y;
        const f32x2 ar = pair(re, re), ai = pair(im, im);
        // A sample's two products are summed first -- exactly: products of
        // int8 values and their sums are integers below 2^24 -- and the sum
        // is added to the accumulator with one rounding.
        xr[k] = add2(xr[k], fma2(ai, bi[cs], mul2(ar, br[cs])));
        xi[k] = add2(xi[k], fma2(ai, br[cs], mul2(ar, nbi[cs])));
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < kParts; ++k) {
    const float2 re = halves(xr[k]), im = halves(xi[k]);
    sum[k] = make_float4(re.x, im.x, re.y, im.y);
  }
  return true;
}

// The whole call by one CTA: the exact phase, then the float phase.  bar0:
// four initialised mbarriers (two a phase).
__device__ __forceinline__ void fp32_whole(const Params &p, uint8_t *dsm, uint32_t bar0, int f,
                                           int rb, int cb) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;   // ty 0..7
  const int i0 = rb * kRows + 2 * ty, j0 = cb * kBlk + 2 * tx;
  auto raw = (uint8_t(*)[2][kRawPanel])dsm;
  if (threadIdx.x == 0) issue_panels<kTcD>(raw[0], bar0, p, p.map, f, rb, cb, p.t0);

  float4 sum[8];
  int ch = 0;
  {
    int4 *wrow = (int4 *)(dsm + 2 * 2 * kRawPanel);   // row words, 16 slots
    int4 *wcol = wrow + kGroups * kRows;               // column words, 32 slots
    const int nchunks = (p.tcount + kTcD - 1) / kTcD;
    int re[2][2][2][2], i1[2][2][2][2], i2[2][2][2][2];
    // The sums continue the buffer's (0 after a clear), so an integration over
    // several calls is one sum in time order.  Sums past 2^24 do not fit the
    // check below: top keeps it from passing, and the float phase reads them
    // again.
    int top = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int rs = e >> 2, cs = (e >> 1) & 1, p1 = e & 1;
      const float4 o = buffer_part(p, f, i0, j0, e);
      if (!(largest(o) <= (float)kExactLimit)) top = kExactLimit;
      re[rs][cs][p1][0] = (int)o.x;
      i1[rs][cs][p1][0] = (int)o.y;
      re[rs][cs][p1][1] = (int)o.z;
      i1[rs][cs][p1][1] = (int)o.w;
      i2[rs][cs][p1][0] = i2[rs][cs][p1][1] = 0;
    }
    int budget = 0;   // chunks that the last check covers
    for (; ch < nchunks; ++ch) {
      const int buf = ch & 1;
      if (budget == 0) {
        int m = top;
#pragma unroll
        for (int a = 0; a < 16; ++a)
          m = max(m, max(abs((&re[0][0][0][0])[a]),
                         abs(difference((&i1[0][0][0][0])[a], (&i2[0][0][0][0])[a]))));
        if (!__syncthreads_or(m > kExactLimit - 4 * kExactChunk)) budget = 4;
        else if (!__syncthreads_or(m > kExactLimit - kExactChunk)) budget = 1;
        else break;
      }
      --budget;
      // Chunk ch+1 goes into the other buffer, free since the end of chunk ch-1.
      if (threadIdx.x == 0 && ch + 1 < nchunks)
        issue_panels<kTcD>(raw[buf ^ 1], bar0 + 8 * (buf ^ 1), p, p.map, f, rb, cb,
                           p.t0 + (ch + 1) * kTcD);
      const bool got = tc::mbar_wait(bar0 + 8 * buf, (ch >> 1) & 1, nullptr);
      if (__syncthreads_or(!got)) {
        panel_timeout(p, bar0 + 8 * (buf ^ 1), ((ch + 1) >> 1) & 1, ch + 1 < nchunks);
        return;
      }
      to_words<kRows>(raw[buf][0], wrow);
      to_words<kBlk>(raw[buf][1], wcol);
      __syncthreads();
      dp4a_chunk(wrow, wcol, ty, tx, re, i1, i2);
      __syncthreads();
    }
    if (ch < nchunks) {
      // chunk ch, already on its way, lands before its place is used again
      const bool got = tc::mbar_wait(bar0 + 8 * (ch & 1), (ch >> 1) & 1, nullptr);
      if (__syncthreads_or(!got)) {
        panel_timeout(p, 0, 0, false);
        return;
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int rs = e >> 2, cs = (e >> 1) & 1, p1 = e & 1;
      sum[e] = make_float4((float)re[rs][cs][p1][0],
                           (float)difference(i1[rs][cs][p1][0], i2[rs][cs][p1][0]),
                           (float)re[rs][cs][p1][1],
                           (float)difference(i1[rs][cs][p1][1], i2[rs][cs][p1][1]));
    }
  }
  if (ch * kTcD < p.tcount) {
    if (ch == 0) {
#pragma unroll
      for (int e = 0; e < 8; ++e) sum[e] = buffer_part(p, f, i0, j0, e);
    }
    report_past(p.past);
    if (!float_phase<8>(p, dsm, bar0 + 16, f, rb, cb, p.t0 + ch * kTcD, 0, sum)) return;
  }
  tc::pdl_trigger();
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if (in_buffer(p, i0, j0, e)) *buffer_slot(p, f, i0, j0, e) = sum[e];
}

// ---- the call split over a cluster
// A launch with few blocks (small arrays, few channels) leaves SMs idle, and
// alone on its SM a block takes 2.0 us per 64 samples where the dp4a pipe
// needs 1.0.  So a cluster of kPieces CTAs shares the block:
//  * first each takes a piece of the call's samples, with exact int32 sums
//    from zero, and the pieces' sums are added through distributed shared
//    memory.  That equals the sums in time order if no partial sum could have
//    passed 2^24 anywhere in the call: within a piece each is at most |sum
//    before the piece| + sum_t |x_i| |x_j| <= |sum before the piece| + the
//    larger of the two inputs' powers in the piece (Cauchy-Schwarz).  The
//    powers come from the converted words on the way, four dp4a an item;
//  * when the buffer's sums are past 2^24 already (checked first), or the bound
//    does not hold at the end, the float phase over all samples, each CTA
//    keeping 8 / kPieces of the eight parts of every thread's tile.
// Per call in chains at N=64, F=10, T=1024: 33 us whole, 18 in four pieces; at
// N=16, F=1, T=512: 18 and 7; with samples of sigma 120, past 2^24 from the
// second call on, at N=64: 101 and 88.
struct SplitShared {
  int past;            // CTAs whose share of the buffer is past 2^24, or breaks the bound
  unsigned power[8];   // each piece's largest input power
};
static_assert(sizeof(SplitShared) <= 40, "room in the dynamic shared memory");
constexpr int kFailed = 1 << 16;   // added to past by a CTA whose panels never came

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t in_cta(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void add_in_cta(uint32_t local, uint32_t rank, unsigned v) {
  asm volatile("red.relaxed.cluster.shared::cluster.add.u32 [%0], %1;" ::"r"(in_cta(local, rank)),
               "r"(v)
               : "memory");
}
__device__ __forceinline__ int4 ld_in_cta(uint32_t local, uint32_t rank) {
  int4 v;
  asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(in_cta(local, rank))
               : "memory");
  return v;
}

// bar0: four initialised mbarriers (two for the pieces, two for the float
// phase).
template <int kPieces>
__device__ __forceinline__ void fp32_split(const Params &p, uint8_t *dsm, uint32_t bar0,
                                           SplitShared *sh, int f, int rb, int cb) {
  constexpr int kParts = 8 / kPieces;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int i0 = rb * kRows + 2 * ty, j0 = cb * kBlk + 2 * tx;
  const int z = (int)blockIdx.z;   // rank in the cluster
  const int e0 = z * kParts;       // this CTA's share of the parts
  const int tbeg = p.t0 + z * p.per, tend = min(p.t0 + p.tcount, tbeg + p.per);
  const int nchunks = tbeg < tend ? (tend - tbeg + kTcD - 1) / kTcD : 0;
  auto raw = (uint8_t(*)[2][kRawPanel])dsm;
  int4 *wrow = (int4 *)(dsm + 2 * 2 * kRawPanel);
  int4 *wcol = wrow + kGroups * kRows;
  const uint32_t past = tc::smem_u32(&sh->past), power = tc::smem_u32(&sh->power[z]);

  if (threadIdx.x == 0) {
    sh->past = 0;
    for (int q = 0; q < 8; ++q) sh->power[q] = 0;
    if (nchunks) issue_panels<kTcD>(raw[0], bar0, p, p.map, f, rb, cb, tbeg);
  }
  bool big = false;
#pragma unroll
  for (int k = 0; k < kParts; ++k)
    big |= !(largest(buffer_part(p, f, i0, j0, e0 + k)) <= (float)kExactLimit);
  big = __syncthreads_or(big);
  cluster_barrier();
  if (big && threadIdx.x < kPieces) add_in_cta(past, threadIdx.x, 1);
  cluster_barrier();
  const bool skip = sh->past != 0;
  bool ok = true;

  int re[2][2][2][2], i1[2][2][2][2], i2[2][2][2][2];
#pragma unroll
  for (int a = 0; a < 16; ++a) {
    (&re[0][0][0][0])[a] = 0;
    (&i1[0][0][0][0])[a] = 0;
    (&i2[0][0][0][0])[a] = 0;
  }
  // powers of the two inputs of the row and of the column station in the slot
  // that this thread converts (threadIdx.x % 16 and % 32)
  int prow[2] = {0, 0}, pcol[2] = {0, 0};
  const int todo = skip ? min(nchunks, 1) : nchunks;   // a skipped piece's first chunk still lands
  for (int ch = 0; ch < todo; ++ch) {
    const int buf = ch & 1;
    if (threadIdx.x == 0 && ch + 1 < todo)
      issue_panels<kTcD>(raw[buf ^ 1], bar0 + 8 * (buf ^ 1), p, p.map, f, rb, cb,
                         tbeg + (ch + 1) * kTcD);
    const bool got = tc::mbar_wait(bar0 + 8 * buf, (ch >> 1) & 1, nullptr);
    if (__syncthreads_or(!got)) {
      panel_timeout(p, bar0 + 8 * (buf ^ 1), ((ch + 1) >> 1) & 1, ch + 1 < todo);
      ok = false;
      break;
    }
    if (skip) break;
    to_words<kRows>(raw[buf][0], wrow, prow);
    to_words<kBlk>(raw[buf][1], wcol, pcol);
    __syncthreads();
    dp4a_chunk(wrow, wcol, ty, tx, re, i1, i2);
    __syncthreads();
  }
  tc::pdl_trigger();
  // The piece's sums into shared memory, part by part, 16 bytes a thread.
  int4 *stage = (int4 *)dsm;
  if (!skip) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int rs = e >> 2, cs = (e >> 1) & 1, p1 = e & 1;
      stage[e * kThreads + threadIdx.x] =
          make_int4(re[rs][cs][p1][0], difference(i1[rs][cs][p1][0], i2[rs][cs][p1][0]),
                    re[rs][cs][p1][1], difference(i1[rs][cs][p1][1], i2[rs][cs][p1][1]));
    }
    // the powers of the block's row and column inputs, where the words were
    unsigned *input = (unsigned *)wrow;
    constexpr int kInputs = 2 * (kRows + kBlk);
    if (threadIdx.x < kInputs) input[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int pol = 0; pol < 2; ++pol) {
      atomicAdd(&input[2 * (threadIdx.x & 15) + pol], (unsigned)prow[pol]);
      atomicAdd(&input[2 * (kRows + (threadIdx.x & 31)) + pol], (unsigned)pcol[pol]);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      unsigned m = 0;
      for (int q = threadIdx.x; q < kInputs; q += 32) m = max(m, input[q]);
      m = __reduce_max_sync(0xffffffffu, m);
      if (threadIdx.x < kPieces) add_in_cta(power, threadIdx.x, m);
    }
  }
  if (!ok && threadIdx.x < kPieces) add_in_cta(past, threadIdx.x, kFailed);
  cluster_barrier();
  float4 sum[kParts];
  big = false;
  if (!skip && ok) {
#pragma unroll
    for (int k = 0; k < kParts; ++k) {
      const float4 old = buffer_part(p, f, i0, j0, e0 + k);
      int4 v = make_int4((int)old.x, (int)old.y, (int)old.z, (int)old.w);
#pragma unroll
      for (int q = 0; q < kPieces; ++q) {
        // the sums before piece q, within 2^24 as long as nothing was big
        const int room = kExactLimit - (int)min(sh->power[q], 2u * kExactLimit);
        big |= max(max(abs(v.x), abs(v.y)), max(abs(v.z), abs(v.w))) > room;
        const int4 w = ld_in_cta(tc::smem_u32(&stage[(e0 + k) * kThreads + threadIdx.x]), q);
        v.x += w.x;
        v.y += w.y;
        v.z += w.z;
        v.w += w.w;
      }
      sum[k] = make_float4((float)v.x, (float)v.y, (float)v.z, (float)v.w);
    }
  }
  big = __syncthreads_or(big);
  if (big && threadIdx.x < kPieces) add_in_cta(past, threadIdx.x, 1);
  cluster_barrier();
  if (sh->past >= kFailed) return;   // the error word is set
  if (sh->past != 0) {
    report_past(p.past);
#pragma unroll
    for (int k = 0; k < kParts; ++k) sum[k] = buffer_part(p, f, i0, j0, e0 + k);
    if (!float_phase<kParts>(p, dsm, bar0 + 16, f, rb, cb, p.t0, e0, sum)) return;
  }
#pragma unroll
  for (int k = 0; k < kParts; ++k)
    if (in_buffer(p, i0, j0, e0 + k)) *buffer_slot(p, f, i0, j0, e0 + k) = sum[k];
}

template <int kPieces>
__global__ void __launch_bounds__(kThreads, 5) xengine_fp32_kernel(const __grid_constant__ Params p) {
  extern __shared__ __align__(128) uint8_t dsm_raw[];
  uint8_t *dsm = (uint8_t *)(((uintptr_t)dsm_raw + 127) & ~(uintptr_t)127);
  const uint32_t bar0 = tc::smem_u32(dsm + kPanelsFp32);
  const int f = p.f0 + (int)blockIdx.y;
  int rb, cb;   // row block of 16 stations, column block of 32
  decode_block(blockIdx.x, rb, cb);
  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&p.map) : "memory");
    for (int q = 0; q < kBarriersFp32; ++q) tc::mbar_init(bar0 + 8 * q, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // Programmatic launch: the prologue runs beside the previous kernel's end.  The
  // next grid is let in only when the sums are done: CTAs that come earlier wait on
  // whichever SMs have room, and then run as unevenly as they came (N=256, F=6,
  // T=2048: 194 us per call in chains against 136; N=128, F=20 101 against 72).
  tc::pdl_wait();
  if constexpr (kPieces > 1) {
    fp32_split<kPieces>(p, dsm, bar0, (SplitShared *)(dsm + kPanelsFp32 + 8 * kBarriersFp32), f,
                        rb, cb);
  } else {
    fp32_whole(p, dsm, bar0, f, rb, cb);
  }
}

}  // namespace plain

// Blocks of 16-station rows r and 32-station columns c <= r / 2
// (decode_block), per channel, times the time splits.
static dim3 plain_grid(const Sizes &s, int fcount, int ksplit = 1) {
  const int nr = (s.n + plain::kRows - 1) / plain::kRows;
  const int m = nr / 2;
  const int blocks = nr % 2 == 0 ? m * (m + 1) : (m + 1) * (m + 1);
  return dim3((unsigned)blocks, (unsigned)fcount, (unsigned)ksplit);
}

long long plain_blocks(const Sizes &s) {
  const dim3 g = plain_grid(s, s.f);
  return (long long)g.x * g.y;
}

// Time splits of a dp4a launch: enough CTAs for one wave of resident CTAs
// (five per SM), or for half of one when the launch may overlap the previous
// adding launch (whose last CTAs, and the next launch's, fill the rest; each
// split costs its ramp and its atomics), to the nearest count (rounded up, 720
// blocks at N=256, F=10 were cut in two for 740 places: 113.4 against 111.6 us for
// a call alone, N=176, F=20 66.9 against 61.9), at least 256 samples per split
// and at most 8 splits.
static int plain_splits(const Sizes &s, int fcount, int tcount, bool overlap) {
  const int slots = 5 * current_device_sms();   // resident dp4a CTAs
  if (!slots) return 1;
  const dim3 g = plain_grid(s, fcount);
  const long long blocks = (long long)g.x * g.y;
  const long long target = overlap ? slots / 2 : slots;
  long long k = (target + blocks / 2) / blocks;
  if (k > tcount / 256) k = tcount / 256;
  if (k > 8) k = 8;
  return k < 1 ? 1 : (int)k;
}

// Pieces of an FP32 launch (fp32_split), for 32768 samples at most (a piece's
// power stays below 2^30).  Eight or four while the CTAs still fit the SMs about
// once (5.5 each: N=128, F=10, 200 blocks, runs 40 us with four pieces, 52
// without); a piece of fewer than 256 samples (eight) or 128 (four) costs more
// in the exchange than it gains, unless the SMs are nearly empty.  Two pieces
// only there: at 288 blocks they gain nothing (N=256, F=4: 55 against 52 us) and
// the float phase loses 10%.
// past: calls of this integration went to the float phase in the middle of the array
// (some calls ago, or none yet: it only chooses the faster way to the same sums).  There
// each CTA converts all samples for its share of the parts, so that eight pieces never
// pay, and four depend on how many of their CTAs come together on an SM: all sums past
// 2^24, T=1024, us a call in chains, four pieces and one CTA a block: 84 blocks 92 and 110,
// 96 128 and 110, 120 133 and 110, 150 (more than one whole block an SM, five CTAs of
// the split) 136 and 161, 192 (a second wave of the split) 228 and 162.
static int fp32_pieces(const Sizes &s, int fcount, int tcount, bool past) {
  const int sms = current_device_sms();
  const dim3 g = plain_grid(s, fcount);
  const long long blocks = (long long)g.x * g.y;
  if (tcount > 32768) return 1;
  if (past && 40 * blocks > 23LL * sms && (blocks <= sms || 4 * blocks > 5LL * sms)) return 1;
  for (int k = past ? 4 : 8; k > 1; k /= 2) {
    const bool sparse = blocks * k <= 2LL * sms;
    const int least = k == 8 ? (sparse ? 64 : 256) : 128;
    if ((sparse || (k > 2 && 2 * blocks * k <= 11LL * sms)) && tcount / k >= least) return k;
  }
  return 1;
}

// The kernels' dynamic shared memory (45.2 KB each), allowed once per
// device.
cudaError_t plain_configure_device() {
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = (dev >= 0 && dev < kDeviceCache) ? 1ull << dev : 0;
  if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
  e = cudaFuncSetAttribute(plain::xengine_dp4a_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           plain::kSmemDp4a);
  const void *fp32[] = {(const void *)plain::xengine_fp32_kernel<1>,
                        (const void *)plain::xengine_fp32_kernel<2>,
                        (const void *)plain::xengine_fp32_kernel<4>,
                        (const void *)plain::xengine_fp32_kernel<8>};
  for (const void *k : fp32)
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, plain::kSmemFp32);
  if (e == cudaSuccess && bit) done.fetch_or(bit, std::memory_order_release);
  return e;
}

static int plain_params(plain::Params *p, const int8_t *in, const Sizes &s, int t0, int tcount,
                        void *state, int overwrite, int per, int *err, int stall, int f0) {
  if (make_panel_map(&p->map, in, s, plain::kTcD) != 0) return -1;
  p->n = s.n;
  p->f = s.f;
  p->t0 = t0;
  p->tcount = tcount;
  p->nbaseline = s.nbaseline;
  p->state = state;
  p->overwrite = overwrite;
  p->per = per;
  p->err = err;
  p->stall = stall;
  p->f0 = f0;
  p->overlap = 0;
  p->past = FloatPast{};
  return 0;
}

cudaError_t launch_plain_dp4a(const int8_t *in, const Sizes &s, int t0, int tcount,
                              int64_t *state, int overwrite, cudaStream_t st, int *err,
                              int stall, int f0, int fcount, int overlap) {
  if (fcount < 0) fcount = s.f - f0;
  if (f0 < 0 || fcount < 1 || f0 + fcount > s.f) return cudaErrorInvalidValue;
  const int ks = plain_splits(s, fcount, tcount, overlap && !overwrite);
  // samples per split: a whole number of 64-sample chunks
  int per = (tcount + ks - 1) / ks;
  per = (per + plain::kTcD - 1) / plain::kTcD * plain::kTcD;
  const int used = (tcount + per - 1) / per;
  if (used > 1 && overwrite) {   // the splits add: clear the channel range first
    const size_t per_channel = (size_t)s.state_elems / s.f;
    cudaError_t e = cudaMemsetAsync(state + (size_t)f0 * per_channel, 0,
                                    (size_t)fcount * per_channel * 8, st);
    if (e != cudaSuccess) return e;
  }
  cudaError_t e = plain_configure_device();
  if (e != cudaSuccess) return e;
  plain::Params p;
  if (plain_params(&p, in, s, t0, tcount, state, overwrite, per, err, stall, f0) != 0)
    return cudaErrorInvalidValue;
  p.overlap = (overlap && !overwrite) ? 1 : 0;
  // Programmatic launch: the grid may start beside the previous kernel's last
  // CTAs (the kernel waits for it where it must).
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = plain_grid(s, fcount, used);
  cfg.blockDim = dim3(plain::kThreads);
  cfg.dynamicSmemBytes = plain::kSmemDp4a;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, plain::xengine_dp4a_kernel, p);
}

cudaError_t launch_plain_fp32(const int8_t *in, const Sizes &s, int t0, int tcount, float *state,
                              int overwrite, cudaStream_t st, int *err, int stall, int f0,
                              int fcount, const FloatPast &past) {
  if (fcount < 0) fcount = s.f - f0;
  if (f0 < 0 || fcount < 1 || f0 + fcount > s.f) return cudaErrorInvalidValue;
  cudaError_t e = plain_configure_device();
  if (e != cudaSuccess) return e;
  const int pieces = fp32_pieces(s, fcount, tcount, past.seen);
  // samples per piece: a whole number of 64-sample chunks
  int per = (tcount + pieces - 1) / pieces;
  per = (per + plain::kTcD - 1) / plain::kTcD * plain::kTcD;
  plain::Params p;
  if (plain_params(&p, in, s, t0, tcount, state, overwrite, per, err, stall, f0) != 0 ||
      make_panel_map(&p.map_float, in, s, plain::kTcF) != 0)
    return cudaErrorInvalidValue;
  p.past = past;
  if (past.seen) p.past.word = nullptr;   // a store over the host link ends a call 3 us later
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = plain_grid(s, fcount, pieces);
  cfg.blockDim = dim3(plain::kThreads);
  cfg.dynamicSmemBytes = plain::kSmemFp32;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = (unsigned)pieces;
  cfg.attrs = attr;
  // Whole blocks that come where a split call's CTAs leave room stay crowded there (the
  // first such call 225 us for 110 at 120 blocks), so they come to an empty GPU.
  const bool plainly = past.seen && cfg.gridDim.x * cfg.gridDim.y < 4u * current_device_sms();
  cfg.numAttrs = pieces > 1 ? 2 : plainly ? 0 : 1;
  switch (pieces) {
    case 8: return cudaLaunchKernelEx(&cfg, plain::xengine_fp32_kernel<8>, p);
    case 4: return cudaLaunchKernelEx(&cfg, plain::xengine_fp32_kernel<4>, p);
    case 2: return cudaLaunchKernelEx(&cfg, plain::xengine_fp32_kernel<2>, p);
    default: return cudaLaunchKernelEx(&cfg, plain::xengine_fp32_kernel<1>, p);
  }
}

}  // namespace xgpu
