// format.cu -- device-side input conversion, output formatting and synthetic
// input.
//
// Output orders (xgpu.h:45-47) are produced on the device from the triangular
// integration buffer, so a dump moves exactly the requested layout to the host.
// The index maps follow the reference's writers and reorderers:
//   TRIANGULAR_ORDER            kernel.cuh:96-117, cpu_util.c:161-162
//   REAL_IMAG_TRIANGULAR_ORDER  kernel.cuh:72-95,  cpu_util.c:112-115
//   REGISTER_TILE_...           kernel.cuh:49-71,  cpu_util.c:66-79
#include <math.h>

#include "internal.h"
#include "packed4.cuh"
#include "tc_common.cuh"

namespace xgpu {

namespace fmt {

__device__ __forceinline__ uint32_t dump_word(long long v, int out_type) {
  if (out_type == XGPU_INT32) return (uint32_t)(unsigned long long)v;  // wraps like int32 sums
  return __float_as_uint(__ll2float_rn(v));
}

__device__ __forceinline__ uint32_t dump_word(float v, int out_type) {
  if (out_type == XGPU_INT32) return (uint32_t)__float2int_rn(v);
  return __float_as_uint(v);
}

// Register-tile order: baseline (i, j) in position k of a channel's slots, 2 x 2
// planes of tiles (I, J) as rows of a triangle; j > i where a slot holds none.
__device__ __forceinline__ void tile_slot(int k, int tiles, int &i, int &j) {
  const int slot = k / tiles, q = k - slot * tiles;
  int I = (int)((sqrtf(8.0f * (float)q + 1.0f) - 1.0f) * 0.5f);
  while (I * (I + 1) / 2 > q) --I;
  while ((I + 1) * (I + 2) / 2 <= q) ++I;
  i = 2 * I + (slot & 1);
  j = 2 * (q - I * (I + 1) / 2) + (slot >> 1);
}

// A dump into device memory: channel f0 + blockIdx.y, one thread per product,
// striding over the channel in the order of the output (32-bit index arithmetic
// within the channel); register-tile order's slots without a baseline get
// zeros.  Programmatic: the launch latency passes under the previous kernel's
// end.  Memory-bound: 16 (int64) or 8 (float) bytes in, 8 out.
template <bool kFloat, bool kTiles>
__global__ void __launch_bounds__(256) format_kernel(const void *state, int n, int nbaseline,
                                                     int f0, const DumpOut o) {
  tc::pdl_wait();
  tc::pdl_trigger();
  const int f = f0 + (int)blockIdx.y;
  const int tiles = (n / 2 + 1) * (n / 4);
  const int words = 4 * (kTiles ? 4 * tiles : nbaseline);
  const long long base = (long long)f * nbaseline * 4;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < words; v += gridDim.x * blockDim.x) {
    int u = v;   // product within the channel, triangular order
    if (kTiles) {
      int i, j;
      tile_slot(v >> 2, tiles, i, j);
      u = j <= i ? 4 * (i * (i + 1) / 2 + j) + (v & 3) : -1;
    }
    uint32_t re = 0, im = 0;
    if (!kTiles || u >= 0) {
      if (kFloat) {
        const float2 x = ((const float2 *)state)[base + u];
        re = dump_word(x.x, o.out_type);
        im = dump_word(x.y, o.out_type);
      } else {
        const longlong2 x = ((const longlong2 *)state)[base + u];
        re = dump_word(x.x, o.out_type);
        im = dump_word(x.y, o.out_type);
      }
    }
    if (!kTiles && o.order == TRIANGULAR_ORDER) {
      *(uint2 *)(o.out + 2 * (base + v)) = make_uint2(re, im);
    } else {
      const long long w = (long long)f * words + v;
      o.out[w] = re;
      o.out[w + o.mat_length] = im;
    }
  }
}

// A dump into host memory that the device maps (16-byte aligned): 16 bytes of
// the output per thread and step, a warp's 512 contiguous.  The host link sets
// the pace: 10.5 MB take 209 us for any grid from 2048 threads on, 50 GB/s.
// What the grid decides is how much waits for it: with the output's lines last
// written by 16 processor cores, 75,000 threads still take 211 us, 2048 threads
// 315 (and a copy engine, 190 us on untouched lines, 350).  Stores that wait
// hold up every other SM's memory accesses meanwhile (a 256 MB read, 67 us
// alone, took 248 beside them), so nothing is gained by running an engine launch
// beside a dump.  Against one 8-byte store per product (16 blocks of 256 threads
// per SM): dumps of 10.5, 16.9 and 6.5 MB 222 to 215, 346 to 338 and 145 to 139
// us; a dumping call over host input (register-tile order, formatted in device
// memory and copied before) 398 to 361 us.
constexpr int kHostThreads = 128;
constexpr int kHostBlocks = 4 * 148;
constexpr long long kHostSmall = 512 << 10;   // bytes of output below which format_kernel's
                                              // shorter code is through first (a call and a
                                              // 33 KB dump: 22 us against 26)
template <bool kFloat, bool kTiles>
__global__ void __launch_bounds__(kHostThreads)
    format_host_kernel(const void *state, int n, int nbaseline, int f0, int fcount,
                       const DumpOut o) {
  tc::pdl_wait();
  tc::pdl_trigger();
  constexpr int kSteps = 4;   // loads of four steps in flight per thread
  const int tiles = (n / 2 + 1) * (n / 4);
  const int slots = kTiles ? 4 * tiles : nbaseline;   // baselines' places per channel
  const bool planes = kTiles || o.order != TRIANGULAR_ORDER;
  const int each = planes ? 4 : 2;                    // products in 16 bytes
  const long long first = (long long)f0 * slots * 4, total = (long long)fcount * slots * 4;
  const long long stride = (long long)gridDim.x * kHostThreads;
  // product `at` in triangular order: its two words
  auto words = [&](long long at, uint32_t &re, uint32_t &im) {
    if (kFloat) {
      const float2 x = ((const float2 *)state)[at];
      re = dump_word(x.x, o.out_type);
      im = dump_word(x.y, o.out_type);
    } else {
      const longlong2 x = ((const longlong2 *)state)[at];
      re = dump_word(x.x, o.out_type);
      im = dump_word(x.y, o.out_type);
    }
  };
  for (long long u0 = blockIdx.x * kHostThreads + threadIdx.x; u0 * each < total;
       u0 += kSteps * stride) {
    uint32_t re[kSteps][4], im[kSteps][4];
#pragma unroll
    for (int s = 0; s < kSteps; ++s) {
      const long long v = (u0 + s * stride) * each;   // product's place in the output
      if (v >= total) break;
      long long at = first + v;
      bool live = true;
      if (kTiles) {
        const int f = f0 + (int)((v >> 2) / slots), q = (int)((v >> 2) % slots);
        int i, j;
        tile_slot(q, tiles, i, j);
        live = j <= i;
        at = ((long long)f * nbaseline + i * (i + 1) / 2 + j) * 4;
      }
#pragma unroll
      for (int pp = 0; pp < 4; ++pp) {
        re[s][pp] = im[s][pp] = 0;
        if (live && pp < each) words(at + pp, re[s][pp], im[s][pp]);
      }
    }
#pragma unroll
    for (int s = 0; s < kSteps; ++s) {
      const long long v = (u0 + s * stride) * each;
      if (v >= total) break;
      uint32_t *d = o.out + (planes ? 1 : 2) * (first + v);
      if (planes) {
        *(uint4 *)d = make_uint4(re[s][0], re[s][1], re[s][2], re[s][3]);
        *(uint4 *)(d + o.mat_length) = make_uint4(im[s][0], im[s][1], im[s][2], im[s][3]);
      } else {
        *(uint4 *)d = make_uint4(re[s][0], im[s][0], re[s][1], im[s][1]);
      }
    }
  }
}

static auto pick_format(int state_is_float, bool tiles) {
  return state_is_float ? (tiles ? format_kernel<true, true> : format_kernel<true, false>)
                        : (tiles ? format_kernel<false, true> : format_kernel<false, false>);
}
static auto pick_format_host(int state_is_float, bool tiles) {
  return state_is_float
             ? (tiles ? format_host_kernel<true, true> : format_host_kernel<true, false>)
             : (tiles ? format_host_kernel<false, true> : format_host_kernel<false, false>);
}

// Conversions stand between two engine launches.  Beside the engine launch before it
// a conversion touches neither that one's input nor its sums, so it starts at once
// and only ends after it (one block's wait keeps the grid; the others leave their
// places to the rest); the engine launch behind it waits for the conversion, and so
// for both.  That launch comes early, its prologue under the conversion, where its CTAs
// can only spread evenly: one fills an SM, or they fill all places.  CTAs of smaller
// grids, several of which fit an SM, would settle where the conversion's blocks leave
// room and then run as unevenly (kConvertLate: they come when it is done).  Plain
// engines, us a call in chains early and late: dp4a, swizzled, N=64, F=10, T=1024 30.2
// and 17.9, N=96, F=16, T=512 31.1 and 22.7, N=256, F=10 (720 CTAs) 106.1 and 107.2;
// FP32, packed, N=128, F=10 50.9 and 40.9, N=176, F=13, T=1552 172 and 143.
__device__ __forceinline__ void begin_conversion(int mode) {
  if (!(mode & kConvertBeside)) tc::pdl_wait();
  if (!(mode & kConvertLate)) tc::pdl_trigger();
}
__device__ __forceinline__ void end_conversion(int mode) {
  if ((mode & kConvertBeside) && blockIdx.x == 0) tc::pdl_wait();
}

// Item u of the compact input (rows of `row` items) in the caller's.  kBand: its rows
// are `pitch` items apart, the band's, of which the context correlates a range; only
// then is the division needed before the load can start.  (With it for every input,
// and 40 registers a thread, six blocks an SM instead of eight, the un-swizzle of
// N=512, F=64, T=4096 took 194 us alone, and the un-blocking 177; 172 and 168 so.)
template <bool kBand>
struct Rows {
  long long row, pitch;
  __device__ __forceinline__ long long at(long long u) const {
    return kBand ? u / row * pitch + u % row : u;
  }
};

// 16 packed samples per thread: one 16-byte load, two 16-byte stores.
template <bool kBand>
__global__ void __launch_bounds__(256, 8)
    unpack4_kernel(const uint4 *in, uint4 *out, long long nquads, Rows<kBand> rows, int mode) {
  begin_conversion(mode);
  for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < nquads;
       u += (long long)gridDim.x * blockDim.x) {
    const uint4 w = in[rows.at(u)];
    const uint2 a = expand_packed4(w.x), b = expand_packed4(w.y), c = expand_packed4(w.z),
                d = expand_packed4(w.w);
    out[2 * u] = make_uint4(a.x, a.y, b.x, b.y);
    out[2 * u + 1] = make_uint4(c.x, c.y, d.x, d.y);
  }
  end_conversion(mode);
}

// xgpuSwizzleInput's layout (cpu_util.c:235-255) back to [t][f][s][p][c]:
// byte e of row-group tq holds samples 4tq..4tq+3 of input byte e.  One thread
// takes 16 bytes (input bytes 4e4..4e4+3, four samples each), transposes them
// 4x4 with byte permutes, and writes one 4-byte word to each of the four
// sample rows (consecutive threads write consecutive words of a row).
template <bool kBand>
__global__ void __launch_bounds__(256, 8)
    unswizzle_kernel(const uint4 *in, uint32_t *out, long long quads, Rows<kBand> rows, int mode) {
  begin_conversion(mode);
  const long long row_words = rows.row;   // f*n, 4 bytes per station; quads = (t/4) * row_words
  for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < quads;
       u += (long long)gridDim.x * blockDim.x) {
    const uint4 w = in[rows.at(u)];
    const long long tq = u / row_words, e4 = u - tq * row_words;
    const uint32_t lo01 = __byte_perm(w.x, w.y, 0x5140), hi01 = __byte_perm(w.x, w.y, 0x7362);
    const uint32_t lo23 = __byte_perm(w.z, w.w, 0x5140), hi23 = __byte_perm(w.z, w.w, 0x7362);
    uint32_t *o = out + 4 * tq * row_words + e4;
    o[0] = __byte_perm(lo01, lo23, 0x5410);
    o[row_words] = __byte_perm(lo01, lo23, 0x7632);
    o[2 * row_words] = __byte_perm(hi01, hi23, 0x5410);
    o[3 * row_words] = __byte_perm(hi01, hi23, 0x7632);
  }
  end_conversion(mode);
}

// xGPU's COMPLEX_BLOCK_SIZE=32 input (read by omp_xengine.c:61-78,
// shared_transfer_4.cuh:69-86) -> [t][f][s][p]{re,im}.  A 64-byte block holds
// 16 consecutive (t,f,s) stations: {X.re,Y.re} pairs in bytes 0-31, {X.im,Y.im}
// pairs in bytes 32-63.  One thread turns 4 stations (8 + 8 bytes) into 16.
template <bool kBand>
__global__ void __launch_bounds__(256, 8)
    unblock32_kernel(const uint2 *in, uint4 *out, long long quads, Rows<kBand> rows, int mode) {
  begin_conversion(mode);
  for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < quads;
       u += (long long)gridDim.x * blockDim.x) {
    const long long blk = rows.at(u >> 2);   // rows of whole blocks (n is a multiple of 16)
    const int q = (int)(u & 3);
    const uint2 re = in[blk * 8 + q];      // bytes 8q .. 8q+7 of the block
    const uint2 im = in[blk * 8 + 4 + q];  // bytes 32+8q ..
    uint4 o;
    o.x = __byte_perm(re.x, im.x, 0x5140);
    o.y = __byte_perm(re.x, im.x, 0x7362);
    o.z = __byte_perm(re.y, im.y, 0x5140);
    o.w = __byte_perm(re.y, im.y, 0x7362);
    out[u] = o;
  }
  end_conversion(mode);
}

// Seeded synthetic bytes; the same hash and tables as the host generator.
struct GenParams {
  uint32_t thr[254];
  int kind;
  unsigned long long seed;
};

__device__ __forceinline__ uint32_t hash32(unsigned long long seed, unsigned long long n) {
  unsigned long long z = seed * 0x9E3779B97F4A7C15ull + n + 0x632BE59BD9B4E019ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (uint32_t)(z >> 32);
}

__device__ __forceinline__ int8_t gen_byte(const GenParams &g, const uint32_t *thr,
                                           unsigned long long n) {
  const uint32_t u = hash32(g.seed, n);
  if (g.kind == 0) {
    int lo = 0, hi = 254;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (u < thr[mid]) hi = mid; else lo = mid + 1;
    }
    return (int8_t)(lo - 127);
  } else if (g.kind == 1) {
    const uint32_t v = hash32(g.seed ^ 0x5A5A5A5A5A5A5A5Aull, n);
    const int re = (int)(((unsigned long long)u * 15u) >> 32) - 7;
    const int im = (int)(((unsigned long long)v * 15u) >> 32) - 7;
    return (int8_t)(((re & 0xF) << 4) | (im & 0xF));
  }
  return (int8_t)((int)(((unsigned long long)u * 15u) >> 32) - 7);
}

__global__ void generate_kernel(int8_t *out, unsigned long long nbytes, const GenParams g) {
  __shared__ uint32_t thr[254];
  for (int q = threadIdx.x; q < 254; q += blockDim.x) thr[q] = g.thr[q];
  __syncthreads();
  const unsigned long long nwords = nbytes / 4;
  for (unsigned long long w = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
       w < nwords; w += (unsigned long long)gridDim.x * blockDim.x) {
    uint32_t v = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) v |= (uint32_t)(uint8_t)gen_byte(g, thr, 4 * w + b) << (8 * b);
    ((uint32_t *)out)[w] = v;
  }
  if (blockIdx.x == 0)
    for (unsigned long long n = nwords * 4 + threadIdx.x; n < nbytes; n += blockDim.x)
      out[n] = gen_byte(g, thr, n);
}

static unsigned grid_for(long long work, int threads) {
  long long b = (work + threads - 1) / threads;
  if (b > 148LL * 16) b = 148LL * 16;
  if (b < 1) b = 1;
  return (unsigned)b;
}

}  // namespace fmt

cudaError_t launch_format(const void *state, int state_is_float, const Sizes &s, const DumpOut &o,
                          cudaStream_t st, int f0, int fcount, bool host_out) {
  if (fcount < 0) fcount = s.f - f0;
  if (f0 < 0 || fcount < 1 || f0 + fcount > s.f) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const bool tiles = o.order == REGISTER_TILE_TRIANGULAR_ORDER;
  if (host_out && ((uintptr_t)o.out & 15) == 0 &&
      s.mat_length / s.f * fcount * 8 >= fmt::kHostSmall) {
    const long long blocks =
        (s.mat_length / s.f * fcount / 2 + fmt::kHostThreads - 1) / fmt::kHostThreads;
    cfg.gridDim = dim3((unsigned)(blocks < fmt::kHostBlocks ? blocks : fmt::kHostBlocks));
    cfg.blockDim = dim3(fmt::kHostThreads);
    return cudaLaunchKernelEx(&cfg, fmt::pick_format_host(state_is_float, tiles), state, s.n,
                              (int)s.nbaseline, f0, fcount, o);
  }
  // about 16 blocks per SM in all, at least one per channel
  const int blocks = (int)((s.mat_length / s.f + 255) / 256);
  const int most = (148 * 16 + fcount - 1) / fcount;
  cfg.gridDim = dim3((unsigned)(blocks < most ? blocks : most), (unsigned)fcount);
  return cudaLaunchKernelEx(&cfg, fmt::pick_format(state_is_float, tiles), state, s.n,
                            (int)s.nbaseline, f0, o);
}

// A launch of one of the conversions over `work` thread items, of s's input.
// Programmatic, except for a long one with nothing to run beside: its blocks would
// come where the engine launch before it leaves room, and then run as unevenly as
// they came (un-swizzle and engine of N=512, T=4096 on a caller's stream: F=64 622 us
// a call, 603 launched plainly, F=16 162 and 159; N=256, F=64, T=1024, 67 MB, 91 either
// way, F=10 19.7 and 20.7; the other formats gain and lose 1% to 2%).
template <class... A>
static cudaError_t launch_conversion(void (*kernel)(A..., int), long long work, const Sizes &s,
                                     int mode, cudaStream_t st, const A &...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(fmt::grid_for(work, 256));
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (mode & kConvertBeside) || 2 * s.vec_length < 128LL << 20 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args..., mode);
}

template <bool kBand>
static cudaError_t load_conversion_kernel(int input_format) {
  switch (input_format) {
    case XGPU_INPUT_PACKED4: return load_kernel((const void *)fmt::unpack4_kernel<kBand>);
    case XGPU_INPUT_DP4A_SWIZZLED: return load_kernel((const void *)fmt::unswizzle_kernel<kBand>);
    case XGPU_INPUT_BLOCK32: return load_kernel((const void *)fmt::unblock32_kernel<kBand>);
    default: return cudaSuccess;
  }
}

cudaError_t load_conversion(int input_format, const Sizes &s) {
  const cudaError_t e = load_conversion_kernel<false>(input_format);
  return e != cudaSuccess || s.fin == s.f ? e : load_conversion_kernel<true>(input_format);
}

cudaError_t load_format(int state_is_float, int order) {
  const bool tiles = order == REGISTER_TILE_TRIANGULAR_ORDER;
  const cudaError_t e = load_kernel((const void *)fmt::pick_format(state_is_float, tiles));
  return e != cudaSuccess ? e
                          : load_kernel((const void *)fmt::pick_format_host(state_is_float, tiles));
}

cudaError_t launch_unpack4(const uint8_t *in, int8_t *out, const Sizes &s, cudaStream_t st,
                           int mode) {
  // 2n bytes a channel, n a multiple of 16
  const long long row = (long long)s.f * s.n / 8, pitch = (long long)s.fin * s.n / 8;
  const long long quads = row * s.t;
  const uint4 *from = (const uint4 *)in;
  uint4 *to = (uint4 *)out;
  if (pitch == row)
    return launch_conversion<const uint4 *, uint4 *, long long, fmt::Rows<false>>(
        fmt::unpack4_kernel<false>, quads, s, mode, st, from, to, quads, {row, pitch});
  return launch_conversion<const uint4 *, uint4 *, long long, fmt::Rows<true>>(
      fmt::unpack4_kernel<true>, quads, s, mode, st, from, to, quads, {row, pitch});
}

cudaError_t launch_unswizzle_dp4a(const int8_t *in, int8_t *out, const Sizes &s, cudaStream_t st,
                                  int mode) {
  // t is a multiple of 4 (ntimepipe % 16 == 0)
  const long long row = (long long)s.f * s.n, pitch = (long long)s.fin * s.n;
  const long long quads = (long long)(s.t / 4) * row;
  const uint4 *from = (const uint4 *)in;
  uint32_t *to = (uint32_t *)out;
  if (pitch == row)
    return launch_conversion<const uint4 *, uint32_t *, long long, fmt::Rows<false>>(
        fmt::unswizzle_kernel<false>, quads, s, mode, st, from, to, quads, {row, pitch});
  return launch_conversion<const uint4 *, uint32_t *, long long, fmt::Rows<true>>(
      fmt::unswizzle_kernel<true>, quads, s, mode, st, from, to, quads, {row, pitch});
}

cudaError_t launch_unblock32(const int8_t *in, int8_t *out, const Sizes &s, cudaStream_t st,
                             int mode) {
  // blocks of 16 stations
  const long long row = (long long)s.f * s.n / 16, pitch = (long long)s.fin * s.n / 16;
  const long long quads = 4 * row * s.t;
  const uint2 *from = (const uint2 *)in;
  uint4 *to = (uint4 *)out;
  if (pitch == row)
    return launch_conversion<const uint2 *, uint4 *, long long, fmt::Rows<false>>(
        fmt::unblock32_kernel<false>, quads, s, mode, st, from, to, quads, {row, pitch});
  return launch_conversion<const uint2 *, uint4 *, long long, fmt::Rows<true>>(
      fmt::unblock32_kernel<true>, quads, s, mode, st, from, to, quads, {row, pitch});
}

void gauss_thresholds(double sigma, uint32_t thr[254]) {
  for (int k = -127; k < 127; k++) {
    double pr = 0.5 * erfc(-((k + 0.5) / sigma) / sqrt(2.0));
    double sc = floor(pr * 4294967296.0);
    if (sc > 4294967295.0) sc = 4294967295.0;
    if (sc < 0) sc = 0;
    thr[k + 127] = (uint32_t)sc;
  }
}

cudaError_t launch_generate(void *out, size_t nbytes, int kind, unsigned long long seed,
                            double sigma, cudaStream_t st) {
  fmt::GenParams g;
  g.kind = kind;
  g.seed = seed;
  if (kind == 0) gauss_thresholds(sigma, g.thr);
  else for (int q = 0; q < 254; ++q) g.thr[q] = 0;
  fmt::generate_kernel<<<fmt::grid_for((long long)(nbytes / 4) + 1, 256), 256, 0, st>>>(
      (int8_t *)out, (unsigned long long)nbytes, g);
  return cudaGetLastError();
}

}  // namespace xgpu
