// PNG encoding of the export's interleaved RGB rows, on the device.
//
// Replaces the PNG arms of export::encode (crates/core/src/export.rs:176-211):
// the reference hands tightly packed 8-bit or 16-bit RGB rows, the ICC
// profile of the output colour space and optional EXIF to the `image`
// crate's PngEncoder (image 0.25, Cargo.toml:39; not vendored). The file here
// decodes to exactly those samples and carries the same metadata chunks; the
// compressed bytes are this encoder's own (any PNG encoder's are).
//
// Six launches on the context's stream:
//  1. png_filter_kernel   one CTA per scanline: PNG filter selection by the
//                         minimum sum of absolute filtered values (the
//                         heuristic the PNG specification recommends, ties to
//                         the lower filter type), then the filtered scanline
//                         with its filter byte into the stream buffer;
//  2. png_histogram_kernel  one CTA per 32 KiB segment of the stream: the
//                         segment's token (literal / run) symbol counts and
//                         Adler-32 partial sums;
//  3. png_code_kernel     one warp per segment: Huffman code and block header;
//  4. png_pack_kernel     one CTA per segment: the byte-aligned deflate block
//                         (deflate.cuh) into the segment's slot;
//  5. png_layout_kernel   one CTA: prefix sum of the IDAT chunk sizes, the
//                         stream's Adler-32, the IEND chunk;
//  6. png_chunk_kernel    one CTA per segment: the IDAT chunk (length, type,
//                         zlib header on the first, Adler-32 on the last) with
//                         its CRC-32, stored at its offset in the file.
// The signature, IHDR, iCCP and eXIf chunks are built on the host and copied
// in front. The stream is HBM-resident byte work: every kernel reads its bytes
// once with coalesced accesses and stages them in shared memory.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "deflate.cuh"
#include "rd_internal.cuh"

namespace rd {
namespace {

using namespace png;

constexpr unsigned FULL_MASK = 0xFFFFFFFFu;

// ---- 1. scanline filters ----------------------------------------------------
// Issue slots bound this pass: a 16-bit 24 MP image has 146 MB to filter five
// ways. Filtered bytes are formed two to a register as f16 numbers, which hold
// these whole numbers exactly and have subtraction, absolute value, minimum and
// comparison in one instruction each; the byte-SIMD intrinsics are sequences.
// Scanlines are staged as they lie in memory, by 16-byte asynchronous copies,
// and aligned on reading. At 16-bit 24 MP
// the pass took 0.65 ms with the byte-SIMD intrinsics and a byte-wise staging,
// now 0.33.
constexpr int FILTER_THREADS = 256;
constexpr int FILTER_TILE = 8192;
constexpr int FILTER_BUF = FILTER_TILE + 64;  // the tile, a pixel and an alignment in front, a word behind

// Bytes 0, 1 (half 0) or 2, 3 (half 1) of w as the f16 pair 1024 + byte.
__device__ __forceinline__ uint32_t spread(uint32_t w, int half) {
  return __byte_perm(w, 0x64646464u, half ? 0x4342u : 0x4140u);
}
__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }
__device__ __forceinline__ uint32_t as_word(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }
__device__ __forceinline__ __half2 diff(uint32_t x, uint32_t y) { return __hsub2(as_half2(x), as_half2(y)); }

// The Paeth predictor of two spread bytes, spread: the neighbour closest to
// p = a + b - c, ties to a, then b; |p - a| = |b - c|, |p - b| = |a - c|,
// |p - c| = |(a - c) + (b - c)|.
__device__ __forceinline__ uint32_t paeth2(uint32_t a, uint32_t b, uint32_t c) {
  const __half2 da = diff(a, c), db = diff(b, c);
  const __half2 pa = __habs2(db), pb = __habs2(da), pc = __habs2(__hadd2(da, db));
  const uint32_t use_a = __hle2_mask(pa, __hmin2(pb, pc)), use_b = __hle2_mask(pb, pc);
  return (a & use_a) | (~use_a & ((b & use_b) | (c & ~use_b)));
}
// floor((a + b) / 2) per byte.
__device__ __forceinline__ uint32_t average4(uint32_t a, uint32_t b) { return (a & b) + (((a ^ b) >> 1) & 0x7F7F7F7Fu); }

// Adds the magnitudes of two filtered bytes read as signed numbers,
// min(|d|, 256 - |d|) of the difference d, each with BIAS on top.
constexpr uint32_t BIAS = 0x6400u;  // the bits of 1024
__device__ __forceinline__ void add_magnitudes(uint32_t& sum, __half2 d) {
  const __half2 m = __hmin2(__hadd2(__habs2(d), __float2half2_rn(1024.0f)),
                            __hsub2(__float2half2_rn(1280.0f), __habs2(d)));
  sum = __dp2a_lo(as_word(m), 0x0101u, sum);
}

__device__ __forceinline__ uint32_t filtered4(int type, uint32_t x, uint32_t a, uint32_t b, uint32_t c) {
  uint32_t p = 0;
  if (type == 1) p = a;
  else if (type == 2) p = b;
  else if (type == 3) p = average4(a, b);
  else if (type == 4)
    p = __byte_perm(paeth2(spread(a, 0), spread(b, 0), spread(c, 0)), paeth2(spread(a, 1), spread(b, 1), spread(c, 1)),
                    0x6420u);
  return __vsub4(x, p);
}

// One scanline's part of a tile in shared memory, as it lies in memory: byte
// p of the line (from BPP before the tile on) is at offset + p - t0.
struct LineTile {
  const uint32_t* words;
  int offset;
  // Line bytes [t0 + at, t0 + at + 4); 16-bit samples most significant byte first.
  template <bool WIDE>
  __device__ __forceinline__ uint32_t word(int at) const {
    const int o = offset + at;
    const uint32_t w = __funnelshift_r(words[o >> 2], words[(o >> 2) + 1], 8 * (o & 3));
    return WIDE ? __byte_perm(w, 0u, 0x2301u) : w;
  }
};

// Starts the copy of line r's bytes [t0 - BPP, t0 + count) (and what shares
// their 16 bytes) into buf. Only whole 16 bytes inside the image are copied so;
// at the image's ends the bytes go one by one.
template <bool WIDE>
__device__ __forceinline__ LineTile stage_line(const uint8_t* __restrict__ rgb, int64_t rb, int rows, int r, int64_t t0,
                                               int count, uint8_t* buf) {
  constexpr int BPP = WIDE ? 6 : 3;
  const uintptr_t image = reinterpret_cast<uintptr_t>(rgb), image_end = image + (uint64_t)rows * (uint64_t)rb;
  const uintptr_t at = image + (uint64_t)r * (uint64_t)rb + (uint64_t)t0;
  const uintptr_t begin = (at - BPP) & ~(uintptr_t)15, end = at + count;
  for (int v = threadIdx.x; begin + 16 * (uintptr_t)v < end; v += FILTER_THREADS) {
    const uintptr_t from = begin + 16 * (uintptr_t)v;
    if (from >= image && from + 16 <= image_end) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(buf + 16 * v)),
                   "l"(from) : "memory");
    } else {
      for (int i = 0; i < 16; ++i) {
        const uintptr_t m = from + i;
        if (m >= image && m < image_end) buf[16 * v + i] = *reinterpret_cast<const uint8_t*>(m);
      }
    }
  }
  return LineTile{reinterpret_cast<const uint32_t*>(buf), (int)(at - begin)};
}

template <bool WIDE>
__global__ void __launch_bounds__(FILTER_THREADS) png_filter_kernel(const void* __restrict__ rgb, int W,
                                                                    uint8_t* __restrict__ stream) {
  constexpr int BPP = WIDE ? 6 : 3;
  __shared__ __align__(16) uint8_t cur_buf[FILTER_BUF];
  __shared__ __align__(16) uint8_t up_buf[FILTER_BUF];
  __shared__ __align__(16) uint32_t done[FILTER_TILE / 4 + 1];
  __shared__ unsigned long long part[FILTER_THREADS / 32][5];
  __shared__ int s_type;
  const int r = blockIdx.x, rows = gridDim.x;
  const int64_t rb = (int64_t)W * BPP;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint8_t* pixels = static_cast<const uint8_t*>(rgb);
  LineTile cur, up;
  auto stage = [&](int64_t t0, int count) {
    cur = stage_line<WIDE>(pixels, rb, rows, r, t0, count, cur_buf);
    if (r > 0) up = stage_line<WIDE>(pixels, rb, rows, r - 1, t0, count, up_buf);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
  };
  // Word k of a tile: bytes 4k..4k+3 of it (x), the bytes a pixel before (a),
  // and the same from the line above (b, c); zero outside the image and past
  // the line.
  auto words = [&](int64_t t0, int count, int k, uint32_t& x, uint32_t& a, uint32_t& b, uint32_t& c) {
    x = cur.template word<WIDE>(4 * k);
    a = cur.template word<WIDE>(4 * k - BPP);
    b = c = 0u;
    if (r > 0) {
      b = up.template word<WIDE>(4 * k);
      c = up.template word<WIDE>(4 * k - BPP);
    }
    if (t0 == 0 && 4 * k < BPP) {
      const uint32_t inside = 4 * k + 4 <= BPP ? 0u : 0xFFFFFFFFu << (8 * (BPP - 4 * k));
      a &= inside;
      c &= inside;
    }
    if (count - 4 * k < 4) {
      const uint32_t keep = (1u << (8 * (count - 4 * k))) - 1u;
      x &= keep;
      a &= keep;
      b &= keep;
      c &= keep;
    }
  };

  unsigned long long sums[5] = {0, 0, 0, 0, 0};
  for (int64_t t0 = 0; t0 < rb; t0 += FILTER_TILE) {
    const int count = (int)min((int64_t)FILTER_TILE, rb - t0);
    stage(t0, count);
    uint32_t s[5] = {0, 0, 0, 0, 0}, n = 0;
    for (int k = tid; 4 * k < count; k += FILTER_THREADS, ++n) {
      uint32_t x, a, b, c;
      words(t0, count, k, x, a, b, c);
      const uint32_t mean = average4(a, b);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t X = spread(x, h), A = spread(a, h), B = spread(b, h), C = spread(c, h);
        add_magnitudes(s[0], diff(X, BIAS | BIAS << 16));
        add_magnitudes(s[1], diff(X, A));
        add_magnitudes(s[2], diff(X, B));
        add_magnitudes(s[3], diff(X, spread(mean, h)));
        add_magnitudes(s[4], diff(X, paeth2(A, B, C)));
      }
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) sums[k] += s[k] - n * (4u * BIAS);
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    unsigned long long v = sums[k];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(FULL_MASK, v, o);
    if (lane == 0) part[warp][k] = v;
  }
  __syncthreads();
  if (tid == 0) {
    int best = 0;
    unsigned long long best_sum = 0;
    for (int k = 0; k < 5; ++k) {
      unsigned long long v = 0;
      for (int w = 0; w < FILTER_THREADS / 32; ++w) v += part[w][k];
      if (k == 0 || v < best_sum) {
        best = k;
        best_sum = v;
      }
    }
    s_type = best;
  }
  __syncthreads();
  const int type = s_type;
  uint8_t* line = stream + (uint64_t)r * (uint64_t)(1 + rb);
  if (tid == 0) line[0] = (uint8_t)type;
  for (int64_t t0 = 0; t0 < rb; t0 += FILTER_TILE) {
    const int count = (int)min((int64_t)FILTER_TILE, rb - t0);
    // A single tile is still resident from the selection pass.
    if (rb > FILTER_TILE) stage(t0, count);
    for (int k = tid; 4 * k < count; k += FILTER_THREADS) {
      uint32_t x, a, b, c;
      words(t0, count, k, x, a, b, c);
      done[k] = filtered4(type, x, a, b, c);
    }
    __syncthreads();
    // Whole words of the stream, the bytes at either end one by one.
    uint8_t* dst = line + 1 + t0;
    const int head = min((int)((4u - (uint32_t)(reinterpret_cast<uintptr_t>(dst) & 3u)) & 3u), count);
    const int nwords = (count - head) / 4;
    const uint8_t* bytes = reinterpret_cast<const uint8_t*>(done);
    if (tid < head) dst[tid] = bytes[tid];
    for (int j = tid; j < nwords; j += FILTER_THREADS)
      reinterpret_cast<uint32_t*>(dst + head)[j] = __funnelshift_r(done[j], done[j + 1], 8 * head);
    const int rest = head + 4 * nwords + tid;
    if (rest < count) dst[rest] = bytes[rest];
    __syncthreads();
  }
}

// ---- 2. deflate segments -----------------------------------------------------
// Three launches: png_histogram_kernel counts each segment's symbols,
// png_code_kernel builds each segment's Huffman code and block header (one
// warp per segment, so every segment's serial tree construction runs at once),
// png_pack_kernel writes the block. A thread of the per-segment kernels holds
// its 32 bytes in registers; runs of repeated bytes are found with a mask of
// the positions where a run cannot continue. Two CTAs of 1024 threads share an
// SM (32 registers, a few spilled), so that one works while the other waits at
// a barrier. A chunk goes token by token only where a run that is long enough
// for a match touches it; one byte in 256 repeats the one before, so that with
// any repeat as the test nearly every warp took both ways, and its CTA waited.
// A literal chunk is taken word by word: with all 32 bytes extracted in advance,
// and kept from the counting pass for the writing one, the packing spilled 280
// bytes a thread, 1.05 GB of a 24 MP file, out to HBM (0.50 ms, histogram 0.21).
// 16-bit 24 MP: histogram 0.42 ms at first, 0.18 now, packing 0.90 and 0.38.
constexpr int DEFLATE_THREADS = SEG / CHUNK;  // 1024
constexpr int DEFLATE_WARPS = DEFLATE_THREADS / 32;
constexpr int HIST_STRIDE = 288;               // literal/length symbols per segment row, padded
constexpr int CODE_WARPS = 4;                  // segments per png_code_kernel CTA

// Code of one segment: its block header (BFINAL, BTYPE and the dynamic
// Huffman header) and the literal/length code.
struct __align__(16) SegCode {
  uint32_t header_bits;
  uint32_t header[HEADER_WORDS];
  uint16_t code[HIST_STRIDE];
  uint8_t len[HIST_STRIDE];
};

struct Chunk {
  uint32_t w[CHUNK_WORDS];
  int c0, count;
  uint64_t breaks;
};

// Bytes [c0, c0 + CHUNK) of the segment that starts at `seg`, n bytes long. The
// stream buffer is padded to 16 bytes and segments start at multiples of SEG,
// so whole 16-byte loads stay inside it; bytes past n are masked by count.
__device__ __forceinline__ void load_chunk(const uint8_t* __restrict__ seg, int n, Chunk& ch) {
  ch.c0 = min((int)threadIdx.x * CHUNK, n);
  ch.count = min(CHUNK, n - ch.c0);
  const uint4* src = reinterpret_cast<const uint4*>(seg + ch.c0);
#pragma unroll
  for (int v = 0; v < CHUNK / 16; ++v) {
    uint4 q = make_uint4(0u, 0u, 0u, 0u);
    if (v * 16 < ch.count) q = __ldg(src + v);
    ch.w[4 * v] = q.x;
    ch.w[4 * v + 1] = q.y;
    ch.w[4 * v + 2] = q.z;
    ch.w[4 * v + 3] = q.w;
  }
  const uint32_t prev = ch.c0 > 0 ? seg[ch.c0 - 1] : 0u;
  ch.breaks = chunk_breaks(ch.w, ch.count, prev, ch.c0 == 0);
}

// The last break before this thread's chunk and the first at or after its end
// (n when none), from every thread's chunk breaks. Block-wide: all threads call.
__device__ __forceinline__ void run_bounds(const Chunk& ch, int n, int* s_last, int* s_first, int* before,
                                           int* after) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int pre = ch.breaks ? ch.c0 + 63 - clz64(ch.breaks) : -1;
  int suf = ch.breaks ? ch.c0 + ctz64(ch.breaks) : n;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(FULL_MASK, pre, o);
    if (lane >= o) pre = max(pre, t);
    const int u = __shfl_down_sync(FULL_MASK, suf, o);
    if (lane + o < 32) suf = min(suf, u);
  }
  if (lane == 31) s_last[warp] = pre;
  if (lane == 0) s_first[warp] = suf;
  __syncthreads();
  int b = __shfl_up_sync(FULL_MASK, pre, 1);
  if (lane == 0) b = -1;
  for (int w = 0; w < warp; ++w) b = max(b, s_last[w]);
  int a = __shfl_down_sync(FULL_MASK, suf, 1);
  if (lane == 31) a = n;
  for (int w = warp + 1; w < DEFLATE_WARPS; ++w) a = min(a, s_first[w]);
  *before = b;
  *after = a;
}

__global__ void __launch_bounds__(DEFLATE_THREADS, 2)
    png_histogram_kernel(const uint8_t* __restrict__ stream, uint64_t total, uint32_t nseg,
                         uint32_t* __restrict__ seg_freq, uint2* __restrict__ seg_sums) {
  __shared__ uint32_t hist[DEFLATE_WARPS][HIST_STRIDE];
  __shared__ int s_last[DEFLATE_WARPS], s_first[DEFLATE_WARPS];
  __shared__ unsigned long long s_sums[DEFLATE_WARPS][2];
  const uint32_t seg = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint64_t base = (uint64_t)seg * SEG;
  const int n = (int)min((uint64_t)SEG, total - base);
  for (int i = tid; i < DEFLATE_WARPS * HIST_STRIDE; i += DEFLATE_THREADS) (&hist[0][0])[i] = 0u;
  Chunk ch;
  load_chunk(stream + base, n, ch);
  // Adler-32 partial sums: S1 = sum d_j, S2 = sum (n - j) d_j over the segment.
  // Within the chunk the weights are CHUNK - j, up to four bytes at a time.
  unsigned long long s1 = 0, s2 = 0;
  {
    uint32_t sum = 0, weighted = 0;
#pragma unroll
    for (int k = 0; k < CHUNK_WORDS; ++k) {
      const int left = ch.count - 4 * k;
      const uint32_t w = left >= 4 ? ch.w[k] : (left <= 0 ? 0u : ch.w[k] & ((1u << (8 * left)) - 1u));
      sum = __dp4a(w, 0x01010101u, sum);
      weighted = __dp4a(w, (uint32_t)(CHUNK - 4 * k) * 0x01010101u - 0x03020100u, weighted);
    }
    s1 = sum;
    s2 = (unsigned long long)((long long)(n - ch.c0 - CHUNK) * (long long)sum + (long long)weighted);
  }
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_down_sync(FULL_MASK, s1, o);
    s2 += __shfl_down_sync(FULL_MASK, s2, o);
  }
  if (lane == 0) {
    s_sums[warp][0] = s1;
    s_sums[warp][1] = s2;
  }
  int before, after;
  run_bounds(ch, n, s_last, s_first, &before, &after);  // includes a block barrier
  uint32_t* mine = hist[warp];
  chunk_tokens(ch.w, ch.breaks, ch.c0, ch.count, before, after, [&](uint32_t lit, int len) {
    int eb, ev;
    atomicAdd(mine + (len ? length_symbol(len, &eb, &ev) : (int)lit), 1u);
  });
  __syncthreads();
  uint32_t* out = seg_freq + (uint64_t)seg * HIST_STRIDE;
  for (int s = tid; s < HIST_STRIDE; s += DEFLATE_THREADS) {
    uint32_t f = s == END_OF_BLOCK ? 1u : 0u;
    for (int w = 0; w < DEFLATE_WARPS; ++w) f += hist[w][s];
    out[s] = f;
  }
  if (tid == 0) {
    uint32_t a = 0, b = 0;
    for (int w = 0; w < DEFLATE_WARPS; ++w) {
      a = (uint32_t)((a + s_sums[w][0]) % ADLER_MOD);
      b = (uint32_t)((b + s_sums[w][1]) % ADLER_MOD);
    }
    seg_sums[seg] = make_uint2(a, b);
  }
}

struct CodeScratch {
  uint32_t freq[LIT_SYMBOLS];
  uint32_t leaf[LIT_SYMBOLS];
  uint32_t weight[2 * LIT_SYMBOLS];
  uint16_t parent[2 * LIT_SYMBOLS];
  uint16_t order[LIT_SYMBOLS];
  uint16_t code[LIT_SYMBOLS];
  uint8_t len[HIST_STRIDE];
  uint32_t count[MAX_BITS + 1];
  uint32_t next[MAX_BITS + 1];
  HeaderScratch header;
  uint32_t header_words[HEADER_WORDS];
};

// Ascending bitonic sort of 512 keys held 16 per lane (key i = lane * 16 + j):
// compare-exchanges within a lane's registers for partners under 16 apart,
// lane shuffles for the rest.
__device__ __forceinline__ void warp_sort512(uint32_t (&e)[16], int lane) {
#pragma unroll
  for (int k = 2; k <= 512; k <<= 1) {
#pragma unroll
    for (int jj = k >> 1; jj > 0; jj >>= 1) {
      if (jj >= 16) {
        const int lm = jj >> 4;
        const bool lower = (lane & lm) == 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const bool asc = ((lane * 16 + j) & k) == 0;
          const uint32_t other = __shfl_xor_sync(FULL_MASK, e[j], lm);
          e[j] = (lower == asc) ? min(e[j], other) : max(e[j], other);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int p = j ^ jj;
          if (p > j) {
            const bool asc = ((lane * 16 + j) & k) == 0;
            const uint32_t a = e[j], b = e[p];
            e[j] = asc ? min(a, b) : max(a, b);
            e[p] = asc ? max(a, b) : min(a, b);
          }
        }
      }
    }
  }
}

// One warp per segment; no block-wide barrier, so a warp past the last
// segment simply returns.
__global__ void __launch_bounds__(32 * CODE_WARPS)
    png_code_kernel(const uint32_t* __restrict__ seg_freq, uint32_t nseg, SegCode* __restrict__ codes) {
  __shared__ CodeScratch scratch[CODE_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t seg = blockIdx.x * CODE_WARPS + warp;
  if (seg >= nseg) return;
  CodeScratch& C = scratch[warp];
  const uint32_t* f = seg_freq + (uint64_t)seg * HIST_STRIDE;
  for (int s = lane; s < HIST_STRIDE; s += 32) {
    if (s < LIT_SYMBOLS) C.freq[s] = f[s];
    C.len[s] = 0;
  }
  for (int i = lane; i < HEADER_WORDS; i += 32) C.header_words[i] = 0u;
  if (lane <= MAX_BITS) C.count[lane] = 0u;
  __syncwarp();
  // Used symbols by ascending (frequency, symbol): keys frequency << 9 | symbol
  // (frequencies are at most SEG + 1 < 2^16), unused symbols last.
  uint32_t keys[16];
  int used = 0;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const int sym = lane * 16 + j;
    const uint32_t fs = sym < LIT_SYMBOLS ? C.freq[sym] : 0u;
    keys[j] = fs ? (fs << 9) | (uint32_t)sym : 0xFFFFFFFFu;
    used += fs != 0u;
  }
  for (int o = 16; o > 0; o >>= 1) used += __shfl_xor_sync(FULL_MASK, used, o);
  warp_sort512(keys, lane);
#pragma unroll
  for (int j = 0; j < 16; ++j)
    if (lane * 16 + j < used) C.order[lane * 16 + j] = (uint16_t)(keys[j] & 511u);
  __syncwarp();
  // used >= 2: the end-of-block symbol and the segment's first byte.
  for (int i = lane; i < used; i += 32) C.leaf[i] = C.freq[C.order[i]];
  const int root = 2 * used - 2;
  for (;;) {
    __syncwarp();
    if (lane == 0) huffman_tree(C.leaf, used, C.weight, C.parent);
    __syncwarp();
    int deepest = 0;
    for (int i = lane; i < used; i += 32) {
      int d = 0;
      for (int j = i; j != root; j = C.parent[j]) ++d;
      C.len[C.order[i]] = (uint8_t)d;
      deepest = max(deepest, d);
    }
    for (int o = 16; o > 0; o >>= 1) deepest = max(deepest, __shfl_xor_sync(FULL_MASK, deepest, o));
    if (deepest <= MAX_BITS) break;
    // Too deep: halve the frequencies (rounding up keeps them non-zero and in order) and rebuild.
    for (int i = lane; i < used; i += 32) C.leaf[i] = (C.leaf[i] + 1) >> 1;
  }
  __syncwarp();
  // Canonical codes (RFC 1951 3.2.2): the next code of each length, then each
  // symbol's rank among the symbols of its length.
  for (int s = lane; s < LIT_SYMBOLS; s += 32)
    if (C.len[s]) atomicAdd(&C.count[C.len[s]], 1u);
  __syncwarp();
  if (lane == 0) {
    uint32_t c = 0;
    C.next[0] = 0;
    for (int bits = 1; bits <= MAX_BITS; ++bits) {
      c = (c + (bits > 1 ? C.count[bits - 1] : 0u)) << 1;
      C.next[bits] = c;
    }
  }
  __syncwarp();
  // Symbols in groups of 32, in order: a symbol's rank within its group among
  // those of its length, plus the codes of that length handed out before.
  if (lane <= MAX_BITS) C.count[lane] = 0u;
  __syncwarp();
  for (int g = 0; g < HIST_STRIDE; g += 32) {
    const int sym = g + lane;
    const int l = sym < LIT_SYMBOLS ? C.len[sym] : 0;
    const unsigned same = __match_any_sync(FULL_MASK, l);
    const uint32_t ahead = (uint32_t)__popc(same & ((1u << lane) - 1u));
    if (sym < LIT_SYMBOLS) C.code[sym] = l ? (uint16_t)reverse_bits(C.next[l] + C.count[l] + ahead, l) : (uint16_t)0;
    __syncwarp();
    if (l && ahead == 0) C.count[l] += (uint32_t)__popc(same);
    __syncwarp();
  }
  uint32_t header_bits = 0;
  if (lane == 0) {
    BitWriter w{C.header_words, 0};
    header_bits = write_dynamic_header(w, seg + 1 == nseg, C.len, C.header);
  }
  header_bits = __shfl_sync(FULL_MASK, header_bits, 0);
  __syncwarp();
  SegCode& out = codes[seg];
  if (lane == 0) out.header_bits = header_bits;
  for (int i = lane; i < HEADER_WORDS; i += 32) out.header[i] = C.header_words[i];
  for (int s = lane; s < HIST_STRIDE; s += 32) {
    out.code[s] = s < LIT_SYMBOLS ? C.code[s] : (uint16_t)0;
    out.len[s] = C.len[s];
  }
}

__global__ void __launch_bounds__(DEFLATE_THREADS, 2)
    png_pack_kernel(const uint8_t* __restrict__ stream, uint64_t total, uint32_t nseg,
                    const SegCode* __restrict__ codes, uint8_t* __restrict__ slots, uint32_t* __restrict__ seg_bytes) {
  __shared__ __align__(16) uint32_t out[SEG_CAP / 4];
  __shared__ uint32_t s_sym[HIST_STRIDE];  // code | length << 16
  __shared__ int s_last[DEFLATE_WARPS], s_first[DEFLATE_WARPS];
  __shared__ uint32_t s_bits[DEFLATE_WARPS];
  const uint32_t seg = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint64_t base = (uint64_t)seg * SEG;
  const int n = (int)min((uint64_t)SEG, total - base);
  const bool last = seg + 1 == nseg;
  const SegCode& sc = codes[seg];
  const uint32_t header_bits = sc.header_bits;
  for (int i = tid; i < SEG_CAP / 4; i += DEFLATE_THREADS) out[i] = i < HEADER_WORDS ? sc.header[i] : 0u;
  for (int s = tid; s < HIST_STRIDE; s += DEFLATE_THREADS) s_sym[s] = sc.code[s] | ((uint32_t)sc.len[s] << 16);
  Chunk ch;
  load_chunk(stream + base, n, ch);
  int before, after;
  run_bounds(ch, n, s_last, s_first, &before, &after);  // includes a block barrier

  // Bit offsets of each thread's tokens.
  uint32_t bits = 0;
  chunk_tokens(ch.w, ch.breaks, ch.c0, ch.count, before, after, [&](uint32_t lit, int len) {
    if (len) {
      int eb, ev;
      bits += (s_sym[length_symbol(len, &eb, &ev)] >> 16) + eb + 1;  // distance symbol 0: one bit
    } else {
      bits += s_sym[lit] >> 16;
    }
  });
  // The words as new values: the second pass takes the bytes from them again
  // instead of finding 32 extracted ones in local memory.
#pragma unroll
  for (int k = 0; k < CHUNK_WORDS; ++k) asm volatile("" : "+r"(ch.w[k]));
  uint32_t incl = bits;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(FULL_MASK, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) s_bits[warp] = incl;
  __syncthreads();
  uint32_t offset = header_bits + incl - bits;
  uint32_t token_bits = 0;
  for (int w = 0; w < DEFLATE_WARPS; ++w) {
    if (w < warp) offset += s_bits[w];
    token_bits += s_bits[w];
  }
  const uint32_t eob_at = header_bits + token_bits;
  const uint32_t end = eob_at + (s_sym[END_OF_BLOCK] >> 16);
  // After the last block the stream pads to a byte; after any other, an empty
  // stored block (3 zero bits, padding, LEN 0, NLEN 0xFFFF) realigns it.
  const uint32_t dyn_bytes = last ? (end + 7) / 8 : (end + 3 + 7) / 8 + 4;
  const uint32_t stored_bytes = (uint32_t)n + STORED_OVERHEAD;
  const bool stored = dyn_bytes >= stored_bytes;  // the same in every thread

  if (!stored) {
    // The thread's bits gather in a 64-bit accumulator that starts at its
    // offset's position within a word; each full word is ORed out (the first
    // and last words of a thread's range are shared with its neighbours').
    uint32_t word = offset >> 5;
    unsigned long long acc = 0;
    int held = (int)(offset & 31u);
    auto emit = [&](uint32_t value, int n) {  // n <= 21, so held stays below 64
      acc |= (unsigned long long)value << held;
      held += n;
      if (held >= 32) {
        if ((uint32_t)acc) atomicOr(out + word, (uint32_t)acc);
        ++word;
        acc >>= 32;
        held -= 32;
      }
    };
    chunk_tokens(ch.w, ch.breaks, ch.c0, ch.count, before, after, [&](uint32_t lit, int len) {
      if (len) {
        int eb, ev;
        const uint32_t e = s_sym[length_symbol(len, &eb, &ev)];
        const int l = (int)(e >> 16);
        // length code, extra bits, then distance symbol 0's one-bit code 0
        emit((e & 0xFFFFu) | ((uint32_t)ev << l), l + eb + 1);
      } else {
        const uint32_t e = s_sym[lit];
        emit(e & 0xFFFFu, (int)(e >> 16));
      }
    });
    if (held > 0 && (uint32_t)acc) atomicOr(out + word, (uint32_t)acc);
    __syncthreads();
    if (tid == 0) {
      BitWriter w{out, eob_at};
      w.put(s_sym[END_OF_BLOCK] & 0xFFFFu, (int)(s_sym[END_OF_BLOCK] >> 16));
      if (!last) {
        uint8_t* bytes = reinterpret_cast<uint8_t*>(out);
        const uint32_t at = (end + 3 + 7) / 8;
        bytes[at + 2] = 0xFF;
        bytes[at + 3] = 0xFF;
      }
    }
  } else {
    // Every thread has read the header words; the block is rewritten as a stored one.
    for (int i = tid; i < HEADER_WORDS; i += DEFLATE_THREADS) out[i] = 0u;
    __syncthreads();
    uint8_t* bytes = reinterpret_cast<uint8_t*>(out);
    if (tid == 0) {
      bytes[0] = last ? 1 : 0;  // BFINAL, BTYPE 00
      bytes[1] = (uint8_t)n;
      bytes[2] = (uint8_t)(n >> 8);
      bytes[3] = (uint8_t)~n;
      bytes[4] = (uint8_t)(~n >> 8);
    }
#pragma unroll
    for (int j = 0; j < CHUNK; ++j)
      if (j < ch.count) bytes[STORED_OVERHEAD + ch.c0 + j] = (uint8_t)chunk_byte(ch.w, j);
  }
  __syncthreads();
  const uint32_t nbytes = stored ? stored_bytes : dyn_bytes;
  uint4* slot = reinterpret_cast<uint4*>(slots + (uint64_t)seg * SEG_CAP);
  const uint4* src = reinterpret_cast<const uint4*>(out);
  for (uint32_t i = tid; i < (nbytes + 15) / 16; i += DEFLATE_THREADS) slot[i] = src[i];
  if (tid == 0) seg_bytes[seg] = nbytes;
}

// ---- 3. file layout ---------------------------------------------------------
constexpr int LAYOUT_THREADS = 1024;

__device__ __forceinline__ uint64_t idat_chunk_bytes(const uint32_t* seg_bytes, uint32_t s, uint32_t nseg) {
  return 12ull + seg_bytes[s] + (s == 0 ? 2u : 0u) + (s + 1 == nseg ? 4u : 0u);
}

__global__ void __launch_bounds__(LAYOUT_THREADS)
    png_layout_kernel(const uint32_t* __restrict__ seg_bytes, const uint2* __restrict__ seg_sums, uint32_t nseg,
                      uint64_t total, uint64_t header_bytes, uint32_t iend_crc, uint64_t* __restrict__ chunk_at,
                      uint32_t* __restrict__ adler_out, uint64_t* __restrict__ png_bytes, uint8_t* __restrict__ png) {
  __shared__ unsigned long long warp_sum[LAYOUT_THREADS / 32][3];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t per = (nseg + LAYOUT_THREADS - 1) / LAYOUT_THREADS;
  const uint32_t s0 = min((uint32_t)tid * per, nseg), s1 = min(s0 + per, nseg);
  unsigned long long mine = 0, a = 0, b = 0;
  for (uint32_t s = s0; s < s1; ++s) {
    mine += idat_chunk_bytes(seg_bytes, s, nseg);
    const uint64_t o = (uint64_t)s * SEG;
    const uint64_t n = min((uint64_t)SEG, total - o);
    const uint2 q = seg_sums[s];
    a += q.x;
    b = (b + adler_combine_term(total, o, n, q.x, q.y)) % ADLER_MOD;
  }
  unsigned long long incl = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(FULL_MASK, incl, o);
    if (lane >= o) incl += t;
  }
  unsigned long long ra = a, rbv = b;
  for (int o = 16; o > 0; o >>= 1) {
    ra += __shfl_down_sync(FULL_MASK, ra, o);
    rbv += __shfl_down_sync(FULL_MASK, rbv, o);
  }
  if (lane == 31) warp_sum[warp][0] = incl;
  if (lane == 0) {
    warp_sum[warp][1] = ra;
    warp_sum[warp][2] = rbv;
  }
  __syncthreads();
  unsigned long long at = header_bytes + incl - mine, all = 0;
  for (int w = 0; w < LAYOUT_THREADS / 32; ++w) {
    if (w < warp) at += warp_sum[w][0];
    all += warp_sum[w][0];
  }
  for (uint32_t s = s0; s < s1; ++s) {
    chunk_at[s] = at;
    at += idat_chunk_bytes(seg_bytes, s, nseg);
  }
  if (tid == 0) {
    unsigned long long asum = 0, bsum = 0;
    for (int w = 0; w < LAYOUT_THREADS / 32; ++w) {
      asum += warp_sum[w][1];
      bsum += warp_sum[w][2];
    }
    const uint32_t A = (uint32_t)((1ull + asum) % ADLER_MOD);
    const uint32_t B = (uint32_t)((total % ADLER_MOD + bsum) % ADLER_MOD);
    *adler_out = (B << 16) | A;
    const uint64_t size = header_bytes + all + 12;
    *png_bytes = size;
    uint8_t* iend = png + size - 12;
    const uint8_t fixed[8] = {0, 0, 0, 0, 'I', 'E', 'N', 'D'};
    for (int k = 0; k < 8; ++k) iend[k] = fixed[k];
    for (int k = 0; k < 4; ++k) iend[8 + k] = (uint8_t)(iend_crc >> (24 - 8 * k));
  }
}

// ---- 4. IDAT chunks ----------------------------------------------------------
constexpr int CHUNK_THREADS = 256;

struct ChunkParams {
  const uint8_t* slots;
  const uint32_t* seg_bytes;
  const uint64_t* chunk_at;
  const uint32_t* adler;
  uint8_t* png;
  uint32_t nseg;
};

static_assert(CHUNK_THREADS == CRC_SHARES, "a thread per share");
__device__ const CrcTree CRC_TREE = crc_tree();

// The segment's block lies in shared memory from byte 16 on, the chunk's length
// and type (and the zlib header) in front of it. CRC-32 takes four bytes a step
// from four tables. 16-bit 24 MP: 0.25 ms with a byte a step and every thread
// advancing its register over the rest of the chunk bit by bit, now 0.08.
__global__ void __launch_bounds__(CHUNK_THREADS) png_chunk_kernel(const __grid_constant__ ChunkParams P) {
  constexpr uint32_t DATA = 16;
  __shared__ __align__(16) uint8_t buf[DATA + SEG_CAP + 48];
  __shared__ uint32_t table[4][256];
  __shared__ CrcTree tree;
  __shared__ uint32_t warp_crc[CHUNK_THREADS / 32];
  const uint32_t s = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool first = s == 0, last = s + 1 == P.nseg;
  const uint32_t nb = P.seg_bytes[s];
  const uint32_t dl = nb + (first ? 2u : 0u) + (last ? 4u : 0u);  // chunk data bytes
  const uint32_t size = dl + 12;
  const uint32_t start = DATA - 8u - (first ? 2u : 0u);  // of the chunk in buf
  table[0][tid] = crc_byte_entry((uint32_t)tid);
  for (int i = tid; i < (int)(sizeof(CrcTree) / 4); i += CHUNK_THREADS)
    (&tree.t[0][0][0])[i] = (&CRC_TREE.t[0][0][0])[i];
  const uint4* src = reinterpret_cast<const uint4*>(P.slots + (uint64_t)s * SEG_CAP);
  for (uint32_t v = tid; v < (nb + 15) / 16; v += CHUNK_THREADS) reinterpret_cast<uint4*>(buf + DATA)[v] = __ldg(src + v);
  __syncthreads();
#pragma unroll
  for (int k = 1; k < 4; ++k) table[k][tid] = crc_zero_bytes(table[0], table[0][tid], k);
  if (tid == 0) {
    uint8_t* c = buf + start;
    for (int k = 0; k < 4; ++k) c[k] = (uint8_t)(dl >> (24 - 8 * k));
    c[4] = 'I';
    c[5] = 'D';
    c[6] = 'A';
    c[7] = 'T';
    if (first) {
      c[8] = 0x78;  // deflate, 32 KiB window
      c[9] = 0x9C;  // default level, no dictionary; 0x789C is a multiple of 31
    }
    if (last) {
      const uint32_t adler = *P.adler;
      for (int k = 0; k < 4; ++k) c[8 + dl - 4 + k] = (uint8_t)(adler >> (24 - 8 * k));
    }
  }
  __syncthreads();
  // Bytes o .. o + 3 of buf.
  const uint32_t* words = reinterpret_cast<const uint32_t*>(buf);
  auto word_at = [&](uint32_t o) { return __funnelshift_r(words[o >> 2], words[(o >> 2) + 1], 8 * (o & 3u)); };
  // CRC-32 over the chunk type and data, each thread over its own bytes.
  const uint32_t from = start + 4;
  uint32_t reg = crc_share(table, (int)(4 + dl), tid, [&](int k) { return (uint32_t)buf[from + k]; },
                           [&](int k) { return word_at(from + k); });
  // Groups to the left of the chunk's start have a zero register.
#pragma unroll
  for (int j = 0; j < 5; ++j) reg = crc_advance(tree.t[j], __shfl_up_sync(FULL_MASK, reg, 1 << j)) ^ reg;
  if (lane == 31) warp_crc[warp] = reg;
  __syncthreads();
  if (warp == 0) {
    reg = warp_crc[lane & 7];
#pragma unroll
    for (int j = 0; j < 3; ++j) reg = crc_advance(tree.t[5 + j], __shfl_up_sync(FULL_MASK, reg, 1 << j)) ^ reg;
  }
  if (tid == 7) {
    const uint32_t crc = reg ^ 0xFFFFFFFFu;
    for (int k = 0; k < 4; ++k) buf[start + 8 + dl + k] = (uint8_t)(crc >> (24 - 8 * k));
  }
  __syncthreads();
  // Whole 32-bit words inside the chunk are stored as words; the bytes at
  // either end share a word with the neighbouring chunk and go one by one.
  const uint64_t at = P.chunk_at[s];
  uint8_t* out = P.png + at;
  const uint32_t head = min((4u - (uint32_t)(reinterpret_cast<uintptr_t>(out) & 3u)) & 3u, size);
  const uint32_t nwords = (size - head) / 4;
  if (tid < head) out[tid] = buf[start + tid];
  uint32_t* ow = reinterpret_cast<uint32_t*>(out + head);
  for (uint32_t w = tid; w < nwords; w += CHUNK_THREADS) ow[w] = word_at(start + head + 4 * w);
  const uint32_t rest = head + 4 * nwords + tid;
  if (rest < size) out[rest] = buf[start + rest];
}

// ---- host: chunks built on the CPU ----------------------------------------
struct HostCrc {
  uint32_t table[256];
  HostCrc() {
    for (uint32_t i = 0; i < 256; ++i) table[i] = crc_byte_entry(i);
  }
  uint32_t operator()(const uint8_t* p, size_t n) const { return crc_update(table, 0xFFFFFFFFu, p, n) ^ 0xFFFFFFFFu; }
};

const HostCrc& host_crc() {
  static const HostCrc crc;
  return crc;
}

void put_be32(std::vector<uint8_t>& v, uint32_t x) {
  for (int k = 0; k < 4; ++k) v.push_back((uint8_t)(x >> (24 - 8 * k)));
}

void add_chunk(std::vector<uint8_t>& out, const char* type, const std::vector<uint8_t>& data) {
  put_be32(out, (uint32_t)data.size());
  const size_t at = out.size();
  out.insert(out.end(), type, type + 4);
  out.insert(out.end(), data.begin(), data.end());
  put_be32(out, host_crc()(out.data() + at, 4 + data.size()));
}

// A zlib stream of stored deflate blocks (RFC 1950/1951): the profile is a
// few kilobytes and rides uncompressed inside its wrapper.
std::vector<uint8_t> zlib_stored(const uint8_t* p, size_t n) {
  std::vector<uint8_t> z = {0x78, 0x01};
  size_t at = 0;
  do {
    const size_t len = std::min<size_t>(65535, n - at);
    const bool final_block = at + len == n;
    z.push_back(final_block ? 1 : 0);
    z.push_back((uint8_t)len);
    z.push_back((uint8_t)(len >> 8));
    z.push_back((uint8_t)~len);
    z.push_back((uint8_t)(~len >> 8));
    z.insert(z.end(), p + at, p + at + len);
    at += len;
  } while (at < n);
  uint32_t a = 1, b = 0;
  for (size_t i = 0; i < n; ++i) {
    a = (a + p[i]) % ADLER_MOD;
    b = (b + a) % ADLER_MOD;
  }
  put_be32(z, (b << 16) | a);
  return z;
}

const char* ICC_PROFILE_NAME = "ICC profile";

}  // namespace

uint64_t png_stream_bytes(int W, int H, int depth) { return (uint64_t)H * (1ull + (uint64_t)W * (depth / 8) * 3); }

uint64_t png_segments(uint64_t stream_bytes) { return (stream_bytes + SEG - 1) / SEG; }

// Largest metadata a PNG chunk carries: the chunk length is a 31-bit count
// and the profile's chunk adds its name and zlib framing.
constexpr uint64_t PNG_METADATA_LIMIT = 0x7FF00000ull;

bool png_metadata_ok(uint64_t icc_len, uint64_t exif_len) {
  return icc_len <= PNG_METADATA_LIMIT && exif_len <= PNG_METADATA_LIMIT;
}

uint64_t png_header_bytes(uint64_t icc_len, uint64_t exif_len) {
  uint64_t n = 8 + 25;  // signature, IHDR
  if (icc_len) {
    const uint64_t blocks = (icc_len + 65534) / 65535;
    n += 12 + std::strlen(ICC_PROFILE_NAME) + 2 + 2 + 5 * blocks + icc_len + 4;
  }
  if (exif_len) n += 12 + exif_len;
  return n;
}

Status png_header(int W, int H, int depth, const uint8_t* icc, size_t icc_len, const uint8_t* exif, size_t exif_len,
                  std::vector<uint8_t>* out) {
  if (!png_metadata_ok(icc_len, exif_len)) return Status{RD_INVALID_INPUT, "metadata too large for a PNG chunk"};
  std::vector<uint8_t>& h = *out;
  h = {0x89, 'P', 'N', 'G', 0x0D, 0x0A, 0x1A, 0x0A};
  std::vector<uint8_t> ihdr;
  put_be32(ihdr, (uint32_t)W);
  put_be32(ihdr, (uint32_t)H);
  ihdr.push_back((uint8_t)depth);
  ihdr.push_back(2);  // truecolour RGB
  ihdr.push_back(0);  // deflate
  ihdr.push_back(0);  // adaptive filtering with the five basic filters
  ihdr.push_back(0);  // no interlace
  add_chunk(h, "IHDR", ihdr);
  if (icc && icc_len) {
    std::vector<uint8_t> iccp(ICC_PROFILE_NAME, ICC_PROFILE_NAME + std::strlen(ICC_PROFILE_NAME));
    iccp.push_back(0);  // name terminator
    iccp.push_back(0);  // compression method: zlib
    const std::vector<uint8_t> z = zlib_stored(icc, icc_len);
    iccp.insert(iccp.end(), z.begin(), z.end());
    if (iccp.size() > 0x7FFFFFFFu) return Status{RD_INVALID_INPUT, "ICC profile does not fit in a PNG chunk"};
    add_chunk(h, "iCCP", iccp);
  }
  if (exif && exif_len) {
    if (exif_len > 0x7FFFFFFFu) return Status{RD_INVALID_INPUT, "EXIF block does not fit in a PNG chunk"};
    add_chunk(h, "eXIf", std::vector<uint8_t>(exif, exif + exif_len));
  }
  return Status{};
}

uint64_t png_bound(int W, int H, int depth, uint64_t header_bytes) {
  const uint64_t L = png_stream_bytes(W, H, depth);
  const uint64_t nseg = png_segments(L);
  // Each segment is at most a stored block; zlib header and Adler-32; IEND.
  return header_bytes + L + nseg * (12 + STORED_OVERHEAD) + 6 + 12;
}

Status run_png_encode(Context& ctx, const void* d_rgb, int W, int H, int depth, const std::vector<uint8_t>& header,
                      uint8_t* d_png, uint64_t* d_png_bytes) {
  const uint64_t L = png_stream_bytes(W, H, depth);
  const uint64_t nseg = png_segments(L);
  if (nseg > 0x7FFFFFFFull) return Status{RD_INVALID_DIMENSIONS, "image too large for one PNG stream"};
  auto round16 = [](uint64_t v) { return (v + 15) & ~15ull; };
  const uint64_t stream_bytes = round16(L);
  const uint64_t slot_bytes = nseg * SEG_CAP;
  const uint64_t count_bytes = round16(nseg * 4);
  const uint64_t sum_bytes = round16(nseg * 8);
  const uint64_t at_bytes = round16(nseg * 8);
  const uint64_t freq_bytes = round16(nseg * HIST_STRIDE * 4);
  const uint64_t code_bytes = nseg * sizeof(SegCode);
  const uint64_t total = stream_bytes + slot_bytes + count_bytes + sum_bytes + at_bytes + 16 + freq_bytes + code_bytes;
  void* scratch = nullptr;
  RD_TRY(device_alloc(ctx, total, &scratch));
  uint8_t* p = static_cast<uint8_t*>(scratch);
  uint8_t* stream = p;
  uint8_t* slots = stream + stream_bytes;
  uint32_t* seg_bytes = reinterpret_cast<uint32_t*>(slots + slot_bytes);
  uint2* seg_sums = reinterpret_cast<uint2*>(reinterpret_cast<uint8_t*>(seg_bytes) + count_bytes);
  uint64_t* chunk_at = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(seg_sums) + sum_bytes);
  uint32_t* adler = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(chunk_at) + at_bytes);
  uint32_t* seg_freq = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(adler) + 16);
  SegCode* codes = reinterpret_cast<SegCode*>(reinterpret_cast<uint8_t*>(seg_freq) + freq_bytes);

  Status st = upload(ctx, d_png, header.data(), header.size());
  if (st.ok()) {
    if (depth == 16) {
      RD_LAUNCH(ctx, K_ENCODE, png_filter_kernel<true><<<H, FILTER_THREADS, 0, ctx.stream>>>(d_rgb, W, stream));
    } else {
      RD_LAUNCH(ctx, K_ENCODE, png_filter_kernel<false><<<H, FILTER_THREADS, 0, ctx.stream>>>(d_rgb, W, stream));
    }
    RD_LAUNCH(ctx, K_ENCODE,
              png_histogram_kernel<<<(unsigned)nseg, DEFLATE_THREADS, 0, ctx.stream>>>(stream, L, (uint32_t)nseg,
                                                                                     seg_freq, seg_sums));
    RD_LAUNCH(ctx, K_ENCODE,
              png_code_kernel<<<(unsigned)((nseg + CODE_WARPS - 1) / CODE_WARPS), 32 * CODE_WARPS, 0, ctx.stream>>>(
                  seg_freq, (uint32_t)nseg, codes));
    RD_LAUNCH(ctx, K_ENCODE,
              png_pack_kernel<<<(unsigned)nseg, DEFLATE_THREADS, 0, ctx.stream>>>(stream, L, (uint32_t)nseg, codes,
                                                                                slots, seg_bytes));
    const uint32_t iend_crc = host_crc()(reinterpret_cast<const uint8_t*>("IEND"), 4);
    RD_LAUNCH(ctx, K_ENCODE,
              png_layout_kernel<<<1, LAYOUT_THREADS, 0, ctx.stream>>>(seg_bytes, seg_sums, (uint32_t)nseg, L,
                                                                      header.size(), iend_crc, chunk_at, adler,
                                                                      d_png_bytes, d_png));
    ChunkParams cp{};
    cp.slots = slots;
    cp.seg_bytes = seg_bytes;
    cp.chunk_at = chunk_at;
    cp.adler = adler;
    cp.png = d_png;
    cp.nseg = (uint32_t)nseg;
    RD_LAUNCH(ctx, K_ENCODE, png_chunk_kernel<<<(unsigned)nseg, CHUNK_THREADS, 0, ctx.stream>>>(cp));
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) st = Status{RD_SYNCHRONIZATION, std::string("PNG encode launch: ") + cudaGetErrorString(e)};
  }
  device_free(ctx, scratch, total);
  return st;
}

}  // namespace rd
