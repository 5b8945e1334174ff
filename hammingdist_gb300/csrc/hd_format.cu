// Device-side text writers.
//
// Replaces lower_triangular_lines / partial_write_lower_triangular
// (include/hamming/hamming_utils.hh:19-104) and DataSet::dump_sparse
// (include/hamming/hamming.hh:79-114), which format on the CPU with fmt.
// The lower-triangular text is formatted as one flat run of entries. The full
// matrix and the sparse lines take one warp per row: per 32 entries each lane
// computes its text length, a warp prefix sum places it, and the lane writes
// its digits; row starts come from a device scan of per-row text lengths.
#include <algorithm>
#include <mutex>

#include "hd_internal.cuh"

namespace hd {

__device__ inline uint32_t ndig(uint32_t v) {
  return v < 10u ? 1 : v < 100u ? 2 : v < 1000u ? 3 : v < 10000u ? 4 : v < 100000u ? 5
       : v < 1000000u ? 6 : v < 10000000u ? 7 : v < 100000000u ? 8 : v < 1000000000u ? 9 : 10;
}

__device__ inline void put_dec(char *dst, uint32_t v, uint32_t nd) {
  for (int k = (int)nd - 1; k >= 0; --k) {
    dst[k] = (char)('0' + v % 10u);
    v /= 10u;
  }
}

__host__ __device__ inline uint64_t row_index(uint64_t i) { return i * (i - 1) / 2; }

// --------------------------------------------------- lower-triangular text
// Row i (i >= 1): "d(i,0),d(i,1),...,d(i,i-1)\n".
//
// The rows' entries follow one another in the lower triangle, and so do their
// texts, so the triangle is formatted as one flat run of entries: each entry's
// digits and a separator, '\n' after a row's last entry. Warps take equal
// stretches whatever the rows' lengths: one pass adds up each stretch's text
// length (k_lt_len), one block turns the sums into offsets, and the write pass
// builds the text in shared memory and copies it out in 16-byte vectors, with
// no synchronisation between warps.
//
// What bounds it (14,000 rows, uint8, 98.0 M entries, 277 MB of text; HBM would
// take 55 us): instructions, 39 per 32 entries in the write pass. 207 us a call:
// lengths 30, offsets 11, text 146 (69% of the issue slots); uint16 412 us.
// One warp per row with byte stores to global memory took 620 us in all; whole
// entries stored byte by byte in shared memory 411 us (77 instructions per 32
// entries).
constexpr int kTextThreads = 256, kTextWarps = kTextThreads / 32;
constexpr uint32_t kTextTile = 512;  // entries per warp and step
// text bytes per entry at most
template <typename T> constexpr uint32_t kTextMax = sizeof(T) == 1 ? 4 : sizeof(T) == 2 ? 6 : 11;

// The flat run: entries [0, n) at lt; e0 is the first one's lower-triangle
// index. Positions count from lt rounded down to 16 bytes (entry k is at
// position shift + k), and stretch g is the positions [g per, (g + 1) per), so
// that stretches start on aligned vectors.
template <typename T>
struct TextRun {
  const T *lt;
  uint64_t e0, n, per;
  __device__ __host__ uint32_t shift() const {
    return (uint32_t)((reinterpret_cast<uintptr_t>(lt) & 15u) / sizeof(T));
  }
};

// Four decimal digits of c < 10000, the first in the low byte, with leading
// zeros.
__device__ __forceinline__ uint32_t four_digits(uint32_t c) {
  const uint32_t q = (c * 5243u) >> 19, r = c - 100u * q;  // c / 100, c % 100
  const uint32_t x = q | (r << 16);
  const uint32_t tens = ((x * 103u) >> 10) & 0x000F000Fu;  // both below 100: no carry into bit 16
  return (tens | ((x - 10u * tens) << 8)) + 0x30303030u;
}
__device__ __forceinline__ uint32_t ndig4(uint32_t c) {
  return 1u + (c >= 10u) + (c >= 100u) + (c >= 1000u);
}

__device__ __forceinline__ uint64_t ceil_pos(uint64_t a, uint64_t b) { return (a + b - 1) / b * b; }

// Text length of 16 bytes of entries: a separator and a digit each, and more
// digits where they are large.
__device__ __forceinline__ uint32_t text_len16(const uint4 &q, uint8_t) {
  uint32_t n = 0;  // two 16-bit sums
  for (uint32_t w : {q.x, q.y, q.z, q.w}) {
    const uint32_t lo = w & 0x00FF00FFu, hi = (w >> 8) & 0x00FF00FFu;
    // bit 8 of each half: the byte is at least 10, at least 100
    n += (((lo + 0x00F600F6u) >> 8) & 0x00010001u) + (((lo + 0x009C009Cu) >> 8) & 0x00010001u);
    n += (((hi + 0x00F600F6u) >> 8) & 0x00010001u) + (((hi + 0x009C009Cu) >> 8) & 0x00010001u);
  }
  return 32u + (n & 0xFFFFu) + (n >> 16);
}
__device__ __forceinline__ uint32_t text_len16(const uint4 &q, uint16_t) {
  uint32_t n = 0;
  for (uint32_t w : {q.x, q.y, q.z, q.w}) n += ndig(w & 0xFFFFu) + ndig(w >> 16) + 2;
  return n;
}
__device__ __forceinline__ uint32_t text_len16(const uint4 &q, uint32_t) {
  return ndig(q.x) + ndig(q.y) + ndig(q.z) + ndig(q.w) + 4;
}

template <typename T>
__global__ void __launch_bounds__(kTextThreads) k_lt_len(TextRun<T> run, uint64_t *sums) {
  const uint32_t lane = threadIdx.x & 31u, shift = run.shift();
  const uint64_t g = (uint64_t)blockIdx.x * kTextWarps + (threadIdx.x >> 5);
  const uint64_t end = run.n + shift;
  const T *base = run.lt - shift;  // position 0
  uint64_t lo = g * run.per, hi = lo + run.per < end ? lo + run.per : end;
  if (lo < shift) lo = shift;
  uint64_t len = 0;
  if (lo < hi) {
    // whole vectors, and entry by entry before and after them
    constexpr uint64_t V = 16 / sizeof(T);
    const uint64_t v_lo = ceil_pos(lo, V) < hi ? ceil_pos(lo, V) : hi, vecs = (hi - v_lo) / V;
    const uint4 *vp = reinterpret_cast<const uint4 *>(base + v_lo);
#pragma unroll 8
    for (uint64_t k = lane; k < vecs; k += 32) len += text_len16(vp[k], T());
    for (uint64_t k = lo + lane; k < v_lo; k += 32) len += ndig(base[k]) + 1;
    for (uint64_t k = v_lo + vecs * V + lane; k < hi; k += 32) len += ndig(base[k]) + 1;
  }
  len = warp_sum(len);
  if (lane == 0) sums[g] = len;
}

// A warp's text on its way out: it gathers in the warp's buffer from byte
// `at` on (the destination's offset mod 16, so that whole 16-byte vectors of
// the buffer go to aligned addresses), and `flush` copies the whole vectors
// out and keeps the rest. The first `skip` bytes of the buffer's first vector
// belong to the stretch before.
struct TextOut {
  uint32_t *buf;
  char *base;     // where the buffer's first vector goes (16-byte aligned)
  uint32_t at;    // bytes in the buffer
  uint32_t skip;
  __device__ __forceinline__ void flush(uint32_t lane, bool last) {
    __syncwarp();
    const char *b = reinterpret_cast<const char *>(buf);
    const uint32_t vecs = at / 16;
    for (uint32_t k = lane + (skip ? 1u : 0u); k < vecs; k += 32)
      reinterpret_cast<uint4 *>(base)[k] = reinterpret_cast<const uint4 *>(buf)[k];
    if (skip && vecs) {
      if (lane >= skip && lane < 16) base[lane] = b[lane];
      skip = 0;
    }
    if (last) {
      const uint32_t from = vecs ? 16 * vecs : skip;
      if (from + lane < at) base[from + lane] = b[from + lane];  // less than 16 bytes
      return;
    }
    const uint32_t keep = lane < 4 ? buf[4 * vecs + lane] : 0u;
    __syncwarp();
    if (lane < 4) buf[lane] = keep;
    __syncwarp();
    base += 16 * vecs;
    at &= 15u;
  }
};

// The row ends among positions [pos, pos + 32 step): lane l's entries are step
// l .. step l + step - 1; `mark(k)` is called for entry k that ends a row.
// row_end: position after the current row's last entry, row: its index.
template <uint32_t kStep, class F>
__device__ __forceinline__ void for_row_ends(uint64_t pos, uint64_t &row, uint64_t &row_end,
                                             uint32_t lane, F &&mark) {
  while (row_end <= pos + 32 * kStep) {
    const uint32_t k = (uint32_t)(row_end - pos) - 1u - kStep * lane;
    if (k < kStep) mark(k);
    row_end += ++row;
  }
}

// The digits of x < 65536 and a separator, n bytes, the first in the low one.
__device__ __forceinline__ uint64_t short_text(uint32_t x, uint32_t sep, uint32_t &n) {
  const uint32_t h = x / 10000u, c = x - 10000u * h, w = four_digits(c);
  const uint32_t nd = h ? 4u : ndig4(c);
  uint64_t t = (uint64_t)(w >> (8 * (4 - nd))) | ((uint64_t)sep << (8 * nd));
  if (h) t = (t << 8) | ('0' + h);
  n = nd + (h ? 2u : 1u);
  return t;
}

// One warp per stretch. Nothing is written if the whole text, *total bytes,
// does not fit in `capacity`.
//
// uint8 and uint16: a lane turns four (two) entries at a time into one string
// in registers (for uint8 a table gives each entry's digits and ','), a prefix
// sum of the lengths places the strings, and each lane stores the whole words
// that end in its string; the bytes before the first of them come from the
// lane before it. Strings have at least four bytes, so a word has bytes of
// two lanes at most. uint32 and the ends of the run: a lane stores every 32nd
// entry byte by byte.
constexpr uint32_t kTabCopies = 16;  // of the uint8 text table: lane l reads copy l % 16
template <typename T>
__global__ void __launch_bounds__(kTextThreads)
    k_lt_write(TextRun<T> run, const uint64_t *offs, const uint64_t *total, uint64_t capacity,
               char *text) {
  constexpr uint32_t kWords = (kTextTile * kTextMax<T> + 32) / 4;
  __shared__ __align__(16) uint32_t s_buf[kTextWarps][kWords];
  __shared__ uint32_t tab[sizeof(T) == 1 ? 256 * kTabCopies : 1];
  if (*total > capacity) return;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  if (sizeof(T) == 1) {
    // value -> its digits and ',', the first character in the low byte
    const uint32_t v = threadIdx.x, nd = ndig4(v);
    const uint32_t w = (four_digits(v) >> (8 * (4 - nd))) | ((uint32_t)',' << (8 * nd));
#pragma unroll
    for (uint32_t c = 0; c < kTabCopies; ++c) tab[v * kTabCopies + c] = w;
    __syncthreads();
  }
  const uint32_t shift = run.shift();
  const uint64_t g = (uint64_t)blockIdx.x * kTextWarps + warp, end = run.n + shift;
  const T *src = run.lt - shift;  // position 0
  uint64_t lo = g * run.per, hi = lo + run.per < end ? lo + run.per : end;
  if (lo < shift) lo = shift;
  if (lo >= hi) return;
  // the row of the stretch's first entry e: i (i - 1) / 2 <= e < i (i + 1) / 2
  // (one lane: double precision is slow here)
  uint64_t row = 0;
  if (lane == 0) {
    const uint64_t e = run.e0 + (lo - shift);
    row = (uint64_t)((1.0 + sqrt(1.0 + 8.0 * (double)e)) * 0.5);
    while (row * (row - 1) / 2 > e) --row;
    while (row * (row + 1) / 2 <= e) ++row;
  }
  row = __shfl_sync(0xffffffffu, row, 0);
  uint64_t row_end = row * (row + 1) / 2 - run.e0 + shift;
  char *dst = text + offs[g];
  const uint32_t skip = (uint32_t)(reinterpret_cast<uintptr_t>(dst) & 15u);
  TextOut out{s_buf[warp], dst - skip, skip, skip};
  char *buf = reinterpret_cast<char *>(out.buf);
  uint32_t carry = 0;  // the bytes of the word at out.at before it
  for (uint64_t t = lo & ~(uint64_t)(kTextTile - 1); t < hi; t += kTextTile) {
    if (sizeof(T) <= 2 && t >= lo && t + kTextTile <= hi) {
      // E entries of a lane at a time, from one 32-bit load each
      constexpr uint32_t E = 4 / sizeof(T), kSteps = kTextTile / (32 * E);
      constexpr uint32_t kFlip = (uint32_t)',' ^ (uint32_t)'\n';
      uint32_t x[kSteps];
#pragma unroll
      for (uint32_t j = 0; j < kSteps; ++j)
        x[j] = reinterpret_cast<const uint32_t *>(src + t)[32 * j + lane];
#pragma unroll
      for (uint32_t j = 0; j < kSteps; ++j) {
        const uint64_t pos = t + 32 * E * j;
        uint32_t a0, a1, a2, a3 = 0, len;  // the lane's string and its bytes
        if (sizeof(T) == 1) {
          const uint32_t lo2 = x[j] & 0x00FF00FFu, hi2 = (x[j] >> 8) & 0x00FF00FFu;
          // 8 x (digits - 1) of entries 0 and 2, of 1 and 3
          const uint32_t d02 = (((lo2 + 0x00F600F6u) >> 5) & 0x00080008u) + (((lo2 + 0x009C009Cu) >> 5) & 0x00080008u);
          const uint32_t d13 = (((hi2 + 0x00F600F6u) >> 5) & 0x00080008u) + (((hi2 + 0x009C009Cu) >> 5) & 0x00080008u);
          const uint32_t b0 = 16u + (d02 & 0xFFu), b1 = 16u + (d13 & 0xFFu);  // bits of entry 0, 1,
          const uint32_t b2 = 16u + (d02 >> 16), b3 = 16u + (d13 >> 16);      // 2 and 3
          const uint32_t *tl = tab + (lane & (kTabCopies - 1));
          uint32_t c0 = tl[(x[j] & 0xFFu) * kTabCopies], c1 = tl[(x[j] >> 8 & 0xFFu) * kTabCopies];
          uint32_t c2 = tl[(x[j] >> 16 & 0xFFu) * kTabCopies], c3 = tl[(x[j] >> 24) * kTabCopies];
          for_row_ends<4>(pos, row, row_end, lane, [&](uint32_t k) {
            if (k == 0) c0 ^= kFlip << (b0 - 8);
            else if (k == 1) c1 ^= kFlip << (b1 - 8);
            else if (k == 2) c2 ^= kFlip << (b2 - 8);
            else c3 ^= kFlip << (b3 - 8);
          });
          // entries 0 and 1, 2 and 3, then all four
          const uint32_t p0 = c0 | __funnelshift_lc(0u, c1, b0), p1 = __funnelshift_lc(c1, 0u, b0);
          const uint32_t q0 = c2 | __funnelshift_lc(0u, c3, b2), q1 = __funnelshift_lc(c3, 0u, b2);
          const uint32_t sh = b0 + b1 - 32;  // the second pair starts in word 1, 0 to 32 bits in
          a0 = p0;
          a1 = p1 | __funnelshift_lc(0u, q0, sh);
          a2 = __funnelshift_lc(q0, q1, sh);
          a3 = __funnelshift_lc(q1, 0u, sh);
          len = (b0 + b1 + b2 + b3) >> 3;
        } else {
          // each entry's digits and separator in 64 bits, then both in 96
          uint32_t sep0 = ',', sep1 = ',';
          for_row_ends<2>(pos, row, row_end, lane, [&](uint32_t k) { (k ? sep1 : sep0) = '\n'; });
          uint32_t n0, n1;
          const uint64_t c0 = short_text(x[j] & 0xFFFFu, sep0, n0);
          const uint64_t c1 = short_text(x[j] >> 16, sep1, n1);
          const uint64_t both = c0 | (c1 << (8 * n0));  // n0 <= 6
          a0 = (uint32_t)both;
          a1 = (uint32_t)(both >> 32);
          a2 = (uint32_t)(c1 >> (64 - 8 * n0));
          len = n0 + n1;
        }
        const uint32_t inc = warp_incl_scan(len);
        const uint32_t q = out.at + inc - len, f = 8 * (q & 3u), words = ((q & 3u) + len) >> 2;
        uint32_t o0 = a0 << f;
        const uint32_t o1 = __funnelshift_l(a0, a1, f), o2 = __funnelshift_l(a1, a2, f);
        const uint32_t o3 = __funnelshift_l(a2, a3, f), o4 = __funnelshift_l(a3, 0u, f);
        // the bytes after the last whole word are the next lane's first
        uint32_t rest;
        if (sizeof(T) == 1) rest = words == 2 ? o2 : words == 3 ? o3 : o4;
        else rest = words == 1 ? o1 : words == 2 ? o2 : o3;
        const uint32_t before = __shfl_up_sync(0xffffffffu, rest, 1);
        o0 |= lane ? before : carry;
        carry = __shfl_sync(0xffffffffu, rest, 31);
        uint32_t *w = out.buf + (q >> 2);
        w[0] = o0;
        if (sizeof(T) == 1 || words > 1) w[1] = o1;
        if (words > 2) w[2] = o2;
        if (sizeof(T) == 1 && words > 3) w[3] = o3;
        out.at += __shfl_sync(0xffffffffu, inc, 31);
      }
      if (lane == 0) out.buf[out.at >> 2] = carry;
    } else {
#pragma unroll 1
      for (uint64_t pos = t; pos < t + kTextTile; pos += 32) {
        if (pos + 32 <= lo || pos >= hi) continue;  // warp-uniform
        const bool on = pos + lane >= lo && pos + lane < hi;
        uint32_t x = on ? (uint32_t)src[pos + lane] : 0u;
        const uint32_t nd = ndig(x), len = on ? nd + 1 : 0u, inc = warp_incl_scan(len);
        char sep = ',';
        for_row_ends<1>(pos, row, row_end, lane, [&](uint32_t) { sep = '\n'; });
        if (on) {
          char *o = buf + out.at + inc - len;
          o[nd] = sep;
          // the last four digits, the four before them, the rest
#pragma unroll
          for (uint32_t h = 0; h < 12; h += 4) {
            const uint32_t w = four_digits(x % 10000u);
#pragma unroll
            for (uint32_t d = 0; d < 4; ++d)
              if (h + d < nd) o[nd - 1 - (h + d)] = (char)(w >> (24 - 8 * d));
            if (h + 4 >= nd) break;
            x /= 10000u;
          }
        }
        out.at += __shfl_sync(0xffffffffu, inc, 31);
      }
      __syncwarp();
      if (sizeof(T) <= 2) carry = out.buf[out.at >> 2] & ((1u << (8 * (out.at & 3u))) - 1u);
    }
    out.flush(lane, t + kTextTile >= hi);
  }
}

static unsigned warp_grid(hd_ctx *ctx, uint64_t rows) {
  uint64_t g = ceil_div(rows * 32, 256);
  uint64_t cap = (uint64_t)ctx->sm_count * 16;
  return (unsigned)(g < cap ? (g ? g : 1) : cap);
}

uint64_t lt_text_bound(uint64_t i_lo, uint64_t i_hi, int dtype_bytes) {
  if (i_lo < 1) i_lo = 1;
  if (i_hi <= i_lo) return 0;
  const uint64_t entries = row_index(i_hi) - row_index(i_lo);
  const uint64_t per = dtype_bytes == 1 ? 4 : dtype_bytes == 2 ? 6 : 11;
  return entries * per;
}

// Stretches of the text: 48 warps per SM at most (six resident blocks).
constexpr uint64_t kMaxStretches = 16384;
static uint64_t max_stretches(hd_ctx *ctx) {
  return std::min<uint64_t>(kMaxStretches, (uint64_t)ctx->sm_count * 48);
}

// Queues the text of rows [i_lo, i_hi) (i_lo >= 1) on the context's stream:
// lengths, offsets, text. `sums` has room for kMaxStretches + kTextWarps
// lengths; the text's length goes to *d_total (device).
template <typename T>
static void queue_lt_text(hd_ctx *ctx, const T *d_lt, uint64_t lt_base, uint64_t i_lo, uint64_t i_hi,
                          uint64_t *sums, uint64_t *d_total, uint64_t capacity, char *d_text) {
  TextRun<T> run{d_lt + (row_index(i_lo) - lt_base), row_index(i_lo),
                 row_index(i_hi) - row_index(i_lo), 0};
  const uint64_t end = run.n + run.shift();
  run.per = round_up(ceil_div(end, max_stretches(ctx)), kTextTile);
  const unsigned blocks = (unsigned)ceil_div(ceil_div(end, run.per), kTextWarps);
  cudaStream_t st = ctx->stream;
  k_lt_len<T><<<blocks, kTextThreads, 0, st>>>(run, sums);
  HD_LAUNCHED(ctx);
  k_scan_top<void><<<1, 1024, 0, st>>>(sums, (uint64_t)blocks * kTextWarps, d_total);
  HD_LAUNCHED(ctx);
  k_lt_write<T><<<blocks, kTextThreads, 0, st>>>(run, sums, d_total, capacity, d_text);
  HD_LAUNCHED(ctx);
}

uint64_t format_lt_rows(hd_ctx *ctx, const void *d_lt, int dtype_bytes, uint64_t lt_base,
                        uint64_t i_lo, uint64_t i_hi, char *d_text) {
  if (i_lo < 1) i_lo = 1;
  if (i_hi <= i_lo) return 0;
  cudaStream_t st = ctx->stream;
  DevBuf sums((kMaxStretches + kTextWarps + 1) * 8, st);
  uint64_t *sp = sums.as<uint64_t>(), *tot = sp + kMaxStretches + kTextWarps;
  if (dtype_bytes == 1)
    queue_lt_text(ctx, (const uint8_t *)d_lt, lt_base, i_lo, i_hi, sp, tot, ~0ull, d_text);
  else if (dtype_bytes == 2)
    queue_lt_text(ctx, (const uint16_t *)d_lt, lt_base, i_lo, i_hi, sp, tot, ~0ull, d_text);
  else
    queue_lt_text(ctx, (const uint32_t *)d_lt, lt_base, i_lo, i_hi, sp, tot, ~0ull, d_text);
  uint64_t total = 0;
  HD_CUDA(cudaMemcpyAsync(&total, tot, 8, cudaMemcpyDeviceToHost, st));
  HD_CUDA(cudaStreamSynchronize(st));
  return total;
}

// ------------------------------------------------------ full matrix text
// DataSet::dump (include/hamming/hamming.hh:63-73): row i of the n x n matrix,
// entries (*this)[{i, j}] (0 on the diagonal, lt[i(i-1)/2 + j] below it and
// lt[j(j-1)/2 + i] above it), ", " between entries, '\n' after the row. An
// index past the `entries` values read as 0 (a triangle whose size is not
// n(n-1)/2, where the reference reads out of bounds).
template <typename T>
__device__ inline uint32_t full_entry(const T *lt, uint64_t entries, uint64_t i, uint64_t j) {
  if (i == j) return 0u;
  const uint64_t k = i > j ? row_index(i) + j : row_index(j) + i;
  return k < entries ? (uint32_t)lt[k] : 0u;
}

template <typename T>
__global__ void k_full_len(const T *lt, uint64_t entries, uint64_t n, uint64_t i_lo, uint64_t rows,
                           uint64_t *row_len) {
  const int lane = threadIdx.x & 31;
  uint64_t wid = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  for (uint64_t q = wid; q < rows; q += nwarps) {
    const uint64_t i = i_lo + q;
    uint64_t len = 0;
    for (uint64_t j = lane; j < n; j += 32) len += ndig(full_entry(lt, entries, i, j)) + 2;
    len = warp_sum(len);
    if (lane == 0) row_len[q] = len - 1;  // the last entry has "\n" instead of ", "
  }
}

template <typename T>
__global__ void k_full_write(const T *lt, uint64_t entries, uint64_t n, uint64_t i_lo, uint64_t rows,
                             const uint64_t *row_off, char *text) {
  const int lane = threadIdx.x & 31;
  uint64_t wid = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  for (uint64_t q = wid; q < rows; q += nwarps) {
    const uint64_t i = i_lo + q;
    uint64_t pos = row_off[q];
    for (uint64_t j0 = 0; j0 < n; j0 += 32) {
      const uint64_t j = j0 + lane;
      const bool on = j < n;
      const bool last = j + 1 == n;
      const uint32_t v = on ? full_entry(lt, entries, i, j) : 0u;
      const uint32_t nd = on ? ndig(v) : 0u;
      const uint32_t len = on ? nd + (last ? 1u : 2u) : 0u;
      const uint32_t inc = warp_incl_scan(len);
      if (on) {
        char *dst = text + pos + inc - len;
        put_dec(dst, v, nd);
        if (last) {
          dst[nd] = '\n';
        } else {
          dst[nd] = ',';
          dst[nd + 1] = ' ';
        }
      }
      pos += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
}

uint64_t full_text_bound(uint64_t n, uint64_t i_lo, uint64_t i_hi, int dtype_bytes) {
  if (i_hi <= i_lo) return 0;
  const uint64_t per = dtype_bytes == 1 ? 5 : dtype_bytes == 2 ? 7 : 12;  // digits + ", "
  return (i_hi - i_lo) * (n * per + 1);
}

uint64_t format_full_rows(hd_ctx *ctx, const void *d_lt, uint64_t entries, int dtype_bytes,
                          uint64_t n, uint64_t i_lo, uint64_t i_hi, char *d_text) {
  if (i_hi <= i_lo) return 0;
  const uint64_t rows = i_hi - i_lo;
  cudaStream_t st = ctx->stream;
  DevBuf len(rows * 8, st), off(rows * 8, st), tot(8, st);
  const unsigned g = warp_grid(ctx, rows);
  if (dtype_bytes == 1)
    k_full_len<uint8_t><<<g, 256, 0, st>>>((const uint8_t *)d_lt, entries, n, i_lo, rows, len.as<uint64_t>());
  else if (dtype_bytes == 2)
    k_full_len<uint16_t><<<g, 256, 0, st>>>((const uint16_t *)d_lt, entries, n, i_lo, rows, len.as<uint64_t>());
  else
    k_full_len<uint32_t><<<g, 256, 0, st>>>((const uint32_t *)d_lt, entries, n, i_lo, rows, len.as<uint64_t>());
  HD_LAUNCHED(ctx);
  scan_exclusive<uint64_t>(ctx, len.as<uint64_t>(), off.as<uint64_t>(), rows, tot.as<uint64_t>());
  if (dtype_bytes == 1)
    k_full_write<uint8_t><<<g, 256, 0, st>>>((const uint8_t *)d_lt, entries, n, i_lo, rows, off.as<uint64_t>(), d_text);
  else if (dtype_bytes == 2)
    k_full_write<uint16_t><<<g, 256, 0, st>>>((const uint16_t *)d_lt, entries, n, i_lo, rows, off.as<uint64_t>(), d_text);
  else
    k_full_write<uint32_t><<<g, 256, 0, st>>>((const uint32_t *)d_lt, entries, n, i_lo, rows, off.as<uint64_t>(), d_text);
  HD_LAUNCHED(ctx);
  uint64_t total = 0;
  HD_CUDA(cudaMemcpyAsync(&total, tot.p, 8, cudaMemcpyDeviceToHost, st));
  HD_CUDA(cudaStreamSynchronize(st));
  return total;
}

// ----------------------------------------------------------- sparse text
// Lines "i j d\n" for j < i with d <= threshold (integer compare, as the
// reference's `*d <= threshold`).
template <typename T>
__global__ void k_sp_len(const T *lt, uint64_t lt_base, uint64_t i_lo, uint64_t rows, int64_t thr,
                         uint64_t *row_bytes, uint64_t *row_lines) {
  const int lane = threadIdx.x & 31;
  uint64_t wid = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  for (uint64_t q = wid; q < rows; q += nwarps) {
    const uint64_t i = i_lo + q;
    const T *rp = lt + (row_index(i) - lt_base);
    const uint32_t ndi = ndig((uint32_t)i);
    uint64_t bytes = 0, lines = 0;
    for (uint64_t j = lane; j < i; j += 32) {
      const uint32_t d = rp[j];
      if ((int64_t)d <= thr) {
        bytes += ndi + ndig((uint32_t)j) + ndig(d) + 3;
        ++lines;
      }
    }
    bytes = warp_sum(bytes);
    lines = warp_sum(lines);
    if (lane == 0) {
      row_bytes[q] = bytes;
      if (row_lines) row_lines[q] = lines;
    }
  }
}

template <typename T>
__global__ void k_sp_write(const T *lt, uint64_t lt_base, uint64_t i_lo, uint64_t rows, int64_t thr,
                           const uint64_t *row_off, char *text) {
  const int lane = threadIdx.x & 31;
  uint64_t wid = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  for (uint64_t q = wid; q < rows; q += nwarps) {
    const uint64_t i = i_lo + q;
    const T *rp = lt + (row_index(i) - lt_base);
    const uint32_t ndi = ndig((uint32_t)i);
    uint64_t pos = row_off[q];
    for (uint64_t j0 = 0; j0 < i; j0 += 32) {
      const uint64_t j = j0 + lane;
      const uint32_t d = j < i ? (uint32_t)rp[j] : 0u;
      const bool on = j < i && (int64_t)d <= thr;
      const uint32_t ndj = ndig((uint32_t)j), ndd = ndig(d);
      const uint32_t len = on ? ndi + ndj + ndd + 3 : 0u;
      const uint32_t inc = warp_incl_scan(len);
      if (on) {
        char *dst = text + pos + inc - len;
        put_dec(dst, (uint32_t)i, ndi);
        dst[ndi] = ' ';
        put_dec(dst + ndi + 1, (uint32_t)j, ndj);
        dst[ndi + 1 + ndj] = ' ';
        put_dec(dst + ndi + ndj + 2, d, ndd);
        dst[ndi + ndj + ndd + 2] = '\n';
      }
      pos += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
}

void sparse_row_sizes(hd_ctx *ctx, const void *d_lt, int dtype_bytes, uint64_t lt_base,
                      uint64_t i_lo, uint64_t i_hi, int64_t threshold, uint64_t *d_row_bytes,
                      uint64_t *d_row_lines) {
  if (i_lo < 1) i_lo = 1;
  if (i_hi <= i_lo) return;
  const uint64_t rows = i_hi - i_lo;
  const unsigned g = warp_grid(ctx, rows);
  cudaStream_t st = ctx->stream;
  if (dtype_bytes == 1)
    k_sp_len<uint8_t><<<g, 256, 0, st>>>((const uint8_t *)d_lt, lt_base, i_lo, rows, threshold, d_row_bytes, d_row_lines);
  else if (dtype_bytes == 2)
    k_sp_len<uint16_t><<<g, 256, 0, st>>>((const uint16_t *)d_lt, lt_base, i_lo, rows, threshold, d_row_bytes, d_row_lines);
  else
    k_sp_len<uint32_t><<<g, 256, 0, st>>>((const uint32_t *)d_lt, lt_base, i_lo, rows, threshold, d_row_bytes, d_row_lines);
  HD_LAUNCHED(ctx);
}

uint64_t format_sparse_rows(hd_ctx *ctx, const void *d_lt, int dtype_bytes, uint64_t lt_base,
                            uint64_t i_lo, uint64_t i_hi, int64_t threshold,
                            const uint64_t *d_row_bytes, char *d_text) {
  if (i_lo < 1) i_lo = 1;
  if (i_hi <= i_lo) return 0;
  const uint64_t rows = i_hi - i_lo;
  cudaStream_t st = ctx->stream;
  DevBuf off(rows * 8, st), tot(8, st);
  scan_exclusive<uint64_t>(ctx, d_row_bytes, off.as<uint64_t>(), rows, tot.as<uint64_t>());
  const unsigned g = warp_grid(ctx, rows);
  if (dtype_bytes == 1)
    k_sp_write<uint8_t><<<g, 256, 0, st>>>((const uint8_t *)d_lt, lt_base, i_lo, rows, threshold, off.as<uint64_t>(), d_text);
  else if (dtype_bytes == 2)
    k_sp_write<uint16_t><<<g, 256, 0, st>>>((const uint16_t *)d_lt, lt_base, i_lo, rows, threshold, off.as<uint64_t>(), d_text);
  else
    k_sp_write<uint32_t><<<g, 256, 0, st>>>((const uint32_t *)d_lt, lt_base, i_lo, rows, threshold, off.as<uint64_t>(), d_text);
  HD_LAUNCHED(ctx);
  uint64_t total = 0;
  HD_CUDA(cudaMemcpyAsync(&total, tot.p, 8, cudaMemcpyDeviceToHost, st));
  HD_CUDA(cudaStreamSynchronize(st));
  return total;
}

}  // namespace hd

// ===================================================== allocation-free text
// A variant of the lower-triangular formatter above for callers that must not
// allocate device memory: code that runs inside a host application whose
// device memory is fully owned by its own allocator or capped by a fixed
// budget, and latency-critical loops that cannot afford cudaMalloc/cudaFree
// (cudaFree synchronises the whole device). Its scratch (the blocks' text
// lengths and offsets) lives in one file-scope device array of fixed size
// instead of pool allocations.
namespace {

constexpr uint64_t kNoAllocMaxRows = 262144;  // rows of text (nsamples - 1)
constexpr uint64_t kNoAllocSums = hd::kMaxStretches + hd::kTextWarps;
constexpr uint64_t kNoAllocWords = kNoAllocSums + 8;

// Held by every GPU that loads the library, until the process exits.
static __device__ __align__(256) uint64_t g_noalloc_scratch[kNoAllocWords];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
uint64_t *g_noalloc_ptr[kNoAllocMaxDevices] = {};

// Device address of the scratch array on `device`, looked up once per device
// with that device current (in host code the array's name is only a host-side
// stand-in, not a device address).
uint64_t *noalloc_scratch(int device) {
  if (device < 0 || device >= kNoAllocMaxDevices)
    hd::fail(HD_ERR_ARG, "device ordinal out of range for the allocation-free formatter");
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_ptr[device]) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess)
      hd::fail(HD_ERR_CUDA, std::string("cudaGetSymbolAddress failed: ") + cudaGetErrorString(e));
    g_noalloc_ptr[device] = static_cast<uint64_t *>(p);
  }
  return g_noalloc_ptr[device];
}

template <typename T>
uint64_t noalloc_text(hd_ctx *ctx, const T *d_lt, uint64_t nsamples, char *d_text,
                      uint64_t capacity, uint64_t *scratch) {
  uint64_t *total = scratch + kNoAllocSums;
  // every scratch word read is written earlier in this call, so nothing has
  // to be cleared between calls; a text above the capacity is not written and
  // the caller reports the shortfall
  hd::queue_lt_text(ctx, d_lt, 0, 1, nsamples, scratch, total, capacity, d_text);
  uint64_t bytes = 0;
  HD_CUDA(cudaMemcpyAsync(&bytes, total, sizeof(bytes), cudaMemcpyDeviceToHost, ctx->stream));
  HD_CUDA(cudaStreamSynchronize(ctx->stream));
  return bytes;
}

}  // namespace

extern "C" int hd_lower_triangular_text_noalloc(hd_ctx *ctx, const void *d_lt, uint64_t nsamples,
                                                int dtype_bytes, char *d_text,
                                                uint64_t text_capacity, uint64_t *text_bytes) {
  if (!ctx || !text_bytes) return HD_ERR_ARG;
  *text_bytes = 0;
  try {
    HD_CUDA(cudaSetDevice(ctx->device));
    if (dtype_bytes != 1 && dtype_bytes != 2 && dtype_bytes != 4)
      hd::fail(HD_ERR_ARG, "dtype_bytes must be 1, 2 or 4");
    if (nsamples > kNoAllocMaxRows)
      hd::fail(HD_ERR_ARG, "hd_lower_triangular_text_noalloc: nsamples " + std::to_string(nsamples) +
                               " exceeds its fixed scratch limit of " +
                               std::to_string(kNoAllocMaxRows) + " rows");
    if (nsamples < 2) return HD_OK;  // no entries, no text
    if (!d_lt || (!d_text && text_capacity)) hd::fail(HD_ERR_ARG, "null buffer");
    uint64_t *scratch = noalloc_scratch(ctx->device);
    uint64_t need;
    if (dtype_bytes == 1)
      need = noalloc_text(ctx, static_cast<const uint8_t *>(d_lt), nsamples, d_text, text_capacity, scratch);
    else if (dtype_bytes == 2)
      need = noalloc_text(ctx, static_cast<const uint16_t *>(d_lt), nsamples, d_text, text_capacity, scratch);
    else
      need = noalloc_text(ctx, static_cast<const uint32_t *>(d_lt), nsamples, d_text, text_capacity, scratch);
    *text_bytes = need;
    if (need > text_capacity)
      hd::fail(HD_ERR_ARG, "text buffer too small: " + std::to_string(need) + " bytes needed");
    return HD_OK;
  } catch (const hd::Error &e) {
    ctx->err = e.msg;
    return e.code;
  }
}

