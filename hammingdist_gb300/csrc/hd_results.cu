// Device readers of the reference's result files.
//
// Replace from_lower_triangular<T> (include/hamming/hamming.hh:152-166) and
// from_csv / DataSet(filename) (hamming.hh:34-55, src/hamming.cc:23-25),
// which parse on the host with std::getline + std::istringstream + std::stoi.
// A field is parsed with the rules of std::stoi by the thread that holds its
// start. The lower triangle is one flat run of fields; for the full matrix the
// device newline index splits the file into lines, one warp walks a line 32
// bytes at a time and finds its commas with a ballot.
//  - from_lower_triangular: every comma-separated field of every line (an
//    empty line or a trailing comma gives an empty field, which std::stoi
//    rejects), values through safe_int_cast<T>
//    (include/hamming/hamming_impl.hh:37-45: above the maximum saturates,
//    below 0 wraps).
//  - from_csv: nsamples = number of '\n'; line i gives its first i fields to
//    result[i(i-1)/2 + j] of nsamples(nsamples+1)/2 zero-initialised values;
//    when the line has fewer, std::getline leaves the last field in place, so
//    the missing fields repeat it; values are truncated to uint8.
// The first field std::stoi would reject, in file order, decides the error:
// no digits (std::invalid_argument) or a value outside int
// (std::out_of_range).
#include <climits>
#include <cmath>

#include "hd_internal.cuh"

namespace hd {

namespace {

// std::stoi on p[a..): C-locale whitespace, an optional sign, then digits up
// to the first non-digit. Returns 0 (value in *v), 1 (no digits) or 2
// (outside int). Bytes past `end` are not read. A field's own end needs no
// check: ',' stops every phase.
__device__ inline int dev_stoi(const uint8_t *p, uint64_t a, uint64_t end, int *v) {
  uint64_t k = a;
  while (k < end) {
    const uint8_t c = p[k];
    if (c == ' ' || c == '\t' || c == '\n' || c == '\v' || c == '\f' || c == '\r') ++k;
    else break;
  }
  bool neg = false;
  if (k < end && (p[k] == '+' || p[k] == '-')) {
    neg = p[k] == '-';
    ++k;
  }
  const uint64_t d0 = k;
  long long acc = 0;
  while (k < end && p[k] >= '0' && p[k] <= '9') {
    if (acc < (1ll << 40)) acc = acc * 10 + (p[k] - '0');
    ++k;
  }
  if (k == d0) return 1;
  if (neg) acc = -acc;
  if (acc > INT_MAX || acc < INT_MIN) return 2;
  *v = (int)acc;
  return 0;
}

// safe_int_cast<T>(x): x above the maximum saturates, otherwise static_cast
template <typename T>
__device__ inline T safe_cast(int x) {
  const int mx = (int)(T)~(T)0;
  return x > mx ? (T)mx : (T)x;
}

// line k of M: [start, end)
__device__ inline void line_span(uint64_t k, const uint64_t *nl, uint64_t m_nl, uint64_t n,
                                 uint64_t &start, uint64_t &end) {
  start = k ? nl[k - 1] + 1 : 0;
  end = k < m_nl ? nl[k] : n;
}

__device__ inline void note_error(unsigned long long *err, uint64_t key, int kind) {
  atomicMin(err, (unsigned long long)((key << 2) | (uint64_t)kind));
}

// Calls f(field index in line, field start) for the fields of line [s, e)
// with index < limit, from the lane that sees the field's start; the warp
// stops after `limit` fields. Returns the line's number of fields seen (all
// of them when the line has fewer than `limit`).
template <class F>
__device__ inline uint64_t walk_fields(const uint8_t *p, uint64_t s, uint64_t e, uint64_t limit,
                                       int lane, F &&f) {
  if (limit == 0) return 0;
  if (lane == 0) f(0ull, s);
  uint64_t commas = 0;
  for (uint64_t x0 = s; x0 < e && commas + 1 < limit; x0 += 32) {
    const uint64_t x = x0 + lane;
    const bool comma = x < e && p[x] == ',';
    const uint32_t m = __ballot_sync(0xffffffffu, comma);
    const uint64_t idx = commas + 1 + __popc(m & ((1u << lane) - 1u));
    if (comma && idx < limit) f(idx, x + 1);
    commas += __popc(m);
  }
  return commas + 1;
}

// from_lower_triangular as one flat run: every ',' and '\n' ends a field, so a
// field's index is the number of separators before it (an unterminated last
// line ends its last field at the end of the file). Blocks take equal
// stretches of the text: one pass counts their separators, one block turns the
// counts into offsets, and the parse pass stages a tile in shared memory, where
// each thread parses the fields that start in its 16 bytes, and writes the
// tile's values out in order.
//
// A field of one to three digits is read as one unaligned word: its digits are
// weighted by a byte dot product. Longer fields and any other character
// (spaces, signs, letters) go through dev_stoi. The parse is issue-bound. 9,001
// rows (40.5 M fields, 117 MB of text): counts 40 us, parse 183 us; the newline
// index, field counts and a parse with one warp per line, byte by byte, took
// 1.20 ms (the parse 1.05).
constexpr int kRdThreads = 256;
constexpr uint32_t kRdTile = kRdThreads * 16;

// 16 bytes at aligned offset x of n text bytes; bytes past the end read as '\n'
__device__ __forceinline__ uint4 text16(const uint8_t *p, uint64_t x, uint64_t n) {
  if (x + 16 <= n) return *reinterpret_cast<const uint4 *>(p + x);
  uint32_t w[4] = {0x0A0A0A0Au, 0x0A0A0A0Au, 0x0A0A0A0Au, 0x0A0A0A0Au};
  for (uint32_t k = 0; k < 16 && x + k < n; ++k)
    w[k >> 2] ^= (uint32_t)(p[x + k] ^ 0x0Au) << (8 * (k & 3));
  return make_uint4(w[0], w[1], w[2], w[3]);
}
// bytes equal to ',' or '\n' (0xFF each)
__device__ __forceinline__ uint32_t seps4(uint32_t w) {
  return __vcmpeq4(w, 0x2C2C2C2Cu) | __vcmpeq4(w, 0x0A0A0A0Au);
}
// the 16 bytes' separators as a bit mask
__device__ __forceinline__ uint32_t sep_mask(const uint4 &v) {
  auto nib = [](uint32_t w) {
    const uint32_t e = seps4(w) & 0x08040201u;
    return (e | (e >> 8) | (e >> 16) | (e >> 24)) & 0xFu;
  };
  return nib(v.x) | (nib(v.y) << 4) | (nib(v.z) << 8) | (nib(v.w) << 12);
}
// of those at offsets below n
__device__ __forceinline__ uint32_t below(uint32_t mask, uint64_t x, uint64_t n) {
  return x + 16 <= n ? mask : x >= n ? 0u : mask & ((1u << (uint32_t)(n - x)) - 1u);
}

__global__ void __launch_bounds__(kRdThreads)
    k_sep_count(const uint8_t *p, uint64_t n, uint32_t per_block, uint64_t *sums) {
  __shared__ uint64_t tmp[33];
  const uint64_t x0 = (uint64_t)blockIdx.x * per_block * kRdTile;
  uint64_t c = 0;
  for (uint32_t t = 0; t < per_block; ++t) {
    const uint64_t x = x0 + (uint64_t)t * kRdTile + threadIdx.x * 16;
    if (x < n) c += __popc(below(sep_mask(text16(p, x, n)), x, n));
  }
  uint64_t total;
  block_excl_scan<uint64_t>(c, tmp, total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

template <typename T>
__global__ void __launch_bounds__(kRdThreads)
    k_lt_parse(const uint8_t *p, uint64_t n, uint32_t per_block, const uint64_t *offs, T *out,
               unsigned long long *err) {
  __shared__ __align__(16) uint32_t tile[kRdTile / 4 + 4];  // and the 16 bytes after it
  __shared__ T vals[kRdTile];
  __shared__ uint32_t tmp[33];
  uint64_t base = offs[blockIdx.x];  // separators before the tile
  for (uint32_t t = 0; t < per_block; ++t) {
    const uint64_t x0 = ((uint64_t)blockIdx.x * per_block + t) * kRdTile;
    if (x0 >= n) return;  // block-uniform
    const uint64_t x = x0 + threadIdx.x * 16;
    const uint4 v = text16(p, x < n ? x : n, n);
    reinterpret_cast<uint4 *>(tile)[threadIdx.x] = v;
    if (threadIdx.x == 0) {
      const uint64_t xe = x0 + kRdTile;
      reinterpret_cast<uint4 *>(tile)[kRdThreads] = text16(p, xe < n ? xe : n, n);
    }
    const uint32_t seps = x < n ? below(sep_mask(v), x, n) : 0u;
    uint32_t total;
    const uint32_t before = block_excl_scan<uint32_t>(__popc(seps), tmp, total);  // also: the tile is staged
    // fields start at the file's first byte and after every separator; the one
    // that starts at byte o has tile index = separators of the tile before o,
    // so the tile's fields are first .. last - 1
    const uint8_t *tb = reinterpret_cast<const uint8_t *>(tile);
    auto is_sep = [](uint8_t c) { return c == ',' || c == '\n'; };
    const bool fresh = x0 == 0 || is_sep(p[x0 - 1]);
    const uint32_t bytes = n - x0 < kRdTile ? (uint32_t)(n - x0) : kRdTile;
    const uint32_t first = fresh ? 0u : 1u, last = total + (is_sep(tb[bytes - 1]) ? 0u : 1u);
    const uint32_t at = threadIdx.x * 16;
    const bool carry = at ? is_sep(tb[at - 1]) : fresh;
    uint32_t starts = x < n ? below((seps << 1 | (carry ? 1u : 0u)) & 0xFFFFu, x, n) : 0u;
    while (starts) {
      const uint32_t k = __ffs(starts) - 1, o = at + k;
      starts &= starts - 1;
      const uint32_t idx = before + __popc(seps & ((1u << k) - 1u));
      const uint32_t w = __funnelshift_r(tile[o >> 2], tile[(o >> 2) + 1], 8 * (o & 3u));
      const uint32_t e = seps4(w), digits = w ^ 0x30303030u;
      const uint32_t len = e ? (__ffs(e) - 1) >> 3 : 4u;
      const uint32_t other = ((digits + 0x76767676u) | digits) & 0x80808080u;  // not 0-9
      uint32_t value;
      if (len - 1u < 3u && !(other & ((1u << (8 * len)) - 1u))) {
        constexpr uint32_t kMax = (T)~(T)0;
        value = __dp4a(digits, 0x00010A64u >> (8 * (3 - len)), 0u);
        value = value > kMax ? kMax : value;
      } else {
        // its own end stops every phase of std::stoi but the whitespace (a '\n'
        // is one): nothing after the number is read, however long the field
        uint64_t s = x + k;
        while (s < n && (p[s] == ' ' || (p[s] >= '\t' && p[s] <= '\r' && p[s] != '\n'))) ++s;
        int r_v = 0;
        const int r = s < n && !is_sep(p[s]) ? dev_stoi(p, s, n, &r_v) : 1;
        if (r) note_error(err, base + idx, r);
        value = r ? 0u : (uint32_t)safe_cast<T>(r_v);
      }
      vals[idx] = (T)value;
    }
    __syncthreads();
    for (uint32_t k = first + threadIdx.x; k < last; k += kRdThreads) out[base + k] = vals[k];
    base += total;
    __syncthreads();  // the tile and the values are rewritten next
  }
}

__global__ void k_csv_parse(const uint8_t *p, uint64_t n, const uint64_t *nl, uint64_t m_nl,
                            uint64_t M, uint8_t *out, unsigned long long *err) {
  const int lane = threadIdx.x & 31;
  uint64_t wid = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  for (uint64_t i = wid; i < M; i += nwarps) {
    if (i == 0) continue;  // line 0 gives no field
    uint64_t s, e;
    line_span(i, nl, m_nl, n, s, e);
    const uint64_t base = i * (i - 1) / 2;
    uint64_t last_start = s;  // start of the last field seen (uniform after the walk)
    const uint64_t seen = walk_fields(p, s, e, i, lane, [&](uint64_t j, uint64_t at) {
      int v = 0;
      const int r = dev_stoi(p, at, e, &v);
      if (r) note_error(err, base + j, r);
      out[base + j] = r ? (uint8_t)0 : (uint8_t)(unsigned)v;
    });
    if (seen >= i) continue;
    // fewer than i fields: fields seen..i-1 repeat the last one (field seen-1)
    unsigned long long mx = 0;
    for (uint64_t x = s + lane; x < e; x += 32)
      if (p[x] == ',') mx = x + 1;
    for (int o = 16; o; o >>= 1) {
      const unsigned long long y = __shfl_xor_sync(0xffffffffu, mx, o);
      mx = y > mx ? y : mx;
    }
    if (mx) last_start = mx;
    int v = 0;
    const int r = dev_stoi(p, last_start, e, &v);
    for (uint64_t j = seen + lane; j < i; j += 32) {
      if (r) note_error(err, base + j, r);
      out[base + j] = r ? (uint8_t)0 : (uint8_t)(unsigned)v;
    }
  }
}

unsigned line_grid(hd_ctx *ctx, uint64_t lines) {
  uint64_t g = ceil_div(lines * 32, 256);
  const uint64_t cap = (uint64_t)ctx->sm_count * 16;
  return (unsigned)(g < cap ? (g ? g : 1) : cap);
}

uint64_t lines_of(const uint8_t *d, uint64_t nbytes, uint64_t m_nl, cudaStream_t st) {
  // a last line without '\n' counts as a line (std::getline)
  if (!nbytes) return 0;
  uint8_t last = 0;
  HD_CUDA(cudaMemcpyAsync(&last, d + nbytes - 1, 1, cudaMemcpyDeviceToHost, st));
  HD_CUDA(cudaStreamSynchronize(st));
  return m_nl + (last != '\n' ? 1 : 0);
}

int decode_error(unsigned long long e) { return e == ~0ull ? 0 : (int)(e & 3ull); }

}  // namespace

ParsedValues read_lower_triangular_device(hd_ctx *ctx, const uint8_t *d, uint64_t nbytes,
                                          int dtype_bytes) {
  cudaStream_t st = ctx->stream;
  ParsedValues res;
  if (nbytes) {
    // about 16 blocks per SM
    const uint64_t tiles = ceil_div(nbytes, (uint64_t)kRdTile);
    const uint64_t per = ceil_div(tiles, (uint64_t)ctx->sm_count * 16), blocks = ceil_div(tiles, per);
    DevBuf sums((blocks + 2) * 8, st);  // offsets, then the separators and the first error
    uint64_t *sp = sums.as<uint64_t>();
    auto *err = reinterpret_cast<unsigned long long *>(sp + blocks + 1);
    HD_CUDA(cudaMemsetAsync(err, 0xff, 8, st));
    k_sep_count<<<(unsigned)blocks, kRdThreads, 0, st>>>(d, nbytes, (uint32_t)per, sp);
    HD_LAUNCHED(ctx);
    k_scan_top<void><<<1, 1024, 0, st>>>(sp, blocks, sp + blocks);
    HD_LAUNCHED(ctx);
    uint64_t F = 0;
    uint8_t tail = 0;
    HD_CUDA(cudaMemcpyAsync(&F, sp + blocks, 8, cudaMemcpyDeviceToHost, st));
    HD_CUDA(cudaMemcpyAsync(&tail, d + nbytes - 1, 1, cudaMemcpyDeviceToHost, st));
    HD_CUDA(cudaStreamSynchronize(st));
    if (tail != '\n') ++F;  // an unterminated last line ends its last field
    res.entries = F;
    res.values = DevBuf((F ? F : 1) * dtype_bytes, st);
    if (dtype_bytes == 1)
      k_lt_parse<uint8_t><<<(unsigned)blocks, kRdThreads, 0, st>>>(d, nbytes, (uint32_t)per, sp,
                                                                  res.values.as<uint8_t>(), err);
    else
      k_lt_parse<uint16_t><<<(unsigned)blocks, kRdThreads, 0, st>>>(d, nbytes, (uint32_t)per, sp,
                                                                   res.values.as<uint16_t>(), err);
    HD_LAUNCHED(ctx);
    unsigned long long e = 0;
    HD_CUDA(cudaMemcpyAsync(&e, err, 8, cudaMemcpyDeviceToHost, st));
    HD_CUDA(cudaStreamSynchronize(st));
    // a ',' that ends the file leaves an empty last field
    if (e == ~0ull && tail == ',') e = ((F - 1) << 2) | 1;
    res.error = decode_error(e);
  } else {
    res.values = DevBuf(dtype_bytes, st);
  }
  // include/hamming/hamming.hh:18-20, 57-61
  res.nsamples = ((uint64_t)std::llround(std::sqrt((double)(8 * res.entries + 1))) + 1) / 2;
  return res;
}

ParsedValues read_csv_device(hd_ctx *ctx, const uint8_t *d, uint64_t nbytes) {
  cudaStream_t st = ctx->stream;
  ParsedValues res;
  uint64_t m_nl = 0;
  DevBuf nl = newline_positions(ctx, d, nbytes, &m_nl);
  const uint64_t M = lines_of(d, nbytes, m_nl, st);
  res.nsamples = m_nl;
  res.entries = m_nl * (m_nl + 1) / 2;
  res.values = DevBuf(res.entries ? res.entries : 1, st);
  if (res.entries) HD_CUDA(cudaMemsetAsync(res.values.p, 0, res.entries, st));
  if (M > 1) {
    DevBuf err(8, st);
    HD_CUDA(cudaMemsetAsync(err.p, 0xff, 8, st));
    k_csv_parse<<<line_grid(ctx, M), 256, 0, st>>>(d, nbytes, nl.as<uint64_t>(), m_nl, M,
                                                   res.values.as<uint8_t>(),
                                                   err.as<unsigned long long>());
    HD_LAUNCHED(ctx);
    unsigned long long e = 0;
    HD_CUDA(cudaMemcpyAsync(&e, err.p, 8, cudaMemcpyDeviceToHost, st));
    HD_CUDA(cudaStreamSynchronize(st));
    res.error = decode_error(e);
  }
  return res;
}

}  // namespace hd
