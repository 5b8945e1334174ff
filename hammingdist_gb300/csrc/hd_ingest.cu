// Device FASTA ingest: newline index, record table, duplicate removal,
// consensus counts, bit-plane packing and reference distances.
//
// Replaces (ssciwr/hammingdist 1.4.0): read_fasta src/hamming_impl.cc:200-242,
// validate_data :80-91, to_dense_data/from_string :190-198/:244-267, the
// consensus of get_reference_expression :142-168 as used by the heuristic of
// include/hamming/hamming_impl.hh:104-118, and fasta_reference_distances /
// fasta_sequence_indices src/hamming.cc:76-141.
#include "hd_internal.cuh"

namespace hd {

// ------------------------------------------------------------ code tables
// Bit p of a code = membership in bit plane p. A pair of sites matches when
// their codes share a bit, so '-' (all ones) matches everything and a code of
// 0 matches nothing.
//  kCodesAnd:     the reference's 4-bit codes (src/hamming_impl.cc:23-44 with
//                 include_x = false): A C G T one-hot, '-' = 1111, else 0000.
//  kCodesSparse:  the sparse rule (src/hamming_impl.cc:93-129) with X invalid:
//                 codes differ and neither is '-' <=> no shared bit, with a
//                 fifth plane for the class of all invalid bytes.
//  kCodesSparseX: the same with X a symbol of its own (6 planes).
void code_table(int table, uint8_t out[256]) {
  for (int c = 0; c < 256; ++c) out[c] = 0;
  if (table == kCodesSparse)
    for (int c = 0; c < 256; ++c) out[c] = 0x10;
  if (table == kCodesSparseX)
    for (int c = 0; c < 256; ++c) out[c] = 0x20;
  out['A'] = 0x1;
  out['C'] = 0x2;
  out['G'] = 0x4;
  out['T'] = 0x8;
  if (table == kCodesAnd) out['-'] = 0x0f;
  if (table == kCodesSparse) out['-'] = 0x1f;
  if (table == kCodesSparseX) {
    out['X'] = 0x10;
    out['-'] = 0x3f;
  }
}

struct Table256 {
  uint8_t v[256];
};

// ------------------------------------------------------------ newline index
constexpr int kNlThreads = 256;
constexpr int kNlIters = 16;
constexpr int kNlBatch = 8;                                               // vectors loaded at once
constexpr int kNlWarps = kNlThreads / 32;
constexpr uint64_t kNlWarpBytes = 32ull * 16 * kNlIters;                  // 8 KB
constexpr uint64_t kNlBlockBytes = kNlWarpBytes * kNlWarps;               // 64 KB

__device__ inline uint32_t nl_nibble(uint32_t w) {
  uint32_t e = __vcmpeq4(w, 0x0a0a0a0au) & 0x01010101u;
  return (e | (e >> 7) | (e >> 14) | (e >> 21)) & 0xfu;
}
// 0x80 bits, nonzero exactly where some byte of w is '\n' (the lowest such
// byte is exact, bytes above it may be flagged too: only whether there is one)
__device__ inline uint32_t nl_any(uint32_t w) {
  const uint32_t x = w ^ 0x0a0a0a0au;
  return (x - 0x01010101u) & ~x & 0x80808080u;
}
// 16-bit mask of the '\n' bytes of a vector
__device__ inline uint32_t nl_mask(uint4 v) {
  if (!(nl_any(v.x) | nl_any(v.y) | nl_any(v.z) | nl_any(v.w))) return 0;
  return nl_nibble(v.x) | (nl_nibble(v.y) << 4) | (nl_nibble(v.z) << 8) | (nl_nibble(v.w) << 12);
}

// 16-bit mask of '\n' bytes in p[off, off+16).
__device__ inline uint32_t nl_mask16(const uint8_t *p, uint64_t off, uint64_t n) {
  if (off + 16 <= n) return nl_mask(__ldg(reinterpret_cast<const uint4 *>(p + off)));
  uint32_t m = 0;
  for (int k = 0; k < 16; ++k)
    if (off + k < n && p[off + k] == '\n') m |= 1u << k;
  return m;
}

// Whether the line after the newline at `pos` is a header: it starts with '>'.
__device__ inline bool header_after(const uint8_t *p, uint64_t pos, uint64_t n) {
  return pos + 1 < n && p[pos + 1] == '>';
}

// Newlines and (kHdr) newlines that a header line follows: per 64 KB block
// (counts: newlines | headers << 32) and per 8 KB warp span (warp_counts[w]:
// newlines | headers << 16). A span with one or two newlines also records
// their offsets in the span with their header flag (warp_counts[W + 2 w] and
// [W + 2 w + 1] = offset << 1 | flag, W = the launch's warps), so that the
// write pass need not read it again: a FASTA line is usually longer than a
// span. Each lane keeps the first two newlines of its own 16-byte slices,
// which it visits in increasing order; the span's first newline is the least
// of the lanes' first ones, and its second the least of the rest.
// DRAM-bound: a lane has 8 vectors in flight, and a vector without a newline
// costs 4 short tests: 598 MB in 83 us, 7.2 TB/s (4 in flight, with a full
// mask of each: 112 us).
template <bool kHdr>
__global__ void __launch_bounds__(kNlThreads)
    k_nl_count(const uint8_t *p, uint64_t n, uint64_t *counts, uint32_t *warp_counts) {
  __shared__ uint32_t sums[kNlWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t wbase = blockIdx.x * kNlBlockBytes + warp * kNlWarpBytes;
  constexpr uint32_t kNone = 0xFFFFFFFFu;
  uint32_t c = 0, h = 0, o0 = kNone, o1 = kNone;
  auto take = [&](uint32_t m, int it) {  // the newlines of slice `it`
    const uint32_t rel = (uint32_t)it * 512u + (uint32_t)lane * 16u;
    while (m) {
      const uint32_t at = rel + (uint32_t)(__ffs(m) - 1);
      m &= m - 1;
      const uint32_t f = kHdr && header_after(p, wbase + at, n) ? 1u : 0u;
      if (c == 0) o0 = at << 1 | f;
      else if (c == 1) o1 = at << 1 | f;
      ++c;
      h += f;
    }
  };
  const uint64_t lbase = wbase + lane * 16;
  for (int i0 = 0; i0 < kNlIters; i0 += kNlBatch) {
    uint4 v[kNlBatch];
#pragma unroll
    for (int k = 0; k < kNlBatch; ++k) {
      const uint64_t at = lbase + (i0 + k) * 512ull;
      v[k] = at + 16 <= n ? __ldg(reinterpret_cast<const uint4 *>(p + at)) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int k = 0; k < kNlBatch; ++k) {
      const uint32_t m = nl_mask(v[k]);
      if (m) take(m, i0 + k);
    }
  }
  // the input's last bytes, less than a vector: the last slice of their lane
  if (n % 16 && n - n % 16 >= lbase && n - n % 16 - lbase < kNlWarpBytes &&
      (n - n % 16 - lbase) % 512 == 0)
    take(nl_mask16(p, n - n % 16, n), (int)((n - n % 16 - lbase) / 512));
  const uint32_t cw = __reduce_add_sync(0xffffffffu, c | h << 16);  // at most 8,192 each
  const uint32_t wid = blockIdx.x * kNlWarps + warp;
  if (lane == 0) {
    warp_counts[wid] = cw;
    sums[warp] = cw;
  }
  const uint32_t cn = cw & 0xFFFFu;
  if (cn >= 1 && cn <= 2) {  // warp-uniform
    const uint32_t q1 = __reduce_min_sync(0xffffffffu, o0);
    const uint32_t q2 = __reduce_min_sync(0xffffffffu, o0 == q1 ? o1 : o0);
    if (lane == 0) {
      uint32_t *pos = warp_counts + gridDim.x * kNlWarps + 2ull * wid;
      pos[0] = q1;
      pos[1] = q2;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint64_t t = 0;
#pragma unroll
    for (int w = 0; w < kNlWarps; ++w) t += (uint64_t)(sums[w] & 0xFFFFu) | (uint64_t)(sums[w] >> 16) << 32;
    counts[blockIdx.x] = t;
  }
}

struct ParseSummary {
  unsigned long long m_nl;      // newlines
  unsigned long long lines;     // M
  unsigned long long headers;   // header lines after the first line
  unsigned long long R;         // records before the n limit
  unsigned long long Rk;        // records kept
  unsigned long long max_len;
  unsigned long long len0;
  unsigned long long skip;      // records left out at the start
  unsigned long long n_limit;
  unsigned int unterminated;    // the last line has no '\n'
  unsigned int unequal;
  unsigned int multi;           // some record spans several non-empty lines
  unsigned int pad;
};

// Number of records the getline loop of read_fasta produces
// (src/hamming_impl.cc:216-233): the first line is skipped; every later
// header closes a record; the loop ends when the stream reaches its end,
// which happens on reading an unterminated last line (last_hdr: that line is
// a header).
__device__ inline void count_records(ParseSummary *s, bool last_hdr) {
  const uint64_t M = s->lines;
  const uint64_t R = M == 0 || (M == 1 && s->unterminated)
                         ? 0 : s->headers + 1 - (last_hdr && s->unterminated ? 1 : 0);
  uint64_t skip = s->skip;
  if (skip == ~0ull) skip = R;
  s->R = R;
  s->skip = skip;
  const uint64_t after = R > skip ? R - skip : 0;
  s->Rk = (s->n_limit && s->n_limit < after) ? s->n_limit : after;
}

// One block: the newlines and headers before each block of k_nl_count (off[2 b]
// and off[2 b + 1]) and the summary. first > 0: the bytes before `first`
// (which follows a '\n') belong to records parsed before, so the records up
// to the header that starts there are left out (s->skip: record 0 and those
// whose header line starts before `first`). Latency-bound: a warp scans 512
// counts from coalesced loads, all queued before the first is used, so up to
// 1 GB of input takes one round.
constexpr int kTopPer = 16;
__global__ void __launch_bounds__(1024)
    k_nl_top(const uint8_t *p, uint64_t n, const uint64_t *counts, uint64_t nblk, uint64_t first,
             uint64_t n_limit, uint64_t *off, ParseSummary *s) {
  __shared__ uint64_t tmp[33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint8_t last = threadIdx.x == 0 && n ? p[n - 1] : (uint8_t)'\n';
  uint64_t before = 0;  // headers before the one at `first`
  for (uint64_t q = threadIdx.x; q + 1 < first; q += blockDim.x)
    before += p[q] == '\n' && p[q + 1] == '>' ? 1 : 0;
  uint64_t nl = 0, hd = 0;
  for (uint64_t b0 = 0; b0 < nblk; b0 += 1024 * kTopPer) {
    // 16,384 blocks of at most 2^16 newlines: both sums fit 32 bits. The
    // round's counts are spread over all warps, `per` rows of 32 each.
    const uint64_t rows = (nblk - b0 + 1023) / 1024;
    const int per = rows < kTopPer ? (int)rows : kTopPer;
    const uint64_t i0 = b0 + (uint64_t)warp * 32 * per + lane;
    uint64_t v[kTopPer], run = 0, tot;
#pragma unroll
    for (int k = 0; k < kTopPer; ++k)
      v[k] = k < per && i0 + 32 * k < nblk ? counts[i0 + 32 * k] : 0;
#pragma unroll
    for (int k = 0; k < kTopPer; ++k) {
      if (k >= per) break;
      const uint64_t inc = warp_incl_scan(v[k]);
      v[k] = run + inc - v[k];
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
    // the warps' sums, from lane 0 of each
    const uint64_t ex = __shfl_sync(0xffffffffu, block_excl_scan<uint64_t>(lane ? 0 : run, tmp, tot), 0);
#pragma unroll
    for (int k = 0; k < kTopPer; ++k) {
      const uint64_t x = ex + v[k];
      if (k < per && i0 + 32 * k < nblk)
        *reinterpret_cast<ulonglong2 *>(off + 2 * (i0 + 32 * k)) =
            make_ulonglong2(nl + (x & 0xFFFFFFFFull), hd + (x >> 32));
    }
    nl += tot & 0xFFFFFFFFull;
    hd += tot >> 32;
  }
  uint64_t tot = 0;
  if (first) block_excl_scan<uint64_t>(before, tmp, tot);
  if (threadIdx.x == 0) {
    ParseSummary t{};
    t.m_nl = nl;
    t.headers = hd;
    t.unterminated = last != '\n' ? 1u : 0u;
    t.lines = nl + t.unterminated;
    t.skip = !first ? 0 : first < n ? tot + 1 : ~0ull;
    t.n_limit = n_limit;
    if (nl == 0) count_records(&t, false);
    *s = t;
  }
}

// Writes the positions of every '\n' in increasing order, and (kHdr) for each
// line k >= 1, which follows newline k - 1, the header lines before it and
// whether it is one (lrec[k] = headers << 1 | flag), and the lines of the
// headers (hline[0] = 0 and hline[h], h = 1, 2, ...): each warp starts at its
// block's offsets plus the counts of the block's earlier warps; a span with
// one or two newlines takes their offsets from the count pass, a span with
// more scans its lanes' counts where some lane holds a newline. (A thread per
// span, with the warp going through the spans of more than two newlines,
// took 5 us instead of 17 on 598 MB of genomes, but leaves too few warps for
// files of short lines: 0.45 ms instead of 0.25 for a 6 MB ingest.) The warp
// that writes the last newline counts the records. Nothing is written when
// there are more than `cap` newlines.
template <bool kHdr>
__global__ void __launch_bounds__(kNlThreads)
    k_nl_write(const uint8_t *p, uint64_t n, const uint64_t *block_off, const uint32_t *warp_counts,
               uint64_t cap, uint64_t *nl, uint64_t *lrec, uint64_t *hline, ParseSummary *s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t wid = blockIdx.x * kNlWarps + warp;
  // the block's spans, one a lane
  uint32_t c = lane < kNlWarps ? warp_counts[blockIdx.x * kNlWarps + lane] : 0;
  const uint32_t cw = __shfl_sync(0xffffffffu, c, warp), cn = cw & 0xFFFFu;
  if (cn == 0) return;
  const uint64_t m_nl = s->m_nl;
  if (m_nl > cap) return;
  const uint64_t wbase = blockIdx.x * kNlBlockBytes + warp * kNlWarpBytes;
  if (lane >= warp) c = 0;
  c = __reduce_add_sync(0xffffffffu, c);  // at most 7 x 8,192 newlines
  uint64_t off = block_off[2 * blockIdx.x] + (c & 0xFFFFu);
  uint64_t hoff = block_off[2 * blockIdx.x + 1] + (c >> 16);
  auto put = [&](uint64_t j, uint64_t pos, uint64_t h, bool hdr) {
    nl[j] = pos;
    if (!kHdr) return;
    lrec[j + 1] = h << 1 | (hdr ? 1u : 0u);
    if (hdr) hline[h + 1] = j + 1;
    if (j == 0) hline[0] = 0;
    if (j + 1 == m_nl) count_records(s, hdr);
  };
  if (cn <= 2) {
    const uint32_t *pos = warp_counts + gridDim.x * kNlWarps + 2ull * wid;
    if (lane < (int)cn) {
      const uint32_t a = pos[lane];
      put(off + lane, wbase + (a >> 1), hoff + (lane == 1 ? pos[0] & 1u : 0u), a & 1u);
    }
    return;
  }
  for (int i0 = 0; i0 < kNlIters; i0 += kNlBatch) {
    uint32_t ms[kNlBatch];
#pragma unroll
    for (int k = 0; k < kNlBatch; ++k)
      ms[k] = nl_mask16(p, wbase + (i0 + k) * 512ull + lane * 16, n);
#pragma unroll
    for (int k = 0; k < kNlBatch; ++k) {
      const uint64_t at = wbase + (i0 + k) * 512ull + lane * 16;
      uint32_t m = ms[k];
      if (!__any_sync(0xffffffffu, m != 0)) continue;
      uint32_t hm = 0;  // the newlines a header follows
      if (kHdr)
        for (uint32_t t = m; t; t &= t - 1)
          if (header_after(p, at + __ffs(t) - 1, n)) hm |= t & (0u - t);
      const uint32_t cnt = __popc(m) | __popc(hm) << 16;
      const uint32_t inc = warp_incl_scan(cnt);  // at most 512 each
      uint64_t pos = off + ((inc - cnt) & 0xFFFFu), h = hoff + ((inc - cnt) >> 16);
      for (; m; m &= m - 1) {
        const bool hdr = hm & m & (0u - m);
        put(pos++, at + __ffs(m) - 1, h, hdr);
        h += hdr;
      }
      const uint32_t all = __shfl_sync(0xffffffffu, inc, 31);
      off += all & 0xFFFFu;
      hoff += all >> 16;
    }
  }
}

// The first line of a parse's lines [a, b) that is not empty, and the bytes of
// all of them. The bytes up to the end of line k, line ends left out, only
// grow with k: the first line that is not empty is found by bisection.
struct LineSpan {
  uint64_t start, len;  // of the first non-empty line (0 if none); of all lines
  bool multi;           // several non-empty lines
};
__device__ inline uint64_t line_end(uint64_t k, const uint64_t *nl, uint64_t m_nl, uint64_t n) {
  return k < m_nl ? nl[k] : n;
}
__device__ inline LineSpan record_span(uint64_t r, const uint64_t *nl, const uint64_t *hline,
                                       uint64_t n, const ParseSummary *s) {
  const uint64_t m_nl = s->m_nl;
  const uint64_t a = hline[r] + 1, b = r < s->headers ? hline[r + 1] : s->lines;
  if (a >= b) return {0, 0, false};
  const uint64_t st = nl[a - 1] + 1;  // a >= 1
  auto upto = [&](uint64_t k) { return line_end(k, nl, m_nl, n) - st - (k - a); };
  const uint64_t len = upto(b - 1);
  if (b - a == 1) return {len ? st : 0, len, false};
  if (!len) return {0, 0, false};
  uint64_t lo = a, hi = b - 1;
  if (upto(a)) hi = a;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) / 2;
    if (upto(mid)) hi = mid;
    else lo = mid + 1;
  }
  return {lo == a ? st : nl[lo - 1] + 1, len, upto(lo) != len};
}

// One thread per record: where it starts and its length, and in the summary
// whether all lengths are equal, the largest one, and whether some record
// spans several non-empty lines. The grid covers `cap` newlines.
__global__ void __launch_bounds__(256)
    k_records(const uint64_t *nl, const uint64_t *hline, uint64_t n, uint64_t cap, ParseSummary *s,
              uint64_t *rec_len, uint64_t *rec_start) {
  __shared__ uint64_t len0;
  if (s->m_nl > cap) return;
  const uint64_t Rk = s->Rk, skip = s->skip;
  if (blockIdx.x * (uint64_t)blockDim.x >= Rk) return;  // block-uniform
  const uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  LineSpan v{0, 0, false};
  if (r < Rk) {
    v = record_span(skip + r, nl, hline, n, s);
    rec_len[r] = v.len;
    rec_start[r] = v.start;
  }
  if (threadIdx.x == 0) {
    len0 = blockIdx.x ? record_span(skip, nl, hline, n, s).len : v.len;
    if (blockIdx.x == 0) {
      s->len0 = v.len;
      atomicMax(&s->max_len, (unsigned long long)v.len);
    }
  }
  __syncthreads();
  const bool differ = r < Rk && v.len != len0;
  if (differ) atomicMax(&s->max_len, (unsigned long long)v.len);
  const int unequal = __syncthreads_or(differ), multi = __syncthreads_or(v.multi);
  if (threadIdx.x == 0) {
    if (unequal) atomicOr(&s->unequal, 1u);
    if (multi) atomicOr(&s->multi, 1u);
  }
}

// Gather of multi-line records: a sequence line of a kept record r goes to its
// place after the record's earlier lines, which start at dst_off[r - skip]. A
// warp takes G neighbouring lines: the lanes find one line's place each, then
// the warp copies line after line. G is about 2 KB of lines: the look-ups
// are chains of four loads, which short lines share.
__global__ void __launch_bounds__(256)
    k_gather_lines(const uint8_t *p, const uint64_t *nl, const uint64_t *lrec,
                   const uint64_t *hline, uint64_t n, const ParseSummary *s,
                   const uint64_t *dst_off, uint8_t *dst, int G) {
  const uint64_t wid = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  const uint64_t M = s->lines, m_nl = s->m_nl, skip = s->skip, Rk = s->Rk;
  for (uint64_t k0 = 1 + wid * G; k0 < M; k0 += nwarps * G) {
    uint64_t st = 0, to = 0, l = 0;
    const uint64_t k = k0 + lane;
    if (lane < G && k < M) {
      const uint64_t v = lrec[k], r = v >> 1;
      if (!(v & 1) && r >= skip && r - skip < Rk) {
        st = nl[k - 1] + 1;
        l = line_end(k, nl, m_nl, n) - st;
        const uint64_t a = hline[r] + 1;
        to = dst_off[r - skip] + (st - (nl[a - 1] + 1) - (k - a));
      }
    }
    for (int j = 0; j < G; ++j) {
      const uint64_t lj = __shfl_sync(0xffffffffu, l, j);
      const uint8_t *src = p + __shfl_sync(0xffffffffu, st, j);
      uint8_t *out = dst + __shfl_sync(0xffffffffu, to, j);
      uint64_t i = lane;
      if (lj > 128) {
        for (; i + 96 < lj; i += 128) {
          const uint8_t b0 = src[i], b1 = src[i + 32], b2 = src[i + 64], b3 = src[i + 96];
          out[i] = b0;
          out[i + 32] = b1;
          out[i + 64] = b2;
          out[i + 96] = b3;
        }
      }
      for (; i < lj; i += 32) out[i] = src[i];
    }
  }
}

static unsigned grid_for(uint64_t n, int threads) {
  uint64_t g = ceil_div(n ? n : 1, threads);
  return (unsigned)(g > 0x7fffffffull ? 0x7fffffffull : g);
}

namespace {
// The scratch of a newline pass: [summary][offsets][counts][warp counts]
struct NlScratch {
  uint64_t nblk;
  DevBuf buf;
  ParseSummary *sum;
  uint64_t *counts, *offs;
  uint32_t *wcounts;
  NlScratch(uint64_t nbytes, cudaStream_t st)
      : nblk(ceil_div(nbytes ? nbytes : 1, kNlBlockBytes)),
        buf(128 + nblk * (16 + 8 + 12 * kNlWarps), st) {
    static_assert(sizeof(ParseSummary) <= 128, "summary");
    uint8_t *b = buf.as<uint8_t>();
    sum = reinterpret_cast<ParseSummary *>(b);
    offs = reinterpret_cast<uint64_t *>(b + 128);
    counts = offs + 2 * nblk;
    wcounts = reinterpret_cast<uint32_t *>(counts + nblk);
  }
};
// the summary, once every launch queued before has run
ParseSummary summary_of(hd_ctx *ctx, const ParseSummary *d) {
  ParseSummary *h = reinterpret_cast<ParseSummary *>(pinned_words(ctx));
  HD_CUDA(cudaMemcpyAsync(h, d, sizeof(*h), cudaMemcpyDeviceToHost, ctx->stream));
  HD_CUDA(cudaStreamSynchronize(ctx->stream));
  return *h;
}
}  // namespace

DevBuf newline_positions(hd_ctx *ctx, const uint8_t *d, uint64_t nbytes, uint64_t *m_nl) {
  cudaStream_t st = ctx->stream;
  NlScratch sc(nbytes, st);
  k_nl_count<false><<<(unsigned)sc.nblk, kNlThreads, 0, st>>>(d, nbytes, sc.counts, sc.wcounts);
  HD_LAUNCHED(ctx);
  k_nl_top<<<1, 1024, 0, st>>>(d, nbytes, sc.counts, sc.nblk, 0, 0, sc.offs, sc.sum);
  HD_LAUNCHED(ctx);
  const uint64_t h = summary_of(ctx, sc.sum).m_nl;
  *m_nl = h;
  DevBuf nl((h + 1) * 8, st);
  if (h) {
    k_nl_write<false><<<(unsigned)sc.nblk, kNlThreads, 0, st>>>(
        d, nbytes, sc.offs, sc.wcounts, h, nl.as<uint64_t>(), nullptr, nullptr, sc.sum);
    HD_LAUNCHED(ctx);
  }
  return nl;
}

// Four launches and one wait: the tables of the lines and records are laid
// out for one newline per 2 KB of input and 8,192 more, which holds records
// of 4 KB and longer and every small file; an input with more newlines
// repeats the last two launches, which wrote nothing, with tables of its size.
Records parse_fasta(hd_ctx *ctx, const uint8_t *d_file, uint64_t nbytes, uint64_t n_limit,
                    uint64_t first) {
  cudaStream_t st = ctx->stream;
  Records rec;
  NlScratch sc(nbytes, st);
  k_nl_count<true><<<(unsigned)sc.nblk, kNlThreads, 0, st>>>(d_file, nbytes, sc.counts, sc.wcounts);
  HD_LAUNCHED(ctx);
  k_nl_top<<<1, 1024, 0, st>>>(d_file, nbytes, sc.counts, sc.nblk, first, n_limit, sc.offs, sc.sum);
  HD_LAUNCHED(ctx);
  DevBuf tab;
  uint64_t *nl = nullptr, *lrec = nullptr, *hline = nullptr;
  ParseSummary hs;
  uint64_t cap = std::min(nbytes, nbytes / 2048 + 8192);
  for (bool again = false;; again = true) {
    // newlines [0, cap), lines [0, cap + 1), headers [0, cap]; the sizes vary
    // with the input: none of the large blocks kept for rows and results
    tab = DevBuf((3 * cap + 5) * 8, st, true);
    nl = tab.as<uint64_t>();
    lrec = nl + cap + 1;
    hline = lrec + cap + 2;
    rec.rec_len = DevBuf((cap + 1) * 8, st, true);  // records <= newlines + 1
    rec.rec_start = DevBuf((cap + 1) * 8, st, true);
    k_nl_write<true><<<(unsigned)sc.nblk, kNlThreads, 0, st>>>(d_file, nbytes, sc.offs, sc.wcounts,
                                                               cap, nl, lrec, hline, sc.sum);
    HD_LAUNCHED(ctx);
    k_records<<<grid_for(cap + 1, 256), 256, 0, st>>>(nl, hline, nbytes, cap, sc.sum,
                                                      rec.rec_len.as<uint64_t>(),
                                                      rec.rec_start.as<uint64_t>());
    HD_LAUNCHED(ctx);
    hs = summary_of(ctx, sc.sum);
    if (hs.m_nl <= cap) break;
    if (again) fail(HD_ERR_CUDA, "newline counts changed between two passes");
    cap = hs.m_nl;
  }
  rec.n = hs.Rk;
  rec.len0 = hs.len0;
  rec.max_len = hs.max_len;
  rec.all_equal = hs.unequal == 0;
  rec.base = d_file;
  rec.bytes = nbytes;
  if (hs.multi) {
    // records spanning several lines: concatenate them into one buffer
    DevBuf gtot(8, st);
    scan_exclusive<uint64_t>(ctx, rec.rec_len.as<uint64_t>(), rec.rec_start.as<uint64_t>(), rec.n,
                             gtot.as<uint64_t>());
    uint64_t *total = pinned_words(ctx);
    HD_CUDA(cudaMemcpyAsync(total, gtot.p, 8, cudaMemcpyDeviceToHost, st));
    HD_CUDA(cudaStreamSynchronize(st));
    const uint64_t total_bytes = *total;
    rec.gathered = DevBuf(total_bytes + 16, st);
    const uint64_t avg = total_bytes / hs.lines + 1;
    const int G = (int)std::min<uint64_t>(32, 2048 / avg + 1);
    k_gather_lines<<<grid_for(ceil_div(hs.lines, (uint64_t)G) * 32, 256), 256, 0, st>>>(
        d_file, nl, lrec, hline, nbytes, sc.sum, rec.rec_start.as<uint64_t>(),
        rec.gathered.as<uint8_t>(), G);
    HD_LAUNCHED(ctx);
    rec.base = rec.gathered.as<uint8_t>();
    rec.bytes = total_bytes;
  }
  return rec;
}

Records records_from_offsets(hd_ctx *ctx, const uint8_t *d_bytes, const uint64_t *h_offsets,
                             uint64_t n) {
  Records rec;
  rec.n = n;
  rec.base = d_bytes;
  std::vector<uint64_t> start(n ? n : 1), len(n ? n : 1);
  for (uint64_t k = 0; k < n; ++k) {
    start[k] = h_offsets[k] - h_offsets[0];
    len[k] = h_offsets[k + 1] - h_offsets[k];
    rec.max_len = len[k] > rec.max_len ? len[k] : rec.max_len;
    if (len[k] != len[0]) rec.all_equal = false;
  }
  rec.len0 = n ? len[0] : 0;
  rec.bytes = n ? h_offsets[n] - h_offsets[0] : 0;
  rec.rec_start = DevBuf(start.size() * 8, ctx->stream);
  rec.rec_len = DevBuf(len.size() * 8, ctx->stream);
  HD_CUDA(cudaMemcpyAsync(rec.rec_start.p, start.data(), start.size() * 8, cudaMemcpyHostToDevice,
                          ctx->stream));
  HD_CUDA(cudaMemcpyAsync(rec.rec_len.p, len.data(), len.size() * 8, cudaMemcpyHostToDevice,
                          ctx->stream));
  HD_CUDA(cudaStreamSynchronize(ctx->stream));  // host vectors go out of scope
  return rec;
}

// ---------------------------------------------------------------- dedupe
__device__ inline uint64_t mix64(uint64_t x) {
  x ^= x >> 30;
  x *= 0xbf58476d1ce4e5b9ull;
  x ^= x >> 27;
  x *= 0x94d049bb133111ebull;
  x ^= x >> 31;
  return x;
}

constexpr unsigned long long kEmpty = ~0ull;
constexpr int kCmpFast = 4;  // 512-byte blocks per step of warp_equal

__device__ inline uint32_t load4_in(uint64_t x, uint64_t lo, uint64_t hi) {
  if (x >= lo && x + 4 <= hi) return *reinterpret_cast<const uint32_t *>(x);
  uint32_t w = 0;
  for (int k = 0; k < 4; ++k)
    if (x + k >= lo && x + k < hi) w |= (uint32_t)*reinterpret_cast<const uint8_t *>(x + k) << (8 * k);
  return w;
}

// Hash of each record's bytes: a sum over its 8-byte groups (at record
// positions 8q; a short last group is zero-filled) of the 64-bit product of
// the group's two 4-byte halves, each XORed with a position-keyed 32-bit
// constant, then one 64-bit mix of the sum and the length (k_tab_insert).
// Different records rarely share a hash, and equal hashes are verified byte
// by byte, so a collision costs a verify round, never a wrong answer. The sum
// does not depend on the order of its terms, so a record is hashed in
// segments of 4 KB of aligned memory (from its first byte's 16-byte vector
// on), one warp each, that add their partial sums to acc[r] (zeroed first):
// many warps per record keep enough loads in flight however few records there
// are. Block (x, y) takes records 8x .. 8x + 7 (one per warp), segment y. A
// lane reads 16 aligned bytes per step, four 512-byte steps at a time; the two
// groups that start in them start at byte d0 mod 8 (d0 = the record's start
// mod 16) and are realigned with funnel shifts, their last bytes from the next
// lane, or for lane 31 from lane 0 of the next step. Only the record's last
// steps mask bytes. 20,000 records of 29,903 bytes: 106 us, 5.7 TB/s (two
// steps at a time, with masks and look-aheads in every step: 158).
constexpr uint32_t kHashSeg = 4096;
constexpr int kHashWarps = 8;
constexpr int kHashSteps = 4;
constexpr uint32_t kHashKx = 0x9e3779b9u, kHashKy = 0x85ebca6bu;  // per group, odd
// Four steps (2 KB) of a record from the 16-byte aligned address A. kHi: the
// lanes' groups start in the second word of their 8 bytes (d0 mod 8 >= 4); h8:
// at this byte of them; sh: the funnel shift; span: bytes from A to the
// record's end; q: the number of lane 0's first group; before: groups that
// start before this byte are not the record's. kFast: all of the steps' groups
// are whole and readable with the 8 bytes after them.
template <bool kHi, bool kFast>
__device__ __forceinline__ uint64_t hash_steps(uint64_t A, int64_t span, uint32_t h8, uint32_t sh,
                                               uint32_t q, uint32_t before, uint64_t lo,
                                               uint64_t hi, int lane) {
  uint4 v[kHashSteps];
  uint2 nx = make_uint2(0u, 0u);  // lane 31: the 8 bytes after its last 16
#pragma unroll
  for (int k = 0; k < kHashSteps; ++k) {
    const uint32_t off = 512 * k + 16 * lane;
    if (kFast) v[k] = __ldg(reinterpret_cast<const uint4 *>(A + off));
    else v[k] = (int64_t)off < span ? load16_in(A + off, lo, hi) : make_uint4(0u, 0u, 0u, 0u);
  }
  if (lane == 31) {
    constexpr uint32_t off = 512 * kHashSteps;
    if (kFast) nx = __ldg(reinterpret_cast<const uint2 *>(A + off));
    else if ((int64_t)off < span) nx = make_uint2(load4_in(A + off, lo, hi), load4_in(A + off + 4, lo, hi));
  }
  uint32_t kx = (q + 2 * lane) * kHashKx + 0x7f4a7c15u;
  uint32_t ky = (q + 2 * lane) * kHashKy + 0x165667b1u;
  uint64_t h = 0;
#pragma unroll
  for (int k = 0; k < kHashSteps; ++k) {
    constexpr int last = kHashSteps - 1;
    // the next lane's first words: for lane 31 those of the next step's lane 0
    const uint4 &vn = v[k < last ? k + 1 : k];
    uint32_t n0 = __shfl_sync(0xffffffffu, lane == 0 ? vn.x : v[k].x, (lane + 1) & 31), n1 = 0;
    if (kHi) n1 = __shfl_sync(0xffffffffu, lane == 0 ? vn.y : v[k].y, (lane + 1) & 31);
    if (k == last && lane == 31) {
      n0 = nx.x;
      n1 = nx.y;
    }
    const uint32_t wd[5] = {kHi ? v[k].y : v[k].x, kHi ? v[k].z : v[k].y, kHi ? v[k].w : v[k].z,
                            kHi ? n0 : v[k].w, kHi ? n1 : n0};
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      uint32_t x = __funnelshift_r(wd[2 * g], wd[2 * g + 1], sh);
      uint32_t y = __funnelshift_r(wd[2 * g + 1], wd[2 * g + 2], sh);
      bool on = k > 0 || 16 * lane + 8 * g + h8 >= before;
      if (!kFast) {
        const int64_t rem = span - (int64_t)(512 * k + 16 * lane + 8 * g + h8);  // bytes left
        on = on && rem > 0;
        if (rem > 0 && rem < 8) {  // the record's last group: bytes from rem on are 0
          const uint32_t m = (uint32_t)rem;
          y = m > 4u ? y & ((1u << (8u * (m - 4u))) - 1u) : 0u;
          if (m < 4u) x &= (1u << (8u * m)) - 1u;
        }
      }
      x ^= kx + (uint32_t)(64 * k + g) * kHashKx;
      y ^= ky + (uint32_t)(64 * k + g) * kHashKy;
      if (on) h += (uint64_t)x * y;
    }
  }
  return h;
}
// One segment of a record (see k_hash) from its aligned address A
template <bool kHi>
__device__ __forceinline__ uint64_t hash_segment(uint64_t A, int64_t span, uint32_t h8, uint32_t sh,
                                                 uint32_t q, uint32_t before, uint64_t lo,
                                                 uint64_t hi, int lane) {
  constexpr uint32_t kStep = 512 * kHashSteps;
  uint64_t h = 0;
#pragma unroll 1
  for (uint32_t b = 0; b < kHashSeg && (int64_t)b < span; b += kStep) {
    const uint64_t at = A + b;
    const int64_t left = span - b;
    const uint32_t qb = q + (b >> 3), bf = b ? 0u : before;
    if (left >= (int64_t)(kStep + 8) && at >= lo && at + kStep + 16 <= hi)
      h += hash_steps<kHi, true>(at, left, h8, sh, qb, bf, lo, hi, lane);
    else
      h += hash_steps<kHi, false>(at, left, h8, sh, qb, bf, lo, hi, lane);
  }
  return h;
}
__global__ void __launch_bounds__(32 * kHashWarps, 5)
    k_hash(const uint8_t *base, uint64_t bytes, const uint64_t *rs, const uint64_t *rl, uint64_t R,
           unsigned long long *acc) {
  const int lane = threadIdx.x & 31;
  const uint64_t r = (uint64_t)blockIdx.x * kHashWarps + (threadIdx.x >> 5);
  if (r >= R) return;  // warp-uniform
  const uint64_t lo = reinterpret_cast<uint64_t>(base), hi = lo + bytes;
  const uint64_t len = rl[r], P = lo + rs[r];
  if (!len) return;
  const uint32_t d0 = (uint32_t)(P & 15u), h8 = d0 & 7u, sh = 8u * (d0 & 3u);
  for (uint64_t j = blockIdx.y; j * kHashSeg < d0 + len; j += gridDim.y) {
    const uint64_t A = P - d0 + j * kHashSeg;
    const int64_t span = (int64_t)(d0 + len - j * kHashSeg);  // to the record's end
    // group numbers count from the record's start, d0 - h8 bytes into it
    const uint32_t q = (uint32_t)(j * (kHashSeg / 8)) - (d0 >> 3);
    const uint32_t before = j ? 0u : d0;
    uint64_t h = (h8 & 4u) ? hash_segment<true>(A, span, h8, sh, q, before, lo, hi, lane)
                           : hash_segment<false>(A, span, h8, sh, q, before, lo, hi, lane);
    h = warp_sum(h);
    if (lane == 0 && h) atomicAdd(&acc[r], (unsigned long long)h);
  }
}
// Hash sums of records [0, R) of rs/rl into out (R > 0), which is zeroed.
void hash_records(hd_ctx *ctx, const Records &rec, const uint64_t *rs, const uint64_t *rl,
                  uint64_t R, uint64_t *out) {
  if (!rec.max_len) return;
  const uint64_t X = ceil_div(R, (uint64_t)kHashWarps), S = ceil_div(rec.max_len + 15, (uint64_t)kHashSeg);
  if (X > 0x7fffffffull) fail(HD_ERR_ARG, "too many records");
  // segments past 65,535 are taken by the warps' loop
  k_hash<<<dim3((unsigned)X, (unsigned)std::min<uint64_t>(S, 65535)), 32 * kHashWarps, 0, ctx->stream>>>(
      rec.base, rec.bytes, rs, rl, R, reinterpret_cast<unsigned long long *>(out));
  HD_LAUNCHED(ctx);
}

__device__ inline uint64_t slot_of(uint64_t h, uint64_t mask) { return (h ^ (h >> 29)) & mask; }

// The records of one round of duplicate removal: record list[i], or r0 + i
// without a list, i < cnt.
struct RoundList {
  const uint64_t *list;
  uint64_t r0, cnt;
  __device__ uint64_t at(uint64_t i) const { return list ? list[i] : r0 + i; }
};

// The records' hashes into the table: each hash's lowest record index. A round
// without a list is the records' first, and makes their hashes of k_hash's
// sums in place.
__global__ void k_tab_insert(uint64_t *hash, const uint64_t *rl, RoundList L,
                             unsigned long long *keys, unsigned long long *mins, uint64_t mask) {
  uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= L.cnt) return;
  const uint64_t r = L.at(i);
  unsigned long long h = hash[r];
  if (!L.list) {
    h = mix64(h ^ (rl[r] * 0xd6e8feb86659fd93ull));
    h = h == kEmpty ? h - 1 : h;
    hash[r] = h;
  }
  uint64_t slot = slot_of(h, mask);
  for (;;) {
    unsigned long long prev = atomicCAS(&keys[slot], kEmpty, h);
    if (prev == kEmpty || prev == h) {
      atomicMin(&mins[slot], (unsigned long long)r);
      return;
    }
    slot = (slot + 1) & mask;
  }
}

// 16 bytes from byte 4 dw + sh / 8 on of the 32 bytes v, n (dw is warp-uniform)
__device__ __forceinline__ uint4 shifted16(uint4 v, uint4 n, uint32_t dw, uint32_t sh) {
  uint32_t w0, w1, w2, w3, w4;
  switch (dw) {
    case 0: w0 = v.x; w1 = v.y; w2 = v.z; w3 = v.w; w4 = n.x; break;
    case 1: w0 = v.y; w1 = v.z; w2 = v.w; w3 = n.x; w4 = n.y; break;
    case 2: w0 = v.z; w1 = v.w; w2 = n.x; w3 = n.y; w4 = n.z; break;
    default: w0 = v.w; w1 = n.x; w2 = n.y; w3 = n.z; w4 = n.w; break;
  }
  return make_uint4(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh),
                    __funnelshift_r(w2, w3, sh), __funnelshift_r(w3, w4, sh));
}

// Whether the len bytes (len < 2^31) at Pa and at Pb, both inside [lo, hi),
// are equal; called by a whole warp, same result in every lane. a is read
// with aligned 16-byte loads; b's bytes at the same relative positions come
// from b's aligned loads and the next lane's, shifted by d = (Pb - Pa) mod 16:
// whole words by a warp-uniform switch, the rest by funnel shifts. Offsets
// inside the span are 32-bit, and only the windows at its two ends mask
// bytes.
__device__ inline bool warp_equal(uint64_t Pa, uint64_t Pb, uint32_t len, uint64_t lo, uint64_t hi,
                                  int lane) {
  const uint64_t Aa = Pa & ~15ull;
  const uint32_t da = (uint32_t)(Pa - Aa);  // a's first byte in its first window
  const uint64_t Bs = Pb - da;              // b's byte at a's window start (may precede b)
  const uint64_t Ab = Bs & ~15ull;
  const uint32_t d = (uint32_t)(Bs - Ab), dw = d >> 2, sh = 8u * (d & 3u);
  const uint32_t span = da + len;                    // a's windows cover [0, span) from Aa
  const uint32_t b_end = (uint32_t)(Pb + len - Ab);  // b's bytes end there, from Ab
  // steps that end inside the span: all loads before the first use, and only
  // the first window has bytes before a's first
  uint32_t b0 = 0;
  for (; b0 + 512 * kCmpFast <= span && Aa >= lo && Ab + b0 >= lo &&
         Ab + b0 + 512 * kCmpFast + 16 <= hi;
       b0 += 512 * kCmpFast) {
    uint4 va[kCmpFast], vb[kCmpFast + 1];
#pragma unroll
    for (int k = 0; k < kCmpFast; ++k) {
      const uint32_t off = b0 + 512 * k + 16 * lane;
      va[k] = __ldg(reinterpret_cast<const uint4 *>(Aa + off));
      vb[k] = __ldg(reinterpret_cast<const uint4 *>(Ab + off));
    }
    vb[kCmpFast] = make_uint4(0u, 0u, 0u, 0u);
    if (d && lane == 0)  // lane 31 takes its next words from lane 0's next step
      vb[kCmpFast] = __ldg(reinterpret_cast<const uint4 *>(Ab + b0 + 512 * kCmpFast));
    uint32_t diff = 0;
#pragma unroll
    for (int k = 0; k < kCmpFast; ++k) {
      uint4 x = vb[k];
      if (d) {  // warp-uniform
        const int to = (lane + 1) & 31;
        uint4 vn;
        vn.x = __shfl_sync(0xffffffffu, lane ? vb[k].x : vb[k + 1].x, to);
        vn.y = __shfl_sync(0xffffffffu, lane ? vb[k].y : vb[k + 1].y, to);
        vn.z = __shfl_sync(0xffffffffu, lane ? vb[k].z : vb[k + 1].z, to);
        vn.w = __shfl_sync(0xffffffffu, lane ? vb[k].w : vb[k + 1].w, to);
        x = shifted16(vb[k], vn, dw, sh);
      }
      x.x ^= va[k].x;
      x.y ^= va[k].y;
      x.z ^= va[k].z;
      x.w ^= va[k].w;
      if (k == 0 && b0 == 0 && lane == 0 && da) {
        x.x &= da >= 4 ? 0u : 0xffffffffu << (8 * da);
        x.y &= da >= 8 ? 0u : da <= 4 ? 0xffffffffu : 0xffffffffu << (8 * (da - 4));
        x.z &= da >= 12 ? 0u : da <= 8 ? 0xffffffffu : 0xffffffffu << (8 * (da - 8));
        x.w &= da <= 12 ? 0xffffffffu : 0xffffffffu << (8 * (da - 12));
      }
      diff |= x.x | x.y | x.z | x.w;
    }
    if (__any_sync(0xffffffffu, diff != 0)) return false;
  }
  for (; b0 < span; b0 += 512) {
    const uint32_t off = b0 + 16 * lane;
    const bool in = off < span;
    const uint4 va = in ? load16_in(Aa + off, lo, hi) : make_uint4(0u, 0u, 0u, 0u);
    const uint4 vb = off < b_end ? load16_in(Ab + off, lo, hi) : make_uint4(0u, 0u, 0u, 0u);
    uint4 vn;
    vn.x = __shfl_down_sync(0xffffffffu, vb.x, 1);
    vn.y = __shfl_down_sync(0xffffffffu, vb.y, 1);
    vn.z = __shfl_down_sync(0xffffffffu, vb.z, 1);
    vn.w = __shfl_down_sync(0xffffffffu, vb.w, 1);
    if (lane == 31)
      vn = (d && off + 16 < b_end) ? load16_in(Ab + off + 16, lo, hi) : make_uint4(0u, 0u, 0u, 0u);
    const uint4 y = shifted16(vb, vn, dw, sh);
    uint32_t x[4] = {va.x ^ y.x, va.y ^ y.y, va.z ^ y.z, va.w ^ y.w};
    if (!(off >= da && off + 16 <= span)) {
      // a window at an end of the span: only the bytes at positions
      // [0, len) from a's first byte count
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int32_t p = (int32_t)(off + 4 * j) - (int32_t)da;  // the word's first byte
        uint32_t m = in ? 0xffffffffu : 0u;
        if (p < 0) m &= p <= -4 ? 0u : (0xffffffffu << (8 * (uint32_t)(-p)));
        if (p + 4 > (int32_t)len)
          m &= p >= (int32_t)len ? 0u : (0xffffffffu >> (8 * (uint32_t)(p + 4 - (int32_t)len)));
        x[j] &= m;
      }
    }
    if (__any_sync(0xffffffffu, (x[0] | x[1] | x[2] | x[3]) != 0)) return false;
  }
  return true;
}

// Each record's first record of equal hash (dup[r]); the records that are not
// their own are listed to be compared with it (pairs[0 .. *n_pairs), any
// order), those of another length marked as unlike it (differs[i]).
__global__ void k_tab_find(const uint64_t *hash, const uint64_t *rl, RoundList L,
                           const unsigned long long *keys, const unsigned long long *mins,
                           uint64_t mask, uint64_t *dup, uint64_t *pairs,
                           unsigned long long *n_pairs, uint32_t *differs) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  bool pair = false;
  if (i < L.cnt) {
    const uint64_t r = L.at(i);
    const unsigned long long h = hash[r];
    uint64_t slot = slot_of(h, mask);
    while (keys[slot] != h) slot = (slot + 1) & mask;
    const uint64_t rep = mins[slot];
    dup[r] = rep;
    if (rep != r) {
      pair = rl[r] == rl[rep];
      if (!pair) differs[i] = 1u;
    }
  }
  const uint32_t on = __ballot_sync(0xffffffffu, pair);
  if (!on) return;
  unsigned long long at = 0;
  const int lane = threadIdx.x & 31;
  if (lane == __ffs(on) - 1) at = atomicAdd(n_pairs, (unsigned long long)__popc(on));
  at = __shfl_sync(0xffffffffu, at, __ffs(on) - 1);
  if (pair) pairs[at + __popc(on & ((1u << lane) - 1u))] = i;
}

// The verify step: the listed records against their first record of equal
// hash, byte by byte; differs[i] marks a difference (a hash collision, a
// record for the next round). A warp compares segments of 4 KB, one after
// another: few duplicates are spread over all SMs. 6,000 duplicates of
// 29,903 bytes among 20,000 records: 67 us, 5 TB/s (a warp for every segment
// of every record, most of which only looked their record up: 113).
constexpr uint64_t kCmpSeg = 4096;
constexpr int kCmpWarps = 8;
__global__ void __launch_bounds__(32 * kCmpWarps)
    k_tab_cmp(const uint8_t *base, uint64_t bytes, const uint64_t *rs, const uint64_t *rl,
              RoundList L, const uint64_t *dup, const uint64_t *pairs,
              const unsigned long long *n_pairs, uint64_t segs, uint32_t *differs) {
  const int lane = threadIdx.x & 31;
  const uint64_t nwarps = (uint64_t)gridDim.x * kCmpWarps, jobs = *n_pairs * segs;
  const uint64_t lo = reinterpret_cast<uint64_t>(base);
  for (uint64_t job = (uint64_t)blockIdx.x * kCmpWarps + (threadIdx.x >> 5); job < jobs; job += nwarps) {
    const uint64_t k = job / segs, i = pairs[k], r = L.at(i), rep = dup[r];
    // the record's bytes in 4 KB of aligned memory
    const uint64_t len = rl[r], P = lo + rs[r], j = job - k * segs;
    const uint64_t o = j ? j * kCmpSeg - (P & 15u) : 0, e = (j + 1) * kCmpSeg - (P & 15u);
    if (o >= len) continue;
    const uint32_t sl = (uint32_t)((len < e ? len : e) - o);
    const bool eq = warp_equal(P + o, lo + rs[rep] + o, sl, lo, lo + bytes, lane);
    if (!eq && lane == 0) differs[i] = 1u;
  }
}

// Which records are the first of their kind: a bit each (bits, a word per 32
// records), those before each word in its tile of 256 (pre), and the tiles'
// sums. A record unlike the first of its hash (differs) goes to `next` and is
// none for now.
constexpr int kDupTile = 256;
__global__ void __launch_bounds__(kDupTile)
    k_dup_flags(uint64_t r0, uint64_t R, const uint32_t *differs, uint64_t *dup, uint64_t *next,
                unsigned long long *next_cnt, uint32_t *bits, uint32_t *pre, uint64_t *sums) {
  __shared__ uint32_t warp_n[kDupTile / 32];
  const uint64_t i = (uint64_t)blockIdx.x * kDupTile + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  bool first = false;
  if (i < R) {
    first = dup[r0 + i] == r0 + i;
    if (differs && differs[i]) {
      next[atomicAdd(next_cnt, 1ull)] = r0 + i;
      dup[r0 + i] = kEmpty;
    }
  }
  const uint32_t word = __ballot_sync(0xffffffffu, first);
  if (lane == 0) warp_n[warp] = __popc(word);
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kDupTile / 32; ++w) {
    if (w < warp) before += warp_n[w];
    all += warp_n[w];
  }
  if (lane == 0 && i < R) {
    bits[i >> 5] = word;
    pre[i >> 5] = before;
  }
  if (threadIdx.x == 0) sums[blockIdx.x] = all;
}

// The records' rows: the first records numbered in order from k0 (their list
// unique_rec and their rows), the others the row of their first record, which
// may be one of the records before r0 (rowid of those is there).
__global__ void k_dup_number(uint64_t r0, uint64_t R, uint64_t k0, const uint64_t *dup,
                             const uint32_t *bits, const uint32_t *pre, const uint64_t *sums,
                             uint64_t *rowid, uint64_t *unique_rec) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= R) return;
  const uint64_t d = dup[r0 + i];
  if (d == kEmpty) return;  // of the next round
  if (d < r0) {
    rowid[r0 + i] = rowid[d];
    return;
  }
  const uint64_t x = d - r0;
  const uint64_t row =
      k0 + sums[x / kDupTile] + pre[x >> 5] + __popc(bits[x >> 5] & ((1u << (x & 31)) - 1u));
  rowid[r0 + i] = row;
  if (d == r0 + i) unique_rec[row] = d;
}

// The records of a round of equal hash but other bytes, for the next round
__global__ void k_dup_next(RoundList L, const uint32_t *differs, uint64_t *next,
                           unsigned long long *next_cnt) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i < L.cnt && differs[i]) next[atomicAdd(next_cnt, 1ull)] = L.at(i);
}

namespace {
// Scratch of duplicate removal for records [0, R): the counts (pairs to
// compare, records for the next round, first records) and per-record marks,
// zeroed together, then the rest
struct DupScratch {
  DevBuf buf;
  unsigned long long *counts;  // 3
  uint32_t *differs, *bits, *pre;
  uint64_t *pairs, *next, *sums;
  uint64_t zeroed;  // bytes from counts on
  DupScratch(uint64_t R, cudaStream_t st) {
    const uint64_t words = ceil_div(R, (uint64_t)32), tiles = ceil_div(R, (uint64_t)kDupTile);
    zeroed = round_up(32 + R * 4, 16);
    buf = DevBuf(zeroed + 2 * R * 8 + tiles * 8 + words * 8, st, true);
    uint8_t *b = buf.as<uint8_t>();
    counts = reinterpret_cast<unsigned long long *>(b);
    differs = reinterpret_cast<uint32_t *>(b + 32);
    pairs = reinterpret_cast<uint64_t *>(b + zeroed);
    next = pairs + R;
    sums = next + R;
    bits = reinterpret_cast<uint32_t *>(sums + tiles);
    pre = bits + words;
  }
};
// Inserts a round's records, finds their first records and compares.
void compare_round(hd_ctx *ctx, const Records &rec, const RoundList &L, uint64_t *hash,
                   unsigned long long *keys, unsigned long long *mins, uint64_t mask, uint64_t *dup,
                   const DupScratch &sc) {
  cudaStream_t st = ctx->stream;
  const uint64_t *rs = rec.rec_start.as<uint64_t>(), *rl = rec.rec_len.as<uint64_t>();
  k_tab_insert<<<grid_for(L.cnt, 256), 256, 0, st>>>(hash, rl, L, keys, mins, mask);
  HD_LAUNCHED(ctx);
  k_tab_find<<<grid_for(L.cnt, 256), 256, 0, st>>>(hash, rl, L, keys, mins, mask, dup, sc.pairs,
                                                   sc.counts, sc.differs);
  HD_LAUNCHED(ctx);
  const uint64_t segs = ceil_div(rec.max_len + 15, kCmpSeg);
  const uint64_t blocks = ceil_div(L.cnt * segs, (uint64_t)kCmpWarps);
  k_tab_cmp<<<(unsigned)std::min<uint64_t>(blocks, (uint64_t)ctx->sm_count * 8), 32 * kCmpWarps, 0,
              st>>>(rec.base, rec.bytes, rs, rl, L, dup, sc.pairs, sc.counts, segs, sc.differs);
  HD_LAUNCHED(ctx);
}
// Numbers the first records among [r0, r0 + R) from k0 on, from dup; those
// marked in sc.differs are left for another round if `check`
void number_round(hd_ctx *ctx, uint64_t r0, uint64_t R, uint64_t k0, uint64_t *dup, bool check,
                  const DupScratch &sc, uint64_t *rowid, uint64_t *unique_rec) {
  cudaStream_t st = ctx->stream;
  const uint64_t tiles = ceil_div(R, (uint64_t)kDupTile);
  k_dup_flags<<<(unsigned)tiles, kDupTile, 0, st>>>(r0, R, check ? sc.differs : nullptr, dup, sc.next,
                                                    sc.counts + 1, sc.bits, sc.pre, sc.sums);
  HD_LAUNCHED(ctx);
  k_scan_top<void><<<1, 1024, 0, st>>>(sc.sums, tiles, reinterpret_cast<uint64_t *>(sc.counts) + 2);
  HD_LAUNCHED(ctx);
  k_dup_number<<<grid_for(R, 256), 256, 0, st>>>(r0, R, k0, dup, sc.bits, sc.pre, sc.sums, rowid,
                                                 unique_rec);
  HD_LAUNCHED(ctx);
}
}  // namespace

// One round and its numbering are queued together, with one wait: a second
// round is needed only where two records of one hash differ.
DevBuf dedupe(hd_ctx *ctx, const Records &rec, uint64_t *n_unique, std::vector<uint64_t> &seqidx) {
  cudaStream_t st = ctx->stream;
  const uint64_t R = rec.n;
  seqidx.resize(R);
  DevBuf unique_rec((R ? R : 1) * 8, st);
  if (R == 0) {
    *n_unique = 0;
    return unique_rec;
  }
  uint64_t T = 64;
  while (T < 2 * R) T <<= 1;
  DevBuf recs(3 * R * 8, st, true), table(2 * T * 8, st, true);
  uint64_t *hash = recs.as<uint64_t>(), *dup = hash + R, *rowid = dup + R;
  unsigned long long *keys = table.as<unsigned long long>(), *mins = keys + T;
  DupScratch sc(R, st);
  HD_CUDA(cudaMemsetAsync(hash, 0, R * 8, st));
  HD_CUDA(cudaMemsetAsync(sc.counts, 0, sc.zeroed, st));
  HD_CUDA(cudaMemsetAsync(keys, 0xff, 2 * T * 8, st));
  hash_records(ctx, rec, rec.rec_start.as<uint64_t>(), rec.rec_len.as<uint64_t>(), R, hash);
  compare_round(ctx, rec, RoundList{nullptr, 0, R}, hash, keys, mins, T - 1, dup, sc);
  number_round(ctx, 0, R, 0, dup, true, sc, rowid, unique_rec.as<uint64_t>());
  uint64_t *h = pinned_words(ctx);
  auto fetch = [&] {
    HD_CUDA(cudaMemcpyAsync(h, sc.counts, 24, cudaMemcpyDeviceToHost, st));
    HD_CUDA(cudaMemcpyAsync(seqidx.data(), rowid, R * 8, cudaMemcpyDeviceToHost, st));
    HD_CUDA(cudaStreamSynchronize(st));
  };
  fetch();
  if (h[1]) {
    DevBuf lists[2] = {DevBuf(h[1] * 8, st), DevBuf(h[1] * 8, st)};
    HD_CUDA(cudaMemcpyAsync(lists[0].p, sc.next, h[1] * 8, cudaMemcpyDeviceToDevice, st));
    uint64_t todo = h[1];
    for (int round = 0; todo; ++round) {
      const RoundList L{lists[round & 1].as<uint64_t>(), 0, todo};
      HD_CUDA(cudaMemsetAsync(sc.counts, 0, 32 + todo * 4, st));
      HD_CUDA(cudaMemsetAsync(keys, 0xff, 2 * T * 8, st));
      compare_round(ctx, rec, L, hash, keys, mins, T - 1, dup, sc);
      k_dup_next<<<grid_for(todo, 256), 256, 0, st>>>(
          L, sc.differs, lists[(round + 1) & 1].as<uint64_t>(), sc.counts + 1);
      HD_LAUNCHED(ctx);
      HD_CUDA(cudaMemcpyAsync(h, sc.counts, 16, cudaMemcpyDeviceToHost, st));
      HD_CUDA(cudaStreamSynchronize(st));
      if (h[1] >= todo) fail(HD_ERR_CUDA, "duplicate removal made no progress");
      todo = h[1];
    }
    number_round(ctx, 0, R, 0, dup, false, sc, rowid, unique_rec.as<uint64_t>());
    fetch();
  }
  *n_unique = h[2];
  return unique_rec;
}

// ------------------------------------------- incremental duplicate removal
void IncDedupe::init(hd_ctx *ctx, uint64_t capacity) {
  cudaStream_t st = ctx->stream;
  cap = capacity ? capacity : 1;
  T = 64;
  while (T < 2 * cap) T <<= 1;
  recs = DevBuf(3 * cap * 8, st, true);
  unique_rec = DevBuf(cap * 8, st, true);
  table = DevBuf(2 * T * 8, st, true);
  HD_CUDA(cudaMemsetAsync(recs.p, 0, cap * 8, st));  // the hashes
  HD_CUDA(cudaMemsetAsync(table.p, 0xff, 2 * T * 8, st));
  seen = 0;
  n_unique = 0;
}

bool IncDedupe::add(hd_ctx *ctx, const Records &rec) {
  cudaStream_t st = ctx->stream;
  const uint64_t r0 = seen, m = rec.n - seen;
  if (rec.n < seen || rec.n > cap) return false;
  if (m == 0) return true;
  uint64_t *hash = recs.as<uint64_t>(), *dup = hash + cap, *rowid = dup + cap;
  unsigned long long *keys = table.as<unsigned long long>(), *mins = keys + T;
  DupScratch sc(m, st);
  HD_CUDA(cudaMemsetAsync(sc.counts, 0, sc.zeroed, st));
  hash_records(ctx, rec, rec.rec_start.as<uint64_t>() + r0, rec.rec_len.as<uint64_t>() + r0, m,
               hash + r0);
  // earlier records hold the smaller indices: they stay each hash's minimum
  compare_round(ctx, rec, RoundList{nullptr, r0, m}, hash, keys, mins, T - 1, dup, sc);
  number_round(ctx, r0, m, n_unique, dup, true, sc, rowid, unique_rec.as<uint64_t>());
  uint64_t *h = pinned_words(ctx);
  HD_CUDA(cudaMemcpyAsync(h, sc.counts, 24, cudaMemcpyDeviceToHost, st));
  HD_CUDA(cudaStreamSynchronize(st));
  // a new record unlike the first record of its hash: the full dedupe decides
  if (h[1]) return false;
  n_unique += h[2];
  seen = rec.n;
  return true;
}

void IncDedupe::rows(hd_ctx *ctx, std::vector<uint64_t> &seqidx) {
  seqidx.resize(seen);
  if (!seen) return;
  HD_CUDA(cudaMemcpyAsync(seqidx.data(), rowid(), seen * 8, cudaMemcpyDeviceToHost, ctx->stream));
  HD_CUDA(cudaStreamSynchronize(ctx->stream));
}

// -------------------------------------------------------------- consensus
// 0x01 in every byte of w that equals the byte of x
__device__ __forceinline__ uint32_t equal_bytes(uint32_t w, uint32_t x) {
  const uint32_t z = w ^ x, ne = ((z & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | z;
  return ~(ne >> 7) & 0x01010101u;
}

// Counts of A, C, G and T per site over a share of at most 128 rows: a thread
// takes four neighbouring sites, whose counts are the bytes of four words, and
// a share is small enough to use all SMs: 120 rows of 1,273 sites take 5.5 us
// (17 with a byte a load and shares of 128), 2,000 of 29,903 57 (57).
constexpr uint32_t kColRows = 128;
__global__ void __launch_bounds__(256)
    k_colcount(const uint8_t *base, uint64_t bytes, const uint64_t *rs, const uint64_t *rows,
               uint64_t n_rows, uint32_t share, uint64_t L, unsigned int *counts) {
  __shared__ uint64_t start[kColRows];
  const uint64_t u0 = (uint64_t)blockIdx.y * share;
  const uint32_t m = (uint32_t)(n_rows - u0 < share ? n_rows - u0 : share);
  const uint64_t lo = reinterpret_cast<uint64_t>(base), hi = lo + bytes;
  for (uint32_t u = threadIdx.x; u < m; u += blockDim.x) start[u] = lo + rs[rows ? rows[u0 + u] : u0 + u];
  __syncthreads();
  const uint64_t s = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) * 4;
  if ((s & ~127ull) >= L) return;  // warp-uniform
  const uint32_t lane = threadIdx.x & 31;
  uint32_t c[4] = {0u, 0u, 0u, 0u};
  constexpr int kAhead = 8;
  for (uint32_t u = 0; u < m; u += kAhead) {
    uint32_t v[kAhead], n[kAhead], sh[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      v[k] = n[k] = sh[k] = 0u;  // past the share: no symbol
      if (u + k < m) {
        const uint64_t P = start[u + k] + s, A = P & ~3ull;
        sh[k] = 8u * (uint32_t)(P - A);
        // the warp's 128 bytes, and the word after them for lane 31
        const bool in = A - 4 * lane >= lo && A - 4 * lane + 132 <= hi;  // warp-uniform
        v[k] = in ? __ldg(reinterpret_cast<const uint32_t *>(A)) : load4_in(A, lo, hi);
        if (lane == 31 && sh[k])
          n[k] = in ? __ldg(reinterpret_cast<const uint32_t *>(A + 4)) : load4_in(A + 4, lo, hi);
      }
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const uint32_t next = __shfl_down_sync(0xffffffffu, v[k], 1);
      const uint32_t w = __funnelshift_r(v[k], lane == 31 ? n[k] : next, sh[k]);
      c[0] += equal_bytes(w, 0x41414141u);
      c[1] += equal_bytes(w, 0x43434343u);
      c[2] += equal_bytes(w, 0x47474747u);
      c[3] += equal_bytes(w, 0x54545454u);
    }
  }
  for (int k = 0; k < 4 && s + k < L; ++k)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t t = (c[j] >> (8 * k)) & 0xFFu;
      if (t) atomicAdd(&counts[4 * (s + k) + j], t);
    }
}

__global__ void k_colmax_sum(const unsigned int *counts, uint64_t L, unsigned long long *sum) {
  __shared__ uint64_t tmp[33];
  uint64_t v = 0;
  for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < L;
       s += (uint64_t)gridDim.x * blockDim.x) {
    unsigned m = max(max(counts[4 * s], counts[4 * s + 1]), max(counts[4 * s + 2], counts[4 * s + 3]));
    v += m;
  }
  uint64_t tot;
  block_excl_scan<uint64_t>(v, tmp, tot);
  if (threadIdx.x == 0) atomicAdd(sum, (unsigned long long)tot);
}

uint64_t consensus_matches(hd_ctx *ctx, const Records &rec, const uint64_t *d_rows,
                           uint64_t n_rows) {
  cudaStream_t st = ctx->stream;
  const uint64_t L = rec.len0;
  if (!L || !n_rows) return 0;
  DevBuf counts(L * 16, st), sum(8, st);
  HD_CUDA(cudaMemsetAsync(counts.p, 0, L * 16, st));
  HD_CUDA(cudaMemsetAsync(sum.p, 0, 8, st));
  // shares of 128 rows, or fewer where that leaves SMs without a block
  const uint64_t X = ceil_div(L, (uint64_t)1024);
  const uint64_t want = ceil_div((uint64_t)ctx->sm_count * 4, X);
  const uint32_t share = (uint32_t)std::min<uint64_t>(kColRows, std::max<uint64_t>(8, n_rows / want));
  const uint64_t chunks = ceil_div(n_rows, (uint64_t)share);
  for (uint64_t c0 = 0; c0 < chunks; c0 += 65535) {
    uint64_t cn = chunks - c0 < 65535 ? chunks - c0 : 65535;
    dim3 grid((unsigned)X, (unsigned)cn);
    const uint64_t *rows = d_rows ? d_rows + c0 * share : nullptr;
    // without a row list the rows are records [c0 * share, ...): shift the starts
    const uint64_t *rs = rec.rec_start.as<uint64_t>() + (d_rows ? 0 : c0 * share);
    k_colcount<<<grid, 256, 0, st>>>(rec.base, rec.bytes, rs, rows, n_rows - c0 * share, share, L,
                                     counts.as<unsigned int>());
    HD_LAUNCHED(ctx);
  }
  k_colmax_sum<<<(unsigned)(ctx->sm_count * 4), 256, 0, st>>>(counts.as<unsigned int>(), L,
                                                             sum.as<unsigned long long>());
  HD_LAUNCHED(ctx);
  uint64_t h = 0;
  HD_CUDA(cudaMemcpyAsync(&h, sum.p, 8, cudaMemcpyDeviceToHost, st));
  HD_CUDA(cudaStreamSynchronize(st));
  return h;
}

// ------------------------------------------------------------------- pack
// Packing: a warp job is kPackCPG chunks of 32 words (1024 sites each) of
// one row. Per chunk the warp reads the 1024 bytes with coalesced byte loads
// (all issued before use), stages their codes in shared memory, and lane i
// then builds word i from its 32 consecutive codes: for plane p, the p bits
// of 4 codes (one per byte) are gathered into 4 bits by one multiply
// ((v & 0x01010101) * 0x01020408 moves bit 8j to bit 24 + j). Sites past L
// get the '-' code, which matches everything, so padding never counts (the
// reference pads with '-' too, src/hamming_impl.cc:256-264).
constexpr int kPackThreads = 256;
constexpr int kPackCPG = 4;
template <int P>
__global__ void __launch_bounds__(kPackThreads)
    k_pack(const uint8_t *base, const uint64_t *rs, const uint64_t *rows, uint64_t n_rows,
           uint64_t L, uint64_t words, Table256 table, uint4 *g0, uint4 *g1) {
  __shared__ uint8_t tbl[256];
  __shared__ __align__(16) uint8_t stage[kPackThreads / 32][1024 + 16];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) tbl[i] = table.v[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  uint8_t *sw = stage[threadIdx.x >> 5];
  const uint64_t chunks = (words + 31) / 32;
  const uint64_t groups = (chunks + kPackCPG - 1) / kPackCPG;
  uint64_t wid = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  for (uint64_t job = wid; job < n_rows * groups; job += nwarps) {
    const uint64_t u = job / groups;
    const uint64_t q0 = (job - u * groups) * kPackCPG;
    const uint64_t r = rows ? rows[u] : u;
    const uint8_t *src = base + rs[r];
    for (uint64_t q = q0; q < q0 + kPackCPG && q < chunks; ++q) {
      const uint8_t *cs = src + q * 1024;
      const int64_t rem64 = (int64_t)L - (int64_t)(q * 1024);
      const int rem = rem64 <= 0 ? 0 : (rem64 >= 1024 ? 1024 : (int)rem64);
      uint8_t ch[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const int s = i * 32 + lane;
        ch[i] = s < rem ? cs[s] : (uint8_t)'-';
      }
#pragma unroll
      for (int i = 0; i < 32; ++i) sw[i * 32 + lane] = tbl[ch[i]];
      __syncwarp();
      const uint4 c0 = *reinterpret_cast<const uint4 *>(sw + lane * 32);
      const uint4 c1 = *reinterpret_cast<const uint4 *>(sw + lane * 32 + 16);
      __syncwarp();  // the next chunk overwrites the staging
      const uint32_t cw[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
      uint32_t x[6] = {0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
      for (int p = 0; p < P; ++p) {
        uint32_t acc = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
          acc |= ((((cw[k] >> p) & 0x01010101u) * 0x01020408u) >> 24 & 0xFu) << (4 * k);
        x[p] = acc;
      }
      const uint64_t w = q * 32 + lane;
      if (w < words) {
        g0[u * words + w] = make_uint4(x[0], x[1], x[2], x[3]);
        if (P > 4) g1[u * words + w] = make_uint4(x[4], x[5], 0u, 0u);
      }
    }
  }
}

__global__ void k_concat_starts(const uint64_t *a, uint64_t na, const uint64_t *b, uint64_t nb,
                                uint64_t b_off, uint64_t *out) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i < na) out[i] = a[i];
  else if (i < na + nb) out[i] = b[i - na] + b_off;
}

Records concat_records(hd_ctx *ctx, const Records &a, const Records &b, uint64_t b_off,
                       uint64_t bytes) {
  cudaStream_t st = ctx->stream;
  Records r;
  r.n = a.n + b.n;
  r.len0 = a.n ? a.len0 : b.len0;
  r.max_len = a.max_len > b.max_len ? a.max_len : b.max_len;
  r.all_equal = a.all_equal && b.all_equal && (!a.n || !b.n || a.len0 == b.len0);
  r.base = a.base;
  r.bytes = bytes;
  r.rec_start = DevBuf((r.n ? r.n : 1) * 8, st);
  r.rec_len = DevBuf((r.n ? r.n : 1) * 8, st);
  if (r.n) {
    k_concat_starts<<<grid_for(r.n, 256), 256, 0, st>>>(a.rec_start.as<uint64_t>(), a.n,
                                                        b.rec_start.as<uint64_t>(), b.n, b_off,
                                                        r.rec_start.as<uint64_t>());
    HD_LAUNCHED(ctx);
    if (a.n)
      HD_CUDA(cudaMemcpyAsync(r.rec_len.p, a.rec_len.p, a.n * 8, cudaMemcpyDeviceToDevice, st));
    if (b.n)
      HD_CUDA(cudaMemcpyAsync(r.rec_len.as<uint64_t>() + a.n, b.rec_len.p, b.n * 8,
                              cudaMemcpyDeviceToDevice, st));
  }
  return r;
}

void pack_rows(hd_ctx *ctx, const Records &rec, const uint64_t *d_rows, hd_alignment *aln,
               bool compared) {
  Table256 t;
  int table = aln->rule == HD_RULE_AND ? kCodesAnd
              : aln->rule == HD_RULE_SPARSE ? kCodesSparse : kCodesSparseX;
  code_table(table, t.v);
  const uint64_t bytes = aln->n_rows * aln->words * 16;
  aln->plane_buf[0] = DevBuf(bytes ? bytes : 16, ctx->stream);
  if (aln->groups > 1) aln->plane_buf[1] = DevBuf(bytes ? bytes : 16, ctx->stream);
  if (!aln->n_rows) return;
  if (aln->planes == 4) {
    // Compared rows come with their tensor-core operand, unless a look at some
    // of their sites says that site lists will do
    uint4 *g = aln->plane_buf[0].as<uint4>();
    const Words sel = compared ? sites_sample(ctx, aln) : Words{};
    if (sel.stride)
      pack_planes(ctx, rec, d_rows, aln->n_rows, aln->length, aln->words, g, nullptr,
                  sel.stride > 1 ? &sel : nullptr);
    const bool lists = sel.stride && sites_likely(ctx, aln, ctx->stream);
    if (lists && sel.stride == 1) return;
    if (compared && !lists && mma_wanted(ctx, aln) &&
        pack_operand(ctx, rec, d_rows, aln, 0, aln->n_rows, nullptr, ctx->stream))
      return;
    pack_planes(ctx, rec, d_rows, aln->n_rows, aln->length, aln->words, g, nullptr);
    return;
  }
  const uint64_t jobs = aln->n_rows * hd::ceil_div((aln->words + 31) / 32, (uint64_t)kPackCPG);
  unsigned grid = grid_for(jobs * 32, kPackThreads);
  uint4 *g0 = aln->plane_buf[0].as<uint4>(), *g1 = aln->plane_buf[1].as<uint4>();
  const uint64_t *rs = rec.rec_start.as<uint64_t>();
  if (aln->planes == 5)
    k_pack<5><<<grid, kPackThreads, 0, ctx->stream>>>(rec.base, rs, d_rows, aln->n_rows, aln->length,
                                             aln->words, t, g0, g1);
  else
    k_pack<6><<<grid, kPackThreads, 0, ctx->stream>>>(rec.base, rs, d_rows, aln->n_rows, aln->length,
                                             aln->words, t, g0, g1);
  HD_LAUNCHED(ctx);
}

// ----------------------------------------------------- reference distances
// Rule of src/hamming.cc:128-136: a site counts when the reference codes of
// the two bytes share no bit, or when the bytes differ and neither is '-'.
// 4-bit site codes of four bytes, as the reference's distance lookup
// classifies them: A 1, C 2, G 4, T 8, '-' 15, X 3 (with include_x), any
// other byte 0. The six symbols differ in their low three bits (X 0, A 1,
// C 3, T 4, '-' 5, G 7), which pick each byte's code from code_lo:code_hi
// and the symbol it must equal from a second table (both with __byte_perm).
__device__ __forceinline__ uint32_t site_codes(uint32_t w, uint32_t code_lo, uint32_t code_hi) {
  const uint32_t sel =
      (w & 0x7u) | ((w >> 4) & 0x70u) | ((w >> 8) & 0x700u) | ((w >> 12) & 0x7000u);
  const uint32_t z = w ^ __byte_perm(kSymLo, kSymHi, sel);
  const uint32_t eq = ~(((z & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | z) & 0x80808080u;  // 0x80: equal
  return __byte_perm(code_lo, code_hi, sel) & ((eq >> 7) * 0xFFu);
}
// Sites of four bytes that count, among those flagged (0x80) in `valid`: a
// pair counts if its codes share no bit, or if the bytes differ and neither
// is '-' (src/hamming.cc:104-141 through the distance lookup).
__device__ __forceinline__ uint32_t count_sites(uint32_t a, uint32_t ca, uint32_t b, uint32_t cb,
                                               uint32_t valid) {
  const uint32_t share = ((ca & cb) + 0x7F7F7F7Fu) & 0x80808080u;  // codes <= 15: no carry
  const uint32_t z = a ^ b;
  const uint32_t differ = (((z & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | z) & 0x80808080u;
  const uint32_t dash = (((ca >> 2) & (ca >> 3)) | ((cb >> 2) & (cb >> 3))) & 0x01010101u;
  return __popc((~share | (differ & ~(dash << 7))) & valid & 0x80808080u);
}

// Block (x, y) compares records 8x .. 8x + 7 (one per warp) over sites
// [y kRefSeg, (y + 1) kRefSeg) and adds each count to out[r], which starts at
// 0, so that short and long records spread evenly over the SMs. The block
// first copies that stretch of the reference, and its site codes, to shared
// memory. Lane l takes 16 consecutive sites per step: the reference's from
// shared memory, the record's from aligned 16-byte loads of its own and the
// next lane's, realigned with funnel shifts, and classifies and compares
// them four at a time, two steps per iteration with both steps' loads
// issued first. 20,000 records of 29,903 sites take 0.39 ms (one step per
// iteration: 0.41 ms; two shared-memory lookups per site: 0.53 ms).
constexpr uint64_t kRefSeg = 4096;
constexpr int kRefWarps = 8;
__global__ void __launch_bounds__(32 * kRefWarps)
    k_refdist(const uint8_t *base, uint64_t bytes, const uint64_t *rs, const uint64_t *rl,
              uint64_t R, uint64_t max_len, const uint8_t *ref, uint32_t code_lo,
              uint32_t code_hi, uint32_t *out) {
  __shared__ uint4 rsm[kRefSeg / 16], csm[kRefSeg / 16];
  const int lane = threadIdx.x & 31;
  const uint64_t r = (uint64_t)blockIdx.x * kRefWarps + (threadIdx.x >> 5);
  const uint64_t len = r < R ? rl[r] : 0;
  const uint64_t lo = reinterpret_cast<uint64_t>(base), hi = lo + bytes;
  const uint64_t S = (max_len + kRefSeg - 1) / kRefSeg;
  for (uint64_t y = blockIdx.y; y < S; y += gridDim.y) {  // block-uniform
    const uint64_t s_lo = y * kRefSeg;                     // < max_len
    // the reference is 16-byte aligned with 16 readable bytes past max_len
    const uint64_t avail = max_len - s_lo < kRefSeg ? max_len - s_lo : kRefSeg;
    const uint4 *rg = reinterpret_cast<const uint4 *>(ref + s_lo);
    __syncthreads();  // no warp still reads the previous stretch
    for (uint64_t i = threadIdx.x; i < (avail + 15) / 16; i += blockDim.x) {
      const uint4 v = rg[i];
      rsm[i] = v;
      csm[i] = make_uint4(site_codes(v.x, code_lo, code_hi), site_codes(v.y, code_lo, code_hi),
                          site_codes(v.z, code_lo, code_hi), site_codes(v.w, code_lo, code_hi));
    }
    __syncthreads();
    if (s_lo >= len) continue;  // warp-uniform (also r >= R)
    const uint64_t seg = len - s_lo < kRefSeg ? len - s_lo : kRefSeg;
    const uint64_t P = lo + rs[r] + s_lo;  // the record's site s_lo
    const uint64_t A = P & ~15ull, end = P + seg;
    const uint32_t d = (uint32_t)(P - A), dw = d >> 2, db = d & 3;
    uint32_t cnt = 0;
    // two 512-site steps per iteration: both steps' loads are issued first
    for (uint64_t o0 = 0; o0 < seg; o0 += 1024) {  // warp-uniform
      uint4 va[2], vx[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint64_t o = o0 + 512 * u + 16 * (uint64_t)lane;
        va[u] = A + o < end ? load16_in(A + o, lo, hi) : make_uint4(0u, 0u, 0u, 0u);
        // lane 31: the 16 bytes after its own, which no lane holds
        vx[u] = (lane == 31 && d && A + o + 16 < end) ? load16_in(A + o + 16, lo, hi)
                                                      : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint64_t o = o0 + 512 * u + 16 * (uint64_t)lane;
        uint4 vn;
        vn.x = __shfl_down_sync(0xffffffffu, va[u].x, 1);
        vn.y = __shfl_down_sync(0xffffffffu, va[u].y, 1);
        vn.z = __shfl_down_sync(0xffffffffu, va[u].z, 1);
        vn.w = __shfl_down_sync(0xffffffffu, va[u].w, 1);
        if (lane == 31) vn = vx[u];
        if (o >= seg) continue;
        const uint4 vr = rsm[o >> 4], vc = csm[o >> 4];
        const uint32_t bw[8] = {va[u].x, va[u].y, va[u].z, va[u].w, vn.x, vn.y, vn.z, vn.w};
        const uint32_t rw[4] = {vr.x, vr.y, vr.z, vr.w}, cw[4] = {vc.x, vc.y, vc.z, vc.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t blo = bw[j], bhi = bw[j + 1];
#pragma unroll
          for (int t = 1; t < 4; ++t)
            if (dw == (uint32_t)t) {
              blo = bw[j + t];
              bhi = bw[j + t + 1];
            }
          const uint32_t aw = __funnelshift_r(blo, bhi, 8 * db);  // record sites o + 4j ..
          const uint64_t rem = seg - o;                           // >= 1
          const uint32_t valid = rem >= (uint64_t)(4 * j + 4) ? 0x80808080u
                                 : rem <= (uint64_t)(4 * j) ? 0u
                                   : 0x80808080u & ((1u << (8 * (uint32_t)(rem - 4 * j))) - 1u);
          cnt += count_sites(aw, site_codes(aw, code_lo, code_hi), rw[j], cw[j], valid);
        }
      }
    }
    cnt = warp_sum(cnt);
    if (lane == 0 && cnt) atomicAdd(&out[r], cnt);
  }
}

void reference_distances_device(hd_ctx *ctx, const Records &rec, const uint8_t *d_ref,
                                int include_x, uint32_t *d_out) {
  if (!rec.n) return;
  // codes by the low three bits of the symbol: X, A, -, C / T, -, -, G
  const uint32_t code_lo = (include_x ? 3u : 0u) | (1u << 8) | (2u << 24);
  const uint32_t code_hi = 8u | (15u << 8) | (4u << 24);
  HD_CUDA(cudaMemsetAsync(d_out, 0, rec.n * sizeof(uint32_t), ctx->stream));
  if (!rec.max_len) return;
  const uint64_t S = ceil_div(rec.max_len, kRefSeg), X = ceil_div(rec.n, (uint64_t)kRefWarps);
  if (X > 0x7fffffffull) fail(HD_ERR_ARG, "too many records");
  // stretches past 65,535 are taken by the blocks' loop
  k_refdist<<<dim3((unsigned)X, (unsigned)std::min<uint64_t>(S, 65535)), 32 * kRefWarps, 0,
              ctx->stream>>>(rec.base, rec.bytes, rec.rec_start.as<uint64_t>(),
                             rec.rec_len.as<uint64_t>(), rec.n, rec.max_len, d_ref, code_lo,
                             code_hi, d_out);
  HD_LAUNCHED(ctx);
}

// Query row (packed with the alignment's AND codes) against every row.
__global__ void k_query(const uint4 *g0, uint64_t words, uint64_t n_rows, const uint4 *q,
                        uint32_t *out) {
  const int lane = threadIdx.x & 31;
  uint64_t wid = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  for (uint64_t u = wid; u < n_rows; u += nwarps) {
    const uint4 *row = g0 + u * words;
    uint32_t cnt = 0;
    for (uint64_t w = lane; w < words; w += 32) {
      uint4 a = row[w], b = q[w];
      cnt += __popc(~((a.x & b.x) | (a.y & b.y) | (a.z & b.z) | (a.w & b.w)));
    }
    cnt = warp_sum(cnt);
    if (lane == 0) out[u] = cnt;
  }
}

void query_distances_async(hd_ctx *ctx, const hd_alignment *aln, const uint8_t *d_query,
                           uint32_t *d_out_rows, DevBuf &q_planes) {
  // pack the query with the AND codes (one row: 3 us), then one warp per row
  q_planes = DevBuf(aln->words * 16, ctx->stream);
  Records q;  // one record, at the start
  q.base = d_query;
  q.bytes = aln->length;
  pack_planes(ctx, q, nullptr, 1, aln->length, aln->words, q_planes.as<uint4>(), nullptr);
  k_query<<<grid_for(aln->n_rows * 32, 256), 256, 0, ctx->stream>>>(
      static_cast<const uint4 *>(aln->planes_ptr(0)), aln->words, aln->n_rows,
      q_planes.as<uint4>(), d_out_rows);
  HD_LAUNCHED(ctx);
}

// out[r] = the distance of record r's row
__global__ void k_gather_rows(const uint32_t *row_dist, const uint64_t *row_of, uint64_t n,
                              uint32_t *out) {
  const uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (r < n) out[r] = row_dist[row_of ? row_of[r] : r];
}

void query_rows_to_records(hd_ctx *ctx, const hd_alignment *aln, const uint8_t *d_query,
                           uint32_t *d_rows, const uint64_t *row_of, uint64_t n, uint32_t *d_out) {
  DevBuf q;  // freed after the kernels in stream order
  query_distances_async(ctx, aln, d_query, d_rows, q);
  k_gather_rows<<<grid_for(n, 256), 256, 0, ctx->stream>>>(d_rows, row_of, n, d_out);
  HD_LAUNCHED(ctx);
}

void alignment_query_distances(hd_ctx *ctx, const hd_alignment *aln, const uint8_t *d_query,
                               uint32_t *d_out_rows) {
  DevBuf q;
  query_distances_async(ctx, aln, d_query, d_out_rows, q);
  HD_CUDA(cudaStreamSynchronize(ctx->stream));
}

}  // namespace hd
