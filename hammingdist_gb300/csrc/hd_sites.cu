// Distances of alignments of similar rows from lists of the sites where a row
// differs from a reference.
//
// Replaces the dense distance loops (ssciwr/hammingdist 1.4.0,
// src/distance_cuda.cu:204-214, include/hamming/hamming_impl.hh:120-175) where
// that does less work, with the same results: rows of one species differ in a
// few sites per thousand, so that nearly all site pairs that a dense
// comparison takes are equal to the reference in both rows.
//
// Per site, r is the commonest code of some rows (any choice gives the same
// distances). Two rows' codes a, b mismatch at a site where a & b == 0. With
//   k = [r & r == 0] (1 where r is the code 0 that matches nothing),
//   m(a) = [a & r == 0] - k,
//   c(a, b) = k + m(a) + m(b) - [a & b == 0],
// m(r) = 0 and c(a, r) = c(r, b) = 0, so a pair's distance is
//   sum of k + sum of m(a) over the row's sites + the same for b
//   - sum of c(a, b) over the sites where BOTH rows differ from r.
// c is 0, 1 or 2. Where r is not 0, a '-' has m = 0 and c = 0 with every code
// but those that r and not '-' mismatches (m = 1, the code not 0), where it is
// 1: '-' entries, of which an alignment's ends have many, are kept in lists of
// their own and only meet those. Two entries of code 0 ('N', in runs) have
// c = 1: a run's first entry (in its 32-site word) meets another run's entry
// for the sites that both still have, and later entries of runs do not meet
// each other.
//
// The lists (SiteLists) are by tiles of 224 rows and ranges of 1,024 sites: the
// entries of a (tile, range) in site order, and where each site's begin. A
// block of k_site_pairs takes a tile pair: its 224 x 224 sums of c are 16-bit
// counters in shared memory, to which it adds c for the pairs of entries that
// the two tiles' lists have at one site.
#include <algorithm>
#include <cstdlib>

#include "hd_internal.cuh"

namespace hd {
namespace {

constexpr uint32_t kT = 224;                 // rows of a tile (two blocks' counters fit an SM)
constexpr uint32_t kPitch = kT / 2;          // counter words per row
constexpr uint32_t kRangeWords = 32;
constexpr uint32_t kRange = 32 * kRangeWords;
constexpr uint32_t kMaxRanges = 64;          // L <= 65,536
constexpr uint32_t kOffPitch = kRange + 8;   // 16-bit starts, and an end
// per (tile, range): where each site's s entries start, its later entries of
// runs among them, and its '-' entries
constexpr uint32_t kOffLater = kOffPitch, kOffDash = 2 * kOffPitch, kOffSlot = 3 * kOffPitch;
constexpr uint32_t kRefRows = 64;            // rows that the reference is taken from
constexpr int kPairThreads = 768;
constexpr uint32_t kPending = 64;            // sites a warp gathers before it takes 32 of them
constexpr uint32_t kStepSites = 128;         // of one range, a warp's step: four to a lane
constexpr uint32_t kMaxSteps = kMaxRanges * (kRange / kStepSites);
constexpr uint32_t kHeavy = 4096;            // meetings of 32 gathered sites that the block's warps share
constexpr uint32_t kPairSmem = kT * kPitch * 4 + kPairThreads / 32 * kPending * 8;
// an entry: site in its range (10 bits), row in its tile (8), code (6), 1 bit:
// a '-' counts against it, 1 bit: the site's r is 0, and for code 0 where r is
// not 0 the sites left of its run (6 bits, else 0)
__device__ __forceinline__ uint32_t e_site(uint32_t e) { return e & 1023u; }
__device__ __forceinline__ uint32_t e_row(uint32_t e) { return (e >> 10) & 255u; }
__device__ __forceinline__ uint32_t e_code(uint32_t e) { return (e >> 18) & 63u; }
__device__ __forceinline__ uint32_t e_run(uint32_t e) { return e >> 26; }
constexpr uint32_t kMeetsDash = 1u << 24, kRefZero = 1u << 25;

struct Planes {
  const uint4 *g0, *g1;
  uint32_t planes;
  uint64_t pitch;  // words per row
  __device__ void load(uint64_t row, uint32_t w, uint4 &a, uint2 &b) const {
    a = __ldg(g0 + row * pitch + w);
    b = make_uint2(0u, 0u);
    if (planes > 4) b = __ldg(reinterpret_cast<const uint2 *>(g1 + row * pitch + w));
  }
};
__device__ __forceinline__ uint32_t valid_mask(uint64_t L, uint32_t w) {
  const uint64_t s0 = 32ull * w;
  return s0 >= L ? 0u : L - s0 >= 32 ? 0xFFFFFFFFu : (1u << (L - s0)) - 1u;
}
// One word of a row against the reference's: the sites with an entry (s), those
// of them that a '-' counts against (x), those of code 0 where r is not 0 (z)
// and the '-' entries (d)
struct Diff {
  uint32_t s, x, z, d;
  __device__ uint32_t later() const { return z & (z << 1); }  // of runs, not their first
};
__device__ __forceinline__ Diff diff_of(const uint4 &a, const uint2 &b, const uint4 &ra,
                                        const uint2 &rb, uint32_t planes, uint32_t valid) {
  uint32_t any = a.x | a.y | a.z | a.w, all = a.x & a.y & a.z & a.w;
  uint32_t ref = ra.x | ra.y | ra.z | ra.w;
  uint32_t df = (a.x ^ ra.x) | (a.y ^ ra.y) | (a.z ^ ra.z) | (a.w ^ ra.w);
  if (planes > 4) {
    any |= b.x | b.y;
    all &= planes > 5 ? b.x & b.y : b.x;
    ref |= rb.x | rb.y;
    df |= (b.x ^ rb.x) | (b.y ^ rb.y);
  }
  df &= valid;
  Diff o;
  o.d = df & all & ref;
  o.s = df & ~o.d;
  o.x = o.s & any & ref;
  o.z = o.s & ~any & ref;
  return o;
}

// Rows of a word's sites, `each` a warp from the q0-th of them on, counted by
// code: 8 bits a slot (bits 0-5, none, '-')
template <uint32_t kEach, class RowOf>
__device__ __forceinline__ unsigned long long count_codes(const Planes &p, uint64_t n, uint32_t w,
                                                          uint32_t lane, RowOf &&row_of) {
  unsigned long long cnt = 0;
#pragma unroll 1
  for (uint32_t h = 0; h < kEach; h += 8) {
    uint4 a[8];
    uint2 b[8];
    uint64_t row[8];
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q) {
      row[q] = row_of(h + q);
      a[q] = make_uint4(0u, 0u, 0u, 0u);
      b[q] = make_uint2(0u, 0u);
      if (row[q] < n) p.load(row[q], w, a[q], b[q]);
    }
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q) {
      const uint32_t code = ((a[q].x >> lane) & 1u) | ((a[q].y >> lane) & 1u) << 1 |
                            ((a[q].z >> lane) & 1u) << 2 | ((a[q].w >> lane) & 1u) << 3 |
                            ((b[q].x >> lane) & 1u) << 4 | ((b[q].y >> lane) & 1u) << 5;
      const uint32_t slot = code == 0 ? 6u : code & (code - 1u) ? 7u : (uint32_t)__ffs(code) - 1u;
      if (row[q] < n) cnt += 1ull << (8u * slot);
    }
  }
  return cnt;
}

// The reference: four warps take a word, 16 rows each, a lane a site: the
// commonest code with one bit (r has at most one) of 64 rows. Where r is 0 a '-'
// is an s entry, so r is 0 only where there are more rows of code 0 than of that
// code and '-' together. Near an alignment's ends the 64 rows can all be '-' at a
// site, or one of them 'N': words with sites that no row gives a code with a bit
// look at 96 rows more. (r taken to be 0 at four sites where all rows but a few
// are '-': 11.3 ms for 14,000 rows instead of 0.3; a code that is not the rows' at
// 18 sites, where 2-12% have one: 0.7 ms.)
__global__ void __launch_bounds__(256)
    k_site_ref(Planes p, uint64_t n, Words sel, uint4 *r0, uint2 *r1) {
  __shared__ unsigned long long part[8][32];
  __shared__ uint32_t more[2];  // the sites of each word to look at again
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, quarter = warp & 3u;
  const uint32_t k = blockIdx.x * 2 + (warp >> 2), w = k < sel.count ? sel.at(k) : sel.words;
  const bool here = w < sel.words;  // warp-uniform
  part[warp][lane] = !here ? 0ull : count_codes<kRefRows / 4>(p, n, w, lane, [&](uint32_t q) {
    q += quarter * (kRefRows / 4);
    return n < kRefRows ? (uint64_t)q : n * q / kRefRows;
  });
  __syncthreads();
  auto sum = [&] {
    return part[warp][lane] + part[warp + 1][lane] + part[warp + 2][lane] + part[warp + 3][lane];
  };
  auto slot = [](unsigned long long c, uint32_t s) { return (uint32_t)(c >> (8u * s)) & 255u; };
  uint32_t best = 0, most = 0;
  auto choose = [&](unsigned long long c) {
    most = slot(c, 0);
#pragma unroll
    for (uint32_t s = 1; s < 6; ++s)
      if (slot(c, s) > most) {
        most = slot(c, s);
        best = s;
      }
    if (slot(c, 6) > most + slot(c, 7)) best = 6;
  };
  uint32_t again = 0;
  if (quarter == 0) {
    choose(sum());
    again = __ballot_sync(0xffffffffu, here && n > kRefRows && most == 0 && best != 6);
    if (lane == 0) more[warp >> 2] = again;
  }
  __syncthreads();
  if (more[warp >> 2]) {
    constexpr uint32_t kMore = 96;
    part[warp][lane] = count_codes<kMore / 4>(p, n, w, lane, [&](uint32_t q) {
      q += quarter * (kMore / 4);
      return n < kRefRows + kMore ? (uint64_t)kRefRows + q : n * (2 * q + 1) / (2 * kMore);
    });
  }
  __syncthreads();
  if (quarter || !here) return;
  if (again >> lane & 1u) choose(sum());
  uint32_t bits[6];
#pragma unroll
  for (uint32_t s = 0; s < 6; ++s) bits[s] = __ballot_sync(0xffffffffu, best == s);
  if (lane == 0) {
    r0[w] = make_uint4(bits[0], bits[1], bits[2], bits[3]);
    r1[w] = make_uint2(bits[4], bits[5]);
  }
}

// Entries per site of the selected words: counts[4 site] s, x, d and the later
// ones of runs. Block (x, y) takes four words of a share of the rows.
__global__ void __launch_bounds__(256)
    k_site_count(Planes p, uint64_t n, uint64_t L, Words sel, const uint4 *r0, const uint2 *r1,
                 uint32_t *counts) {
  __shared__ uint32_t cnt[4][128];
  for (uint32_t i = threadIdx.x; i < 512; i += blockDim.x) (&cnt[0][0])[i] = 0;
  __syncthreads();
  const uint32_t k = threadIdx.x & 3u, w = sel.at(blockIdx.x * 4 + k);
  if (w < sel.words) {
    const uint32_t valid = valid_mask(L, w);
    const uint4 ra = r0[w];
    const uint2 rb = r1[w];
    for (uint64_t r = blockIdx.y * 64ull + (threadIdx.x >> 2); r < n; r += gridDim.y * 64ull) {
      uint4 a;
      uint2 b;
      p.load(r, w, a, b);
      const Diff f = diff_of(a, b, ra, rb, p.planes, valid);
      for (uint32_t m = f.s; m; m &= m - 1) atomicAdd(&cnt[0][32 * k + __ffs(m) - 1], 1u);
      for (uint32_t m = f.x; m; m &= m - 1) atomicAdd(&cnt[1][32 * k + __ffs(m) - 1], 1u);
      for (uint32_t m = f.d; m; m &= m - 1) atomicAdd(&cnt[2][32 * k + __ffs(m) - 1], 1u);
      for (uint32_t m = f.later(); m; m &= m - 1) atomicAdd(&cnt[3][32 * k + __ffs(m) - 1], 1u);
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < 512; i += blockDim.x) {
    const uint32_t v = (&cnt[0][0])[i];
    if (v) atomicAdd(&counts[(blockIdx.x * 128 + (i & 127u)) * 4 + (i >> 7)], v);
  }
}
// One block: the entries (s, x, d), the pairs of s entries of one site that
// meet, and the pairs of an x and a d entry: of the sites before `edge` in
// out[0 .. 5), of the others in out[5 .. 10)
__global__ void __launch_bounds__(1024)
    k_site_cost(const uint32_t *counts, uint32_t edge, uint32_t sites, unsigned long long *out) {
  __shared__ unsigned long long sum[10];
  if (threadIdx.x < 10) sum[threadIdx.x] = 0;
  __syncthreads();
  for (int part = 0; part < 2; ++part) {
    unsigned long long v[5] = {0, 0, 0, 0, 0};
    const uint32_t end = part ? sites : edge;
    for (uint32_t i = (part ? edge : 0u) + threadIdx.x; i < end; i += blockDim.x) {
      const unsigned long long s = counts[4 * i], x = counts[4 * i + 1], d = counts[4 * i + 2];
      const unsigned long long l = counts[4 * i + 3];
      v[0] += s;
      v[1] += x;
      v[2] += d;
      v[3] += (s * s - l * l) / 2;
      v[4] += x * d;
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      v[k] = warp_sum(v[k]);
      if ((threadIdx.x & 31) == 0 && v[k]) atomicAdd(&sum[5 * part + k], v[k]);
    }
  }
  __syncthreads();
  if (threadIdx.x < 10) out[threadIdx.x] = sum[threadIdx.x];
}

// What building the lists leaves (device)
struct BuildSums {
  unsigned long long s, d;     // entries
  unsigned long long pairs;    // of s entries that meet
  unsigned long long dashes;   // of an s and a '-' entry of one site
  uint32_t full;               // some list did not fit
  uint32_t zero;               // sites where r is 0
  uint32_t max_weight;
  uint32_t peak;               // most meetings of a tile with itself, of its sites with many
};

// The lists of one (range, tile): a warp takes four rows at a time, a lane a
// word. The block counts the entries of its sites, places them and, reading
// the rows again (from the caches), files them. weight: sum of m per row.
// first_rows: block row 0 is the alignment's first tile (not that of a later
// launch), which counts the sites where r is 0.
// 14,000 rows of 29,903 sites: 150 us, bound by the instructions and the chains
// of ballots, shuffles and atomics of a row's entries (a lane a word's entries
// instead, one after another: 217 us; a row at a time: 173).
template <bool kWide>  // more than four planes
__global__ void __launch_bounds__(256, 4)
    k_site_lists(Planes p, uint64_t n, uint64_t L, uint32_t words, const uint4 *r0, const uint2 *r1,
                 uint32_t ranges, uint64_t cap_s, uint64_t cap_d, uint4 *base, uint16_t *off,
                 uint32_t *es, uint8_t *ed, uint32_t *weight, bool first_rows, BuildSums *sums) {
  __shared__ uint32_t cnt[3][kRange];  // first entries, later ones of runs, '-'
  __shared__ uint64_t tmp[33];
  __shared__ unsigned long long at_s, at_d;
  __shared__ uint32_t fits;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t tile = blockIdx.y, range = blockIdx.x, w = range * kRangeWords + lane;
  const uint64_t row0 = (uint64_t)tile * kT;
  const uint32_t rows = n - row0 < kT ? (uint32_t)(n - row0) : kT;
  for (uint32_t i = threadIdx.x; i < kRange; i += blockDim.x) cnt[0][i] = cnt[1][i] = cnt[2][i] = 0;
  const uint32_t valid = w < words ? valid_mask(L, w) : 0u;
  uint4 ra = make_uint4(0u, 0u, 0u, 0u);
  uint2 rb = make_uint2(0u, 0u);
  if (valid) {
    ra = r0[w];
    rb = r1[w];
  }
  const uint32_t zero = valid & ~(ra.x | ra.y | ra.z | ra.w | rb.x | rb.y);
  __syncthreads();
  constexpr uint32_t kBatch = 4;
  const uint32_t planes = kWide ? p.planes : 4u;
  // rows i, i + 8, ... of a batch: this lane's words, and for each row f(row,
  // words, diff) by the whole warp; a lane past the row's words has none
  auto each_row = [&](auto &&f) {
    for (uint32_t i0 = warp; i0 < rows; i0 += 8 * kBatch) {
      uint4 a[kBatch];
      uint2 b[kBatch];
#pragma unroll
      for (uint32_t k = 0; k < kBatch; ++k) {
        a[k] = ra;  // no entries
        b[k] = rb;
        if (valid && i0 + 8 * k < rows) {
          a[k] = __ldg(p.g0 + (row0 + i0 + 8 * k) * p.pitch + w);
          if (kWide) b[k] = __ldg(reinterpret_cast<const uint2 *>(p.g1 + (row0 + i0 + 8 * k) * p.pitch + w));
        }
      }
#pragma unroll
      for (uint32_t k = 0; k < kBatch; ++k)
        if (i0 + 8 * k < rows) f(i0 + 8 * k, a[k], b[k], diff_of(a[k], b[k], ra, rb, planes, valid));
    }
  };
  // a word with entries at a time, a lane a site: a run of 'N' or '-' costs no
  // more than one entry
  each_row([&](uint32_t i, const uint4 &, const uint2 &, const Diff &f) {
    for (uint32_t on = __ballot_sync(0xffffffffu, f.s | f.d); on; on &= on - 1) {
      const int src = __ffs(on) - 1;
      const uint32_t ms = __shfl_sync(0xffffffffu, f.s, src), md = __shfl_sync(0xffffffffu, f.d, src);
      const uint32_t ml = __shfl_sync(0xffffffffu, f.later(), src);
      const uint32_t kind = (ml >> lane & 1u) | (md >> lane & 1u) << 1;
      if ((ms | md) >> lane & 1u) atomicAdd(&cnt[kind][32 * src + lane], 1u);
    }
    const uint32_t m = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(f.s & ~zero));
    if (lane == 0 && m) atomicAdd(&weight[row0 + i], m);
  });
  if (first_rows && tile == 0 && warp == 0) {
    const uint32_t z = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(zero));
    if (lane == 0 && z) atomicAdd(&sums->zero, z);
  }
  __syncthreads();
  uint32_t c[3][4];
  uint64_t v = 0, total;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
#pragma unroll
    for (int j = 0; j < 3; ++j) c[j][k] = cnt[j][4 * threadIdx.x + k];
    v += (uint64_t)(c[0][k] + c[1][k]) | (uint64_t)c[2][k] << 32;
  }
  uint64_t ex = block_excl_scan<uint64_t>(v, tmp, total);
  const uint32_t ns = (uint32_t)total, nd = (uint32_t)(total >> 32);
  if (threadIdx.x == 0) {
    at_s = atomicAdd(&sums->s, (unsigned long long)ns);
    at_d = atomicAdd(&sums->d, (unsigned long long)nd);
    fits = ns <= 65535u && nd <= 65535u && at_s + ns <= cap_s && at_d + nd <= cap_d ? 1u : 0u;
    if (!fits) atomicOr(&sums->full, 1u);
  }
  __syncthreads();
  const uint64_t slot = (uint64_t)tile * ranges + range;
  uint16_t *o = off + slot * kOffSlot;
  if (threadIdx.x == 0)
    base[slot] = fits ? make_uint4((uint32_t)at_s, ns, (uint32_t)at_d, nd) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t s = 4 * threadIdx.x + k;
    const uint32_t first = (uint32_t)ex, later = first + c[0][k], dash = (uint32_t)(ex >> 32);
    cnt[0][s] = first;
    cnt[1][s] = later;
    cnt[2][s] = dash;
    o[s] = (uint16_t)(fits ? first : 0u);
    o[kOffLater + s] = (uint16_t)(fits ? later : 0u);
    o[kOffDash + s] = (uint16_t)(fits ? dash : 0u);
    ex += (uint64_t)(c[0][k] + c[1][k]) | (uint64_t)c[2][k] << 32;
  }
  if (threadIdx.x == 0) {
    o[kRange] = (uint16_t)(fits ? ns : 0u);
    o[kOffDash + kRange] = (uint16_t)(fits ? nd : 0u);
  }
  __syncthreads();
  if (!fits) return;
  each_row([&](uint32_t i, const uint4 &a, const uint2 &b, const Diff &f) {
    for (uint32_t on = __ballot_sync(0xffffffffu, f.s | f.d); on; on &= on - 1) {
      const int src = __ffs(on) - 1;
      const uint32_t ms = __shfl_sync(0xffffffffu, f.s, src), md = __shfl_sync(0xffffffffu, f.d, src);
      const uint32_t mn = __shfl_sync(0xffffffffu, f.z, src), ml = mn & (mn << 1);
      uint32_t *at = &cnt[(ml >> lane & 1u) | (md >> lane & 1u) << 1][32 * src + lane];
      if (ms) {  // warp-uniform
        const uint32_t mx = __shfl_sync(0xffffffffu, f.x, src), mz = __shfl_sync(0xffffffffu, zero, src);
        uint32_t code = ((__shfl_sync(0xffffffffu, a.x, src) >> lane) & 1u) |
                        ((__shfl_sync(0xffffffffu, a.y, src) >> lane) & 1u) << 1 |
                        ((__shfl_sync(0xffffffffu, a.z, src) >> lane) & 1u) << 2 |
                        ((__shfl_sync(0xffffffffu, a.w, src) >> lane) & 1u) << 3;
        if (kWide)
          code |= ((__shfl_sync(0xffffffffu, b.x, src) >> lane) & 1u) << 4 |
                  ((__shfl_sync(0xffffffffu, b.y, src) >> lane) & 1u) << 5;
        if (ms >> lane & 1u)
        {
          // the run's sites from here on: the ones of mn up to the next 0
          const uint32_t up = ~(mn >> lane);  // bit 0 is 0 for an entry of a run
          const uint32_t run = mn >> lane & 1u ? (up ? (uint32_t)__ffs(up) - 1u : 32u) : 0u;
          es[at_s + atomicAdd(at, 1u)] = (32 * src + lane) | i << 10 | code << 18 |
                                         (mx >> lane & 1u ? kMeetsDash : 0u) |
                                         (mz >> lane & 1u ? kRefZero : 0u) | run << 26;
        }
      }
      if (md >> lane & 1u) ed[at_d + atomicAdd(at, 1u)] = (uint8_t)i;
    }
  });
}

// The pairs of s entries that meet over all tiles, of s and '-' entries, the
// largest weight, and the tile whose own entries meet most (no pair of tiles has
// more), by the 32 neighbouring sites that have many: tile_sum, one a tile, starts
// at 0. A lane takes a site, the block's warps a share of the tiles each.
__global__ void __launch_bounds__(256)
    k_site_check(const uint16_t *off, uint32_t tiles, uint32_t ranges, const uint32_t *weight,
                 uint64_t n, uint32_t *tile_sum, BuildSums *sums) {
  __shared__ uint32_t part[3][8][32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t range = blockIdx.x / (kRange / 32), s = (blockIdx.x % (kRange / 32)) * 32 + lane;
  uint32_t k = 0, l = 0, d = 0;
  for (uint32_t t = warp; t < tiles; t += 8) {
    const uint16_t *o = off + ((uint64_t)t * ranges + range) * kOffSlot + s;
    const uint32_t kt = (uint32_t)o[1] - o[0], lt = (uint32_t)o[1] - o[kOffLater];
    const uint32_t own = __reduce_add_sync(0xffffffffu, kt * kt - lt * lt);
    if (own >= 1024 && lane == 0) atomicMax(&sums->peak, atomicAdd(&tile_sum[t], own) + own);
    k += kt;
    l += lt;
    d += (uint32_t)o[kOffDash + 1] - o[kOffDash];
  }
  part[0][warp][lane] = k;
  part[1][warp][lane] = l;
  part[2][warp][lane] = d;
  __syncthreads();
  if (warp == 0) {
    unsigned long long v[3] = {0, 0, 0};
#pragma unroll
    for (int w = 0; w < 8; ++w)
#pragma unroll
      for (int j = 0; j < 3; ++j) v[j] += part[j][w][lane];
    const unsigned long long pairs = warp_sum((v[0] * v[0] - v[1] * v[1]) / 2);
    const unsigned long long dashes = warp_sum(v[0] * v[2]);
    if (lane == 0 && pairs) atomicAdd(&sums->pairs, pairs);
    if (lane == 0 && dashes) atomicAdd(&sums->dashes, dashes);
  }
  uint32_t m = 0;
  for (uint64_t r = blockIdx.x * 256ull + threadIdx.x; r < n; r += gridDim.x * 256ull)
    m = max(m, weight[r]);
  m = __reduce_max_sync(0xffffffffu, m);
  if (lane == 0 && m) atomicMax(&sums->max_weight, m);
}

// The tile pair's distances from its counters: a warp a row, a lane a column of
// every 32. kDiag: the pair of a tile with itself, whose rows end at themselves.
template <class T, bool kDiag>
__device__ __forceinline__ void store_tile(const SiteJob &J, const uint32_t *acc, uint32_t ti,
                                           uint32_t tj) {
  constexpr uint32_t kWarps = kPairThreads / 32;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t half = (lane & 1u) ? 0x4432u : 0x4410u;  // its 16 bits of a counter word
  uint32_t wj[kT / 32];
#pragma unroll
  for (uint32_t k = 0; k < kT / 32; ++k) {
    const uint64_t j = (uint64_t)tj * kT + 32 * k + lane;
    wj[k] = j < J.n ? __ldg(J.weight + j) + J.zero : 0u;
  }
  const uint64_t r0 = (uint64_t)ti * kT;
  for (uint32_t i = warp; i < kT; i += kWarps) {
    const uint64_t r = r0 + i;
    if (r < J.row_lo || r >= J.row_hi) continue;
    const uint32_t wi = __ldg(J.weight + r);
    T *out = static_cast<T *>(J.out) + (r * (r - 1) / 2 + (uint64_t)tj * kT - J.out_base) + lane;
    const uint32_t *row = acc + i * kPitch + (lane >> 1);
#pragma unroll
    for (uint32_t k = 0; k < kT / 32; ++k) {
      const uint32_t d = wi + wj[k] - __byte_perm(row[16 * k], 0u, half);
      if (!kDiag || 32 * k + lane < i) out[32 * k] = (T)min(d, J.max_dist);
    }
  }
}
template <class T>
__device__ __forceinline__ void store_rows(const SiteJob &J, const uint32_t *acc, uint32_t ti,
                                           uint32_t tj) {
  if (ti == tj) store_tile<T, true>(J, acc, ti, tj);
  else store_tile<T, false>(J, acc, ti, tj);
}

// 1 to every '-' entry's counter: column j (row i) of the list's rows, for up
// to 224 of them, all loaded before the first is used
template <bool kRow>
__device__ __forceinline__ void meet_dashes(uint32_t *acc, const uint8_t *list, uint32_t n,
                                            uint32_t fixed, uint32_t lane) {
  uint32_t v[kT / 32];
#pragma unroll
  for (uint32_t k = 0; k < kT / 32; ++k) v[k] = 32 * k + lane < n ? __ldg(list + 32 * k + lane) : 255u;
#pragma unroll
  for (uint32_t k = 0; k < kT / 32; ++k) {
    if (32 * k >= n) break;  // warp-uniform
    const uint32_t i = kRow ? fixed : v[k], j = kRow ? v[k] : fixed;
    if (v[k] != 255u) atomicAdd(&acc[i * kPitch + (j >> 1)], 1u << (16u * (j & 1u)));
  }
}

// The entries of n <= 32 sites of one range that meet, one a lane at a time:
// per site, the first entries of the row tile's list with all of the column
// tile's, and its later ones with the column tile's first ones. kShare: one warp's
// part of them, every 24th 32 meetings; else false, and nothing is done, if there
// are more than kHeavy.
template <bool kShare>
__device__ __forceinline__ bool meet_sites(uint32_t *acc, const uint2 *sites, uint32_t n,
                                           const uint32_t *li, const uint32_t *lj, uint32_t lane) {
  const uint2 me = lane < n ? sites[lane] : make_uint2(0u, 0u);
  const uint32_t fa = me.y & 255u, la = (me.y >> 8) & 255u, fb = (me.y >> 16) & 255u, lb = me.y >> 24;
  const uint32_t mine = fa * (fb + lb) + la * fb;
  const uint32_t inc = warp_incl_scan(mine), total = __shfl_sync(0xffffffffu, inc, 31);
  if (!kShare && total > kHeavy) return false;
  for (uint32_t m0 = kShare ? threadIdx.x & ~31u : 0u; m0 < total; m0 += kShare ? kPairThreads : 32) {
    const uint32_t m = m0 + lane;
    uint32_t src = 0;  // the lane whose site the m-th meeting is of
#pragma unroll
    for (uint32_t h = 16; h; h >>= 1)
      if (__shfl_sync(0xffffffffu, inc, src + h - 1) <= m) src += h;
    const uint32_t at = __shfl_sync(0xffffffffu, me.x, src), c = __shfl_sync(0xffffffffu, me.y, src);
    uint32_t rest = m - __shfl_sync(0xffffffffu, inc - mine, src);
    if (m < total) {
      const uint32_t sa = c & 255u, sb = (c >> 16) & 255u, all = sb + (c >> 24);
      // the quotients are of numbers below 2^16: a half more than the dividend
      // keeps them off whole numbers by far more than the division's error
      uint32_t u = 0, per = all;
      if (rest >= sa * all) {
        rest -= sa * all;
        u = sa;
        per = sb;
      }
      const uint32_t q = (uint32_t)__fdividef((float)rest + 0.5f, (float)per);
      const uint32_t e = __ldg(li + (at & 0xFFFFu) + u + q), f = __ldg(lj + (at >> 16) + rest - q * per);
      const uint32_t run = min(e_run(e), e_run(f));  // both of code 0, r not 0
      const uint32_t one = ((e & kRefZero) ? 1u : 2u) - ((e_code(e) & e_code(f)) ? 0u : 1u);
      const uint32_t w = run ? run : one, j = e_row(f);
      if (w) atomicAdd(&acc[e_row(e) * kPitch + (j >> 1)], w << (16u * (j & 1u)));
    }
  }
  return true;
}

// A step's sites, four to a lane: those with entries in both tiles are gathered in
// `pending` and taken in batches of 32, take(bit, sites, n) for the batch (bit q: of
// those a lane's q-th sites complete, 4: the rest).
template <class Take>
__device__ __forceinline__ void gather_sites(const uint16_t *a, const uint16_t *b, uint2 *pending,
                                             uint32_t lane, Take &&take) {
  uint32_t count = 0;
  const uint2 af = __ldg(reinterpret_cast<const uint2 *>(a));
  const uint2 al = __ldg(reinterpret_cast<const uint2 *>(a + kOffLater));
  const uint2 bf = __ldg(reinterpret_cast<const uint2 *>(b));
  const uint2 bl = __ldg(reinterpret_cast<const uint2 *>(b + kOffLater));
  uint32_t an = __shfl_down_sync(0xffffffffu, af.x, 1) & 0xFFFFu;
  uint32_t bn = __shfl_down_sync(0xffffffffu, bf.x, 1) & 0xFFFFu;
  if (lane == 31) {
    an = a[4];
    bn = b[4];
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t a0 = (q & 1) ? (q < 2 ? af.x : af.y) >> 16 : (q < 2 ? af.x : af.y) & 0xFFFFu;
    const uint32_t b0 = (q & 1) ? (q < 2 ? bf.x : bf.y) >> 16 : (q < 2 ? bf.x : bf.y) & 0xFFFFu;
    const uint32_t a1 = (q & 1) ? (q < 2 ? al.x : al.y) >> 16 : (q < 2 ? al.x : al.y) & 0xFFFFu;
    const uint32_t b1 = (q & 1) ? (q < 2 ? bl.x : bl.y) >> 16 : (q < 2 ? bl.x : bl.y) & 0xFFFFu;
    const uint32_t a2 = q == 0 ? af.x >> 16 : q == 1 ? af.y & 0xFFFFu : q == 2 ? af.y >> 16 : an;
    const uint32_t b2 = q == 0 ? bf.x >> 16 : q == 1 ? bf.y & 0xFFFFu : q == 2 ? bf.y >> 16 : bn;
    // some first entry here, and some entry there
    const bool on = (a1 > a0 && b2 > b0) || (b1 > b0 && a2 > a0);
    const uint32_t mask = __ballot_sync(0xffffffffu, on);
    if (on)
      pending[count + __popc(mask & ((1u << lane) - 1u))] =
          make_uint2(a0 | b0 << 16, (a1 - a0) | (a2 - a1) << 8 | (b1 - b0) << 16 | (b2 - b1) << 24);
    count += __popc(mask);
    __syncwarp();
    if (count >= 32) {  // the sites gathered last
      count -= 32;
      take(q, pending + count, 32u);
      __syncwarp();
    }
  }
  if (count) {
    take(4, pending, count);
    __syncwarp();
  }
}

// The distances of a tile pair (see the top of the file). The warps draw steps
// from a queue: first the s entries that a '-' counts against, 32 at a time, in
// the ranges where the other tile has '-' entries (a list of up to 224 rows
// each: the longest steps), then 128 sites at a time the s entries that meet,
// which 32 lanes share evenly. Where many rows of both tiles differ from the
// reference (a lineage's substitutions), one warp would be at a batch long after the
// others' steps: batches of more than 4,096 meetings are left to the end, and all
// warps share them (10 neighbouring sites where half of the rows differ: 7.2 -> 1.06
// ms, 60 of a clade of a tenth of the rows 23.8 -> 1.69; lines at 8,192 and 16,384:
// 400 sites with a tenth 1.69, 1.98 and 3.25). What bounds the kernel is the
// instructions of finding the meetings (IPC 3.3 of 4). 14,000 rows of 29,903 sites, one
// substitution per 1,000: 300 us (about 30 for the '-', 110 for the meetings,
// 65 to gather their sites, 30 to store), where the tensor-core engine takes 1,910. A
// lane an entry of the row tile instead, which looks its site up, took 655
// (the blocks' warps waited half of the time for those with '-' entries), 32
// sites at a time without gathering them and with every pair of a run 410.
__global__ void __launch_bounds__(kPairThreads, 2) k_site_pairs(SiteJob J) {
  extern __shared__ __align__(16) uint32_t acc[];
  __shared__ uint32_t chunks[2][kMaxRanges + 1];  // 32-entry chunks before each range
  __shared__ uint32_t queue, some_left;
  __shared__ __align__(4) uint8_t left[kMaxSteps];  // a step's batches of more than kHeavy meetings
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint2 *pending = reinterpret_cast<uint2 *>(acc + kT * kPitch) + warp * kPending;
  const uint64_t idx = J.first + blockIdx.x;
  uint32_t ti = (uint32_t)((sqrtf(8.0f * (float)idx + 1.0f) - 1.0f) * 0.5f);
  while ((uint64_t)ti * (ti + 1) / 2 > idx) --ti;
  while ((uint64_t)(ti + 1) * (ti + 2) / 2 <= idx) ++ti;
  const uint32_t tj = (uint32_t)(idx - (uint64_t)ti * (ti + 1) / 2);
  for (uint32_t i = threadIdx.x; i < kT * kPitch / 4; i += kPairThreads)
    reinterpret_cast<uint4 *>(acc)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (threadIdx.x == 0) queue = some_left = 0;
  for (uint32_t i = threadIdx.x; i < kMaxSteps / 4; i += kPairThreads) reinterpret_cast<uint32_t *>(left)[i] = 0u;
  const uint4 *bi = J.base + (uint64_t)ti * J.ranges, *bj = J.base + (uint64_t)tj * J.ranges;
  const uint16_t *oi = J.off + (uint64_t)ti * J.ranges * kOffSlot;
  const uint16_t *oj = J.off + (uint64_t)tj * J.ranges * kOffSlot;
  if (warp < 2) {
    const uint4 *b = warp ? bj : bi, *d = warp ? bi : bj;
    uint32_t run = 0;
    for (uint32_t r0 = 0; r0 < J.ranges; r0 += 32) {
      const uint32_t r = r0 + lane;
      const uint32_t k = r < J.ranges && d[r].w ? (b[r].y + 31u) / 32u : 0u;
      const uint32_t inc = warp_incl_scan(k);
      if (r < J.ranges) chunks[warp][r] = run + inc - k;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) chunks[warp][J.ranges] = run;
  }
  __syncthreads();
  const uint32_t ci = chunks[0][J.ranges], cd = ci + chunks[1][J.ranges];
  const uint32_t steps = cd + J.ranges * (kRange / kStepSites);
  for (;;) {
    uint32_t c = 0;
    if (lane == 0) c = atomicAdd(&queue, 1u);
    c = __shfl_sync(0xffffffffu, c, 0);
    if (c >= steps) break;
    if (c < cd) {
      // a '-' of one tile against the other's s entries
      const uint32_t side = c < ci ? 0u : 1u;
      if (side) c -= ci;
      uint32_t r = 0;  // its range: the last one that starts at or before c
      for (uint32_t r0 = 0; r0 < J.ranges; r0 += 32)
        r += __popc(__ballot_sync(0xffffffffu, r0 + lane < J.ranges && chunks[side][r0 + lane + 1] <= c));
      const uint4 mine = side ? bj[r] : bi[r], other = side ? bi[r] : bj[r];
      const uint32_t at = (c - chunks[side][r]) * 32 + lane;
      uint32_t e = 0, o0 = 0, len = 0;
      if (at < mine.y) {
        e = __ldg(J.es + mine.x + at);
        if (e & kMeetsDash) {
          const uint16_t *o = (side ? oi : oj) + (uint64_t)r * kOffSlot + kOffDash + e_site(e);
          o0 = o[0];
          len = o[1] - o0;
        }
      }
      const uint8_t *list = J.ed + other.z;
      for (uint32_t on = __ballot_sync(0xffffffffu, len > 0); on; on &= on - 1) {
        const int src = __ffs(on) - 1;
        const uint32_t row = e_row(__shfl_sync(0xffffffffu, e, src));
        const uint32_t n = __shfl_sync(0xffffffffu, len, src);
        const uint8_t *l = list + __shfl_sync(0xffffffffu, o0, src);
        if (side) meet_dashes<false>(acc, l, n, row, lane);
        else meet_dashes<true>(acc, l, n, row, lane);
      }
      continue;
    }
    const uint32_t k = c - cd, r = k / (kRange / kStepSites);
    const uint32_t at = r * kOffSlot + (k % (kRange / kStepSites)) * kStepSites + 4 * lane;
    const uint32_t *li = J.es + bi[r].x, *lj = J.es + bj[r].x;
    gather_sites(oi + at, oj + at, pending, lane, [&](int bit, const uint2 *sites, uint32_t n) {
      if (!meet_sites<false>(acc, sites, n, li, lj, lane) && lane == 0) {
        left[k] |= (uint8_t)(1u << bit);
        some_left = 1;
      }
    });
  }
  __syncthreads();
  if (some_left) {  // block-uniform: the batches left, shared by all warps
    for (uint32_t k0 = 0; k0 < steps - cd; k0 += 32) {
      uint32_t on = __ballot_sync(0xffffffffu, k0 + lane < steps - cd && left[k0 + lane] != 0);
      for (; on; on &= on - 1) {
        const uint32_t k = k0 + __ffs(on) - 1, r = k / (kRange / kStepSites);
        const uint32_t at = r * kOffSlot + (k % (kRange / kStepSites)) * kStepSites + 4 * lane;
        const uint32_t *li = J.es + bi[r].x, *lj = J.es + bj[r].x;
        gather_sites(oi + at, oj + at, pending, lane, [&](int bit, const uint2 *sites, uint32_t n) {
          if (left[k] >> bit & 1u) meet_sites<true>(acc, sites, n, li, lj, lane);
        });
      }
    }
    __syncthreads();
  }
  if (J.dtype == 1) store_rows<uint8_t>(J, acc, ti, tj);
  else if (J.dtype == 2) store_rows<uint16_t>(J, acc, ti, tj);
  else store_rows<uint32_t>(J, acc, ti, tj);
}

// Estimated times of a call in us, from measurements. The distances alone (dense /
// lists, us) at 1e-3, 3e-3, 1e-2, 1.5e-2 and 3e-2 substitutions per site:
//   n = 14,000, L = 29,903: 1,920 / 295, 471, 1,331, 2,188, 6,112
//   n = 5,000, L = 29,903: 363 / 55, 92, 256, 407, 1,097
//   n = 14,000, L = 3,000: 254 / 129, 182, 372, 540, 1,173
//   n = 8,000, L = 10,000: 261 / 65, 98, 245, 383, 965
//   n = 16,000, L = 600: 168 / 107, 147, 227, 324, 733
// and at 1e-3 with 10, 20 and 40 sites where half of 14,000 rows differ 1,193,
// 2,068 and 3,823. pairs: meetings of entries by the sample, which also counts those
// of 'N' runs and '-' (2.5e-6 us each puts the line between 1.2e-2 and 1.5e-2; 2e-6
// took the lists at 1.5e-2, 3.2e-6 the dense kernel at 1.2e-2).
// Building the lists costs about what expanding the operand does.
double dense_us(uint64_t n, uint64_t L, uint32_t planes) {
  const double pairs = 0.5 * (double)n * (double)n;
  return 60.0 + 1e-6 * pairs + 6.2e-10 * pairs * (double)L * (double)planes / 4.0;
}
double lists_us(uint64_t n, uint64_t L, double pairs) {
  const double tiles = (double)ceil_div(n, (uint64_t)kT), ranges = (double)ceil_div(L, (uint64_t)kRange);
  return 40.0 + 0.95e-6 * 0.5 * (double)n * (double)n +
         3.3e-3 * 0.5 * tiles * (tiles + 1) * ranges + 2.5e-6 * pairs;
}

Planes planes_of(const hd_alignment *a) {
  return Planes{a->plane_buf[0].as<uint4>(), a->planes > 4 ? a->plane_buf[1].as<uint4>() : nullptr,
                (uint32_t)a->planes, a->words};
}
uint64_t ref_bytes(const hd_alignment *a) { return a->words * (16 + 8); }

// -1: never, 1: always (where the lists can be used), 0: by the estimates
int forced() {
  if (std::getenv("HAMMINGDIST_KERNEL")) return -1;
  if (const char *e = std::getenv("HAMMINGDIST_SITE_LISTS")) return std::atoi(e) ? 1 : -1;
  return 0;
}
bool usable(hd_ctx *ctx, const hd_alignment *a, uint64_t rows) {
  return !a->base && ctx->engine_force < 0 && rows >= 2 && rows < (1ull << 31) &&
         a->length >= 1 && a->length <= (uint64_t)kMaxRanges * kRange &&
         (a->planes == 4 || a->groups == 2);
}

}  // namespace

Words sites_sample(hd_ctx *ctx, const hd_alignment *a, uint64_t rows) {
  if (!rows) rows = a->n_rows;
  const int f = forced();
  if (f < 0 || !usable(ctx, a, rows)) return Words{};
  // below this the launches and waits that build lists for one call cost what
  // they save (about 100 us)
  if (f == 0 && dense_us(rows, a->length, (uint32_t)a->planes) < 200.0) return Words{};
  const uint32_t w = (uint32_t)ceil_div(a->length, (uint64_t)32);
  return Words::of(w, w < 256 ? 1 : w < 512 ? 8 : 16);
}

bool sites_likely(hd_ctx *ctx, const hd_alignment *a, cudaStream_t st, uint64_t have, uint64_t rows) {
  if (!rows) rows = a->n_rows;
  if (!have) have = rows;
  const Words sel = sites_sample(ctx, a, rows);
  if (!sel.stride) return false;
  std::lock_guard<std::recursive_mutex> lk(a->lazy);
  if (a->sites && a->sites->verdict) return a->sites->verdict > 0;
  if (!a->sites) a->sites = std::make_unique<SiteLists>();
  SiteLists &S = *a->sites;
  if (forced() > 0) {
    S.verdict = 1;
    S.est_s = (double)rows * (double)a->length;  // room for anything (tests)
    S.est_d = S.est_s;
    return true;
  }
  const uint32_t quads = (uint32_t)ceil_div((uint64_t)sel.count, (uint64_t)4);
  const uint64_t count_bytes = (uint64_t)quads * 128 * 4 * 4;
  DevBuf buf(ref_bytes(a) + 80 + count_bytes, st);
  uint4 *r0 = buf.as<uint4>();
  uint2 *r1 = reinterpret_cast<uint2 *>(r0 + a->words);
  auto *sums = reinterpret_cast<unsigned long long *>(r1 + a->words);
  uint32_t *counts = reinterpret_cast<uint32_t *>(sums + 10);
  HD_CUDA(cudaMemsetAsync(counts, 0, count_bytes, st));
  const Planes p = planes_of(a);
  k_site_ref<<<(unsigned)ceil_div((uint64_t)sel.count, (uint64_t)2), 256, 0, st>>>(p, have, sel, r0,
                                                                                   r1);
  HD_LAUNCHED(ctx);
  // two rounds of a block's 64 rows: the rows' latency is most of its time
  const uint64_t shares = std::min<uint64_t>(ceil_div(have, (uint64_t)128), 65535);
  k_site_count<<<dim3(quads, (unsigned)shares), 256, 0, st>>>(p, have, a->length, sel, r0, r1, counts);
  HD_LAUNCHED(ctx);
  k_site_cost<<<1, 1024, 0, st>>>(counts, 32 * sel.edges(), quads * 128, sums);
  HD_LAUNCHED(ctx);
  uint64_t *h = pinned_words(ctx);
  HD_CUDA(cudaMemcpyAsync(h, sums, 80, cudaMemcpyDeviceToHost, st));
  HD_CUDA(cudaStreamSynchronize(st));
  const double inner = sel.words - sel.edges();
  const double up = sel.stride > 1 ? inner / std::min<double>(inner, sel.count - sel.edges()) : 1.0;
  const double more = (double)rows / (double)have;
  auto est = [&](int k) { return (double)h[k] + up * (double)h[5 + k]; };
  S.est_s = more * est(0);
  S.est_x = more * est(1);
  S.est_d = more * est(2);
  S.est_xd = more * more * est(4);
  const double t = lists_us(rows, a->length, more * more * (est(3) + est(4)));
  S.verdict = t < 0.9 * dense_us(rows, a->length, (uint32_t)a->planes) ? 1 : -1;
  return S.verdict > 0;
}

// (the stream is waited for before the lists count as there, for other threads
// and streams too)
bool ensure_sites(hd_ctx *ctx, const hd_alignment *a, cudaStream_t st) {
  if (!sites_sample(ctx, a).stride) return false;
  std::lock_guard<std::recursive_mutex> lk(a->lazy);
  if (!sites_likely(ctx, a, st)) return false;
  SiteLists &S = *a->sites;
  if (S.tiles) return true;
  const uint32_t words = (uint32_t)ceil_div(a->length, (uint64_t)32);
  const uint32_t ranges = (uint32_t)ceil_div((uint64_t)words, (uint64_t)kRangeWords);
  const uint64_t tiles = ceil_div(a->n_rows, (uint64_t)kT), slots = tiles * ranges;
  S.verdict = -1;  // until the lists are there
  const uint64_t all = a->n_rows * a->length;
  const uint64_t cap_s = std::min<uint64_t>(all, (uint64_t)(2.0 * S.est_s) + 16 * a->n_rows + 65536);
  const uint64_t cap_d = std::min<uint64_t>(all, (uint64_t)(2.0 * S.est_d) + 64 * a->n_rows + 65536);
  if (cap_s > 0xFFFFFFFFull || cap_d > 0xFFFFFFFFull) return false;
  DevBuf ref;
  const uint64_t tile_bytes = round_up(tiles * 4, 16);
  try {
    S.off = DevBuf(slots * kOffSlot * 2, st, true);
    S.base = DevBuf(slots * 16, st, true);
    S.es = DevBuf(cap_s * 4, st, true);
    S.ed = DevBuf(cap_d + 16, st, true);
    S.weight = DevBuf(a->n_rows * 4, st, true);
    ref = DevBuf(ref_bytes(a) + sizeof(BuildSums) + tile_bytes, st, true);
  } catch (const Error &e) {
    if (e.code != HD_ERR_OOM) throw;
    cudaGetLastError();
    S.release();
    return false;  // the engines need less memory
  }
  auto *sums = ref.as<BuildSums>();
  uint32_t *tile_sum = reinterpret_cast<uint32_t *>(sums + 1);
  uint4 *r0 = reinterpret_cast<uint4 *>(ref.as<uint8_t>() + sizeof(BuildSums) + tile_bytes);
  uint2 *r1 = reinterpret_cast<uint2 *>(r0 + a->words);
  static_assert(sizeof(BuildSums) % 16 == 0, "the reference follows");
  HD_CUDA(cudaMemsetAsync(sums, 0, sizeof(BuildSums) + tile_bytes, st));
  HD_CUDA(cudaMemsetAsync(S.weight.p, 0, a->n_rows * 4, st));
  const Planes p = planes_of(a);
  const Words sel = Words::of(words, 1);
  k_site_ref<<<(unsigned)ceil_div((uint64_t)words, (uint64_t)2), 256, 0, st>>>(
      p, a->n_rows, sel, r0, r1);
  HD_LAUNCHED(ctx);
  for (uint64_t t0 = 0; t0 < tiles; t0 += 65535) {
    const uint64_t tn = std::min<uint64_t>(65535, tiles - t0), row = t0 * kT;
    Planes q = p;
    q.g0 += row * p.pitch;
    if (q.g1) q.g1 += row * p.pitch;
    (q.planes > 4 ? k_site_lists<true> : k_site_lists<false>)<<<dim3(ranges, (unsigned)tn), 256, 0, st>>>(
        q, a->n_rows - row, a->length, words, r0, r1, ranges, cap_s, cap_d,
        S.base.as<uint4>() + t0 * ranges, S.off.as<uint16_t>() + t0 * ranges * kOffSlot,
        S.es.as<uint32_t>(), S.ed.as<uint8_t>(), S.weight.as<uint32_t>() + row, t0 == 0, sums);
    HD_LAUNCHED(ctx);
  }
  k_site_check<<<ranges * (kRange / 32), 256, 0, st>>>(
      S.off.as<uint16_t>(), (uint32_t)tiles, ranges, S.weight.as<uint32_t>(), a->n_rows, tile_sum, sums);
  HD_LAUNCHED(ctx);
  auto *h = reinterpret_cast<BuildSums *>(pinned_words(ctx));
  HD_CUDA(cudaMemcpyAsync(h, sums, sizeof(BuildSums), cudaMemcpyDeviceToHost, st));
  HD_CUDA(cudaStreamSynchronize(st));
  // every list fits, a pair's sum of c (at most the distance's other terms)
  // fits 16 bits, and the true count of pairs still costs less than the engine
  const bool fits = !h->full && 2ull * h->max_weight + h->zero <= 65535;
  // meetings with '-': the pairs found, by the sample's share of s entries that
  // do meet a '-', if the sample saw fewer
  const double dash = std::max(S.est_xd, (double)h->dashes * S.est_x / std::max(1.0, S.est_s));
  // a block with `peak` meetings takes 0.5 ns each, beyond the average ones': 40
  // lineages of 350 neighbouring rows, 60 sites each, take 2.6-3.0 ms, and 1.9 on the
  // tensor cores
  const double t = lists_us(a->n_rows, a->length, (double)h->pairs + dash) + 0.5e-3 * h->peak;
  if (!fits || (forced() == 0 && t > dense_us(a->n_rows, a->length, (uint32_t)a->planes))) {
    S.release();
    return false;
  }
  S.zero = h->zero;
  S.tiles = (uint32_t)tiles;
  S.ranges = ranges;
  S.verdict = 1;
  return true;
}

void prepare_site_jobs(hd_ctx *ctx, const std::vector<PairJobSpec> &specs, cudaStream_t stream,
                       PairLaunchPlan *plan, std::vector<char> &taken) {
  for (size_t k = 0; k < specs.size(); ++k) {
    const PairJobSpec &sp = specs[k];
    const hd_alignment *a = sp.aln;
    if (a->n_rows < 2 || sp.tile_hi <= sp.tile_lo || !ensure_sites(ctx, a, stream)) continue;
    const uint64_t edge = sp.cfg.tile > 0 ? (uint64_t)sp.cfg.tile : kTile;
    const uint64_t lo = sp.tile_lo * edge, hi = std::min<uint64_t>(sp.tile_hi * edge, a->n_rows);
    const SiteLists &S = *a->sites;
    PairLaunchPlan::Launch L;
    L.sites = true;
    L.jobs = 1;
    L.tile = kTile;
    L.tiles = mma_size_tiles(lo, hi);
    const uint64_t t0 = lo / kT, t1 = ceil_div(hi, (uint64_t)kT);
    L.grid = t1 * (t1 + 1) / 2 - t0 * (t0 + 1) / 2;
    if (L.grid > 0x7fffffffull) continue;
    SiteJob &J = L.site;
    J.base = S.base.as<uint4>();
    J.off = S.off.as<uint16_t>();
    J.es = S.es.as<uint32_t>();
    J.ed = S.ed.as<uint8_t>();
    J.weight = S.weight.as<uint32_t>();
    J.out = sp.d_out;
    J.out_base = sp.out_base;
    J.row_lo = lo;
    J.row_hi = hi;
    J.first = t0 * (t0 + 1) / 2;
    J.n = a->n_rows;
    J.ranges = S.ranges;
    J.zero = S.zero;
    J.max_dist = sp.max_dist;
    J.dtype = (uint32_t)sp.dtype;
    plan->launches.push_back(L);
    taken[k] = 1;
  }
}

void launch_sites(hd_ctx *ctx, const PairLaunchPlan::Launch &L, cudaStream_t stream) {
  static OncePerDevice once;
  once.run(ctx->device, [] {
    HD_CUDA(cudaFuncSetAttribute(k_site_pairs, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem));
  });
  k_site_pairs<<<(unsigned)L.grid, kPairThreads, kPairSmem, stream>>>(L.site);
  HD_LAUNCHED(ctx);
  ctx->last_pair_tiles += L.tiles;
}

}  // namespace hd
