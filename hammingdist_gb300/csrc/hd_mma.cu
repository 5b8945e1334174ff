// Tensor-core lower-triangle distances (tcgen05, block-scaled FP4) for the
// dense AND rule and the sparse rules.
//
// Replaces the reference's Dist<T> kernel (src/distance_cuda.cu:9-202) and,
// for use_gpu=False, its CPU loops (include/hamming/hamming_impl.hh:120-175).
// A site pair matches when the two codes share a bit: the dense rule's
// 4-bit codes (src/distance_cuda.cu:57-65; src/hamming_impl.cc:23-44: A, C,
// G, T one-hot, '-' all four bits, every other byte 0) or the sparse rules'
// one-hot classes over P = 5 or 6 planes with '-' as all P bits
// (src/hamming_impl.cc:93-129).
//
// For those codes the match indicator is a bilinear form. With e(x) the P
// plane bits of x and d(x) = [x = '-'],
//   match(a, b) = <e(a), e(b)> - (P - 1) d(a) d(b):
// the plane dot product is 1 for equal symbols and for a symbol against '-',
// P for '-' against '-' (hence the -(P - 1)), and 0 otherwise. Summed over
// the sites of two rows this is one dot product of P + 1 values per site, the
// dash value being 1 on the row side and -(P - 1) on the column side. All
// values are 0, 1, -3 or -4, exact in E2M1 (FP4: 0, 0.5, 1, 1.5, 2, 3, 4, 6
// and their negatives); -5 (P = 6) is not, so there the column side's dash
// is -4 and -1 in two blocks, each paired with the row side's +1. The MMAs
// are kind::mxf4 with every UE8M0 scale factor 1.0 and FP32 accumulation,
// exact while P L < 2^24. mismatches = L - matches.
//
// K order: first the P plane blocks of every 192-site chunk (partial sums up
// to P L), then the dash products, only for the chunks where some row of the
// operand has a '-' (the expansion marks them): elsewhere every dash product
// is 0. On aligned genomes the '-' sit mostly in leading and trailing runs, so
// a row's P + 1 blocks per chunk shrink to about P.
//
// Operand (one buffer serves rows and columns): each row's bit planes are
// expanded to packed E2M1, two sites per byte, in the layout the tensor
// cores read without a swizzle: for 8 rows (a row group) and 192 sites, the P
// planes (1.0), the dash as 1.0 (read for rows) and the dash as -(P - 1)
// (read for columns; -4 and -1 for P = 6) are blocks of 768 bytes, each six
// 128-byte core matrices (8 rows x 16 bytes = 32 sites). Sites past L are 0; the
// dash blocks of a large operand are written for the listed chunks only. A row
// group's blocks follow one another, so a TMA box of 16 groups brings one block
// of 128 rows. An alignment caches its operand; a view of a resident alignment (a
// serving window) gets one of its own rows.
//
// One launch serves a job table of matrices. Persistent pairs of CTAs (a
// cluster of two SMs, 352 threads each) walk a list of items: 256 rows x up to
// 496 columns of one job, in bands of tile rows, column-major within a band,
// so that resident pairs share operands in L2.
//  * warps 0 and 10 (one thread each) take turns to issue the TMA loads of one
//    96-byte K block of the CTA's 128 rows and of its half of the columns, 6
//    stages of 36,096 B; both CTAs' loads count on the first CTA's full barriers.
//    The first CTA's first producer also draws the items of a queued launch;
//    warp 0 allocates and frees the TMEM;
//  * warp 1 of the first CTA (one thread) issues tcgen05.mma.cta_group::2
//    .kind::mxf4.block_scale with K = 96 (the shape only sm_103a has: 1.5
//    times the rate of K = 64), M = 256 and N = 256 and 240, two K steps per
//    block, into both CTAs' TMEM (columns 0-255 and 256-495); the unit scale
//    factors sit in columns 496-511. Each stage's MMAs are committed to both
//    CTAs' empty barriers, an item's last ones to `done`;
//  * warps 2-9, two per TMEM lane quarter, each read 32 rows x 248 columns
//    (tcgen05.ld), form min(L - matches, max_dist) (safe_int_cast,
//    include/hamming/hamming_impl.hh:37-45) as packed 16-bit values in
//    registers and release the accumulators (`tmem_free`) at once: the next
//    item's MMAs run while the warp turns 32 x 28 pieces around in shared
//    memory and stores them row by row. 32-bit outputs are stored piece by
//    piece before the release.
// Where items do not divide evenly among the pairs (few rows, or the last
// round), the rest is split along K at chunk boundaries: a piece leaves its
// partial distances in a workspace, and k_pair_fix adds a tile's pieces.
// Every wait is bounded; on a timeout the CTA records it in the status word,
// waits (bounded) for its own copies and MMAs, frees its TMEM and returns.
//
// What bounds it (n = 14,000, L = 29,903, 8.05 FLOP per pair-site): the loads.
// A pair's K block takes 497 cycles of MMAs and brings 72 KB; measured alone,
// the loads reach 77 B per cycle and SM, the MMAs 14.4 PFLOP/s.
//   form (K block x stages), alone             operand in L2 / over 100 MB
//   single CTAs, K = 96, 96 B x 3              9.1 / 8.0 PFLOP/s
//   CTA pairs, K = 96, 96 B x 6               13.4 / 12.9
//   CTA pairs, K = 96, 144 B x 4              14.5 / 12.6
//   CTA pairs, K = 96, 192 B x 3              14.5 / 12.2
// The smaller blocks let the loads run further ahead of the MMAs, and two TMA
// threads keep up with them: 4 x 144 B with one 1,985 us, 6 x 96 B with one
// 1,940, with two 1,925 (531 cycles a block; 500 with every load from the same
// rows), 84% of the FP4 rate hd_measure_mma_peak reports.
// Pairs halve the column bytes an SM loads and its MMAs read.
#include <algorithm>
#include <cstdlib>
#include <functional>
#include <queue>
#include <string>
#include <type_traits>
#include <vector>

#include "hd_internal.cuh"

namespace hd {
namespace {

constexpr int kEpiWarps = 8;      // two per TMEM lane quarter
// warp 0: TMA, warp 1: MMA, warps 2-9: epilogue, warp 10: TMA
constexpr int kMmaThreads = 96 + 32 * kEpiWarps;
constexpr uint32_t kProducers = 2;  // the TMA warps take K blocks in turn
constexpr int kMmaStages = 6;
static_assert(kMmaStages % kProducers == 0, "a stage always has the same producer");
constexpr uint32_t kTM = 128;                          // rows of a tile row, and of a CTA in a pair
constexpr uint32_t kRowsPerItem = 2 * kTM;             // M of a CTA pair's MMA
constexpr uint32_t kN0 = 256, kN1 = 240;               // N of an item's two MMAs
constexpr uint32_t kItemCols = kN0 + kN1;
constexpr uint32_t kChunkWords = 6;                    // 32-site words per chunk (192 sites)
constexpr uint32_t kChunkSites = 32 * kChunkWords;
constexpr uint32_t kBlockK = 16 * kChunkWords;         // bytes of K per row and block (96)
constexpr uint32_t kGroupBytes = 8 * kBlockK;          // one block of 8 rows (768)
constexpr uint32_t kKStep = 48;                        // bytes of K per MMA (96 values)
constexpr uint32_t kABytes = kTM / 8 * kGroupBytes;              // 128 rows
constexpr uint32_t kB0Bytes = kN0 / 16 * kGroupBytes;            // a CTA's half of 256 columns
constexpr uint32_t kBBytes = kItemCols / 16 * kGroupBytes;       // and of all 496
constexpr uint32_t kStageBytes = kABytes + kBBytes;              // 36,096
// the epilogue warps' pieces: 32 rows x 14 words (28 16-bit columns), row r
// at words 15 r (conflict-free by row and by column)
constexpr uint32_t kPieceWords = 14, kPiecePitch = 15;
constexpr uint32_t kEpiBytes = kEpiWarps * 32 * kPiecePitch * 4;
constexpr int kMmaSmem = kMmaStages * kStageBytes + kEpiBytes + 128;
static_assert(kBlockK % kKStep == 0 && kStageBytes % 128 == 0, "K steps and TMA destinations");
static_assert(kMmaSmem + 256 <= 232448, "shared memory above the per-block limit");
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kHalfCols = kItemCols / 2;         // columns per epilogue warp (248 at most)
constexpr uint32_t kHalfWords = kHalfCols / 2;        // packed 16-bit pairs (124)
constexpr uint32_t kSfColA = kItemCols, kSfColB = kItemCols + 8;  // unit scale factors
constexpr uint32_t kSfWord = 0x7F7F7F7Fu;             // four UE8M0 scale factors of 2^0
constexpr uint64_t kMmaWaitNs = 1000000000ull;        // 1 s
constexpr uint32_t kMmaBand = 16;  // item rows (256 rows) per L2 band (HAMMINGDIST_MMA_BAND overrides)
constexpr int kItemRing = 4;                          // item indices handed to the other warps
// arrivals that free a ring slot: the MMA warp, the producers but the one that
// fills it, and both CTAs' epilogue warps
constexpr uint32_t kRingReaders = 1 + (2 * kProducers - 1) + 2 * kEpiWarps;
constexpr uint32_t kNoItem = 0xFFFFFFFFu;             // end of this pair's items
constexpr uint32_t kNoSlot = 0xFFFFFFFFu;             // an item that covers all of K
// A split tile's partial distances of one K piece: 16-bit pairs, per CTA,
// column half, lane quarter and word the 32 lanes of a warp
constexpr uint64_t kSlotBytes = 2ull * 2 * 4 * kHalfWords * 32 * 4;
// K pieces of fewer chunks than this cost more in barriers, workspace traffic
// and k_pair_fix than they spread (six chunks of four planes run 6.5 us). A call
// with pieces of 3, 6 and 10 chunks: 700 rows of 8,000 sites 72.2, 66.7 and
// 74.2 us, 1,500 of 1,273 (7 chunks) 63.5, 62.3 and 61.8.
constexpr uint32_t kMinPart = 6;
// blocks of 192 sites per row and chunk in the operand: the P planes, the row
// side's dash and the column side's dash (two blocks for P = 6: -4 and -1)
__host__ __device__ constexpr uint32_t op_blocks(uint32_t planes) {
  return planes + (planes == 6 ? 3u : 2u);
}
__host__ __device__ constexpr uint32_t op_chunks(uint64_t sites) {
  return (uint32_t)((sites + kChunkSites - 1) / kChunkSites);
}
// operand bytes of 8 rows
__host__ __device__ constexpr uint64_t op_group_bytes(uint32_t planes, uint64_t sites) {
  return (uint64_t)op_chunks(sites) * op_blocks(planes) * kGroupBytes;
}
uint64_t op_bytes(uint32_t planes, uint64_t sites, uint64_t rows) {
  return ceil_div(rows, (uint64_t)8) * op_group_bytes(planes, sites);
}
// E2M1 codes: 1.0, and the column side's -(P - 1): -3 for P = 4, -4 else
// (then -1 for P = 6)
constexpr uint32_t kE2M1One = 0x2u, kE2M1Neg1 = 0xAu;
__device__ __forceinline__ uint32_t dash_neg(uint32_t planes) { return planes == 4 ? 0xDu : 0xEu; }
// instruction descriptor (block-scaled kinds): A and B E2M1 (1 at bits 7-9
// and 10-12), both K-major, N >> 3 at bits 17-22, scale factors UE8M0 (bit
// 23), M >> 4 at bits 24-28, scale factor ids 0, K = 96 (bit 31); D is FP32
__host__ __device__ constexpr uint32_t idesc_mxf4(uint32_t n) {
  return (1u << 7) | (1u << 10) | ((n >> 3) << 17) | (1u << 23) |
         ((kRowsPerItem >> 4) << 24) | (1u << 31);
}

}  // namespace

// One matrix of a launch (device copy): its output and the chunks whose dash
// products count. Its operand's tensor maps are at 2 job of the launch's maps
// (boxes of one block of 128 and of 248 rows).
struct MmaJob {
  void *out;                     // lt index out_base at out[0]
  unsigned long long out_base;
  uint32_t row_hi, sites, max_dist, dtype;  // rows end, L, cap, 1/2/4 bytes
  uint32_t planes;                          // P
  uint32_t chunks;                          // 192-site chunks per row
  const uint32_t *dash_list;                // the chunks whose dash products count
  const uint32_t *dash_rank;                // per chunk: listed chunks before it (chunks + 1)
  unsigned long long pairs;                 // lower-triangle pairs of this launch
};

// One work item: rows [row0, row0 + 256) x columns [col0, col0 + n0 + n1) of
// job `job` over the chunks [c_lo, c_hi); a piece of a split tile leaves its
// partial distances in workspace slot `slot`. n0 and n1, the N of the item's
// MMAs, in units of 16; n1 > 0 only after n0 = 256 / 16.
struct MmaItem {
  uint32_t job, row0, col0;  // job kNoItem: none (padding of the static order)
  uint8_t n0_16, n1_16, planes, pad;
  uint32_t c_lo, c_hi, slot, pad2;
  __host__ __device__ uint32_t n0() const { return 16u * n0_16; }
  __host__ __device__ uint32_t n1() const { return 16u * n1_16; }
};
static_assert(sizeof(MmaItem) == 32, "items are read as two 16-byte vectors");
// One split tile: the workspace slots [slot, slot + parts) of its pieces.
struct MmaFix {
  uint32_t job, row0, col0, cols, slot, parts;
};

namespace {

// 8 bits -> 8 nibbles (bit i -> the low bit of nibble i), times the E2M1
// code `v` (no carries: each nibble is 0 or 1 before the multiply)
__device__ __forceinline__ uint32_t nib8(uint32_t b, uint32_t v) {
  b = (b | (b << 12)) & 0x000F000Fu;
  b = (b | (b << 6)) & 0x03030303u;
  b = (b | (b << 3)) & 0x11111111u;
  return b * v;
}
// 32 sites (one plane word) -> 16 bytes of E2M1: site s in nibble s (byte
// s / 2, low nibble for even s), `v` where the bit is set, else 0
__device__ __forceinline__ void put16(uint8_t *dst, uint32_t w, uint32_t v) {
  *reinterpret_cast<uint4 *>(dst) =
      make_uint4(nib8(w & 0xFFu, v), nib8((w >> 8) & 0xFFu, v), nib8((w >> 16) & 0xFFu, v),
                 nib8(w >> 24, v));
}

// the dash blocks' 16 bytes of a word
__device__ __forceinline__ void put_dash(uint8_t *dst, uint32_t dash, uint32_t planes) {
  put16(dst, dash, kE2M1One);                       // 1.0: the row side
  put16(dst + kGroupBytes, dash, dash_neg(planes));  // the column side
  if (planes == 6) put16(dst + 2 * kGroupBytes, dash, kE2M1Neg1);
}

// One extension of an operand: rows [row_lo, row_hi) of the planes g0, g1 in x.
struct OpRows {
  const uint4 *g0, *g1;
  uint8_t *x;
  uint32_t *marks;  // per chunk, and a count of k_expand_op's blocks (0 between launches)
  uint32_t *list;   // the marked chunks, then the listed ones before each chunk (chunks + 1)
  unsigned long long row_lo, row_hi, sites;
  uint32_t planes, words, ext;
  uint32_t blocks;  // the listed chunks' dash blocks are to be written (k_dash_blocks)
};

// The ascending list of the chunks whose mark is set, and for every chunk the
// listed ones before it; by a whole block.
__device__ __forceinline__ void list_marked(const OpRows &o, uint32_t *tmp /*[33]*/) {
  const uint32_t chunks = op_chunks(o.sites);
  uint32_t *before = o.list + chunks, n = 0;
  for (uint32_t c0 = 0; c0 < chunks; c0 += blockDim.x) {
    const uint32_t c = c0 + threadIdx.x;
    const uint32_t on = c < chunks && __ldcg(o.marks + c) != 0u ? 1u : 0u;
    uint32_t total;
    const uint32_t at = n + block_excl_scan<uint32_t>(on, tmp, total);
    if (on) o.list[at] = c;
    if (c < chunks) before[c] = at;
    n += total;
  }
  if (threadIdx.x == 0) before[chunks] = n;
}

// Rows of a P-plane alignment (P = 4: the AND rule; 5, 6: the sparse rules,
// planes 4-5 in the second group) -> the plane blocks of their E2M1 operand
// rows and, unless k_dash_blocks follows, the dash blocks of every chunk. One
// thread per (row, 32-site word): 16 or 32 bytes read, 16 bytes written per block.
// A warp takes one row group x 4 words, lane l row l % 8, so that each of its
// stores fills whole 128-byte core matrices; a block of 256 threads takes 32
// words. The words past the alignment's, up to whole chunks, are written as 0.
// The dash is the AND of the P planes ('-' has every plane); a chunk where some
// row has its first '-' is marked with `ext`. The block that ends last lists the
// marked chunks (kList).
template <bool kList>
__global__ void __launch_bounds__(256) k_expand_op(OpRows o) {
  __shared__ uint32_t tmp[33];
  __shared__ bool last;
  const uint32_t nb = op_blocks(o.planes), chunks = op_chunks(o.sites);
  const uint32_t w = blockIdx.x * 32 + threadIdx.x / 8;
  const uint32_t c = w / kChunkWords;
  const uint64_t s0 = (uint64_t)w * 32;
  const uint32_t valid = s0 >= o.sites ? 0u : (o.sites - s0 >= 32 ? 0xffffffffu : ((1u << (o.sites - s0)) - 1u));
  const uint64_t in_group = (uint64_t)c * nb * kGroupBytes + (w - c * kChunkWords) * 128u +
                            (threadIdx.x & 7u) * 16u;
  const uint64_t group_bytes = op_group_bytes(o.planes, o.sites);
  for (uint64_t g = o.row_lo / 8 + blockIdx.y; c < chunks && g * 8 < o.row_hi; g += gridDim.y) {
    const uint64_t r = g * 8 + (threadIdx.x & 7u);
    if (r < o.row_lo || r >= o.row_hi) continue;
    uint4 p = make_uint4(0u, 0u, 0u, 0u), p1 = p;
    if (w < o.words) {
      p = __ldg(o.g0 + r * o.words + w);
      if (o.planes > 4) p1 = __ldg(o.g1 + r * o.words + w);
    }
    uint32_t dash = p.x & p.y & p.z & p.w & valid;
    if (o.planes > 4) dash &= p1.x;
    if (o.planes > 5) dash &= p1.y;
    uint8_t *blk = o.x + g * group_bytes + in_group;
    put16(blk, p.x & valid, kE2M1One);
    put16(blk + kGroupBytes, p.y & valid, kE2M1One);
    put16(blk + 2 * kGroupBytes, p.z & valid, kE2M1One);
    put16(blk + 3 * kGroupBytes, p.w & valid, kE2M1One);
    if (o.planes > 4) put16(blk + 4 * kGroupBytes, p1.x & valid, kE2M1One);
    if (o.planes > 5) put16(blk + 5 * kGroupBytes, p1.y & valid, kE2M1One);
    if (!o.blocks) put_dash(blk + o.planes * kGroupBytes, dash, o.planes);
    if (dash && !o.marks[c]) o.marks[c] = o.ext;  // every writer stores the same
  }
  if (!kList) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();  // the block's marks, before its count
    last = atomicAdd(o.marks + chunks, 1u) == gridDim.x * gridDim.y - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  list_marked(o, tmp);
  if (threadIdx.x == 0) o.marks[chunks] = 0;
}

// The dash blocks of the marked chunks (the job's list): of rows [row_lo,
// row_hi), and for a chunk that extension `ext` marked first of the rows
// before them, which have no '-' there. The other chunks' blocks are never
// read, and stay unwritten: two of an operand's six blocks (four planes),
// 0.4 of 1.3 GB for 14,000 rows of 29,903 sites. A thread per (row, word):
// 48 threads take one row group of a chunk. Block row y takes job y of `jobs`,
// or `one` without them.
constexpr uint32_t kDashGroups = 4;  // row groups per block
__global__ void __launch_bounds__(kDashGroups * 8 * kChunkWords)
    k_dash_blocks(OpRows one, const OpRows *__restrict__ jobs, uint32_t n_jobs) {
  const uint32_t sub = threadIdx.x / (8 * kChunkWords), u = threadIdx.x % (8 * kChunkWords);
  for (uint32_t q = blockIdx.y; q < n_jobs; q += gridDim.y) {
    const OpRows j = jobs ? jobs[q] : one;
    if (!j.blocks) continue;
    const uint32_t nb = op_blocks(j.planes), chunks = op_chunks(j.sites);
    const uint64_t group_bytes = op_group_bytes(j.planes, j.sites);
    const uint64_t batches = ((j.row_hi + 7) / 8 + kDashGroups - 1) / kDashGroups;
    const uint64_t work = batches * j.list[2 * chunks];
    for (uint64_t t = blockIdx.x; t < work; t += gridDim.x) {
      const uint64_t i = t / batches, g = (t - i * batches) * kDashGroups + sub;
      const uint32_t c = j.list[i], w = c * kChunkWords + u / 8;
      const uint64_t r = g * 8 + (u & 7u), s0 = (uint64_t)w * 32;
      if (r >= j.row_hi || (r < j.row_lo && j.marks[c] != j.ext)) continue;
      uint32_t dash = s0 >= j.sites ? 0u : (j.sites - s0 >= 32 ? 0xffffffffu : ((1u << (j.sites - s0)) - 1u));
      if (w < j.words) {
        const uint4 p = j.g0[r * j.words + w];
        dash &= p.x & p.y & p.z & p.w;
        if (j.planes > 4) {
          const uint4 p1 = j.g1[r * j.words + w];
          dash &= p1.x;
          if (j.planes > 5) dash &= p1.y;
        }
      }
      uint8_t *blk = j.x + g * group_bytes + ((uint64_t)c * nb + j.planes) * kGroupBytes + u * 16u;
      put_dash(blk, dash, j.planes);
    }
  }
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
// The AND rule's codes of 8 sites (bytes of w0 and w1, in order: A 1, C 2, G 4,
// T 8, '-' 15, any other byte 0), one a byte, to c0 and c1. The low three bits
// of a byte pick its symbol and the symbol's code; a byte unlike its symbol
// has code 0 (0x80 of `ne`, spread over the byte).
__device__ __forceinline__ void and_codes(uint32_t w0, uint32_t w1, uint32_t &c0, uint32_t &c1) {
  constexpr uint32_t kCodeLo = 0x02000100u, kCodeHi = 0x04000F08u;  // X A . C / T - . G
  uint32_t a = w0 & 0x07070707u, b = w1 & 0x07070707u;
  a |= a >> 4;
  b |= b >> 4;
  const uint32_t sel = prmt(a, b, 0x6420u), sel1 = sel >> 16;  // a nibble a site
  const uint32_t x0 = w0 ^ prmt(kSymLo, kSymHi, sel), x1 = w1 ^ prmt(kSymLo, kSymHi, sel1);
  const uint32_t ne0 = ((x0 & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x0;
  const uint32_t ne1 = ((x1 & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x1;
  c0 = prmt(kCodeLo, kCodeHi, sel) & ~prmt(ne0, 0u, 0xBA98u);
  c1 = prmt(kCodeLo, kCodeHi, sel1) & ~prmt(ne1, 0u, 0xBA98u);
}

// 32 sites, the bytes of v[0 .. 8] from bit db on -> their codes as nibbles z in
// site order, 8 sites a word, and the plane words pl. kTail: the sites from
// `valid` on are past L, '-' in the planes and 0 in z.
template <bool kTail>
__device__ __forceinline__ void pack_sites(const uint32_t *v, uint32_t db, uint32_t valid,
                                           uint32_t *z, uint32_t *pl) {
  uint32_t t[4];  // byte p: plane p's bits of 8 sites
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    uint32_t c0, c1;
    and_codes(__funnelshift_r(v[2 * m], v[2 * m + 1], db),
              __funnelshift_r(v[2 * m + 1], v[2 * m + 2], db), c0, c1);
    const uint32_t k = valid > 8u * m ? valid - 8u * m : 0u;  // sites of these 8 and after
    if (kTail && k < 8u) {
      const uint32_t m0 = k >= 4u ? 0xFFFFFFFFu : (1u << (8u * k)) - 1u;
      const uint32_t m1 = k <= 4u ? 0u : (1u << (8u * (k - 4u))) - 1u;
      c0 = (c0 & m0) | (0x0F0F0F0Fu & ~m0);
      c1 = (c1 & m1) | (0x0F0F0F0Fu & ~m1);
    }
    uint32_t y = c0 + (c1 << 4);  // bit 8 (s mod 4) + 4 (s / 4) + p
    uint32_t q = (y ^ (y >> 14)) & 0x0000CCCCu;  // bit 4 of the index with bit 1
    y ^= q ^ (q << 14);
    q = (y ^ (y >> 7)) & 0x00AA00AAu;  // bit 3 with bit 0
    t[m] = y ^ q ^ (q << 7);
    z[m] = prmt(c0 | (c0 >> 4), c1 | (c1 >> 4), 0x6420u);
    if (kTail && k < 8u) z[m] &= (1u << (4u * k)) - 1u;
  }
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const uint32_t sel = (uint32_t)p | ((uint32_t)(4 + p) << 4);
    pl[p] = prmt(prmt(t[0], t[1], sel), prmt(t[2], t[3], sel), 0x5410u);
  }
}

// The text of rows [row_lo, row_hi) of the AND rule -> their plane words and
// the plane blocks of their E2M1 operand rows, in one pass: row row_lo + i is
// record rows[i] (none: i; no rs: one record, at the start). Thread and store layout as in k_expand_op; the
// sites past L are '-' in the planes and 0 in the operand. A thread reads the
// 32 bytes of its sites as aligned 16-byte vectors. Eight sites' codes are
// one word of nibbles z, in site order, in which plane p's E2M1 ones are the
// bits p moved to bit 1 of each nibble; with the codes of sites k and k + 4
// in a byte instead, two exchanges of bits leave plane p's 8 bits in byte p.
// 14,000 rows of 29,903 sites move 1.47 GB (6.2 TB/s) in 238 us. Packing
// and then expanding, with the planes read back and dash blocks written for
// every chunk, took 198 + 212 us (1.9 GB).
template <bool kOp>
__global__ void __launch_bounds__(256, 6)
    k_pack_op(const uint8_t *base, uint64_t bytes, const uint64_t *__restrict__ rs,
              const uint64_t *__restrict__ rows, uint64_t row_lo, uint64_t row_hi, uint64_t L,
              uint32_t words, uint4 *__restrict__ g0, uint4 *__restrict__ g1,
              uint8_t *__restrict__ x, uint32_t *dash_chunk, uint32_t ext, Words sel) {
  constexpr uint32_t kPlanes = 4, nb = op_blocks(kPlanes);
  const uint32_t op_words = kOp ? op_chunks(L) * kChunkWords : 0u;
  // without the operand a warp takes 32 words of one row instead
  const uint32_t k = blockIdx.x * 32 + (kOp ? threadIdx.x / 8 : threadIdx.x & 31u);
  const uint32_t w = kOp ? k : sel.at(k);
  const uint32_t row = kOp ? threadIdx.x & 7u : threadIdx.x >> 5;
  if (w >= words && w >= op_words) return;
  const uint32_t c = w / kChunkWords;
  const uint64_t s0 = (uint64_t)w * 32;
  const uint32_t valid = s0 >= L ? 0u : L - s0 >= 32 ? 32u : (uint32_t)(L - s0);  // sites
  const uint64_t in_group = (uint64_t)c * nb * kGroupBytes + (w - c * kChunkWords) * 128u +
                            (threadIdx.x & 7u) * 16u;
  const uint64_t group_bytes = op_group_bytes(kPlanes, L);
  const uint64_t lo = reinterpret_cast<uint64_t>(base), hi = lo + bytes;
  // the record starts of a group's rows are fetched one group ahead
  auto start_of = [&](uint64_t r) -> uint64_t {
    if (!valid || r < row_lo || r >= row_hi) return 0;
    return lo + s0 + (rs ? rs[rows ? rows[r - row_lo] : r - row_lo] : 0);
  };
  uint64_t r = row_lo / 8 * 8 + blockIdx.y * 8 + row;
  uint64_t next = start_of(r);
  uint8_t *blk = x + (r / 8) * group_bytes + in_group;
  const uint64_t blk_step = gridDim.y * group_bytes;
  for (; (r & ~7ull) < row_hi; r += gridDim.y * 8, blk += blk_step) {
    const uint64_t P = next;
    next = start_of(r + gridDim.y * 8);
    if (r < row_lo || r >= row_hi) continue;
    uint32_t v[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) v[k] = 0u;
    uint32_t dw = 0, db = 0;
    if (valid) {
      const uint64_t A = P & ~15ull;
      const uint32_t d = (uint32_t)(P - A);
      dw = d >> 2;
      db = 8u * (d & 3u);
      uint4 a, b, e = make_uint4(0u, 0u, 0u, 0u);
      if (A >= lo && A + 48 <= hi) {
        const uint4 *q = reinterpret_cast<const uint4 *>(A);
        a = __ldg(q);
        b = __ldg(q + 1);
        if (d) e = __ldg(q + 2);
      } else {
        a = load16_in(A, lo, hi);
        b = load16_in(A + 16, lo, hi);
        if (d) e = load16_in(A + 32, lo, hi);
      }
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
      v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
      v[8] = e.x; v[9] = e.y; v[10] = e.z; v[11] = e.w;
    }
    // the words from byte 4 dw on
    if (kOp) {
#pragma unroll
      for (int k = 0; k < 11; ++k) v[k] = (dw & 1u) ? v[k + 1] : v[k];
#pragma unroll
      for (int k = 0; k < 9; ++k) v[k] = (dw & 2u) ? v[k + 2] : v[k];
    } else {  // the same for the whole warp but its words past the row's end, which read 0
      if (__any_sync(__activemask(), dw & 1u)) {
#pragma unroll
        for (int k = 0; k < 11; ++k) v[k] = v[k + 1];
      }
      if (__any_sync(__activemask(), dw & 2u)) {
#pragma unroll
        for (int k = 0; k < 9; ++k) v[k] = v[k + 2];
      }
    }
    uint32_t z[4], pl[4];
    if (valid == 32u) pack_sites<false>(v, db, valid, z, pl);
    else pack_sites<true>(v, db, valid, z, pl);
    if (w < words) {
      const uint4 o = make_uint4(pl[0], pl[1], pl[2], pl[3]);
      g0[r * words + w] = o;
      if (g1) g1[r * words + w] = o;
    }
    if (kOp && w < op_words) {
      constexpr uint32_t kOne = 0x22222222u;  // E2M1 1.0 in every nibble
      uint4 *out = reinterpret_cast<uint4 *>(blk);
      constexpr uint32_t kNext = kGroupBytes / 16;
      out[0] = make_uint4((z[0] << 1) & kOne, (z[1] << 1) & kOne, (z[2] << 1) & kOne,
                          (z[3] << 1) & kOne);
      out[kNext] = make_uint4(z[0] & kOne, z[1] & kOne, z[2] & kOne, z[3] & kOne);
      out[2 * kNext] = make_uint4((z[0] >> 1) & kOne, (z[1] >> 1) & kOne, (z[2] >> 1) & kOne,
                                  (z[3] >> 1) & kOne);
      out[3 * kNext] = make_uint4((z[0] >> 2) & kOne, (z[1] >> 2) & kOne, (z[2] >> 2) & kOne,
                                  (z[3] >> 2) & kOne);
      uint32_t dash = pl[0] & pl[1] & pl[2] & pl[3];
      if (valid < 32u) dash &= (1u << valid) - 1u;
      if (dash && !dash_chunk[c]) dash_chunk[c] = ext;  // every writer stores the same
    }
  }
}

// ------------------------------------------------------- tcgen05 helpers
// Shared-memory matrix descriptor, K-major, no swizzle: start address >> 4
// (bits 0-13), 128 B between the core matrices along K (bits 16-29), one
// block between 8-row groups (bits 32-45), descriptor version 1 (bits 46-47).
__device__ __forceinline__ uint64_t core_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(128 >> 4) << 16) |
         ((uint64_t)(kGroupBytes >> 4) << 32) | ((uint64_t)1 << 46);
}
__device__ __forceinline__ void tmem_alloc(uint32_t *dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// address, in the cluster's shared memory, of CTA `rank`'s copy of a local one
__device__ __forceinline__ uint32_t map_rank(uint32_t saddr, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
  return a;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// the same without ordering memory: it does not wait for the stores in flight
__device__ __forceinline__ void cluster_sync_relaxed() {
  asm volatile("barrier.cluster.arrive.relaxed;\n\tbarrier.cluster.wait;" ::: "memory");
}
// D (+)= A B^T over K = 96 E2M1 values on the pair's tensor cores, every block
// of 32 scaled by the UE8M0 factors at TMEM addresses sfa and sfb
__device__ __forceinline__ void mma_f4(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                       uint32_t idesc, uint32_t accumulate, uint32_t sfa,
                                       uint32_t sfb) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf4.block_scale.block32 [%0], %1, %2, %3, [%5], "
      "[%6], p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
      : "memory");
}
// One K block (96 bytes a row) of an item: its two K steps against both
// column halves, or the first alone.
template <bool kSecond>
__device__ __forceinline__ void mma_block(uint32_t tmem, uint64_t a_desc, uint32_t id0, uint32_t id1,
                                          bool accumulate) {
  constexpr uint64_t kStep = 128 * (kKStep / 16) >> 4;  // three core matrices
  const uint64_t b0 = a_desc + (kABytes >> 4), b1 = b0 + (kB0Bytes >> 4);  // after 128 columns
#pragma unroll
  for (uint32_t k = 0; k < kBlockK / kKStep; ++k) {
    const uint32_t acc = (accumulate || k) ? 1u : 0u;
    mma_f4(tmem, a_desc + k * kStep, b0 + k * kStep, id0, acc, tmem + kSfColA, tmem + kSfColB);
    if (kSecond)
      mma_f4(tmem + kN0, a_desc + k * kStep, b1 + k * kStep, id1, acc, tmem + kSfColA, tmem + kSfColB);
  }
}
// one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(p));
  return p != 0;
}
// The unit scale factors: this warp writes kSfWord to the NC TMEM columns
// from col0 in its lane quarter (lane base `t_lane`) and waits for the
// stores; the caller fences before the MMAs read them.
template <uint32_t NC>
__device__ __forceinline__ void write_unit_scales(uint32_t t_lane, uint32_t col0) {
#pragma unroll
  for (uint32_t c = col0; c < col0 + NC; c += 4)
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(t_lane + c),
                 "r"(kSfWord), "r"(kSfWord), "r"(kSfWord), "r"(kSfWord)
                 : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// arrives on both CTAs' barrier at `bar` once every earlier tcgen05.mma of
// this thread has completed
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%0], %1;" ::"r"(bar),
      "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
// bounded wait for a phase that the copies or the tensor cores complete, or
// (kCluster) that a thread of either CTA completes to hand over what it wrote
template <bool kCluster>
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  if (kCluster)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  return ok != 0;
}
template <bool kCluster = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
  if (mbar_try<kCluster>(bar, parity)) return true;
  const long long t0 = clock64(), limit = wait_cycles(limit_ns);
  for (;;) {
    if (mbar_try<kCluster>(bar, parity)) return true;
    if (clock64() - t0 > limit) return false;
  }
}
// TMA box of a pair's CTA: into its own shared memory, completion counted on
// the barrier `bar` of the first CTA
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap *map, int32_t x,
                                              int32_t y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// 32 lanes x 16 consecutive 32-bit columns
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {"
      "%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15 "
      "}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
// 32 lanes x 8 consecutive 32-bit columns
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]),
                 "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// min(sites - matches, cap) of two accumulator columns as packed 16-bit
// values (cap <= 65535). FP32 throughout: every operand is an integer below
// 2^24, and adding 2^23 leaves the value in the low mantissa bits, which
// avoids the quarter-rate float-to-integer conversion while the accumulators
// are held.
__device__ __forceinline__ uint32_t pack2(uint32_t d0, uint32_t d1, float sites, float cap) {
  const float m0 = fminf(sites - __uint_as_float(d0), cap) + 8388608.0f;
  const float m1 = fminf(sites - __uint_as_float(d1), cap) + 8388608.0f;
  return __byte_perm(__float_as_uint(m0), __float_as_uint(m1), 0x5410u);
}

// This warp's 32 rows x 128 columns from t0 and 120 from t1, packed: word w
// holds columns 2 w and 2 w + 1 of row `lane`.
__device__ __forceinline__ void load_packed(uint32_t t0, uint32_t t1, float sites, float cap,
                                            uint32_t (&v)[kHalfWords]) {
#pragma unroll
  for (uint32_t g = 0; g < 7; ++g) {
    const uint32_t t = g < 4 ? t0 + 32 * g : t1 + 32 * (g - 4);
    uint32_t d[16], e[16];
    tmem_ld16(t, d);
    tmem_ld16(t + 16, e);
    tmem_ld_wait();
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
      v[16 * g + k] = pack2(d[2 * k], d[2 * k + 1], sites, cap);
      v[16 * g + 8 + k] = pack2(e[2 * k], e[2 * k + 1], sites, cap);
    }
  }
  uint32_t d[16], e[8];
  tmem_ld16(t1 + 96, d);
  tmem_ld8(t1 + 112, e);
  tmem_ld_wait();
#pragma unroll
  for (uint32_t k = 0; k < 8; ++k) v[112 + k] = pack2(d[2 * k], d[2 * k + 1], sites, cap);
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) v[120 + k] = pack2(e[2 * k], e[2 * k + 1], sites, cap);
}

// Rows i0 .. i0 + rows - 1 x columns j0 .. j0 + cols - 1 (cols <= 28) from the
// warp's piece (row r's 16-bit values from word 15 r), row by row: lane l
// stores column j0 + l of row i0 + r, lower-triangle entry tri(i0 + r) + j0 +
// l = e0 + r i0 + r (r - 1) / 2, where it is below the diagonal. Eight rows
// are read before they are stored: the compiler cannot tell the output from
// the piece, and one row at a time waits for shared memory 32 times over (27 k
// cycles for an item's 248 columns).
template <typename T>
__device__ __forceinline__ void store_piece(T *out, unsigned long long e0, uint32_t i0,
                                            uint32_t rows, uint32_t j0, uint32_t cols,
                                            const uint32_t *buf, uint32_t lane) {
  // lanes past the columns read a column that is there (the piece has 30)
  const uint16_t *h = reinterpret_cast<const uint16_t *>(buf) + (lane < cols ? lane : 0u);
  // bit r: row i0 + r has column j0 + lane (rows first .. rows - 1)
  const uint32_t first = j0 + lane < i0 ? 0u : j0 + lane + 1 - i0;
  uint32_t on = rows >= 32 ? 0xffffffffu : (1u << rows) - 1u;
  on = first < 32 ? on & (0xffffffffu << first) : 0u;
  if (lane >= cols) on = 0;
  T *o = out + e0;
#pragma unroll
  for (uint32_t r0 = 0; r0 < 32; r0 += 8) {
    T x[8];
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) x[k] = (T)h[2 * kPiecePitch * (r0 + k)];
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
      if (on & (1u << (r0 + k))) *o = x[k];
      o += i0 + r0 + k;  // tri(i + 1) - tri(i) = i
    }
  }
}

// The packed columns of one epilogue warp (rows i0 .., columns j0 .. j0 + 247,
// those below col_end) to the output.
template <typename T>
__device__ __forceinline__ void store_packed(const MmaJob &job, uint32_t i0, uint32_t j0,
                                             uint32_t col_end, const uint32_t (&v)[kHalfWords],
                                             uint32_t lane, uint32_t *buf) {
  const uint32_t rows = job.row_hi - i0 < 32u ? job.row_hi - i0 : 32u;
  T *out = static_cast<T *>(job.out);
  const unsigned long long t0 = (unsigned long long)i0 * (i0 - 1) / 2 - job.out_base + lane;
#pragma unroll
  for (uint32_t q = 0; q * kPieceWords < kHalfWords; ++q) {
    constexpr uint32_t kAll = kHalfWords;
    const uint32_t j = j0 + 2 * kPieceWords * q;
    // no row reaches column j, or the item ends before it (warp-uniform)
    if (j >= col_end || j + 1 >= i0 + rows) break;
    const uint32_t words = kAll - q * kPieceWords < kPieceWords ? kAll - q * kPieceWords : kPieceWords;
    const uint32_t cols = col_end - j < 2 * words ? col_end - j : 2 * words;
    __syncwarp();  // the previous piece has been read
#pragma unroll
    for (uint32_t w = 0; w < words; ++w) buf[lane * kPiecePitch + w] = v[q * kPieceWords + w];
    __syncwarp();
    store_piece<T>(out, t0 + j, i0, rows, j, cols, buf, lane);
  }
}

// 32-bit outputs: 8 columns at a time straight from the accumulators, four
// rows per store.
__device__ __forceinline__ void store_wide(const MmaJob &job, uint32_t t_lo, uint32_t t_hi, uint32_t i0,
                                           uint32_t j0, uint32_t col_end, uint32_t lane,
                                           uint32_t *buf) {
  const uint32_t rows = job.row_hi - i0 < 32u ? job.row_hi - i0 : 32u;
  uint32_t *out = static_cast<uint32_t *>(job.out);
  const unsigned long long t0 = (unsigned long long)i0 * (i0 - 1) / 2 - job.out_base;
#pragma unroll 1
  for (uint32_t c = 0; c < kHalfCols; c += 8) {
    const uint32_t j = j0 + c;
    if (j >= col_end || j + 1 >= i0 + rows) break;  // warp-uniform
    uint32_t d[8];
    tmem_ld8(c < kN0 / 2 ? t_lo + c : t_hi + (c - kN0 / 2), d);
    tmem_ld_wait();
    __syncwarp();
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
      const uint32_t mism = job.sites - (uint32_t)__uint_as_float(d[k]);
      buf[lane * 9 + k] = mism < job.max_dist ? mism : job.max_dist;
    }
    __syncwarp();
    const uint32_t k = lane & 7u;
#pragma unroll
    for (uint32_t r = lane >> 3; r < 32; r += 4)
      if (r < rows && j + k < col_end && j + k < i0 + r)
        out[t0 + j + k + (unsigned long long)r * i0 + r * (r - 1) / 2] = buf[r * 9 + k];
  }
}
static_assert(32 * 9 <= 32 * kPiecePitch, "the wide piece fits the warp's buffer");

// Sites of a job in the chunks [c_lo, c_hi).
__device__ __forceinline__ uint32_t sites_in(const MmaJob &job, uint32_t c_lo, uint32_t c_hi) {
  const uint32_t hi = c_hi * kChunkSites, lo = c_lo * kChunkSites;
  return (hi < job.sites ? hi : job.sites) - (lo < job.sites ? lo : job.sites);
}
// K blocks of the chunks [c_lo, c_hi): P per chunk, then the dash products of
// the listed ones.
__device__ __forceinline__ uint32_t blocks_in(const MmaJob &job, uint32_t c_lo, uint32_t c_hi) {
  const uint32_t d = job.dash_rank[c_hi] - job.dash_rank[c_lo];
  return job.planes * (c_hi - c_lo) + (job.planes == 6 ? 2 * d : d);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kMmaThreads, 1)
    k_pairwise_mma(const CUtensorMap *__restrict__ tms, const MmaJob *__restrict__ jobs,
                   uint32_t n_jobs, const MmaItem *__restrict__ items, uint32_t n_items,
                   unsigned *__restrict__ counter, uint32_t queue, uint32_t *__restrict__ ws,
                   unsigned long long *macs, int *status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full[kMmaStages], empty[kMmaStages], done, tmem_free, fin;
  __shared__ __align__(8) uint64_t item_full[kItemRing], item_empty[kItemRing];
  __shared__ uint32_t s_item[kItemRing];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  const uint32_t smem = (smem_u32(smem_raw) + 127u) & ~127u;
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_rank(), unit = blockIdx.x >> 1, units = gridDim.x >> 1;
  if (tid == 0) {
    for (int s = 0; s < kMmaStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int r = 0; r < kItemRing; ++r) {
      mbar_init(&item_full[r], 1);
      mbar_init(&item_empty[r], kRingReaders);
    }
    mbar_init(&done, 1);
    mbar_init(&tmem_free, 2 * kEpiWarps);
    mbar_init(&fin, 1);
    fence_mbar_init();
    s_abort = 0;
  }
  if (warp == 0) {
    tmem_alloc(&s_tmem, kTmemCols);
    tmem_relinquish();
  }
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  const uint32_t tmem = s_tmem;
  // the unit scale factors, once per CTA: warps 2-5 cover the lane quarters
  if (warp >= 2 && warp < 6) write_unit_scales<16>(tmem + (((warp & 3u) * 32) << 16), kSfColA);
  tc_before_sync();
  __syncthreads();
  cluster_sync();  // both CTAs' barriers and scale factors are ready
  tc_after_sync();

  const uint32_t full0 = smem_u32(&full[0]), empty0 = smem_u32(&empty[0]);
  const uint32_t ring_full0 = smem_u32(&item_full[0]);
  // barriers of the first CTA, where both CTAs' threads arrive
  const uint32_t lead_full0 = map_rank(full0, 0);
  const uint32_t lead_ring_empty0 = map_rank(smem_u32(&item_empty[0]), 0);
  if (warp == 0 || warp == 2 + kEpiWarps) {
    if (lane == 0) {
      // producers: load their CTA's share of every K block of this pair's
      // items, taking the blocks in turn (a block costs one thread about 460
      // cycles of waits and issues; its MMAs last 497).
      // Static order: items unit, unit + units, ...; every warp walks them by
      // itself. With `queue`, item `unit` and then the launch's counter: the
      // first CTA's first producer hands each index to all other warps.
      const uint32_t peer_item0 = map_rank(smem_u32(&s_item[0]), 1);
      const uint32_t peer_ring_full0 = map_rank(ring_full0, 1);
      const bool fills = rank == 0 && warp == 0;  // the ring
      uint32_t turn = warp == 0 ? 0u : 1u;        // blocks until this thread's next one
      uint32_t s = 0, ph = 1;  // stage, and the parity its empty barrier is waited for
      bool ok = true;
      for (uint32_t k = 0; ok; ++k) {
        const uint32_t r = k % kItemRing;
        uint32_t t = unit + k * units;
        if (queue && fills) {
          if (k >= (uint32_t)kItemRing &&
              !mbar_wait<true>(smem_u32(&item_empty[r]), ((k / kItemRing) - 1) & 1u, 4 * kMmaWaitNs)) {
            ok = false;
            break;
          }
          if (k) t = units + atomicAdd(counter, 1u);
          if (t >= n_items || *(volatile int *)&s_abort) t = kNoItem;
          *(volatile uint32_t *)&s_item[r] = t;
          asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer_item0 + 4 * r), "r"(t) : "memory");
          mbar_arrive_cluster(peer_ring_full0 + 8 * r);  // releases the index
          mbar_arrive_cluster(map_rank(ring_full0 + 8 * r, 0));
        } else if (queue) {
          if (!mbar_wait<true>(ring_full0 + 8 * r, (k / kItemRing) & 1u, 4 * kMmaWaitNs)) {
            ok = false;
            break;
          }
          t = *(volatile uint32_t *)&s_item[r];
          mbar_arrive_cluster(lead_ring_empty0 + 8 * r);
        }
        if (t >= n_items) break;
        const MmaItem it = items[t];
        if (it.job == kNoItem) break;
        // boxes of one block of 128 rows, and of 248 for both MMAs' columns
        const bool second = it.n1_16 != 0;
        const CUtensorMap *ta = tms + 2 * it.job, *tb = ta + (second ? 1 : 0);
        prefetch_tmap(ta);
        prefetch_tmap(tb);
        // row groups of this CTA's 128 rows, and of its half of the columns
        const int32_t ya = (int32_t)(it.row0 / 8 + rank * (kTM / 8));
        const int32_t yb = (int32_t)(it.col0 / 8 + rank * (it.n0_16 + it.n1_16));
        const uint32_t bytes = 2 * (kABytes + (second ? kBBytes : kB0Bytes));
        auto issue = [&](int32_t xa, int32_t xb) {
          if (turn == 0) {
            if (!mbar_wait(empty0 + 8 * s, ph, kMmaWaitNs)) return false;
            if (rank == 0) mbar_expect(full0 + 8 * s, bytes);
            const uint32_t st = smem + s * kStageBytes, bar = lead_full0 + 8 * s;
            tma_load_pair(st, ta, xa, ya, bar);
            tma_load_pair(st + kABytes, tb, xb, yb, bar);
            turn = kProducers;
          }
          --turn;
          if (++s == (uint32_t)kMmaStages) {
            s = 0;
            ph ^= 1u;
          }
          return true;
        };
        // K order: the P plane blocks of every chunk, then the dash products
        // of the listed chunks (the rows' +1 block against the columns'
        // -(P - 1) block; for P = 6 the +1 block twice, against -4 and -1).
        // Coordinates count 8-byte elements: a block is 96 of them.
        const uint32_t P = it.planes, NB = op_blocks(P);
        int32_t x = (int32_t)(it.c_lo * NB * kBlockK);
        for (uint32_t c = it.c_lo; ok && c < it.c_hi; ++c, x += (int32_t)((NB - P) * kBlockK))
          for (uint32_t p = 0; p < P; ++p, x += (int32_t)kBlockK)
            if (!issue(x, x)) {
              ok = false;
              break;
            }
        const MmaJob &job = jobs[it.job];
        const uint32_t d_hi = job.dash_rank[it.c_hi];
        for (uint32_t d = job.dash_rank[it.c_lo]; ok && d < d_hi; ++d) {
          const int32_t xd = (int32_t)((job.dash_list[d] * NB + P) * kBlockK);
          ok = issue(xd, xd + (int32_t)kBlockK);
          if (ok && P == 6) ok = issue(xd, xd + 2 * (int32_t)kBlockK);
        }
      }
      if (!ok) {
        atomicExch(&s_abort, 1);
        atomicExch(status, kStatusTmaTimeout);
        // the copies in flight land (microseconds) before the CTA may leave
        const uint64_t t0 = global_ns();
        while (global_ns() - t0 < 10000000ull) {
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // MMA issuer of the pair: the whole warp walks the loop, so that the
      // descriptors stay in uniform registers, and one elected lane issues
      const bool lead = elect_one();
      uint32_t s = 0, ph = 0;
      const uint64_t desc0 = core_desc(smem);
      uint64_t desc = desc0;
      bool ok = true;
      for (uint32_t k = 0; ok; ++k) {
        uint32_t t = unit + k * units;
        if (queue) {
          const uint32_t r = k % kItemRing;
          if (!mbar_wait<true>(ring_full0 + 8 * r, (k / kItemRing) & 1u, 4 * kMmaWaitNs)) {
            ok = false;
            break;
          }
          t = __shfl_sync(0xffffffffu, *(volatile uint32_t *)&s_item[r], 0);
          if (lead) mbar_arrive_cluster(lead_ring_empty0 + 8 * r);
        }
        if (t >= n_items) break;
        const MmaItem it = items[t];
        if (it.job == kNoItem) break;
        const uint32_t nkb = __shfl_sync(0xffffffffu, blocks_in(jobs[it.job], it.c_lo, it.c_hi), 0);
        const uint32_t n0 = __shfl_sync(0xffffffffu, it.n0(), 0);
        const uint32_t n1 = __shfl_sync(0xffffffffu, it.n1(), 0);
        const uint32_t id0 = idesc_mxf4(n0), id1 = idesc_mxf4(n1);
        // both CTAs' epilogues have read the previous item's accumulators
        if (k > 0 && !mbar_wait(smem_u32(&tmem_free), (k - 1) & 1u, kMmaWaitNs)) {
          ok = false;
          break;
        }
        tc_after_sync();
        for (uint32_t kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(full0 + 8 * s, ph, kMmaWaitNs)) {
            ok = false;
            break;
          }
          tc_after_sync();
          if (lead) {
            if (n1) mma_block<true>(tmem, desc, id0, id1, kb != 0);
            else mma_block<false>(tmem, desc, id0, id1, kb != 0);
            mma_commit(empty0 + 8 * s);
          }
          __syncwarp();
          desc += kStageBytes >> 4;
          if (++s == (uint32_t)kMmaStages) {
            s = 0;
            ph ^= 1u;
            desc = desc0;
          }
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (lead) mma_commit(smem_u32(&done));
      }
      if (lead) {
        if (!ok) {
          atomicExch(&s_abort, 1);
          atomicExch(status, kStatusTmaTimeout);
          mma_commit(smem_u32(&done));  // releases the epilogues waiting for this item
        }
        // every MMA of this thread has completed before TMEM is freed
        mma_commit(smem_u32(&fin));
        mbar_wait(smem_u32(&fin), 0, 4 * kMmaWaitNs);
      }
    } else if (unit == 0) {
      // the launch's multiply-adds (pairs x 192 values per K block)
      for (uint32_t q = lane; q < n_jobs; q += 32)
        atomicAdd(macs, jobs[q].pairs * (unsigned long long)kChunkSites *
                            blocks_in(jobs[q], 0, jobs[q].chunks));
    }
  } else {
    // epilogue warps 2 .. 9: warp w reads TMEM lanes 32 (w % 4) .. + 31, which
    // are rows 32 (w % 4) + lane of the CTA's 128, in the columns that the
    // first (w < 6) or the second CTA brings: `cols` of them, up to 128 in the
    // first MMA's accumulators and the rest in the second's
    const uint32_t sub = warp & 3u, half = warp < 6 ? 0u : 1u;
    const uint32_t t_lane = tmem + ((sub * 32) << 16);
    const uint32_t lead_free = map_rank(smem_u32(&tmem_free), 0);
    uint32_t *buf = reinterpret_cast<uint32_t *>(smem_raw + (smem - smem_u32(smem_raw)) +
                                                 kMmaStages * kStageBytes) +
                    (warp - 2) * 32 * kPiecePitch;
    for (uint32_t k = 0;; ++k) {
      uint32_t t = unit + k * units;
      bool got = true;
      if (queue) {
        // lane 0 waits and reads the index; the warp takes its answer
        const uint32_t r = k % kItemRing;
        if (lane == 0) {
          got = mbar_wait<true>(ring_full0 + 8 * r, (k / kItemRing) & 1u, 4 * kMmaWaitNs);
          if (got) {
            t = *(volatile uint32_t *)&s_item[r];
            mbar_arrive_cluster(lead_ring_empty0 + 8 * r);
          }
        }
        got = __shfl_sync(0xffffffffu, got ? 1u : 0u, 0) != 0;
        t = __shfl_sync(0xffffffffu, t, 0);
        if (!got) {
          atomicExch(&s_abort, 1);
          atomicExch(status, kStatusTmaTimeout);
        }
      }
      if (t >= n_items) break;
      const MmaItem it = items[t];
      if (it.job == kNoItem) break;
      const MmaJob &job = jobs[it.job];
      got = mbar_wait(smem_u32(&done), k & 1u, 4 * kMmaWaitNs);
      if (!got) {
        atomicExch(&s_abort, 1);
        atomicExch(status, kStatusTmaTimeout);
      }
      // one decision per warp: tcgen05.ld needs the whole warp
      if (__any_sync(0xffffffffu, !got || *(volatile int *)&s_abort)) break;
      tc_after_sync();
      const uint32_t cols = (it.n0() + it.n1()) / 2;
      const uint32_t i0 = it.row0 + rank * kTM + sub * 32, j0 = it.col0 + half * cols;
      const uint32_t col_end = j0 + cols;
      const uint32_t t0 = t_lane + half * (it.n0() / 2), t1 = t_lane + kN0 + half * (it.n1() / 2);
      // nothing below the diagonal, or past the rows or columns (warp-uniform)
      const bool any = i0 < job.row_hi && j0 < col_end && j0 + 1 < i0 + 32;
      if (job.dtype == 4) {
        if (any) store_wide(job, t0, t1, i0, j0, col_end, lane, buf);
        tc_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(lead_free);
        continue;
      }
      uint32_t v[kHalfWords];
      if (any) {
        const uint32_t top = it.slot != kNoSlot ? 65535u : job.max_dist;
        load_packed(t0, t1, (float)sites_in(job, it.c_lo, it.c_hi), (float)top, v);
      }
      // the accumulators may be overwritten
      tc_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(lead_free);
      if (!any) continue;
      if (it.slot != kNoSlot) {
        uint32_t *w = ws + (((uint64_t)it.slot * 2 + rank) * 8 + half * 4 + sub) * kHalfWords * 32 + lane;
#pragma unroll
        for (uint32_t q = 0; q < kHalfWords; ++q) w[32 * q] = v[q];
      } else if (job.dtype == 1) {
        store_packed<uint8_t>(job, i0, j0, col_end, v, lane, buf);
      } else {
        store_packed<uint16_t>(job, i0, j0, col_end, v, lane, buf);
      }
    }
  }
  tc_before_sync();
  __syncthreads();
  // neither CTA leaves while the other may still signal it or read its operands
  cluster_sync_relaxed();
  tc_after_sync();
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tmem, kTmemCols);
  }
}

// The split tiles: each warp adds one piece (32 rows x 28 columns) of a tile
// over the tile's K pieces, saturating at 65,535 (the results saturate at
// max_dist <= 65,535 anyway), and stores it as the epilogue does. The
// workspace was written just before and is read from L2.
constexpr uint32_t kFixPieces = (kHalfWords + kPieceWords - 1) / kPieceWords;  // per 248 columns
constexpr uint32_t kFixWarps = 2 * 8 * kFixPieces;                             // per tile
constexpr uint32_t kLastWords = kHalfWords - (kFixPieces - 1) * kPieceWords;     // the last piece's
__global__ void __launch_bounds__(256)
    k_pair_fix(const MmaJob *__restrict__ jobs, const MmaFix *__restrict__ fix, uint32_t n_fix,
               const uint32_t *__restrict__ ws) {
  __shared__ uint32_t s_buf[8][32 * kPiecePitch];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t id = blockIdx.x * 8 + warp;
  if (id >= n_fix * kFixWarps) return;
  const MmaFix f = fix[id / kFixWarps];
  const MmaJob &job = jobs[f.job];
  const uint32_t q = id % kFixPieces, part = id / kFixPieces % 16;  // (rank, half, quarter)
  const uint32_t i0 = f.row0 + (part >> 3) * kTM + (part & 3u) * 32;
  const uint32_t half = (part >> 2 & 1u) * (f.cols / 2), end = f.col0 + half + f.cols / 2;
  const uint32_t j = f.col0 + half + 2 * kPieceWords * q;
  if (i0 >= job.row_hi) return;
  const uint32_t rows = job.row_hi - i0 < 32u ? job.row_hi - i0 : 32u;
  if (j >= end || j + 1 >= i0 + rows) return;
  const uint32_t words = kHalfWords - q * kPieceWords < kPieceWords ? kHalfWords - q * kPieceWords
                                                                    : kPieceWords;
  uint32_t v[kPieceWords];
#pragma unroll
  for (uint32_t w = 0; w < kPieceWords; ++w) v[w] = 0;
  const uint32_t *src = ws + (((uint64_t)f.slot * 16 + part) * kHalfWords + q * kPieceWords) * 32 + lane;
  // the last piece's missing words repeat its last one (they are not stored),
  // so that the loads of four parts go out together
  auto add = [&](auto parts) {
    constexpr uint32_t U = decltype(parts)::value;
    uint32_t x[U][kPieceWords];
#pragma unroll
    for (uint32_t u = 0; u < U; ++u)
#pragma unroll
      for (uint32_t w = 0; w < kPieceWords; ++w)
        x[u][w] = __ldcg(src + u * (kSlotBytes / 4) + 32 * (w < kLastWords ? w : min(w, words - 1)));
#pragma unroll
    for (uint32_t u = 0; u < U; ++u)
#pragma unroll
      for (uint32_t w = 0; w < kPieceWords; ++w) v[w] = __vaddus2(v[w], x[u][w]);
    src += U * (kSlotBytes / 4);
  };
  uint32_t p = 0;
  for (; p + 4 <= f.parts; p += 4) add(std::integral_constant<uint32_t, 4>());
  for (; p < f.parts; ++p) add(std::integral_constant<uint32_t, 1>());
  const uint32_t cap = job.max_dist * 0x10001u;
  uint32_t *buf = s_buf[warp];
#pragma unroll
  for (uint32_t w = 0; w < kPieceWords; ++w) buf[lane * kPiecePitch + w] = __vminu2(v[w], cap);
  __syncwarp();
  const uint32_t cols = end - j < 2 * words ? end - j : 2 * words;
  const unsigned long long e0 = (unsigned long long)i0 * (i0 - 1) / 2 - job.out_base + lane + j;
  if (job.dtype == 1)
    store_piece<uint8_t>(static_cast<uint8_t *>(job.out), e0, i0, rows, j, cols, buf, lane);
  else
    store_piece<uint16_t>(static_cast<uint16_t *>(job.out), e0, i0, rows, j, cols, buf, lane);
}

// FP4 (kind::mxf4) MMA rate from shared memory alone (no loads): CTA pairs
// issue `rounds` K blocks of the engine's own MMAs (M = 256, N = 256 and 240,
// K = 96) on zeroed stages (the values do not change the rate).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(128, 1)
    k_peak_mma(uint32_t rounds, int *status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t s_tmem;
  const uint32_t smem = (smem_u32(smem_raw) + 127u) & ~127u;
  uint8_t *stage = smem_raw + (smem - smem_u32(smem_raw));
  for (uint32_t k = threadIdx.x; k < kStageBytes / 16; k += blockDim.x)
    reinterpret_cast<uint4 *>(stage)[k] = make_uint4(0, 0, 0, 0);
  // the generic-proxy writes above, before the tensor cores read them
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  if (threadIdx.x < 32) {
    tmem_alloc(&s_tmem, kTmemCols);
    tmem_relinquish();
  }
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  const uint32_t tmem = s_tmem;
  write_unit_scales<16>(tmem + (((threadIdx.x >> 5) * 32) << 16), kSfColA);
  tc_before_sync();
  __syncthreads();
  cluster_sync();
  tc_after_sync();
  if (threadIdx.x == 0) {
    if (cluster_rank() == 0) {
      const uint64_t desc = core_desc(smem);
      for (uint32_t r = 0; r < rounds; ++r)
        mma_block<true>(tmem, desc, idesc_mxf4(kN0), idesc_mxf4(kN1), r != 0);
      mma_commit(smem_u32(&bar));
    }
    if (!mbar_wait(smem_u32(&bar), 0, 4 * kMmaWaitNs)) atomicExch(status, kStatusTmaTimeout);
  }
  tc_before_sync();
  __syncthreads();
  cluster_sync();
  tc_after_sync();
  if (threadIdx.x < 32) {
    __syncwarp();
    tmem_dealloc(tmem, kTmemCols);
  }
}

// The list of the marked chunks (a block for each of `jobs`, or one for `one`)
__global__ void __launch_bounds__(512) k_dash_list(OpRows one, const OpRows *__restrict__ jobs) {
  __shared__ uint32_t tmp[33];
  const OpRows o = jobs ? jobs[blockIdx.x] : one;
  list_marked(o, tmp);
}

void set_smem_once(int device) {
  static OncePerDevice once;
  once.run(device, [] {
    HD_CUDA(cudaFuncSetAttribute(k_pairwise_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, kMmaSmem));
  });
}

// Map of an operand's row groups: boxes of one block of `box_rows` rows.
void make_tmap_op(hd_ctx *ctx, CUtensorMap *tm, const void *base, uint32_t planes, uint64_t sites,
                  uint64_t rows, uint32_t box_rows) {
  const uint64_t group = op_group_bytes(planes, sites);
  cuuint64_t dims[2] = {group / 8, ceil_div(rows, (uint64_t)8)};
  cuuint64_t strides[1] = {group};
  cuuint32_t box[2] = {kGroupBytes / 8, box_rows / 8};
  cuuint32_t es[2] = {1, 1};
  CUresult r = ctx->encode_tiled(tm, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, const_cast<void *>(base),
                                 dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                 CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    fail(HD_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
}

// uint32s of the marks and the block count, and of the list and ranks made of them
uint64_t mark_words(uint64_t sites) { return (uint64_t)op_chunks(sites) + 1; }
uint64_t list_words(uint64_t sites) { return 2 * (uint64_t)op_chunks(sites) + 1; }

// The list of the extension's marked chunks, and their dash blocks if they are
// not written: launches
uint64_t list_chunks(const OpRows &o, int sm_count, cudaStream_t stream) {
  k_dash_list<<<1, 512, 0, stream>>>(o, nullptr);
  if (!o.blocks) return 1;
  const uint64_t work = ceil_div(ceil_div((uint64_t)o.row_hi, (uint64_t)8), (uint64_t)kDashGroups) *
                        op_chunks(o.sites);
  k_dash_blocks<<<(unsigned)std::min<uint64_t>(work, (uint64_t)sm_count * 8),
                  kDashGroups * 8 * kChunkWords, 0, stream>>>(o, nullptr, 1);
  return 2;
}

// The operand's rows and its last list are written by what is queued on the
// stream so far: other streams wait for that.
void mark_operand(hd_ctx *ctx, const hd_alignment *o, cudaStream_t stream,
                  std::shared_ptr<StreamMark> &mark) {
  if (!mark) {
    mark = stream == ctx->stream ? ctx->op_mark : nullptr;
    if (!mark) {
      mark = std::make_shared<StreamMark>();
      HD_CUDA(cudaEventCreateWithFlags(&mark->ev, cudaEventDisableTiming));
      if (stream == ctx->stream) ctx->op_mark = mark;
    }
    HD_CUDA(cudaEventRecord(mark->ev, stream));
  }
  o->op_mark = mark;
  o->op_stream = stream;
}
// The stream's next work follows what wrote the operand.
void follow_operand(const hd_alignment *o, cudaStream_t stream) {
  if (o->op_mark && o->op_stream != stream) HD_CUDA(cudaStreamWaitEvent(stream, o->op_mark->ev, 0));
}

// A plan's extensions whose marked chunks are not listed yet, and the large ones'
// dash blocks not written: two launches for all of them. A list by each one's
// last block costs 2 us a matrix there, since the launches follow one another
// (first run of a batch of 200 matrices of 20 to 128 rows: 2.0 ms, with one
// launch for all lists 1.6, with two launches for each matrix 3.2; 50 served
// windows of 100 rows 1.63, 1.57, 1.84). Left early, each has its own launches:
// their alignments count the rows as there.
struct DashLater {
  hd_ctx *ctx;
  cudaStream_t stream;
  std::vector<OpRows> jobs;
  std::vector<const hd_alignment *> owners;  // the alignments among them
  void mark() {
    std::shared_ptr<StreamMark> at;
    for (const hd_alignment *o : owners) mark_operand(ctx, o, stream, at);
    owners.clear();
  }
  ~DashLater() {
    for (const OpRows &o : jobs) list_chunks(o, ctx->sm_count, stream);
    try {
      mark();
    } catch (const Error &) {
      cudaStreamSynchronize(stream);
    }
  }
  // d_jobs: their copy on the device
  void launch(const OpRows *d_jobs) {
    if (jobs.empty()) return;
    const unsigned n = (unsigned)jobs.size(), y = std::min(n, 65535u);
    k_dash_list<<<n, 512, 0, stream>>>(OpRows{}, d_jobs);
    HD_LAUNCHED(ctx);
    const bool blocks = std::any_of(jobs.begin(), jobs.end(), [](const OpRows &o) { return o.blocks != 0; });
    if (blocks) {
      const unsigned x = (unsigned)ceil_div((uint64_t)ctx->sm_count * 32, (uint64_t)y);
      k_dash_blocks<<<dim3(x, y), kDashGroups * 8 * kChunkWords, 0, stream>>>(OpRows{}, d_jobs, n);
      HD_LAUNCHED(ctx);
    }
    jobs.clear();
    mark();
  }
};

dim3 op_grid(uint64_t words, uint64_t lo, uint64_t hi) {
  const uint64_t groups = ceil_div(hi, (uint64_t)8) - lo / 8;
  return dim3((unsigned)ceil_div(words, (uint64_t)32),
              (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(groups, 65535)));
}

// Expands the rows and lists the chunks with a '-', now or with the plan's
// others. Where the dash blocks of all chunks are few bytes they are written with
// the others and the last block makes the list: one launch instead of three. A
// first call with 1,500 rows of 1,273 sites takes 103 us, with three launches
// 113; with 3,000 of 3,000 (9 MB) 123 and 136. On large operands the blocks'
// counting costs more than the launches (14,000 rows of 29,903 sites: 60 us).
// Rows after others go the longer way: a chunk that they mark first needs dash
// blocks of the earlier rows too.
constexpr uint64_t kDashBytes = 16ull << 20;
void expand_rows(hd_ctx *ctx, OpRows o, cudaStream_t stream, DashLater *later) {
  const uint64_t bytes = (o.row_hi - o.row_lo) * op_chunks(o.sites) * (op_blocks(o.planes) - o.planes) * kBlockK;
  o.blocks = bytes > kDashBytes || o.row_lo > 0 ? 1u : 0u;
  const bool list = !later && !o.blocks;
  (list ? k_expand_op<true> : k_expand_op<false>)<<<
      op_grid((uint64_t)op_chunks(o.sites) * kChunkWords, o.row_lo, o.row_hi), 256, 0, stream>>>(o);
  HD_LAUNCHED(ctx);
  if (later) {
    later->jobs.push_back(o);
  } else if (!list) {
    ctx->launches += list_chunks(o, ctx->sm_count, stream);
    check_cuda(cudaGetLastError(), "kernel launch");
  }
}

}  // namespace

int mma_band_of(const TileConfig &c) {
  if (const char *e = std::getenv("HAMMINGDIST_MMA_BAND")) return std::max(2, std::atoi(e)) & ~1;
  return c.mma_band > 0 ? std::max(2, c.mma_band) & ~1 : (int)kMmaBand;
}
int mma_rows_of(const TileConfig &c) {
  if (const char *e = std::getenv("HAMMINGDIST_MMA_ROWS")) return std::atoi(e) == 1 ? 1 : 2;
  return c.mma_rows == 1 ? 1 : 2;
}

bool mma_eligible(const hd_alignment *aln) {
  if (const char *e = std::getenv("HAMMINGDIST_KERNEL"))
    if (std::string(e) == "lop3") return false;
  // the AND rule (4 planes) or a sparse rule (5, 6 planes); FP32 sums of up
  // to P L are exact below 2^24
  const uint64_t P = (uint64_t)aln->planes;
  const bool shape = (P == 4 && aln->groups == 1) || ((P == 5 || P == 6) && aln->groups == 2);
  return shape && aln->length >= 1 && aln->length * P < (1ull << 24) && aln->n_rows >= 2 &&
         aln->n_rows < (1ull << 31);
}

namespace {
// Room for `rows` rows in the operand of the alignment o, and for the list of
// its next extension; false if there is no memory for it.
bool grow_operand(hd_ctx *ctx, const hd_alignment *o, uint64_t rows, cudaStream_t stream,
                  uint64_t cap_hint) {
  const uint32_t P = (uint32_t)o->planes;
  const uint64_t words = o->words;
  if (rows > o->op_cap) {
    // room for the rows asked for, or for what the caller says will come
    const uint64_t plane_rows = o->plane_buf[0].bytes / (words * 16);
    const uint64_t cap = std::max(rows, std::min(cap_hint, plane_rows));
    DevBuf grown;
    try {
      grown = DevBuf(op_bytes(P, o->length, cap), stream);
    } catch (const Error &e) {
      if (e.code != HD_ERR_OOM) throw;
      cudaGetLastError();
      return false;  // the bit-plane engine needs no extra memory
    }
    if (o->op_rows) {
      HD_CUDA(cudaMemcpyAsync(grown.p, o->op.p, op_bytes(P, o->length, o->op_rows),
                              cudaMemcpyDeviceToDevice, stream));
      // launches on the context's other streams may still read the old
      // operand: they finish before it is freed
      for (cudaStream_t st : {ctx->side, ctx->stream}) HD_CUDA(cudaStreamSynchronize(st));
    }
    o->op = std::move(grown);
    o->op_cap = cap;
  }
  // a list of its own for every extension (the first one's after the marks):
  // launches on other streams may still read an earlier one
  if (!o->op_dash.p) {
    const uint64_t marks = mark_words(o->length);
    o->op_dash = DevBuf((marks + list_words(o->length)) * 4, stream);
    HD_CUDA(cudaMemsetAsync(o->op_dash.p, 0, marks * 4, stream));
  } else {
    o->op_lists.emplace_back(list_words(o->length) * 4, stream);
  }
  return true;
}
// The list of the operand's last extension
uint32_t *last_list(const hd_alignment *o) {
  return o->op_lists.empty() ? o->op_dash.as<uint32_t>() + mark_words(o->length)
                             : o->op_lists.back().as<uint32_t>();
}
// The extension to rows [op_rows, rows) that grow_operand made room for
OpRows extension_of(const hd_alignment *o, uint64_t rows) {
  OpRows j{};
  j.g0 = o->plane_buf[0].as<uint4>();
  j.g1 = o->planes > 4 ? o->plane_buf[1].as<uint4>() : nullptr;
  j.x = o->op.as<uint8_t>();
  j.marks = o->op_dash.as<uint32_t>();
  j.list = last_list(o);
  j.row_lo = o->op_rows;
  j.row_hi = rows;
  j.sites = o->length;
  j.planes = (uint32_t)o->planes;
  j.words = (uint32_t)o->words;
  j.ext = (uint32_t)o->op_lists.size() + 1;
  j.blocks = 1;
  return j;
}
bool extend_operand(hd_ctx *ctx, const hd_alignment *o, uint64_t rows, cudaStream_t stream,
                    uint64_t cap_hint, DashLater *later) {
  std::lock_guard<std::recursive_mutex> lk(o->lazy);
  follow_operand(o, stream);
  if (o->op_rows >= rows) return true;
  if (!grow_operand(ctx, o, rows, stream, cap_hint)) return false;
  expand_rows(ctx, extension_of(o, rows), stream, later);
  o->op_rows = rows;
  std::shared_ptr<StreamMark> mark;
  if (later) later->owners.push_back(o);
  else mark_operand(ctx, o, stream, mark);
  return true;
}
}  // namespace

bool ensure_operand(hd_ctx *ctx, const hd_alignment *aln, uint64_t rows, cudaStream_t stream,
                    uint64_t cap_hint) {
  return extend_operand(ctx, aln->base ? aln->base : aln, rows, stream, cap_hint, nullptr);
}

namespace {
// up to 8 row groups a block, while that leaves four rounds of blocks
dim3 pack_grid(hd_ctx *ctx, uint64_t words, uint64_t lo, uint64_t hi) {
  dim3 grid = op_grid(words, lo, hi);
  const uint64_t rounds = (uint64_t)grid.x * grid.y / ((uint64_t)ctx->sm_count * 6 * 4);
  grid.y = (unsigned)ceil_div(grid.y, std::min<uint64_t>(8, std::max<uint64_t>(1, rounds)));
  return grid;
}
}  // namespace

void pack_planes(hd_ctx *ctx, const Records &rec, const uint64_t *d_rows, uint64_t n_rows,
                 uint64_t length, uint64_t words, uint4 *g0, uint4 *g1, const Words *sel) {
  if (!n_rows) return;
  const Words all = Words::of((uint32_t)words, 1);
  if (!sel) sel = &all;
  k_pack_op<false><<<pack_grid(ctx, sel->count, 0, n_rows), 256, 0, ctx->stream>>>(
      rec.base, rec.bytes, rec.rec_start.as<uint64_t>(), d_rows, 0, n_rows, length,
      (uint32_t)words, g0, g1, nullptr, nullptr, 0, *sel);
  HD_LAUNCHED(ctx);
}

bool pack_operand(hd_ctx *ctx, const Records &rec, const uint64_t *d_rows, const hd_alignment *aln,
                  uint64_t lo, uint64_t hi, uint4 *copy, cudaStream_t stream, uint64_t cap_hint) {
  if (aln->base || aln->planes != 4 || aln->op_rows != lo || hi <= lo) return false;
  std::lock_guard<std::recursive_mutex> lk(aln->lazy);
  follow_operand(aln, stream);
  if (!grow_operand(ctx, aln, hi, stream, cap_hint)) return false;
  const OpRows j = extension_of(aln, hi);
  const uint64_t op_words = (uint64_t)op_chunks(aln->length) * kChunkWords;
  k_pack_op<true><<<pack_grid(ctx, std::max(aln->words, op_words), lo, hi), 256, 0, stream>>>(
      rec.base, rec.bytes, rec.rec_start.as<uint64_t>(), d_rows, lo, hi, aln->length,
      (uint32_t)aln->words, aln->plane_buf[0].as<uint4>(), copy, j.x, j.marks, j.ext,
      Words::of(0, 1));
  HD_LAUNCHED(ctx);
  ctx->launches += list_chunks(j, ctx->sm_count, stream);
  check_cuda(cudaGetLastError(), "kernel launch");
  aln->op_rows = hi;
  std::shared_ptr<StreamMark> mark;
  mark_operand(ctx, aln, stream, mark);
  return true;
}

uint64_t mma_operand_bytes(uint32_t planes, uint64_t sites, uint64_t rows) {
  return op_bytes(planes, sites, rows);
}

double measure_mma_peak(hd_ctx *ctx) {
  static OncePerDevice once;
  once.run(ctx->device, [] {
    HD_CUDA(cudaFuncSetAttribute(k_peak_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, kMmaSmem));
  });
  const uint32_t rounds = 4096, pairs = std::max(1, ctx->sm_count / 2);
  k_peak_mma<<<2 * pairs, 128, kMmaSmem, ctx->stream>>>(256, ctx->d_status);  // warm-up
  HD_LAUNCHED(ctx);
  HD_CUDA(cudaEventRecord(ctx->ev_start, ctx->stream));
  k_peak_mma<<<2 * pairs, 128, kMmaSmem, ctx->stream>>>(rounds, ctx->d_status);
  HD_LAUNCHED(ctx);
  HD_CUDA(cudaEventRecord(ctx->ev_stop, ctx->stream));
  HD_CUDA(cudaStreamSynchronize(ctx->stream));
  float ms = 0;
  HD_CUDA(cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
  const double flop = (double)pairs * rounds * 2.0 * kRowsPerItem * kItemCols * kChunkSites;
  return flop / (ms / 1e3);
}

// The E2M1 operand rows of a job: the alignment's own cache (an alignment, or
// a view at row 0 of a base whose cache already holds its rows: the streamed
// from_fasta), else the view's rows expanded into a buffer the plan keeps
// until the kernel has run (a serving window must not expand a large base).
// False if there is no memory for it.
bool operand_for(hd_ctx *ctx, const hd_alignment *a, cudaStream_t stream, PairLaunchPlan *plan,
                 const uint8_t *&op, const uint32_t *&dash, DashLater *later) {
  const hd_alignment *o = a->base ? a->base : a;
  if (!a->base) {
    if (!extend_operand(ctx, a, a->n_rows, stream, 0, later)) return false;
    std::lock_guard<std::recursive_mutex> lk(a->lazy);
    op = a->op.as<uint8_t>();
    dash = last_list(a);
    return true;
  }
  std::unique_lock<std::recursive_mutex> lk(o->lazy, std::defer_lock);
  if (a->row0 == 0) lk.lock();
  if (a->row0 == 0 && o->op.p && o->op_rows >= a->n_rows) {
    follow_operand(o, stream);
    // the base's listed chunks cover its other rows too: a chunk listed for
    // them only adds dash products of 0
    op = o->op.as<uint8_t>();
    dash = last_list(o);
    return true;
  }
  if (lk) lk.unlock();
  const uint32_t P = (uint32_t)o->planes;
  const uint64_t bytes = op_bytes(P, o->length, a->n_rows);
  const uint64_t marks = mark_words(o->length), flag_bytes = (marks + list_words(o->length)) * 4;
  if (bytes > (8ull << 30)) return false;  // the bit-plane engine needs no extra memory
  DevBuf tmp;
  try {
    tmp = DevBuf(bytes + flag_bytes, stream);
  } catch (const Error &e) {
    if (e.code != HD_ERR_OOM) throw;
    cudaGetLastError();
    return false;
  }
  uint32_t *flags = reinterpret_cast<uint32_t *>(tmp.as<uint8_t>() + bytes);
  HD_CUDA(cudaMemsetAsync(flags, 0, marks * 4, stream));
  OpRows j{};
  j.g0 = static_cast<const uint4 *>(a->planes_ptr(0));
  j.g1 = P > 4 ? static_cast<const uint4 *>(a->planes_ptr(1)) : nullptr;
  j.x = tmp.as<uint8_t>();
  j.marks = flags;
  j.list = flags + marks;
  j.row_hi = a->n_rows;
  j.sites = o->length;
  j.planes = P;
  j.words = (uint32_t)o->words;
  j.ext = 1;
  plan->blocks.push_back(std::move(tmp));
  expand_rows(ctx, j, stream, later);
  op = j.x;
  dash = j.list;
  return true;
}

namespace {

// The items of a launch and how the CTA pairs share them.
struct MmaPlan {
  // static order: pair u of `pairs` runs items u, u + pairs, ... up to the
  // padding (job kNoItem)
  std::vector<MmaItem> items;
  std::vector<MmaFix> fix;
  uint32_t slots = 0;
  uint32_t pairs = 0;  // CTA pairs with work
  // a tile's item, cut along K at the chunks `cuts` (first and last included)
  void add_pieces(const MmaItem &tile, const std::vector<uint32_t> &cuts, std::vector<MmaItem> &out) {
    if (cuts.size() <= 2) {
      out.push_back(tile);
      return;
    }
    fix.push_back({tile.job, tile.row0, tile.col0, tile.n0() + tile.n1(), slots,
                   (uint32_t)cuts.size() - 1});
    for (size_t k = 0; k + 1 < cuts.size(); ++k) {
      MmaItem it = tile;
      it.c_lo = cuts[k];
      it.c_hi = cuts[k + 1];
      it.slot = slots++;
      out.push_back(it);
    }
  }
};

// Cost of an item per K block, in units of 177 cycles (0.09 us): 531 cycles for
// both column halves; one half alone waits for its loads (24.6 KB at the 72 B
// per cycle and SM that the L2 gives), about 340.
constexpr double kCostUs = 0.09;
// What splitting costs: the pieces' workspace traffic and one more launch. Calls,
// split and whole: 1,000 rows of 2,400 sites (7.5 us of pieces' gain) 80 and 75
// us, of 3,000 (10.8) 73 and 77, of 5,000 74 and 89; 3,000 rows of 4,000 (9.0) 97
// and 86, of 5,000 (11.6) 92 and 93, of 8,000 (18) 106 and 109.
constexpr double kSplitUs = 10.0;
uint64_t block_cost(const MmaItem &it) { return it.n1_16 ? 3 : 2; }

// One matrix: every pair of CTAs gets the same share of the work to within a
// chunk. Whole items go round in list order while every pair has one more;
// the rest is dealt out in K pieces that fill each pair up to the average, unless
// that gains less than it costs: then the rest goes to the least loaded pairs.
void plan_static(std::vector<MmaItem> &list, uint32_t units, uint32_t planes, bool may_split,
                 MmaPlan &plan) {
  // The items of both column halves first: they all take the same time, so
  // that the pairs working on one band stay at the same K and read its rows
  // while the L2 holds them.
  std::stable_partition(list.begin(), list.end(), [](const MmaItem &it) { return it.n1_16 != 0; });
  const size_t m = list.size();
  auto cost_of = [&](const MmaItem &it) {
    return block_cost(it) * planes * (it.c_hi - it.c_lo);
  };
  uint64_t total = 0, most = 1;
  for (const MmaItem &it : list) {
    total += cost_of(it);
    most = std::max(most, cost_of(it));
  }
  // a pair's share: the average, at least the shortest piece of a full tile
  const uint64_t share = std::max<uint64_t>(ceil_div(total, units), 3ull * planes * kMinPart);
  const size_t whole = std::min<size_t>(m, (size_t)(total / units / most) * units);
  // items in the order that their pairs take them, and each one's pair
  std::vector<MmaItem> out;
  std::vector<uint32_t> owner;
  std::vector<uint64_t> load(units, 0);
  out.reserve(m + 2 * units);
  owner.reserve(m + 2 * units);
  for (size_t k = 0; k < whole; ++k) {
    out.push_back(list[k]);
    owner.push_back((uint32_t)(k % units));
    load[k % units] += cost_of(list[k]);
  }
  const uint64_t unsplit = (whole / units + ceil_div(m - whole, (size_t)units)) * most;
  const bool split = may_split && (double)(unsplit - std::min(unsplit, share)) * kCostUs > kSplitUs;
  if (!split) {
    // each to the least loaded pair, the first of equals
    using Load = std::pair<uint64_t, uint32_t>;
    std::priority_queue<Load, std::vector<Load>, std::greater<Load>> least;
    for (uint32_t v = 0; v < units; ++v) least.push({load[v], v});
    for (size_t k = whole; k < m; ++k) {
      const Load v = least.top();
      least.pop();
      out.push_back(list[k]);
      owner.push_back(v.second);
      least.push({v.first + cost_of(list[k]), v.second});
    }
  } else {
    // the rest as one row of chunks; pair u's end on it is the sum of the room
    // up to u, so that rounding to whole chunks does not add up
    auto room = [&](uint32_t v) { return load[v] < share ? share - load[v] : 0; };
    uint32_t u = 0;
    uint64_t at = 0, end = room(0);
    std::vector<uint32_t> cuts;
    for (size_t k = whole; k < m; ++k) {
      const MmaItem &it = list[k];
      const uint64_t per = block_cost(it) * planes;  // cost of one chunk
      cuts.assign(1, it.c_lo);
      for (uint32_t c = it.c_lo; c < it.c_hi;) {
        const uint32_t left = it.c_hi - c;
        uint64_t take = end > at ? (end - at + per / 2) / per : 0;
        if (u + 1 < units && take < kMinPart && left > take) {
          end += room(++u);  // this pair is full
          continue;
        }
        if (u + 1 == units || take > left || left - take < kMinPart) take = left;
        c += (uint32_t)take;
        at += take * per;
        cuts.push_back(c);
        owner.push_back(u);
      }
      plan.add_pieces(it, cuts, out);
    }
  }
  std::vector<uint32_t> depth(units, 0);
  for (uint32_t v : owner) ++depth[v];
  uint32_t deepest = 0;
  for (uint32_t v = 0; v < units; ++v) {
    deepest = std::max(deepest, depth[v]);
    if (depth[v]) plan.pairs = v + 1;
  }
  MmaItem none{};
  none.job = kNoItem;
  plan.items.assign((size_t)deepest * plan.pairs, none);
  std::fill(depth.begin(), depth.end(), 0u);
  for (size_t k = 0; k < out.size(); ++k)
    plan.items[(size_t)depth[owner[k]]++ * plan.pairs + owner[k]] = out[k];
}

// Several matrices: the pairs draw items from a queue, the costliest first
// (list order). Items longer than half of a pair's average share (a small
// batch) are cut along K to about that length.
void plan_queue(std::vector<MmaItem> &list, uint32_t units, const std::vector<uint32_t> &planes,
                const std::vector<char> &may_split, MmaPlan &plan) {
  uint64_t total = 0;
  for (const MmaItem &it : list)
    total += block_cost(it) * planes[it.job] * (it.c_hi - it.c_lo);
  const uint64_t half = std::max<uint64_t>(1, total / units / 2);
  for (const MmaItem &it : list) {
    const uint32_t n = it.c_hi - it.c_lo;
    const uint64_t cost = block_cost(it) * planes[it.job] * n;
    uint64_t parts = may_split[it.job] ? std::min<uint64_t>(cost / half, n / kMinPart) : 1;
    // (between 2 and 12 us this line makes no difference to a batch)
    if ((double)(cost - std::min(cost, half)) * kCostUs < kSplitUs) parts = 1;
    std::vector<uint32_t> cuts{it.c_lo};
    for (uint64_t k = 1; k <= std::max<uint64_t>(parts, 1); ++k)
      cuts.push_back(it.c_lo + (uint32_t)(n * k / std::max<uint64_t>(parts, 1)));
    plan.add_pieces(it, cuts, plan.items);
  }
  plan.pairs = (uint32_t)std::min<uint64_t>(units, plan.items.size());
}

// The item, or (halves) its column halves as items of their own.
void push_item(std::vector<MmaItem> &list, MmaItem it, bool halves) {
  if (halves && it.n1_16) {
    MmaItem first = it;
    first.n1_16 = 0;
    list.push_back(first);
    it.col0 += it.n0();
    it.n0_16 = it.n1_16;
    it.n1_16 = 0;
  }
  list.push_back(it);
}

}  // namespace

// Size of the tile rows [lo, hi) in tiles of 128 x kMmaCols pairs: what the
// launch thresholds and the reported tile counts are in.
static uint64_t size_tiles(uint64_t lo, uint64_t hi) {
  uint64_t n = 0;
  for (uint64_t I = lo; I < hi; ++I) n += ((I + 1) * kTM - 2) / kMmaCols + 1;
  return n;
}

uint64_t mma_size_tiles(uint64_t lo, uint64_t hi) {
  return size_tiles(lo / kTM, ceil_div(hi, (uint64_t)kTM));
}

bool mma_wanted(hd_ctx *ctx, const hd_alignment *aln) {
  if (ctx->engine_force == 0 || !mma_eligible(aln)) return false;
  const uint64_t min_items = ctx->engine_force == 1 ? 0 : mma_min_items_for(ctx, aln->length);
  return size_tiles(0, ceil_div(aln->n_rows, (uint64_t)kTM)) >= min_items;
}

void prepare_mma_jobs(hd_ctx *ctx, const std::vector<PairJobSpec> &specs, cudaStream_t stream,
                      PairLaunchPlan *plan, int sm_limit, std::vector<char> &taken) {
  taken.resize(specs.size(), 0);
  std::vector<const uint8_t *> ops(specs.size(), nullptr);  // each job's operand rows
  std::vector<const uint32_t *> dash_lists(specs.size(), nullptr);  // and its listed chunks
  struct Job {
    size_t k;
    uint32_t t_lo, t_hi;
    double cost;
  };
  std::vector<Job> js;
  // Rows whose lists follow with the plan's others are nobody else's to read
  // until then: their alignments stay locked (in the order of their addresses)
  std::vector<std::unique_lock<std::recursive_mutex>> locks;
  DashLater dash_later{ctx, stream, {}, {}};
  // A small launch leaves SMs idle: below a minimum size, counted in tiles of
  // 128 x kMmaCols pairs (mma_min_items_for, autotuned per row length), the
  // bit-plane engine's finer tiles finish first; a batch of small matrices
  // still goes here when together they are enough.
  if (ctx->engine_force == 0) return;
  uint64_t items_total = 0, max_len = 0;
  for (size_t k = 0; k < specs.size(); ++k) {
    const PairJobSpec &sp = specs[k];
    if (taken[k] || !mma_eligible(sp.aln) || sp.tile_hi <= sp.tile_lo) continue;
    max_len = std::max<uint64_t>(max_len, sp.aln->length);
    const uint64_t edge = sp.cfg.tile > 0 ? (uint64_t)sp.cfg.tile : kTile;
    const uint64_t lo = sp.tile_lo * edge / kTM;
    const uint64_t hi = ceil_div(std::min<uint64_t>(sp.tile_hi * edge, sp.aln->n_rows), kTM);
    items_total += size_tiles(lo, hi);
  }
  const uint64_t min_items = ctx->engine_force == 1 ? 0 : mma_min_items_for(ctx, max_len);
  if (items_total < min_items) return;
  if (specs.size() > 1) {
    std::vector<const hd_alignment *> shared;
    for (const PairJobSpec &sp : specs)
      if (!sp.aln->base || sp.aln->row0 == 0) shared.push_back(sp.aln->base ? sp.aln->base : sp.aln);
    std::sort(shared.begin(), shared.end(), std::less<const hd_alignment *>());
    shared.erase(std::unique(shared.begin(), shared.end()), shared.end());
    locks.reserve(shared.size());
    for (const hd_alignment *o : shared) locks.emplace_back(o->lazy);
  }
  for (size_t k = 0; k < specs.size(); ++k) {
    const PairJobSpec &sp = specs[k];
    const hd_alignment *a = sp.aln;
    if (taken[k] || !mma_eligible(a) || sp.tile_hi <= sp.tile_lo) continue;
    // the caller's tile rows are in units of its configuration's tile edge
    const uint64_t edge = sp.cfg.tile > 0 ? (uint64_t)sp.cfg.tile : kTile;
    const uint64_t row_lo = sp.tile_lo * edge, row_hi = std::min<uint64_t>(sp.tile_hi * edge, a->n_rows);
    if (row_lo % kTM || row_hi <= row_lo) continue;
    if (!operand_for(ctx, a, stream, plan, ops[k], dash_lists[k], specs.size() > 1 ? &dash_later : nullptr))
      continue;
    const uint32_t lo = (uint32_t)(row_lo / kTM), hi = (uint32_t)ceil_div(row_hi, kTM);
    js.push_back({k, lo, hi, (double)a->words * ((double)hi * hi - (double)lo * lo)});
    taken[k] = 1;
  }
  if (js.empty()) return;
  // Each job's K blocks: the P plane blocks of every chunk, and the dash
  // products of the chunks its rows have a '-' in, whose list stays on the
  // device (k_dash_list); the host orders the jobs by the plane blocks.
  auto owner_of = [&](const Job &j) {
    const hd_alignment *a = specs[j.k].aln;
    return a->base ? a->base : a;
  };
  auto kcost = [&](const Job &j) {
    const hd_alignment *o = owner_of(j);
    return (uint64_t)o->planes * op_chunks(o->length);
  };
  // the costliest items first (an item's cost is its K length), biggest jobs
  // first among equals, so that the cheap items fill the tail
  std::stable_sort(js.begin(), js.end(), [&](const Job &a, const Job &b) {
    return kcost(a) != kcost(b) ? kcost(a) > kcost(b) : a.cost > b.cost;
  });
  // Items of each job: 256 rows x 496 columns (with mma_rows 1, each column
  // half by itself) up to the last column any of their rows needs, in bands of
  // mma_band tile rows, column-major within a band. Near the diagonal an item
  // is as wide as its rows need, in the 16 columns an MMA's N counts in.
  const size_t nj = js.size();
  std::vector<MmaItem> list;
  std::vector<uint32_t> planes(nj);
  std::vector<char> may_split(nj);
  for (uint32_t q = 0; q < (uint32_t)nj; ++q) {
    const PairJobSpec &sp = specs[js[q].k];
    const hd_alignment *o = owner_of(js[q]);
    planes[q] = (uint32_t)o->planes;
    const uint32_t chunks = op_chunks(o->length);
    may_split[q] = sp.dtype <= 2 && chunks >= 2 * kMinPart;
    const uint32_t band = (uint32_t)mma_band_of(sp.cfg) * kRowsPerItem;
    const bool halves = mma_rows_of(sp.cfg) == 1;
    const uint32_t lo = js[q].t_lo * kTM;
    const uint32_t hi = (uint32_t)std::min<uint64_t>((uint64_t)js[q].t_hi * kTM, sp.aln->n_rows);
    for (uint32_t b = lo; b < hi; b += band) {
      const uint32_t e = std::min(b + band, hi);
      for (uint32_t col = 0; col + 1 < e; col += kItemCols)
        for (uint32_t r = b; r < e; r += kRowsPerItem) {
          const uint32_t last = std::min(r + kRowsPerItem, e);  // rows [r, last) need columns < last - 1
          if (col + 1 >= last) continue;
          const uint32_t need = (uint32_t)round_up(std::min(last - 1 - col, kItemCols), 16);
          const uint32_t n0 = std::min(need, kN0), n1 = need - n0;
          MmaItem it{q, r, col, (uint8_t)(n0 / 16), (uint8_t)(n1 / 16), (uint8_t)planes[q], 0, 0,
                     chunks, kNoSlot, 0};
          push_item(list, it, halves);
        }
    }
  }
  // HAMMINGDIST_MMA_SCHEDULE=static|queue picks one for every launch (several
  // matrices always go through the queue)
  const int sms = sm_limit > 0 && sm_limit < ctx->sm_count ? sm_limit : ctx->sm_count;
  const uint32_t units = (uint32_t)std::max(1, sms / 2);
  // 32-bit outputs are not split along K: where two thirds of an item's time
  // for twice the items leave every pair one at most, they are cut into column
  // halves (a call with 1,000 rows of 29,903 sites 233 -> 177 us)
  if (nj == 1 && specs[js[0].k].dtype == 4 && 2 * list.size() <= units) {
    std::vector<MmaItem> cut;
    for (const MmaItem &it : list) push_item(cut, it, true);
    list.swap(cut);
  }
  bool queue = nj > 1;
  if (const char *e = std::getenv("HAMMINGDIST_MMA_SCHEDULE"))
    queue = queue || std::string(e) == "queue";
  // the pieces' workspace: the context's for this stream, else the plan's own.
  // (Allocated for each launch on the side stream, it held a streamed call up
  // for 0.7 ms.)
  MmaPlan mp;
  DevBuf own;
  DevBuf *ws = plan->replayed ? &own : stream == ctx->stream ? &ctx->mma_ws[0]
               : stream == ctx->side ? &ctx->mma_ws[1] : &own;
  for (;;) {
    if (queue) plan_queue(list, units, planes, may_split, mp);
    else plan_static(list, units, planes[0], may_split[0], mp);
    const uint64_t need = mp.slots * kSlotBytes;
    if (need <= ws->bytes) break;
    try {
      ws->release();  // in stream order, after the launches that use it
      *ws = DevBuf(round_up(need, 4ull << 20), stream, true);
      break;
    } catch (const Error &e) {
      if (e.code != HD_ERR_OOM) throw;
      cudaGetLastError();
      mp = MmaPlan();  // no room for the pieces: whole items
      may_split.assign(nj, 0);
    }
  }
  // one device block: [tensor maps (2 per job)][jobs][items][split tiles]
  // [queue counter][dash blocks to write]
  const size_t tm_bytes = nj * 2 * sizeof(CUtensorMap);
  const size_t job_at = tm_bytes, item_at = job_at + round_up(nj * sizeof(MmaJob), 64);
  const size_t fix_at = item_at + mp.items.size() * sizeof(MmaItem);
  const size_t counter_at = fix_at + round_up(mp.fix.size() * sizeof(MmaFix), 16);
  const size_t dash_at = counter_at + 16;
  std::vector<uint8_t> host(dash_at + dash_later.jobs.size() * sizeof(OpRows), 0);
  DevBuf dev(host.size(), stream);
  auto *tms = reinterpret_cast<CUtensorMap *>(host.data());
  auto *jobs = reinterpret_cast<MmaJob *>(host.data() + job_at);
  for (size_t q = 0; q < nj; ++q) {
    const PairJobSpec &sp = specs[js[q].k];
    const hd_alignment *a = sp.aln, *o = owner_of(js[q]);
    make_tmap_op(ctx, &tms[2 * q], ops[js[q].k], planes[q], o->length, a->n_rows, kTM);
    make_tmap_op(ctx, &tms[2 * q + 1], ops[js[q].k], planes[q], o->length, a->n_rows, kItemCols / 2);
    MmaJob &m = jobs[q];
    m.out = sp.d_out;
    m.out_base = sp.out_base;
    m.chunks = op_chunks(o->length);
    m.dash_list = dash_lists[js[q].k];
    m.dash_rank = m.dash_list + m.chunks;
    // the launch's lower-triangle pairs (for its multiply-add count)
    const uint64_t r_lo = (uint64_t)js[q].t_lo * kTM, r_hi = std::min<uint64_t>((uint64_t)js[q].t_hi * kTM, a->n_rows);
    m.row_hi = (uint32_t)r_hi;
    m.pairs = r_hi * (r_hi - 1) / 2 - (r_lo ? r_lo * (r_lo - 1) / 2 : 0);
    m.planes = planes[q];
    m.sites = (uint32_t)a->length;
    m.max_dist = sp.max_dist;
    m.dtype = (uint32_t)sp.dtype;
  }
  std::memcpy(host.data() + item_at, mp.items.data(), mp.items.size() * sizeof(MmaItem));
  std::memcpy(host.data() + fix_at, mp.fix.data(), mp.fix.size() * sizeof(MmaFix));
  std::memcpy(host.data() + dash_at, dash_later.jobs.data(), dash_later.jobs.size() * sizeof(OpRows));
  // staged in pinned memory (pageable for a large table): `host` may go when this returns
  upload_table(ctx, dev.p, host.data(), host.size(), stream);
  uint8_t *d = dev.as<uint8_t>();
  dash_later.launch(reinterpret_cast<const OpRows *>(d + dash_at));
  PairLaunchPlan::Launch L;
  L.mma = true;
  L.fn = reinterpret_cast<const void *>(k_pairwise_mma);
  L.smem = kMmaSmem;
  L.tile = kTM;
  L.jobs = nj;
  for (const Job &j : js) L.tiles += size_tiles(j.t_lo, j.t_hi);
  L.items = mp.items.size();
  L.grid = 2 * mp.pairs;
  L.d_jobs = d + job_at;
  L.d_items = d + item_at;
  L.d_tms = d;
  L.d_fix = d + fix_at;
  L.fixes = mp.fix.size();
  L.d_ws = ws->p;
  L.d_counter = reinterpret_cast<unsigned long long *>(d + counter_at);
  L.queue = queue;
  plan->launches.push_back(L);
  plan->blocks.push_back(std::move(dev));
  if (own.p) plan->blocks.push_back(std::move(own));
}

void launch_mma(hd_ctx *ctx, const PairLaunchPlan::Launch &L, cudaStream_t stream) {
  set_smem_once(ctx->device);
  // the item queue starts empty at every launch (also when a graph replays it)
  if (L.queue) HD_CUDA(cudaMemsetAsync(L.d_counter, 0, sizeof(unsigned), stream));
  k_pairwise_mma<<<(unsigned)L.grid, kMmaThreads, kMmaSmem, stream>>>(
      static_cast<const CUtensorMap *>(L.d_tms), static_cast<const MmaJob *>(L.d_jobs),
      (uint32_t)L.jobs, static_cast<const MmaItem *>(L.d_items), (uint32_t)L.items,
      reinterpret_cast<unsigned *>(L.d_counter), L.queue ? 1u : 0u,
      static_cast<uint32_t *>(L.d_ws), mma_mac_counter(ctx), ctx->d_status);
  HD_LAUNCHED(ctx);
  if (L.fixes) {
    k_pair_fix<<<(unsigned)ceil_div(L.fixes * kFixWarps, (uint64_t)8), 256, 0, stream>>>(
        static_cast<const MmaJob *>(L.d_jobs), static_cast<const MmaFix *>(L.d_fix),
        (uint32_t)L.fixes, static_cast<const uint32_t *>(L.d_ws));
    HD_LAUNCHED(ctx);
  }
  ctx->last_pair_tiles += L.tiles;
}

bool pairwise_mma(hd_ctx *ctx, const hd_alignment *aln, int dtype_bytes, uint32_t max_dist,
                  void *d_out, uint64_t out_base, uint32_t tile_lo, uint32_t tile_hi,
                  cudaStream_t stream, int sm_limit) {
  if (!mma_eligible(aln)) return false;
  std::vector<PairJobSpec> specs(1);
  PairJobSpec &sp = specs[0];
  sp.aln = aln;
  sp.dtype = dtype_bytes;
  sp.max_dist = max_dist;
  sp.d_out = d_out;
  sp.out_base = out_base;
  // the tensor-core settings of the whole matrix's bucket; row tiles of 128
  sp.cfg = tile_config_for(ctx, aln->n_rows, aln->length, dtype_bytes);
  sp.cfg.tile = kTM;
  sp.tile_lo = tile_lo;
  sp.tile_hi = std::min<uint32_t>(tile_hi, (uint32_t)ceil_div(aln->n_rows, kTM));
  if (sp.tile_hi <= sp.tile_lo) return true;
  PairLaunchPlan plan;
  std::vector<char> taken;
  prepare_mma_jobs(ctx, specs, stream, &plan, sm_limit, taken);
  if (!taken[0]) return false;
  for (const auto &L : plan.launches) launch_mma(ctx, L, stream);
  return true;  // the plan's device block is freed in stream order, after the kernel
}

}  // namespace hd
