// census_tc.cuh — the census matcher (9x7 descriptors, 5x5 Hamming sums,
// winner-take-all in both directions) with its window sums on the tensor cores.
//
// With the 64 descriptor bits as +1 / -1, the Hamming distance of two
// descriptors is (64 - a . b) / 2, so the 5x5 cost of left pixel x and right
// pixel x' is (1600 - S(x, x')) / 2 with
//   S(x, x') = sum over rows r = y-2 .. y+2 and i = -2 .. 2 of
//              a(x + i, r) . b(x' + i, r):
// per image row and shift i a product of two matrices, A (left pixels, one
// descriptor a row) times B^T (right pixels). +-1 is exact in 4-bit floating
// point (e2m1), so the products run as tcgen05.mma kind::mxf4 (K = 64, one
// descriptor; block scales all 1), four times the f16 rate; the fp32 sums are
// small integers, exact. A tile is 128 left pixels x up to 240 right pixels;
// its accumulator in TMEM keeps the running window sum down a strip of rows,
// S(y+1) = S(y) + row y+3 - row y-2 (subtracted by the descriptor's negate-A
// bit): 10 MMAs a row. The shift by i pixels is i * 16 bytes on the operands'
// start addresses (K-major, no swizzle: pixel rows 16 bytes apart).
//
// The accumulator starts at 2048 - d / 256 (d the pair's disparity, relative
// to the minimum) inside the searched band and at -30000 outside it, so that
// every value read back is already the winner-take-all key: larger is a lower
// cost, then a lower d (fp32 holds it exactly: 12 + 8 bits), and nothing needs
// masking. (A tile that finds nothing keeps the empty key 0.)
// Both directions take their maxima from the same values: along the row
// (left pixel) and along the column (right pixel).
//
// A CTA (one an SM) works on a pair of tiles, so that one tile's maxima run
// while the other's MMAs do: two neighbouring column tiles of a strip, or the
// two halves of one tile's right pixels when the disparities need more than
// 240 columns. (Two CTAs an SM instead, each with one tile, fell into step:
// both waited for their MMAs, then both ran their maxima with the tensor core
// idle.) 20 warps, 5 a scheduler, which lets each have 96 registers:
//   warps 0-7, 8-15  maxima of tile 0 and of tile 1: lane quarter q = warp % 4
//               (the TMEM lanes a warp may read), the quarter's band in
//               40-column pieces, alternating between its two warps. A row's
//               results merge in shared memory and leave two rows later;
//   warps 16-18 descriptors of the rows ahead, global -> e2m1 in shared memory
//               (a ring of 8 rows: 5 of the window, the leaving one, 2 ahead);
//   warp 19     the MMAs of both tiles in turn (issued by a warp each, both
//               tiles' MMAs ran at once, ended together, and left the tensor
//               core idle while both tiles' maxima ran).
// What waits for MMAs does so on mbarriers, boundedly.
//
// What bounds it: at 1920x1080, D = 128 (18 column tiles of 107 pixels, 240
// columns, strips of 68 rows: 144 CTAs) a row of a tile pair takes 20 MMAs of
// 120 cycles = 2400 cycles; the left view alone runs at that rate (2400 cycles
// a row traced), both views at about 2900, by the maxima's instructions (3830 a
// tile and row, 2.6 of 4 issued per cycle). Whole calls there: left view 121 us
// (223 on the CUDA cores), both views and check 144 us (266).
//
#pragma once

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "census_match.cuh"
#include "ct_device.cuh"

namespace ct {
namespace ctc {

constexpr int kM = 128;                 // left pixels of a tile: MMA M, TMEM lanes
constexpr int kNMax = 240;              // right pixels of a tile: MMA N, accumulator columns
constexpr int kR = 2;                   // window radius
constexpr int kWin = 2 * kR + 1;
constexpr int kSlots = 8;               // descriptor rows in the ring
constexpr int kAP = 2 * kM + 2 * kR;    // left pixels of a staged row (both tiles)
constexpr int kBP = 392;                // right pixels: 128 + 240 + 4, or 2 * 192 + 4
constexpr int kSlotBytes = (kAP + kBP) * 32;
constexpr int kPiece = 40;              // accumulator columns a warp reduces at a time
constexpr int kTileWarps = 8, kRowWarps = 3;
constexpr int kTileT = kTileWarps * 32, kMaxT = 2 * kTileT, kRowT = kRowWarps * 32;
constexpr int kNT = kMaxT + kRowT + 32;
constexpr int kRowPx = 7;               // staged pixels of a row a thread converts: 7 * 96 >= 256 + 4 + 368 + 4
constexpr uint32_t kTmemCols = 512, kScaleCol = 2 * kNMax;  // columns 480 .. 495: block scales
// shared memory
constexpr int kRowsL = 8, kRowsR = 4;   // rows of keys kept
constexpr int kKeyN = 256;              // right keys of a quarter's row (kNMax, a power of 2)
constexpr int kOffKeyL = kSlots * kSlotBytes;               // kRowsL x 2 tiles x 2 warps of a quarter x kM keys
constexpr int kOffKeyR = kOffKeyL + kRowsL * 4 * kM * 4;    // 2 tiles x kRowsR x 4 quarters x kNMax keys
constexpr int kOffBar = kOffKeyR + 2 * kRowsR * 4 * kKeyN * 4;
constexpr int kBars = 8 + kRowsL + 1;  // ready, merged, drained
constexpr int kOffMisc = kOffBar + kBars * 8;
constexpr int kSmemBytes = kOffMisc + 32;
static_assert(kOffKeyL % 16 == 0 && kOffBar % 8 == 0 && kSmemBytes <= 227 * 1024, "shared memory");

struct Args {
    int W, H, D;        // relative disparities 0 .. D-1
    int dmin;           // relative d matches column x - (dmin + d) and is stored as dmin + d
    int mo, n, th;      // tile: left pixels (<= 128), columns (multiple of 16), rows
    int lstep, rstep;   // tile 1 of a pair: left pixels + lstep (mo or 0), right pixels + rstep (mo or n)
    const uint64_t* left;
    const uint64_t* right;
    size_t pitch;       // descriptor rows, elements
    void* out;          // left-to-right map (null when not asked for)
    size_t out_pitch;
    int out_type;
    uint32_t* r_keys;   // right-to-left winners: bids (null when not asked for)
    size_t key_pitch;   // words
    uint32_t tag;       // the call's tag: bids are tag | 23 bits that grow with the key (cm::MaxKeys)
    int32_t* status;
    uint32_t polls;     // limit of every wait (kPolls; less in tests)
};

struct Shape {
    int mo, n, lstep, rstep, tiles_x;  // tiles_x: pairs of tiles in a strip
    double row_cost;                   // cycles of a pair's row (estimate)
};

// Shape of the tile pair: neighbouring column tiles, or (from about 150
// disparities) one column tile whose right pixels are cut in two; the one
// with the fewer cycles for a strip's row. A row of a pair takes the longer
// of its MMAs (n / 2 cycles each, or 32 + n / 4 where the operands' shared
// memory reads, 128 bytes a cycle, take longer) and its maxima (about 55
// cycles a 40-column piece and 300 a tile).
inline Shape pick_shape(int W, int D) {
    Shape best{};
    double best_cost = -1;
    for (int split = 0; split < 2; ++split) {
        const int most = split ? kM : std::min(kM, kNMax - (D - 1));
        if (most < 16) continue;
        Shape s{};
        const int per = split ? most : 2 * most;
        s.tiles_x = (W + per - 1) / per;
        s.mo = split ? (W + s.tiles_x - 1) / s.tiles_x : (W + 2 * s.tiles_x - 1) / (2 * s.tiles_x);
        const int span = s.mo + D - 1;
        s.n = std::max(((split ? (span + 1) / 2 : span) + 15) / 16 * 16, 48);
        s.lstep = split ? 0 : s.mo;
        s.rstep = split ? s.n : s.mo;
        const double mma = 20.0 * std::max(s.n / 2, 32 + s.n / 4);
        const double alu = 2.0 * (4 * ((std::min(s.n, D + 31) + kPiece - 1) / kPiece) * 55.0 + 300.0);
        s.row_cost = std::max(mma, alu);
        const double cost = s.tiles_x * s.row_cost;
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = s;
        }
    }
    return best;
}

// Strip height: waves of tile pairs over the SMs x a pair's rows, the first
// window (15 more MMAs) and the start of the pipeline worth about 4 rows.
inline int pick_rows(int H, int tiles, int sms) {
    int best = H;
    long best_cost = -1;
    for (int th = 4; th <= H || th == 4; ++th) {
        const long items = long((H + th - 1) / th) * tiles;
        const long cost = (items + sms - 1) / sms * (std::min(th, H) + 4);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = th;
        }
    }
    return best;
}

// Instruction descriptor, kind::mxf4: A and B e2m1 (bits 7, 10 = 1), negate A
// (bit 13), both K-major, N >> 3 at bit 17, ue8m0 scales (bit 23), M >> 7 at
// bit 27.
__device__ __forceinline__ uint32_t idesc(int n, bool negate_a) {
    return (1u << 7) | (1u << 10) | (uint32_t(negate_a) << 13) | (uint32_t(n >> 3) << 17) | (1u << 23) |
           (uint32_t(kM >> 7) << 27);
}
// Shared-memory matrix descriptor: start, leading byte offset (the second half
// of K), stride byte offset 128 (the next 8 pixel rows), version 1, no swizzle.
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo) {
    return uint64_t((saddr >> 4) & 0x3FFF) | (uint64_t((lbo >> 4) & 0x3FFF) << 16) | (uint64_t(128 >> 4) << 32) |
           (uint64_t(1) << 46);
}
// Issued by the warp's elected lane, from code that the whole warp runs (its
// operands then stay in uniform registers).
__device__ __forceinline__ void mma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t id, uint32_t scales) {
    asm volatile(
        "{\n.reg .pred p, e;\nsetp.ne.b32 p, 1, 0;\nelect.sync _|e, 0xffffffff;\n"
        "@e tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%4], [%4], p;\n}\n" ::"r"(
            tmem_d),
        "l"(a), "l"(b), "r"(id), "r"(scales)
        : "memory");
}
__device__ __forceinline__ void commit(uint64_t* bar) {
    asm volatile(
        "{\n.reg .pred e;\nelect.sync _|e, 0xffffffff;\n"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(
            dev::smem_u32(bar))
        : "memory");
}
// Waits for phase `parity` of `bar`, suspended for up to 20 us a poll (waiting
// warps that poll more often take the maxima's issue slots), for `polls` polls.
// Returns the polls for the next wait: the same (about a second), or 0 once a
// wait gave up.
constexpr uint32_t kPolls = 1u << 16;
__device__ __forceinline__ uint32_t wait(uint64_t* bar, uint32_t parity, uint32_t polls) {
    const uint32_t addr = dev::smem_u32(bar);
    for (uint32_t i = 0; i < polls; ++i) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(addr), "r"(parity), "r"(20000u)
            : "memory");
        if (done) return polls;
    }
    return 0;
}
__device__ __forceinline__ void arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(dev::smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Eight accumulator columns of this thread's lane.
__device__ __forceinline__ void st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]),
                 "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Columns taddr .. taddr + 39 of the warp's 32 lanes, waited for: lane t holds
// of each 8 columns g the columns 8 g + 2 (t % 4) + e of rows t / 4 + 8 k:
// v[k][2 g + e].
__device__ __forceinline__ void ld_piece(uint32_t taddr, float (&v)[4][10]) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const uint32_t ta = taddr + (uint32_t(16 * half) << 16);
        float (&lo)[10] = v[2 * half];
        float (&hi)[10] = v[2 * half + 1];
        asm volatile(
            "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=f"(lo[0]), "=f"(lo[1]), "=f"(hi[0]), "=f"(hi[1]), "=f"(lo[2]), "=f"(lo[3]), "=f"(hi[2]), "=f"(hi[3]),
              "=f"(lo[4]), "=f"(lo[5]), "=f"(hi[4]), "=f"(hi[5]), "=f"(lo[6]), "=f"(lo[7]), "=f"(hi[6]), "=f"(hi[7])
            : "r"(ta)
            : "memory");
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];"
                     : "=f"(lo[8]), "=f"(lo[9]), "=f"(hi[8]), "=f"(hi[9])
                     : "r"(ta + 32)
                     : "memory");
    }
    // the waited-for values pass through the wait, so that no use of them can
    // be placed before it
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int j = 0; j < 10; ++j) asm volatile("" : "+f"(v[k][j]));
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Of two values a lane holds, the one its bit (`upper`: hi) says, and the
// maximum of that with the lane's that differs in that bit.
__device__ __forceinline__ float halve(float lo, float hi, bool upper, int mask) {
    const float give = upper ? lo : hi, keep = upper ? hi : lo;
    return fmaxf(keep, __shfl_xor_sync(0xffffffffu, give, mask));
}

// Hand-overs to the MMA warp by hardware barriers, which answer in tens of
// cycles (an mbarrier takes about 200 beside the MMAs' operand reads, longer
// than the MMAs that wait in the tensor core's queue last): the accumulator of
// tile t read (barriers 3, 4), staged row r (5-12 in turn). A phase ends with
// its last arrival, whoever that is, so nobody may arrive for row r + kRowBars
// before the MMA warp has joined row r: the staging warps write kSlots rows
// without waiting for anything, and row k >= kSlots once the MMAs of step k - 7
// are complete, which the MMA warp issued after it joined row k - 3.
// A warp whose wait gave up (about a second without an answer) keeps taking part
// in every hand-over, so that the MMA warp, which waits on nothing else, comes
// to its end and the CTA can report. It arrives for a row once the MMA warp has
// passed the hand-over that the wait stood behind (Cta::passed), and stages
// nothing more: every row then leaves a window as it came in, also in MMAs that
// it did not wait for, so that accumulators read unfinished lie between those of
// finished rows. Their keys are wrong but as bounded as others: columns outside
// the band stay below 0 and bid for nothing. (Holding back the keys as well cost
// 1.6% of a batch.)
constexpr int kRowBars = 8;
static_assert(kRowBars >= kSlots && 5 + kRowBars <= 16,
              "staged rows come round to a barrier after the MMA warp has joined it");
template <int ID, int N>
__device__ __forceinline__ void bar_arrive() {
    asm volatile("barrier.cta.arrive %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
template <int ID, int N>
__device__ __forceinline__ void bar_sync() {
    asm volatile("barrier.cta.sync %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
__device__ __forceinline__ void read_arrive(int t) { t == 0 ? bar_arrive<3, kTileT + 32>() : bar_arrive<4, kTileT + 32>(); }
__device__ __forceinline__ void read_sync(int t) { t == 0 ? bar_sync<3, kTileT + 32>() : bar_sync<4, kTileT + 32>(); }
__device__ __forceinline__ void row_arrive(int r) {
    asm volatile("barrier.cta.arrive %0, %1;" ::"r"(5 + (r & (kRowBars - 1))), "n"(kRowT + 32) : "memory");
}
__device__ __forceinline__ void row_sync(int r) {
    asm volatile("barrier.cta.sync %0, %1;" ::"r"(5 + (r & (kRowBars - 1))), "n"(kRowT + 32) : "memory");
}
// One tile's maxima warps (barriers 1, 2).
__device__ __forceinline__ void tile_sync(int t) { t == 0 ? bar_sync<1, kTileT>() : bar_sync<2, kTileT>(); }

// Shared memory of a CTA and the rows its tiles have completed (the same in
// every thread between tile pairs).
struct Cta {
    unsigned char* smem;
    uint64_t* ready;   // [2 tiles][4] window sums of a row complete (commit and the MMA warp's arrival), rows in turn
    uint64_t* merged;  // [kRowsL] tile 0's keys of a row written (kTileWarps arrivals; pairs that share left pixels)
    uint64_t* drained; // MMAs complete after a wait gave up
    uint32_t* misc;    // TMEM address; rows that the MMA warp has begun, per tile
    uint32_t steps0, steps1, merges;  // rows done by tile 0, by tile 1, with merged
    uint32_t tmem;
    __device__ explicit Cta(unsigned char* raw)
        : smem(raw),
          ready(reinterpret_cast<uint64_t*>(raw + kOffBar)),
          merged(ready + 8),
          drained(merged + kRowsL),
          misc(reinterpret_cast<uint32_t*>(raw + kOffMisc)),
          steps0(0),
          steps1(0),
          merges(0),
          tmem(0) {}
    __device__ uint32_t step(int t, int s) const { return (t ? steps1 : steps0) + uint32_t(s); }
    // Row s of the tile: its barrier, and the wait for it (nobody waits more
    // than 2 rows behind the MMAs, so 4 barriers leave the phase unambiguous).
    __device__ uint64_t* ready_bar(int t, int s) const { return &ready[4 * t + (step(t, s) & 3)]; }
    // After it, by the whole warp, the MMA warp has passed the hand-overs before
    // the row's MMAs, also when the wait gave up.
    __device__ uint32_t wait_ready(int t, int s, uint32_t polls) const {
        polls = wait(ready_bar(t, s), (step(t, s) >> 2) & 1, polls);
        if (polls == 0) passed(t, s);
        __syncwarp();
        return polls;
    }
    __device__ void begin(int t, int s) const { *static_cast<volatile uint32_t*>(misc + 1 + t) = step(t, s) + 1; }
    // Waits until the MMA warp has begun the row: it waits only for the other
    // warps' arrivals, each about a second away at most (the limit is about 20).
    __device__ void passed(int t, int s) const {
        const volatile uint32_t* begun = misc + 1 + t;
        for (uint32_t i = 0; i < (1u << 20) && int32_t(*begun - step(t, s)) <= 0; ++i) __nanosleep(20000);
    }
};

// Barriers, TMEM, block scales, keys and a ring of zeros (the operands of
// lanes and columns beyond a tile stay finite); ends with a CTA barrier.
__device__ __forceinline__ void cta_begin(Cta& c) {
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) {
        for (int i = 0; i < 8; ++i) dev::mbar_init(&c.ready[i], 2);
        for (int i = 0; i < kRowsL; ++i) dev::mbar_init(&c.merged[i], kTileWarps);
        dev::mbar_init(c.drained, 1);
        c.misc[1] = c.misc[2] = 0;
        dev::fence_barrier_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dev::smem_u32(c.misc)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i < kOffBar / 16; i += kNT) reinterpret_cast<uint4*>(c.smem)[i] = make_uint4(0, 0, 0, 0);
    dev::fence_proxy_async();
    fence_before();
    __syncthreads();
    fence_after();
    c.tmem = c.misc[0];
    if (warp < 4) {  // scales: 2^0 everywhere
        const uint32_t ones[8] = {0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu,
                                  0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu};
        const uint32_t t = c.tmem + (uint32_t(32 * warp) << 16) + kScaleCol;
        st8(t, ones);
        st8(t + 8, ones);
        wait_st();
    }
    fence_before();
    __syncthreads();
    fence_after();
}

__device__ __forceinline__ void cta_end(Cta& c) {
    fence_before();
    __syncthreads();
    fence_after();
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.tmem), "r"(kTmemCols) : "memory");
}

// A key (positive) as an integer of the same order, 0x47000000 + 23 bits: the
// sum's last mantissa bit is 1 / 256, so its low byte is minus the relative
// disparity.
__device__ __forceinline__ uint32_t key_bits(float key) { return __float_as_uint(key + 49152.0f); }

// One tile pair: strip by, pair bx. Every thread of the CTA calls it; returns
// false if a wait gave up (the status word is set; the CTA must take no
// further tile).
__device__ __forceinline__ bool run_tile(Cta& c, const Args& a, int bx, int by) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int x0 = bx * (a.mo + a.lstep), y0 = by * a.th;
    const int rows = min(a.th, a.H - y0);
    const int xb = x0 - a.dmin - (a.D - 1);   // right pixel of tile 0's column 0
    const int nrows = rows + 2 * kR;          // staged rows
    const int tiles = x0 + a.lstep < a.W ? 2 : 1;  // a strip's last pair may have one tile only
    const bool share = a.lstep == 0;               // the tiles have the same left pixels
    uint32_t polls = a.polls;

    if (warp >= (kMaxT + kRowT) / 32) {
        // ---- MMAs
        const uint32_t id_add = idesc(a.n, false), id_sub = idesc(a.n, true);
        const uint32_t tmem = __shfl_sync(0xffffffffu, c.tmem, 0), scales = tmem + kScaleCol;
        const uint64_t a0 = sdesc(dev::smem_u32(c.smem), kAP * 16);
        const uint64_t b0 = sdesc(dev::smem_u32(c.smem) + kAP * 32, kBP * 16);
        auto row_mmas = [&](int t, int k, uint32_t id) {  // staged row k into tile t's accumulator
            const uint32_t s = uint32_t(k % kSlots) * (kSlotBytes / 16);
            const uint64_t da = a0 + (s + uint32_t(t * a.lstep)), db = b0 + (s + uint32_t(t * a.rstep));
#pragma unroll
            for (int i = 0; i < kWin; ++i) mma(tmem + uint32_t(t * kNMax), da + i, db + i, id, scales);
        };
        // Row s of tile t. Nothing else is done here: the tensor core's queue
        // holds about 4 MMAs, and a second commit would wait for it to drain.
        auto step = [&](int t, int s) {
            read_sync(t);
            if (lane == 0) arrive(c.ready_bar(t, s));  // hands on what the reads' arrivals ordered
            __syncwarp();
            fence_after();
            if (s == 0) {
                for (int k = 0; k < kWin; ++k) row_mmas(t, k, id_add);
            } else {
                row_mmas(t, s + 2 * kR, id_add);
                row_mmas(t, s - 1, id_sub);
            }
            commit(c.ready_bar(t, s));
            if (lane == 0) c.begin(t, s);  // (after the MMAs: before them it cost 1%)
        };
        for (int k = 0; k < kWin - 1; ++k) row_sync(k);
        for (int s = 0; s < rows; ++s) {
            row_sync(s + kWin - 1);
            step(0, s);
            if (tiles == 2) step(1, s);
        }
        for (int t = 0; t < tiles; ++t) read_sync(t);
    } else if (warp >= kMaxT / 32) {
        // ---- descriptors of the strip's rows
        const int ti = tid - kMaxT;
        const int na = a.mo + a.lstep + 2 * kR, nb = a.n + a.rstep + 2 * kR;  // staged left and right pixels
        // Pixels outside the image read some pixel inside it: they only meet
        // windows that leave the image, which are outside every band. So do
        // rows; threads beyond the row's pixels repeat its last one.
        const uint64_t* src[kRowPx];             // the thread's pixels in the row fetched next
        uint32_t dst0[kRowPx], dst1[kRowPx];     // in a ring slot: the two halves of K
#pragma unroll
        for (int j = 0; j < kRowPx; ++j) {
            const int i = min(ti + kRowT * j, na + nb - 1);
            const bool isl = i < na;
            const int x = min(max(isl ? x0 - kR + i : xb - kR + (i - na), 0), a.W - 1);
            src[j] = (isl ? a.left : a.right) + size_t(max(y0 - kR, 0)) * a.pitch + x;
            dst0[j] = uint32_t(16 * i + (isl ? 0 : kAP * 32 - 16 * na));
            dst1[j] = dst0[j] + (isl ? kAP * 16 : kBP * 16);
        }
        int y_next = y0 - kR;
        auto fetch = [&](uint64_t (&v)[kRowPx]) {
            const size_t step = y_next >= 0 && y_next < a.H - 1 ? a.pitch : 0;
            ++y_next;
#pragma unroll
            for (int j = 0; j < kRowPx; ++j) {
                v[j] = __ldg(src[j]);
                src[j] += step;
            }
        };
        auto stage = [&](int k, const uint64_t (&v)[kRowPx]) {
            // row k - 8 left both windows with the last tile's step k - 7
            if (k >= kSlots) polls = c.wait_ready(tiles - 1, k - kSlots + 1, polls);
            unsigned char* s = c.smem + (k % kSlots) * kSlotBytes;
#pragma unroll
            for (int j = 0; j < kRowPx; ++j) {
                if (polls == 0) break;
                // bit -> sign of a nibble holding 1.0; the order of the bits is
                // the same for both operands
                auto e2m1 = [](uint32_t w, int q) { return ((w << q) & 0x88888888u) | 0x22222222u; };
                const uint32_t lo = uint32_t(v[j]), hi = uint32_t(v[j] >> 32);
                *reinterpret_cast<uint4*>(s + dst0[j]) =
                    make_uint4(e2m1(lo, 0), e2m1(lo, 1), e2m1(lo, 2), e2m1(lo, 3));
                *reinterpret_cast<uint4*>(s + dst1[j]) =
                    make_uint4(e2m1(hi, 0), e2m1(hi, 1), e2m1(hi, 2), e2m1(hi, 3));
            }
            dev::fence_proxy_async();  // generic-proxy writes -> the tensor core's reads
            row_arrive(k);
        };
        // the loads of the two rows after the one being converted are in flight
        uint64_t v0[kRowPx], v1[kRowPx];
        fetch(v0);
        fetch(v1);
        for (int k = 0; k < nrows; k += 2) {
            stage(k, v0);
            fetch(v0);
            if (k + 1 < nrows) stage(k + 1, v1);
            fetch(v1);
        }
    } else if (warp / kTileWarps < tiles) {
        // ---- maxima
        const int t = warp / kTileWarps, q = warp & 3, h = (warp >> 2) & 1, tt = tid & (kTileT - 1);
        const int xl = x0 + t * a.lstep, xr0 = xb + t * a.rstep;  // the tile's first left and right pixels
        const uint32_t tq = c.tmem + (uint32_t(32 * q) << 16) + uint32_t(t * kNMax);
        {  // the accumulator's start: keys of cost sum 0 inside the searched band
            const int m = 32 * q + lane, x = xl + m;
            // its columns n: right pixel xr0 + n inside, d = x - xr0 - n - dmin in 0 .. D-1
            const int dn = x - xr0 - a.dmin;
            const int lo = max(kR - xr0, dn - (a.D - 1)), hi = min(a.W - kR - 1 - xr0, dn);
            const uint32_t count = m < a.mo && x >= kR && x < a.W - kR && hi >= lo ? uint32_t(hi - lo + 1) : 0u;
            const float f0 = 2048.0f - float(dn) * (1.0f / 256.0f);
            for (int n0 = 8 * h; n0 < a.n; n0 += 16) {
                uint32_t w[8];
                const float f = f0 + float(n0) * (1.0f / 256.0f);
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    w[j] = __float_as_uint(uint32_t(n0 + j - lo) < count ? f + float(j) * (1.0f / 256.0f) : -30000.0f);
                st8(tq + uint32_t(n0), w);
            }
            wait_st();
            fence_before();
            read_arrive(t);
        }
        // columns that meet the band of the quarter's 32 pixels, from a
        // multiple of 8, in pieces of 40
        const int c_lo = max(xl + 32 * q - a.dmin - (a.D - 1) - xr0, 0) & ~7;
        const int c_hi = min(xl + 32 * q + 31 - a.dmin - xr0, a.n - 1);
        const int pieces = c_hi < c_lo ? 0 : (c_hi - c_lo + kPiece) / kPiece;
        // Keys of a row, a place of its own for each writer (no shared
        // atomics: the MMAs' operand reads and these share the memory's
        // bandwidth): left keys [row % kRowsL][tile][h][pixel], right keys
        // [row % kRowsR][q][column]; columns no piece covers stay 0.
        float* keyL = reinterpret_cast<float*>(c.smem + kOffKeyL);
        float* keyR = reinterpret_cast<float*>(c.smem + kOffKeyR) + kRowsR * 4 * kKeyN * t;
        for (int i = tt; i < kRowsR * 4 * kKeyN; i += kTileT) keyR[i] = 0.0f;
        tile_sync(t);
        const bool f0 = lane & 1, f1 = lane & 2, f2 = lane & 4, f3 = lane & 8, f4 = lane & 16;
        // the column (of its piece) of the lane's first result (columns 0-31),
        // and of its second one (columns 32-39, lanes with bits 2, 3 clear)
        const int j0 = 4 * (lane >> 4) + 2 * ((lane >> 2) & 1) + ((lane >> 3) & 1);
        const int col0 = 8 * (j0 >> 1) + 2 * (lane & 3) + (j0 & 1);
        const int col1 = 32 + 2 * (lane & 3) + (lane >> 4);
        const int row = 32 * q + (lane >> 2) + 8 * (lane & 3);  // the lane's left pixel
        // Row r's results: two right pixels a thread (warps 0-3 of the tile) or
        // one left pixel (warps 4-7). The keys are read (take), then written
        // out (put, rows in order). Tiles that share left pixels leave those
        // to tile 1's warps.
        const int lt = tt - kM, rt = 2 * tt;
        const bool put_l = a.out && lt >= 0 && lt < a.mo && (!share || t == 1) && xl + lt < a.W;
        // (n is even; the image's first and last columns have no disparity)
        const bool put_r = a.r_keys && rt < a.n && xr0 + rt >= 0 && xr0 + rt + 1 < a.W;
        const bool u8 = a.out_type == CT_PIX_U8;
        char* out = static_cast<char*>(a.out) + size_t(y0) * a.out_pitch + (xl + lt) * (u8 ? 1 : 2);
        uint32_t* bids = a.r_keys + size_t(y0) * a.key_pitch + (xr0 + rt);
        const uint32_t tag = a.tag - 0x47000000u;
        auto inside = [&](int r) { return uint32_t(y0 + r - kR) < uint32_t(max(a.H - 2 * kR, 0)); };
        auto take = [&](int r, float& k0, float& k1) {
            if (put_l) {
                const float* p = keyL + (r & (kRowsL - 1)) * (4 * kM) + lt;
                k0 = fmaxf(p[2 * t * kM], p[(2 * t + 1) * kM]);
                if (share) k0 = max3(k0, p[0], p[kM]);
            }
            if (put_r) {
                const float2* p = reinterpret_cast<const float2*>(keyR + (r & (kRowsR - 1)) * (4 * kKeyN) + rt);
                const float2 p0 = p[0], p1 = p[kKeyN / 2], p2 = p[kKeyN], p3 = p[3 * kKeyN / 2];
                k0 = fmaxf(max3(p0.x, p1.x, p2.x), p3.x);
                k1 = fmaxf(max3(p0.y, p1.y, p2.y), p3.y);
            }
        };
        auto put = [&](int r, float k0, float k1) {
            const bool yin = inside(r);
            if (put_l) {
                const uint32_t d = ((0u - key_bits(k0)) & 255u) + uint32_t(a.dmin);
                const bool found = yin && k0 > 0.0f;
                if (u8) *reinterpret_cast<uint8_t*>(out) = found ? uint8_t(d) : uint8_t(0xFF);
                else *reinterpret_cast<uint16_t*>(out) = found ? uint16_t(d + 1) : uint16_t(0xFFFF);
            }
            if (put_r && yin) {
                if (k0 > 0.0f) atomicMax(bids, key_bits(k0) + tag);
                if (k1 > 0.0f) atomicMax(bids + 1, key_bits(k1) + tag);
            }
            out += a.out_pitch;
            bids += a.key_pitch;
        };
        // Left keys of tile 0's row r, for tile 1 when they share pixels. Tile
        // 0 is less than kRowsL rows ahead of what tile 1 has put: its MMAs of
        // row s are issued after tile 1's of row s - 1, which follow that
        // tile's reads of row s - 2 and so its put of row s - 5.
        auto wait_merged = [&](int r) {
            const uint32_t g = c.merges + uint32_t(r);
            if (share && t == 1) polls = wait(&c.merged[g & (kRowsL - 1)], (g / kRowsL) & 1, polls);
        };
        float* const put_kl = keyL + (2 * t + h) * kM + row;
        float* const put_kr = keyR + q * kKeyN;
        for (int s = 0; s < rows; ++s) {
            polls = c.wait_ready(t, s, polls);
            fence_after();
            float rm[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            // Maxima of a piece: along the rows into rm, along the columns
            // (over the thread's 4 rows) into w.
            auto reduce = [&](const float (&v)[4][10], float (&w)[10]) {
                if (a.out) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int j = 0; j < 10; j += 2) rm[k] = max3(rm[k], v[k][j], v[k][j + 1]);
                }
                if (a.r_keys) {
#pragma unroll
                    for (int j = 0; j < 10; ++j) w[j] = fmaxf(max3(v[0][j], v[1][j], v[2][j]), v[3][j]);
                }
            };
            // Two pieces at a time; the accumulator is given back before what
            // needs no more of it. (Rows whose windows leave the image are not
            // written out.)
            int p = h;
            if (p >= pieces) {
                fence_before();
                read_arrive(t);
            }
            auto reduce_pieces = [&](auto pair) {
                constexpr bool kTwo = decltype(pair)::value;
                const int na = min(c_lo + kPiece * p, a.n - kPiece);
                const int nb = min(c_lo + kPiece * (p + 2), a.n - kPiece);
                float v[4][10], wa[10], wb[10];
                ld_piece(tq + uint32_t(na), v);
                if constexpr (kTwo) {
                    reduce(v, wa);
                    ld_piece(tq + uint32_t(nb), v);
                }
                if (p + 4 >= pieces) {
                    fence_before();
                    read_arrive(t);
                }
                if constexpr (kTwo) reduce(v, wb);
                else reduce(v, wa);
                if (!a.r_keys) return;
                // The column maxima over the 8 lanes of equal t % 4, halving
                // the columns a lane keeps while it can: of w[0..3], w[8] and
                // w[4..7], w[9], then of the four, then of the two. Both
                // pieces level by level, so that one's shuffles cover the
                // other's latency.
                float ua[4], ub[4], za, zb;
#pragma unroll
                for (int j = 0; j < 4; ++j) ua[j] = halve(wa[j], wa[j + 4], f4, 16);
                za = halve(wa[8], wa[9], f4, 16);
                if constexpr (kTwo) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) ub[j] = halve(wb[j], wb[j + 4], f4, 16);
                    zb = halve(wb[8], wb[9], f4, 16);
                }
                ua[0] = halve(ua[0], ua[1], f3, 8);
                ua[2] = halve(ua[2], ua[3], f3, 8);
                za = fmaxf(za, __shfl_xor_sync(0xffffffffu, za, 8));
                if constexpr (kTwo) {
                    ub[0] = halve(ub[0], ub[1], f3, 8);
                    ub[2] = halve(ub[2], ub[3], f3, 8);
                    zb = fmaxf(zb, __shfl_xor_sync(0xffffffffu, zb, 8));
                }
                ua[0] = halve(ua[0], ua[2], f2, 4);
                za = fmaxf(za, __shfl_xor_sync(0xffffffffu, za, 4));
                if constexpr (kTwo) {
                    ub[0] = halve(ub[0], ub[2], f2, 4);
                    zb = fmaxf(zb, __shfl_xor_sync(0xffffffffu, zb, 4));
                }
                float* d = put_kr + (s & (kRowsR - 1)) * (4 * kKeyN);
                d[na + col0] = ua[0];
                if constexpr (kTwo) d[nb + col0] = ub[0];
                if (!(lane & 12)) {
                    d[na + col1] = za;
                    if constexpr (kTwo) d[nb + col1] = zb;
                }
            };
            for (; p < pieces; p += 4) {
                if (p + 2 < pieces) reduce_pieces(std::true_type{});
                else reduce_pieces(std::false_type{});
            }
            // row s - 2: every warp wrote its keys before it read row s - 1's
            // accumulator, which the MMAs of this row waited for
            float k0 = 0.0f, k1 = 0.0f;
            if (s >= 2) {
                wait_merged(s - 2);
                take(s - 2, k0, k1);
            }
            if (a.out) {
                const float r0 = halve(rm[0], rm[1], f0, 1), r1 = halve(rm[2], rm[3], f0, 1);
                const float r = halve(r0, r1, f1, 2);
                put_kl[(s & (kRowsL - 1)) * (4 * kM)] = r;
            }
            if (share && t == 0) {
                __syncwarp();
                if (lane == 0) arrive(&c.merged[(c.merges + uint32_t(s)) & (kRowsL - 1)]);
            }
            if (s >= 2) put(s - 2, k0, k1);
        }
        // the last two rows
        tile_sync(t);
        for (int r = max(rows - 2, 0); r < rows; ++r) {
            float k0 = 0.0f, k1 = 0.0f;
            wait_merged(r);
            take(r, k0, k1);
            put(r, k0, k1);
        }
    }
    c.steps0 += uint32_t(rows);
    if (tiles == 2) c.steps1 += uint32_t(rows);
    if (share) c.merges += uint32_t(rows);
    const bool failed = __syncthreads_or(polls == 0);
    if (failed) {
        if (tid == 0) dev::report(a.status, CT_ETIMEOUT);
        if (warp == kNT / 32 - 1) {  // the MMA warp: none may be in flight when the CTA ends
            commit(c.drained);
            wait(c.drained, 0, kPolls);
        }
        __syncthreads();
    }
    return !failed;
}

}  // namespace ctc
}  // namespace ct
