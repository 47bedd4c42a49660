// ncc_guided.cuh — the guided NCC matcher (match_ncc.cu): every 16 x 16 block
// of pixels searches its own range of disparities (guide.cuh). Included by
// match_ncc.cu after the CUDA-core kernel; scores, ranking and maps are the
// same.
//
// A CTA (2 warps) is one block, so that it searches its own range and not the
// union over a wide tile (118 x 32 pixels: on a scene of slanted planes nearly
// every disparity). A thread owns a column of the block and 4 neighbouring
// disparities; it walks down the block's rows and keeps their window sums. A
// row's part of a window, 2R+1 products, is 3 dp4a (2 for R = 2) on words of 4
// pixels, cut from aligned words by funnel shifts; 4 neighbouring disparities
// share them. The vertical sum adds the new row and drops the one 2R+1 above
// from registers.
//
// The score decides as in ncc_match_kernel: the thread's 4 disparities by an
// estimate with a relative error of about 1e-6, the IEEE score for those within
// 1e-5 of the best estimate, and only where that comes within 1e-5 of the
// pixel's best score so far.
//
// What bounds it: instructions and their latency with 14 warps an SM (67% of
// the issue slots, the ALU 51%). A row of 4 disparities takes 47 instructions a
// disparity; with 26 rows for 16 and ranges filled up to 16 disparities that is
// 112 a searched pixel and disparity. At 1920x1080 (slanted planes, D = 128, 11
// x 11: 13 disparities a pixel) the launch of 8160 blocks takes 156 us, against
// 448 us for the wide tiles.
//
// Every guided call runs here. Its time grows with the blocks' own ranges, that
// of the wide tiles with their union; whole calls at 1920x1080, D = 128, 11 x 11
// (here / wide tiles, two scenes): checked coarse maps 168 / 424 and 168 / 443
// us, unchecked ones 190 / 450 and 211 / 467, uniform noise for a coarse map
// (every block searches nearly everything) 610 / 690 and 622 / 690. With noise
// the wide tiles, whose passes hold 64 disparities, are ahead at D = 64 only
// (346 / 340, 356 / 341), and unguided matching (440 us) is from D = 128: no
// line is drawn for a coarse map that says nothing.
#pragma once

namespace ct {
namespace ncc {
namespace gd {

constexpr int kB = guide::kBlock;   // pixels a side
constexpr int kThreads = 64;
constexpr int kDT = 4;              // disparities a thread
constexpr int kDC = 32;             // disparities staged at a time
constexpr int kPass = kThreads / kB * kDT;  // disparities the CTA matches at a time
static_assert(kB == 16 && kDC % kPass == 0, "block mapping");

constexpr int kLW = 8, kRW = 16;    // staged words a row: left view from x0 - 8, right view of a chunk

// The aligned word at column xa (a multiple of 4) of row y; columns and rows
// outside the image read some pixel inside it (only windows that leave the
// image meet them). Rows are padded to whole words.
__device__ __forceinline__ uint32_t word_at(const uint8_t* img, size_t pitch, int xa, int y, int W, int H) {
    const int yc = min(max(y, 0), H - 1), xc = min(max(xa, 0), (W - 1) & ~3);
    return __ldg(reinterpret_cast<const uint32_t*>(img + size_t(yc) * pitch + xc));
}

}  // namespace gd

template <int R>
__global__ void __launch_bounds__(gd::kThreads)
    ncc_guided_kernel(const uint8_t* __restrict__ Limg, size_t pl, const uint8_t* __restrict__ Rimg, size_t pr, Args a) {
    using namespace gd;
    constexpr int K = 2 * R + 1, n = K * K, NW = (K + 3) / 4, NR = kB + 2 * R;
    constexpr int NS = kB - 1 + kDC;  // right-view columns with statistics
    constexpr uint32_t kLast = 0xFFFFFFFFu >> (8 * (4 * NW - K));  // the last word's pixels inside the window
    static_assert(R <= 8 && kB + 7 + 4 * NW - R <= 4 * kLW, "the left words cover the block's windows");
    static_assert(kB - 1 + kDC - kDT + 4 * NW + 3 + 4 <= 4 * kRW, "the right words cover a chunk's windows");
    __shared__ uint32_t sl[NR][kLW];
    __shared__ uint32_t sr[NR][kRW];
    __shared__ int2 ss[kB][NS];        // right view: Sy, vy
    __shared__ int4 sp[kB][kB];        // left view: Sx, Tx, ~1 / sqrt(vx), float(vx)
    __shared__ int4 ring[K][kThreads];  // the last K rows' parts of a thread's 4 windows
    __shared__ float bs[kThreads / kB][kB][kB];  // each 4 disparities' best score of a pixel
    __shared__ int bd[kThreads / kB][kB][kB];    // and its disparity (-1: none)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int x0 = blockIdx.x * kB, y0 = blockIdx.y * kB;
    const uint32_t g = a.guide[(size_t)blockIdx.y * a.guide_gw + blockIdx.x];
    const int lo = int(g & 0xFFFFu), hi = min(int(g >> 16), a.D - 1);

#pragma unroll
    for (int i = tid; i < kThreads / kB * kB * kB; i += kThreads) {
        (&bs[0][0][0])[i] = -INFINITY;
        (&bd[0][0][0])[i] = -1;
    }
    if (lo <= hi) {
#pragma unroll
        for (int i = tid; i < NR * kLW; i += kThreads)
            sl[i / kLW][i % kLW] = word_at(Limg, pl, x0 - 8 + 4 * (i % kLW), y0 - R + i / kLW, a.W, a.H);
#pragma unroll
        for (int i = tid; i < kB * kB; i += kThreads) {
            const int x = min(x0 + i % kB, a.W - 1), y = min(y0 + i / kB, a.H - 1);
            const size_t o = (size_t)y * a.W + x;
            const float fvx = __int2float_rn(a.Vx[o]);
            sp[i / kB][i % kB] = make_int4(a.Sx[o], a.Tx[o], __float_as_int(rsqrtf(fvx)), __float_as_int(fvx));
        }
    }
    const int xi = lane & (kB - 1), x = x0 + xi;
    const int dt = kDT * (2 * warp + (lane >> 4));  // the thread's first disparity of a pass
    const int grp = 2 * warp + (lane >> 4);
    const bool xin = x >= R && x < a.W - R;
    for (int c0 = lo; c0 <= hi; c0 += kDC) {
        __syncthreads();  // the chunk before is matched
        const int xr0 = x0 - a.dmin - c0 - (kDC - 1);  // first right-view column of the chunk
        const int rb = (xr0 - R) & ~3;                 // column of its first word
#pragma unroll
        for (int i = tid; i < NR * kRW; i += kThreads)
            sr[i / kRW][i % kRW] = word_at(Rimg, pr, rb + 4 * (i % kRW), y0 - R + i / kRW, a.W, a.H);
#pragma unroll
        for (int i = tid; i < kB * NS; i += kThreads) {
            const int c = i % NS, r = i / NS, y = min(y0 + r, a.H - 1), xr = min(max(xr0 + c, 0), a.W - 1);
            const size_t o = (size_t)y * a.W + xr;
            ss[r][c] = make_int2(a.Sy[o], a.Vy[o]);
        }
        __syncthreads();
        for (int p = 0; p < kDC; p += kPass) {
            const int d0 = c0 + p + dt;  // its disparities d0 .. d0 + 3, relative to dmin
            // searched: in the block's range, the matched window inside the image
            const int dmax = min(hi, x - a.dmin - R);
            const int nd = xin ? min(max(dmax - d0 + 1, 0), kDT) : 0;
            if (!__any_sync(0xffffffffu, nd > 0)) continue;
            // column of disparity d0 + 3 in ss; first byte of its window in sr,
            // of the pixel's in sl
            const int col = xi + (kDC - 1) - (p + dt) - (kDT - 1);
            const int br = xr0 - R + col - rb, bl = xi + 8 - R;
            const uint32_t shr = 8 * (br & 3), shl = 8 * (bl & 3);
            int V[kDT] = {};
            // Rows are a loop, the window's rows and the best scores live in
            // shared memory: unrolled with both in registers the code was 26
            // rows long and the warps waited for instructions (222 us where
            // this takes 167).
            int slot = 0;
#pragma unroll 1
            for (int r = 0; r < NR; ++r) {
                uint32_t A[NW + 1], B[NW];
                {
                    const uint32_t* q = &sr[r][br >> 2];
                    uint32_t w0 = q[0];
#pragma unroll
                    for (int w = 0; w <= NW; ++w) {
                        const uint32_t w1 = q[w + 1];
                        A[w] = __funnelshift_r(w0, w1, shr);
                        w0 = w1;
                    }
                    const uint32_t* l = &sl[r][bl >> 2];
                    w0 = l[0];
#pragma unroll
                    for (int w = 0; w < NW; ++w) {
                        const uint32_t w1 = l[w + 1];
                        B[w] = __funnelshift_r(w0, w1, shl);
                        w0 = w1;
                    }
                    B[NW - 1] &= kLast;
                }
                int H[kDT];
#pragma unroll
                for (int k = 0; k < kDT; ++k) {
                    uint32_t h = 0;
#pragma unroll
                    for (int w = 0; w < NW; ++w) h = __dp4a(B[w], __funnelshift_r(A[w], A[w + 1], 8 * (kDT - 1 - k)), h);
                    H[k] = int(h);
                    V[k] += H[k];
                }
                if (r >= K) {
                    const int4 o = ring[slot][tid];
                    V[0] -= o.x; V[1] -= o.y; V[2] -= o.z; V[3] -= o.w;
                }
                ring[slot][tid] = make_int4(H[0], H[1], H[2], H[3]);
                slot = slot + 1 < K ? slot + 1 : 0;
                if (r < 2 * R) continue;
                const int y = r - 2 * R;  // the block's row whose windows end here
                const int4 px = sp[y][xi];
                float best = bs[grp][y][xi];
                int num[kDT], vy[kDT];
                float e[kDT];
                float emax = -INFINITY;
#pragma unroll
                for (int k = 0; k < kDT; ++k) {
                    const int2 st = ss[y][col + (kDT - 1 - k)];
                    num[k] = n * V[k] - px.x * st.x;
                    vy[k] = st.y;
                    // 0 when sigma_x sigma_y < 1 (the score is +0 then, and
                    // only then or for num = 0)
                    e[k] = st.y >= px.y ? __int2float_rn(num[k]) * rsqrtf(__int2float_rn(st.y)) : 0.0f;
                    e[k] = k < nd ? e[k] : -INFINITY;
                    emax = fmaxf(emax, e[k]);
                }
                // (in the estimate's scale: times sqrt(vx))
                const float es = emax * __int_as_float(px.z);
                if (nd > 0 && (emax == 0.0f ? 0.0f > best : es >= best - fabsf(best) * 1e-5f)) {
                    const float thr = emax - fabsf(emax) * 1e-5f;
                    auto score = [&](int nk, int vk) {
                        return vk >= px.y ? __fdiv_rn(__int2float_rn(nk), __fsqrt_rn(__fmul_rn(__int_as_float(px.w),
                                                                                               __int2float_rn(vk))))
                                          : 0.0f;
                    };
                    auto take = [&](float sc, int d) {
                        if (sc > best) {  // disparities in order: the lowest of equals stays
                            best = sc;
                            bs[grp][y][xi] = sc;
                            bd[grp][y][xi] = d;
                        }
                    };
                    // the lowest disparity near the thread's best estimate,
                    // then, rarely, the others near it
                    int k1 = kDT - 1, n1 = num[kDT - 1], v1 = vy[kDT - 1];
                    uint32_t near = e[kDT - 1] >= thr ? 1u << (kDT - 1) : 0u;
#pragma unroll
                    for (int k = kDT - 2; k >= 0; --k)
                        if (e[k] >= thr) {
                            k1 = k;
                            n1 = num[k];
                            v1 = vy[k];
                            near |= 1u << k;
                        }
                    take(score(n1, v1), d0 + k1);
                    near &= near - 1;
                    if (near && emax != 0.0f)
#pragma unroll
                        for (int k = 1; k < kDT; ++k)
                            if ((near >> k) & 1u) take(score(num[k], vy[k]), d0 + k);
                }
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < kB * kB; i += kThreads) {
        const int px = x0 + i % kB, py = y0 + i / kB;
        unsigned long long key = 0ull;
#pragma unroll
        for (int q = 0; q < kThreads / kB; ++q) {
            const int d = bd[q][i / kB][i % kB];
            const unsigned long long k2 =
                d < 0 ? 0ull : ((unsigned long long)ordered(bs[q][i / kB][i % kB]) << 32) | (0xFFFFFFFFu - uint32_t(d));
            key = k2 > key ? k2 : key;
        }
        if (px < a.W && py < a.H)
            store_ncc(a, px, py, px >= R && px < a.W - R && py >= R && py < a.H - R, key);
    }
}

}  // namespace ncc
}  // namespace ct
