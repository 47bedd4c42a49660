// batch.cu — census stereo (both directions + cross-check) for many pairs of
// mixed sizes and disparity ranges in one persistent, work-queue-scheduled
// matching launch, replayable as a CUDA graph.
//
// Per process call, on one stream:
//   1. a copy of the per-call pair table (caller image tensor maps, output
//      pointers) from pinned host memory, and a memset of the queue counter;
//   2. one census launch: every CTA is one 64 x 32 census tile of one image of
//      one pair (census_tile.cuh), found by a scan of per-pair prefix counts;
//   3. one persistent matching launch, one CTA per SM: each CTA takes work
//      items (pair, strip, tile pair) from a global atomic counter, the
//      longest first, and runs the tensor-core census tile (census_tc.cuh: the
//      left map, and the right view's winners bid into the pair's right-view
//      key plane) on the pair's descriptors;
//   4. one cross-check launch, a CTA a row of a pair: the caller's map from the
//      left map and the right-view keys, which it then resets.
// Results are bit-identical to processing each pair alone: every tile's
// arithmetic is the same and the winner-take-all keys are order-free.
#include "ct_internal.h"
#include "ct_device.cuh"
#include "census_match.cuh"
#include "census_tc.cuh"
#include "census_tile.cuh"

#include <algorithm>
#include <functional>
#include <map>
#include <queue>
#include <tuple>
#include <vector>

namespace ct {
namespace batch {

constexpr int kMaxPairs = 256;

// Device-side description of one pair (fixed at configure, except the
// per-call fields at the end, rewritten by every process call).
struct PairDev {
    int W, H, D, th, tiles_x, strips, tol;
    int mo, n, lstep, rstep;                 // tile pair (ctc::Shape)
    int census_tx, census_ty, census_item0;  // census tiles per image, prefix over census CTAs
    int match_item0, match_items;            // prefix over matching items
    int row0;                                // prefix over rows
    uint64_t* desc[2];                       // row-major descriptors: left, right
    size_t desc_pitch;                       // elements
    uint16_t* map;                           // U16 left-to-right disparity map
    size_t map_pitch;                        // bytes
    uint32_t* rl_keys;                       // right-view keys (kTag), 0 between calls
    size_t rl_pitch;                         // words
    // per call
    void* out;
    size_t out_pitch;
    int out_type;
    int pad;
};

constexpr uint32_t kTag = 1u << cm::kRLTagShift;

// Per-call tensor maps of the caller's images, 64-byte aligned in device memory.
struct alignas(64) CallMaps {
    CUtensorMap img[2];  // left, right
};

__device__ __forceinline__ void tmap_acquire(const CUtensorMap* m) {
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(reinterpret_cast<uint64_t>(m))
                 : "memory");
}

// Last pair whose first item (PairDev member FIRST) is <= item.
template <int PairDev::*FIRST>
__device__ __forceinline__ int find_pair(const PairDev* pairs, int n, int item) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pairs[mid].*FIRST <= item) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(census::kNT) census_batch_kernel(const PairDev* pairs, int n,
                                                                    const CallMaps* maps, int32_t* status) {
    __shared__ __align__(128) census::TileSmem sm;
    const int item = blockIdx.x;
    const int p = find_pair<&PairDev::census_item0>(pairs, n, item);
    const PairDev& P = pairs[p];
    const int local = item - P.census_item0;
    const int per_img = P.census_tx * P.census_ty;
    if (local < 0 || local >= 2 * per_img) {  // table inconsistent with the grid
        if (threadIdx.x == 0) dev::report(status, CT_EINTERNAL);
        return;
    }
    const int img = local / per_img, t = local % per_img;
    const CUtensorMap* tm = &maps[p].img[img];
    if (threadIdx.x == 0) tmap_acquire(tm);
    __syncthreads();
    census::census_tile(tm, P.W, P.H, (t % P.census_tx) * census::kTX, (t / P.census_tx) * census::kTY,
                        P.desc[img], P.desc_pitch, 0, status, sm);
}

// Cross-check of one row of a pair from its U16 left map and the right-view
// keys into the caller's map (CrossCheckDisparityMaps.cu:63-110 rule,
// left-to-right: the right view's code at x - d, as its map would hold it,
// within tol of the left code), 8 pixels a thread; then the row's keys are
// reset. A launch of its own: run by the matching CTA that finished a strip,
// it kept that CTA's tensor core idle for a strip's dependent loads.
constexpr int kCheckT = 128;
__global__ void __launch_bounds__(kCheckT) check_batch_kernel(const PairDev* pairs, int n) {
    const int p = find_pair<&PairDev::row0>(pairs, n, blockIdx.x);
    const PairDev& P = pairs[p];
    const int W = P.W, y = blockIdx.x - P.row0;
    const bool yin = y >= cm::kAR && y < P.H - cm::kAR;
    const cm::MaxKeys how{kTag, 0};
    const uint16_t* map = reinterpret_cast<const uint16_t*>(reinterpret_cast<const char*>(P.map) + (size_t)y * P.map_pitch);
    uint32_t* keys = P.rl_keys + (size_t)y * P.rl_pitch;
    char* row = static_cast<char*>(P.out) + (size_t)y * P.out_pitch;
    for (int x0 = 8 * threadIdx.x; x0 < W; x0 += 8 * kCheckT) {
        // the map's and the caller's rows are 16-byte aligned; the map's pitch
        // is a multiple of 256
        const uint4 q = *reinterpret_cast<const uint4*>(map + x0);
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        uint32_t o16[4] = {0, 0, 0, 0}, o8[2] = {0, 0};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint16_t v = uint16_t(w[i >> 1] >> (16 * (i & 1)));
            const bool disp = v >= CT_DISP_FIRST && v <= CT_DISP_LAST && x0 + i < W;
            const int xo = x0 + i - (int(v) - 1);
            bool keep = false;
            if (disp && xo >= 0 && xo < W) {
                const uint16_t vo = how.code<uint16_t>(keys[xo], yin && xo >= cm::kAR && xo < W - cm::kAR);
                keep = abs(int(vo) - int(v)) <= P.tol;  // raw codes, CrossCheckDisparityMaps.cu:94
            }
            o16[i >> 1] |= uint32_t(keep ? v : (disp ? uint16_t(CT_DISP_INCONSISTENT) : v)) << (16 * (i & 1));
            o8[i >> 2] |= uint32_t(keep ? uint8_t(v - 1) : uint8_t(0xFF)) << (8 * (i & 3));
        }
        if (P.out_type == CT_PIX_U8) {
            uint8_t* o = reinterpret_cast<uint8_t*>(row) + x0;
            if (x0 + 8 <= W) *reinterpret_cast<uint2*>(o) = make_uint2(o8[0], o8[1]);
            else
                for (int i = 0; x0 + i < W; ++i) o[i] = uint8_t(o8[i >> 2] >> (8 * (i & 3)));
        } else {
            uint16_t* o = reinterpret_cast<uint16_t*>(row) + x0;
            if (x0 + 8 <= W) *reinterpret_cast<uint4*>(o) = make_uint4(o16[0], o16[1], o16[2], o16[3]);
            else
                for (int i = 0; x0 + i < W; ++i) o[i] = uint16_t(o16[i >> 1] >> (16 * (i & 1)));
        }
    }
    __syncthreads();  // every read of the row's keys done
    for (int i = 4 * threadIdx.x; i < int(P.rl_pitch); i += 4 * kCheckT)
        *reinterpret_cast<uint4*>(keys + i) = make_uint4(0, 0, 0, 0);
}

__global__ void __launch_bounds__(ctc::kNT, 1)
    match_batch_kernel(const PairDev* pairs, int n, int total_items, unsigned* queue, uint32_t polls, int32_t* status) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ int s_item;
    ctc::Cta c(smem_raw);
    ctc::cta_begin(c);
    const int tid = threadIdx.x;
    for (;;) {
        if (tid == 0) s_item = int(atomicAdd(queue, 1u));
        __syncthreads();
        const int item = s_item;
        __syncthreads();
        if (item >= total_items) break;
        const int p = find_pair<&PairDev::match_item0>(pairs, n, item);
        const PairDev& P = pairs[p];
        const int local = item - P.match_item0;
        if (local < 0 || local >= P.match_items || P.match_items != P.strips * P.tiles_x) {
            if (tid == 0) dev::report(status, CT_EINTERNAL);  // table inconsistent
            break;
        }
        const int by = local / P.tiles_x;
        ctc::Args a{};
        a.W = P.W; a.H = P.H; a.D = P.D;
        a.mo = P.mo; a.n = P.n; a.th = P.th;
        a.lstep = P.lstep; a.rstep = P.rstep;
        a.left = P.desc[0]; a.right = P.desc[1];
        a.pitch = P.desc_pitch;
        a.out = P.map; a.out_pitch = P.map_pitch; a.out_type = CT_PIX_U16;
        a.r_keys = P.rl_keys;
        a.key_pitch = P.rl_pitch;
        a.tag = kTag;
        a.status = status;
        a.polls = polls;
        if (!ctc::run_tile(c, a, local % P.tiles_x, by)) break;  // status already set; the CTA takes no more work
    }
    ctc::cta_end(c);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
// Pinned host staging of one call's pair table and image tensor maps. The
// host rewrites a slot only after the copies that read it have run (event
// `copied`, recorded behind them): cuTensorMapEncodeTiled does not write a
// descriptor in one store, so a copy racing a rewrite could deliver a torn
// tensor map even when the new bytes equal the old ones.
struct Staging {
    PairDev* pairs = nullptr;
    CallMaps* maps = nullptr;
    cudaEvent_t copied = nullptr;
    bool pending = false;  // `copied` recorded and not yet waited for
    int wait() {
        if (pending) CT_CUDA_TRY(cudaEventSynchronize(copied));
        pending = false;
        return CT_OK;
    }
    int alloc(int n) {
        if (!copied) CT_CUDA_TRY(cudaEventCreateWithFlags(&copied, cudaEventDisableTiming));
        release_host();
        CT_CUDA_TRY(cudaMallocHost(&pairs, sizeof(PairDev) * n));
        CT_CUDA_TRY(cudaMallocHost(&maps, sizeof(CallMaps) * n));
        return CT_OK;
    }
    void release_host() {
        wait();
        cudaFreeHost(pairs);
        cudaFreeHost(maps);
        pairs = nullptr;
        maps = nullptr;
    }
    void release() {
        release_host();
        if (copied) cudaEventDestroy(copied);
        copied = nullptr;
    }
};

// Staging slots used in turn by process calls, so the host fills call k + 1
// while the copies of call k are still queued behind earlier work.
constexpr int kSlots = 3;

struct BatchHandle : ct_handle {
    BatchHandle() : ct_handle(Kind::Batch) {}
    ~BatchHandle() override {
        if (device >= 0) cudaSetDevice(device);
        if (graph_exec) cudaGraphExecDestroy(graph_exec);
        for (Staging& st : stage) st.release();
        graph_stage.release();
        cudaFree(arena);
    }
    int n = 0;
    int tol = 1;
    std::vector<ct_batch_shape> shapes;
    std::vector<PairDev> pairs;          // host copy (per-call fields filled per call)
    std::vector<int> order;              // pair index -> position in the device table
    int total_census = 0, total_match = 0, total_rows = 0;
    unsigned char* arena = nullptr;      // one device allocation for all scratch
    PairDev* d_pairs = nullptr;
    CallMaps* d_maps = nullptr;
    unsigned* d_queue = nullptr;
    Staging stage[kSlots];               // process calls
    int next_slot = 0;
    Staging graph_stage;                 // snapshot read by every graph launch; `copied`
                                         // is recorded behind each launch
    cudaGraphExec_t graph_exec = nullptr;
    int sms = 148;
};

int fill_call(BatchHandle* h, const ct_batch_item* items, int n, PairDev* pd, CallMaps* cm_) {
    if (n != h->n) return fail(CT_EFORMAT, "item count %d differs from the configured %d", n, h->n);
    for (int i = 0; i < n; ++i) {
        const ct_batch_item& it = items[i];
        const ct_batch_shape& s = h->shapes[i];
        if (int rc = check_image(&it.left, "left", 1u << CT_PIX_U8)) return rc;
        if (int rc = check_image(&it.right, "right", 1u << CT_PIX_U8)) return rc;
        if (int rc = check_image(&it.disp, "disp", (1u << CT_PIX_U8) | (1u << CT_PIX_U16))) return rc;
        if (it.left.width != s.width || it.left.height != s.height || it.right.width != s.width ||
            it.right.height != s.height || it.disp.width != s.width || it.disp.height != s.height)
            return fail(CT_EFORMAT, "pair %d: image sizes differ from the configured shape", i);
        if (it.disp.type == CT_PIX_U8 && s.disp_count > 255)
            return fail(CT_ETYPE, "pair %d: U8 maps need disp_count <= 255", i);
        const int slot = h->order[i];
        PairDev& P = pd[slot];
        P = h->pairs[slot];
        P.out = it.disp.ptr;
        P.out_pitch = it.disp.pitch_bytes;
        P.out_type = it.disp.type;
        const ct_image* im[2] = {&it.left, &it.right};
        for (int k = 0; k < 2; ++k)
            if (int rc = make_tmap_2d(&cm_[slot].img[k], im[k]->ptr, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, s.width,
                                      s.height, im[k]->pitch_bytes, census::kBoxW, census::kBoxH))
                return rc;
    }
    return CT_OK;
}

// Enqueues one call: table copies from `st` (its event recorded behind them
// unless `record` is false, as inside a stream capture), queue reset, census
// launch, matching launch.
int enqueue(BatchHandle* h, Staging& st, bool record, cudaStream_t s) {
    CT_CUDA_TRY(cudaMemcpyAsync(h->d_pairs, st.pairs, sizeof(PairDev) * h->n, cudaMemcpyHostToDevice, s));
    CT_CUDA_TRY(cudaMemcpyAsync(h->d_maps, st.maps, sizeof(CallMaps) * h->n, cudaMemcpyHostToDevice, s));
    if (record) {
        CT_CUDA_TRY(cudaEventRecord(st.copied, s));
        st.pending = true;
    }
    CT_CUDA_TRY(cudaMemsetAsync(h->d_queue, 0, sizeof(unsigned), s));
    census_batch_kernel<<<h->total_census, census::kNT, 0, s>>>(h->d_pairs, h->n, h->d_maps, h->d_status);
    CT_LAUNCH_CHECK();
    match_batch_kernel<<<std::min(h->sms, h->total_match), ctc::kNT, ctc::kSmemBytes, s>>>(
        h->d_pairs, h->n, h->total_match, h->d_queue, h->wait_polls, h->d_status);
    CT_LAUNCH_CHECK();
    check_batch_kernel<<<h->total_rows, kCheckT, 0, s>>>(h->d_pairs, h->n);
    CT_LAUNCH_CHECK();
    return CT_OK;
}

// Strip heights keep the form 5 k + 1 that callers of ct_batch_strip_height know.
constexpr int strip_form(int th) { return th + (6 - th % 5) % 5; }

// Strip heights: the same target for every pair, the one whose items finish
// first when handed out longest first. An item takes its rows, the first
// window and the start of its pipeline (about 7 rows' worth) times the tile
// pair's cost of a row. With very many items their order no longer matters and
// tall strips repeat fewer rows.
std::vector<int> pick_strips(const std::vector<ct_batch_shape>& shapes, int sms) {
    const int n = int(shapes.size());
    std::vector<ctc::Shape> sh(n);
    for (int i = 0; i < n; ++i) sh[i] = ctc::pick_shape(shapes[i].width, shapes[i].disp_count);
    std::vector<int> best(n), th(n);
    double best_time = -1;
    for (int target : {8, 12, 16, 24, 32, 48, 64, 80, 96, 128, 160, 192, 256}) {
        std::vector<std::pair<double, long>> items;  // cost, how many
        long count = 0;
        double total = 0;
        for (int i = 0; i < n; ++i) {
            const int strips = (shapes[i].height + target - 1) / target;
            th[i] = strip_form((shapes[i].height + strips - 1) / strips);
            const double cost = (std::min(th[i], shapes[i].height) + 7) * sh[i].row_cost;
            const long k = long((shapes[i].height + th[i] - 1) / th[i]) * sh[i].tiles_x;
            items.push_back({cost, k});
            count += k;
            total += cost * k;
        }
        double time = total / sms;
        if (count <= 64L * sms) {
            std::sort(items.begin(), items.end(), std::greater<>());
            std::priority_queue<double, std::vector<double>, std::greater<>> cta;
            for (int k = 0; k < sms; ++k) cta.push(0.0);
            for (auto& it : items)
                for (long k = 0; k < it.second; ++k) {
                    const double t = cta.top() + it.first;
                    cta.pop();
                    cta.push(t);
                    time = std::max(time, t);
                }
        }
        if (best_time < 0 || time < best_time) {
            best_time = time;
            best = th;
        }
    }
    return best;
}

// Lays out the table (longest items first), item prefixes and scratch for the
// current shapes and strip heights.
int layout(BatchHandle* h, const std::vector<int>& th) {
    const int n = h->n;
    std::vector<int> idx(n);
    for (int i = 0; i < n; ++i) idx[i] = i;
    auto cost = [&](int i) {
        return (std::min(th[i], h->shapes[i].height) + 7) *
               ctc::pick_shape(h->shapes[i].width, h->shapes[i].disp_count).row_cost;
    };
    std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) { return cost(a) > cost(b); });
    h->order.assign(n, 0);
    for (int k = 0; k < n; ++k) h->order[idx[k]] = k;
    // sizes
    size_t bytes = 0;
    auto take = [&](size_t b) { const size_t o = bytes; bytes += (b + 255) / 256 * 256; return o; };
    struct Off { size_t desc[2], map, rl; };
    std::vector<Off> off(n);
    h->pairs.assign(n, PairDev{});
    int census0 = 0, match0 = 0, row0 = 0;
    for (int k = 0; k < n; ++k) {
        const int i = idx[k];
        const ct_batch_shape& s = h->shapes[i];
        PairDev& P = h->pairs[k];
        P.W = s.width; P.H = s.height; P.D = s.disp_count; P.th = th[i];
        const ctc::Shape shape = ctc::pick_shape(P.W, P.D);
        P.mo = shape.mo; P.n = shape.n; P.lstep = shape.lstep; P.rstep = shape.rstep;
        P.tiles_x = shape.tiles_x;
        P.strips = (P.H + P.th - 1) / P.th;
        P.tol = h->tol;
        P.census_tx = (P.W + census::kTX - 1) / census::kTX;
        P.census_ty = (P.H + census::kTY - 1) / census::kTY;
        P.census_item0 = census0;
        census0 += 2 * P.census_tx * P.census_ty;
        P.match_item0 = match0;
        P.match_items = P.strips * P.tiles_x;
        match0 += P.match_items;
        P.row0 = row0;
        row0 += P.H;
        P.map_pitch = ((size_t)P.W * 2 + 255) / 256 * 256;
        Off& o = off[k];
        P.desc_pitch = ((size_t)P.W + 1) / 2 * 2;  // 16-byte rows
        for (int v = 0; v < 2; ++v) o.desc[v] = take(P.desc_pitch * P.H * 8);
        o.map = take(P.map_pitch * P.H);
        P.rl_pitch = cm::rl_pitch_words(P.W);
        o.rl = take(P.rl_pitch * P.H * 4);
    }
    const size_t o_pairs = take(sizeof(PairDev) * n), o_maps = take(sizeof(CallMaps) * n);
    const size_t o_queue = take(256);
    cudaFree(h->arena);
    h->arena = nullptr;
    if (cudaMalloc(&h->arena, bytes) != cudaSuccess) return fail(CT_ENOMEM, "batch scratch (%zu bytes)", bytes);
    CT_CUDA_TRY(cudaMemset(h->arena, 0, bytes));  // right-view keys start at 0
    unsigned char* A = h->arena;
    for (int k = 0; k < n; ++k) {
        PairDev& P = h->pairs[k];
        for (int v = 0; v < 2; ++v) P.desc[v] = reinterpret_cast<uint64_t*>(A + off[k].desc[v]);
        P.map = reinterpret_cast<uint16_t*>(A + off[k].map);
        P.rl_keys = reinterpret_cast<uint32_t*>(A + off[k].rl);
    }
    h->d_pairs = reinterpret_cast<PairDev*>(A + o_pairs);
    h->d_maps = reinterpret_cast<CallMaps*>(A + o_maps);
    h->d_queue = reinterpret_cast<unsigned*>(A + o_queue);
    h->total_census = census0;
    h->total_match = match0;
    h->total_rows = row0;
    if (h->graph_exec) {
        cudaGraphExecDestroy(h->graph_exec);
        h->graph_exec = nullptr;
    }
    return CT_OK;
}

BatchHandle* as_batch(ct_handle* h) { return (h && h->kind == Kind::Batch) ? static_cast<BatchHandle*>(h) : nullptr; }

}  // namespace batch
}  // namespace ct

using namespace ct;
using namespace ct::batch;

extern "C" {

int ct_batch_create(ct_handle** out) {
    clear_error();
    if (!out) return fail(CT_EINVAL, "null output handle pointer");
    *out = new BatchHandle();
    return CT_OK;
}

int ct_batch_configure(ct_handle* hh, int32_t device, const ct_batch_shape* shapes, int32_t n, int32_t tol) {
    clear_error();
    auto* h = as_batch(hh);
    if (!h) return fail(CT_ESTATE, "not a batch handle");
    if (!shapes || n < 1 || n > kMaxPairs) return fail(CT_EINVAL, "need 1..%d pair shapes", kMaxPairs);
    if (tol < 0) return fail(CT_EINVAL, "tol must be >= 0");
    for (int i = 0; i < n; ++i) {
        const ct_batch_shape& s = shapes[i];
        if (s.width < 8 || s.height < 8 || s.width > 32768 || s.height > 32768)
            return fail(CT_EINVAL, "pair %d: size %dx%d out of range", i, s.width, s.height);
        if (s.disp_count < 1 || s.disp_count > 256) return fail(CT_EINVAL, "pair %d: disp_count must be 1..256", i);
    }
    if (int rc = use_device(device)) return rc;
    h->device = device;
    if (int rc = h->init_status()) return rc;
    CT_CUDA_TRY(cudaFuncSetAttribute(match_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     ctc::kSmemBytes));
    h->sms = sm_count(device);
    h->n = n;
    h->tol = tol;
    h->shapes.assign(shapes, shapes + n);
    const std::vector<int> th = pick_strips(h->shapes, h->sms);
    if (int rc = layout(h, th)) return rc;
    for (Staging& st : h->stage)
        if (int rc = st.alloc(n)) return rc;
    h->configured = true;
    return CT_OK;
}

int ct_batch_process(ct_handle* hh, const ct_batch_item* items, int32_t n, ct_stream stream) {
    clear_error();
    auto* h = as_batch(hh);
    if (!h) return fail(CT_ESTATE, "not a batch handle");
    if (!h->configured) return fail(CT_ESTATE, "process before configure");
    if (!items) return fail(CT_EINVAL, "null items");
    if (int rc = use_device(h->device)) return rc;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    h->last_stream = s;
    Staging& st = h->stage[h->next_slot];
    if (int rc = st.wait()) return rc;  // the slot may still feed a copy of an earlier call
    if (int rc = fill_call(h, items, n, st.pairs, st.maps)) return rc;
    h->next_slot = (h->next_slot + 1) % kSlots;
    return enqueue(h, st, true, s);
}

int ct_batch_autotune(ct_handle* hh, const ct_batch_item* items, int32_t n, ct_stream stream) {
    clear_error();
    auto* h = as_batch(hh);
    if (!h) return fail(CT_ESTATE, "not a batch handle");
    if (!h->configured) return fail(CT_ESTATE, "autotune before configure");
    if (!items) return fail(CT_EINVAL, "null items");
    if (int rc = use_device(h->device)) return rc;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    // current strip heights by original pair index
    std::vector<int> th(h->n);
    for (int i = 0; i < h->n; ++i) th[i] = h->pairs[h->order[i]].th;
    // distinct (W, H, D) shapes
    std::map<std::tuple<int, int, int>, std::vector<int>> groups;
    for (int i = 0; i < h->n; ++i)
        groups[{h->shapes[i].width, h->shapes[i].height, h->shapes[i].disp_count}].push_back(i);
    cudaEvent_t e0, e1;
    CT_CUDA_TRY(cudaEventCreate(&e0));
    CT_CUDA_TRY(cudaEventCreate(&e1));
    auto time_batch = [&](float* ms_out) -> int {
        float best = 1e30f;
        for (int rep = 0; rep < 3; ++rep) {
            if (int rc = ct_batch_process(hh, items, n, stream)) return rc;
            cudaEventRecord(e0, s);
            if (int rc = ct_batch_process(hh, items, n, stream)) return rc;
            cudaEventRecord(e1, s);
            const cudaError_t e = cudaEventSynchronize(e1);
            if (e != cudaSuccess) return fail(CT_ECUDA, "autotune timing failed: %s", cudaGetErrorString(e));
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            best = std::min(best, ms);
        }
        *ms_out = best;
        return CT_OK;
    };
    int rc = CT_OK;
    float cur = 0.f;
    if ((rc = time_batch(&cur))) goto done;
    // one pass of coordinate descent over the shapes' strip heights
    for (auto& g : groups) {
        const int base = th[g.second[0]];
        int best_th = base;
        for (int cand : {strip_form(base / 2), strip_form(base * 2), strip_form(base * 3 / 2), 31, 66}) {
            if (cand < 6 || cand > h->shapes[g.second[0]].height || cand == best_th) continue;
            for (int i : g.second) th[i] = cand;
            if ((rc = layout(h, th))) goto done;
            float t = 0.f;
            if ((rc = time_batch(&t))) goto done;
            if (t < cur) { cur = t; best_th = cand; }
        }
        for (int i : g.second) th[i] = best_th;
        if ((rc = layout(h, th))) goto done;
    }
done:
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return rc;
}

int ct_batch_strip_height(ct_handle* hh, int32_t pair, int32_t* strip_height) {
    clear_error();
    auto* h = as_batch(hh);
    if (!h || !h->configured) return fail(CT_ESTATE, "not a configured batch handle");
    if (pair < 0 || pair >= h->n || !strip_height) return fail(CT_EINVAL, "bad pair index");
    *strip_height = h->pairs[h->order[pair]].th;
    return CT_OK;
}

int ct_batch_graph_create(ct_handle* hh, const ct_batch_item* items, int32_t n) {
    clear_error();
    auto* h = as_batch(hh);
    if (!h) return fail(CT_ESTATE, "not a batch handle");
    if (!h->configured) return fail(CT_ESTATE, "graph before configure");
    if (!items) return fail(CT_EINVAL, "null items");
    if (int rc = use_device(h->device)) return rc;
    if (h->graph_exec) {
        cudaGraphExecDestroy(h->graph_exec);
        h->graph_exec = nullptr;
    }
    if (!h->graph_stage.pairs) {
        if (int rc = h->graph_stage.alloc(kMaxPairs)) return rc;
    }
    if (int rc = h->graph_stage.wait()) return rc;  // earlier launches read the snapshot
    if (int rc = fill_call(h, items, n, h->graph_stage.pairs, h->graph_stage.maps)) return rc;
    cudaStream_t cs;
    CT_CUDA_TRY(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaGraph_t g = nullptr;
    int rc = CT_OK;
    if (cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        rc = fail(CT_ECUDA, "stream capture failed to begin");
    } else {
        rc = enqueue(h, h->graph_stage, false, cs);
        const cudaError_t e = cudaStreamEndCapture(cs, &g);
        if (!rc && e != cudaSuccess) rc = fail(CT_ECUDA, "stream capture failed: %s", cudaGetErrorString(e));
    }
    if (!rc && cudaGraphInstantiate(&h->graph_exec, g, 0) != cudaSuccess) rc = fail(CT_ECUDA, "graph instantiate failed");
    if (g) cudaGraphDestroy(g);
    cudaStreamDestroy(cs);
    return rc;
}

int ct_batch_graph_launch(ct_handle* hh, ct_stream stream) {
    clear_error();
    auto* h = as_batch(hh);
    if (!h || !h->graph_exec) return fail(CT_ESTATE, "no graph: call ct_batch_graph_create first");
    if (int rc = use_device(h->device)) return rc;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    h->last_stream = s;
    CT_CUDA_TRY(cudaGraphLaunch(h->graph_exec, s));
    CT_CUDA_TRY(cudaEventRecord(h->graph_stage.copied, s));
    h->graph_stage.pending = true;
    return CT_OK;
}

}  // extern "C"
