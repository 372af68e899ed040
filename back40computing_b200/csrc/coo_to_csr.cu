// COO -> CSR on the GPU: the conversion CsrGraph::FromCoo does on the host
// with a stable sort by row (csr_graph.cuh:109-152), as a stable LSD radix
// sort of the edges by row, then the row offsets from the sorted rows.  Within
// a row the edges keep their input order, so the result equals FromCoo's byte
// for byte.
//
// The digits are as wide as the fewest passes allow (at most 11 bits: rows
// below 2^11 take one pass, below 2^22 two, all others three).  Every pass cuts
// the input into one contiguous run of tiles per CTA:
//   digit_count  per-CTA digit counts, stored digit-major (hist[d * ctas + c]);
//   digit_scan   per digit, an exclusive scan over the CTAs and the digit's total;
//   scatter      every CTA walks its tiles in order, keeping the next output
//                slot of every digit in shared memory: a tile is ranked (counters
//                per warp, matching lanes where digits collide), regrouped by
//                digit in shared memory and written out in runs of equal digits.
// A pass reads 4 + 8 and writes 8 bytes per edge, mostly
// through L2; the ranking and its barriers, not that traffic, bound it.
// 16.8 M edges, 2^20 rows: 4.85 -> 0.53 ms a call (three 8-bit passes in steps
// of 256 edges behind CTA barriers, one global atomic per edge for the offsets
// and seven allocations, before).
#include <algorithm>
#include <mutex>

#include "problem.h"

namespace b40c {
namespace coo {

constexpr int kThreads = 512;  // digit counts
constexpr int kCtasPerSm = 2;
constexpr int kMaxDigitBits = 11;
constexpr int kMaxBins = 1 << kMaxDigitBits;
// Scatter tiles: one long tile per SM (1024 threads, 16 edges each), whose
// runs of equal digits fill whole sectors, or, for lists that would leave SMs
// idle that way, short ones (512 threads, 4 edges each).  16.8 M edges, 2^20
// rows: 533 us with long tiles of 16384 edges, 648 us with 8192; 1 M edges: 132
// us with long tiles, 100 us with short ones.
constexpr int kLongThreads = 1024, kLongPer = 16;
constexpr int kShortThreads = 512, kShortPer = 4;

// Digit counts of each CTA's tiles.  The first pass (cols given) also checks
// the ids: out of range sets *bad, after which no later kernel does anything.
__global__ void __launch_bounds__(kThreads) digit_count_kernel(const int32_t *keys, const int32_t *cols, int64_t m,
                                                               int32_t n, int shift, int bins, int64_t per_cta,
                                                               int32_t *hist, int32_t *bad)
{
    extern __shared__ int32_t count[];
    if (!cols && *bad) return;
    for (int d = threadIdx.x; d < bins; d += kThreads) count[d] = 0;
    __syncthreads();
    const int64_t b = (int64_t)blockIdx.x * per_cta, e = min(m, b + per_cta);
    constexpr int U = 8;
    for (int64_t i0 = b + threadIdx.x; i0 < e; i0 += (int64_t)U * kThreads) {
        int32_t k[U], c[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int64_t i = i0 + (int64_t)u * kThreads;
            k[u] = i < e ? keys[i] : 0;
            c[u] = (cols && i < e) ? cols[i] : 0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (i0 + (int64_t)u * kThreads < e) {
                if (cols && ((uint32_t)k[u] >= (uint32_t)n || (uint32_t)c[u] >= (uint32_t)n)) *bad = 1;
                atomicAdd(&count[(k[u] >> shift) & (bins - 1)], 1);
            }
        }
    }
    __syncthreads();
    for (int d = threadIdx.x; d < bins; d += kThreads) hist[(int64_t)d * gridDim.x + blockIdx.x] = count[d];
}

// One warp per digit: exclusive scan of its counts over the CTAs, in place,
// and the digit's total.
__global__ void digit_scan_kernel(int32_t *hist, int ctas, int bins, int32_t *totals)
{
    const int lane = threadIdx.x & 31, d = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (d >= bins) return;
    int32_t *row = hist + (int64_t)d * ctas;
    int carry = 0;
    for (int c0 = 0; c0 < ctas; c0 += 32) {
        const int c = c0 + lane;
        const int x = c < ctas ? row[c] : 0;
        int inc = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (c < ctas) row[c] = carry + inc - x;
        carry += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) totals[d] = carry;
}

// Exclusive scan, in place, of the CTA's `bins` shared counters (a multiple of
// 32, at most kMaxBins): each thread takes up to kMaxBins / THREADS
// neighbouring ones.
template <int THREADS>
__device__ __forceinline__ void scan_bins(int32_t *x, int bins, int32_t *warp_sums)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per = (bins + THREADS - 1) / THREADS;
    int v[kMaxBins / THREADS];
    int sum = 0;
#pragma unroll
    for (int k = 0; k < kMaxBins / THREADS; k++) {
        const int d = tid * per + k;
        v[k] = (k < per && d < bins) ? x[d] : 0;
        sum += v[k];
    }
    int inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    int run = inc - sum;
    for (int w = 0; w < warp; w++) run += warp_sums[w];
#pragma unroll
    for (int k = 0; k < kMaxBins / THREADS; k++) {
        const int d = tid * per + k;
        if (k < per && d < bins) x[d] = run;
        run += v[k];
    }
    __syncthreads();
}

// Shared memory of the scatter: next output slot and tile-local start of every
// digit, then the warps' counters, whose space the regrouped tile takes once
// the ranks are known.
template <int THREADS, int PER>
size_t scatter_smem(int bins)
{
    const size_t counters = sizeof(uint16_t) * (THREADS / 32) * bins, tile = 2 * sizeof(int32_t) * THREADS * PER;
    return 2 * sizeof(int32_t) * bins + std::max(counters, tile);
}

template <int THREADS, int PER>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
    scatter_kernel(const int32_t *keys, const int32_t *vals, int64_t m, int shift, int bits, int64_t per_cta,
                   const int32_t *hist, const int32_t *totals, int32_t *keys_out, int32_t *vals_out,
                   const int32_t *bad)
{
    constexpr int kTile = THREADS * PER, kWarps = THREADS / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int32_t warp_sums[kWarps];
    if (*bad) return;
    const int bins = 1 << bits, mask = bins - 1;
    int32_t *next = reinterpret_cast<int32_t *>(smem);  // next output slot of each digit
    int32_t *start = next + bins;                       // the digit's first slot in the regrouped tile
    uint16_t *cnt = reinterpret_cast<uint16_t *>(start + bins);  // [warp][digit]
    int32_t *skey = start + bins, *sval = skey + kTile;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int d = tid; d < bins; d += THREADS) next[d] = totals[d];
    __syncthreads();
    scan_bins<THREADS>(next, bins, warp_sums);
    for (int d = tid; d < bins; d += THREADS) next[d] += hist[(int64_t)d * gridDim.x + blockIdx.x];
    const int64_t b = (int64_t)blockIdx.x * per_cta, e = min(m, b + per_cta);
    for (int64_t t0 = b; t0 < e; t0 += kTile) {
        const int len = (int)min((int64_t)kTile, e - t0);
        __syncthreads();  // the last tile has been written out
        {
            // (bins * kWarps uint16 counters, bins a multiple of 32)
            uint4 *z = reinterpret_cast<uint4 *>(cnt);
            const int n16 = bins * kWarps / 8;
            for (int i = tid; i < n16; i += THREADS) z[i] = make_uint4(0u, 0u, 0u, 0u);
        }
        // a warp's items are contiguous and taken 32 at a time, so counting them
        // in this order keeps the input order among equal digits
        const int w0 = warp * (32 * PER);
        int32_t key[PER], val[PER];
        uint16_t pos[PER];
#pragma unroll
        for (int k = 0; k < PER; k++) {
            const int i = w0 + k * 32 + lane;
            key[k] = i < len ? keys[t0 + i] : 0;
        }
#pragma unroll
        for (int k = 0; k < PER; k++) {
            const int i = w0 + k * 32 + lane;
            val[k] = i < len ? vals[t0 + i] : 0;
        }
        __syncthreads();
        uint16_t *mine = cnt + warp * bins;
#pragma unroll
        for (int k = 0; k < PER; k++) {
            const bool valid = w0 + k * 32 + lane < len;
            const int d = (key[k] >> shift) & mask;
            // two digits' counters share a word.  Lanes of different digits count
            // alone; where some lanes' digits are equal, the atomic's order among
            // them is not theirs, and the matching lanes rank themselves
            unsigned *word = reinterpret_cast<unsigned *>(mine) + (d >> 1);
            const int sh = (d & 1) * 16;
            unsigned old = 0, now = 0;
            if (valid) old = (atomicAdd(word, 1u << sh) >> sh) & 0xffffu;
            __syncwarp();
            if (valid) now = (*reinterpret_cast<volatile unsigned *>(word) >> sh) & 0xffffu;
            __syncwarp();
            int before = (int)old, rank = 0;
            if (__any_sync(0xffffffffu, valid && now != old + 1)) {
                const unsigned peers = __match_any_sync(0xffffffffu, valid ? d : -1 - lane);
                before = (int)now - __popc(peers);
                rank = __popc(peers & dev::lanemask_lt());
            }
            pos[k] = (uint16_t)(before + rank);
        }
        __syncthreads();
        // counters -> exclusive prefix over the warps; digit totals -> tile starts
        for (int d = tid; d < bins; d += THREADS) {
            int run = 0;
#pragma unroll
            for (int w = 0; w < kWarps; w++) {
                const int c = cnt[w * bins + d];
                cnt[w * bins + d] = (uint16_t)run;
                run += c;
            }
            start[d] = run;
        }
        __syncthreads();
        scan_bins<THREADS>(start, bins, warp_sums);
#pragma unroll
        for (int k = 0; k < PER; k++) {
            const int d = (key[k] >> shift) & mask;
            pos[k] = (uint16_t)(pos[k] + start[d] + mine[d]);
        }
        __syncthreads();  // the counters are consumed: their space takes the tile
#pragma unroll
        for (int k = 0; k < PER; k++) {
            if (w0 + k * 32 + lane < len) {
                skey[pos[k]] = key[k];
                sval[pos[k]] = val[k];
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < PER; k++) {
            const int j = k * THREADS + tid;
            if (j < len) {
                const int32_t kk = skey[j];
                const int d = (kk >> shift) & mask;
                const int32_t o = next[d] + (j - start[d]);
                keys_out[o] = kk;
                vals_out[o] = sval[j];
            }
        }
        __syncthreads();
        for (int d = tid; d < bins; d += THREADS) next[d] += (d + 1 < bins ? start[d + 1] : len) - start[d];
    }
}

// First position of the sorted keys not below `row`: every lane probes its own
// point of the range, so a step narrows it 33-fold.
__device__ __forceinline__ int64_t warp_lower_bound(const int32_t *keys, int64_t lo, int64_t hi, int64_t row)
{
    const int lane = threadIdx.x & 31;
    while (lo < hi) {
        // probe points lo <= p_0 <= .. <= p_31 < hi
        const int64_t p = lo + (hi - lo) * (lane + 1) / 33;
        const unsigned below = __ballot_sync(0xffffffffu, keys[p] < row);
        const int c = __popc(below);  // probes below form a prefix
        const int64_t last = __shfl_sync(0xffffffffu, p, max(c - 1, 0)), first = __shfl_sync(0xffffffffu, p, min(c, 31));
        if (c > 0) lo = last + 1;
        if (c < 32) hi = first;
    }
    return lo;
}

// Row offsets from the sorted rows: a warp takes `span` rows, finds their edge
// range with all its lanes, then each lane searches its rows inside it.
__global__ void row_offsets_kernel(const int32_t *keys, int64_t m, int64_t n, int span, int32_t *ro,
                                   const int32_t *bad)
{
    if (*bad) return;
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t r0 = warp * span, r1 = min(n + 1, r0 + span);  // row n is the end
    if (r0 > n) return;
    const int64_t lo = warp_lower_bound(keys, 0, m, r0);
    const int64_t hi = warp_lower_bound(keys, lo, m, r1);
    int64_t from = lo;
    for (int64_t r = r0 + lane; r < r1; r += 32) {
        int64_t a = from, b = hi;
        while (a < b) {
            const int64_t mid = (a + b) >> 1;
            if (keys[mid] < r) a = mid + 1; else b = mid;
        }
        ro[r] = (int32_t)a;
        from = a;
    }
}

// Temporary memory of a conversion, stream-ordered, from one pool per device that
// is safe with any thread and stream.  A conversion of 16 M edges needs 200 MB, and
// mapping that anew costs more than the sort; the pool keeps up to kPoolKeep bytes
// between calls.  A conversion frees its workspace ahead of its last wait, so what is
// kept is settled when it returns: more than kPoolKeep goes back to the device
// there, the rest with b40c_coo_release_memory, after a problem_create_coo and when an
// allocation of this library runs short.
constexpr uint64_t kPoolKeep = 512ull << 20;
constexpr int kMaxDevices = 64;
static cudaMemPool_t g_pool[kMaxDevices];
static std::mutex g_pool_mutex;

static int pool_of(int device, cudaMemPool_t *out)
{
    if (device < 0 || device >= kMaxDevices) return b40c::fail(B40C_ERROR_INVALID_VALUE, "device %d", device);
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    if (!g_pool[device]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool;
        CUDA_TRY(cudaMemPoolCreate(&pool, &props), "conversion pool");
        uint64_t keep = kPoolKeep;
        const cudaError_t e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e != cudaSuccess) {
            cudaMemPoolDestroy(pool);
            CUDA_TRY(e, "conversion pool threshold");
        }
        g_pool[device] = pool;
    }
    *out = g_pool[device];
    return B40C_SUCCESS;
}

// Gives back what the device's pool holds beyond the conversions in progress.
static void trim_pool(int device)
{
    if (device < 0 || device >= kMaxDevices) return;
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    if (g_pool[device] && cudaMemPoolTrimTo(g_pool[device], 0) != cudaSuccess) cudaGetLastError();
}

struct Workspace {
    unsigned char *p = nullptr;
    cudaStream_t s;
    explicit Workspace(cudaStream_t stream) : s(stream) {}
    // Before the caller's last wait: the pool counts freed memory as its own only
    // once the host has seen the free done.
    cudaError_t release()
    {
        void *q = p;
        p = nullptr;
        return q ? cudaFreeAsync(q, s) : cudaSuccess;
    }
    ~Workspace()
    {
        if (!p) return;
        release();  // a failed conversion
        cudaStreamSynchronize(s);
        cudaGetLastError();
    }
};

template <int THREADS, int PER>
int sort_passes(const int32_t *d_rows, const int32_t *d_cols, int64_t nodes, int64_t edges, int passes, int bits,
                int32_t *const (&kbuf)[2], int32_t *const (&vbuf)[2], int32_t *d_ci, int32_t *hist, int32_t *totals,
                int32_t *bad, int ctas, cudaStream_t s, const int32_t **sorted)
{
    const int bins = 1 << bits;
    const int64_t tile = THREADS * PER, tiles = (edges + tile - 1) / tile;
    const int64_t per_cta = (tiles + ctas - 1) / ctas * tile;
    const int grid = (int)((edges + per_cta - 1) / per_cta);
    const size_t smem = scatter_smem<THREADS, PER>(bins);
    // (the limit belongs to the kernel: every conversion sets the same one, for the
    // widest digit, so none running beside it finds its own launch above the limit)
    CUDA_TRY(cudaFuncSetAttribute(scatter_kernel<THREADS, PER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)scatter_smem<THREADS, PER>(kMaxBins)),
             "smem attribute");
    const int32_t *kin = d_rows, *vin = d_cols;
    for (int pass = 0; pass < passes; pass++) {
        int32_t *kout = kbuf[pass & 1], *vout = pass == passes - 1 ? d_ci : vbuf[pass & 1];
        const int shift = bits * pass;
        digit_count_kernel<<<grid, kThreads, sizeof(int32_t) * bins, s>>>(kin, pass == 0 ? d_cols : nullptr, edges,
                                                                          (int32_t)nodes, shift, bins, per_cta, hist, bad);
        digit_scan_kernel<<<(bins * 32 + 255) / 256, 256, 0, s>>>(hist, grid, bins, totals);
        scatter_kernel<THREADS, PER><<<grid, THREADS, smem, s>>>(kin, vin, edges, shift, bits, per_cta, hist, totals,
                                                                 kout, vout, bad);
        CUDA_TRY(cudaGetLastError(), "radix pass launch");
        kin = kout;
        vin = vout;
    }
    *sorted = kin;
    return B40C_SUCCESS;
}

}  // namespace coo

namespace rt {

void release_conversion_memory(int device) { coo::trim_pool(device); }

namespace {

struct DeviceBuffer {
    void *p = nullptr;
    ~DeviceBuffer()
    {
        if (p) cudaFree(p);
    }
};

}  // namespace

// Stable by-row conversion of a device COO list into device CSR arrays
// (row_offsets[nodes + 1], column_indices[edges]); synchronous on `s`.
int coo_to_csr_device(const int32_t *d_rows, const int32_t *d_cols, int64_t nodes, int64_t edges, int32_t *d_ro,
                      int32_t *d_ci, cudaStream_t s, int device, int sms)
{
    using namespace coo;
    if (edges == 0) {
        CUDA_TRY(cudaMemsetAsync(d_ro, 0, sizeof(int32_t) * (nodes + 1), s), "offset reset");
        CUDA_TRY(cudaStreamSynchronize(s), "offset reset");
        return B40C_SUCCESS;
    }
    // the row ids' significant bits in equal digits (at least 5 bits: the
    // kernels clear and scan the counters of 32 digits at a time)
    int row_bits = 1;
    while (row_bits < 31 && ((int64_t)1 << row_bits) < nodes) row_bits++;
    // (a single pass would write columns over input it has not read, where a caller
    // converts in place)
    const auto overlaps = [&](const int32_t *in) { return in < d_ci + edges && d_ci < in + edges; };
    const int fewest = (row_bits + kMaxDigitBits - 1) / kMaxDigitBits;
    const int passes = fewest == 1 && (overlaps(d_rows) || overlaps(d_cols)) ? 2 : fewest;
    const int bits = std::max(5, (row_bits + passes - 1) / passes);
    const int ctas = sms * kCtasPerSm;

    // workspace: flag, digit totals, digit counts, then the passes' outputs (the
    // last one writes the column indices in place; its rows give the offsets)
    auto align = [](int64_t x) { return (x + 255) / 256 * 256; };
    const int64_t list = align(sizeof(int32_t) * edges), bins = (int64_t)1 << bits;
    const int64_t totals_at = 256, hist_at = totals_at + align(sizeof(int32_t) * bins);
    const int64_t lists_at = hist_at + align(sizeof(int32_t) * bins * ctas);
    const int key_lists = std::min(passes, 2), val_lists = std::min(passes - 1, 2);
    cudaMemPool_t pool;
    int rc = pool_of(device, &pool);
    if (rc) return rc;
    Workspace ws(s);
    {
        const int64_t need = lists_at + (key_lists + val_lists) * list;
        const cudaError_t e = cudaMallocFromPoolAsync((void **)&ws.p, (size_t)need, pool, s);
        if (e != cudaSuccess) {
            cudaGetLastError();
            ws.p = nullptr;
            return b40c::fail(e == cudaErrorMemoryAllocation ? B40C_ERROR_MEMORY_ALLOCATION : (int)e,
                              "conversion workspace (%lld bytes) failed: %s", (long long)need, cudaGetErrorString(e));
        }
    }
    int32_t *flag = (int32_t *)ws.p, *totals = (int32_t *)(ws.p + totals_at), *hist = (int32_t *)(ws.p + hist_at);
    int32_t *kbuf[2] = {}, *vbuf[2] = {};
    for (int i = 0; i < key_lists; i++) kbuf[i] = (int32_t *)(ws.p + lists_at + i * list);
    for (int i = 0; i < val_lists; i++) vbuf[i] = (int32_t *)(ws.p + lists_at + (key_lists + i) * list);
    CUDA_TRY(cudaMemsetAsync(flag, 0, sizeof(int32_t), s), "flag reset");

    // long tiles once every SM gets one
    const int32_t *sorted = nullptr;
    const bool long_tiles = edges >= (int64_t)sms * kLongThreads * kLongPer;
    rc = long_tiles ? sort_passes<kLongThreads, kLongPer>(d_rows, d_cols, nodes, edges, passes, bits, kbuf, vbuf, d_ci,
                                                          hist, totals, flag, sms, s, &sorted)
                    : sort_passes<kShortThreads, kShortPer>(d_rows, d_cols, nodes, edges, passes, bits, kbuf, vbuf,
                                                            d_ci, hist, totals, flag, ctas, s, &sorted);
    if (rc) return rc;
    // few edges per row: longer spans, so that the warps' searches stay a small part
    const int span = nodes > 8 * edges ? 1024 : 128;
    const int64_t warps = (nodes + 1 + span - 1) / span;
    row_offsets_kernel<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, s>>>(sorted, edges, nodes, span, d_ro, flag);
    CUDA_TRY(cudaGetLastError(), "row offsets launch");
    int32_t h_bad = 0;
    CUDA_TRY(cudaMemcpyAsync(&h_bad, flag, sizeof(int32_t), cudaMemcpyDeviceToHost, s), "flag read");
    CUDA_TRY(ws.release(), "conversion workspace release");
    CUDA_TRY(cudaStreamSynchronize(s), "conversion");
    if (h_bad) return b40c::fail(B40C_ERROR_INVALID_VALUE, "COO vertex id out of [0, %lld)", (long long)nodes);
    return B40C_SUCCESS;
}

}  // namespace rt
}  // namespace b40c

using namespace b40c;
using namespace b40c::rt;

extern "C" {

int b40c_coo_to_csr_device(const int32_t *d_rows, const int32_t *d_cols, int64_t nodes, int64_t edges,
                           int32_t *d_row_offsets, int32_t *d_column_indices, void *cuda_stream)
{
    b40c::clear_error();
    if (((!d_rows || !d_cols || !d_column_indices) && edges > 0) || !d_row_offsets || nodes <= 0 || edges < 0 ||
        nodes >= INT32_MAX || edges >= INT32_MAX)
        return b40c::fail(B40C_ERROR_INVALID_VALUE, "b40c_coo_to_csr_device: bad arguments");
    int device = 0, sms = 0;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        cudaGetLastError();
        return b40c::fail(B40C_ERROR_NO_DEVICE, "no usable current CUDA device");
    }
    return coo_to_csr_device(d_rows, d_cols, nodes, edges, d_row_offsets, d_column_indices,
                             (cudaStream_t)cuda_stream, device, sms);
}

int b40c_coo_release_memory(int device)
{
    b40c::clear_error();
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count < 1) {
        cudaGetLastError();
        return b40c::fail(B40C_ERROR_NO_DEVICE, "no CUDA device");
    }
    if (device < 0 || device >= count) return b40c::fail(B40C_ERROR_INVALID_VALUE, "device %d", device);
    release_conversion_memory(device);
    return B40C_SUCCESS;
}

int b40c_bfs_problem_create_coo(const int32_t *h_rows, const int32_t *h_cols, int64_t nodes, int64_t edges,
                                int mark_predecessors, int device, b40c_bfs_problem **out)
{
    b40c::clear_error();
    if (!out) return b40c::fail(B40C_ERROR_INVALID_VALUE, "null output handle");
    *out = nullptr;
    if ((!h_rows || !h_cols) && edges > 0)
        return b40c::fail(B40C_ERROR_INVALID_VALUE, "null COO arrays");
    if (nodes <= 0 || edges < 0 || nodes >= (int64_t)1 << 30 || edges >= (int64_t)INT32_MAX)
        return b40c::fail(B40C_ERROR_INVALID_VALUE,
                          "invalid COO (nodes %lld, edges %lld; need 0 < nodes < 2^30, edges < 2^31)",
                          (long long)nodes, (long long)edges);
    auto load = [&](b40c_bfs_problem *p) -> int {
        int rc;
        if ((rc = alloc_dev((void **)&p->d_ro, sizeof(int32_t) * (nodes + 1), "row offsets"))) return rc;
        if ((rc = alloc_dev((void **)&p->d_ci, sizeof(int32_t) * std::max<int64_t>(edges, 1), "column indices")))
            return rc;
        DeviceBuffer rows, cols;
        const size_t bytes = sizeof(int32_t) * (size_t)std::max<int64_t>(edges, 1);
        if ((rc = alloc_dev(&rows.p, bytes, "COO rows"))) return rc;
        if ((rc = alloc_dev(&cols.p, bytes, "COO columns"))) return rc;
        if (edges > 0) {
            CUDA_TRY(cudaMemcpyAsync(rows.p, h_rows, bytes, cudaMemcpyHostToDevice, p->stream), "COO upload");
            CUDA_TRY(cudaMemcpyAsync(cols.p, h_cols, bytes, cudaMemcpyHostToDevice, p->stream), "COO upload");
        }
        rc = coo_to_csr_device((const int32_t *)rows.p, (const int32_t *)cols.p, nodes, edges, p->d_ro, p->d_ci,
                               p->stream, p->device, p->sms);
        release_conversion_memory(p->device);  // one conversion per handle: its memory is for the searches
        return rc;
    };
    return create_problem(nodes, edges, mark_predecessors, 0, device, load, out);
}

}  // extern "C"
