// Readout: the raster (read, or staged on the device and collected), neuron
// state, weights, the CSR, partition statistics and handle information.
#include <memory>

#include "sim.h"

using namespace mgc;

namespace {

constexpr int32_t kRasterBits = kStatusRasterIds | kStatusRasterSteps;

// ns steps' counts c32 and their ni ids hid (step after step, ascending inside
// a step) into the caller's arrays.
mgc_status finish_raster(int64_t step0, int64_t ns, int64_t ni, const int32_t* c32, bool truncated, int32_t status,
                         int64_t* first_step, int64_t* counts, int64_t counts_cap, int64_t ids_cap, int64_t* n_steps,
                         int64_t* n_ids)
{
    truncated = truncated || ns > counts_cap || ni > ids_cap;
    if (counts)
        for (int64_t i = 0; i < std::min(ns, counts_cap); ++i) counts[i] = c32[i];
    if (first_step) *first_step = step0;
    if (n_steps) *n_steps = std::min(ns, counts_cap);
    if (n_ids) *n_ids = std::min(ni, ids_cap);
    if (truncated) return fail(MGC_ERR_OVERFLOW, "raster truncated (device status %d)", status);
    return MGC_OK;
}

// ---------------------------------------------------------------------------
// A raster's ids put in ascending order inside each step, on the device (the
// host's sort of 6.3e6 ids, 6,270 a step, took 24 ms on 16 threads).  The ids
// of a step are distinct, so a long step is sorted by marking its ids in a
// bitmap in shared memory and reading the bitmap out in order; up to
// kSortBitonic ids take a bitonic sort in shared memory, up to 32 one warp's.
// Bound by the ids read and written once (and n/8 bytes of shared memory
// cleared and read per long step).
// ---------------------------------------------------------------------------
constexpr int kSortBlock = 256;
constexpr int kSortBitonic = 2048;
constexpr int kSortWords = 48 * 1024;                 // bitmap words in shared memory (1.57e6 neurons)
constexpr int64_t kSortBitmaps = int64_t(256) << 20;  // larger networks: bitmaps in device memory, at most

// meta: {first step, steps, ids, raster status bits, the handle's step}; off:
// running sums of the steps' counts.  One block.
__global__ void __launch_bounds__(1024) k_raster_offsets(StepArgs a, const int32_t* counts, int64_t steps_cap,
                                                         int64_t ids_cap, int64_t* meta, int64_t* off)
{
    __shared__ int64_t part[32];
    __shared__ int64_t carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t ns = min(*a.step - *a.raster_step0, steps_cap);
    if (threadIdx.x == 0) {
        carry = 0;
        off[0] = 0;
        meta[0] = *a.raster_step0;
        meta[1] = ns;
        meta[2] = min(*a.raster_pos, ids_cap);
        meta[3] = *a.status & kRasterBits;
        meta[4] = *a.step;
    }
    __syncthreads();
    for (int64_t b = 0; b < ns; b += blockDim.x) {
        const int64_t i = b + threadIdx.x;
        int64_t c = i < ns ? counts[i] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t v = __shfl_up_sync(0xffffffffu, c, o);
            if (lane >= o) c += v;
        }
        if (lane == 31) part[warp] = c;
        __syncthreads();
        if (warp == 0) {
            int64_t p = part[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t v = __shfl_up_sync(0xffffffffu, p, o);
                if (lane >= o) p += v;
            }
            part[lane] = p;
        }
        __syncthreads();
        c += carry + (warp ? part[warp - 1] : 0);
        if (i < ns) off[i + 1] = c;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = c;
        __syncthreads();
    }
}

// Steps of 2 to 32 ids, a warp each: a bitonic sort through shuffles.
__global__ void __launch_bounds__(kSortBlock) k_raster_sort_short(const int64_t* meta, const int64_t* off, int32_t* ids)
{
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < meta[1]; s += nw) {
        const int64_t b = off[s];
        const int64_t c = off[s + 1] - b;
        if (c < 2 || c > 32 || b + c > meta[2]) continue;
        int32_t x = lane < c ? ids[b + lane] : 0x7fffffff;
#pragma unroll
        for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
            for (int j = k >> 1; j >= 1; j >>= 1) {
                const int32_t y = __shfl_xor_sync(0xffffffffu, x, j);
                const bool up = (lane & k) == 0, low = (lane & j) == 0;
                x = (up == low) ? min(x, y) : max(x, y);
            }
        if (lane < c) ids[b + lane] = x;
    }
}

// Steps of more than 32 ids, a block each.  bitmap: null when the network's
// `words` words fit in shared memory, else `words` of device memory per block.
__global__ void __launch_bounds__(kSortBlock) k_raster_sort_long(const int64_t* meta, const int64_t* off, int32_t* ids,
                                                                 int64_t words, uint32_t* bitmap)
{
    extern __shared__ uint32_t sort_mem[];
    __shared__ int32_t part[kSortBlock / 32];
    uint32_t* bits_of = bitmap ? bitmap + (int64_t)blockIdx.x * words : sort_mem;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = kSortBlock / 32;
    for (int64_t s = blockIdx.x; s < meta[1]; s += gridDim.x) {
        const int64_t b = off[s];
        const int64_t c64 = off[s + 1] - b;
        if (c64 <= 32 || b + c64 > meta[2]) continue;
        const int c = (int)c64;
        int32_t* x = ids + b;
        if (c <= kSortBitonic) {
            int m = 64;
            while (m < c) m <<= 1;
            int32_t* v = reinterpret_cast<int32_t*>(sort_mem);
            for (int i = threadIdx.x; i < m; i += kSortBlock) v[i] = i < c ? x[i] : 0x7fffffff;
            __syncthreads();
            for (int k = 2; k <= m; k <<= 1)
                for (int j = k >> 1; j >= 1; j >>= 1) {
                    for (int i = threadIdx.x; i < m / 2; i += kSortBlock) {
                        const int p = 2 * i - (i & (j - 1)), q = p + j;  // the pair at distance j
                        const int32_t u = v[p], w = v[q];
                        if ((u > w) == ((p & k) == 0)) {
                            v[p] = w;
                            v[q] = u;
                        }
                    }
                    __syncthreads();
                }
            for (int i = threadIdx.x; i < c; i += kSortBlock) x[i] = v[i];
            __syncthreads();
            continue;
        }
        for (int64_t i = threadIdx.x; i < words; i += kSortBlock) bits_of[i] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < c; i += kSortBlock) {
            const int64_t w = (uint32_t)x[i] >> 5;
            if (w < words) atomicOr(bits_of + w, 1u << (x[i] & 31));
        }
        __syncthreads();
        // each warp a stretch of the words: their bits counted, then written out
        const int64_t per = (words + nwarp * 32 - 1) / (nwarp * 32) * 32;
        const int64_t w0 = warp * per, w1 = min(words, w0 + per);
        int cnt = 0;
        for (int64_t i = w0 + lane; i < w1; i += 32) cnt += __popc(bits_of[i]);
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        if (lane == 0) part[warp] = cnt;
        __syncthreads();
        int at = 0;
        for (int w = 0; w < warp; ++w) at += part[w];
        for (int64_t i0 = w0; i0 < w1; i0 += 32) {
            const int64_t i = i0 + lane;
            uint32_t bits = i < w1 ? bits_of[i] : 0u;
            const int n = __popc(bits);
            int incl = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            int p = at + incl - n;
            for (; bits; bits &= bits - 1, ++p) x[p] = (int32_t)(32 * i + (__ffs(bits) - 1));
            at += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncthreads();
    }
}

// Enqueues the offsets and the sort of a raster (counts, ids); meta as above.
mgc_status sort_raster(mgc_sim* s, const int32_t* counts, int32_t* ids, int64_t* meta)
{
    k_raster_offsets<<<1, 1024, 0, s->stream>>>(s->a, counts, s->raster_steps_cap, s->raster_ids_cap, meta,
                                                s->raster_off);
    k_raster_sort_short<<<s->sort_grid, kSortBlock, 0, s->stream>>>(meta, s->raster_off, ids);
    k_raster_sort_long<<<s->sort_grid, kSortBlock, s->sort_smem, s->stream>>>(meta, s->raster_off, ids, s->sort_words,
                                                                               s->sort_bitmap);
    CK(cudaGetLastError());
    s->launches += 3;
    return MGC_OK;
}

// The raster so far into a stage (block-strided copies), then the clock of
// the next raster (k_raster_restart, once the copies and the offsets are made).
__global__ void k_raster_stage(StepArgs a, int32_t* ids, int32_t* counts, int64_t steps_cap, int64_t ids_cap)
{
    const int64_t ns = min(*a.step - *a.raster_step0, steps_cap);
    const int64_t ni = min(*a.raster_pos, ids_cap);
    GRID_STRIDE(i, ns) counts[i] = a.raster_counts[i];
    GRID_STRIDE(i, ni) ids[i] = a.raster_ids[i];
}

__global__ void k_raster_restart(StepArgs a)
{
    *a.raster_step0 = *a.step;
    *a.raster_pos = 0;
    atomicAnd(a.status, ~kRasterBits);
}

// Weights into synapse-list order.
__global__ void k_weights_out(const uint2* words, const int64_t* idx, int64_t S, float* out)
{
    GRID_STRIDE(p, S) out[idx[p]] = as_f(words[p].y);
}

// The six state arrays side by side, for one copy to the host.
__global__ void k_state_out(StepArgs a, uint32_t* out, int32_t n)
{
    const uint32_t* in[6] = {reinterpret_cast<const uint32_t*>(a.V), reinterpret_cast<const uint32_t*>(a.Iexc),
                             reinterpret_cast<const uint32_t*>(a.Iinh), reinterpret_cast<const uint32_t*>(a.refrac),
                             reinterpret_cast<const uint32_t*>(a.last_fired),
                             reinterpret_cast<const uint32_t*>(a.fire_cnt)};
    GRID_STRIDE(i, n)
    {
#pragma unroll
        for (int k = 0; k < 6; ++k) out[(size_t)k * n + i] = in[k][i];
    }
}

// Up to this many neurons the state comes over as one copy: six copies of
// 17 KB took 110 us, one of 100 KB and the host's copies out of it 45.
constexpr int32_t kStateOneCopy = 1 << 16;

}  // namespace

namespace mgc {

// The raster's sort: its sums, its launch shape, and bitmaps for networks whose
// ids' bitmap does not fit in shared memory (fewer of them, each for a block,
// where the device has no room for all).
static mgc_status init_raster(mgc_sim* s)
{
    if (!s->a.record) return MGC_OK;
    CKS(s->alloc(&s->raster_meta, 5));
    CKS(s->alloc(&s->raster_off, (size_t)s->raster_steps_cap + 1, false));
    s->sort_words = (std::max<int64_t>(s->n, s->n_src) + 31) / 32;  // whole-network ids
    int sms = 0, occ = 0;
    CKS(device_attr(cudaDevAttrMultiProcessorCount, s->device, &sms));
    const bool chip = s->sort_words <= kSortWords;
    s->sort_smem = 4 * (size_t)std::max<int64_t>(chip ? s->sort_words : 0, kSortBitonic);
    CK(cudaFuncSetAttribute(k_raster_sort_long, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kSortWords));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_raster_sort_long, kSortBlock, s->sort_smem));
    s->sort_grid = sms * std::max(1, occ);
    if (!chip) {
        s->sort_grid = (int)std::max<int64_t>(1, std::min<int64_t>(sms, kSortBitmaps / (4 * s->sort_words)));
        for (;; s->sort_grid /= 2) {
            const mgc_status st = s->alloc(&s->sort_bitmap, (size_t)s->sort_grid * (size_t)s->sort_words, false);
            if (st == MGC_OK) break;
            if (st != MGC_ERR_NOMEM || s->sort_grid == 1) return st;
        }
    }
    return MGC_OK;
}

mgc_status init_readout(mgc_sim* s)
{
    if (s->n <= kStateOneCopy) {
        CKS(s->alloc(&s->state_buf, 6 * (size_t)s->n, false));
        s->state_host.resize(6 * (size_t)s->n);
    }
    CKS(init_raster(s));
    // weights that change are read again and again (cudaMalloc and cudaFree in
    // the call took up to 600 ms on a busy driver); without the buffer, each
    // call finds its own
    if (!s->stdp || s->S == 0) return MGC_OK;
    const mgc_status st = s->alloc(&s->weights_buf, s->S, false);
    return st == MGC_ERR_NOMEM ? MGC_OK : st;
}

}  // namespace mgc

extern "C" {

mgc_status mgc_read_raster(mgc_sim* s, int64_t* first_step, int64_t* counts, int64_t counts_cap, int32_t* ids,
                           int64_t ids_cap, int64_t* n_steps, int64_t* n_ids)
{
    if (!s) return fail(MGC_ERR_INVALID, "null handle");
    if (!s->a.record) return fail(MGC_ERR_INVALID, "raster recording is off for this handle");
    if (s->staged) return fail(MGC_ERR_INVALID, "collect the staged rasters first (mgc_raster_collect)");
    CK(cudaSetDevice(s->device));
    CKS(sort_raster(s, s->a.raster_counts, s->a.raster_ids, s->raster_meta));
    // the next raster starts here; only the raster's status bits are cleared
    k_raster_restart<<<1, 1, 0, s->stream>>>(s->a);
    CK(cudaGetLastError());
    s->launches += 1;
    int64_t meta[5];
    CK(cudaMemcpyAsync(meta, s->raster_meta, sizeof(meta), cudaMemcpyDeviceToHost, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    const int64_t step0 = meta[0], ns = meta[1], ni = meta[2];
    const int32_t status = (int32_t)meta[3];
    std::vector<int32_t> c32(ns);
    if (ns) CK(cudaMemcpyAsync(c32.data(), s->a.raster_counts, 4 * ns, cudaMemcpyDeviceToHost, s->stream));
    if (ids && std::min(ni, ids_cap) > 0)
        CK(cudaMemcpyAsync(ids, s->a.raster_ids, 4 * std::min(ni, ids_cap), cudaMemcpyDeviceToHost, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    return finish_raster(step0, ns, ni, c32.data(), status != 0, status, first_step, counts, counts_cap, ids_cap,
                         n_steps, n_ids);
}

mgc_status mgc_raster_stage(mgc_sim* s)
{
    if (!s) return fail(MGC_ERR_INVALID, "null handle");
    if (!s->a.record) return fail(MGC_ERR_INVALID, "raster recording is off for this handle");
    if (s->staged == 2) return fail(MGC_ERR_INVALID, "two rasters are staged already: collect one first");
    CK(cudaSetDevice(s->device));
    mgc_sim::RasterStage& g = s->stages[(s->stage_head + s->staged) & 1];
    if (!g.ids) {
        CKS(s->alloc(&g.ids, (size_t)s->raster_ids_cap, false));
        CKS(s->alloc(&g.counts, (size_t)s->raster_steps_cap, false));
        CKS(s->alloc(&g.meta, 5));
        CK(cudaEventCreateWithFlags(&g.ev, cudaEventDisableTiming));
    }
    if (!s->copy_stream) CK(cudaStreamCreateWithFlags(&s->copy_stream, cudaStreamNonBlocking));
    k_raster_stage<<<grid_for(s->raster_ids_cap), 256, 0, s->stream>>>(s->a, g.ids, g.counts, s->raster_steps_cap,
                                                                        s->raster_ids_cap);
    CK(cudaGetLastError());
    CKS(sort_raster(s, g.counts, g.ids, g.meta));
    k_raster_restart<<<1, 1, 0, s->stream>>>(s->a);
    CK(cudaGetLastError());
    CK(cudaEventRecord(g.ev, s->stream));
    s->launches += 2;
    s->staged += 1;
    return MGC_OK;
}

mgc_status mgc_raster_collect(mgc_sim* s, int64_t* first_step, int64_t* counts, int64_t counts_cap, int32_t* ids,
                              int64_t ids_cap, int64_t* n_steps, int64_t* n_ids)
{
    if (!s) return fail(MGC_ERR_INVALID, "null handle");
    if (!s->staged) return fail(MGC_ERR_INVALID, "no raster is staged (mgc_raster_stage)");
    CK(cudaSetDevice(s->device));
    mgc_sim::RasterStage& g = s->stages[s->stage_head];
    // the stage's copies are done; the steps enqueued after it keep running
    CK(cudaStreamWaitEvent(s->copy_stream, g.ev, 0));
    int64_t meta[5];
    CK(cudaMemcpyAsync(meta, g.meta, sizeof(meta), cudaMemcpyDeviceToHost, s->copy_stream));
    CK(cudaStreamSynchronize(s->copy_stream));
    const int64_t step0 = meta[0], ns = meta[1], ni = meta[2];
    const int32_t status = (int32_t)meta[3];
    std::vector<int32_t> c32(ns);
    if (ns) CK(cudaMemcpyAsync(c32.data(), g.counts, 4 * ns, cudaMemcpyDeviceToHost, s->copy_stream));
    if (ids && std::min(ni, ids_cap) > 0)
        CK(cudaMemcpyAsync(ids, g.ids, 4 * std::min(ni, ids_cap), cudaMemcpyDeviceToHost, s->copy_stream));
    CK(cudaStreamSynchronize(s->copy_stream));
    s->stage_head ^= 1;
    s->staged -= 1;
    return finish_raster(step0, ns, ni, c32.data(), status != 0, status, first_step, counts, counts_cap, ids_cap,
                         n_steps, n_ids);
}

mgc_status mgc_read_state(mgc_sim* s, float* v, float* i_exc, float* i_inh, int32_t* refrac, int32_t* last_fired,
                          int32_t* fire_cnt)
{
    if (!s) return fail(MGC_ERR_INVALID, "null handle");
    CK(cudaSetDevice(s->device));
    const size_t n = s->n;
    if (s->n <= kStateOneCopy) {
        k_state_out<<<grid_for(s->n), 256, 0, s->stream>>>(s->a, s->state_buf, s->n);
        CK(cudaGetLastError());
        s->launches += 1;
        CK(cudaMemcpyAsync(s->state_host.data(), s->state_buf, 24 * n, cudaMemcpyDeviceToHost, s->stream));
        CK(cudaStreamSynchronize(s->stream));
        void* to[6] = {v, i_exc, i_inh, refrac, last_fired, fire_cnt};
        for (int k = 0; k < 6; ++k)
            if (to[k]) memcpy(to[k], s->state_host.data() + k * n, 4 * n);
        if (v)
            for (size_t k = 0; k < s->pois_idx.size(); ++k) v[s->pois_idx[k]] = s->pois_v[k];
        return MGC_OK;
    }
    CK(cudaStreamSynchronize(s->stream));
    if (v) {
        CK(cudaMemcpy(v, s->a.V, 4 * n, cudaMemcpyDeviceToHost));
        for (size_t k = 0; k < s->pois_idx.size(); ++k) v[s->pois_idx[k]] = s->pois_v[k];
    }
    if (i_exc) CK(cudaMemcpy(i_exc, s->a.Iexc, 4 * n, cudaMemcpyDeviceToHost));
    if (i_inh) CK(cudaMemcpy(i_inh, s->a.Iinh, 4 * n, cudaMemcpyDeviceToHost));
    if (refrac) CK(cudaMemcpy(refrac, s->a.refrac, 4 * n, cudaMemcpyDeviceToHost));
    if (last_fired) CK(cudaMemcpy(last_fired, s->a.last_fired, 4 * n, cudaMemcpyDeviceToHost));
    if (fire_cnt) CK(cudaMemcpy(fire_cnt, s->a.fire_cnt, 4 * n, cudaMemcpyDeviceToHost));
    return MGC_OK;
}

mgc_status mgc_read_weights(mgc_sim* s, float* weight)
{
    if (!s || !weight) return fail(MGC_ERR_INVALID, "null argument");
    if (!s->csr_syn64) return fail(MGC_ERR_INVALID, "procedural networks have no synapse-list order");
    CK(cudaSetDevice(s->device));
    CK(cudaStreamSynchronize(s->stream));
    if (!s->S) return MGC_OK;
    // put into synapse-list order on the device (15 MB come over for 3.8e6
    // synapses instead of the words and their places, 61 MB, and a host loop)
    const uint2* src_words = s->a.pull ? s->a.in_ent : s->a.syn;  // the pull method's live weights
    const int64_t* src_idx = s->a.pull ? s->in_syn64 : s->csr_syn64;
    DevTmp t;
    float* out = s->weights_buf;
    if (!out) {
        const mgc_status st = tmp_alloc(t, &out, s->S);
        if (st == MGC_ERR_NOMEM) {  // a full device: a stretch at a time in host memory
            const int64_t step = std::min<int64_t>(s->S, int64_t(1) << 22);
            std::vector<uint2> words(step);
            std::vector<int64_t> idx(step);
            for (int64_t b = 0; b < s->S; b += step) {
                const int64_t c = std::min(step, s->S - b);
                CK(cudaMemcpy(words.data(), src_words + b, 8 * c, cudaMemcpyDeviceToHost));
                CK(cudaMemcpy(idx.data(), src_idx + b, 8 * c, cudaMemcpyDeviceToHost));
                for (int64_t p = 0; p < c; ++p) memcpy(&weight[idx[p]], &words[p].y, 4);
            }
            return MGC_OK;
        }
        CKS(st);
    }
    k_weights_out<<<grid_for(s->S), 256, 0, s->stream>>>(src_words, src_idx, s->S, out);
    CK(cudaGetLastError());
    s->launches += 1;
    CK(cudaMemcpyAsync(weight, out, 4 * (size_t)s->S, cudaMemcpyDeviceToHost, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    return MGC_OK;
}

mgc_status mgc_export_csr(mgc_sim* s, int64_t* row_ptr, int32_t* tgt, float* weight, int32_t* delay)
{
    if (!s) return fail(MGC_ERR_INVALID, "null handle");
    CK(cudaSetDevice(s->device));
    CK(cudaStreamSynchronize(s->stream));
    if (row_ptr) CK(cudaMemcpy(row_ptr, s->a.row_ptr, 8 * ((size_t)s->n_src + 1), cudaMemcpyDeviceToHost));
    if (tgt || weight || delay) {
        // in pieces, so a large CSR needs no second full-size host copy
        const int64_t piece = int64_t(1) << 24;
        std::vector<uint2> buf((size_t)std::min<int64_t>(piece, std::max<int64_t>(s->S, 1)));
        for (int64_t p0 = 0; p0 < s->S; p0 += piece) {
            const int64_t c = std::min(piece, s->S - p0);
            CK(cudaMemcpy(buf.data(), s->a.syn + p0, 8 * c, cudaMemcpyDeviceToHost));
            for (int64_t q = 0; q < c; ++q) {
                if (tgt) tgt[p0 + q] = (int32_t)(buf[q].x & s->a.tmask);
                if (delay) delay[p0 + q] = (int32_t)(buf[q].x >> s->a.tbits);
                if (weight) memcpy(&weight[p0 + q], &buf[q].y, 4);
            }
        }
    }
    return MGC_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Partition statistics on the device: one warp per source row of the CSR,
// the zones' counters in shared memory, flushed once per block.
// ---------------------------------------------------------------------------
namespace {

constexpr int kMaxZones = 4096;

__global__ void k_partition_stats(const int64_t* row_ptr, const uint2* syn, int32_t n_src, uint32_t tmask,
                                  int32_t tar_base, const int32_t* part, int32_t nparts, unsigned long long* out)
{
    extern __shared__ unsigned int zc[];  // [3][nparts]: syn by source zone, out by source zone, in by target zone
    for (int z = threadIdx.x; z < 3 * nparts; z += blockDim.x) zc[z] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t src = warp; src < n_src; src += nwarps) {
        const int64_t b = row_ptr[src], e = row_ptr[src + 1];
        if (e == b) continue;
        const int32_t zs = part[src];
        unsigned int crossing = 0;
        for (int64_t q = b + lane; q < e; q += 32) {
            const int32_t zt = part[(int32_t)(syn[q].x & tmask) + tar_base];
            if (zt != zs) {
                ++crossing;
                atomicAdd(&zc[2 * nparts + zt], 1u);
            }
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) crossing += __shfl_xor_sync(0xffffffffu, crossing, o);
        if (lane == 0) {
            atomicAdd(&zc[zs], (unsigned int)(e - b));
            atomicAdd(&zc[nparts + zs], crossing);
        }
    }
    __syncthreads();
    for (int z = threadIdx.x; z < 3 * nparts; z += blockDim.x)
        if (zc[z]) atomicAdd(out + z, (unsigned long long)zc[z]);
}

}  // namespace

extern "C" {

mgc_status mgc_partition_stats(mgc_sim* s, const int32_t* part, int32_t nparts, int64_t* cut, int64_t* zone_neurons,
                               int64_t* zone_syn, int64_t* zone_out, int64_t* zone_in)
{
    if (!s || !part) return fail(MGC_ERR_INVALID, "null argument");
    if (nparts < 1 || nparts > kMaxZones) return fail(MGC_ERR_INVALID, "1..%d zones (got %d)", kMaxZones, nparts);
    const int32_t n = s->n_src;
    std::vector<int64_t> zn(nparts, 0);
    for (int32_t i = 0; i < n; ++i) {
        if (part[i] < 0 || part[i] >= nparts)
            return fail(MGC_ERR_INVALID, "neuron %d in zone %d, outside 0..%d", i, part[i], nparts - 1);
        zn[part[i]] += 1;
    }
    CK(cudaSetDevice(s->device));
    DevTmp tp, to;
    int32_t* dpart;
    unsigned long long* dout;
    CKS(tmp_alloc(tp, &dpart, (size_t)n));
    CKS(tmp_alloc(to, &dout, 3 * (size_t)nparts));
    CK(cudaMemcpyAsync(dpart, part, 4 * (size_t)n, cudaMemcpyHostToDevice, s->stream));
    CK(cudaMemsetAsync(dout, 0, 8 * 3 * (size_t)nparts, s->stream));
    cudaDeviceProp prop;
    CK(cudaGetDeviceProperties(&prop, s->device));
    const size_t smem = 4 * 3 * (size_t)nparts;
    if (smem > 48 * 1024) CKS(allow_shared((const void*)k_partition_stats, s->device));
    // a partition handle's targets are local ids; their zones are those of
    // the whole-network ids from its first neuron on
    k_partition_stats<<<prop.multiProcessorCount * 4, 256, smem, s->stream>>>(s->a.row_ptr, s->a.syn, n, s->a.tmask,
                                                                              s->a.src_base, dpart, nparts, dout);
    CK(cudaGetLastError());
    s->launches += 1;
    std::vector<unsigned long long> h(3 * (size_t)nparts);
    CK(cudaMemcpyAsync(h.data(), dout, 8 * h.size(), cudaMemcpyDeviceToHost, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    int64_t total_cut = 0;
    for (int32_t z = 0; z < nparts; ++z) {
        if (zone_neurons) zone_neurons[z] = zn[z];
        if (zone_syn) zone_syn[z] = (int64_t)h[z];
        if (zone_out) zone_out[z] = (int64_t)h[nparts + z];
        if (zone_in) zone_in[z] = (int64_t)h[2 * nparts + z];
        total_cut += (int64_t)h[nparts + z];
    }
    if (cut) *cut = total_cut;
    return MGC_OK;
}

mgc_status mgc_get_info(mgc_sim* s, mgc_info* info)
{
    if (!s || !info) return fail(MGC_ERR_INVALID, "null argument");
    CK(cudaSetDevice(s->device));
    CK(cudaStreamSynchronize(s->stream));
    memset(info, 0, sizeof(*info));
    info->n_neurons = s->n;
    info->ring_len = s->M;
    info->min_delay = s->dmin;
    info->max_delay = s->dmax;
    info->n_synapses = s->S;
    CK(cudaMemcpy(&info->step, s->a.step, 8, cudaMemcpyDeviceToHost));
    unsigned long long ev = 0;
    CK(cudaMemcpy(&ev, s->a.events, 8, cudaMemcpyDeviceToHost));
    info->events = (int64_t)ev;
    info->mode = s->mode;
    info->graph_steps = s->graph_steps ? s->graph_steps : kGraphSteps;
    info->device_bytes = (int64_t)s->bytes;
    info->persistent = s->a.deferred && !sched_wanted(s) ? s->persistent : 0;
    info->first_neuron = s->a.src_base;
    info->total_neurons = s->n_src;
    info->window = s->fused ? s->window : 0;
    info->accumulation = s->a.fx ? MGC_ACC_FIXED : MGC_ACC_FLOAT;
    info->fx_shift = s->fx_shift;
    return MGC_OK;
}


}  // extern "C"
