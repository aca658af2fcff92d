// The tiled step group's host side: which networks take it, the synapses cut
// by tile, and the kernel instantiations.
#include "sim.h"

using namespace mgc;

namespace mgc {
namespace {

constexpr int kTileRowBlock = 256;
// Above this many neurons, networks with fewer than 4 records a segment keep the
// other step groups: every tile looks up a segment per spike, and at 200,000
// neurons with 2 records a segment a driven step took 9.3 us against 5.8 for
// the windowed group (a quiet one 2.4 against 3.2); at 100,000 neurons with 0.7
// the tiles are the faster form on both loads (1.1 / 3.7 against 2.6 / 4.2).
constexpr int kTileThinNeurons = 1 << 17;

// Networks with several delays whose segment offsets (4 bytes per neuron and tile)
// take more than this keep the other step groups: the look-ups, one per spike and
// tile, then miss L2 (126 MB).  Inputs at 20, 100, 200 and 500 Hz, in-degree 1,000,
// delays of 4 to 8 steps, us a step here and (in brackets) in the other groups:
// 220,000 neurons (130 MB) 2.1, 4.0, 11.1 and 26.8 (5.6, 7.8, 13.3, 25.6), 275,000
// (163 MB) 2.3, 4.9, 14.4 and 33.1 (5.8, 9.6, 14.6, 29.6), 330,000 (195 MB) 2.5, 5.9,
// 17.8 and 39.9 (5.9, 10.5, 15.9, 34.1), 550,000 3.4, 11.2, 31.3 and 77.3 (7.9, 12.3,
// 22.4, 65.1).  With one delay the group stays the faster one at 200 Hz (550,000
// neurons, delay 3: 21.6 against 23.7): a quarter of the record bytes.  So it does with
// a minimum delay of one step, where the others pay two barriers a step (330,000
// neurons, delays of 1 to 5 steps: 7.1, 10.0, 20.5 and 50.5 against 9.6, 14.0, 25.2 and
// 57.2; 495,000 at 200 Hz 30.8 against 26.9, below that 1.2 to 1.3 times as fast).
constexpr int64_t kTileOffsetBytes = 160 << 20;

// The same for networks with fixed-point sums, whose records take 8 bytes: above this
// many synapses the records a driven step reads (with the vectors' padding more than
// the CSR's) outweigh the exchanges saved.  In-degree 1,000, inputs at 20, 100, 200 and
// 500 Hz, delays of 5 to 8 steps: 4e7 synapses 1.4, 4.3, 7.7 and 17.9 us a step (7.5,
// 8.6, 9.2, 14.0), 5e7 1.4, 5.2, 9.4 and 24.9 (7.6, 8.1, 9.5, 16.2), 6e7 1.5, 5.9, 11.2
// and 28.4 (7.5, 8.8, 10.1, 18.2); delays of 10 to 30 at 200 Hz, 4e7 7.3 (9.0), 4.5e7
// 10.3 (9.3).  Not with a minimum delay of one step (1.25e8 synapses at 200 Hz 29
// against 52 to 67).
constexpr int64_t kTileFixedSynapses = 40 << 20;

// Plastic networks: a tile takes its own spikes' incoming plastic synapses one spike
// after another, so long lists keep the ring kernels.  us a step here and (there), the
// inputs at 32 Hz in the mean: 2,000 plastic inputs onto each of 3,000 neurons 7.9 (11.9),
// 3,000 onto 3,000 9.7 (12.7), 4,000 onto 4,000 23.3 (19.6); at 127 Hz 15.4 (14.5), 27.7
// (20.9), 33.8 (24.2).
constexpr uint32_t kTilePlasticInputs = 3072;

// The shortest call that runs in the group.  A launch costs 15 us and more over
// its steps (the state into shared memory and back, an exchange at the end), a step
// of the other forms 3 to 8: calls of 1, 2, 4 and 8 steps took 20.7, 21.3, 22.5 and
// 24.4 us in it and 14.0, 20.6, 33.0 and 58.6 pipelined (36,000 neurons, delays of 18
// steps, 73 spikes a step).  With more neurons than threads in a tile its launch
// costs more: 744 a tile, 34.5, 35.8, 36.6 and 37.5 against 13.2, 19.8, 30.8 and 52.7
// (or 38 windowed).  Plastic networks (784 -> 1,600), one and two steps: 17.0 and
// 22.4, 15.7 and 30.8 with the ring kernels.
int64_t shortest_call(const TileArgs& t, bool stdp)
{
    return stdp ? 2 : 4 + (std::max(0, t.nl - kTileThreads) + 63) / 64;
}

// Records per vector.
__host__ __device__ constexpr int vec_records(bool fx, bool one) { return !fx && one ? 4 : 2; }

// Vectors of every (source, tile) segment, one block per source row at a time;
// with fp32 sums also each neuron's in-degree, the smallest and largest weight
// word per sign, and whether some source has synapses of both signs
// (wstat[5]).
template <bool FX, bool ONE, uint32_t V = vec_records(FX, ONE)>
__global__ void __launch_bounds__(kTileRowBlock) k_tile_count(const int64_t* row_ptr, const uint2* syn, int32_t n_src,
                                                              int32_t T, uint32_t tmask, uint32_t* off,
                                                              uint32_t* indeg, uint32_t* wstat)
{
    __shared__ uint32_t cnt[kMaxTiles];
    uint32_t st[4] = {0xffffffffu, 0u, 0xffffffffu, 0u};  // exc min, max, inh min, max (words)
    for (int64_t row = blockIdx.x; row < n_src; row += gridDim.x) {
        const int64_t b = row_ptr[row], e = row_ptr[row + 1];
        const bool first_exc = !FX && b < e && as_f(syn[b].y) > 0.0f;
        for (int t = threadIdx.x; t < T; t += blockDim.x) cnt[t] = 0;
        __syncthreads();
        for (int64_t p = b + threadIdx.x; p < e; p += blockDim.x) {
            const uint2 w = syn[p];
            const uint32_t tgt = w.x & tmask;
            atomicAdd(cnt + (tgt >> 2) % (uint32_t)T, 1u);
            if (!FX) {
                const float x = as_f(w.y);
                const int h = x > 0.0f ? 0 : 2;
                if ((x > 0.0f) != first_exc) wstat[5] = 1u;
                st[h] = min(st[h], w.y);
                st[h + 1] = max(st[h + 1], w.y);
                atomicAdd(indeg + tgt, 1u);
            }
        }
        __syncthreads();
        for (int t = threadIdx.x; t < T; t += blockDim.x) off[(size_t)row * T + t] = (cnt[t] + V - 1) / V;
        __syncthreads();
    }
    if (!FX) {
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1)
#pragma unroll
            for (int h = 0; h < 4; h += 2) {
                st[h] = min(st[h], __shfl_xor_sync(0xffffffffu, st[h], o));
                st[h + 1] = max(st[h + 1], __shfl_xor_sync(0xffffffffu, st[h + 1], o));
            }
        if ((threadIdx.x & 31) == 0)
            for (int h = 0; h < 4; h += 2) {
                atomicMin(wstat + h, st[h]);
                atomicMax(wstat + h + 1, st[h + 1]);
            }
    }
}

constexpr uint32_t kIndex = 0x7fffffffu;  // off: vector index, the source's sign above (ONE)

// The records into their segments (their order inside a segment does not
// matter: the sums are counts or integers), the last vector filled up.
template <bool FX, bool ONE>
__global__ void __launch_bounds__(kTileRowBlock) k_tile_fill(const int64_t* row_ptr, const uint2* syn, int32_t n_src,
                                                             int32_t T, uint32_t tmask, int tbits, int32_t nl,
                                                             uint32_t* off, void* rec)
{
    __shared__ uint32_t pos[kMaxTiles];
    constexpr uint32_t V = vec_records(FX, ONE);
    auto put = [&](uint32_t at, uint32_t local, uint32_t d, uint32_t w, bool inh) {
        if (FX)
            reinterpret_cast<uint2*>(rec)[at] = make_uint2(local | (d << 16), w);
        else if (ONE)
            reinterpret_cast<uint16_t*>(rec)[at] = (uint16_t)(4u * local);
        else
            reinterpret_cast<uint32_t*>(rec)[at] = local | (d << 16) | (inh ? 0x80000000u : 0u);
    };
    for (int64_t row = blockIdx.x; row < n_src; row += gridDim.x) {
        const int64_t b = row_ptr[row], e = row_ptr[row + 1];
        for (int t = threadIdx.x; t < T; t += blockDim.x) pos[t] = (off[(size_t)row * T + t] & kIndex) * V;
        __syncthreads();
        for (int64_t p = b + threadIdx.x; p < e; p += blockDim.x) {
            const uint2 w = syn[p];
            const uint32_t tgt = w.x & tmask;
            const uint32_t g = tgt >> 2, q = g / (uint32_t)T;
            const uint32_t at = atomicAdd(pos + (g - q * (uint32_t)T), 1u);
            put(at, (q << 2) + (tgt & 3u), w.x >> tbits, w.y, !(as_f(w.y) > 0.0f));
        }
        __syncthreads();
        const uint32_t sign = ONE && b < e && !(as_f(syn[b].y) > 0.0f) ? ~kIndex : 0u;
        for (int t = threadIdx.x; t < T; t += blockDim.x) {
            // (the next entry may belong to another block's row, which sets only its top bit)
            const uint32_t end = (*(volatile uint32_t*)(off + (size_t)row * T + t + 1) & kIndex) * V;
            for (uint32_t at = pos[t]; at < end; ++at) put(at, ONE ? (uint32_t)nl : 0u, 0x7fffu, 0u, false);
            if (sign) off[(size_t)row * T + t] |= sign;
        }
        __syncthreads();
    }
}

// Plastic networks: the records with their plastic flag and CSR position, and
// the plastic synapses onto each local neuron counted.
__global__ void __launch_bounds__(kTileRowBlock) k_tile_fill_stdp(const int64_t* row_ptr, const uint2* syn,
                                                                  const uint8_t* plastic, int32_t n_src, int32_t T,
                                                                  int32_t nl, uint32_t tmask, int tbits,
                                                                  const uint32_t* off, uint2* rec, uint32_t* cpos,
                                                                  uint32_t* in_cnt)
{
    __shared__ uint32_t pos[kMaxTiles];
    for (int64_t row = blockIdx.x; row < n_src; row += gridDim.x) {
        const int64_t b = row_ptr[row], e = row_ptr[row + 1];
        for (int t = threadIdx.x; t < T; t += blockDim.x) pos[t] = off[(size_t)row * T + t];
        __syncthreads();
        for (int64_t p = b + threadIdx.x; p < e; p += blockDim.x) {
            const uint2 w = syn[p];
            const uint32_t tgt = w.x & tmask;
            const uint32_t g = tgt >> 2, q = g / (uint32_t)T, t = g - q * (uint32_t)T;
            const uint32_t local = (q << 2) + (tgt & 3u);
            const bool pl = !plastic || plastic[p];
            const uint32_t at = atomicAdd(pos + t, 1u);
            rec[at] = make_uint2(local | ((w.x >> tbits) << 16) | (pl ? 0x80000000u : 0u), w.y);
            cpos[at] = (uint32_t)p;
            if (pl) atomicAdd(in_cnt + (size_t)t * nl + local, 1u);
        }
        __syncthreads();
    }
}

// The incoming lists {source, record} of the plastic synapses (each synapse is
// updated by itself, so their order does not matter); at: running places.
__global__ void k_tile_in(const uint2* rec, const uint32_t* cpos, const int32_t* csr_src, const uint2* syn, int64_t S,
                          int32_t T, int32_t nl, uint32_t tmask, uint32_t* at, uint2* in_ent)
{
    GRID_STRIDE(r, S)
    {
        const uint2 w = rec[r];
        if (!(w.x >> 31)) continue;
        const uint32_t p = cpos[r];
        const uint32_t t = ((syn[p].x & tmask) >> 2) % (uint32_t)T;
        in_ent[atomicAdd(at + (size_t)t * nl + (w.x & 0xffffu), 1u)] = make_uint2((uint32_t)csr_src[p], (uint32_t)r);
    }
}

// The records' weights from the CSR, after other step forms changed it.
__global__ void k_tile_refresh(const uint2* syn, const uint32_t* cpos, int64_t S, uint2* rec)
{
    GRID_STRIDE(r, S) rec[r].y = syn[cpos[r]].y;
}

// Each neuron's weight per sign: the network's (word of each sign), or from its
// synapses.
__global__ void k_tile_weights(const uint2* syn, int64_t S, uint32_t tmask, float* we, float* wi)
{
    GRID_STRIDE(p, S)
    {
        const uint2 w = syn[p];
        const float x = as_f(w.y);
        (x > 0.0f ? we : wi)[w.x & tmask] = x;
    }
}
__global__ void k_tile_weight(const uint32_t* wstat, int64_t n, float* we, float* wi)
{
    GRID_STRIDE(i, n)
    {
        we[i] = as_f(wstat[0]);
        wi[i] = as_f(wstat[2]);
    }
}

__global__ void k_max_u32(const uint32_t* v, int64_t n, uint32_t* out)
{
    uint32_t m = 0;
    GRID_STRIDE(i, n) m = max(m, v[i]);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// chain[h][k]: k additions of the sign's weight from zero.
__global__ void k_chain(const uint32_t* wstat, float* chain)
{
    const int h = threadIdx.x;
    if (h >= 2) return;
    const float w = as_f(wstat[2 * h]);
    float v = 0.0f;
    for (int k = 0; k < kTileTable; ++k) {
        chain[h * kTileTable + k] = v;
        v = fadd_ftz(v, w);
    }
}

template <bool FX, bool ONE>
static TileKernel tile_of(bool cur)
{
    return cur ? k_tile<true, FX, ONE> : k_tile<false, FX, ONE>;
}

}  // namespace

TileKernel tile_kernel(const mgc_sim* s)
{
    if (s->stdp) return s->a.has_cur ? k_tile_stdp<true> : k_tile_stdp<false>;
    if (s->a.fx) return tile_of<true, false>(s->a.has_cur);
    return s->tile_one ? tile_of<false, true>(s->a.has_cur) : tile_of<false, false>(s->a.has_cur);
}

void drop_tiles(mgc_sim* s)
{
    cudaStreamSynchronize(s->stream);
    TileArgs& t = s->tile;
    for (const void* p : {(const void*)t.off, t.rec, (const void*)t.pend, (const void*)t.pend_step, (const void*)t.we, (const void*)t.wi, (const void*)t.chain,
                          (const void*)t.list, (const void*)t.mail, (const void*)t.cnt, (const void*)t.cpos,
                          (const void*)t.in_off, (const void*)t.in_ent})
        if (p) s->release(const_cast<void*>(p));
    t = TileArgs{};
    s->tile_ok = s->tile_on = false;
}

mgc_status forget_tile_rings(mgc_sim* s)
{
    if (s->tile.pend_step) CK(cudaMemsetAsync(s->tile.pend_step, 0xff, sizeof(int64_t), s->stream));
    return MGC_OK;
}

static mgc_status lay_tiles(mgc_sim* s)
{
    StepArgs& a = s->a;
    const bool stdp = s->stdp && !a.deferred && !a.pull && a.fx;  // the ring method with STDP
    if ((!a.deferred && !stdp) || s->partition || s->S <= 0 || (s->hetero && !a.fx) || s->dmax > kTileMaxDelay)
        return MGC_OK;
    int sms = 0, optin = 0;
    CKS(device_attr(cudaDevAttrMultiProcessorCount, s->device, &sms));
    CKS(device_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin, s->device, &optin));
    sms = std::min(sms, kMaxTiles);
    const bool fx = a.fx != 0, cur = a.has_cur != 0;
    bool one = !fx && s->dmax == s->dmin;  // and one sign per source, checked below
    const size_t room = (size_t)optin - 1024;  // (static shared memory)
    const int64_t groups = a.ns / 4;
    if (a.ns >= (1 << kTileStepShift)) return MGC_OK;
    auto nl_of = [&](int T) { return (int64_t)((groups + T - 1) / T * 4); };
    auto fits = [&](int T) {
        const int64_t nl = nl_of(T);
        if (stdp) return nl < 0x10000 && tile_stdp_bytes((int)nl, s->dmax, T, cur, s->n) <= room;
        return nl < (one ? 0x3fff : 0x10000) && tile_smem_bytes((int)nl, s->dmax, T, fx, cur, !fx) <= room;
    };
    // As many tiles as SMs, fewer only where a mean segment would hold less than half
    // a record: the more tiles, the fewer events a tile (us a step on 16, 32, 64, 100
    // and 148 tiles: volleys of 11,000 neurons 3.41, 2.83, 1.99, 1.59, 1.36; 24 networks
    // in one batch 2.92, 2.93, 0.96, 0.76, 0.62).  Windows of one step are mostly
    // exchange, whose cost grows with the tiles: 4,000 neurons 3.38, 3.09, 2.96, 3.02,
    // 3.18, so up to 7 % are left there.
    int T = (int)std::max<int64_t>(1, std::min<int64_t>({(int64_t)sms, groups, 2 * s->S / s->n}));
    while (T < sms && !fits(T)) ++T;
    const int64_t avg = s->S / ((int64_t)s->n * T);  // records per segment
    if (!fits(T) || 2 * s->S / T < s->n || (avg < 4 && s->n > kTileThinNeurons)) return MGC_OK;
    auto offsets_fit = [&] { return !s->fused || one || 4 * (int64_t)s->n * T <= kTileOffsetBytes; };
    if (!offsets_fit() || (fx && s->fused && s->S > kTileFixedSynapses)) return MGC_OK;
    const size_t vec_bytes = fx ? 16 : 8;
    // at most one vector in each segment is not full
    const size_t most = ((size_t)s->S / 2 + (size_t)s->n * T) * vec_bytes;
    const int W = stdp ? 1 : std::min(kTileWindow, s->dmin);
    const size_t ring = stdp ? 0 : (fx ? 16 : 4) * (size_t)s->dmax * tile_stride((int)nl_of(T));  // of a tile
    const size_t need = most + (stdp ? 12 * (size_t)s->S : 0) + ((size_t)s->n * T + 1) * 4 +
                        kTileLists * (size_t)W * nl_of(T) * T * 4 + 32 * (size_t)T * T * kTileChunks +
                        16 * (size_t)a.ns + ring * T;
    // offsets in vectors, and in records while they are filled
    if ((int64_t)s->n * T + 1 > (int64_t)0x7fffffff || most / vec_bytes > kIndex / 2) return MGC_OK;
    size_t free_b = 0, total_b = 0;
    CK(cudaMemGetInfo(&free_b, &total_b));
    // the copy only saves time: it leaves seven eighths of what is free to others
    if (need > free_b / 8) return MGC_OK;
    TileArgs& t = s->tile;
    t.T = T;
    t.nl = (int32_t)nl_of(T);
    t.stride = tile_stride(t.nl);
    t.R = s->dmax;
    t.W = W;
    t.dmin = s->dmin;
    t.dmax = s->dmax;
    t.ahead = s->fused ? 1 : 0;
    s->tile_min = shortest_call(t, stdp);
    uint32_t* off;
    float *we = nullptr, *wi = nullptr, *chain = nullptr;
    CKS(s->alloc(&off, (size_t)s->n * T + 1, false));
    t.off = off;
    CKS(s->alloc(&t.list, kTileLists * (size_t)T * t.nl * W, false));
    CKS(s->alloc(&t.mail, 2 * (size_t)T * T * kTileChunks));
    t.epoch = 1;
    CKS(s->alloc(&t.cnt, 4 * kTileWindow * kTileLine));
    if (!stdp) {
        char* pend;
        CKS(s->alloc(&pend, ring * T, false));
        t.pend = pend;
        CKS(s->alloc(&t.pend_step, 1, false));
        CKS(forget_tile_rings(s));
    }
    DevTmp t_deg, t_stat;
    uint32_t *indeg = nullptr, *wstat = nullptr;
    if (!fx) {
        CKS(s->alloc(&we, a.ns));
        t.we = we;
        CKS(s->alloc(&wi, a.ns));
        t.wi = wi;
        CKS(s->alloc(&chain, 2 * kTileTable, false));
        t.chain = chain;
        CKS(tmp_alloc(t_deg, &indeg, a.ns));
        CKS(tmp_alloc(t_stat, &wstat, 6));
        const uint32_t init[6] = {0xffffffffu, 0u, 0xffffffffu, 0u, 0u, 0u};
        CK(cudaMemsetAsync(indeg, 0, 4 * (size_t)a.ns, s->stream));
        CK(cudaMemcpyAsync(wstat, init, sizeof(init), cudaMemcpyHostToDevice, s->stream));
    }
    const int grid = (int)std::min<int64_t>(s->n, (int64_t)sms * 8);
    uint32_t h[6] = {};
    auto count = [&]() -> mgc_status {
        auto k = stdp ? k_tile_count<true, false, 1> : fx ? k_tile_count<true, false> : (one ? k_tile_count<false, true> : k_tile_count<false, false>);
        k<<<grid, kTileRowBlock, 0, s->stream>>>(a.row_ptr, a.syn, s->n, T, a.tmask, off, indeg, wstat);
        CKS(scan_offsets(off, (int64_t)s->n * T, s->stream));
        if (!fx) {
            k_max_u32<<<grid_for(a.ns), 256, 0, s->stream>>>(indeg, a.ns, wstat + 4);
            k_chain<<<1, 32, 0, s->stream>>>(wstat, chain);
            CK(cudaMemcpyAsync(h, wstat, sizeof(h), cudaMemcpyDeviceToHost, s->stream));
        }
        CK(cudaMemcpyAsync(&t.n_vec, off + (size_t)s->n * T, 4, cudaMemcpyDeviceToHost, s->stream));
        CK(cudaStreamSynchronize(s->stream));
        return MGC_OK;
    };
    CKS(count());
    if (one && h[5]) {  // a source with synapses of both signs: a sign in every record
        one = false;
        if (!offsets_fit()) {
            drop_tiles(s);
            return MGC_OK;
        }
        CK(cudaMemsetAsync(indeg, 0, 4 * (size_t)a.ns, s->stream));
        CKS(count());
    }
    if (!fx) {
        if (h[4] > 0xffffu) {  // a step's count of one sign might not fit its half word
            drop_tiles(s);
            return MGC_OK;
        }
        t.table = (h[0] >= h[1] && h[2] >= h[3]) ? 1 : 0;
        if (t.table)
            k_tile_weight<<<grid_for(a.ns), 256, 0, s->stream>>>(wstat, a.ns, we, wi);
        else
            k_tile_weights<<<grid_for(s->S), 256, 0, s->stream>>>(a.syn, s->S, a.tmask, we, wi);
    }
    t.lanes_log2 = avg < 10 * vec_records(fx, one) ? 0 : 2;
    if (stdp) {
        uint2 *srec, *in_ent;
        uint32_t *cpos, *in_off;
        const int64_t locals = (int64_t)T * t.nl;
        CKS(s->alloc(&srec, s->S, false));
        t.rec = srec;
        CKS(s->alloc(&cpos, s->S, false));
        t.cpos = cpos;
        CKS(s->alloc(&in_off, locals + 1));
        t.in_off = in_off;
        DevTmp t_at;
        uint32_t* at;
        CKS(tmp_alloc(t_at, &at, locals + 1));
        k_tile_fill_stdp<<<grid, kTileRowBlock, 0, s->stream>>>(a.row_ptr, a.syn, a.plastic, s->n, T, t.nl, a.tmask,
                                                                a.tbits, off, srec, cpos, in_off);
        uint32_t n_in = 0, longest = 0;
        DevTmp t_max;
        uint32_t* d_max;
        CKS(tmp_alloc(t_max, &d_max, 1));
        CK(cudaMemsetAsync(d_max, 0, 4, s->stream));
        k_max_u32<<<grid_for(locals), 256, 0, s->stream>>>(in_off, locals, d_max);
        CK(cudaMemcpyAsync(&longest, d_max, 4, cudaMemcpyDeviceToHost, s->stream));
        CK(cudaStreamSynchronize(s->stream));
        if (longest > kTilePlasticInputs) {
            drop_tiles(s);
            return MGC_OK;
        }
        CKS(scan_offsets(in_off, locals, s->stream));
        CK(cudaMemcpyAsync(&n_in, in_off + locals, 4, cudaMemcpyDeviceToHost, s->stream));
        CK(cudaMemcpyAsync(at, in_off, 4 * (size_t)locals, cudaMemcpyDeviceToDevice, s->stream));
        CK(cudaStreamSynchronize(s->stream));
        CKS(s->alloc(&in_ent, n_in, false));
        t.in_ent = in_ent;
        k_tile_in<<<grid_for(s->S), 256, 0, s->stream>>>(srec, cpos, a.csr_src, a.syn, s->S, T, t.nl, a.tmask, at,
                                                         in_ent);
        CK(cudaGetLastError());
        CK(cudaStreamSynchronize(s->stream));
        s->tile_smem = tile_stdp_bytes(t.nl, t.R, T, cur, s->n);
        CKS(allow_shared((const void*)tile_kernel(s), s->device));
        s->tile_ok = true;
        s->tile_on = s->tile_wanted;
        s->tile_stale = false;
        return MGC_OK;
    }
    char* rec;
    CKS(s->alloc(&rec, std::max<size_t>(1, t.n_vec) * vec_bytes, false));
    t.rec = rec;
    auto fill = fx ? k_tile_fill<true, false> : (one ? k_tile_fill<false, true> : k_tile_fill<false, false>);
    fill<<<grid, kTileRowBlock, 0, s->stream>>>(a.row_ptr, a.syn, s->n, T, a.tmask, a.tbits, t.nl, off, rec);
    CK(cudaGetLastError());
    s->tile_one = one;
    s->tile_smem = tile_smem_bytes(t.nl, t.R, T, fx, cur, t.table != 0);
    CKS(allow_shared((const void*)tile_kernel(s), s->device));
    s->tile_ok = true;
    s->tile_on = s->tile_wanted;
    return MGC_OK;
}

static size_t mail_bytes(const TileArgs& t) { return 2 * (size_t)t.T * t.T * kTileChunks * sizeof(ulonglong2); }

mgc_status build_tiles(mgc_sim* s)
{
    drop_tiles(s);
    const mgc_status st = lay_tiles(s);
    if (st == MGC_OK) return st;
    drop_tiles(s);
    return st == MGC_ERR_NOMEM ? MGC_OK : st;  // the network runs without them
}

cudaError_t launch_tiles(mgc_sim* s, StepArgs& a, int32_t n, int32_t blocks)
{
    const uint32_t windows = (uint32_t)((n + s->tile.W - 1) / s->tile.W + 1);  // and the end
    if (s->tile.epoch > 0xffffffffu - windows) {
        // epochs that wrapped would meet chunks last written 2^32 windows ago
        const cudaError_t e = cudaMemsetAsync(s->tile.mail, 0, mail_bytes(s->tile), s->stream);
        if (e != cudaSuccess) return e;
        s->tile.epoch = 1;
    }
    void* args[] = {&a, &s->tile, &n};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)tile_kernel(s), dim3(blocks), dim3(kTileThreads),
                                                      args, s->tile_smem, s->stream);
    if (e == cudaSuccess) s->tile.epoch += windows;
    return e;
}

mgc_status clear_tile_counters(mgc_sim* s)
{
    if (s->tile.cnt) CK(cudaMemsetAsync(s->tile.cnt, 0, 4 * sizeof(int32_t) * kTileWindow * kTileLine, s->stream));
    CK(cudaMemsetAsync(s->a.done, 0, sizeof(unsigned int), s->stream));
    return MGC_OK;
}

mgc_status refresh_tiles(mgc_sim* s)
{
    if (!s->tile_stale) return MGC_OK;
    k_tile_refresh<<<grid_for(s->S), 256, 0, s->stream>>>(s->a.syn, s->tile.cpos, s->S,
                                                           static_cast<uint2*>(const_cast<void*>(s->tile.rec)));
    CK(cudaGetLastError());
    s->launches += 1;
    s->tile_stale = false;
    return MGC_OK;
}

}  // namespace mgc

extern "C" mgc_status mgc_selftest_tile_timeout(mgc_sim* s)
{
    if (!s) return fail(MGC_ERR_INVALID, "null handle");
    if (!s->tile_on || s->tile.T < 2) return fail(MGC_ERR_INVALID, "the handle's steps do not run on two or more tiles");
    CK(cudaSetDevice(s->device));
    CKS(refresh_tiles(s));
    StepArgs a = s->a;
    a.trace = nullptr;
    CK(launch_tiles(s, a, 1, s->tile.T - 1));  // the last tile's block never publishes
    s->launches += 1;
    return MGC_OK;
}

extern "C" mgc_status mgc_selftest_tile_epoch(mgc_sim* s, uint32_t epoch)
{
    if (!s || epoch == 0) return fail(MGC_ERR_INVALID, "null handle, or epoch 0");
    if (!s->tile_on) return fail(MGC_ERR_INVALID, "the handle's steps do not run on tiles");
    CK(cudaSetDevice(s->device));
    CK(cudaMemsetAsync(s->tile.mail, 0, mail_bytes(s->tile), s->stream));  // as if the epochs up to it had passed
    s->tile.epoch = epoch;
    return MGC_OK;
}
