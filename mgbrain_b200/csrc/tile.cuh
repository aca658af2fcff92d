// Tiled step group (deferred method, networks whose state fits on the chip):
// the neurons are dealt to one block per SM ("tiles"), each block keeps its
// neurons' state and their input of the steps to come in shared memory for
// the whole launch, and delivers every spike to its own targets itself,
// from a copy of the synapses cut by tile.  An event is then one
// shared-memory reduction; only spike ids cross between blocks, once per
// window of W <= minimum delay steps.
//
// What bounds it: the step forms that reduce into L2 run at the chip's rate
// of scattered reductions (1.64e11/s measured) plus two or more grid barriers
// and about seven dependent L2 round trips per window or step; here the
// events are bounded by the shared-memory atomics and the instructions of
// 148 SMs, and a window pays one exchange (a store and a poll) and two or
// three dependent round trips (spike ids beyond the first two of a tile,
// segment offsets, records).
//
// Layout: neuron group g (four neurons) belongs to tile g % T as its local
// group g / T, so that populations (POISSON inputs, inhibitory cells) spread
// evenly.  The synapses of source s towards tile t are the records
// [off[s*T + t], off[s*T + t + 1]); a record is
//   one delay, fp32 sums     16 bits: 4 * local target, the sign of the source's
//     (one sign per source)  synapses in bit 31 of off
//   several delays, fp32     32 bits: local target | delay << 16 | sign << 31
//   fixed-point sums         64 bits: local target | delay << 16, weight
// read as vectors of 8 bytes (16 with fixed point); a segment is filled up to
// whole vectors (off counts vectors) with records that go nowhere.
// With fp32 sums every neuron receives one weight per sign (the handle uses
// the tiles only then), so the input of a step is a count per sign, kept as
// two 16-bit halves of one word, and the fp32 sum is the chain of `count`
// additions of the weight from zero with red.add's rounding: the bits the
// scattered reductions give in any order.  Fixed-point sums are the exact
// 64-bit integers.  So every result equals the other step forms' bit for bit.
//
// Input ring: the arrivals of step x in slot x % R, R = the longest delay: a
// window's updates clear its W slots before its spikes are delivered, which
// arrive W to W - 1 + R steps after its first step.  The group starts and
// ends in the state of the single-step kernels: the prologue delivers the
// spikes of the history that arrive after the first step (whose arrivals the
// accumulators hold), the last windows' spikes are written into the
// history, and the arrivals of the step after the last go into the
// accumulators.  With a minimum delay of one step the single-step kernels
// start a step without its arrivals; there the prologue includes them and
// the accumulators stay empty.
//
// Exchange of window k: a tile writes its spikes (id, step in the window) into
// its list of buffer k & 1, then sends every tile a 16-byte header {epoch of
// the window and count, first two spikes}, one store each, into that tile's
// mailbox; thread l of a block polls the place of tile l in its own mailbox,
// which no other block reads.  No counter is shared, so no atomic waits its
// turn, no line is polled by more than one block, and a quiet window's spikes
// arrive with the poll; only a tile with more spikes than the header carries
// orders its list before the header with a fence, and only their readers
// wait for one.  (One set of headers polled by all blocks, with a release
// store: 5.0 us an exchange on 148 tiles; mailboxes: see DESIGN.)  A tile
// overwrites a buffer two windows later, when every tile has published the
// window between, which it does after reading the buffer.  Waits are bounded
// (kStatusBarrier).
//
// Raster: a step's place in it needs the step's spikes of all tiles, so each
// tile adds its counts to the window's 16 step counters when it publishes,
// and writes its spikes' places one window later, when every tile's counts
// are in: none of it is waited for.  The counters of window k (slot k % 4)
// are read in window k+1 before its deliveries end and cleared by tile 0 in
// window k+3, before anyone adds to them again in window k+4.
#pragma once
#include "kernels.cuh"

namespace mgc {

constexpr int kTileThreads = 512;   // 128 registers a thread: no spills (768 and 1,024 threads spill and ran slower)
constexpr int kTileWindow = 16;     // longest window (a neuron's spikes of a window: 16 bits)
constexpr int kTileMaxDelay = 512;  // longest delay (the prologue's prefix, shared memory)
constexpr int kTileTable = 512;     // entries of each chain table

struct TileArgs {
    int32_t T;            // tiles = blocks
    int32_t nl;           // neurons per tile (a multiple of 4)
    int32_t stride;       // entries of a ring row: nl, a spare one for fillers, padding
    int32_t R;            // ring slots: the longest delay
    int32_t W;            // steps per window (<= minimum delay)
    int32_t dmin, dmax;
    int32_t lanes_log2;   // lanes that share a segment in the delivery (0: one lane a segment)
    int32_t table;        // one weight per sign in the whole network: chains from the tables
    int32_t ahead;        // the accumulators hold the first step's arrivals (minimum delay >= 2)
    uint32_t n_vec;       // vectors of records
    const uint32_t* off;  // [n*T + 1]
    const void* rec;
    const float* we;      // [ns] weight per sign of each neuron (fp32 sums)
    const float* wi;
    const float* chain;   // [2][kTileTable] sums of k weights (exc, inh), when table
    uint32_t* list;       // [2][T][nl*W] spikes of a window: id | step in the window << 28
    ulonglong2* mail;     // [2][T reader][T] headers {epoch << 32 | count, first spikes}
    uint32_t epoch;       // epoch of the launch's first window (they count on over the launches)
    int32_t* cnt;         // [4][kTileWindow] spikes of a window's steps; zero between launches
    // plastic networks (k_tile_stdp): rec holds single records (off counts them)
    const uint32_t* cpos;   // [S] CSR position of a record
    const uint32_t* in_off; // [T*nl + 1] plastic synapses onto each local neuron, tile after tile:
    const uint2* in_ent;    //   {source, record}
};

constexpr int kTileInline = 2;      // spikes a header carries
constexpr int kTileSpikes = 4096;   // spikes of a window gathered in shared memory
constexpr int kTileStepShift = 28;  // spike word: id below, step in the window above

// Shared memory of a block, in this order.
struct TileSmem {
    void* ring;       // FLOAT: u32 [R][stride]; FIXED: u64 [2][R][stride]
    float *V, *we, *wi, *ie, *ii, *tab;
    int32_t* rf;
    int32_t* cnt;     // spikes of each list (a window's tiles, the prologue's steps)
    int32_t* at;      // [T] a tile's place in `spikes`
    uint32_t* spikes; // [kTileSpikes] a window's spikes, when they fit
    uint16_t* pg;     // [nl/4] local groups with POISSON neurons
    int8_t* type;
};

// A ring row: nl entries and the fillers' one, a multiple of 4.
__host__ __device__ inline int tile_stride(int nl) { return nl + 4; }

__host__ __device__ inline int tile_lists(int R, int T) { return R > T ? R : T; }

__host__ __device__ inline size_t tile_smem_bytes(int nl, int R, int T, bool fx, bool cur, bool table)
{
    const size_t per = 8 + (fx ? 0 : 8) + (cur ? 8 : 0) + 1;
    return (fx ? 16 : 4) * (size_t)R * (size_t)tile_stride(nl) + per * (size_t)nl + 4 * (size_t)(tile_lists(R, T) + T) +
           4 * (size_t)kTileSpikes + (size_t)nl / 2 + (table ? 8 * (size_t)kTileTable : 0) + 64;
}

template <bool CUR, bool FX>
__device__ __forceinline__ TileSmem tile_smem(unsigned char* base, const TileArgs& t)
{
    TileSmem m{};
    unsigned char* p = base;
    const size_t nl = t.nl;
    m.ring = p;
    p += (FX ? 16 : 4) * (size_t)t.R * t.stride;
    auto take_f = [&](size_t n) {
        float* q = reinterpret_cast<float*>(p);
        p += 4 * n;
        return q;
    };
    m.V = take_f(nl);
    m.rf = reinterpret_cast<int32_t*>(take_f(nl));
    if (!FX) {
        m.we = take_f(nl);
        m.wi = take_f(nl);
        if (t.table) m.tab = take_f(2 * kTileTable);
    }
    if (CUR) {
        m.ie = take_f(nl);
        m.ii = take_f(nl);
    }
    m.cnt = reinterpret_cast<int32_t*>(take_f(tile_lists(t.R, t.T)));
    m.at = reinterpret_cast<int32_t*>(take_f(t.T));
    m.spikes = reinterpret_cast<uint32_t*>(take_f(kTileSpikes));
    m.pg = reinterpret_cast<uint16_t*>(p);
    p += nl / 2;
    m.type = reinterpret_cast<int8_t*>(p);
    return m;
}

// Network neuron of local neuron i of this block's tile.
__device__ __forceinline__ int32_t tile_neuron(const TileArgs& t, int i, int tile)
{
    return (((i >> 2) * t.T + tile) << 2) + (i & 3);
}

// The sum of c additions of w from zero, as red.add.f32 makes it.
__device__ __forceinline__ float chain_sum(uint32_t c, float w, const float* tab)
{
    float v = 0.0f;
    if (tab && c) {
        const uint32_t k = c < kTileTable ? c : kTileTable - 1;
        v = tab[k];
        c -= k;
    }
    for (; c; --c) v = fadd_ftz(v, w);
    return v;
}

// A neuron's spikes of a window (bit j: step w0 + j) into the tile's list.
__device__ __forceinline__ void tile_spikes(const TileArgs& t, int32_t gi, uint32_t fm, uint32_t* list,
                                            uint32_t* first, int* count, int* scnt)
{
    int pos = atomicAdd(count, __popc(fm));
    for (; fm; fm &= fm - 1, ++pos) {
        const int j = __ffs(fm) - 1;
        atomicAdd(scnt + j, 1);
        const uint32_t e = (uint32_t)gi | ((uint32_t)j << kTileStepShift);
        if (pos < kTileInline) first[pos] = e;
        if (pos < t.nl * t.W) list[pos] = e;
    }
}

// The tile's POISSON neurons through the wl steps from w0: a thread takes
// one group of four neurons and one step, whose draws are one Philox block.
// Threads from the block's end, since the other neurons start at its front.
__device__ __forceinline__ void tile_poisson(const StepArgs& a, const TileArgs& t, const TileSmem& m, int64_t w0,
                                             int wl, int npg, uint32_t* list, uint32_t* first, int* count, int* scnt)
{
    for (int x = blockDim.x - 1 - threadIdx.x; x < npg * wl; x += blockDim.x) {
        const int j = x / npg, g = m.pg[x - j * npg];
        const int32_t gi = tile_neuron(t, 4 * g, blockIdx.x);
        float u[4];
        poisson_uniform4(a.seed, (int64_t)gi + a.id_offset, w0 + j, u);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (m.type[4 * g + q] != kPOISSON || !(m.V[4 * g + q] > u[q])) continue;  // (V holds the probability)
            atomicAdd(a.fire_cnt + gi + q, 1);
            atomicMax(a.last_fired + gi + q, (int32_t)(w0 + j));  // another thread has the group's other steps
            tile_spikes(t, gi + q, 1u << j, list, first, count, scnt);
        }
    }
}

// The tile's other neurons through the wl steps from w0 (ring slot `slot`),
// one neuron a lane, four steps at a time.  `from_acc`: the first step's
// input is in the accumulators (the launch's first step), which are cleared.
// The spikes go into `list` (and `first`), counted in *count and per step.
// Warps without LIF or LIFE neurons take lifb_step for every lane and keep
// its result where the neuron is LIFB: no branches, few instructions (a
// window's update is one warp's chain of dependent instructions).
template <bool CUR, bool FX>
__device__ __forceinline__ void tile_update(const StepArgs& a, const TileArgs& t, const TileSmem& m, int64_t w0,
                                            int wl, int slot, bool from_acc, uint32_t* list, uint32_t* first,
                                            int* count, int* scnt)
{
    const int lane = threadIdx.x & 31;
    const int tile = blockIdx.x;
    const int plane = t.R * t.stride;  // fixed point: the inh sums follow the exc ones
    for (int b = threadIdx.x - lane; b < t.nl; b += blockDim.x) {
        const int i = b + lane;
        const int type = i < t.nl ? m.type[i] : (int)kRAW;
        const bool input = i < t.nl && type != kPOISSON;
        if (!__any_sync(0xffffffffu, input && type != kRAW)) continue;  // (padding is RAW)
        const int32_t gi = tile_neuron(t, i, tile);
        float v = 0.f, we = 0.f, wi = 0.f, ie = 0.f, ii = 0.f;
        int32_t rf = 0;
        if (input) {
            v = m.V[i];
            rf = m.rf[i];
            if (!FX) {
                we = m.we[i];
                wi = m.wi[i];
            }
            if (CUR) {
                ie = m.ie[i];
                ii = m.ii[i];
            }
        }
        const bool lifb = type == kLIFB;
        const bool any_cur = CUR && __any_sync(0xffffffffu, type == kLIF || type == kLIFE);
        uint32_t fm = 0;
        int row = slot;
#pragma unroll 1
        for (int h = 0; h < wl; h += 4) {
            float re[4], ri[4];
            int at[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                at[k] = row * t.stride + i;
                row = row + 1 == t.R ? 0 : row + 1;
            }
            if (FX) {
                long long* ring = reinterpret_cast<long long*>(m.ring);
                long long fe[4], fi[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    fe[k] = fi[k] = 0;
                    if (input && h + k < wl) {
                        fe[k] = ring[at[k]];
                        fi[k] = ring[plane + at[k]];
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (fe[k] | fi[k]) ring[at[k]] = ring[plane + at[k]] = 0;
                    re[k] = from_fx(fe[k], a.fx_unscale);
                    ri[k] = from_fx(fi[k], a.fx_unscale);
                }
            } else {
                uint32_t* ring = reinterpret_cast<uint32_t*>(m.ring);
                uint32_t c[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    c[k] = 0;
                    if (input && h + k < wl) {
                        c[k] = ring[at[k]];
                        ring[at[k]] = 0;
                    }
                }
                if (m.tab) {  // tab[0] is 0; counts past the tables are finished one by one
                    constexpr uint32_t kMask = kTileTable - 1;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        re[k] = m.tab[c[k] & kMask];
                        ri[k] = m.tab[kTileTable + ((c[k] >> 16) & kMask)];
                    }
                    if ((c[0] | c[1] | c[2] | c[3]) & ~(kMask | (kMask << 16))) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            re[k] = chain_sum(c[k] & 0xffffu, we, m.tab);
                            ri[k] = chain_sum(c[k] >> 16, wi, m.tab + kTileTable);
                        }
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        re[k] = chain_sum(c[k] & 0xffffu, we, nullptr);
                        ri[k] = chain_sum(c[k] >> 16, wi, nullptr);
                    }
                }
            }
            if (from_acc && h == 0 && input && gi < a.ns) {
                typename AccT<FX>::type* pe = acc_buf<FX>(a, a.acc_e, w0) + gi;
                typename AccT<FX>::type* pi = acc_buf<FX>(a, a.acc_i, w0) + gi;
                if (FX) {
                    re[0] = from_fx((long long)*pe, a.fx_unscale);
                    ri[0] = from_fx((long long)*pi, a.fx_unscale);
                } else {
                    re[0] = *pe;
                    ri[0] = *pi;
                }
                *pe = 0;
                *pi = 0;
            }
            if (any_cur) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (h + k < wl && input)
                        fm |= (update_one<false>(a, type, gi, w0 + h + k, v, rf, re[k], ri[k], ie, ii, 0.f) ? 1u : 0u)
                              << (h + k);
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float nv = v;
                    int32_t nr = rf;
                    const bool go = lifb && h + k < wl;  // the window's last batch may be partial
                    const bool f = lifb_step(a, nv, nr, re[k], ri[k]) && go;
                    v = go ? nv : v;
                    rf = go ? nr : rf;
                    fm |= (f ? 1u : 0u) << (h + k);
                }
            }
        }
        if (input) {
            m.V[i] = v;
            m.rf[i] = rf;
            if (CUR) {
                m.ie[i] = ie;
                m.ii[i] = ii;
            }
            if (fm) {
                atomicAdd(a.fire_cnt + gi, __popc(fm));
                a.last_fired[gi] = (int32_t)(w0 + (31 - __clz(fm)));
                tile_spikes(t, gi, fm, list, first, count, scnt);
            }
        }
    }
}

// One record into the ring.  base: the ring row of the spike's step (ONE: of
// its arrival step); j: the step's place in the batch.
template <bool FX, bool ONE>
__device__ __forceinline__ void tile_apply(const StepArgs& a, const TileArgs& t, const TileSmem& m, uint32_t x,
                                           uint32_t wbits, int base, int j, int lo_rel, unsigned span, uint32_t& ev)
{
    if (ONE) {  // base: byte offset of the row | the sign; fillers go to the row's spare column
        if (!MGC_OK_INDEX((x >> 2) < (uint32_t)t.stride && !(x & 3u))) return;
        atomicAdd(reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(m.ring) + ((base & ~1) + x)),
                  (base & 1) ? 0x10000u : 1u);
    } else {    // a filler's delay is past every arrival window
        const int d = (int)((x >> 16) & 0x7fffu);
        if ((unsigned)(j + d - lo_rel - 1) >= span) return;
        int row = base + d;
        if (row >= t.R) row -= t.R;
        if (!MGC_OK_INDEX(row < t.R && (x & 0xffffu) < (uint32_t)t.nl)) return;
        ++ev;
        const int at = row * t.stride + (int)(x & 0xffffu);
        if (FX) {
            const float w = as_f(wbits);
            unsigned long long* ring = reinterpret_cast<unsigned long long*>(m.ring);
            if (!(w > 0.0f)) ring += (size_t)t.R * t.stride;
            atomicAdd(ring + at, (unsigned long long)to_fx(w, a.fx_scale));
        } else {
            atomicAdd(reinterpret_cast<uint32_t*>(m.ring) + at, (x >> 31) ? 0x10000u : 1u);
        }
    }
}

// One vector of records: 8 bytes (four 16-bit or two 32-bit records), or 16
// (two fixed-point records).
template <bool FX> struct TileVec { using type = uint2; };
template <> struct TileVec<true> { using type = uint4; };

template <bool FX, bool ONE>
__device__ __forceinline__ void tile_apply_vec(const StepArgs& a, const TileArgs& t, const TileSmem& m,
                                               const typename TileVec<FX>::type& v, int base, int j, int lo_rel,
                                               unsigned span, uint32_t& ev)
{
    if constexpr (FX) {
        tile_apply<FX, ONE>(a, t, m, v.x, v.y, base, j, lo_rel, span, ev);
        tile_apply<FX, ONE>(a, t, m, v.z, v.w, base, j, lo_rel, span, ev);
    } else if constexpr (ONE) {
        tile_apply<FX, ONE>(a, t, m, v.x & 0xffffu, 0u, base, j, lo_rel, span, ev);
        tile_apply<FX, ONE>(a, t, m, v.x >> 16, 0u, base, j, lo_rel, span, ev);
        tile_apply<FX, ONE>(a, t, m, v.y & 0xffffu, 0u, base, j, lo_rel, span, ev);
        tile_apply<FX, ONE>(a, t, m, v.y >> 16, 0u, base, j, lo_rel, span, ev);
    } else {
        tile_apply<FX, ONE>(a, t, m, v.x, 0u, base, j, lo_rel, span, ev);
        tile_apply<FX, ONE>(a, t, m, v.y, 0u, base, j, lo_rel, span, ev);
    }
}

// Where a warp's batches of spikes come from: begin(n) starts its next batch
// (false: none left; n <= 32 U spikes), load(i, j) returns spike i of the batch
// and its step (j steps after the first).
constexpr int kTileU = 2;           // segments a lane takes in a batch
constexpr int kTileD = 4;           // 8-byte vectors of each it loads at once (half as many of 16)
constexpr int kTileBatch = 32 * kTileU;
constexpr uint32_t kTileId = (1u << kTileStepShift) - 1u;

struct TileGathered {  // the window's spikes in shared memory
    const uint32_t* spikes;
    int total, per, next, at;
    __device__ TileGathered(const uint32_t* sp, int n) : spikes(sp), total(n)
    {
        const int nw = blockDim.x >> 5, need = (n + nw - 1) / nw;
        per = need < kTileBatch ? (need > 0 ? need : 1) : kTileBatch;
        next = (threadIdx.x >> 5) * per;
        at = 0;
    }
    __device__ __forceinline__ bool begin(int& n)
    {
        at = next;
        n = min(per, total - at);
        next += (blockDim.x >> 5) * per;
        return n > 0;
    }
    __device__ __forceinline__ int32_t load(int i, int& j) const
    {
        const uint32_t e = spikes[at + i];
        j = (int)(e >> kTileStepShift);
        return (int32_t)(e & kTileId);
    }
};

// Lists in device memory (get(l, q, j): spike q of list l), cut into batches
// dealt to the block's warps in turn; cnt: their lengths, in shared memory.
template <class Get> struct TileListed {
    Get get;
    const int32_t* cnt;
    int lists, l, q, skip, cl, cq;
    __device__ TileListed(Get g, const int32_t* c, int n) : get(g), cnt(c), lists(n), l(0), q(0), cl(0), cq(0)
    {
        skip = threadIdx.x >> 5;
    }
    __device__ __forceinline__ bool begin(int& n)
    {
        q += skip;
        skip = blockDim.x >> 5;
        int b = 0;
        for (; l < lists; ++l, q -= b) {
            b = (cnt[l] + kTileBatch - 1) / kTileBatch;
            if (q < b) break;
        }
        if (l >= lists) return false;
        cl = l;
        cq = q * kTileBatch;
        n = min(kTileBatch, cnt[l] - cq);
        return true;
    }
    __device__ __forceinline__ int32_t load(int i, int& j) const { return get(cl, cq + i, j); }
};

// Delivers spikes of the steps x0, x0+1, ... to this tile's targets: the
// records whose arrival step is in (lo, hi].  slot0: the ring slot of x0.
// A warp's batches run as a pipeline of three dependent loads: the spike ids
// of the batch after next, the segment offsets of the next and the records
// of this one are in flight together, and a lane loads kTileD vectors of each
// of its segments at once, so that a batch waits for about one round trip to
// L2 (walking a segment one vector at a time, with no batch ahead, took 7.6 us
// a batch).  Long segments are shared by 1 << lanes_log2 lanes.
template <bool FX, bool ONE, class Src>
__device__ __forceinline__ void tile_deliver(const StepArgs& a, const TileArgs& t, const TileSmem& m, int64_t x0,
                                             int slot0, int64_t lo, int64_t hi, Src src, unsigned long long& events)
{
    using Vec = typename TileVec<FX>::type;
    constexpr int U = kTileU, D = FX ? kTileD / 2 : kTileD;
    const Vec* rec = reinterpret_cast<const Vec*>(t.rec);
    const int lane = threadIdx.x & 31;
    // arrival windows relative to x0, as one unsigned comparison
    const int64_t hr = hi - x0, lr = lo - x0;
    const int lo_rel = (int)(lr < -1 ? -1 : lr);
    const int hi_rel = (int)(hr > 4 * kTileMaxDelay ? 4 * kTileMaxDelay : hr);
    const unsigned span = hi_rel > lo_rel ? (unsigned)(hi_rel - lo_rel) : 0u;
    uint32_t ev = 0;

    struct Seg {
        uint32_t k, e;
        int base, j;
    };
    int32_t id1[U];  // ids and steps of the batch whose offsets come next
    int j1[U];
    Seg s0[U];       // segments of the batch to deliver
    auto ids = [&](bool any, int n) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            id1[u] = -1;
            j1[u] = 0;
            if (any && u * 32 + lane < n) id1[u] = src.load(u * 32 + lane, j1[u]);
        }
    };
    auto offsets = [&]() {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            Seg& g = s0[u];
            g.k = g.e = 0;
            if (id1[u] >= 0 && MGC_OK_INDEX(id1[u] < a.n_src)) {
                const uint32_t* o = t.off + (size_t)id1[u] * t.T + blockIdx.x;
                g.k = __ldg(o);
                g.e = __ldg(o + 1);
            }
            g.j = j1[u];
        }
    };
    int n0 = 0, n1 = 0;
    bool more = src.begin(n1);
    if (!more) return;
    ids(true, n1);
    offsets();
    n0 = n1;
    more = src.begin(n1);
    ids(more, n1);
    for (;;) {
        // this batch's segments, their first vectors
        Seg c[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            c[u] = s0[u];
            int sl = slot0 + c[u].j;
            if (sl >= t.R) sl -= t.R;
            if (ONE) {  // (R = dmin: the arrival row is the spike's own)
                sl = sl * t.stride * 4 + (int)(c[u].k >> 31);
                c[u].k &= 0x7fffffffu;
                c[u].e &= 0x7fffffffu;
                if ((unsigned)(c[u].j + t.dmin - lo_rel - 1) >= span) c[u].e = c[u].k;
            }
            c[u].base = sl;
            if (!MGC_OK_INDEX(c[u].k <= c[u].e && c[u].e <= t.n_vec)) c[u].e = c[u].k;
        }
        const int n = n0;
        if (t.lanes_log2 == 0) {
            Vec v[U][D];
            auto fetch = [&]() {
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int d = 0; d < D; ++d)
                        if (c[u].k + d < c[u].e) v[u][d] = __ldg(rec + c[u].k + d);
            };
            fetch();
            if (more) {  // the next batch's offsets, and the ids after it
                offsets();
                n0 = n1;
                const bool m2 = src.begin(n1);
                ids(m2, n1);
                more = m2;
            } else {
                n0 = 0;
            }
            for (;;) {
                bool rest = false;
#pragma unroll
                for (int u = 0; u < U; ++u) {
#pragma unroll
                    for (int d = 0; d < D; ++d)
                        if (c[u].k + d < c[u].e)
                            tile_apply_vec<FX, ONE>(a, t, m, v[u][d], c[u].base, c[u].j, lo_rel, span, ev);
                    c[u].k += D;
                    rest |= c[u].k < c[u].e;
                }
                if (!rest) break;
                fetch();
            }
        } else {
            const int G = 1 << t.lanes_log2, round = 32 >> t.lanes_log2;
            const int gl = lane & (G - 1), gq = lane >> t.lanes_log2;
            if (more) {
                offsets();
                n0 = n1;
                const bool m2 = src.begin(n1);
                ids(m2, n1);
                more = m2;
            } else {
                n0 = 0;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                for (int q0 = 0; q0 < 32 && u * 32 + q0 < n; q0 += round) {
                    const int q = q0 + gq;
                    uint32_t k = __shfl_sync(0xffffffffu, c[u].k, q) + gl;
                    const uint32_t e = __shfl_sync(0xffffffffu, c[u].e, q);
                    const int base = __shfl_sync(0xffffffffu, c[u].base, q);
                    const int j = ONE ? 0 : __shfl_sync(0xffffffffu, c[u].j, q);
                    while (k < e) {
                        Vec v[D];
#pragma unroll
                        for (int d = 0; d < D; ++d)
                            if (k + d * G < e) v[d] = __ldg(rec + k + d * G);
#pragma unroll
                        for (int d = 0; d < D; ++d)
                            if (k + d * G < e) tile_apply_vec<FX, ONE>(a, t, m, v[d], base, j, lo_rel, span, ev);
                        k += D * G;
                    }
                    __syncwarp();
                }
            }
        }
        if (!n0) break;
    }
    events += ev;
}

// 16 bytes as one access (neither half is seen without the other).
__device__ __forceinline__ void st_head(ulonglong2* p, ulonglong2 v)
{
    asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
                 "l"(v.x), "l"(v.y)
                 : "memory");
}
__device__ __forceinline__ ulonglong2 ld_head(const ulonglong2* p)
{
    ulonglong2 v;
    asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
                 : "=l"(v.x), "=l"(v.y)
                 : "l"(p)
                 : "memory");
    return v;
}

// The tile's header of window k (c spikes, the first in `first`) into every
// tile's mailbox.  Called by the whole block after a block barrier.
__device__ __forceinline__ void tile_publish(const TileArgs& t, int k, int c, const uint32_t* first, bool fence)
{
    if ((int)threadIdx.x < t.T) {
        ulonglong2 h;
        h.x = ((unsigned long long)(t.epoch + (uint32_t)k) << 32) | (uint32_t)c;
        h.y = (unsigned long long)first[0] | ((unsigned long long)first[1] << 32);
        if (fence || c > kTileInline) asm volatile("fence.acq_rel.gpu;" ::: "memory");
        st_head(t.mail + ((size_t)(k & 1) * t.T + threadIdx.x) * t.T + blockIdx.x, h);
    }
}

// Waits until every tile has published window k.  *n (zero on entry) gets the
// window's spikes, m.cnt the tiles' counts; when the spikes fit, they are all
// in m.spikes.  False on a time-out.
__device__ __forceinline__ bool tile_gather(const StepArgs& a, const TileArgs& t, const TileSmem& m, int k,
                                            const uint32_t* lists, size_t list_len, int* n, int* abort_flag)
{
    bool listed = false;  // the tile has more spikes than its header carries
    if ((int)threadIdx.x < t.T) {
        const ulonglong2* p = t.mail + ((size_t)(k & 1) * t.T + blockIdx.x) * t.T + threadIdx.x;
        ulonglong2 v = ld_head(p);
        for (unsigned it = 0; (uint32_t)(v.x >> 32) != t.epoch + (uint32_t)k; v = ld_head(p)) {
            if (++it > kBarrierSpins) {
                atomicOr(a.status, kStatusBarrier);
                *abort_flag = 1;
                v.x = 0;
                break;
            }
            if (it > 64) __nanosleep(32);
        }
        const int c = (int)(uint32_t)v.x;
        int at = 0;
        if (c > 0) {
            at = atomicAdd(n, c);
            listed = c > kTileInline;
            if (listed) asm volatile("fence.acq_rel.gpu;" ::: "memory");
            if (at + c <= kTileSpikes) {
                m.spikes[at] = (uint32_t)v.y;
                if (c > 1) m.spikes[at + 1] = (uint32_t)(v.y >> 32);
            }
        }
        m.cnt[threadIdx.x] = c;
        m.at[threadIdx.x] = at;
    }
    const bool any = __syncthreads_or(listed);
    if (any && *n <= kTileSpikes) {  // eight lanes a tile
        for (int l = threadIdx.x >> 3; l < t.T; l += blockDim.x >> 3) {
            const int c = m.cnt[l];
            const uint32_t* from = lists + (size_t)l * list_len;
            for (int q = kTileInline + (threadIdx.x & 7); q < c; q += 8) m.spikes[m.at[l] + q] = __ldcg(from + q);
        }
        __syncthreads();
    }
    return *abort_flag == 0;
}

template <bool CUR, bool FX, bool ONE>
__global__ void __launch_bounds__(kTileThreads, 1) k_tile(StepArgs a, TileArgs t, int32_t nsteps)
{
    extern __shared__ __align__(16) unsigned char tile_raw[];
    __shared__ int abort_flag;
    __shared__ unsigned long long blk_ev;
    __shared__ int count, npg, total;  // the tile's spikes of the window, its POISSON groups, all tiles' spikes
    __shared__ uint32_t mine[kTileInline];
    __shared__ int scnt[kTileWindow];      // this window's spikes per step
    __shared__ int32_t sbase[2][kTileWindow], stot[kTileWindow + 1];  // places reserved in the steps, the steps' totals
    const TileSmem m = tile_smem<CUR, FX>(tile_raw, t);
    const int tile = blockIdx.x, tid = threadIdx.x;
    const int64_t s0 = *a.step;
    const int32_t slot0 = a.slots[0], h0 = a.slots[1];
    const bool rec = a.record != 0;
    int64_t rbase = rec ? *a.raster_pos : 0;
    const int64_t rstep0 = *a.raster_step0;
    const int64_t s_end = s0 + nsteps;
    // arrivals this launch delivers and counts: (lo, hi]
    const int64_t lo = t.ahead ? s0 : s0 - 1, hi = t.ahead ? s_end : s_end - 1;
    auto hs_of = [&](int64_t x) {  // history slot of a step within H of s0, or later
        int64_t h = (h0 + (x - s0)) % a.H;
        return (int32_t)(h < 0 ? h + a.H : h);
    };
    unsigned long long ev = 0;

    // state of the tile, empty ring
    {
        uint32_t* z = reinterpret_cast<uint32_t*>(m.ring);
        const int words = (FX ? 4 : 1) * t.R * t.stride;
        for (int k = tid; k < words; k += blockDim.x) z[k] = 0;
        for (int i = tid; i < t.nl; i += blockDim.x) {
            const int32_t gi = tile_neuron(t, i, tile);
            const bool in = gi < a.ns;
            m.type[i] = in ? a.type[gi] : (int8_t)kRAW;
            m.V[i] = in ? a.V[gi] : 0.f;
            m.rf[i] = in ? a.refrac[gi] : 0;
            if (!FX) {
                m.we[i] = in ? t.we[gi] : 0.f;
                m.wi[i] = in ? t.wi[gi] : 0.f;
            }
            if (CUR) {
                m.ie[i] = in ? a.Iexc[gi] : 0.f;
                m.ii[i] = in ? a.Iinh[gi] : 0.f;
            }
        }
        if (!FX && m.tab)
            for (int k = tid; k < 2 * kTileTable; k += blockDim.x) m.tab[k] = t.chain[k];
        if (tid < kTileWindow) scnt[tid] = 0;
        if (tid == 0) {
            abort_flag = 0;
            blk_ev = 0;
            count = npg = total = 0;
        }
    }
    __syncthreads();
    for (int g = tid; g < t.nl / 4; g += blockDim.x) {
        bool p = false;
        for (int q = 0; q < 4; ++q) p |= m.type[4 * g + q] == kPOISSON;
        if (p) m.pg[atomicAdd(&npg, 1)] = (uint16_t)g;
    }
    __syncthreads();
    const int n_pg = npg;
    // prologue: the spikes of the last R steps before s0 that arrive later
    {
        const int64_t x0 = s0 - t.R > 0 ? s0 - t.R : 0;
        const int nst = (int)(s0 - x0);
        for (int j = tid; j < nst; j += blockDim.x) m.cnt[j] = __ldcg(a.hist_cnt + hs_of(x0 + j));
        __syncthreads();
        auto get = [&](int l, int q, int& j) {
            j = l;
            return __ldcg(a.hist_ids + (size_t)hs_of(x0 + l) * (size_t)a.n_src + q);
        };
        tile_deliver<FX, ONE>(a, t, m, x0, (int)(x0 % t.R), lo, hi, TileListed<decltype(get)>(get, m.cnt, nst), ev);
        if (ONE)  // whole rows, counted by one block a step
            for (int j = tile; j < nst; j += t.T) {
                const int64_t x = x0 + j;
                if (x + t.dmin <= lo || x + t.dmin > hi) continue;
                for (int q = tid; q < m.cnt[j]; q += blockDim.x) {
                    const int32_t id = __ldcg(a.hist_ids + (size_t)hs_of(x) * (size_t)a.n_src + q);
                    if (MGC_OK_INDEX(id >= 0 && id < a.n_src))
                        ev += (unsigned long long)(a.row_ptr[id + 1] - a.row_ptr[id]);
                }
            }
        __syncthreads();
    }
    // the spikes of window k (w steps from x0): their raster places, and the
    // history of the launch's last steps; the counters of the window are final
    const size_t list_len = (size_t)t.nl * t.W;
    auto my_list = [&](int k) { return t.list + ((size_t)(k & 1) * t.T + tile) * list_len; };
    auto record = [&](int k, int64_t x0, int w, int c) {  // stot, sbase ready; c: this tile's spikes
        for (int q = tid; q < c; q += blockDim.x) {
            const uint32_t e = my_list(k)[q];
            const int32_t id = (int32_t)(e & kTileId);
            const int j = (int)(e >> kTileStepShift);
            const int at = atomicAdd(&sbase[k & 1][j], 1);  // any order inside a step
            const int64_t x = x0 + j, rb = rbase + stot[j] + at;
            if (rec && rb < a.raster_ids_cap) a.raster_ids[rb] = id;
            if (x > s_end - a.H && MGC_OK_INDEX(at < a.n_src)) a.hist_ids[(size_t)hs_of(x) * (size_t)a.n_src + at] = id;
            if (ONE && x + t.dmin <= hi) ev += (unsigned long long)(a.row_ptr[id + 1] - a.row_ptr[id]);
        }
        if (tile == 0 && tid < w) {
            const int64_t x = x0 + tid;
            const int c_all = stot[tid + 1] - stot[tid];
            if (x > s_end - a.H) a.hist_cnt[hs_of(x)] = c_all;
            if (rec) {
                if (x - rstep0 < a.raster_steps_cap)
                    a.raster_counts[x - rstep0] = c_all;
                else
                    atomicOr(a.status, kStatusRasterSteps);
                if (rbase + stot[tid + 1] > a.raster_ids_cap) atomicOr(a.status, kStatusRasterIds);
            }
        }
        rbase += stot[w];
    };
    // running sums of window k's step totals, by the first warp
    auto totals = [&](int k, int w) {
        if (tid < 32) {
            int c = tid < w ? __ldcg(t.cnt + (k & 3) * kTileWindow + tid) : 0;
#pragma unroll
            for (int o = 1; o < kTileWindow; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, c, o);
                if (tid >= o) c += v;
            }
            if (tid < w) stot[tid + 1] = c;
            if (tid == 0) stot[0] = 0;
        }
    };
    int slot = (int)(s0 % t.R);
    int k = 0, c_prev = 0, w_prev = 0;  // the window before: this tile's spikes, steps
    int64_t w0 = s0;
    for (; w0 < s_end; ++k) {
        const int wl = (int)(s_end - w0 < t.W ? s_end - w0 : t.W);
        if (n_pg) tile_poisson(a, t, m, w0, wl, n_pg, my_list(k), mine, &count, scnt);
        tile_update<CUR, FX>(a, t, m, w0, wl, slot, t.ahead && k == 0, my_list(k), mine, &count, scnt);
        if (tile == 0 && tid < kTileWindow) t.cnt[((k + 1) & 3) * kTileWindow + tid] = 0;
        __syncthreads();
        const int c_now = count;
        tile_publish(t, k, c_now, mine, tile == 0);  // (tile 0 cleared counters)
        // the steps' places for this tile's spikes, needed a window later
        int place = 0;
        if (tid >= 32 && tid < 32 + wl && scnt[tid - 32])
            place = atomicAdd(t.cnt + (k & 3) * kTileWindow + tid - 32, scnt[tid - 32]);
        const uint32_t* lists = t.list + (size_t)(k & 1) * t.T * list_len;
        if (!tile_gather(a, t, m, k, lists, list_len, &total, &abort_flag)) return;
        if (tid >= 32 && tid < 32 + kTileWindow) {
            sbase[k & 1][tid - 32] = place;
            scnt[tid - 32] = 0;
        }
        if (tid == 0) count = 0;
        if (k > 0) totals(k - 1, w_prev);
        if (total <= kTileSpikes) {
            tile_deliver<FX, ONE>(a, t, m, w0, slot, lo, hi, TileGathered(m.spikes, total), ev);
        } else {
            auto get = [&](int l, int q, int& j) {
                const uint32_t e = __ldcg(lists + (size_t)l * list_len + q);
                j = (int)(e >> kTileStepShift);
                return (int32_t)(e & kTileId);
            };
            tile_deliver<FX, ONE>(a, t, m, w0, slot, lo, hi, TileListed<decltype(get)>(get, m.cnt, t.T), ev);
        }
        __syncthreads();
        if (tid == 0) total = 0;
        if (k > 0) record(k - 1, w0 - w_prev, w_prev, c_prev);
        c_prev = c_now;
        w_prev = wl;
        w0 += wl;
        slot += wl;
        if (slot >= t.R) slot -= t.R;
    }
    // the last window's raster and history: an empty window makes its counters final
    tile_publish(t, k, 0, mine, true);
    if (!tile_gather(a, t, m, k, t.list, 0, &total, &abort_flag)) return;
    totals(k - 1, w_prev);
    __syncthreads();
    record(k - 1, w0 - w_prev, w_prev, c_prev);
    // back to the single-step form: the state, and the arrivals of s_end
    for (int i = tid; i < t.nl; i += blockDim.x) {
        const int32_t gi = tile_neuron(t, i, tile);
        if (gi >= a.ns) continue;
        if (m.type[i] == kPOISSON) continue;  // keeps its probability, ignores its input
        a.V[gi] = m.V[i];
        a.refrac[gi] = m.rf[i];
        if (CUR) {
            a.Iexc[gi] = m.ie[i];
            a.Iinh[gi] = m.ii[i];
        }
        if (t.ahead) {
            const size_t at = (size_t)slot * t.stride + i;
            if (FX) {
                const unsigned long long* e = reinterpret_cast<const unsigned long long*>(m.ring);
                acc_buf<FX>(a, a.acc_e, s_end)[gi] = (typename AccT<FX>::type)e[at];
                acc_buf<FX>(a, a.acc_i, s_end)[gi] = (typename AccT<FX>::type)e[(size_t)t.R * t.stride + at];
            } else {
                const uint32_t c = reinterpret_cast<const uint32_t*>(m.ring)[at];
                acc_buf<FX>(a, a.acc_e, s_end)[gi] = (typename AccT<FX>::type)chain_sum(c & 0xffffu, m.we[i], m.tab);
                acc_buf<FX>(a, a.acc_i, s_end)[gi] =
                    (typename AccT<FX>::type)chain_sum(c >> 16, m.wi[i], m.tab ? m.tab + kTileTable : nullptr);
            }
        }
    }
    if (ev) atomicAdd(&blk_ev, ev);
    __syncthreads();
    if (tid == 0 && blk_ev) atomicAdd(a.events, blk_ev);
    // the clock, by the last block to finish
    if (last_block(a.done) && tid == 0) {
        if (rec) *a.raster_pos = rbase;
        if (a.ev_mark) *a.ev_mark = *(volatile unsigned long long*)a.events;
        a.hist_cnt[hs_of(s_end)] = 0;
        for (int j = 0; j < 4 * kTileWindow; ++j) t.cnt[j] = 0;
        *a.done = 0;
        a.slots[0] = (int32_t)((slot0 + nsteps) % a.M);
        a.slots[1] = hs_of(s_end);
        *a.step = s_end;
    }
}

// ---------------------------------------------------------------------------
// The same for the ring method with STDP (fixed-point sums): one step per
// window, since a step's pushes read the weights that the spikes of the step
// before changed.  A tile owns the synapses onto its neurons, so both sides of
// STDP are its own work: its records of a spiking source are pushed and
// depressed, the plastic records onto a spiking neuron of its own are
// potentiated (those whose source spiked too belong to the first, as in
// k_push_stdp), and no weight has two writers.  last_fired of the whole network
// and the step's spikes as a bitmap are kept in shared memory by every block,
// from the spike ids that the exchange brings.  A weight is written to its record
// and to the CSR, which stays current for readers and the other step forms
// (records are refreshed from it after those ran).  The launch takes over
// the global ring's pending input and hands it back.
//
// Bound by the step's chain of dependent accesses: exchange, segment
// offsets, records, and after a spike of its own the incoming list and its
// weights.  784 -> 1,600 plastic network, 1.9e4 events a step: see DESIGN.
// ---------------------------------------------------------------------------
struct TileStdpSmem {
    int32_t* lf;       // [n] last spike of every neuron
    uint32_t* fired;   // [n/32] this step's spikes
    uint32_t* in_off;  // [nl + 1] this tile's part of t.in_off
};

__host__ __device__ inline size_t tile_stdp_bytes(int nl, int R, int T, bool cur, int n)
{
    const size_t base = (tile_smem_bytes(nl, R, T, true, cur, false) + 15) / 16 * 16;
    return base + 4 * ((size_t)n + (n + 31) / 32 + nl + 1);
}

template <bool CUR>
__global__ void __launch_bounds__(kTileThreads, 1) k_tile_stdp(StepArgs a, TileArgs t, int32_t nsteps)
{
    extern __shared__ __align__(16) unsigned char tile_raw[];
    __shared__ int abort_flag;
    __shared__ unsigned long long blk_ev;
    __shared__ int count, npg, total;
    __shared__ uint32_t mine[kTileInline];
    __shared__ int scnt[kTileWindow];
    __shared__ int32_t sbase[2], stot;   // places reserved in a step, a step's spikes
    const TileSmem m = tile_smem<CUR, true>(tile_raw, t);
    TileStdpSmem q;
    {
        unsigned char* p = tile_raw + (tile_smem_bytes(t.nl, t.R, t.T, true, CUR, false) + 15) / 16 * 16;
        q.lf = reinterpret_cast<int32_t*>(p);
        q.fired = reinterpret_cast<uint32_t*>(q.lf + a.n);
        q.in_off = q.fired + (a.n + 31) / 32;
    }
    const int tile = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const int64_t s0 = *a.step;
    const int32_t slot0 = a.slots[0];
    const bool rec_on = a.record != 0;
    int64_t rbase = rec_on ? *a.raster_pos : 0;
    const int64_t rstep0 = *a.raster_step0;
    const int64_t s_end = s0 + nsteps;
    unsigned long long ev = 0;
    uint2* rec = reinterpret_cast<uint2*>(const_cast<void*>(t.rec));
    unsigned long long* ring = reinterpret_cast<unsigned long long*>(m.ring);
    const int plane = t.R * t.stride;
    unsigned long long* gring[2] = {reinterpret_cast<unsigned long long*>(a.ring_e),
                                    reinterpret_cast<unsigned long long*>(a.ring_i)};

    // state of the tile, the pending input of steps s0 .. s0 + R - 1
    for (int i = tid; i < t.nl; i += blockDim.x) {
        const int32_t gi = tile_neuron(t, i, tile);
        const bool in = gi < a.ns;
        m.type[i] = in ? a.type[gi] : (int8_t)kRAW;
        m.V[i] = in ? a.V[gi] : 0.f;
        m.rf[i] = in ? a.refrac[gi] : 0;
        if (CUR) {
            m.ie[i] = in ? a.Iexc[gi] : 0.f;
            m.ii[i] = in ? a.Iinh[gi] : 0.f;
        }
        for (int x = 0; x < t.R; ++x) {
            const int row = (int)((s0 + x) % t.R);
            const size_t from = (size_t)((slot0 + x) % a.M) * (size_t)a.ns + gi;
            for (int h = 0; h < 2; ++h) ring[h * plane + row * t.stride + i] = in ? gring[h][from] : 0ull;
        }
    }
    for (int i = tid; i < a.n; i += blockDim.x) q.lf[i] = a.last_fired[i];
    for (int i = tid; i < (a.n + 31) / 32; i += blockDim.x) q.fired[i] = 0;
    for (int i = tid; i <= t.nl; i += blockDim.x) q.in_off[i] = t.in_off[(size_t)tile * t.nl + i];
    if (tid < kTileWindow) scnt[tid] = 0;
    if (tid == 0) {
        abort_flag = 0;
        blk_ev = 0;
        count = npg = total = 0;
    }
    __syncthreads();
    for (int g = tid; g < t.nl / 4; g += blockDim.x) {
        bool p = false;
        for (int x = 0; x < 4; ++x) p |= m.type[4 * g + x] == kPOISSON;
        if (p) m.pg[atomicAdd(&npg, 1)] = (uint16_t)g;
    }
    __syncthreads();
    const int n_pg = npg;
    const size_t list_len = (size_t)t.nl * t.W;
    auto my_list = [&](int k) { return t.list + ((size_t)(k & 1) * t.T + tile) * list_len; };
    // f(id) for every spike of the step, the block's threads (or groups of
    // `width` of them) in turn
    auto each_spike = [&](int k, int group, int groups, auto f) {
        if (total <= kTileSpikes) {
            for (int x = group; x < total; x += groups) f((int32_t)(m.spikes[x] & kTileId));
        } else {
            const uint32_t* lists = t.list + (size_t)(k & 1) * t.T * list_len;
            for (int l = 0; l < t.T; ++l)
                for (int x = group; x < m.cnt[l]; x += groups) f((int32_t)(__ldcg(lists + (size_t)l * list_len + x) & kTileId));
        }
    };
    // raster places of step x's spikes (the step's counter is final), one step late
    auto record = [&](int k, int64_t x, int c) {
        for (int y = tid; y < c; y += blockDim.x) {
            const int32_t id = (int32_t)(my_list(k)[y] & kTileId);
            const int64_t rb = rbase + atomicAdd(&sbase[k & 1], 1);  // any order inside a step
            if (rec_on && rb < a.raster_ids_cap) a.raster_ids[rb] = id;
            ev += (unsigned long long)(a.row_ptr[id + 1] - a.row_ptr[id]);
        }
        if (tile == 0 && tid == 0 && rec_on) {
            if (x - rstep0 < a.raster_steps_cap)
                a.raster_counts[x - rstep0] = stot;
            else
                atomicOr(a.status, kStatusRasterSteps);
            if (rbase + stot > a.raster_ids_cap) atomicOr(a.status, kStatusRasterIds);
        }
        rbase += stot;
    };
    int slot = (int)(s0 % t.R);
    int k = 0, c_prev = 0;
    for (int64_t s = s0; s < s_end; ++s, ++k) {
        if (n_pg) tile_poisson(a, t, m, s, 1, n_pg, my_list(k), mine, &count, scnt);
        tile_update<CUR, true>(a, t, m, s, 1, slot, false, my_list(k), mine, &count, scnt);
        if (tile == 0 && tid == 0) t.cnt[((k + 1) & 3) * kTileWindow] = 0;
        __syncthreads();
        const int c_now = count;
        tile_publish(t, k, c_now, mine, tile == 0);  // (tile 0 cleared a counter)
        int place = 0;
        if (tid == 32 && c_now) place = atomicAdd(t.cnt + (k & 3) * kTileWindow, c_now);
        if (!tile_gather(a, t, m, k, t.list + (size_t)(k & 1) * t.T * list_len, list_len, &total, &abort_flag)) return;
        if (tid == 32) {
            sbase[k & 1] = place;
            scnt[0] = 0;
        }
        if (tid == 0) {
            count = 0;
            if (k > 0) stot = __ldcg(t.cnt + ((k - 1) & 3) * kTileWindow);
        }
        each_spike(k, tid, blockDim.x, [&](int32_t id) {
            if (!MGC_OK_INDEX(id >= 0 && id < a.n)) return;
            q.lf[id] = (int32_t)s;
            atomicOr(q.fired + (id >> 5), 1u << (id & 31));
        });
        __syncthreads();
        // this tile's synapses of the spiking sources, eight lanes a source
        each_spike(k, tid >> 3, blockDim.x >> 3, [&](int32_t id) {
            if (!MGC_OK_INDEX(id >= 0 && id < a.n)) return;
            const uint32_t* o = t.off + (size_t)id * t.T + tile;
            const uint32_t b = __ldg(o), e = __ldg(o + 1);
            if (!MGC_OK_INDEX(b <= e && e <= t.n_vec)) return;
            for (uint32_t r0 = b + (lane & 7); r0 < e; r0 += 32) {
                uint2 x[4];
                uint32_t cp[4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (r0 + 8 * u < e) {
                        x[u] = __ldcg(rec + r0 + 8 * u);
                        cp[u] = __ldg(t.cpos + r0 + 8 * u);
                    }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (r0 + 8 * u >= e) continue;
                    const int local = (int)(x[u].x & 0xffffu), d = (int)((x[u].x >> 16) & 0x7fffu);
                    int row = slot + d;
                    if (row >= t.R) row -= t.R;
                    if (!MGC_OK_INDEX(local < t.nl && row < t.R && cp[u] < (uint64_t)a.n_syn)) continue;
                    const float w = as_f(x[u].y);
                    atomicAdd(ring + (w > 0.0f ? 0 : plane) + row * t.stride + local,
                              (unsigned long long)to_fx(w, a.fx_scale));
                    if (x[u].x >> 31) {
                        const uint32_t nw = as_u(stdp_weight((int32_t)s - q.lf[tile_neuron(t, local, tile)], w, a.P));
                        rec[r0 + 8 * u].y = nw;
                        a.syn[cp[u]].y = nw;
                    }
                }
            }
        });
        // the plastic synapses onto this tile's spiking neurons, the block on each
        for (int y = 0; y < c_now; ++y) {
            const int32_t id = (int32_t)((y < kTileInline ? mine[y] : __ldcg(my_list(k) + y)) & kTileId);
            const int g = id >> 2, local = g / t.T * 4 + (id & 3);
            const uint32_t e = q.in_off[local + 1];
            for (uint32_t p0 = q.in_off[local] + tid; p0 < e; p0 += 2 * blockDim.x) {
                uint2 en[2];
                uint32_t w[2], cp[2];
                bool go[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    go[u] = p0 + u * blockDim.x < e;
                    if (go[u]) en[u] = __ldg(t.in_ent + p0 + u * blockDim.x);
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    go[u] = go[u] && MGC_OK_INDEX(en[u].x < (uint32_t)a.n && en[u].y < t.n_vec) &&
                            !bit_of(q.fired, (int32_t)en[u].x);
                    if (go[u]) {
                        w[u] = __ldcg(&rec[en[u].y].y);
                        cp[u] = __ldg(t.cpos + en[u].y);
                    }
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (!go[u]) continue;
                    const uint32_t nw = as_u(stdp_weight(q.lf[en[u].x] - (int32_t)s, as_f(w[u]), a.P));
                    rec[en[u].y].y = nw;
                    a.syn[cp[u]].y = nw;
                }
            }
        }
        __syncthreads();
        each_spike(k, tid, blockDim.x, [&](int32_t id) { q.fired[id >> 5] = 0; });
        if (k > 0) record(k - 1, s - 1, c_prev);
        c_prev = c_now;
        slot = slot + 1 == t.R ? 0 : slot + 1;
        __syncthreads();
        if (tid == 0) total = 0;
    }
    // the last step's raster: an empty window makes its counter final
    __syncthreads();
    tile_publish(t, k, 0, mine, true);
    if (!tile_gather(a, t, m, k, t.list, 0, &total, &abort_flag)) return;
    if (tid == 0) stot = __ldcg(t.cnt + ((k - 1) & 3) * kTileWindow);
    __syncthreads();
    record(k - 1, s_end - 1, c_prev);
    for (int i = tid; i < t.nl; i += blockDim.x) {
        const int32_t gi = tile_neuron(t, i, tile);
        if (gi >= a.ns) continue;
        const int32_t slot_end = (int32_t)((slot0 + nsteps) % a.M);
        const bool pois = m.type[i] == kPOISSON;
        for (int x = 0; x < a.M; ++x) {
            const int row = (int)((s_end + x) % t.R);
            const size_t to = (size_t)((slot_end + x) % a.M) * (size_t)a.ns + gi;
            for (int h = 0; h < 2; ++h)  // (a POISSON neuron's input is read by nobody)
                gring[h][to] = x < t.R && !pois ? ring[h * plane + row * t.stride + i] : 0ull;
        }
        if (pois) continue;
        a.V[gi] = m.V[i];
        a.refrac[gi] = m.rf[i];
        if (CUR) {
            a.Iexc[gi] = m.ie[i];
            a.Iinh[gi] = m.ii[i];
        }
    }
    if (ev) atomicAdd(&blk_ev, ev);
    __syncthreads();
    if (tid == 0 && blk_ev) atomicAdd(a.events, blk_ev);
    if (last_block(a.done) && tid == 0) {
        if (rec_on) *a.raster_pos = rbase;
        for (int j = 0; j < 4 * kTileWindow; ++j) t.cnt[j] = 0;
        *a.done = 0;
        a.slots[0] = (int32_t)((slot0 + nsteps) % a.M);
        *a.step = s_end;
    }
}

}  // namespace mgc
