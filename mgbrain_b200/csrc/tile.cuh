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
// ends in the state of the single-step kernels: the last windows' spikes are
// written into the history, and the arrivals of the step after the last go into
// the accumulators.  The later ones are kept as they stand in the ring (`pend`,
// valid for a launch that starts at that step: `pend_step`).  A launch after
// steps of another form delivers the history's spikes that arrive after its first
// step (whose arrivals the accumulators hold) once more, which every call paid at
// first: 12,000 neurons, 9.8e6 synapses of 10 to 50 steps, 2,460 spikes a step, in
// calls of one step: 298 us a call, 45 with the kept ring.  With a minimum
// delay of one step the single-step kernels start a step without its arrivals;
// there the ring includes them and the accumulators stay empty.
//
// Events are counted by the spike's own tile, from the CSR's (source, delay)
// offsets: those of a launch's steps, whichever launch delivered them.
//
// Exchange of window k: a tile sends every tile its spikes (id, step in the
// window) in 16-byte chunks, one store each, into that tile's mailbox: {epoch of
// the window and count, first two spikes}, then {epoch, three spikes}.  Every
// chunk carries the epoch, so none has to be ordered after another, and no
// fence is needed; thread l of a block polls the place of tile l in its own
// mailbox, which no other block reads, so no counter or line is shared.  Only a
// tile with more spikes than a mailbox holds sends just the count; they are in
// its list of buffer k % kTileLists, with a fence before and at its readers.
// (11,000 neurons: 5.0 us an exchange with one set of headers polled by all
// blocks and release stores, 2.1 with mailboxes; 44,700 neurons, 13 spikes a
// tile and window: 8.0 us with two spikes a header and fenced lists.)  A tile
// overwrites a mailbox place two windows later, when every tile has published
// the window between, which it does after reading the place.  A list is read a
// second time, by its own tile's raster writes at the end of the window after
// its own; no block barrier lies between those and the next window's updates,
// which write the list of two windows on.  So there are three list buffers, not
// two: the buffer of window k is written again in window k + 3, behind the
// barriers of window k + 2.  Waits are bounded (kStatusBarrier).
//
// Raster: a step's place in it needs the step's spikes of all tiles, so each
// tile adds its counts to the window's 16 step counters when it publishes,
// and writes its spikes' places one window later, when every tile's counts
// are in: hardly ever waited for.  The counters (slot k % 4) run on over the
// windows of a launch; every block keeps their last totals.  Nothing orders a
// tile's additions before its next mailbox stores (both are relaxed), so a
// reader reads the counters until the steps add up to the window's spikes, which
// the mailboxes have told it; the first time while it waits for the next
// window's mailboxes.
//
// Measured per step, the faster of the other step groups and this one: 4,000
// neurons, minimum delay 1: 6.5 and 3.2 us; 11,000 neurons, windows of 15 steps
// quiet: 5.0 and 0.31, with volleys: 8.7 and 1.36; balanced networks of 1e8
// synapses, quiet: 6.6 and 0.98, and of 3e7 at POISSON rates of 1 kHz: 20.9 and
// 4.6; 9,000 neurons with a range of delays: 7.8 and 1.1.
#pragma once
#include <type_traits>

#include "kernels.cuh"

namespace mgc {

constexpr int kTileThreads = 512;   // 128 registers a thread: no spills (768 and 1,024 threads spill and ran slower)
constexpr int kTileWindow = 16;     // longest window (a neuron's spikes of a window: 16 bits)
constexpr int kTileMaxDelay = 512;  // longest delay (the prologue's prefix, shared memory)
constexpr int kTileTable = 512;     // entries of each chain table

struct TileArgs {
    int32_t T;            // tiles = blocks
    int32_t nl;           // neurons per tile (a multiple of 4)
    int32_t stride;       // entries of a ring row: nl, one for fillers, an empty one, padding
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
    uint32_t* list;       // [kTileLists][T][nl*W] spikes of a window: id | step in the window << 28
    ulonglong2* mail;     // [2][T reader][T][kTileChunks]
    uint32_t epoch;       // epoch of the launch's first window (they count on over the launches; never 0,
                          //   which the mailboxes hold at first, and never past 2^32 - 1: launch_tiles)
    int32_t* cnt;         // [4][kTileWindow] counters (tile_counter) of a window's steps' spikes; zero between launches
    void* pend;           // [T] rings as the last launch left them (of the steps after its end),
    int64_t* pend_step;   //   and the step they continue at (-1: none)
    // plastic networks (k_tile_stdp): rec holds single records (off counts them)
    const uint32_t* cpos;   // [S] CSR position of a record
    const uint32_t* in_off; // [T*nl + 1] plastic synapses onto each local neuron, tile after tile:
    const uint2* in_ent;    //   {source, record}
};

constexpr int kTileLine = 32;       // a counter has a line to itself: 148 blocks add to 16 of them at once, and
                                    // on one line those atomics queued for 8 to 70 us a window
constexpr int kTileChunks = 16;     // chunks of a mailbox place
constexpr int kTileInline = 2 + 3 * (kTileChunks - 1);  // spikes they carry
constexpr int kTileLists = 3;       // list buffers (see the exchange above)
constexpr int kTileSpikes = 8192;   // spikes of a window gathered in shared memory; every mailbox full fits
constexpr int kMaxTiles = kTileSpikes / kTileInline;
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

// A ring row: nl entries, the fillers' one and an empty one, a multiple of 4.
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

__device__ __forceinline__ int32_t* tile_counter(const TileArgs& t, int k, int j)
{
    return t.cnt + ((k & 3) * kTileWindow + j) * kTileLine;
}
__device__ __forceinline__ int32_t tile_count(const TileArgs& t, int k, int j)
{
    int32_t v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(tile_counter(t, k, j)) : "memory");
    return v;
}
// One more read of counters that did not add up; false: the limit is reached.
__device__ __forceinline__ bool tile_again(const StepArgs& a, unsigned& it, int* late)
{
    if (++it > kBarrierSpins) {
        atomicOr(a.status, kStatusBarrier);
        *late = 1;
        return false;
    }
    if (it > 64) __nanosleep(32);
    return true;
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
#pragma unroll 1
    for (; c; --c) v = fadd_ftz(v, w);
    return v;
}

// A neuron's spikes of a window (bit j: step w0 + j) into the tile's list.
__device__ __forceinline__ void tile_spikes(const TileArgs& t, int32_t gi, uint32_t fm, uint32_t* list,
                                            uint32_t* first, int* count, int* scnt)
{
    int pos = atomicAdd(count, __popc(fm));
#pragma unroll 1
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
#pragma unroll 1
    for (int x = blockDim.x - 1 - threadIdx.x; x < npg * wl; x += blockDim.x) {
        const int j = x / npg, g = m.pg[x - j * npg];
        const int32_t gi = tile_neuron(t, 4 * g, blockIdx.x);
        const int64_t id = (int64_t)gi + a.id_offset;
        float u[4] = {0.f, 0.f, 0.f, 0.f};
        if ((id & 3) == 0) {
            const uint64_t st = (uint64_t)(w0 + j);
            const U32x4 r = philox4x32_10((uint32_t)st, (uint32_t)(st >> 32), (uint32_t)((uint64_t)id >> 2),
                                          kTagPoisson, (uint32_t)a.seed, (uint32_t)(a.seed >> 32));
#pragma unroll
            for (int q = 0; q < 4; ++q) u[q] = unit_open0(pick(r, q));
        } else {  // ids that start inside a Philox block
#pragma unroll 1
            for (int q = 0; q < 4; ++q) {
                const float x = poisson_uniform(a.seed, id + q, w0 + j);
#pragma unroll
                for (int y = 0; y < 4; ++y) u[y] = y == q ? x : u[y];
            }
        }
        unsigned f = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q)  // (V holds the probability)
            f |= (m.type[4 * g + q] == kPOISSON && m.V[4 * g + q] > u[q] ? 1u : 0u) << q;
#pragma unroll 1
        for (; f; f &= f - 1) {
            const int32_t nrn = gi + __ffs(f) - 1;
            atomicAdd(a.fire_cnt + nrn, 1);
            atomicMax(a.last_fired + nrn, (int32_t)(w0 + j));  // another thread has the group's other steps
            tile_spikes(t, nrn, 1u << j, list, first, count, scnt);
        }
    }
}

// Inputs of the steps whose ring words are at[0..N), which are cleared.
template <bool FX, int N>
__device__ __forceinline__ void tile_inputs(const StepArgs& a, const TileArgs& t, const TileSmem& m, const int* at,
                                            float we, float wi, float* re, float* ri)
{
    if (FX) {
        const int plane = t.R * t.stride;  // the inh sums follow the exc ones
        long long* ring = reinterpret_cast<long long*>(m.ring);
        long long fe[N], fi[N];
#pragma unroll
        for (int k = 0; k < N; ++k) {
            fe[k] = ring[at[k]];
            fi[k] = ring[plane + at[k]];
            ring[at[k]] = 0;
            ring[plane + at[k]] = 0;
        }
#pragma unroll
        for (int k = 0; k < N; ++k) {
            re[k] = from_fx(fe[k], a.fx_unscale);
            ri[k] = from_fx(fi[k], a.fx_unscale);
        }
        return;
    }
    uint32_t* ring = reinterpret_cast<uint32_t*>(m.ring);
    constexpr uint32_t kMask = kTileTable - 1;
    uint32_t c[N], any = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        c[k] = ring[at[k]];
        ring[at[k]] = 0;
        any |= c[k];
    }
    if (m.tab && !__any_sync(0xffffffffu, (any & ~(kMask | (kMask << 16))) != 0)) {  // (tab[0] is 0)
#pragma unroll
        for (int k = 0; k < N; ++k) {
            re[k] = m.tab[c[k] & kMask];
            ri[k] = m.tab[kTileTable + (c[k] >> 16)];
        }
        return;
    }
    // counts past the tables, or no tables: all chains an addition at a time
#pragma unroll
    for (int k = 0; k < N; ++k) {
        re[k] = ri[k] = 0.0f;
        if (m.tab) {
            const uint32_t ce = min(c[k] & 0xffffu, kMask), ci = min(c[k] >> 16, kMask);
            re[k] = m.tab[ce];
            ri[k] = m.tab[kTileTable + ci];
            c[k] -= ce | (ci << 16);
        }
    }
#pragma unroll 1
    while (__any_sync(0xffffffffu, any != 0)) {
        any = 0;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            if (c[k] & 0xffffu) {
                re[k] = fadd_ftz(re[k], we);
                c[k] -= 1u;
            }
            if (c[k] >> 16) {
                ri[k] = fadd_ftz(ri[k], wi);
                c[k] -= 0x10000u;
            }
            any |= c[k];
        }
    }
}

// The tile's other neurons through the wl steps from w0 (ring slot `slot`),
// one neuron a lane, eight steps at a time.  `from_acc`: the first step's
// input is in the accumulators (the launch's first step), which are cleared.
// The spikes go into `list` (and `first`), counted in *count and per step.
// Warps without LIF or LIFE neurons take lifb_step for every lane, whatever its
// neuron, and keep the result of LIFB neurons at the end; lanes without input,
// and steps past the window, read a column of the rows that stays empty, so
// that a batch has no branches.
template <bool CUR, bool FX>
__device__ __forceinline__ void tile_update(const StepArgs& a, const TileArgs& t, const TileSmem& m, int64_t w0,
                                            int wl, int slot, bool from_acc, uint32_t* list, uint32_t* first,
                                            int* count, int* scnt)
{
    const int lane = threadIdx.x & 31;
    const int tile = blockIdx.x;
#pragma unroll 1
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
        const bool any_cur = CUR && __any_sync(0xffffffffu, type == kLIF || type == kLIFE);
        uint32_t fm = 0;
        const int empty = t.nl + 1, wrap = t.R * t.stride;
        int place = slot * t.stride + (input ? i : empty);
        auto batch = [&](auto width, int h, int n) {
            constexpr int N = decltype(width)::value;
            float re[N], ri[N];
            int at[N];
#pragma unroll
            for (int k = 0; k < N; ++k) {
                at[k] = N == 1 || k < n ? place : empty;
                place += t.stride;
                place = place >= wrap ? place - wrap : place;
            }
            tile_inputs<FX, N>(a, t, m, at, we, wi, re, ri);
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
#pragma unroll
            for (int k = 0; k < N; ++k) {
                if (N > 1 && k >= n) break;
                bool f;
                if (any_cur)
                    f = input && update_one<false>(a, type, gi, w0 + h + k, v, rf, re[k], ri[k], ie, ii, 0.f);
                else
                    f = lifb_step(a, v, rf, re[k], ri[k]);
                fm |= (f ? 1u : 0u) << (h + k);
            }
        };
        constexpr int kWide = CUR ? 4 : 8;  // (update_one is long: fewer copies of it)
        int h = 0;
#pragma unroll 1
        for (; wl - h > 1; h += kWide) {
            if (!CUR && wl - h <= 4)
                batch(std::integral_constant<int, 4>{}, h, wl - h);
            else
                batch(std::integral_constant<int, kWide>{}, h, wl - h);
        }
        if (wl - h == 1) batch(std::integral_constant<int, 1>{}, h, 1);
        if (!input || !(any_cur || type == kLIFB)) continue;
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

// One record into the ring.  base: the ring row of the spike's step (ONE: of
// its arrival step); j: the step's place in the batch.
template <bool FX, bool ONE>
__device__ __forceinline__ void tile_apply(const StepArgs& a, const TileArgs& t, const TileSmem& m, uint32_t x,
                                           uint32_t wbits, int base, int j, int lo_rel, unsigned span)
{
    if (ONE) {  // base: byte offset of the row | the sign; fillers go to the row's spare column
        if (!MGC_OK_INDEX((x >> 2) < (uint32_t)t.stride && !(x & 3u))) return;
        atomicAdd(reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(m.ring) + ((base & ~1) + x)),
                  (base & 1) ? 0x10000u : 1u);
    } else {    // a filler's delay is past every arrival
        const int d = (int)((x >> 16) & 0x7fffu);
        if ((unsigned)(j + d - lo_rel - 1) >= span) return;
        int row = base + d;
        if (row >= t.R) row -= t.R;
        if (!MGC_OK_INDEX(row < t.R && (x & 0xffffu) < (uint32_t)t.nl)) return;
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
                                               unsigned span)
{
    if constexpr (FX) {
        tile_apply<FX, ONE>(a, t, m, v.x, v.y, base, j, lo_rel, span);
        tile_apply<FX, ONE>(a, t, m, v.z, v.w, base, j, lo_rel, span);
    } else if constexpr (ONE) {
        tile_apply<FX, ONE>(a, t, m, v.x & 0xffffu, 0u, base, j, lo_rel, span);
        tile_apply<FX, ONE>(a, t, m, v.x >> 16, 0u, base, j, lo_rel, span);
        tile_apply<FX, ONE>(a, t, m, v.y & 0xffffu, 0u, base, j, lo_rel, span);
        tile_apply<FX, ONE>(a, t, m, v.y >> 16, 0u, base, j, lo_rel, span);
    } else {
        tile_apply<FX, ONE>(a, t, m, v.x, 0u, base, j, lo_rel, span);
        tile_apply<FX, ONE>(a, t, m, v.y, 0u, base, j, lo_rel, span);
    }
}

// 2, 3 and 4 segments (2, 6 and 8 vectors) a lane ran no faster on driven
// networks, and their code is longer, which every quiet window pays for.
constexpr int kTileU = 1;           // segments a lane takes in a batch
constexpr int kTileD = 4;           // 8-byte vectors of each it loads at once (half as many of 16)
constexpr int kTileBatch = 32 * kTileU;
constexpr uint32_t kTileId = (1u << kTileStepShift) - 1u;

// Tile l's list of window k, and spike q of the tile from its mailbox place.
__device__ __forceinline__ const uint32_t* tile_list(const TileArgs& t, int k, int l)
{
    return t.list + ((size_t)(k % kTileLists) * t.T + l) * ((size_t)t.nl * t.W);
}
__device__ __forceinline__ uint32_t tile_mail(const TileArgs& t, int k, int l, int q)
{
    const uint32_t* p = reinterpret_cast<const uint32_t*>(
        t.mail + (((size_t)(k & 1) * t.T + blockIdx.x) * t.T + l) * kTileChunks);
    const int g = q < 2 ? 0 : (q - 2) / 3 + 1;  // words: count, epoch, 2 spikes; then spike, epoch, 2 spikes
    const int r = q < 2 ? q + 2 : q - 2 - 3 * (g - 1);
    return __ldcg(p + 4 * g + (q < 2 ? r : (r == 0 ? 0 : r + 1)));
}

// Where a warp's batches of spikes come from: the window's spikes gathered in
// shared memory, the tiles' mailboxes and lists of a window with more, or the
// history's lists (the prologue); lists are cut into batches dealt to the
// block's warps in turn.  One struct for the three, so that the delivery is
// in the code once (the kernel's loop is run through once a window, and
// instruction fetches are a good part of a quiet window).
struct TileSource {
    enum { kGathered, kTiles, kHistory };
    int kind, k;              // k: the window
    int total, per, next;     // gathered
    int lists, l, q, skip;    // lists: m.cnt holds their lengths
    int at;                   // the batch's first spike
    const uint32_t* from;     // its list (null: the mailbox)
    int32_t h0;               // history slot of the first list

    __device__ __forceinline__ void gathered(int n)
    {
        kind = kGathered;
        total = n;
        const int nw = blockDim.x >> 5, need = (n + nw - 1) / nw;
        per = need < kTileBatch ? (need > 0 ? need : 1) : kTileBatch;
        next = (threadIdx.x >> 5) * per;
    }
    __device__ __forceinline__ void listed(int kind_, int n, int k_or_slot)
    {
        kind = kind_;
        k = h0 = k_or_slot;
        lists = n;
        l = q = 0;
        skip = threadIdx.x >> 5;
    }
    // begins the warp's next batch of n <= kTileBatch spikes; false: none left
    __device__ __forceinline__ bool begin(const StepArgs& a, const TileArgs& t, const TileSmem& m, int& n)
    {
        if (kind == kGathered) {
            at = next;
            n = min(per, total - at);
            next += (blockDim.x >> 5) * per;
            return n > 0;
        }
        q += skip;
        skip = blockDim.x >> 5;
        int b = 0;
#pragma unroll 1
        for (; l < lists; ++l, q -= b) {
            b = (m.cnt[l] + kTileBatch - 1) / kTileBatch;
            if (q < b) break;
        }
        if (l >= lists) return false;
        at = q * kTileBatch;
        n = min(kTileBatch, m.cnt[l] - at);
        if (kind == kHistory) {
            const int h = h0 + l;
            from = reinterpret_cast<const uint32_t*>(a.hist_ids) + (size_t)(h >= a.H ? h - a.H : h) * (size_t)a.n_src;
        } else {
            from = m.cnt[l] > kTileInline ? tile_list(t, k, l) : nullptr;
        }
        return true;
    }
    // spike i of the batch, j steps after the first
    __device__ __forceinline__ int32_t load(const TileArgs& t, const TileSmem& m, int i, int& j) const
    {
        uint32_t e;
        if (kind == kGathered)
            e = m.spikes[at + i];
        else if (from)
            e = __ldcg(from + at + i);
        else
            e = tile_mail(t, k, l, at + i);
        j = kind == kHistory ? l : (int)(e >> kTileStepShift);
        return (int32_t)(kind == kHistory ? e : e & kTileId);
    }
};

// Delivers spikes of the steps x0, x0+1, ... to this tile's targets: the
// records whose arrival step is after lo.  slot0: the ring slot of x0.
// A warp's batches run as a pipeline of three dependent loads: the spike ids
// of the batch after next, the segment offsets of the next and the records
// of this one are in flight together, and a lane loads kTileD vectors of each
// of its segments at once, so that a batch waits for about one round trip to
// L2 (walking a segment one vector at a time, with no batch ahead, took 7.6 us
// a batch).  Long segments are cut for 1 << lanes_log2 lanes.
template <bool FX, bool ONE>
__device__ __forceinline__ void tile_deliver(const StepArgs& a, const TileArgs& t, const TileSmem& m, int64_t x0,
                                             int slot0, int64_t lo, TileSource src)
{
    using Vec = typename TileVec<FX>::type;
    constexpr int U = kTileU, D = FX ? kTileD / 2 : kTileD;
    const Vec* rec = reinterpret_cast<const Vec*>(t.rec);
    const int lane = threadIdx.x & 31;
    const int lg = t.lanes_log2;
    // the arrivals that count, relative to x0, as one unsigned comparison
    const int64_t lr = lo - x0;
    const int lo_rel = (int)(lr < -1 ? -1 : lr);
    const unsigned span = (unsigned)(4 * kTileMaxDelay - lo_rel);  // (a filler's delay is past it)
    // a batch of n spikes is n << lg parts of segments; `done` of them taken
    int n = 0, done = 0;
    bool more = src.begin(a, t, m, n);
    int32_t id1[U];   // ids and steps of the parts whose offsets come next
    int j1[U];
    uint32_t k0[U], e0[U];  // segments of the parts to deliver, their steps
    int j0[U];
    auto ids = [&]() {      // the next parts' ids; begins the next batch after the last
#pragma unroll
        for (int u = 0; u < U; ++u) {
            id1[u] = -1;
            j1[u] = 0;
            const int p = done + u * 32 + lane;
            if (more && (p >> lg) < n) id1[u] = src.load(t, m, p >> lg, j1[u]);
        }
    };
    auto offsets = [&]() {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            k0[u] = e0[u] = 0;
            if (id1[u] >= 0 && MGC_OK_INDEX(id1[u] < a.n_src)) {
                const uint32_t* o = t.off + (size_t)id1[u] * t.T + blockIdx.x;
                k0[u] = __ldg(o);
                e0[u] = __ldg(o + 1);
            }
            j0[u] = j1[u];
        }
    };
    auto advance = [&]() {  // past the parts whose ids are loaded
        done += kTileBatch;
        if (done >= n << lg) {
            done = 0;
            more = src.begin(a, t, m, n);
        }
    };
    if (!more) return;
    ids();
    offsets();
    int part = done;  // first part of the batch whose segments come next
    advance();
    ids();
#pragma unroll 1
    for (bool go = true; go;) {
        // these parts' segments
        uint32_t k[U], e[U];
        int base[U], j[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            j[u] = j0[u];
            int sl = slot0 + j[u];
            if (sl >= t.R) sl -= t.R;
            k[u] = k0[u];
            e[u] = e0[u];
            if (ONE) {  // (R = dmin: the arrival row is the spike's own)
                sl = sl * t.stride * 4 + (int)(k[u] >> 31);
                k[u] &= 0x7fffffffu;
                e[u] &= 0x7fffffffu;
                if ((unsigned)(j[u] + t.dmin - lo_rel - 1) >= span) e[u] = k[u];
            }
            base[u] = sl;
            if (!MGC_OK_INDEX(k[u] <= e[u] && e[u] <= t.n_vec)) e[u] = k[u];
            if (lg) {
                const uint32_t len = e[u] - k[u], p = (uint32_t)(part + u * 32 + lane) & ((1u << lg) - 1u);
                e[u] = k[u] + ((len * (p + 1)) >> lg);
                k[u] += (len * p) >> lg;
            }
        }
        go = more;
#pragma unroll 1
        for (bool first = true;; first = false) {
            Vec v[U][D];
            bool rest = false;
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int d = 0; d < D; ++d)
                    if (k[u] + d < e[u]) v[u][d] = __ldg(rec + k[u] + d);
            if (first && go) {  // behind them, the next parts' offsets and the ids after those
                offsets();
                part = done;
                advance();
                ids();
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
#pragma unroll
                for (int d = 0; d < D; ++d)
                    if (k[u] + d < e[u])
                        tile_apply_vec<FX, ONE>(a, t, m, v[u][d], base[u], j[u], lo_rel, span);
                k[u] += D;
                rest |= k[u] < e[u];
            }
            if (!rest) break;
        }
    }
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

// The tile's c spikes of window k (the first kTileInline in `first`) into every
// tile's mailbox, thread r into tile r's.  Called by the whole block after a
// block barrier.
__device__ __forceinline__ void tile_publish(const TileArgs& t, int k, int c, const uint32_t* first)
{
    if ((int)threadIdx.x < t.T) {
        ulonglong2* p = t.mail + (((size_t)(k & 1) * t.T + threadIdx.x) * t.T + blockIdx.x) * kTileChunks;
        const unsigned long long epoch = (unsigned long long)(t.epoch + (uint32_t)k) << 32;
        if (c > kTileInline) asm volatile("fence.acq_rel.gpu;" ::: "memory");
        st_head(p, make_ulonglong2(epoch | (uint32_t)c, (unsigned long long)first[0] | ((unsigned long long)first[1] << 32)));
        if (c > 2 && c <= kTileInline)
            for (int q = 2; q < c; q += 3)  // (the last chunk may hold stale words past c)
                st_head(p + 1 + (q - 2) / 3, make_ulonglong2(epoch | first[q], (unsigned long long)first[q + 1] |
                                                                                 ((unsigned long long)first[q + 2] << 32)));
    }
}

// A chunk of the wanted epoch, waited for.
__device__ __forceinline__ ulonglong2 tile_wait(const StepArgs& a, const ulonglong2* p, uint32_t epoch, int* abort_flag)
{
    ulonglong2 v = ld_head(p);
    for (unsigned it = 0; (uint32_t)(v.x >> 32) != epoch; v = ld_head(p)) {
        if (++it > kBarrierSpins) {
            atomicOr(a.status, kStatusBarrier);
            *abort_flag = 1;
            return make_ulonglong2(0, 0);
        }
        if (it > 64) __nanosleep(32);
    }
    return v;
}

// Waits until every tile has published window k.  *n (zero on entry) gets the
// window's spikes, m.cnt the tiles' counts; when the spikes fit, they are all
// in m.spikes.  False on a time-out.
__device__ __forceinline__ bool tile_gather(const StepArgs& a, const TileArgs& t, const TileSmem& m, int k,
                                            const uint32_t* lists, size_t list_len, int* n, int* abort_flag)
{
    bool listed = false;  // the tile has more spikes than its mailbox place holds
    if ((int)threadIdx.x < t.T) {
        const uint32_t epoch = t.epoch + (uint32_t)k;
        const ulonglong2* p = t.mail + (((size_t)(k & 1) * t.T + blockIdx.x) * t.T + threadIdx.x) * kTileChunks;
        const ulonglong2 v = tile_wait(a, p, epoch, abort_flag);
        const int c = (int)(uint32_t)v.x;
        int at = 0;
        if (c > 0) {
            at = atomicAdd(n, c);
            listed = c > kTileInline;
            if (listed) asm volatile("fence.acq_rel.gpu;" ::: "memory");
            const bool fits = at + c <= kTileSpikes;
            uint32_t* out = m.spikes + at;
            if (fits) {
                out[0] = (uint32_t)v.y;
                if (c > 1) out[1] = (uint32_t)(v.y >> 32);
            }
            if (!listed) {
                const int chunks = (c - 2 + 2) / 3;  // after the first
#pragma unroll 1
                for (int g = 0; g < chunks; g += 5) {
                    ulonglong2 w[5];
#pragma unroll
                    for (int u = 0; u < 5; ++u)  // in flight together
                        if (g + u < chunks) w[u] = ld_head(p + 1 + g + u);
#pragma unroll
                    for (int u = 0; u < 5; ++u) {
                        if (g + u >= chunks) continue;
                        if ((uint32_t)(w[u].x >> 32) != epoch) w[u] = tile_wait(a, p + 1 + g + u, epoch, abort_flag);
                        const int q = 2 + 3 * (g + u);
                        if (!fits) continue;
                        out[q] = (uint32_t)w[u].x;
                        if (q + 1 < c) out[q + 1] = (uint32_t)w[u].y;
                        if (q + 2 < c) out[q + 2] = (uint32_t)(w[u].y >> 32);
                    }
                }
            }
        }
        m.cnt[threadIdx.x] = c;
        m.at[threadIdx.x] = at;
    }
    const bool any = __syncthreads_or(listed);
    if (any && *n <= kTileSpikes) {  // the lists, eight lanes a tile
        for (int l = threadIdx.x >> 3; l < t.T; l += blockDim.x >> 3) {
            const int c = m.cnt[l];
            if (c <= kTileInline) continue;
            const uint32_t* from = lists + (size_t)l * list_len;
#pragma unroll 4
            for (int q = 2 + (threadIdx.x & 7); q < c; q += 8) m.spikes[m.at[l] + q] = __ldcg(from + q);
        }
        __syncthreads();
    }
    return *abort_flag == 0;
}

// After a wait that ran out, the step counters and a.done hold part of that
// launch: places computed from them could lie outside the history.  No launch
// runs any more until a checkpoint is loaded, which clears them and the status.
__device__ __forceinline__ int tile_refused(const StepArgs& a)
{
    return (*(volatile int32_t*)a.status & kStatusBarrier) != 0;
}

template <bool CUR, bool FX, bool ONE>
__global__ void __launch_bounds__(kTileThreads, 1) k_tile(StepArgs a, TileArgs t, int32_t nsteps)
{
    extern __shared__ __align__(16) unsigned char tile_raw[];
    __shared__ int abort_flag;
    __shared__ unsigned long long blk_ev;
    __shared__ int count, npg, total;  // the tile's spikes of the window, its POISSON groups, all tiles' spikes
    __shared__ uint32_t mine[kTileInline + 2];  // (a chunk's words past the last spike are read)
    __shared__ int scnt[kTileWindow];      // this window's spikes per step
    __shared__ int32_t sbase[2][kTileWindow], stot[kTileWindow + 1];  // places reserved in the steps, the steps' totals
    __shared__ int32_t ctot[4][kTileWindow];  // the counters' last totals
    const TileSmem m = tile_smem<CUR, FX>(tile_raw, t);
    const int tile = blockIdx.x, tid = threadIdx.x;
    const int64_t s0 = *a.step;
    const int32_t slot0 = a.slots[0], h0 = a.slots[1];
    const bool rec = a.record != 0;
    int64_t rbase = rec ? *a.raster_pos : 0;
    const int64_t rstep0 = *a.raster_step0;
    const int64_t s_end = s0 + nsteps;
    // arrivals of this launch, whose events it counts: (lo, hi]
    const int64_t lo = t.ahead ? s0 : s0 - 1, hi = t.ahead ? s_end : s_end - 1;
    auto hs_of = [&](int64_t x) {  // history slot of a step within H of s0, or later
        int64_t h = (h0 + (x - s0)) % a.H;
        return (int32_t)(h < 0 ? h + a.H : h);
    };
    unsigned long long ev = 0;
    auto events_of = [&](int32_t id, int64_t x) {  // a spike's synapses whose arrival is in (lo, hi]
        if (ONE) return (unsigned long long)(x + t.dmin > lo && x + t.dmin <= hi ? a.row_ptr[id + 1] - a.row_ptr[id] : 0);
        const int64_t a0 = lo - x - t.dmin + 1, a1 = hi - x - t.dmin + 1;
        const int64_t* bk = a.bucket + (size_t)id * a.D;
        const int k0 = (int)(a0 < 0 ? 0 : a0 > a.D ? a.D : a0), k1 = (int)(a1 < 0 ? 0 : a1 > a.D ? a.D : a1);
        return (unsigned long long)(k0 < k1 ? bk[k1] - bk[k0] : 0);
    };
    // the ring, words of 16 bytes (a row's entries are a multiple of 4)
    const int ring_words = (FX ? 4 : 1) * t.R * t.stride / 4;
    uint4* pend = reinterpret_cast<uint4*>(t.pend) + (size_t)tile * ring_words;
    const bool kept = *t.pend_step == s0;

    // state of the tile, its ring
    {
        uint4* z = reinterpret_cast<uint4*>(m.ring);
#pragma unroll 4
        for (int k = tid; k < ring_words; k += blockDim.x) {
            const uint4 v = __ldcg(pend + k);  // (loaded before it is known whether it counts)
            z[k] = kept ? v : make_uint4(0, 0, 0, 0);
        }
#pragma unroll 1
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
#pragma unroll 1
            for (int k = tid; k < 2 * kTileTable; k += blockDim.x) m.tab[k] = t.chain[k];
        if (tid < kTileWindow) scnt[tid] = 0;
        if (tid < 4 * kTileWindow) ctot[tid / kTileWindow][tid % kTileWindow] = 0;
        if (tid == 0) {
            abort_flag = tile_refused(a);
            blk_ev = 0;
            count = npg = total = 0;
        }
    }
    __syncthreads();
    if (abort_flag) return;
    for (int g = tid; g < t.nl / 4; g += blockDim.x) {
        bool p = false;
        for (int q = 0; q < 4; ++q) p |= m.type[4 * g + q] == kPOISSON;
        if (p) m.pg[atomicAdd(&npg, 1)] = (uint16_t)g;
    }
    __syncthreads();
    const int n_pg = npg;
    // the last R steps before s0: their spikes that arrive later, when the ring was
    // not kept, and the events of this launch's steps, a warp a step or part of one
    {
        const int64_t x0 = s0 - t.R > 0 ? s0 - t.R : 0;
        const int nst = (int)(s0 - x0);
        if (!kept) {
#pragma unroll 1
            for (int j = tid; j < nst; j += blockDim.x) m.cnt[j] = __ldcg(a.hist_cnt + hs_of(x0 + j));
            __syncthreads();
            TileSource src;
            src.listed(TileSource::kHistory, nst, hs_of(x0));
            tile_deliver<FX, ONE>(a, t, m, x0, (int)(x0 % t.R), lo, src);
        }
        const int lane = tid & 31, warps = t.T * (int)(blockDim.x >> 5);
        const int each = nst > 0 && warps > nst ? warps / nst : 1;  // warps of a step
        const int h_first = hs_of(x0);
#pragma unroll 1
        for (int w = tile + (tid >> 5) * t.T; w < nst * each; w += warps) {
            const int j = w / each, part = w - j * each;
            if (x0 + j + t.dmin > hi || x0 + j + t.dmax <= lo) continue;
            const int h = h_first + j, hs = h >= a.H ? h - a.H : h;
            const int c = __ldcg(a.hist_cnt + hs);
#pragma unroll 1
            for (int q = part * 32 + lane; q < c; q += each * 32) {
                const int32_t id = __ldcg(a.hist_ids + (size_t)hs * (size_t)a.n_src + q);
                if (MGC_OK_INDEX(id >= 0 && id < a.n_src)) ev += events_of(id, x0 + j);
            }
        }
        __syncthreads();
    }
    // the spikes of window k (w steps from x0): their raster places, and the
    // history of the launch's last steps; the counters of the window are final
    const size_t list_len = (size_t)t.nl * t.W;
    auto my_list = [&](int k) { return t.list + ((size_t)(k % kTileLists) * t.T + tile) * list_len; };
    const int32_t h_end = hs_of(s_end);
    auto hs_last = [&](int64_t x) {  // history slot of a step less than H before s_end
        const int32_t h = h_end - (int32_t)(s_end - x);
        return h < 0 ? h + a.H : h;
    };
    auto record = [&](int k, int64_t x0, int w, int c) {  // stot, sbase ready; c: this tile's spikes
#pragma unroll 1
        for (int q = tid; q < c; q += blockDim.x) {
            const uint32_t e = my_list(k)[q];
            const int32_t id = (int32_t)(e & kTileId);
            const int j = (int)(e >> kTileStepShift);
            const int at = atomicAdd(&sbase[k & 1][j], 1);  // any order inside a step
            const int64_t x = x0 + j, rb = rbase + stot[j] + at;
            if (rec && rb < a.raster_ids_cap) a.raster_ids[rb] = id;
            if (x > s_end - a.H && MGC_OK_INDEX(at < a.n_src)) a.hist_ids[(size_t)hs_last(x) * (size_t)a.n_src + at] = id;
            ev += events_of(id, x);
        }
        if (tile == 0 && tid < w) {
            const int64_t x = x0 + tid;
            const int c_all = stot[tid + 1] - stot[tid];
            if (x > s_end - a.H) a.hist_cnt[hs_last(x)] = c_all;
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
    // running sums of window k's step totals (n_all in all), by the last warp, which
    // has the fewest spikes to deliver; now: the counters as read before
    const int last = tid - (kTileThreads - 32);
    int gave_up = 0;  // (counters that never added up)
    auto totals = [&](int k, int w, int n_all, int32_t now) {
        if (last >= 0) {
            int c;
            for (unsigned it = 0;;) {
                c = last < w ? now - ctot[k & 3][last] : 0;
#pragma unroll
                for (int o = 1; o < kTileWindow; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, c, o);
                    if (last >= o) c += v;
                }
                if (__shfl_sync(0xffffffffu, c, kTileWindow - 1) == n_all || !tile_again(a, it, &gave_up)) break;
                if (last < w) now = tile_count(t, k, last);
            }
            if (last < w) ctot[k & 3][last] = now;
            if (last < w) stot[last + 1] = c;
            if (last == 0) stot[0] = 0;
        }
    };
    int slot = (int)(s0 % t.R);
    int k = 0, c_prev = 0, w_prev = 0, n_prev = 0;  // the window before: this tile's spikes, steps, all spikes
    int64_t w0 = s0;
    for (; w0 < s_end; ++k) {
        const int wl = (int)(s_end - w0 < t.W ? s_end - w0 : t.W);
        if (n_pg) tile_poisson(a, t, m, w0, wl, n_pg, my_list(k), mine, &count, scnt);
        tile_update<CUR, FX>(a, t, m, w0, wl, slot, t.ahead && k == 0, my_list(k), mine, &count, scnt);
        __syncthreads();
        const int c_now = count;
        tile_publish(t, k, c_now, mine);
        // the steps' places for this tile's spikes, needed a window later
        int place = 0;
        if (tid >= 32 && tid < 32 + wl && scnt[tid - 32])
            place = atomicAdd(tile_counter(t, k, tid - 32), scnt[tid - 32]);
        const int32_t early = k > 0 && last >= 0 && last < w_prev ? tile_count(t, k - 1, last) : 0;
        const uint32_t* lists = t.list + (size_t)(k % kTileLists) * t.T * list_len;
        if (!tile_gather(a, t, m, k, lists, list_len, &total, &abort_flag)) return;
        if (tid >= 32 && tid < 32 + kTileWindow) {
            sbase[k & 1][tid - 32] = place - ctot[k & 3][tid - 32];
            scnt[tid - 32] = 0;
        }
        if (tid == 0) count = 0;
        if (k > 0) totals(k - 1, w_prev, n_prev, early);
        TileSource src;
        n_prev = total;
        if (n_prev <= kTileSpikes)
            src.gathered(n_prev);
        else
            src.listed(TileSource::kTiles, t.T, k);
        tile_deliver<FX, ONE>(a, t, m, w0, slot, lo, src);
        if (__syncthreads_or(gave_up)) return;
        if (tid == 0) total = 0;
        if (k > 0) record(k - 1, w0 - w_prev, w_prev, c_prev);
        c_prev = c_now;
        w_prev = wl;
        w0 += wl;
        slot += wl;
        if (slot >= t.R) slot -= t.R;
    }
    // the last window's raster and history: an empty window makes its counters final
    tile_publish(t, k, 0, mine);
    if (!tile_gather(a, t, m, k, t.list, 0, &total, &abort_flag)) return;
    totals(k - 1, w_prev, n_prev, last >= 0 && last < w_prev ? tile_count(t, k - 1, last) : 0);
    if (__syncthreads_or(gave_up)) return;
    record(k - 1, w0 - w_prev, w_prev, c_prev);
    // back to the single-step form: the state, and the arrivals of s_end
#pragma unroll 1
    for (int i = tid; i < t.nl; i += blockDim.x) {
        const int32_t gi = tile_neuron(t, i, tile);
        if (gi >= a.ns) continue;
        if (m.type[i] == kPOISSON || m.type[i] == kRAW) continue;  // they keep V and ignore their input (whose
                                                                   // ring words may run over: 32 bits each)
        a.V[gi] = m.V[i];
        a.refrac[gi] = m.rf[i];
        if (CUR) {
            a.Iexc[gi] = m.ie[i];
            a.Iinh[gi] = m.ii[i];
        }
        if (t.ahead) {
            const size_t at = (size_t)slot * t.stride + i;
            if (FX) {
                unsigned long long* e = reinterpret_cast<unsigned long long*>(m.ring);
                acc_buf<FX>(a, a.acc_e, s_end)[gi] = (typename AccT<FX>::type)e[at];
                acc_buf<FX>(a, a.acc_i, s_end)[gi] = (typename AccT<FX>::type)e[(size_t)t.R * t.stride + at];
                e[at] = e[(size_t)t.R * t.stride + at] = 0;
            } else {
                uint32_t* ring = reinterpret_cast<uint32_t*>(m.ring);
                const uint32_t c = ring[at];
                acc_buf<FX>(a, a.acc_e, s_end)[gi] = (typename AccT<FX>::type)chain_sum(c & 0xffffu, m.we[i], m.tab);
                acc_buf<FX>(a, a.acc_i, s_end)[gi] =
                    (typename AccT<FX>::type)chain_sum(c >> 16, m.wi[i], m.tab ? m.tab + kTileTable : nullptr);
                ring[at] = 0;
            }
        }
    }
    __syncthreads();
#pragma unroll 4
    for (int k = tid; k < ring_words; k += blockDim.x) pend[k] = reinterpret_cast<const uint4*>(m.ring)[k];
    if (ev) atomicAdd(&blk_ev, ev);
    __syncthreads();
    if (tid == 0 && blk_ev) atomicAdd(a.events, blk_ev);
    // the clock, by the last block to finish
    if (last_block(a.done) && tid == 0) {
        if (rec) *a.raster_pos = rbase;
        if (a.ev_mark) *a.ev_mark = *(volatile unsigned long long*)a.events;
        a.hist_cnt[h_end] = 0;
        for (int j = 0; j < 4 * kTileWindow; ++j) t.cnt[j * kTileLine] = 0;
        *a.done = 0;
        a.slots[0] = (int32_t)((slot0 + nsteps) % a.M);
        a.slots[1] = h_end;
        *a.step = s_end;
        *t.pend_step = s_end;
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
// weights.  784 -> 1,600 plastic network, 1.9e4 events a step: 12.1 us a step
// with the single-step ring kernels, 5.1 here.
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
    __shared__ int abort_flag, late;  // waits that ran out: for the mailboxes, the counters
    __shared__ unsigned long long blk_ev;
    __shared__ int count, npg, total;
    __shared__ uint32_t mine[kTileInline + 2];
    __shared__ int scnt[kTileWindow];
    __shared__ int32_t sbase[2], stot, ctot[4];   // places reserved in a step, a step's spikes, the counters' totals
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
#pragma unroll 1
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
    // (a faster block may already have written a spike of step s0 here, which the
    // exchange brings this block before anything reads it)
    for (int i = tid; i < a.n; i += blockDim.x) q.lf[i] = __ldcg(a.last_fired + i);
    for (int i = tid; i < (a.n + 31) / 32; i += blockDim.x) q.fired[i] = 0;
    for (int i = tid; i <= t.nl; i += blockDim.x) q.in_off[i] = t.in_off[(size_t)tile * t.nl + i];
    if (tid < kTileWindow) scnt[tid] = 0;
    if (tid < 4) ctot[tid] = 0;
    if (tid == 0) {
        abort_flag = tile_refused(a);
        late = 0;
        blk_ev = 0;
        count = npg = total = 0;
    }
    __syncthreads();
    if (abort_flag) return;
    for (int g = tid; g < t.nl / 4; g += blockDim.x) {
        bool p = false;
        for (int x = 0; x < 4; ++x) p |= m.type[4 * g + x] == kPOISSON;
        if (p) m.pg[atomicAdd(&npg, 1)] = (uint16_t)g;
    }
    __syncthreads();
    const int n_pg = npg;
    const size_t list_len = (size_t)t.nl * t.W;
    auto my_list = [&](int k) { return t.list + ((size_t)(k % kTileLists) * t.T + tile) * list_len; };
    // f(id) for every spike of the step, the block's threads (or groups of
    // `width` of them) in turn
    auto each_spike = [&](int k, int group, int groups, auto f) {
        if (total <= kTileSpikes) {
#pragma unroll 1
            for (int x = group; x < total; x += groups) f((int32_t)(m.spikes[x] & kTileId));
        } else {
#pragma unroll 1
            for (int l = 0; l < t.T; ++l)
#pragma unroll 1
                for (int x = group; x < m.cnt[l]; x += groups)
                    f((int32_t)((m.cnt[l] > kTileInline ? __ldcg(tile_list(t, k, l) + x) : tile_mail(t, k, l, x)) & kTileId));
        }
    };
    // step k's spikes, n_all in all (one thread); now: the counter as read before
    auto total_of = [&](int k, int n_all, int32_t now) {
        for (unsigned it = 0; now - ctot[k & 3] != n_all && tile_again(a, it, &late);) now = tile_count(t, k, 0);
        stot = now - ctot[k & 3];
        ctot[k & 3] = now;
    };
    // raster places of step x's spikes (the step's counter is final), one step late
    auto record = [&](int k, int64_t x, int c) {
#pragma unroll 1
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
    int k = 0, c_prev = 0, n_prev = 0;
    for (int64_t s = s0; s < s_end; ++s, ++k) {
        if (n_pg) tile_poisson(a, t, m, s, 1, n_pg, my_list(k), mine, &count, scnt);
        tile_update<CUR, true>(a, t, m, s, 1, slot, false, my_list(k), mine, &count, scnt);
        __syncthreads();
        const int c_now = count;
        tile_publish(t, k, c_now, mine);
        int place = 0;
        if (tid == 32 && c_now) place = atomicAdd(tile_counter(t, k, 0), c_now);
        const int32_t early = k > 0 && tid == kTileThreads - 1 ? tile_count(t, k - 1, 0) : 0;
        if (!tile_gather(a, t, m, k, tile_list(t, k, 0), list_len, &total, &abort_flag)) return;
        if (tid == 32) {
            sbase[k & 1] = place - ctot[k & 3];
            scnt[0] = 0;
        }
        if (tid == 0) count = 0;
        if (k > 0 && tid == kTileThreads - 1) total_of(k - 1, n_prev, early);  // (it has the fewest spikes to deliver)
        n_prev = total;
        each_spike(k, tid, blockDim.x, [&](int32_t id) {
            if (!MGC_OK_INDEX(id >= 0 && id < a.n)) return;
            q.lf[id] = (int32_t)s;
            atomicOr(q.fired + (id >> 5), 1u << (id & 31));
        });
        __syncthreads();
        if (late) return;
        // this tile's synapses of the spiking sources, eight lanes a source
        each_spike(k, tid >> 3, blockDim.x >> 3, [&](int32_t id) {
            if (!MGC_OK_INDEX(id >= 0 && id < a.n)) return;
            const uint32_t* o = t.off + (size_t)id * t.T + tile;
            const uint32_t b = __ldg(o), e = __ldg(o + 1);
            if (!MGC_OK_INDEX(b <= e && e <= t.n_vec)) return;
#pragma unroll 1
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
            const int32_t id = (int32_t)((y < kTileInline ? mine[y] : __ldcg(my_list(k) + y)) & kTileId);  // (uniform)
            const int g = id >> 2, local = g / t.T * 4 + (id & 3);
            const uint32_t e = q.in_off[local + 1];
#pragma unroll 1
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
    tile_publish(t, k, 0, mine);
    if (!tile_gather(a, t, m, k, t.list, 0, &total, &abort_flag)) return;
    if (tid == 0) total_of(k - 1, n_prev, tile_count(t, k - 1, 0));
    __syncthreads();
    if (late) return;
    record(k - 1, s_end - 1, c_prev);
#pragma unroll 1
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
        for (int j = 0; j < 4 * kTileWindow; ++j) t.cnt[j * kTileLine] = 0;
        *a.done = 0;
        a.slots[0] = (int32_t)((slot0 + nsteps) % a.M);
        *a.step = s_end;
    }
}

}  // namespace mgc
