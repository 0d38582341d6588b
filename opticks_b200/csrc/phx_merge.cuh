// phx_merge.cuh : hit merging on the device — select records by flag mask, group them by
// (identity, time bucket) and reduce each group to one record with a summed hit count.
//
// Semantics follow SPM::merge_partial_select (sysrap/SPM.cu:110-200) with the record functors of
// sysrap/sphoton.h:292-320 (sphoton, 64 B) and sysrap/sphotonlite.h:68-97 (sphotonlite, 16 B):
//   select   (flagmask & mask) != 0, or every record when mask == 0xffffffff (already selected)
//   key      (uint64(identity) << 48) | unsigned(time / window)   (identity bits above 16 drop out)
//   order    groups ascending by key; within a group the input order decides ties
//   reduce   sphoton     : the earliest-time record (ties: first in input order), flagmask = OR,
//                          hitcount = sum (16 bits)
//            sphotonlite : the first record in input order, time = min, flagmask = OR,
//                          hitcount = sum (16 bits)
//   window 0 : selection only, records in input order
//
// The reference sorts with thrust::sort_by_key and folds with thrust::reduce_by_key.  Every reduction
// above is associative and commutative over (time, position), so no order is needed to compute it,
// only the rank of a key among the keys that occur:
//   1. k_merge_range   keys of the selected records, their count and the ranges of identity and bucket
//   2. k_merge_present one bit per (identity, bucket) cell of that range, set where a key occurs
//   3. k_merge_rank    popcount prefix of the bit table: a cell's rank is its group index, and groups
//                      come out in ascending key order
//   4. k_merge_fold    atomics of each record into its group: min (time, position), OR, sum
//   5. k_merge_groups  the representative record of each group with the reduced fields
// in one go without a host read (the table's size comes from n, the range stays on the device).  1M
// sphoton records with a fifth selected, 1 ns windows: 79 us a call, against 247 us through the sort
// (35 launches and three host reads); what is left is six launches and one read at 4-20 us apiece.
// Ranges whose cells outnumber the table (phx_merge_cells) are left to a stable sort of the keys.  They are
// ordinary: with 17,612 sensors the 2^24 cells of a small event are 952 buckets, so one microsecond-late
// selected record at 1 ns is enough.  The failed attempt (a read of the records and five launches that leave
// at once) is paid back by its keys: 4M records, a fifth selected, 433 us before there was a table, 500 with
// the sort started over, 396 with the keys taken over; 100,000 all selected 212, 236, 225; 1,000 162, 192, 152.
//   1. ordered selection from the keys (ballot + tile offsets) -> input positions and keys
//   2. passes only over the key bytes in use
//   3. stable LSD radix sort, 8-bit digits: per-tile digit histograms (digit-major), one scan,
//      a scatter ranking equal digits by __match_any_sync so every pass is stable
//   4. group heads + scan -> group index; warp-segmented reductions (__reduce_*_sync over the
//      lanes of one group) with one atomic per (warp, group): min (time, position), min position,
//      OR flagmask, sum hitcount
//   5. one thread per group writes the representative record with the reduced fields
// Scratch: the table form takes 24 B an input record (28 for sphotonlite) and the table, the sort form 25 B a
// selected record besides.  Where either has no room in device memory the range alone is found and the
// sort form starts from the records, at 33 B a selected one and 16 to 20 a group.
// Each form picks the record the left fold of reduce_op picks.  Included by phx_engine.cu after
// DevBuf and PHX_CU.
#pragma once
#include <stdint.h>

#define PHX_MERGE_TILE_ITEMS 8
#define PHX_MERGE_TILE (256 * PHX_MERGE_TILE_ITEMS)
#define PHX_MERGE_SCAN_TILE 1024

// word offsets of the fields a merge reads/writes, per record kind
template <int LITE> struct PhxRec;
template <> struct PhxRec<0> {       // sphoton (sysrap/sphoton.h:171-192)
    static constexpr int W = 16, TIME = 3, HC = 7, ID = 13, FLAG = 15;
    static constexpr uint32_t IDMASK = 0xffffffu;
};
template <> struct PhxRec<1> {       // sphotonlite (sysrap/sphotonlite.h:47-51)
    static constexpr int W = 4, TIME = 1, HC = 0, ID = 0, FLAG = 3;
    static constexpr uint32_t IDMASK = 0xffffu;
};

// monotone map of float bits to u32 order; NaN after +inf (fminf ignores NaN)
__device__ __forceinline__ uint32_t phx_time_order(uint32_t b)
{
    if ((b & 0x7fffffffu) > 0x7f800000u) return 0xffffffffu;
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ uint32_t phx_time_unorder(uint32_t o)
{
    if (o == 0xffffffffu) return 0x7fc00000u;
    return (o & 0x80000000u) ? (o & 0x7fffffffu) : ~o;
}

// ---------------------------------------------------------------- table form
// Bits of the cell table for n records: 32 per record (4 B), and never fewer than 2^24 (2 MB).  The
// whole table is cleared on each call, and the range's part of it read and its offsets written (8 B a
// word): against a 16 B record at most three quarters of its bytes, below 524,288 records 2 MB whatever n.
__host__ __device__ inline unsigned long long phx_merge_cells(long long n)
{
    const unsigned long long c = 32ull * (unsigned long long)n;
    return c < (1ull << 24) ? (1ull << 24) : c < (1ull << 31) ? ((c + 32767ull) & ~32767ull) : (1ull << 31);
}

// what k_merge_range finds out (zeroed before it); minima are kept as maxima of the complement
struct PhxMergeRange {
    uint32_t id_max, id_cmin, bk_max, bk_cmin;
    unsigned long long count;
    long long groups;
};

// the cells of a range: identities x buckets, 0 when nothing was selected
struct PhxMergeMap {
    uint32_t id0, bk0, nbk;
    unsigned long long cells;
};
__host__ __device__ inline PhxMergeMap phx_merge_map(const PhxMergeRange& r)
{
    PhxMergeMap m;
    m.id0 = ~r.id_cmin;
    m.bk0 = ~r.bk_cmin;
    m.nbk = r.bk_max - m.bk0 + 1u;                   // 0: 2^32 buckets
    const unsigned long long nb = m.nbk ? (unsigned long long)m.nbk : (1ull << 32);
    m.cells = r.count ? (unsigned long long)(r.id_max - m.id0 + 1u) * nb : 0ull;
    return m;
}

// does key byte b (0-3 bucket, 4-5 unused, 6-7 identity) hold a bit of any key?
__host__ __device__ inline bool phx_merge_byte_used(const PhxMergeRange& r, int b)
{
    if (b < 4) return (r.bk_max >> (8 * b)) != 0u;
    return b >= 6 && (r.id_max >> (8 * (b - 6))) != 0u;
}

#define PHX_MERGE_NONE 0xffffffffffffffffull         // key of a record that is not selected (identities are 16 bits)

template <int LITE>
__device__ __forceinline__ unsigned long long phx_merge_key(const uint32_t* r, float tw)
{
    const uint32_t id = r[PhxRec<LITE>::ID] & PhxRec<LITE>::IDMASK;
    const unsigned bucket = static_cast<unsigned>(__uint_as_float(r[PhxRec<LITE>::TIME]) / tw);
    return ((unsigned long long)id << 48) | (unsigned long long)bucket;
}

template <int LITE>
__device__ __forceinline__ void phx_merge_clear(long long g, unsigned long long* amin, uint32_t* pmin, uint32_t* gor, uint32_t* gsum)
{
    amin[g] = 0xffffffffffffffffull;
    if (LITE) pmin[g] = 0xffffffffu;
    gor[g] = 0u;
    gsum[g] = 0u;
}

// 1. keys and their ranges; also clears the cell table (key null: the range alone)
template <int LITE>
__global__ void __launch_bounds__(256) k_merge_range(const uint32_t* in, long long n, uint32_t mask, float tw, unsigned long long* key,
                                                     PhxMergeRange* range, uint32_t* cell, long long ncellw)
{
    __shared__ uint32_t s_id, s_idc, s_bk, s_bkc, s_cnt;
    if (threadIdx.x == 0) s_id = s_idc = s_bk = s_bkc = s_cnt = 0u;
    __syncthreads();
    const long long at = (long long)blockIdx.x * blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
    for (long long j = at; j < ncellw / 4; j += stride) reinterpret_cast<uint4*>(cell)[j] = make_uint4(0u, 0u, 0u, 0u);
    uint32_t id = 0u, idc = 0u, bk = 0u, bkc = 0u, cnt = 0u;
    for (long long j = at; j < n; j += stride) {
        const uint32_t* r = in + j * PhxRec<LITE>::W;
        unsigned long long k = PHX_MERGE_NONE;
        if (mask == 0xffffffffu || (r[PhxRec<LITE>::FLAG] & mask) != 0u) {
            k = phx_merge_key<LITE>(r, tw);
            const uint32_t i = (uint32_t)(k >> 48), b = (uint32_t)k;
            id = max(id, i); idc = max(idc, ~i); bk = max(bk, b); bkc = max(bkc, ~b);
            cnt++;
        }
        if (key) key[j] = k;
    }
    const unsigned FULL = 0xffffffffu;
    id = __reduce_max_sync(FULL, id); idc = __reduce_max_sync(FULL, idc);
    bk = __reduce_max_sync(FULL, bk); bkc = __reduce_max_sync(FULL, bkc);
    cnt = __reduce_add_sync(FULL, cnt);
    if ((threadIdx.x & 31) == 0 && cnt) {
        atomicMax(&s_id, id); atomicMax(&s_idc, idc); atomicMax(&s_bk, bk); atomicMax(&s_bkc, bkc);
        atomicAdd(&s_cnt, cnt);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_cnt) {
        atomicMax(&range->id_max, s_id); atomicMax(&range->id_cmin, s_idc);
        atomicMax(&range->bk_max, s_bk); atomicMax(&range->bk_cmin, s_bkc);
        atomicAdd(&range->count, (unsigned long long)s_cnt);
    }
}

__device__ __forceinline__ uint32_t phx_merge_cell(const PhxMergeMap& m, unsigned long long k)
{
    return ((uint32_t)(k >> 48) - m.id0) * m.nbk + ((uint32_t)k - m.bk0);
}

// 2. the cells that occur
__global__ void __launch_bounds__(256) k_merge_present(const unsigned long long* key, long long n, const PhxMergeRange* range,
                                                       unsigned long long most, uint32_t* cell)
{
    const PhxMergeMap m = phx_merge_map(*range);
    if (m.cells == 0ull || m.cells > most) return;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += stride) {
        const unsigned long long k = key[j];
        if (k == PHX_MERGE_NONE) continue;
        const uint32_t c = phx_merge_cell(m, k);
        const uint32_t bit = 1u << (c & 31u);
        if (!(cell[c >> 5] & bit)) atomicOr(cell + (c >> 5), bit);   // a stale read only costs the atomic
    }
}

// 3. popcount prefix of the table, 1024 words a block (offsets within the block, block totals); also clears the
// group slots, where the table form goes on
template <int LITE>
__global__ void __launch_bounds__(256) k_merge_rank(const uint32_t* cell, const PhxMergeRange* range, unsigned long long most,
                                                    uint32_t* off, uint32_t* blocksum, long long n, unsigned long long* amin,
                                                    uint32_t* pmin, uint32_t* gor, uint32_t* gsum)
{
    const PhxMergeMap m = phx_merge_map(*range);
    if (m.cells <= most) {
        const long long stride = (long long)gridDim.x * blockDim.x;
        for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < n; g += stride) phx_merge_clear<LITE>(g, amin, pmin, gor, gsum);
    }
    const unsigned long long w0 = (unsigned long long)blockIdx.x * 1024ull;
    if (m.cells > most || w0 * 32ull >= m.cells) {
        if (threadIdx.x == 0) blocksum[blockIdx.x] = 0u;
        return;
    }
    __shared__ uint32_t wt[8];
    const uint4 v = reinterpret_cast<const uint4*>(cell)[w0 / 4 + threadIdx.x];
    const uint32_t c0 = __popc(v.x), c1 = __popc(v.y), c2 = __popc(v.z), s = c0 + c1 + c2 + __popc(v.w);
    uint32_t inc = s;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) { const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += y; }
    if (lane == 31) wt[wid] = inc;
    __syncthreads();
    uint32_t run = inc - s;
    for (int k = 0; k < wid; k++) run += wt[k];
    reinterpret_cast<uint4*>(off)[w0 / 4 + threadIdx.x] = make_uint4(run, run + c0, run + c0 + c1, run + c0 + c1 + c2);
    if (threadIdx.x == 255) blocksum[blockIdx.x] = run + s;
}

// 4. each record into its group.  Lanes of a warp that share a group are reduced first, so that many
// records of one group do not queue on its atomics one by one.
template <int LITE>
__global__ void __launch_bounds__(256) k_merge_fold(const uint32_t* in, const unsigned long long* key, long long n,
                                                    const PhxMergeRange* range, unsigned long long most, const uint32_t* cell,
                                                    const uint32_t* off, const uint32_t* blocksum, unsigned long long* amin,
                                                    uint32_t* pmin, uint32_t* gor, uint32_t* gsum)
{
    const PhxMergeMap m = phx_merge_map(*range);
    if (m.cells == 0ull || m.cells > most) return;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += stride) {
        const long long j = base + lane;
        const unsigned long long k = j < n ? key[j] : PHX_MERGE_NONE;
        const bool ok = k != PHX_MERGE_NONE;
        uint32_t g = 0xffffffffu, tb = 0xffffffffu, fl = 0u, hc = 0u, pos = (uint32_t)j;
        if (ok) {
            const uint32_t c = phx_merge_cell(m, k), w = c >> 5;
            g = blocksum[w >> 10] + off[w] + __popc(cell[w] & ((1u << (c & 31u)) - 1u));
            const uint32_t* r = in + j * PhxRec<LITE>::W;
            tb = phx_time_order(r[PhxRec<LITE>::TIME]);
            fl = r[PhxRec<LITE>::FLAG];
            hc = r[PhxRec<LITE>::HC] >> 16;
        }
        if (!__any_sync(FULL, ok)) continue;
        const uint32_t peers = __match_any_sync(FULL, g);
        bool lead = ok;
        uint32_t pfirst = pos, pm = pos;
        if (__any_sync(FULL, ok && (peers & (peers - 1u)) != 0u)) {
            const uint32_t tmin = __reduce_min_sync(peers, tb);
            pfirst = __reduce_min_sync(peers, tb == tmin ? pos : 0xffffffffu);
            pm = __reduce_min_sync(peers, pos);
            fl = __reduce_or_sync(peers, fl);
            hc = __reduce_add_sync(peers, hc);
            tb = tmin;
            lead = ok && __ffs(peers) - 1 == lane;
        }
        if (lead) {
            atomicMin(amin + g, ((unsigned long long)tb << 32) | (unsigned long long)pfirst);
            if (LITE) atomicMin(pmin + g, pm);
            atomicOr(gor + g, fl);
            atomicAdd(gsum + g, hc);
        }
    }
}

// 5. representative record per group with the reduced fields, a 16 B row a thread
template <int LITE>
__global__ void __launch_bounds__(256) k_merge_groups(const uint32_t* in, const PhxMergeRange* range, unsigned long long most,
                                                      long long cap, const unsigned long long* amin, const uint32_t* pmin,
                                                      const uint32_t* gor, const uint32_t* gsum, uint32_t* out)
{
    constexpr int Q = PhxRec<LITE>::W / 4;
    const long long ng = range->groups;
    if (phx_merge_map(*range).cells > most || ng > cap) return;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x; x < ng * Q; x += stride) {
        const long long g = x / Q;
        const int q = (int)(x - g * Q);
        const unsigned long long a = amin[g];
        const long long i = LITE ? (long long)pmin[g] : (long long)(a & 0xffffffffull);
        uint32_t r[4];
        for (int w = 0; w < 4; w++) r[w] = in[i * PhxRec<LITE>::W + 4 * q + w];
        if (LITE) r[PhxRec<LITE>::TIME & 3] = phx_time_unorder((uint32_t)(a >> 32));
        if (q == PhxRec<LITE>::FLAG / 4) r[PhxRec<LITE>::FLAG & 3] = gor[g];
        if (q == PhxRec<LITE>::HC / 4) r[PhxRec<LITE>::HC & 3] = (r[PhxRec<LITE>::HC & 3] & 0xffffu) | ((gsum[g] & 0xffffu) << 16);
        for (int w = 0; w < 4; w++) out[x * 4 + w] = r[w];
    }
}

// ---------------------------------------------------------------- sort form
// record i is selected: by its key, where step 1 of the table form left one, or by its flags
template <int LITE>
__device__ __forceinline__ bool phx_merge_selected(const uint32_t* in, const unsigned long long* key, long long i, uint32_t mask)
{
    return key ? key[i] != PHX_MERGE_NONE : (in[i * PhxRec<LITE>::W + PhxRec<LITE>::FLAG] & mask) != 0u;
}

// 1a. per-tile selected counts
template <int LITE>
__global__ void __launch_bounds__(256) k_merge_sel_count(const uint32_t* in, const unsigned long long* key, long long n, uint32_t mask,
                                                          uint32_t* tcount)
{
    __shared__ uint32_t wsum[8];
    const long long tile = (long long)blockIdx.x * PHX_MERGE_TILE;
    uint32_t c = 0;
    for (int r = 0; r < PHX_MERGE_TILE_ITEMS; r++) {
        const long long i = tile + (long long)r * 256 + threadIdx.x;
        if (i < n) c += phx_merge_selected<LITE>(in, key, i, mask);
    }
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t s = 0;
        for (int k = 0; k < 8; k++) s += wsum[k];
        tcount[blockIdx.x] = s;
    }
}

// 1b. ordered write of selected positions, and of their keys where there are any (tile offsets already scanned)
template <int LITE>
__global__ void __launch_bounds__(256) k_merge_sel_write(const uint32_t* in, const unsigned long long* key, long long n, uint32_t mask,
                                                          const uint32_t* toff, uint32_t* sel, unsigned long long* sel_key)
{
    __shared__ uint32_t wsum[8];
    __shared__ uint32_t base;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) base = toff[blockIdx.x];
    __syncthreads();
    const long long tile = (long long)blockIdx.x * PHX_MERGE_TILE;
    for (int r = 0; r < PHX_MERGE_TILE_ITEMS; r++) {
        const long long i = tile + (long long)r * 256 + threadIdx.x;
        const bool s = i < n && phx_merge_selected<LITE>(in, key, i, mask);
        const uint32_t b = __ballot_sync(0xffffffffu, s);
        if (lane == 0) wsum[w] = __popc(b);
        __syncthreads();
        uint32_t before = base;
        for (int k = 0; k < w; k++) before += wsum[k];
        if (s) {
            const uint32_t p = before + __popc(b & ((1u << lane) - 1u));
            sel[p] = (uint32_t)i;
            if (sel_key) sel_key[p] = key[i];
        }
        __syncthreads();
        if (threadIdx.x == 0) { uint32_t t = 0; for (int k = 0; k < 8; k++) t += wsum[k]; base += t; }
        __syncthreads();
    }
}

// selection only (window 0): gather selected records in order
template <int LITE>
__global__ void k_merge_gather(const uint32_t* in, const uint32_t* sel, long long m, uint32_t* out)
{
    constexpr int W = PhxRec<LITE>::W;
    const long long total = m * W;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += (long long)gridDim.x * blockDim.x) {
        const long long j = k / W;
        const int w = (int)(k - j * W);
        const long long i = sel ? (long long)sel[j] : j;
        out[k] = in[i * W + w];
    }
}

// 2. keys of the selected records, where there is no room for the table form and so none yet
template <int LITE>
__global__ void k_merge_keys(const uint32_t* in, const uint32_t* sel, long long m, float tw, unsigned long long* key)
{
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < m; j += (long long)gridDim.x * blockDim.x) {
        const long long i = sel ? (long long)sel[j] : j;
        key[j] = phx_merge_key<LITE>(in + i * PhxRec<LITE>::W, tw);
    }
}

// 3a. digit histogram per tile, digit-major: hist[d * ntile + tile]
__global__ void __launch_bounds__(256) k_radix_hist(const unsigned long long* key, long long m, int shift, uint32_t* hist, int ntile)
{
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0u;
    __syncthreads();
    const long long tile = (long long)blockIdx.x * PHX_MERGE_TILE;
    for (int r = 0; r < PHX_MERGE_TILE_ITEMS; r++) {
        const long long j = tile + (long long)r * 256 + threadIdx.x;
        if (j < m) atomicAdd(&h[(uint32_t)(key[j] >> shift) & 0xffu], 1u);
    }
    __syncthreads();
    hist[(size_t)threadIdx.x * ntile + blockIdx.x] = h[threadIdx.x];
}

// 3b. stable scatter: equal digits ranked by (round, warp, lane), i.e. by position in the tile (vin null: the
// values are the positions)
__global__ void __launch_bounds__(256) k_radix_scatter(const unsigned long long* kin, const uint32_t* vin, unsigned long long* kout,
                                                       uint32_t* vout, long long m, int shift, const uint32_t* off, int ntile)
{
    __shared__ uint32_t base[256];
    __shared__ uint32_t wcnt[8][256];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    base[t] = off[(size_t)t * ntile + blockIdx.x];
    const long long tile = (long long)blockIdx.x * PHX_MERGE_TILE;
    for (int r = 0; r < PHX_MERGE_TILE_ITEMS; r++) {
        for (int q = 0; q < 8; q++) wcnt[q][t] = 0u;
        __syncthreads();
        const long long j = tile + (long long)r * 256 + t;
        const bool ok = j < m;
        const unsigned long long k = ok ? kin[j] : 0ull;
        const uint32_t v = !ok ? 0u : vin ? vin[j] : (uint32_t)j;
        const uint32_t d = ok ? ((uint32_t)(k >> shift) & 0xffu) : 0x100u;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
        if (ok && rank == 0u) wcnt[w][d] = __popc(peers);
        __syncthreads();
        {
            uint32_t run = base[t];
            for (int q = 0; q < 8; q++) { const uint32_t c = wcnt[q][t]; wcnt[q][t] = run; run += c; }
            base[t] = run;
        }
        __syncthreads();
        if (ok) {
            const uint32_t p = wcnt[w][d] + rank;
            kout[p] = k;
            vout[p] = v;
        }
        __syncthreads();
    }
}

// exclusive scan of u32 in tiles of 1024 (256 threads x 4): local scan + tile sums
__global__ void __launch_bounds__(256) k_scan_tile(uint32_t* x, long long n, uint32_t* tsum)
{
    __shared__ uint32_t wt[8];
    const long long b = (long long)blockIdx.x * PHX_MERGE_SCAN_TILE + (long long)threadIdx.x * 4;
    uint32_t v[4], s = 0;
    for (int k = 0; k < 4; k++) { v[k] = (b + k < n) ? x[b + k] : 0u; s += v[k]; }
    uint32_t inc = s;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) { const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += y; }
    if (lane == 31) wt[wid] = inc;
    __syncthreads();
    uint32_t before = 0;
    for (int k = 0; k < wid; k++) before += wt[k];
    uint32_t run = before + inc - s;
    for (int k = 0; k < 4; k++) { if (b + k < n) x[b + k] = run; run += v[k]; }
    if (threadIdx.x == 255) tsum[blockIdx.x] = before + inc;
}
__global__ void k_scan_add(uint32_t* x, long long n, const uint32_t* tsum)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] += tsum[i / PHX_MERGE_SCAN_TILE];
}

template <int LITE>
__global__ void k_merge_clear(long long ng, unsigned long long* amin, uint32_t* pmin, uint32_t* gor, uint32_t* gsum)
{
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g < ng) phx_merge_clear<LITE>(g, amin, pmin, gor, gsum);
}

// 4a. group heads
__global__ void k_merge_heads(const unsigned long long* key, long long m, uint32_t* head)
{
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < m) head[j] = (j == 0 || key[j] != key[j - 1]) ? 1u : 0u;
}

// 4b. warp-segmented reduction per group, one atomic per (warp, group); val: input positions (null: 0, 1, ...)
template <int LITE>
__global__ void k_merge_reduce(const uint32_t* in, const unsigned long long* key, const uint32_t* val, const uint32_t* gexcl,
                               long long m, unsigned long long* amin, uint32_t* pmin, uint32_t* gor, uint32_t* gsum)
{
    const int lane = threadIdx.x & 31;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < m; base += stride) {
        const long long j = base + lane;
        const bool ok = j < m;
        uint32_t g = 0xffffffffu, pos = 0xffffffffu, tb = 0xffffffffu, fl = 0u, hc = 0u;
        if (ok) {
            const uint32_t head = (j == 0 || key[j] != key[j - 1]) ? 1u : 0u;
            g = gexcl[j] + head - 1u;
            pos = val ? val[j] : (uint32_t)j;
            const uint32_t* r = in + (long long)pos * PhxRec<LITE>::W;
            tb = phx_time_order(r[PhxRec<LITE>::TIME]);
            fl = r[PhxRec<LITE>::FLAG];
            hc = r[PhxRec<LITE>::HC] >> 16;
        }
        const uint32_t peers = __match_any_sync(0xffffffffu, g);
        const uint32_t tmin = __reduce_min_sync(peers, tb);
        const uint32_t pfirst = __reduce_min_sync(peers, tb == tmin ? pos : 0xffffffffu);
        const uint32_t pm = __reduce_min_sync(peers, pos);
        const uint32_t fo = __reduce_or_sync(peers, fl);
        const uint32_t hs = __reduce_add_sync(peers, hc);
        if (ok && (__ffs(peers) - 1) == lane) {
            atomicMin(amin + g, ((unsigned long long)tmin << 32) | (unsigned long long)pfirst);
            if (LITE) atomicMin(pmin + g, pm);
            atomicOr(gor + g, fo);
            atomicAdd(gsum + g, hs);
        }
    }
}

// 5. representative record per group with the reduced fields
template <int LITE>
__global__ void k_merge_write(const uint32_t* in, long long ng, const unsigned long long* amin, const uint32_t* pmin,
                              const uint32_t* gor, const uint32_t* gsum, uint32_t* out)
{
    constexpr int W = PhxRec<LITE>::W;
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ng) return;
    const long long i = LITE ? (long long)pmin[g] : (long long)(amin[g] & 0xffffffffull);
    uint32_t r[W];
    for (int w = 0; w < W; w++) r[w] = in[i * W + w];
    if (LITE) r[PhxRec<LITE>::TIME] = phx_time_unorder((uint32_t)(amin[g] >> 32));
    r[PhxRec<LITE>::FLAG] = gor[g];
    r[PhxRec<LITE>::HC] = (r[PhxRec<LITE>::HC] & 0xffffu) | ((gsum[g] & 0xffffu) << 16);
    for (int w = 0; w < W; w++) out[g * W + w] = r[w];
}
