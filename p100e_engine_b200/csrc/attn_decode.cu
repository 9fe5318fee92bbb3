// Split-KV decode / MTP-verify attention over the paged f16 / q8_0 / q4_0 cache, sm_100a.
//
// Work unit = (slot, kv head, key chunk): one CTA of 4 warps walks its chunk in 64-key tiles; four CTAs per SM for three row
// tiles (q_len 3..4), five for two, six for one (q_len 1), two for f16 caches.
//   staging   the K rows and the V rows of a tile (one kv head, 64 positions) are each fetched by ONE tiled TMA copy through a
//             tensor map of the cache (x = row bytes, y = position in page, z = page) into a ring of half-tile slots,
//             completion counted on mbarriers; rows keep their cache format in shared memory.  The warp that is last to
//             finish with a slot issues its refill.  f16 rows go through a rank-4 map with the 128-byte swizzle.  What a
//             ragged last tile holds past the last key is masked; pages under 64 rows are staged row by row through registers instead.
//   QK^T      warp w owns keys 16w..16w+15 of the tile: keys on the MMA M axis, the slot's 6 * q_len query rows on N
//             (all GQA heads and verify rows share one pass over the KV bytes).  int8 / nibbles are widened to f16
//             exactly in registers (byte permute + one f16x2 subtract), products accumulate in fp32 on the tensor
//             cores (mma.sync m16n8k16), the per-32 block scale multiplies the fp32 partial sums.
//   softmax   online, per row, base 2, against a reference maximum that all warps share and that may trail the true
//             maximum by 2^7: a tile whose scores stay under it needs one block barrier (P to shared memory as f16, then
//             P V); only a tile that outgrows it makes the warps exchange maxima, redo P and rescale O.
//   PV        warp w owns output dims 64w..64w+63: V^T tiles on M, rows on N, fp32 accumulators in registers.
//   partials  each unit writes unnormalised (O, m, l); a merge kernel combines a row's chunks in a fixed order, applies
//             the optional sigmoid gate and normalises (reference formula: dec2_combine_k, src/fast/attn_dec2.cu:430-450).
// The chunk grid is fixed by absolute key index, and a chunk's arithmetic never depends on the other rows of the call:
// a row's result is a function of its own keys and of chunk_keys only (row t of a T-row call == the 1-row call).
//
// Batched calls of several slots that let the library choose the split (chunk_keys < 0) cut the batch evenly over the CTAs that fit the GPU
// (decode_split_k; one plan per model step when the caller declares the step, b200_attn_step_begin).  There q8_0 caches
// with two to four rows per slot run on a second kernel, decode_tc_k (decode_tc.cuh): tcgen05 MMAs with K in tensor
// memory and V as an f16 image in shared memory, one CTA per SM (one slot of such rows too); q8_0 with one row per slot and q4_0 with one or
// two on a third, decode_warp_k (decode_warp.cuh).  Everything else, and every fixed-chunk call, runs on the kernel described above.
//
// Reference counterpart: dec2_k / attn_decode2 (src/fast/attn_dec2.cu:210-530), fp32 FFMA on sm_60.
#include "umma.cuh"

#include <dlfcn.h>
#include <cuda.h>   // CUtensorMap and its enums only: the encoder is looked up at run time, nothing links against libcuda
#include <algorithm>
#include <atomic>
#include <cstring>
#include <cstdlib>
#include <mutex>

namespace b200 {
namespace {

constexpr int TILE = 64;              // keys per tile
constexpr int NWARP = 4, NTHR = NWARP * 32;
constexpr int PGS = 64;               // page-table entries of a chunk kept in shared memory
constexpr int HDR = 1024;             // shared-memory header: barriers, counters, page entries; the slots start 1024-aligned
#ifndef DEC_CTAS
#define DEC_CTAS 4
#endif
constexpr int CTAS_Q = DEC_CTAS;      // CTAs per SM the quantised kernels are compiled for (register budget 65536 / (128 * CTAS_Q))
// fewer query rows need fewer accumulator registers: one row tile (q_len 1) runs six CTAs per SM, two run five
template <uint32_t KT, int NT> constexpr int ctas_per_sm() { return KT == B200_KV_F16 ? 2 : NT == 1 ? CTAS_Q + 2 : NT == 2 ? CTAS_Q + 1 : CTAS_Q; }
constexpr int QSTR = 576;             // bytes per Q row in shared memory (256 f16 + 64: rows g, g+1 on different bank halves)
constexpr int PSTR = 144;             // bytes per P row (64 f16 + 16)
constexpr int SDSTR = 132;            // bytes per V-scale row (64 f16 + 4)
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;
constexpr float PSHIFT = 8.0f;        // P (and l) are kept times 2^8 inside the kernels
constexpr float REF_GAP = 7.0f;       // a row's reference maximum may trail its true maximum by this much (log2 units)

template <uint32_t KT> struct traits {
    static constexpr int HB = head_bytes(KT);                       // bytes of a head row in the cache
    static constexpr int SROW = HB;                                 // bytes per key row in shared memory
    static constexpr int SLOT = TILE * SROW;                        // one ring slot: the K rows or the V rows of a tile
    static constexpr bool SCALED = KT != B200_KV_F16;
};
// Verify calls on quantised caches (two or three row tiles) keep 32 or 48 output accumulators per thread, which are idle
// during Q K^T and the softmax: there they are parked in tensor memory (tcgen05.st / tcgen05.ld, this warp's own 32 lanes),
// so the compiler has those registers for loads in flight.  PARK_COLS columns are allocated per CTA.
#ifndef DEC_PARK
#define DEC_PARK 1
#endif

template <uint32_t KT, int NT> constexpr bool parks() { return DEC_PARK && KT != B200_KV_F16 && NT >= 2; }
constexpr uint32_t PARK_COLS = 64;

// f16 slots hold four sub-tiles [64 rows][128 B] (dims 64 c .. 64 c + 63) with the 128-byte swizzle of the TMA unit: the
// 16-byte chunk j of a sub-tile row sits at chunk j ^ (row & 7), which keeps 16-byte and ldmatrix accesses of eight
// different rows on different banks.  chunk16 = 16-byte chunk of the 512-byte head row.
__device__ __forceinline__ int f16_slot_off(int row, int chunk16) {
    return (chunk16 >> 3) * (TILE * 128) + row * 128 + (((chunk16 & 7) ^ (row & 7)) << 4);
}

// M-row (0..7) -> key of the warp's 16-key group, chosen so that the A-fragment loads of a phase hit distinct banks
template <uint32_t KT> __device__ __forceinline__ int key_perm(int g) {
    if constexpr (KT == B200_KV_F16) return (g >> 1) + 4 * (g & 1);       // 16-byte loads: lanes of a phase 4 keys apart
    else if constexpr (KT == B200_KV_Q8_0) return 2 * (g & 3) + (g >> 2); // 8-byte loads: 2 keys apart
    else return g;
}
// position of head dim d inside the shared-memory Q row, so that lane t of a quad reads dims of block b for both
// k-steps of the block with one 16-byte load at 64 b + 16 t
template <uint32_t KT> __device__ __forceinline__ int q_slot(int d) {
    if constexpr (KT == B200_KV_Q4_0) {
        const int b = d >> 5, i = d & 31;          // nibble order: byte j = dims j | j + 16
        return b * 32 + ((i & 15) >> 2) * 8 + (i >> 4) * 4 + (i & 3);
    } else return d;
}

// Chunk grids of the fixed-chunk modes, by absolute key index.  CH > 0: chunks of CH keys.  CH <= 0, the grid of the row entry
// points (position_grid): 64 keys up to position 4096, then 32 chunks per doubling (128 keys from 4096, 256 from 8192, ..) up to chunks of 64 << -CH keys.  A short context
// is cut finely enough to fill the chip whatever the cache's capacity, and a long one into little more than one wave of equal units.
// One row, q8_0, 4 kv heads: chunks of 512 keys everywhere take 22.3 / 24.8 / 69.1 us at 4096 / 16384 / 131072 keys, of 64 keys
// 12.7 / 24.8 / 124.1 us.
__host__ __device__ __forceinline__ int chunk_of(int CH, int p) {
    if (CH > 0) return p / CH;
    int k = 0;
    while (k < -CH && (p >> (12 + k)) != 0) ++k;
    return 32 * k + (p >> (6 + k));
}
__host__ __device__ __forceinline__ long long chunk_lo(int CH, int c) {
    if (CH > 0) return (long long) c * CH;
    const int k = c < 64 ? 0 : (c >> 5) - 1 < -CH ? (c >> 5) - 1 : -CH;
    return (long long) (c - 32 * k) << (6 + k);
}

struct dec_args {
    const float * q;
    kv_view g;
    float * po; float * pm; float * pl;   // partials [unit][R][256], [unit][R], [unit][R]
    const int32_t * pos;                  // per-row positions (device) or nullptr
    const int32_t * p0p;                  // device first position or nullptr
    int p0;
    int q_len, n_slots, Hq;
    float qscale;                         // softmax scale * log2(e)
    int CH, max_chunks;                   // chunk grid (chunk_of / chunk_lo); chunks of the longest slot
    int hk0, nhk;                         // kv heads of this launch: hk0 .. hk0 + nhk - 1 (all of them but in the allocation-free entry)
    unsigned * status;
    int n_ctx;                            // rows of a contiguous cache
    int tiled;                            // set by the launcher: whole tiles are fetched through the tensor maps
    int chunked;                          // fixed chunks: every chunk of the grid leaves its own partial
    // run plan (decode_split_k): the batch's 64-key tiles, slot after slot, are cut into one contiguous run per CTA; nullptr = fixed
    // chunks without a plan (one slot, or few units: see decode_part_k)
    const int4 * segs;                    // (slot, first key, end key, 0) in CTA order; a run that crosses a slot boundary has several
    const int * cta_seg;                  // [n_cta + 1] first segment of each CTA
    const int2 * slot_seg;                // [n_slots] (first segment, segments) of each slot
    int max_cta;                          // runs per kv head that a plan may hold
    int solo;                             // > 0: one slot in even runs without a plan (solo_runs), at most so many
    const int * n_cta;                    // CTAs (per kv head) that hold work; < 0: -n_cta segments, CTA c takes c, c + CTAs of the head, ..
};

// keys of a slot that the call may touch: 1 + its largest row position, held to the caller's max_n (the grid and the
// partials are sized for max_chunks chunks) and to n_ctx for a contiguous cache.  A position beyond the limit is recorded
// in the status word and its keys past the limit are left out.
__device__ __forceinline__ int key_limit(const dec_args & a) {
    const long long lim = chunk_lo(a.CH, a.max_chunks);
    const int l = (int) (lim < 0x7fffffffLL ? lim : 0x7fffffffLL);
    return a.g.pt ? l : min(l, a.n_ctx);
}

__device__ __forceinline__ int row_pos(const dec_args & a, int slot, int j);

// One slot in an even split: its 64-key tiles (returned) in `runs` runs per kv head, of two tiles (decode_tc_k walks pairs) where there are so few; run c takes tiles [c W / runs, (c + 1) W / runs).  The
// decode kernel and the merge find this by themselves: a plan kernel would cost the call 3 us.  Called by whole warps.
__device__ __forceinline__ int solo_runs(const dec_args & a, int & runs) {
    const int lane = threadIdx.x & 31, n = __reduce_max_sync(0xffffffffu, lane < a.q_len ? row_pos(a, 0, lane) : -1) + 1;
    const int W = (max(0, min(n, key_limit(a))) + TILE - 1) / TILE;
    runs = min(a.solo, (W + 1) / 2);
    return W;
}

// One tiled copy (TMA unit) of a box of a rank-3 tensor into shared memory, completion counted in bytes on an mbarrier.
// x is in 16-bit elements and x * 2 must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_box3(void * dst, const CUtensorMap * map, int x, int y, int z, uint64_t * bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ int row_pos(const dec_args & a, int slot, int j) {
    const int r = slot * a.q_len + j;
    if (a.pos) return a.pos[r];
    return (a.p0p ? *a.p0p : a.p0) + r;
}

// two int8 (already offset by 128) at bytes (2 * HI, 2 * HI + 1) of u -> f16x2
template <int HI> __device__ __forceinline__ uint32_t cvt_i8x2(uint32_t u) {
    return hsub2_u32(__byte_perm(u, 0x64646464u, HI ? 0x7362 : 0x5140), 0x64806480u);
}
// bytes holding values 0..15 (+8 bias) at bytes (2 * HI, 2 * HI + 1) -> f16x2 of (value - 8)
template <int HI> __device__ __forceinline__ uint32_t cvt_n4x2(uint32_t u) {
    return hsub2_u32(__byte_perm(u, 0x64646464u, HI ? 0x7362 : 0x5140), 0x64086408u);
}

__device__ __forceinline__ void tma_box4(void * dst, const CUtensorMap * map, int x, int y, int z, int w, uint64_t * bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar)) : "memory");
}

// One unit of work: the keys k_lo .. k_cap-1 (as far as the slot has them) of one slot and kv head, all its query rows; writes
// the unnormalised partial (O, m, l) number `unit`, or with RUNS (planned runs of fixed chunks) one partial per chunk, unit,
// unit + 1, ..: sums and references start afresh at every chunk, so a chunk's bits do not depend on where a unit begins or
// ends. Called by all threads of the CTA.  A CTA that runs several units keeps its ring of copy slots, their barriers and the
// arrival counters going from one unit to the next: tiles_before is the number of tiles its earlier units walked (two ring
// items each); the function returns this unit's tile count. t_slot: where the tensor-memory base of the parked accumulators is written.
template <uint32_t KT, int NT, bool RUNS>
__device__ __forceinline__ int decode_unit(const dec_args & a, const int nslot, const CUtensorMap & mapK, const CUtensorMap & mapV,
                                           unsigned char * smem, const int hk, const int slot, const int k_lo, const int k_cap,
                                           unsigned unit, const int tiles_before, const uint32_t * t_slot) {
    using TR = traits<KT>;
    constexpr int HB = TR::HB, SROW = TR::SROW;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
    const int R = a.q_len * GQA;

    // What the unit reads before its first copy is asked for at once, the positions (lane j: row j), the query rows (this thread's share, in
    // registers) and the place of the page table; the start of a unit is a chain of such loads, and with one tile per CTA most of the kernel's time.
    const int posv = lane < a.q_len ? row_pos(a, slot, lane) : -1;
    const int rt = a.g.pt && a.g.rtab ? a.g.rtab[slot * a.q_len] : 0;
    constexpr int QN = NT * 8 * (DH / 4) / NTHR;
    float4 qv[QN];
#pragma unroll
    for (int k = 0; k < QN; ++k) {
        const int i = tid + k * NTHR, r = i / (DH / 4), d4 = (i - r * (DH / 4)) * 4, j = r / GQA, hh = r - j * GQA;
        qv[k] = r < R ? *reinterpret_cast<const float4 *>(a.q + ((size_t) (slot * a.q_len + j) * a.Hq + hk * GQA + hh) * DH + d4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    // visible keys of the slot = 1 + the largest row position
    int n_slot = __reduce_max_sync(0xffffffffu, posv) + 1;
    const int rmin = __reduce_min_sync(0xffffffffu, lane < a.q_len ? posv : 0x7fffffff);
    {
        const int lim = key_limit(a);
        if (n_slot > lim) { if (tid == 0) atomicOr(a.status, ST_BAD_POS); n_slot = lim; }
    }
    if (k_lo >= n_slot) return 0;
    const int k_hi = min(k_cap, n_slot);
    const int ntiles = (k_hi - k_lo + TILE - 1) / TILE;
    const int ring0 = (2 * tiles_before) % nslot;                       // ring slot of this unit's first item
    const uint32_t ring0_par = (uint32_t) ((2 * tiles_before) / nslot) & 1u;   // and the parity of that slot's use count

    // shared memory carve-up
    uint64_t * full = reinterpret_cast<uint64_t *>(smem);                    // [nslot]
    int * done = reinterpret_cast<int *>(smem + 96);                         // warps that finished Q K^T / P V (two counters)
    int * flag = reinterpret_cast<int *>(smem + 104);                        // [3] "some warp's scores outgrew the references"
    int * pgs = reinterpret_cast<int *>(smem + 128);                         // [PGS] page-table entries of the chunk's pages
    unsigned char * stg = smem + HDR;                                        // nslot * SLOT
    unsigned char * Qs = stg + (size_t) nslot * TR::SLOT;                    // [NT*8][QSTR]
    unsigned char * Ps = Qs + NT * 8 * QSTR;                                 // [NT*8][PSTR]
    unsigned char * Sd = Ps + NT * 8 * PSTR;                                 // [8][SDSTR]  V block scales, transposed
    float * wmax = reinterpret_cast<float *>(Sd + 8 * SDSTR);                // [NWARP][NT*8]
    float * wl = wmax + NWARP * NT * 8;                                      // [NWARP][NT*8]
    float4 * Qb = reinterpret_cast<float4 *>(wl + NWARP * NT * 8);           // [NBLK][NT][4] block sums of Q (quantised caches)

    const int32_t * tab = a.g.pt ? a.g.pt + rt : nullptr;
    const unsigned long long hoff = (unsigned long long) hk * HB;
    // the chunk's page-table entries are staged in shared memory when there are at most PGS of them, so that a refill does
    // not wait for a global load
    const int pg0 = tab ? k_lo >> a.g.psh : 0;
    const bool pg_staged = tab && ((k_hi - 1) >> a.g.psh) - pg0 < PGS;

    // staging: the K rows and the V rows of the tiles form one sequence q = 2 * tile (K), 2 * tile + 1 (V) that walks a ring
    // of nslot half-tile slots.  The warp that is last to finish the Q K^T (P V) of a tile refills that tile's K (V) slot with
    // item q + nslot, so a copy is in flight while the other half of the tile is being computed.  A tile is one tiled
    // copy through the cache's tensor map (box = 64 rows of this head, inside one page), a slot's last, ragged tile too: what lies
    // past its last key (stale rows of the page; zeros past the end of a contiguous cache) is masked in the softmax and
    // enters P V as zeros.  One warp moving that tile row by row held its CTA for 30 us (q8_0) to 60 us (f16), longer than everything
    // else in a call of 30011 keys (50.2 us in all).  Caches without a tensor map (small pages) are still moved that way, rows past the slot's
    // last key replaced by that key.
    // page entries of the first copies: lane q that of item q
    const int pg_first = w == 0 && tab && lane < nslot && lane < 2 * ntiles ? tab[(k_lo + (lane >> 1) * TILE) >> a.g.psh] : 0;
    auto page_of = [&](int p) { return pg_staged ? pgs[(p >> a.g.psh) - pg0] : tab[p >> a.g.psh]; };
    auto issue = [&](int q, int s, bool first) {   // s = q mod nslot; called by one whole warp
        const int zf = first ? __shfl_sync(0xffffffffu, pg_first, q) : 0;
        if (q >= 2 * ntiles) return;
        const int it = q >> 1;
        unsigned char * dst = stg + (size_t) s * TR::SLOT;
        const char * base = (q & 1) ? a.g.v : a.g.k;
        const int p_t = k_lo + it * TILE;
        if (a.tiled) {
            if (lane == 0) {
                int y = p_t, z = 0;
                if (tab) {
                    z = first ? zf : page_of(p_t);
                    y = p_t & ((1 << a.g.psh) - 1);
                    if (z < 0) { atomicOr(a.status, ST_BAD_PAGE); z = 0; }
                }
                mbar_expect_tx(&full[s], (uint32_t) TILE * HB);
                if constexpr (KT == B200_KV_F16) tma_box4(dst, (q & 1) ? &mapV : &mapK, 0, y, 4 * hk, z, &full[s]);
                else tma_box3(dst, (q & 1) ? &mapV : &mapK, hk * (HB / 2), y, z, &full[s]);
            }
            __syncwarp();
            return;
        }
        // row by row through registers, 16 bytes per lane and step; the slot is published by a plain arrival
        constexpr int CPR = HB / 16;
#pragma unroll 4
        for (int idx = lane; idx < TILE * CPR; idx += 32) {
            const int row = idx / CPR, c = idx - row * CPR;
            const int p = min(p_t + row, n_slot - 1);
            unsigned long long off;
            if (tab) {
                const int pg = first ? tab[p >> a.g.psh] : page_of(p);
                if (pg < 0) { atomicOr(a.status, ST_BAD_PAGE); off = 0; }
                else off = (unsigned long long) pg * a.g.pstride + (unsigned long long) (p & ((1 << a.g.psh) - 1)) * a.g.rowb;
            } else off = (unsigned long long) p * a.g.rowb;
            const uint4 v = __ldg(reinterpret_cast<const uint4 *>(base + off + hoff) + c);
            const int o = KT == B200_KV_F16 ? f16_slot_off(row, c) : row * SROW + c * 16;
            *reinterpret_cast<uint4 *>(dst + o) = v;
        }
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full[s])) : "memory");
    };
    // warp 0 starts the first copies before anything else, so that they fly while Q is staged
    if (w == 0) {   // every slot is free at the start of a unit: all items of the earlier units have been consumed
        int s = ring0;
        for (int q0 = 0; q0 < nslot; ++q0) {
            issue(q0, s, true);
            if (++s == nslot) s = 0;
        }
    }
    constexpr bool PARK = parks<KT, NT>();
    if (pg_staged)
        for (int j = tid; j <= ((k_hi - 1) >> a.g.psh) - pg0; j += NTHR) pgs[j] = tab[pg0 + j];
    // Q rows -> shared memory as f16, scaled; row r = j * 6 + hh (verify row j, head hh of the group).  For the quantised
    // caches the middle two of every four dims are swapped (d0 d2 d1 d3): a 32-bit word of cache bytes then splits into the
    // f16 pairs (byte 0, byte 2) and (byte 1, byte 3) with one mask and one byte permute (see the Q K^T loop).
    // The cache integers enter the tensor cores as f16 subnormals u * 2^-24 with u = q + 128 (q8_0) or the nibble itself
    // (q4_0, value = nibble - 8).  The offset is taken out again through the accumulator's starting value: for block b and
    // row r it is -OFFS * 2^-24 * (sum of the block's 32 scaled f16 query values, which eight neighbouring lanes hold), kept per (block, row tile,
    // lane quad position) in the order of an accumulator fragment {row 2t, row 2t+1, row 2t, row 2t+1}.
#pragma unroll
    for (int k = 0; k < QN; ++k) {
        const int i = tid + k * NTHR, r = i / (DH / 4), d4 = (i - r * (DH / 4)) * 4;
        const float4 v = qv[k];
        // four consecutive dims stay together under q_slot (it permutes groups of four): one 8-byte store
        uint2 pk;
        if constexpr (TR::SCALED) pk = make_uint2(pack_h2(v.x * a.qscale, v.z * a.qscale), pack_h2(v.y * a.qscale, v.w * a.qscale));
        else pk = make_uint2(pack_h2(v.x * a.qscale, v.y * a.qscale), pack_h2(v.z * a.qscale, v.w * a.qscale));
        *reinterpret_cast<uint2 *>(Qs + r * QSTR + q_slot<KT>(d4) * 2) = pk;
        if constexpr (TR::SCALED) {
            constexpr float OFFS = KT == B200_KV_Q8_0 ? 128.0f : 8.0f;
            const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&pk.x)), hi = __half22float2(*reinterpret_cast<const __half2 *>(&pk.y));
            float sum = (lo.x + lo.y) + (hi.x + hi.y);
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            sum += __shfl_xor_sync(0xffffffffu, sum, 4);
            if ((lane & 7) == 0) {
                const int b = d4 >> 5;
                const float x = -OFFS * 5.9604644775390625e-8f * sum;
                float * dst = reinterpret_cast<float *>(Qb + (b * NT + (r >> 3)) * 4 + ((r & 7) >> 1));
                dst[r & 1] = x; dst[2 + (r & 1)] = x;
            }
        }
    }
    if constexpr (parks<KT, NT>()) umma::fence_before_sync();
    __syncthreads();
    if constexpr (parks<KT, NT>()) umma::fence_after_sync();
    const uint32_t t_base = parks<KT, NT>() ? *t_slot : 0u;

    // arrive(c): this warp is done with the K (c = 0) or V (c = 1) item of the tile; lane 0 learns whether it was the last of
    // the four warps.  refill_if_last: that warp refills the slot.  The two are apart in the instruction stream so that the
    // round trip of the shared-memory atomic is covered by other work.
    auto arrive = [&](int c) {
        asm volatile("" ::: "memory");   // the item's shared-memory reads stay above this point
        int last = 0;
        if (lane == 0) last = (atomicAdd(&done[c], 1) & (NWARP - 1)) == NWARP - 1;
        return last;
    };
    auto refill_if_last = [&](int last, int q, int s) {
        if (__shfl_sync(0xffffffffu, last, 0)) issue(q + nslot, s, false);
    };

    // per-lane row bookkeeping: this lane's score / output columns are rows 8i + 2t and 8i + 2t + 1
    int rpos[NT][2];
    float m_run[NT][2], l_run[NT][2];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int r = 8 * i + 2 * t + e;
            const int pr = __shfl_sync(0xffffffffu, posv, min(r / GQA, 31));
            rpos[i][e] = r < R ? pr : -1;
            m_run[i][e] = B200_NEG_INF;
            l_run[i][e] = 0.0f;
        }
    float O[4][NT][4];
#pragma unroll
    for (int mt = 0; mt < 4; ++mt)
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) O[mt][i][e] = 0.0f;
    // parked accumulators: 16 * NT columns of this warp's 32 tensor-memory lanes
    uint32_t t_O = 0;
    auto park = [&]() {
        const float * o = &O[0][0][0];
#pragma unroll
        for (int c = 0; c < NT; ++c) {
            uint32_t r[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) r[e] = __float_as_uint(o[16 * c + e]);
            umma::tmem_st16(t_O + 16 * c, r);
        }
        umma::tmem_st_wait();
    };
    auto unpark = [&]() {
        float * o = &O[0][0][0];
#pragma unroll
        for (int c = 0; c < NT; ++c) {
            uint32_t r[16];
            umma::tmem_ld16(t_O + 16 * c, r);
#pragma unroll
            for (int e = 0; e < 16; ++e) o[16 * c + e] = __uint_as_float(r[e]);
        }
        umma::tmem_ld_wait();
    };
    if constexpr (PARK) {
        t_O = t_base + ((uint32_t) (32 * w) << 16);
        park();
    }

    const int kA = 16 * w + key_perm<KT>(g), kB = kA + 8;   // this lane's two keys (tile-relative) in the QK phase
    const int mask_from = min(k_hi, rmin + 1);   // the mask is only evaluated in tiles that reach past some row's last key or the chunk's end

    // writes partial `unit` from the accumulators
    auto flush = [&]() {
        // l: sum over the lanes that share this row pair (same t), then over the warps
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float l = l_run[i][e];
                l += __shfl_xor_sync(0xffffffffu, l, 4);
                l += __shfl_xor_sync(0xffffffffu, l, 8);
                l += __shfl_xor_sync(0xffffffffu, l, 16);
                if (g == 0) wl[w * NT * 8 + 8 * i + 2 * t + e] = l;
            }
        __syncthreads();
        if (w == 0 && g == 0) {
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int r = 8 * i + 2 * t + e;
                    if (r < R) {
                        a.pm[(size_t) unit * R + r] = m_run[i][e];
                        a.pl[(size_t) unit * R + r] = (wl[r] + wl[NT * 8 + r]) + (wl[2 * NT * 8 + r] + wl[3 * NT * 8 + r]);
                    }
                }
        }
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = 8 * i + 2 * t + e;
                if (r >= R) continue;
                float * dst = a.po + ((size_t) unit * R + r) * DH;
                if constexpr (KT == B200_KV_F16) {
#pragma unroll
                    for (int mt = 0; mt < 4; ++mt) {
                        dst[64 * w + 16 * mt + g] = O[mt][i][e];
                        dst[64 * w + 16 * mt + g + 8] = O[mt][i][2 + e];
                    }
                } else if constexpr (KT == B200_KV_Q8_0) {
#pragma unroll
                    for (int y = 0; y < 2; ++y)
                        *reinterpret_cast<float4 *>(dst + 64 * w + 32 * y + 4 * g) =
                            make_float4(O[2 * y][i][e], O[2 * y][i][2 + e], O[2 * y + 1][i][e], O[2 * y + 1][i][2 + e]);
                } else {
#pragma unroll
                    for (int y = 0; y < 2; ++y) {
                        *reinterpret_cast<float2 *>(dst + 64 * w + 32 * y + 2 * g) = make_float2(O[2 * y][i][e], O[2 * y][i][2 + e]);
                        *reinterpret_cast<float2 *>(dst + 64 * w + 32 * y + 16 + 2 * g) = make_float2(O[2 * y + 1][i][e], O[2 * y + 1][i][2 + e]);
                    }
                }
            }
    };
    auto end_from = [&](int key) { return (int) min((long long) k_hi, chunk_lo(a.CH, chunk_of(a.CH, key) + 1)); };
    int part_end = 0;
    if constexpr (RUNS) part_end = end_from(k_lo);   // first key that the partial being summed does not cover

    // ring position of the tile's K item (2 it) and V item (2 it + 1): slot index and the parity of its use count
    int last_v = 0, sv_prev = 0;
    int sk = ring0, sv = ring0 + 1;
    uint32_t phk = ring0_par, phv = ring0_par;
    if (sv >= nslot) { sv -= nslot; phv ^= 1u; }
    for (int it = 0; it < ntiles; ++it) {
        const unsigned char * Ks = stg + (size_t) sk * TR::SLOT;
        const unsigned char * Vs = stg + (size_t) sv * TR::SLOT;
        uint64_t * const bar_k = &full[sk], * const bar_v = &full[sv];
        const uint32_t par_k = phk, par_v = phv;
        const int sk_now = sk, sv_now = sv;
        sk += 2; if (sk >= nslot) { sk -= nslot; phk ^= 1u; }
        sv += 2; if (sv >= nslot) { sv -= nslot; phv ^= 1u; }
        mbar_wait(bar_k, par_k, a.status);
        if (it > 0) refill_if_last(last_v, 2 * it - 1, sv_prev);   // the V slot of the previous tile

        // ---------------- S = K Q^T for the warp's 16 keys ----------------
        float S[NT][4];
#pragma unroll
        for (int i = 0; i < NT; ++i) { S[i][0] = S[i][1] = S[i][2] = S[i][3] = 0.0f; }
        const unsigned char * rowA = Ks + kA * SROW, * rowB = Ks + kB * SROW;
        if constexpr (KT == B200_KV_F16) {
#pragma unroll
            for (int b = 0; b < NBLK; ++b) {
                const uint4 wa = *reinterpret_cast<const uint4 *>(Ks + f16_slot_off(kA, 4 * b + t));
                const uint4 wb = *reinterpret_cast<const uint4 *>(Ks + f16_slot_off(kB, 4 * b + t));
                const uint32_t a0[4] = {wa.x, wb.x, wa.y, wb.y}, a1[4] = {wa.z, wb.z, wa.w, wb.w};
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    const uint4 qv = *reinterpret_cast<const uint4 *>(Qs + (8 * i + g) * QSTR + 64 * b + 16 * t);
                    mma16816(S[i], a0, qv.x, qv.y);
                    mma16816(S[i], a1, qv.z, qv.w);
                }
            }
        } else {
            // Integers -> f16 without arithmetic: a 16-bit lane holding a value u in 0..255 in its low byte IS the f16
            // subnormal u * 2^-24, and the tensor cores take subnormal operands at full rate.  A word of four cache bytes
            // gives the pairs (byte 0, byte 2) by a mask and (byte 1, byte 3) by one byte permute; the query dims are
            // stored in the matching order.  The sign offset (q8_0: u = q + 128 after flipping the top bits; q4_0: the
            // nibble carries +8) comes out through the accumulator's starting value Qb, the factor 2^24 through the scale.
            constexpr float UNSUB = 16777216.0f;
            uint4 sA, sB;   // the 8 block scales of each key (q8_0); q4_0 reads them block by block
            if constexpr (KT == B200_KV_Q8_0) {
                sA = *reinterpret_cast<const uint4 *>(rowA);
                sB = *reinterpret_cast<const uint4 *>(rowB);
            }
#pragma unroll
            for (int b = 0; b < NBLK; ++b) {
                uint32_t a0[4], a1[4];
                float dA, dB;
                if constexpr (KT == B200_KV_Q8_0) {
                    const uint2 wa = *reinterpret_cast<const uint2 *>(rowA + 16 + 32 * b + 8 * t);
                    const uint2 wb = *reinterpret_cast<const uint2 *>(rowB + 16 + 32 * b + 8 * t);
                    const uint32_t ax = wa.x ^ 0x80808080u, ay = wa.y ^ 0x80808080u;
                    const uint32_t bx = wb.x ^ 0x80808080u, by = wb.y ^ 0x80808080u;
                    a0[0] = ax & 0x00ff00ffu; a0[1] = bx & 0x00ff00ffu; a0[2] = __byte_perm(ax, 0u, 0x4341); a0[3] = __byte_perm(bx, 0u, 0x4341);
                    a1[0] = ay & 0x00ff00ffu; a1[1] = by & 0x00ff00ffu; a1[2] = __byte_perm(ay, 0u, 0x4341); a1[3] = __byte_perm(by, 0u, 0x4341);
                    const uint32_t swA = (&sA.x)[b >> 1], swB = (&sB.x)[b >> 1];
                    dA = __half2float(__ushort_as_half((unsigned short) ((b & 1) ? swA >> 16 : swA & 0xffffu))) * UNSUB;
                    dB = __half2float(__ushort_as_half((unsigned short) ((b & 1) ? swB >> 16 : swB & 0xffffu))) * UNSUB;
                } else {
                    // block at byte 18 b: f16 d, then 16 bytes; this lane takes bytes 4t..4t+3 (dims 4t.. low nibbles,
                    // 16+4t.. high nibbles).  The 16 bytes start on a 2-byte boundary for even b.
                    uint32_t qa, qb;
                    if ((b & 1) == 0) {
                        const uint32_t * pa = reinterpret_cast<const uint32_t *>(rowA + 18 * b + 4 * t);
                        const uint32_t * pb = reinterpret_cast<const uint32_t *>(rowB + 18 * b + 4 * t);
                        qa = __funnelshift_r(pa[0], pa[1], 16);
                        qb = __funnelshift_r(pb[0], pb[1], 16);
                    } else {
                        qa = *reinterpret_cast<const uint32_t *>(rowA + 18 * b + 2 + 4 * t);
                        qb = *reinterpret_cast<const uint32_t *>(rowB + 18 * b + 2 + 4 * t);
                    }
                    // nibble pairs: low nibbles of bytes (0, 2) and (1, 3) feed the first k-step, the high nibbles the second
                    a0[0] = qa & 0x000f000fu; a0[1] = qb & 0x000f000fu; a0[2] = (qa >> 8) & 0x000f000fu; a0[3] = (qb >> 8) & 0x000f000fu;
                    a1[0] = (qa >> 4) & 0x000f000fu; a1[1] = (qb >> 4) & 0x000f000fu; a1[2] = (qa >> 12) & 0x000f000fu; a1[3] = (qb >> 12) & 0x000f000fu;
                    dA = __half2float(*reinterpret_cast<const __half *>(rowA + 18 * b)) * UNSUB;
                    dB = __half2float(*reinterpret_cast<const __half *>(rowB + 18 * b)) * UNSUB;
                }
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    const uint4 qv = *reinterpret_cast<const uint4 *>(Qs + (8 * i + g) * QSTR + 64 * b + 16 * t);
                    float c[4];
                    mma16816_from(c, Qb[(b * NT + i) * 4 + t], a0, qv.x, qv.y);
                    mma16816(c, a1, qv.z, qv.w);
                    S[i][0] = fmaf(dA, c[0], S[i][0]); S[i][1] = fmaf(dA, c[1], S[i][1]);
                    S[i][2] = fmaf(dB, c[2], S[i][2]); S[i][3] = fmaf(dB, c[3], S[i][3]);
                }
            }
        }
        const int last_k = arrive(0);
        // causal / chunk mask, warp-level row maxima
        const int keyA = k_lo + it * TILE + kA, keyB = keyA + 8;
        if (k_lo + (it + 1) * TILE > mask_from) {
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (keyA > rpos[i][e] || keyA >= k_hi) S[i][e] = B200_NEG_INF;
                    if (keyB > rpos[i][e] || keyB >= k_hi) S[i][2 + e] = B200_NEG_INF;
                }
        }
        // ---------------- online softmax, P -> shared memory ----------------
        // Every row has a reference maximum m_run, the same in all four warps, that trails its true maximum by at most
        // REF_GAP (P = 2^(S - m_run + PSHIFT) <= 2^15 stays inside f16).  A warp whose keys stay under m_run + REF_GAP needs
        // nothing from the other warps: it writes P at once.  Only when some warp of the CTA sees a larger score (always on
        // the first tile) do the warps exchange their maxima after the barrier, move the references, redo P and rescale O.
        bool grow = false;
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) grow = grow || fmaxf(S[i][e], S[i][2 + e]) > m_run[i][e] + REF_GAP;
        const int ph = (tiles_before + it) % 3;   // three flags in turn: the one of the next tile is cleared two barriers after its last reader
        if (__any_sync(0xffffffffu, grow) && lane == 0) flag[ph] = 1;
        if (tid == 0) flag[ph == 2 ? 0 : ph + 1] = 0;
        refill_if_last(last_k, 2 * it, sk_now);
        // P and the V scales of this tile replace those of the previous tile: every warp must be done with its P V
        if (it > 0) {
            int spins = 0;
            while (*reinterpret_cast<volatile int *>(&done[1]) < NWARP * (tiles_before + it))
                if (++spins > (1 << 24)) { atomicOr(a.status, ST_WAIT_TIMEOUT); break; }
        }
        float lsum[NT][2];
        auto write_p = [&]() {   // P carries a factor 2^PSHIFT (numerator and denominator alike): keeps small weights out of
                                 // the f16 subnormal range; 2^(-inf) = 0 for a masked key
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int r = 8 * i + 2 * t + e;
                    const float msafe = m_run[i][e] == B200_NEG_INF ? 0.0f : m_run[i][e];
                    const __half pa = __float2half_rn(ex2f(S[i][e] - msafe + PSHIFT));
                    const __half pb = __float2half_rn(ex2f(S[i][2 + e] - msafe + PSHIFT));
                    lsum[i][e] = __half2float(pa) + __half2float(pb);
                    *reinterpret_cast<__half *>(Ps + r * PSTR + kA * 2) = pa;
                    *reinterpret_cast<__half *>(Ps + r * PSTR + kB * 2) = pb;
                }
        };
        write_p();
        mbar_wait(bar_v, par_v, a.status);   // this tile's V rows
        const int v_keys = k_hi - (k_lo + it * TILE);   // rows of the tile that hold keys: 64 or more but in the last tile
        if constexpr (TR::SCALED) {   // V block scales, transposed to [block][key]; zero for rows past the last key (their bytes may be anything)
            const int key = tid >> 1, b0 = (tid & 1) * 4;
#pragma unroll
            for (int b = b0; b < b0 + 4; ++b) {
                const unsigned char * src = KT == B200_KV_Q8_0 ? Vs + key * SROW + 2 * b : Vs + key * SROW + 18 * b;
                const uint16_t d = *reinterpret_cast<const uint16_t *>(src);
                *reinterpret_cast<uint16_t *>(Sd + b * SDSTR + key * 2) = key < v_keys ? d : (uint16_t) 0;
            }
        } else if (v_keys < TILE) {
            unsigned char * vz = stg + (size_t) sv_now * TR::SLOT;
            for (int i = tid; i < (TILE - v_keys) * 32; i += NTHR)
                *reinterpret_cast<uint4 *>(vz + f16_slot_off(v_keys + (i >> 5), i & 31)) = make_uint4(0, 0, 0, 0);
            umma::fence_async_smem();   // the slot's next fill comes through the async proxy
        }
        __syncthreads();   // P, the V scales, the warps' maxima and the flag are visible
        if constexpr (PARK) unpark();
        if (flag[ph]) {
            // the warps' row maxima over their 16 keys, exchanged through shared memory
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float mx = fmaxf(S[i][e], S[i][2 + e]);
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                    if (g == 0) wmax[w * NT * 8 + 8 * i + 2 * t + e] = mx;
                }
            __syncthreads();
            float fsc[NT][2];
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int r = 8 * i + 2 * t + e;
                    const float mx = fmaxf(fmaxf(wmax[r], wmax[NT * 8 + r]), fmaxf(wmax[2 * NT * 8 + r], wmax[3 * NT * 8 + r]));
                    const float mnew = mx > m_run[i][e] + REF_GAP ? mx : m_run[i][e];
                    fsc[i][e] = ex2f(m_run[i][e] - (mnew == B200_NEG_INF ? 0.0f : mnew));
                    m_run[i][e] = mnew;
                }
            write_p();   // rows whose reference stayed get the same bits again
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) l_run[i][e] = fmaf(l_run[i][e], fsc[i][e], lsum[i][e]);
#pragma unroll
            for (int mt = 0; mt < 4; ++mt)
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    O[mt][i][0] *= fsc[i][0]; O[mt][i][1] *= fsc[i][1];
                    O[mt][i][2] *= fsc[i][0]; O[mt][i][3] *= fsc[i][1];
                }
            __syncthreads();   // the rewritten P is visible
        } else {
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) l_run[i][e] += lsum[i][e];
        }

        // ---------------- O^T += V^T P^T for the warp's 64 output dims ----------------
#pragma unroll
        for (int u = 0; u < TILE / 16; ++u) {
            uint32_t pw[NT][2];
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                pw[i][0] = *reinterpret_cast<const uint32_t *>(Ps + (8 * i + g) * PSTR + (16 * u + 2 * t) * 2);
                pw[i][1] = *reinterpret_cast<const uint32_t *>(Ps + (8 * i + g) * PSTR + (16 * u + 2 * t + 8) * 2);
            }
            if constexpr (KT == B200_KV_F16) {
#pragma unroll
                for (int mt = 0; mt < 4; ++mt) {
                    // four 8x8 tiles, transposed on load: (keys 0-7 | 8-15) x (dims 0-7 | 8-15) of this m-tile
                    const int mj = lane >> 3, mr = lane & 7;
                    const unsigned char * p = Vs + f16_slot_off(16 * u + (mj >> 1) * 8 + mr, 8 * w + 2 * mt + (mj & 1));
                    uint32_t av[4];
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(av[0]), "=r"(av[1]), "=r"(av[2]), "=r"(av[3]) : "r"(smem_u32(p)));
#pragma unroll
                    for (int i = 0; i < NT; ++i) mma16816(O[mt][i], av, pw[i][0], pw[i][1]);
                }
            } else {
                const unsigned char * v0 = Vs + (16 * u + 2 * t) * SROW, * v1 = v0 + SROW, * v2 = v0 + 8 * SROW, * v3 = v2 + SROW;
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    const int blk = 2 * w + y;
                    uint32_t ax[4], ay[4];   // m-tiles X and Y of this block
                    if constexpr (KT == B200_KV_Q8_0) {
                        const int col = 16 + 32 * blk + 4 * g;
                        const uint32_t w0 = *reinterpret_cast<const uint32_t *>(v0 + col) ^ 0x80808080u;
                        const uint32_t w1 = *reinterpret_cast<const uint32_t *>(v1 + col) ^ 0x80808080u;
                        const uint32_t w2 = *reinterpret_cast<const uint32_t *>(v2 + col) ^ 0x80808080u;
                        const uint32_t w3 = *reinterpret_cast<const uint32_t *>(v3 + col) ^ 0x80808080u;
                        // interleave key pairs: e01 = (k0.d0, k1.d0, k0.d1, k1.d1), f01 = (k0.d2, k1.d2, k0.d3, k1.d3)
                        const uint32_t e01 = __byte_perm(w0, w1, 0x5140), f01 = __byte_perm(w0, w1, 0x7362);
                        const uint32_t e23 = __byte_perm(w2, w3, 0x5140), f23 = __byte_perm(w2, w3, 0x7362);
                        ax[0] = cvt_i8x2<0>(e01); ax[1] = cvt_i8x2<1>(e01); ax[2] = cvt_i8x2<0>(e23); ax[3] = cvt_i8x2<1>(e23);
                        ay[0] = cvt_i8x2<0>(f01); ay[1] = cvt_i8x2<1>(f01); ay[2] = cvt_i8x2<0>(f23); ay[3] = cvt_i8x2<1>(f23);
                    } else {
                        const int col = 18 * blk + 2 + 2 * g;   // bytes 2g, 2g+1 of the block: dims 2g, 2g+1 | 16+2g, 17+2g
                        const uint32_t h0 = *reinterpret_cast<const uint16_t *>(v0 + col), h1 = *reinterpret_cast<const uint16_t *>(v1 + col);
                        const uint32_t h2 = *reinterpret_cast<const uint16_t *>(v2 + col), h3 = *reinterpret_cast<const uint16_t *>(v3 + col);
                        const uint32_t w01 = h0 | (h1 << 16), w23 = h2 | (h3 << 16);   // bytes (k0.B0, k0.B1, k1.B0, k1.B1)
                        const uint32_t l01 = w01 & 0x0f0f0f0fu, u01 = (w01 >> 4) & 0x0f0f0f0fu;
                        const uint32_t l23 = w23 & 0x0f0f0f0fu, u23 = (w23 >> 4) & 0x0f0f0f0fu;
                        // (k0.x, k1.x) pairs: bytes 0 and 2 -> dim 2g (+16), bytes 1 and 3 -> dim 2g+1 (+16)
                        ax[0] = hsub2_u32(__byte_perm(l01, 0x64646464u, 0x6240), 0x64086408u);
                        ax[1] = hsub2_u32(__byte_perm(l01, 0x64646464u, 0x7351), 0x64086408u);
                        ax[2] = hsub2_u32(__byte_perm(l23, 0x64646464u, 0x6240), 0x64086408u);
                        ax[3] = hsub2_u32(__byte_perm(l23, 0x64646464u, 0x7351), 0x64086408u);
                        ay[0] = hsub2_u32(__byte_perm(u01, 0x64646464u, 0x6240), 0x64086408u);
                        ay[1] = hsub2_u32(__byte_perm(u01, 0x64646464u, 0x7351), 0x64086408u);
                        ay[2] = hsub2_u32(__byte_perm(u23, 0x64646464u, 0x6240), 0x64086408u);
                        ay[3] = hsub2_u32(__byte_perm(u23, 0x64646464u, 0x7351), 0x64086408u);
                    }
                    const uint32_t sd0 = *reinterpret_cast<const uint32_t *>(Sd + blk * SDSTR + (16 * u + 2 * t) * 2);
                    const uint32_t sd1 = *reinterpret_cast<const uint32_t *>(Sd + blk * SDSTR + (16 * u + 2 * t + 8) * 2);
                    // block scale of each key pair folded into V (f16 product of an exact integer and the f16 scale)
                    ax[0] = hmul2_u32(ax[0], sd0); ax[1] = hmul2_u32(ax[1], sd0); ax[2] = hmul2_u32(ax[2], sd1); ax[3] = hmul2_u32(ax[3], sd1);
                    ay[0] = hmul2_u32(ay[0], sd0); ay[1] = hmul2_u32(ay[1], sd0); ay[2] = hmul2_u32(ay[2], sd1); ay[3] = hmul2_u32(ay[3], sd1);
#pragma unroll
                    for (int i = 0; i < NT; ++i) {
                        mma16816(O[2 * y][i], ax, pw[i][0], pw[i][1]);
                        mma16816(O[2 * y + 1][i], ay, pw[i][0], pw[i][1]);
                    }
                }
            }
        }
        last_v = arrive(1);
        sv_prev = sv_now;
        if (RUNS && k_lo + (it + 1) * TILE >= part_end) {
            flush();
            if (it + 1 < ntiles) {   // the next chunk starts afresh
                ++unit;
                part_end = end_from(part_end);
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    m_run[i][0] = m_run[i][1] = B200_NEG_INF;
                    l_run[i][0] = l_run[i][1] = 0.0f;
#pragma unroll
                    for (int mt = 0; mt < 4; ++mt) O[mt][i][0] = O[mt][i][1] = O[mt][i][2] = O[mt][i][3] = 0.0f;
                }
            }
        }
        if constexpr (PARK) park();
    }
    if constexpr (!RUNS) {
        if constexpr (PARK) unpark();
        flush();
    }
    return ntiles;
}

#include "decode_tc.cuh"
#include "decode_warp.cuh"

// The kernel.  With a run plan: every segment of the CTA's run one after the other.  Fixed chunks without a plan (one slot;
// no more chunks than CTAs; more slots than a plan holds): units u = index, + CTAs of the kv head, .., one chunk each, the highest chunk
// index first, so that the long chunks start first and the short ones fill the tail.  (One long context as contiguous runs,
// cut at chunk boundaries like the plans: 401 us against 364 for four layers of 131000 keys, because a CTA got either 8 or 16
// tiles.)
template <uint32_t KT, int NT, bool RUNS>
__global__ void __launch_bounds__(NTHR, ctas_per_sm<KT, NT>())
decode_part_k(const dec_args a, const int nslot, const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapV) {
    pdl_enter();
    extern __shared__ __align__(1024) unsigned char smem[];
    // kv head = block index mod heads: the heads of one (slot, key range) are neighbours in launch order, so the four
    // head rows of a position are fetched close together in time
    const int hl = (int) (blockIdx.x % (unsigned) a.nhk), ui = (int) (blockIdx.x / (unsigned) a.nhk);
    int s0, s1, nch = a.max_chunks, step = (int) (gridDim.x / (unsigned) a.nhk);
    const bool one_wave = (long long) a.max_chunks * a.n_slots <= step;   // no CTA has two chunks: their order does not matter, nor who has how many
    if (a.segs) {
        const int c = min(ui, a.max_cta - 1), n = *a.n_cta, c0 = a.cta_seg[c], c1 = a.cta_seg[c + 1];   // loads that do not wait for one another
        if (RUNS && n < 0) { s0 = ui; s1 = -n; }
        else {
            if (ui >= n) return;
            s0 = c0; s1 = c1; step = 1;
        }
    } else {
        if (one_wave) nch = a.max_chunks;
        else if (a.n_slots == 1) {   // the chunks the slot has (a position beyond the limit is reported by the unit that runs)
            const int p = (threadIdx.x & 31) < a.q_len ? row_pos(a, 0, threadIdx.x & 31) : -1;
            const int n = min(__reduce_max_sync(0xffffffffu, p) + 1, key_limit(a));
            nch = n > 0 ? chunk_of(a.CH, n - 1) + 1 : 0;
        }
        s0 = ui; s1 = (int) min((long long) nch * a.n_slots, 0x7fffffffLL);
    }
    if (s0 >= s1) return;
    // barriers of the copy ring, arrival counters and flags: made once per CTA
    if (threadIdx.x == 0) {
        uint64_t * full = reinterpret_cast<uint64_t *>(smem);
        for (int s = 0; s < nslot; ++s) mbar_init(&full[s], 1);
        mbar_fence_init();
        int * cnt = reinterpret_cast<int *>(smem + 96);   // done[2], flag[3]
        cnt[0] = cnt[1] = cnt[2] = cnt[3] = cnt[4] = 0;
    }
    // (a unit's first barrier makes them and the tensor-memory base known to all; the warp that starts the first copies has made them itself)
    uint32_t * t_slot = reinterpret_cast<uint32_t *>(smem + 120);
    if constexpr (parks<KT, NT>()) {
        if (threadIdx.x >= 32 && threadIdx.x < 64) umma::tmem_alloc(t_slot, PARK_COLS);
    }
    __syncwarp();
    int tiles = 0;
    for (int u = s0; u < s1; u += step) {
        int slot, chunk = -1, k_lo, k_cap;
        unsigned unit;
        if (a.segs) {
            const int4 e = a.segs[u];
            slot = e.x; k_lo = e.y; k_cap = e.z;
            unit = (unsigned) u * a.nhk + hl;
            if constexpr (RUNS) chunk = chunk_of(a.CH, k_lo);
        } else {
            slot = u % a.n_slots; chunk = nch - 1 - u / a.n_slots;
            k_lo = (int) min(0x7fffffffLL, chunk_lo(a.CH, chunk));
            k_cap = (int) min(0x7fffffffLL, chunk_lo(a.CH, chunk + 1));
        }
        if (chunk >= 0) unit = ((unsigned) slot * a.nhk + hl) * a.max_chunks + chunk;   // below 2^31 (decode_geometry)
        if (tiles) __syncthreads();   // the previous unit's shared memory is no longer read
        tiles += decode_unit<KT, NT, RUNS>(a, nslot, mapK, mapV, smem, a.hk0 + hl, slot, k_lo, k_cap, unit, tiles, t_slot);
        if (u > 0x7fffffff - step) break;
    }
    if constexpr (parks<KT, NT>()) {
        umma::fence_before_sync();
        __syncthreads();
        if (threadIdx.x >= 32 && threadIdx.x < 64) {
            umma::fence_after_sync();
            umma::tmem_dealloc(*t_slot, PARK_COLS);
        }
    }
}

// Merge a row's chunk partials.  Chunk c belongs to summation stream c mod MERGE_STREAMS; a stream is summed in ascending order in an
// accumulator of its own and the streams are added in stream order: an order that depends on the number of chunks only, not on the
// rest of the call.
//   out != nullptr : out = num / den (* sigmoid(gate)); rows that saw no key give zeros
//   fo  != nullptr : unnormalised num, max in natural-log units, den (for a cross-GPU merge)
// What both kernels below do once a row's partials are summed: lanes hold four dims each, oi = float4 index of the result.
__device__ __forceinline__ void merge_finish(const dec_args & a, float4 num, float den, float M, size_t oi, size_t row, int h, bool live, bool first, float4 gv,
                                             const float * gate, float * out, float * fo, float * fm, float * fl, __half2 * qbuf, size_t rows) {
    if (fo && live) {   // public partials are plain sums: take the internal 2^PSHIFT out (exact)
        constexpr float U = 1.0f / 256.0f;
        static_assert(PSHIFT == 8.0f, "U must be 2^-PSHIFT");
        reinterpret_cast<float4 *>(fo)[oi] = make_float4(num.x * U, num.y * U, num.z * U, num.w * U);
        if (first) { fm[row * a.Hq + h] = M * LN2; fl[row * a.Hq + h] = den * U; }
    }
    if (out) {
        float4 y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (den > 0.0f) {
            const float inv = 1.0f / den;
            y = make_float4(num.x * inv, num.y * inv, num.z * inv, num.w * inv);
            if (gate) {
                y.x *= 1.0f / (1.0f + expf(-gv.x)); y.y *= 1.0f / (1.0f + expf(-gv.y));
                y.z *= 1.0f / (1.0f + expf(-gv.z)); y.w *= 1.0f / (1.0f + expf(-gv.w));
            }
        }
        if (live) reinterpret_cast<float4 *>(out)[oi] = y;
        // the projection that follows attention reads its input in the a16 format: emitted here, from registers
        if (qbuf) a16_store_lanes8(y, qbuf, oi >> 3, rows * (a.Hq * (DH / 32)), live);
    }
}

// Few partials on a grid that fills the GPU: grid (rows, Hq), 64 threads of one float4 each, the partials one after the other.  CHUNKED: the
// roundings of one chunk per stream (at most MERGE_STREAMS chunks).
constexpr int MERGE_STREAMS = 16;
template <bool CHUNKED>
__global__ void __launch_bounds__(64) decode_merge_k(const dec_args a, const float * __restrict__ gate, float * __restrict__ out, float * __restrict__ fo,
                                                     float * __restrict__ fm, float * __restrict__ fl, __half2 * __restrict__ qbuf) {
    pdl_enter();
    const int lane4 = threadIdx.x;
    const int row = blockIdx.x, slot = row / a.q_len, j = row - slot * a.q_len;
    const int hl = blockIdx.y / GQA, hh = blockIdx.y - hl * GQA, h = a.hk0 * GQA + blockIdx.y, r = j * GQA + hh, R = a.q_len * GQA;
    const int pos = min(row_pos(a, slot, j), key_limit(a) - 1);   // a row past the limit merges the chunks that exist
    // partials of the row's kv head: consecutive units of stride ustr from unit0 (a segment the row does not reach holds m = -inf)
    int nch;
    size_t unit0, ustr;
    if constexpr (!CHUNKED) {
        int2 sg;
        if (a.solo) { sg.x = 0; solo_runs(a, sg.y); }
        else sg = a.slot_seg[slot];
        nch = pos < 0 ? 0 : sg.y;
        unit0 = (size_t) sg.x * a.nhk + hl; ustr = a.nhk;
    } else {
        nch = pos < 0 ? 0 : chunk_of(a.CH, pos) + 1;
        unit0 = ((size_t) slot * a.nhk + hl) * a.max_chunks; ustr = 1;
    }
    const float * pm = a.pm + unit0 * R + r, * pl = a.pl + unit0 * R + r;
    const float4 * po = reinterpret_cast<const float4 *>(a.po + (unit0 * R + r) * DH) + lane4;
    const size_t st = ustr * R;   // from one partial of the row to the next, in values (pm, pl) and head rows (po)
    float M = B200_NEG_INF;
    for (int c = 0; c < nch; ++c) M = fmaxf(M, pm[c * st]);
    float den = 0.0f;
    float4 num = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
    for (int c = 0; c < nch; ++c) {   // no early continue: the loads of several chunks are in flight together
        const float ms = pm[c * st], lc = pl[c * st];
        const float4 o = po[c * st * (DH / 4)];
        const float f = ms == B200_NEG_INF ? 0.0f : ex2f(ms - M);   // a chunk the row did not see holds zeros: adds nothing
        if constexpr (CHUNKED) {
            den += __fmul_rn(f, lc);
            num.x += __fmul_rn(f, o.x); num.y += __fmul_rn(f, o.y); num.z += __fmul_rn(f, o.z); num.w += __fmul_rn(f, o.w);
        } else {
            den = fmaf(f, lc, den);
            num.x = fmaf(f, o.x, num.x); num.y = fmaf(f, o.y, num.y); num.z = fmaf(f, o.z, num.z); num.w = fmaf(f, o.w, num.w);
        }
    }
    const size_t oi = ((size_t) row * a.Hq + h) * (DH / 4) + lane4;
    const float4 gv = gate ? reinterpret_cast<const float4 *>(gate)[oi] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    merge_finish(a, num, den, M, oi, row, h, true, lane4 == 0, gv, gate, out, fo, fm, fl, qbuf, gridDim.x);
}

// Everything else: grid (rows, Hq, 256 / 64), a thread per (stream, four dims) of a 64-dim slice.  Bound by a chain of dependent loads
// (position, number of partials, maxima, partials) with nothing else to hide it, so all loads that can go out do so at once: the gate, the
// position and the first AHEAD partials of every stream, which lie inside the scratch whether the row has them or not and are left out
// once the position is known.  Against CTAs of up to 1024 threads per (row, head) that loaded one after the other (64 registers: one such CTA
// on an SM): 16 layers of one row at 4096 keys 311 -> 283 us, four layers of one row at 131000 keys (q4_0) 321 -> 305, 16 layers of 1 + 3 rows at
// 30011 keys 609 -> 592, four layers of 8 rows of up to 16384 keys 337 -> 330.
constexpr int MERGE_DL = 16, MERGE_THR = MERGE_STREAMS * MERGE_DL;
template <int AHEAD>
__global__ void __launch_bounds__(MERGE_THR, AHEAD > 4 ? 2 : 4) decode_merge_streams_k(const dec_args a, const float * __restrict__ gate, float * __restrict__ out,
                                                                    float * __restrict__ fo, float * __restrict__ fm, float * __restrict__ fl,
                                                                    __half2 * __restrict__ qbuf) {
    pdl_enter();
    __shared__ float4 snum[MERGE_STREAMS][MERGE_DL];
    __shared__ float sden[MERGE_STREAMS], smax[MERGE_THR / 32];
    const int tid = threadIdx.x, dl = tid & (MERGE_DL - 1), s = tid / MERGE_DL;
    const int row = blockIdx.x, slot = row / a.q_len, j = row - slot * a.q_len;
    const int hl = blockIdx.y / GQA, hh = blockIdx.y - hl * GQA, h = a.hk0 * GQA + blockIdx.y, r = j * GQA + hh, R = a.q_len * GQA;
    const size_t oi = ((size_t) row * a.Hq + h) * (DH / 4) + blockIdx.z * MERGE_DL + dl;
    float4 gv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (gate && s < 2) gv = reinterpret_cast<const float4 *>(gate)[oi];   // the first warp finishes the row
    size_t unit0, ustr;
    int most;   // partials that may be read
    if (a.chunked) {
        most = a.max_chunks;
        unit0 = ((size_t) slot * a.nhk + hl) * a.max_chunks; ustr = 1;
    } else {
        int2 sg;
        if (a.solo) { sg.x = 0; solo_runs(a, sg.y); }
        else sg = a.slot_seg[slot];
        most = sg.y;
        unit0 = (size_t) sg.x * a.nhk + hl; ustr = a.nhk;
    }
    // the stream's next partial; from one partial of the row to the next, ustr * R values (pm, pl) and head rows (po)
    const size_t i0 = (unit0 + s * ustr) * R + r, st = MERGE_STREAMS * ustr * R;
    const float * pm = a.pm + i0;
    const ptrdiff_t to_pl = a.pl - a.pm;
    const float4 * po = reinterpret_cast<const float4 *>(a.po + i0 * DH) + blockIdx.z * MERGE_DL + dl;
    float ms[AHEAD], ls[AHEAD];
    float4 o[AHEAD];
    auto fetch = [&](int c0, int n) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            ms[u] = B200_NEG_INF; ls[u] = 0.0f; o[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (c0 + u * MERGE_STREAMS < n) { ms[u] = *pm; ls[u] = pm[to_pl]; o[u] = *po; }
            pm += st; po += st * (DH / 4);
        }
    };
    fetch(s, most);
    const int pos = min(row_pos(a, slot, j), key_limit(a) - 1);   // a row past the limit merges the chunks that exist
    const int nch = pos < 0 ? 0 : a.chunked ? chunk_of(a.CH, pos) + 1 : most;
    float M = B200_NEG_INF;
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
        if (s + u * MERGE_STREAMS >= nch) { ms[u] = B200_NEG_INF; ls[u] = 0.0f; o[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f); }
        M = fmaxf(M, ms[u]);
    }
    for (int c = AHEAD * MERGE_STREAMS + tid; c < nch; c += MERGE_THR) M = fmaxf(M, a.pm[(unit0 + c * ustr) * R + r]);
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, k));
    if ((tid & 31) == 0) smax[tid >> 5] = M;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MERGE_THR / 32; ++i) M = fmaxf(M, smax[i]);
    float d = 0.0f;
    float4 n = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int c0 = s;;) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const float f = ms[u] == B200_NEG_INF ? 0.0f : ex2f(ms[u] - M);   // a chunk the row did not see holds zeros: adds nothing
            d = fmaf(f, ls[u], d);
            n.x = fmaf(f, o[u].x, n.x); n.y = fmaf(f, o[u].y, n.y); n.z = fmaf(f, o[u].z, n.z); n.w = fmaf(f, o[u].w, n.w);
        }
        c0 += AHEAD * MERGE_STREAMS;
        if (c0 >= nch) break;
        fetch(c0, nch);
    }
    snum[s][dl] = n;
    if (dl == 0) sden[s] = d;
    __syncthreads();
    if (tid >= 32) return;   // both halves of the first warp add up the streams, the first one writes
    float den = 0.0f;
    float4 num = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int ns = min(nch, MERGE_STREAMS);   // the other streams are empty
    for (int k = 0; k < ns; ++k) {
        const float4 v = snum[k][dl];
        num.x += v.x; num.y += v.y; num.z += v.z; num.w += v.w;
        den += sden[k];
    }
    merge_finish(a, num, den, M, oi, row, h, tid < MERGE_DL, blockIdx.z == 0 && dl == 0, gv, gate, out, fo, fm, fl, qbuf, gridDim.x);
}

// Merge of caller-provided partials (cross-GPU sequence split): part s has O [R][D] at po + s * so, m (natural log) [R] at
// pm + s * sm and l [R] at pl + s * sm (strides in floats); one block per row, D/4 threads.
__global__ void merge_parts_k(const float * __restrict__ po, const float * __restrict__ pm, const float * __restrict__ pl,
                              int nparts, int R, int D, const float * __restrict__ gate, float * __restrict__ out, size_t so,
                              size_t sm, __half2 * __restrict__ qbuf) {
    pdl_enter();
    const int r = blockIdx.x, i = threadIdx.x;
    float M = B200_NEG_INF;
    for (int s = 0; s < nparts; ++s) M = fmaxf(M, pm[s * sm + r]);
    float den = 0.0f;
    float4 num = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int s = 0; s < nparts; ++s) {
        const float ms = pm[s * sm + r];
        if (ms == B200_NEG_INF) continue;
        const float f = ex2f((ms - M) * LOG2E);
        den = fmaf(f, pl[s * sm + r], den);
        const float4 o = reinterpret_cast<const float4 *>(po + s * so + (size_t) r * D)[i];
        num.x = fmaf(f, o.x, num.x); num.y = fmaf(f, o.y, num.y); num.z = fmaf(f, o.z, num.z); num.w = fmaf(f, o.w, num.w);
    }
    float4 y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (den > 0.0f) {
        const float inv = 1.0f / den;
        y = make_float4(num.x * inv, num.y * inv, num.z * inv, num.w * inv);
        if (gate) {
            const float4 gv = reinterpret_cast<const float4 *>(gate + (size_t) r * D)[i];
            y.x *= 1.0f / (1.0f + expf(-gv.x)); y.y *= 1.0f / (1.0f + expf(-gv.y));
            y.z *= 1.0f / (1.0f + expf(-gv.z)); y.w *= 1.0f / (1.0f + expf(-gv.w));
        }
    }
    reinterpret_cast<float4 *>(out + (size_t) r * D)[i] = y;
    // a16 copy of the gated output (rows of row_len = heads * D values): group index = float index / 32
    if (qbuf) a16_store_lanes8(y, qbuf, ((size_t) r * D + 4 * i) / 32, (size_t) R * D / 32, true);
}

// The same merge with the shards' partials read in place: shard s of a sequence split keeps its partial [O (R*D) | m (R) | l (R)]
// in a buffer that its peers have mapped (part[s]: this GPU's own buffer for s == me, a peer mapping otherwise) and a row of
// flag words flag[s][0..n_seq) that shard j writes at index j.  A call with epoch e (1, 2, .. in step on all shards)
//   1. tells every peer "my partial of call e is complete" (the kernel that wrote it ran before this one on the stream),
//   2. waits, bounded, until every peer has said the same,
//   3. merges in shard order, reading the peers' rows over NVLink with plain loads that bypass L1.
// The caller alternates two partial buffers by the parity of e: a peer that announces call e + 1 has finished reading the
// buffer of call e, and this shard passes step 2 of call e + 1 before the kernel that rewrites that buffer (call e + 2)
// can start.  One block per row, D/4 threads; the first four blocks announce, every block waits by itself.
constexpr int MAX_PEERS = 8;
struct peer_parts { const float * part[MAX_PEERS]; unsigned * flag[MAX_PEERS]; };

__device__ __forceinline__ float4 ld_sys_f4(const float * p) {
    float4 v;
    asm volatile("ld.relaxed.sys.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float ld_sys_f(const float * p) {
    float v;
    asm volatile("ld.relaxed.sys.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}

__global__ void merge_peers_k(const peer_parts pp, int n_seq, int me, unsigned epoch, int R, int D, const float * __restrict__ gate,
                              float * __restrict__ out, __half2 * __restrict__ qbuf, unsigned * __restrict__ status) {
    const int r = blockIdx.x, i = threadIdx.x;
    // the first blocks of the grid announce (any one would do; a few, so that the announcement does not hang on one block's
    // turn); every block waits by itself
    if (r < 4 && i < n_seq && i != me)
        asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(pp.flag[i] + me), "r"(epoch) : "memory");
    if (i < n_seq && i != me) {
        const unsigned * f = pp.flag[me] + i;
        unsigned v;
        const unsigned long long t0 = globaltimer_ns();
        for (int it = 0;; ++it) {
            asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
            if ((int) (v - epoch) >= 0) break;
            if ((it & 63) == 63 && globaltimer_ns() - t0 > 2000000000ull) { atomicOr(status, ST_WAIT_TIMEOUT); break; }
        }
    }
    __syncthreads();
    const size_t om = (size_t) R * D, ol = om + R;
    float ms[MAX_PEERS];
    float M = B200_NEG_INF;
#pragma unroll
    for (int s = 0; s < MAX_PEERS; ++s) {
        ms[s] = B200_NEG_INF;
        if (s < n_seq) ms[s] = s == me ? pp.part[s][om + r] : ld_sys_f(pp.part[s] + om + r);
        M = fmaxf(M, ms[s]);
    }
    float den = 0.0f;
    float4 num = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int s = 0; s < MAX_PEERS; ++s) {
        if (s >= n_seq || ms[s] == B200_NEG_INF) continue;
        const float f = ex2f((ms[s] - M) * LOG2E);
        const float * po = pp.part[s] + (size_t) r * D + 4 * i;
        const float l = s == me ? pp.part[s][ol + r] : ld_sys_f(pp.part[s] + ol + r);
        const float4 o = s == me ? *reinterpret_cast<const float4 *>(po) : ld_sys_f4(po);
        den = fmaf(f, l, den);
        num.x = fmaf(f, o.x, num.x); num.y = fmaf(f, o.y, num.y); num.z = fmaf(f, o.z, num.z); num.w = fmaf(f, o.w, num.w);
    }
    float4 y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (den > 0.0f) {
        const float inv = 1.0f / den;
        y = make_float4(num.x * inv, num.y * inv, num.z * inv, num.w * inv);
        if (gate) {
            const float4 gv = reinterpret_cast<const float4 *>(gate + (size_t) r * D)[i];
            y.x *= 1.0f / (1.0f + expf(-gv.x)); y.y *= 1.0f / (1.0f + expf(-gv.y));
            y.z *= 1.0f / (1.0f + expf(-gv.z)); y.w *= 1.0f / (1.0f + expf(-gv.w));
        }
    }
    reinterpret_cast<float4 *>(out + (size_t) r * D)[i] = y;
    if (qbuf) a16_store_lanes8(y, qbuf, ((size_t) r * D + 4 * i) / 32, (size_t) R * D / 32, true);
}

// Even split of a batch over the resident CTAs (used when the chunk is chosen from the batch).  The 64-key tiles of all slots,
// slot after slot, form one sequence per kv head; CTA c of n_cta takes tiles [c W / n_cta, (c + 1) W / n_cta), so every CTA
// has the same work to within one tile however ragged the contexts are, and all CTAs fit the machine at once.  A run that
// crosses slot boundaries becomes several segments; each segment yields one partial.  n_cta = min(max_cta, W / min_tiles): the
// tcgen05 kernel walks tiles of 128 keys, so its runs hold at least two of these.  Fixed chunks (chunked): the same runs,
// their ends moved to the nearest chunk boundary, so that a CTA streams neighbouring chunks of one slot instead of starting
// afresh for each chunk of a work list (four layers of 8 rows of 700 .. 16384 keys, f16: 389 -> 341 us).  As many
// chunks as CTAs or fewer: one chunk each, without a plan where the host can tell (cut by tiles, CTAs without a chunk lie between the others and leave SMs
// idle: 512 chunks of 512 keys, q4_0, one head, 888 CTAs: 53.8 us a call, 37.3 with a CTA per chunk).  Few slots of a quantised cache with chunks
// of two tiles on average or more (list_cap): a list of all chunks, the highest first, over more CTAs than are resident.  There the chip is busy with
// arithmetic, and what counts is that an SM gets its next chunk when it has room: 8 rows at 100003 keys, q4_0, two heads 182.9 us in runs, 158.5
// in a list; f16, four heads, 30011 keys 136.7 and 158.4.  One block; n_slots
// <= PLAN_MAX_SLOTS.
constexpr int SPLIT_THR = 1024, SPLIT_MAX_SLOTS = 2048, PLAN_MAX_SLOTS = 8192, SPLIT_MAX_CTA = 1024, LIST_SLOTS = 8, LIST_MAX = 8192;
__global__ void __launch_bounds__(SPLIT_THR) decode_split_k(const dec_args a, int max_cta, int list_cap, int min_tiles, int4 * __restrict__ segs, int * __restrict__ cta_seg,
                                                            int2 * __restrict__ slot_seg, int * __restrict__ n_cta_out) {
    pdl_enter();
    __shared__ int pre[PLAN_MAX_SLOTS + 1];      // tiles before slot s
    __shared__ int cseg[SPLIT_MAX_CTA + 1];      // segments before CTA c
    __shared__ int scut[SPLIT_MAX_CTA + 1];      // first tile of CTA c
    __shared__ short first_slot[SPLIT_MAX_CTA];
    __shared__ int n_chunks;
    const int tid = threadIdx.x, lim = key_limit(a);
    auto slot_keys = [&](int s) {
        int n = 0;
        for (int j = 0; j < a.q_len; ++j) n = max(n, row_pos(a, s, j) + 1);
        return min(n, lim);
    };
    int my_chunks = 0;
    for (int s = tid; s < a.n_slots; s += SPLIT_THR) {
        const int n = slot_keys(s);
        pre[s + 1] = (n + TILE - 1) / TILE;
        if (a.chunked && n > 0) my_chunks += chunk_of(a.CH, n - 1) + 1;
    }
    if (tid == 0) { pre[0] = 0; n_chunks = 0; }
    __syncthreads();
    if (a.chunked) {
        my_chunks = __reduce_add_sync(0xffffffffu, my_chunks);
        if ((tid & 31) == 0 && my_chunks) atomicAdd(&n_chunks, my_chunks);
    }
    if (tid < 32) {   // inclusive scan of pre[1..n_slots], 32 entries at a time with a running carry
        int carry = 0;
        for (int base = 1; base <= a.n_slots; base += 32) {
            const int i = base + tid;
            int v = i <= a.n_slots ? pre[i] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, v, o); if (tid >= o) v += u; }
            if (i <= a.n_slots) pre[i] = v + carry;
            carry += __shfl_sync(0xffffffffu, v, 31);
        }
    }
    __syncthreads();
    const long long W = pre[a.n_slots];
    if (a.chunked && (n_chunks <= max_cta || (n_chunks <= list_cap && W >= 2LL * n_chunks))) {   // a list of chunks
        if (a.n_slots <= LIST_SLOTS) {
            if (tid < a.n_slots) { const int n = (pre[tid + 1] - pre[tid]) * TILE; cseg[tid] = n > 0 ? chunk_of(a.CH, n - 1) + 1 : 0; }
            __syncthreads();
            for (int s = 0; s < a.n_slots; ++s)
                for (int c = tid; c < cseg[s]; c += SPLIT_THR) {
                    int o = 0;   // chunks of a higher index, and of this index in earlier slots
                    for (int r = 0; r < a.n_slots; ++r) o += max(0, cseg[r] - 1 - c) + (r < s && cseg[r] > c);
                    segs[o] = make_int4(s, (int) chunk_lo(a.CH, c), (int) min((long long) (pre[s + 1] - pre[s]) * TILE, chunk_lo(a.CH, c + 1)), 0);
                }
        } else {   // a CTA each: in any order
            if (tid == 0) cseg[0] = 0;
            __syncthreads();
            for (int s = tid; s < a.n_slots; s += SPLIT_THR) {
                const int n = (pre[s + 1] - pre[s]) * TILE, k = n > 0 ? chunk_of(a.CH, n - 1) + 1 : 0;
                int o = k ? atomicAdd(&cseg[0], k) : 0;
                for (int c = 0; c < k; ++c, ++o) segs[o] = make_int4(s, (int) chunk_lo(a.CH, c), (int) min((long long) n, chunk_lo(a.CH, c + 1)), 0);
            }
        }
        if (tid == 0) *n_cta_out = -n_chunks;
        return;
    }
    const int n_cta = (int) max(1LL, min((long long) min(max_cta, SPLIT_MAX_CTA), W / min_tiles));
    if (tid <= n_cta) {
        int x = (int) (W * tid / n_cta);
        if (a.chunked && tid > 0 && tid < n_cta) {
            int l = 0, r = a.n_slots;               // last slot with pre[s] <= x
            while (r - l > 1) { const int m = (l + r) >> 1; if (pre[m] <= x) l = m; else r = m; }
            const int len = pre[l + 1] - pre[l], off = x - pre[l];   // x < W, so off < len
            const int c = chunk_of(a.CH, off * TILE);
            const int lo = (int) (chunk_lo(a.CH, c) / TILE), hi = (int) min((long long) len, chunk_lo(a.CH, c + 1) / TILE);
            x = pre[l] + (off - lo <= hi - off ? lo : hi);
        }
        scut[tid] = x;
    }
    __syncthreads();
    auto cut = [&](int c) { return scut[c]; };
    // segments per CTA: the slots its run intersects
    int my_first = 0, my_cnt = 0;
    if (tid < n_cta) {
        const int lo = cut(tid), hi = cut(tid + 1);
        if (hi > lo) {
            int l = 0, r = a.n_slots;               // last slot with pre[s] <= lo
            while (r - l > 1) { const int m = (l + r) >> 1; if (pre[m] <= lo) l = m; else r = m; }
            while (pre[l + 1] <= lo) ++l;           // skip empty slots
            my_first = l;
            int e = l;
            while (e < a.n_slots && pre[e] < hi) { if (pre[e + 1] > pre[e] && pre[e + 1] > lo) ++my_cnt; ++e; }
        }
        first_slot[tid] = (short) my_first;
        cseg[tid + 1] = my_cnt;
    }
    if (tid == 0) cseg[0] = 0;
    __syncthreads();
    if (tid < 32) {
        int carry = 0;
        for (int base = 1; base <= n_cta; base += 32) {
            const int i = base + tid;
            int v = i <= n_cta ? cseg[i] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, v, o); if (tid >= o) v += u; }
            if (i <= n_cta) cseg[i] = v + carry;
            carry += __shfl_sync(0xffffffffu, v, 31);
        }
    }
    __syncthreads();
    if (tid <= n_cta) cta_seg[tid] = cseg[tid];
    if (tid == 0) *n_cta_out = W > 0 ? n_cta : 0;
    if (tid < n_cta && my_cnt > 0) {
        const int lo = cut(tid), hi = cut(tid + 1);
        int o = cseg[tid];
        for (int s = my_first; s < a.n_slots && pre[s] < hi; ++s) {
            if (pre[s + 1] <= pre[s] || pre[s + 1] <= lo) continue;
            const int t0 = max(lo, pre[s]) - pre[s], t1 = min(hi, pre[s + 1]) - pre[s];
            segs[o++] = make_int4(s, t0 * TILE, t1 * TILE, 0);
        }
    }
    if (a.chunked) return;   // a chunk's partial has its own place
    // the segments of a slot are consecutive: from the CTA that holds its first tile to the one that holds its last
    for (int s = tid; s < a.n_slots; s += SPLIT_THR) {
        if (pre[s + 1] <= pre[s]) { slot_seg[s] = make_int2(0, 0); continue; }
        auto cta_of = [&](int tile) {
            int c = (int) min((long long) n_cta - 1, ((long long) tile * n_cta) / max(W, 1LL));
            while (c > 0 && cut(c) > tile) --c;
            while (c + 1 < n_cta && cut(c + 1) <= tile) ++c;
            return c;
        };
        const int c0 = cta_of(pre[s]), c1 = cta_of(pre[s + 1] - 1);
        // inside CTA c0 the slot's segment comes after those of the non-empty slots first_slot[c0] .. s-1
        int before = 0;
        for (int z = first_slot[c0]; z < s; ++z) if (pre[z + 1] > pre[z] && pre[z + 1] > cut(c0)) ++before;
        slot_seg[s] = make_int2(cseg[c0] + before, c1 - c0 + 1);
    }
}

// ------------------------------------------------------------------------------------------------ host side ----
constexpr int DEFAULT_CHUNK = 512;
constexpr int MAX_DEFAULT_CHUNKS = 256;   // the default chunk grows with n_ctx so that a context never has more chunks than this
int g_chunk = 0;            // 0 = not read yet; else B200ATTN_CHUNK or DEFAULT_CHUNK
bool g_chunk_from_env = false;
int g_nsplit_override = 0;  // set_nsplit: chunks per full context

int round_tile(long long v) { return (int) ((std::max<long long>(v, TILE) + TILE - 1) / TILE * TILE); }
int env_chunk(bool * from_env) {
    const char * e = getenv("B200ATTN_CHUNK");
    const bool have = e && *e && atoi(e) > 0;
    if (from_env) *from_env = have;
    return round_tile(have ? atoi(e) : DEFAULT_CHUNK);
}
int default_chunk() {
    if (!g_chunk) g_chunk = env_chunk(&g_chunk_from_env);
    return g_chunk;
}
// Chunks of the calls that name none: functions of the cache's capacity and of settings only, so that a row's bits do not depend on the
// batch it is decoded in.  set_nsplit(n) pins n chunks per full context, B200ATTN_CHUNK pins the keys, for both grids.
int pinned_chunk(int n_ctx) {
    const int base = default_chunk();
    if (g_nsplit_override > 0) return round_tile(((long long) std::max(n_ctx, 1) + g_nsplit_override - 1) / g_nsplit_override);
    return g_chunk_from_env ? base : 0;
}
// Batched entry points with chunk_keys = 0.  A batch fills the chip with long chunks, and every chunk costs its partials: with the
// position grid 64 slots x 4 rows at 4096 keys (q8_0, 4 kv heads) take 441 us against 214, 8 x 1 rows 37 against 29, and eight times the scratch.
int fixed_chunk(int n_ctx) {
    const int pinned = pinned_chunk(n_ctx);
    return pinned ? pinned : std::max(default_chunk(), round_tile(((long long) std::max(n_ctx, 1) + MAX_DEFAULT_CHUNKS - 1) / MAX_DEFAULT_CHUNKS));
}
// Row entry points (attn_decode and its kin, at most 8 rows): the position grid, whose longest chunk is
// 512 keys up to a capacity of 229376 and n_ctx / 448 rounded up to a power of two beyond.  One row, 4 heads, chunks of up to 512 / 1024 keys: q4_0 at
// 65664 of 131328 keys 44.7 / 54.5 us, q8_0 48.6 / 61.1 (the longest CTA walks 8 or 16 tiles); q4_0 at 262141 of 262144 125.9 / 115.1, at half of it
// 70.2 / 76.2.
int position_grid(int n_ctx) {
    const int pinned = pinned_chunk(n_ctx);
    if (pinned) return pinned;
    int k = 3;
    while (((long long) 448 * TILE << k) < n_ctx) ++k;
    return -k;
}

// Split partials and the run plan live in one library-owned buffer per (device, stream), as in the reference
// (src/fast/attn_dec2.cu:452-464,503-517): sized on the first call or by b200_attn_reserve, and from then on calls that
// fit neither allocate nor synchronise, and the pointer does not move (recorded work stays valid).  A call that needs more
// gets a new, larger buffer; the old one is kept allocated until the process exits, so nothing that was recorded against
// it ever reads freed memory, and no stream is synchronised.
// A run plan depends on the rows' positions only, which a model step does not change from layer to layer.
// Between b200_attn_step_begin(stream, positions, bytes) and the next one (or b200_attn_step_end) the plan that the first
// batched call of a given shape, with its positions inside the declared array, leaves in the stream's scratch is used again by
// the following calls of the same shape instead of being recomputed: what identifies the plan is kept here, and any other
// call on the stream drops it.  A recorded call's plan does not exist until the recording is replayed, and a replay comes with
// positions of its own, so a plan serves only calls of the recording it was recorded in (`rec`), or only calls outside of any.  Plans
// of recorded calls and of the others have a place each at the front of the buffer, away from all partials: a replay between two
// calls of a step leaves their plan alone.
struct plan_key {
    unsigned long long rec = 0;

    const void * scr = nullptr, * pos = nullptr, * p0p = nullptr;
    int p0 = 0, n_slots = 0, q_len = 0, CH = 0, max_chunks = 0, max_cta = 0, Hkv = 0, n_ctx = 0, paged = 0;
    int list_cap = 0, split = 0, tc = 0;   // an even split has slot_seg, a plan of fixed chunks has not; they can agree in all the rest
    size_t part_floats = 0;
    bool operator==(const plan_key & o) const {
        return rec == o.rec && scr == o.scr && pos == o.pos && p0p == o.p0p && p0 == o.p0 && n_slots == o.n_slots && q_len == o.q_len && CH == o.CH &&
               max_chunks == o.max_chunks && max_cta == o.max_cta && Hkv == o.Hkv && n_ctx == o.n_ctx && paged == o.paged && list_cap == o.list_cap && split == o.split && tc == o.tc &&
               part_floats == o.part_floats;
    }
};
// the longest plan (run_list_ints), in whole 256-byte units
constexpr int SCR_PLAN_INTS = (6 * PLAN_MAX_SLOTS + 5 * SPLIT_MAX_CTA + 4 + 63) / 64 * 64;
struct scratch {
    int dev = -1; cudaStream_t s = nullptr; float * p = nullptr; size_t cap = 0;
    bool step_mode = false, plan_valid = false;
    const char * step_lo = nullptr, * step_hi = nullptr;   // the position array the caller declared fixed for the step
    plan_key key;
};
scratch g_scr[64];
int g_nscr = 0;
std::mutex g_mu;

// `floats`: partials of the call (0: no buffer is needed)
scratch * scratch_entry(cudaStream_t s, size_t floats, size_t floats_hint) {
    if (floats) floats += 2 * SCR_PLAN_INTS;
    if (floats_hint) floats_hint += 2 * SCR_PLAN_INTS;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_mu);
    scratch * e = nullptr;
    for (int i = 0; i < g_nscr; ++i) if (g_scr[i].dev == dev && g_scr[i].s == s) e = &g_scr[i];
    if (!e) {
        if (g_nscr == 64) return nullptr;
        e = &g_scr[g_nscr++];
        e->dev = dev; e->s = s;
    }
    if (floats > e->cap) {
        const size_t want = std::max(std::max(floats, floats_hint), std::max(e->cap + e->cap / 2, (size_t) 1 << 20));
        float * p = nullptr;
        if (cudaMalloc(&p, want * sizeof(float)) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        e->p = p;      // the previous buffer, if any, stays allocated (see above)
        e->cap = want;
        e->plan_valid = false;
    }
    return e;
}
float * scratch_for(cudaStream_t s, size_t floats, size_t floats_hint) {
    scratch * e = scratch_entry(s, floats, floats_hint);
    return e ? e->p : nullptr;
}

// ---- tensor maps of the cache ----------------------------------------------------------------------------------
// K and V as rank-3 tensors of 16-bit elements: x = the row of one position (all kv heads), y = position inside a page
// (or in the whole cache when it is contiguous), z = page.  The box is one head's bytes of 64 consecutive positions.
// f16 rows (512 B per head) are wider than a box may be, and their shared-memory image is swizzled: rank 4 with x = 64
// elements (128 B), y = position, z = 128-byte chunk of the row, w = page; box = 64 x 64 x 4 chunks, 128-byte swizzle.
using encode_tiled_fn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                     const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                     CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
encode_tiled_fn tensor_map_encoder() {
    static encode_tiled_fn fn = [] {
        void * p = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &r) != cudaSuccess || r != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return (encode_tiled_fn) p;
    }();
    return fn;
}
// Encoding a map is pure host arithmetic on (base, geometry); the last few are kept, since a serving loop calls with the
// same caches (one K and one V per layer) every step.
struct map_entry { const char * base; unsigned long long rowb, pstride, rows; int HB, box_rows; bool paged; CUtensorMap m; };
constexpr int MAP_CACHE = 256;
map_entry g_maps[MAP_CACHE];
int g_nmaps = 0, g_map_next = 0;
std::mutex g_map_mu;

bool make_cache_map(CUtensorMap * m, const char * base, const dec_args & a, int HB, int box_rows = TILE) {
    encode_tiled_fn enc = tensor_map_encoder();
    if (!enc) return false;
    const bool paged = a.g.pt != nullptr;
    const cuuint64_t rows = paged ? (cuuint64_t) 1 << a.g.psh : (cuuint64_t) a.n_ctx;
    const unsigned long long pstr = paged ? a.g.pstride : 0;
    {
        std::lock_guard<std::mutex> lk(g_map_mu);
        for (int i = 0; i < g_nmaps; ++i) {
            const map_entry & e = g_maps[i];
            if (e.base == base && e.rowb == a.g.rowb && e.pstride == pstr && e.rows == rows && e.HB == HB && e.box_rows == box_rows && e.paged == paged) {
                *m = e.m;
                return true;
            }
        }
    }
    const cuuint64_t npages = paged ? (cuuint64_t) 0x7fffffff : 1, pbytes = paged ? a.g.pstride : a.g.rowb * rows;
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult rc;
    if (HB == head_bytes(B200_KV_F16)) {
        const cuuint64_t gdim[4] = {64, rows, a.g.rowb / 128, npages};
        const cuuint64_t gstr[3] = {a.g.rowb, 128, pbytes};
        const cuuint32_t box[4] = {64, (cuuint32_t) TILE, 4, 1};
        rc = enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT16, 4, (void *) base, gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                 CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    } else {
        const cuuint64_t gdim[3] = {a.g.rowb / 2, rows, npages};
        const cuuint64_t gstr[2] = {a.g.rowb, pbytes};
        const cuuint32_t box[3] = {(cuuint32_t) HB / 2, (cuuint32_t) box_rows, 1};
        rc = enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, (void *) base, gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                 CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    if (rc != CUDA_SUCCESS) return false;
    std::lock_guard<std::mutex> lk(g_map_mu);
    map_entry & e = g_maps[g_map_next];
    g_map_next = (g_map_next + 1) % MAP_CACHE;
    if (g_nmaps < MAP_CACHE) ++g_nmaps;
    e.base = base; e.rowb = a.g.rowb; e.pstride = pstr; e.rows = rows; e.HB = HB; e.box_rows = box_rows; e.paged = paged; e.m = *m;
    return true;
}

template <uint32_t KT, int NT> size_t smem_bytes(int nslot) {
    return HDR + (size_t) nslot * traits<KT>::SLOT + NT * 8 * (QSTR + PSTR) + 8 * SDSTR + 2 * NWARP * NT * 8 * sizeof(float) +
           (traits<KT>::SCALED ? NBLK * NT * 4 * sizeof(float4) : 0);
}

template <uint32_t KT, int NT, bool RUNS>
int launch_part(const dec_args & a_in, unsigned blocks, cudaStream_t s) {
    dec_args a = a_in;
    CUtensorMap mapK, mapV;
    memset(&mapK, 0, sizeof mapK);
    memset(&mapV, 0, sizeof mapV);
    // tiled copies need a tile inside one page (pages of at least 64 rows), 16-byte row strides and a contiguous cache short
    // enough for the stride field; anything else keeps the row-by-row copies
    a.tiled = 0;
    if ((!a.g.pt || a.g.psh >= 6) && a.g.rowb % 16 == 0 &&
        (a.g.pt ? a.g.pstride < ((unsigned long long) 1 << 40) : (a.n_ctx >= 1 && a.g.rowb * (unsigned long long) a.n_ctx < ((unsigned long long) 1 << 40))))
        a.tiled = make_cache_map(&mapK, a.g.k, a, traits<KT>::HB) && make_cache_map(&mapV, a.g.v, a, traits<KT>::HB);
    // as many CTAs per SM as the kernel is compiled for, if a ring of two half-tile slots fits that often into the 227 KB of
    // an SM; then the deepest ring (up to 8 slots) that still fits
    auto fits = [](int n, int ctas) { return (size_t) ctas * (smem_bytes<KT, NT>(n) + 1024) <= (size_t) 227 * 1024; };
    int ctas = ctas_per_sm<KT, NT>();
    while (ctas > 1 && !fits(2, ctas)) --ctas;
    int nslot = 2;
    while (nslot < 8 && fits(nslot + 1, ctas)) ++nslot;
    const size_t sm = smem_bytes<KT, NT>(nslot);
    static std::atomic<bool> attr_done[64];   // per instantiation and device; setting the attribute twice is harmless
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_done[dev & 63].load(std::memory_order_acquire)) {
        if (cudaFuncSetAttribute(decode_part_k<KT, NT, RUNS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sm) != cudaSuccess)
            return launch_status("attn_decode (shared memory attribute)");
        cudaFuncSetAttribute(decode_part_k<KT, NT, RUNS>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        attr_done[dev & 63].store(true, std::memory_order_release);
    }
    decode_part_k<KT, NT, RUNS><<<blocks, NTHR, sm, s>>>(a, nslot, mapK, mapV);
    return B200_OK;
}

template <uint32_t KT, int NT>
int launch_warp(const dec_args & a_in, unsigned runs, cudaStream_t s) {
    dec_args a = a_in;
    CUtensorMap mapK, mapV;
    memset(&mapK, 0, sizeof mapK);
    memset(&mapV, 0, sizeof mapV);
    a.tiled = 0;
    if ((!a.g.pt || a.g.psh >= 6) && a.g.rowb % 16 == 0 &&
        (a.g.pt ? a.g.pstride < ((unsigned long long) 1 << 40) : (a.n_ctx >= 1 && a.g.rowb * (unsigned long long) a.n_ctx < ((unsigned long long) 1 << 40))))
        a.tiled = make_cache_map(&mapK, a.g.k, a, traits<KT>::HB, WT) && make_cache_map(&mapV, a.g.v, a, traits<KT>::HB, WT);
    constexpr size_t sm = wk<KT, NT>::smem(wk<KT, NT>::slots());
    static std::atomic<bool> attr_done[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_done[dev & 63].load(std::memory_order_acquire)) {
        if (cudaFuncSetAttribute(decode_warp_k<KT, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sm) != cudaSuccess)
            return launch_status("attn_decode (shared memory attribute)");
        cudaFuncSetAttribute(decode_warp_k<KT, NT>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        attr_done[dev & 63].store(true, std::memory_order_release);
    }
    decode_warp_k<KT, NT><<<(runs + 1) / 2, WK_THR, sm, s>>>(a, (int) runs, mapK, mapV);
    return B200_OK;
}
template <uint32_t KT, bool RUNS>
int launch_part_runs(const dec_args & a, unsigned blocks, cudaStream_t s) {
    const int nt = (a.q_len * GQA + 7) / 8;
    return nt == 1 ? launch_part<KT, 1, RUNS>(a, blocks, s) : nt == 2 ? launch_part<KT, 2, RUNS>(a, blocks, s) : launch_part<KT, 3, RUNS>(a, blocks, s);
}
template <uint32_t KT>
int launch_part_nt(const dec_args & a, unsigned blocks, cudaStream_t s) {
    return a.chunked && a.segs ? launch_part_runs<KT, true>(a, blocks, s) : launch_part_runs<KT, false>(a, blocks, s);
}

// whole tiles can be fetched through tensor maps: pages of at least 64 rows, 16-byte row strides, strides inside the map's fields
bool cache_tiles(const kv_view & g, int n_ctx) {
    return (!g.pt || g.psh >= 6) && g.rowb % 16 == 0 &&
           (g.pt ? g.pstride < ((unsigned long long) 1 << 40) : (n_ctx >= 1 && g.rowb * (unsigned long long) n_ctx < ((unsigned long long) 1 << 40)));
}
// The tensor-core kernel serves the even split of q8_0 caches that can be tiled, for two to four rows per slot (one row
// per slot and q4_0 are faster on the mma.sync kernel: their tiles cost fewer instructions there); B200ATTN_TC=0 keeps the
// mma.sync kernel everywhere.
int g_tc = -1;   // -1 = not read yet
bool tc_enabled() {
    if (g_tc < 0) { const char * e = getenv("B200ATTN_TC"); g_tc = (e && *e == '0') ? 0 : 1; }
    return g_tc != 0;
}
bool tc_eligible(const b200_kv_cache & c, int q_len) {
    return tc_enabled() && c.type == B200_KV_Q8_0 && q_len >= 2 && cache_tiles(view_of(c), c.n_ctx) && tensor_map_encoder() != nullptr;
}

template <int NC, bool EX>
int launch_tc(const dec_args & a_in, unsigned blocks, cudaStream_t s) {
    dec_args a = a_in;
    CUtensorMap mapK, mapV;
    memset(&mapK, 0, sizeof mapK);
    memset(&mapV, 0, sizeof mapV);
    if (!make_cache_map(&mapK, a.g.k, a, TC_HB) || !make_cache_map(&mapV, a.g.v, a, TC_HB))
        B200_REFUSE(B200_ERR_CUDA, "attn_decode: the cache's tensor map could not be encoded");
    a.tiled = 1;
    constexpr size_t sm = tc_smem_bytes(EX);
    static std::atomic<bool> attr_done[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_done[dev & 63].load(std::memory_order_acquire)) {
        if (cudaFuncSetAttribute(decode_tc_k<NC, EX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sm) != cudaSuccess)
            return launch_status("attn_decode (shared memory attribute)");
        attr_done[dev & 63].store(true, std::memory_order_release);
    }
    // a step of few rows is short enough for the gap before the kernel to count
    if (a.n_slots * a.q_len <= 64) launch(decode_tc_k<NC, EX>, blocks, TC_THR, sm, s, a, mapK, mapV);
    else decode_tc_k<NC, EX><<<blocks, TC_THR, sm, s>>>(a, mapK, mapV);
    return B200_OK;
}
int launch_tc_nc(const dec_args & a, unsigned blocks, cudaStream_t s) {
    if (a.solo) return a.q_len <= 2 ? launch_tc<16, true>(a, blocks, s) : launch_tc<32, true>(a, blocks, s);
    return a.q_len <= 2 ? launch_tc<16, false>(a, blocks, s) : launch_tc<32, false>(a, blocks, s);
}

int sm_count() {
    int sms = 148, dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// CTAs of decode_part_k<type, row tiles> that fit an SM at once (the same rule as launch_part)
template <uint32_t KT, int NT> int ctas_fitting() {
    int ctas = ctas_per_sm<KT, NT>();
    while (ctas > 1 && (size_t) ctas * (smem_bytes<KT, NT>(2) + 1024) > (size_t) 227 * 1024) --ctas;
    return ctas;
}
template <uint32_t KT> int ctas_fitting_nt(int nt) { return nt == 1 ? ctas_fitting<KT, 1>() : nt == 2 ? ctas_fitting<KT, 2>() : ctas_fitting<KT, 3>(); }
int resident_ctas(uint32_t type, int q_len) {
    const int nt = (q_len * GQA + 7) / 8;
    const int per_sm = type == B200_KV_F16 ? ctas_fitting_nt<B200_KV_F16>(nt) : type == B200_KV_Q8_0 ? ctas_fitting_nt<B200_KV_Q8_0>(nt)
                                                                                                 : ctas_fitting_nt<B200_KV_Q4_0>(nt);
    return per_sm * sm_count();
}

// runs of decode_warp_k that fit the GPU at once, 0 = not its call.  q4_0: only where the runs may be two tiles long.  Shorter ones have nothing to
// amortise and half the warps per run: 9 slots of up to 3433 keys, two layers, 79 us for 74 (8 slots x 2 rows of 2839 keys 94 for 88); 40 slots of
// 13880 keys 377 for 419.
int warp_runs(uint32_t type, int n_slots, int q_len, int max_n, int Hkv) {
    if (type == B200_KV_Q8_0) return q_len == 1 ? 2 * wk<B200_KV_Q8_0, 1>::CTAS * sm_count() : 0;
    if (type != B200_KV_Q4_0 || q_len > 2) return 0;
    const int n = 2 * (q_len == 1 ? wk<B200_KV_Q4_0, 1>::CTAS : wk<B200_KV_Q4_0, 2>::CTAS) * sm_count();
    return (long long) n_slots * ((max_n + TILE - 1) / TILE) * Hkv >= 2LL * n ? n : 0;
}

int auto_chunk(long long total_keys, int Hkv) {
    // enough units for several waves over the SMs, chunks between 256 and 4096 keys
    const long long units = 8LL * sm_count();
    long long ch = total_keys * Hkv / units;
    int c = 256;
    while (c < 4096 && c < ch) c *= 2;
    return c;
}

// One slot: the position grid up to auto_chunk's chunk, which short contexts need to fill the chip; a long one in equal chunks.  4 rows of
// 2 heads, q8_0, 30011 keys: 29.9 us, with the row entry points' grid (chunks of up to 512 keys) 36.5; 131000 keys 66.9 and 62.1.
int single_grid(int max_n, int Hkv) {
    const int c = auto_chunk(max_n / 2, Hkv);
    int k = 0;
    while (TILE << k < c) ++k;
    return max_n > 65536 ? c : -k;
}

// geometry of a call: chunk, chunks per slot, partial floats, work-list ints
//   split   (chunk chosen from the batch, two to SPLIT_MAX_SLOTS slots; one slot for decode_tc_k): one contiguous run of tiles per resident CTA
//   planned (fixed chunks of several slots, more units than a wave): the same runs, cut at chunk boundaries
//   else    see decode_part_k
// rows: a call of the row entry points (chunk_keys = 0: the position grid).
// One slot with chunk_keys < 0: two to four rows of a q8_0 cache run on decode_tc_k in its exact form (K as integers, references renewed every 256 keys),
// which is no further from 64-bit attention than chunks of 256 keys on decode_part_k (4 rows, 30011 / 65536 keys: 3.48e-4 / 3.50e-4 against 3.54e-4);
// 16 layers of 1 + 3 rows at 30011 keys, two heads, 587 -> 443 us, 8 layers at 1500 keys 159 -> 139, at 130000 (four heads) 1029 -> 694.  All else stays on decode_part_k in
// chunks (single_grid) that are nowhere longer than auto_chunk's.
//   the plan holds `segs` segments, the runs' or (listed) every chunk
size_t run_list_ints(size_t segs, int max_cta, int n_slots) { return (4 * segs + 2 * (size_t) n_slots + max_cta + 2 + 3) & ~(size_t) 3; }
static_assert(SCR_PLAN_INTS >= 4 * (SPLIT_MAX_CTA + PLAN_MAX_SLOTS) + 2 * PLAN_MAX_SLOTS + SPLIT_MAX_CTA + 2 &&
              SCR_PLAN_INTS >= 4 * LIST_MAX + 2 * LIST_SLOTS + SPLIT_MAX_CTA + 4, "a plan fits its place");
// the recording the stream takes part in, 0 if none; false = unknown
bool recording_of(cudaStream_t s, unsigned long long & id) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamGetCaptureInfo(s, &st, &id) != cudaSuccess) { cudaGetLastError(); return false; }
    if (st == cudaStreamCaptureStatusNone) id = 0;
    return st != cudaStreamCaptureStatusInvalidated;
}
struct dec_geom { int CH, max_chunks, R, max_cta, list_cap; size_t units, segs, part_floats, list_ints; bool planned, split, tc, warp; };

bool decode_geometry(dec_geom & g, uint32_t type, int n_slots, int q_len, int max_n, int n_ctx, int Hkv, int chunk_keys, bool tc = false, bool rows = false, bool warp = true) {
    if (max_n < 1) max_n = 1;
    g.tc = g.warp = false;
    g.R = q_len * GQA;
    g.split = chunk_keys < 0 && (n_slots > 1 || (tc && type == B200_KV_Q8_0 && q_len >= 2)) && n_slots <= SPLIT_MAX_SLOTS;
    g.planned = false;
    g.max_cta = g.list_cap = 0;
    if (g.split) {
        g.CH = TILE;
        g.max_chunks = (max_n + TILE - 1) / TILE;
        g.tc = tc && type == B200_KV_Q8_0 && q_len >= 2;   // the tensor-core kernel: one CTA per SM
        const int runs = g.tc || !warp ? 0 : warp_runs(type, n_slots, q_len, max_n, Hkv);
        g.warp = runs > 0;
        g.max_cta = std::max(1, std::min(SPLIT_MAX_CTA, (g.tc ? sm_count() : g.warp ? runs : resident_ctas(type, q_len)) / Hkv));
        g.segs = (size_t) g.max_cta + n_slots;
        g.units = g.segs * Hkv;
        g.part_floats = g.units * g.R * (DH + 2);
        g.list_ints = n_slots > 1 ? run_list_ints(g.segs, g.max_cta, n_slots) : 0;
        return true;
    }
    g.CH = chunk_keys > 0 ? round_tile(chunk_keys) : chunk_keys < 0 && n_slots > 1 ? auto_chunk((long long) n_slots * max_n / 2, Hkv) :
           chunk_keys < 0 ? single_grid(max_n, Hkv) : rows ? position_grid(n_ctx) : fixed_chunk(n_ctx);
    g.max_chunks = chunk_of(g.CH, max_n - 1) + 1;
    g.units = (size_t) n_slots * Hkv * g.max_chunks;
    if (g.units >= ((size_t) 1 << 31) || (size_t) n_slots * g.max_chunks >= ((size_t) 1 << 30)) return false;
    g.part_floats = g.units * g.R * (DH + 2);
    g.max_cta = std::max(1, std::min(SPLIT_MAX_CTA, resident_ctas(type, q_len) / Hkv));
    // a plan pays once there are more chunks than resident CTAs; fewer are enumerated
    g.planned = n_slots > 1 && n_slots <= PLAN_MAX_SLOTS && (size_t) n_slots * g.max_chunks > (size_t) g.max_cta;
    if (g.planned && type != B200_KV_F16 && n_slots <= LIST_SLOTS && n_slots * g.max_chunks <= LIST_MAX) g.list_cap = n_slots * g.max_chunks;
    g.segs = std::max((size_t) g.max_cta + n_slots, (size_t) g.list_cap);
    g.list_ints = g.planned ? run_list_ints(g.segs, g.max_cta, n_slots) : 0;
    return true;
}

int decode_check(const float * q, const b200_kv_cache * c, const float * out, const float * gate, int n_slots, int q_len, int Hq,
                 const char * who) {
    if (!c || !q || !c->k || !c->v) B200_REFUSE(B200_ERR_SHAPE, "%s: null argument", who);
    if (c->D != DH || Hq != GQA * c->Hkv || c->Hkv <= 0) B200_REFUSE(B200_ERR_SHAPE, "%s: unsupported shape (D=%d Hq=%d Hkv=%d)", who, c->D, Hq, c->Hkv);
    if (c->type != B200_KV_F16 && c->type != B200_KV_Q8_0 && c->type != B200_KV_Q4_0) B200_REFUSE(B200_ERR_SHAPE, "%s: unsupported cache type %u", who, c->type);
    if (n_slots < 1 || n_slots > 65535 || q_len < 1 || q_len > B200_MAX_QLEN) B200_REFUSE(B200_ERR_SHAPE, "%s: unsupported rows (slots=%d q_len=%d)", who, n_slots, q_len);
    if (!aligned16(c->k) || !aligned16(c->v) || !aligned16(q) || (out && !aligned16(out)) || (gate && !aligned16(gate)) ||
        (c->pt && c->pstride % 16))
        B200_REFUSE(B200_ERR_SHAPE, "%s: cache base, page stride, q, out and gate must be 16-byte aligned", who);
    if (c->pt && (c->psh < 0 || c->psh > 30)) B200_REFUSE(B200_ERR_SHAPE, "%s: bad page shift %d", who, c->psh);
    return B200_OK;
}

struct merge_out { float * out; const float * gate; float * fo, * fm, * fl; void * qbuf; };

// the kernels of one call, partials in `scr`, run plan in `list` (nullptr: behind the partials)
int decode_launch(const float * q, const b200_kv_cache * c, const merge_out & mo, int n_slots, int q_len, const int32_t * pos,
                  const int32_t * p0p, int p0, int Hq, float scale, const dec_geom & gm, float * scr, int * list, unsigned * st, cudaStream_t s,
                  const char * who, bool reuse_plan = false, int hk0 = 0, int nhk = 0) {
    dec_args a;
    a.q = q; a.g = view_of(*c);
    const int heads = nhk ? nhk : c->Hkv;
    const size_t units = gm.units / c->Hkv * heads, part_floats = units * gm.R * (DH + 2);
    a.po = scr; a.pm = scr + units * gm.R * DH; a.pl = a.pm + units * gm.R;
    a.pos = pos; a.p0p = p0p; a.p0 = p0;
    a.q_len = q_len; a.n_slots = n_slots; a.Hq = Hq;
    a.qscale = scale * LOG2E;
    a.CH = gm.CH; a.max_chunks = gm.max_chunks; a.status = st;
    a.hk0 = hk0; a.nhk = heads;
    a.n_ctx = c->n_ctx; a.tiled = 0;
    a.chunked = gm.split ? 0 : 1;
    a.segs = nullptr; a.cta_seg = nullptr; a.slot_seg = nullptr; a.n_cta = nullptr;
    a.solo = gm.split && n_slots == 1 ? gm.max_cta : 0;
    a.max_cta = gm.max_cta;
    int launches = 2;
    // fixed chunks without a plan: at most one wave of CTAs, a multiple of the heads
    unsigned blocks = (unsigned) std::min<size_t>((size_t) n_slots * gm.max_chunks, (size_t) gm.max_cta) * (unsigned) a.nhk;
    if (a.solo) blocks = (unsigned) gm.max_cta * (unsigned) a.nhk;
    else if (gm.split || gm.planned) {
        if (!list) list = reinterpret_cast<int *>(scr + part_floats);
        int4 * segs = reinterpret_cast<int4 *>(list);
        int2 * slot_seg = reinterpret_cast<int2 *>(list + 4 * gm.segs);
        int * cta_seg = list + 4 * gm.segs + 2 * (size_t) n_slots;
        int * n_cta = cta_seg + gm.max_cta + 1;
        a.segs = segs; a.cta_seg = cta_seg; a.slot_seg = slot_seg; a.n_cta = n_cta;
        if (!reuse_plan) {   // else the lists of an earlier call of this step, same shape, same positions, are still there
            launch(decode_split_k, 1, SPLIT_THR, 0, s, a, gm.max_cta, gm.list_cap, gm.tc ? 2 : 1, segs, cta_seg, slot_seg, n_cta);
            ++launches;
        }
        // a list is dealt out to up to four waves of CTAs; CTAs without a chunk come last and leave at once
        blocks = (unsigned) (gm.list_cap ? std::min(gm.list_cap, 4 * gm.max_cta) : gm.max_cta) * (unsigned) a.nhk;
    }
    int rc;
    if (gm.split && gm.tc) rc = launch_tc_nc(a, blocks, s);
    else if (c->type == B200_KV_F16) rc = launch_part_nt<B200_KV_F16>(a, blocks, s);
    else if (gm.warp) rc = c->type == B200_KV_Q8_0 ? launch_warp<B200_KV_Q8_0, 1>(a, blocks, s) : q_len == 1 ? launch_warp<B200_KV_Q4_0, 1>(a, blocks, s) : launch_warp<B200_KV_Q4_0, 2>(a, blocks, s);
    else if (c->type == B200_KV_Q8_0) rc = launch_part_nt<B200_KV_Q8_0>(a, blocks, s);
    else rc = launch_part_nt<B200_KV_Q4_0>(a, blocks, s);
    if (rc != B200_OK) return rc;
    // Few partials (of a typical slot): one group of threads per (row, head), for fixed chunks on grids beyond eight CTAs per SM up to one
    // chunk per stream.  Measured, us, with one group / 256 threads: 8 partials on 24 (row, head) pairs 6.6 / 5.2, on 6144 17.3 / 36.2.  Eight partials of a stream
    // at once cost occupancy: 118 partials of 48 pairs (16 layers, 609 at the start) 595, with four 601; up to 128 of 192 pairs 341 and 331.
    const int parts = gm.split ? gm.max_cta / n_slots + 2 : gm.max_chunks, sms = sm_count();
    const dim3 mg(n_slots * q_len, GQA * a.nhk);
    const long long grid = (long long) mg.x * mg.y;
    const bool one = gm.split ? parts <= 8 : parts <= 4 || (parts <= MERGE_STREAMS && grid > 8LL * sms);
    if (one) launch(gm.split ? decode_merge_k<false> : decode_merge_k<true>, mg, 64, 0, s, a, mo.gate, mo.out, mo.fo, mo.fm, mo.fl, (__half2 *) mo.qbuf);
    // (early up to eight CTAs per SM: they are small and behind kernels of one wave; 768 CTAs, four layers of 8 rows of up to
    // 16384 keys 306 -> 302 us, of up to 4000 keys 158 -> 149)
    else launch_if(grid * (DH / 4 / MERGE_DL) < 2 * (long long) PDL_MAX_CTAS, parts > 4 * MERGE_STREAMS && grid * (DH / 4 / MERGE_DL) <= 2LL * sms ? decode_merge_streams_k<8> : decode_merge_streams_k<4>, dim3(mg.x, mg.y, DH / 4 / MERGE_DL), MERGE_THR, 0, s, a, mo.gate, mo.out, mo.fo, mo.fm, mo.fl, (__half2 *) mo.qbuf);
    count_launch(launches);
    return launch_status(who);
}

}  // namespace

// q [rows][Hq][256]; rows = n_slots * q_len. Exactly one of (pos), (p0p), (p0) gives the positions.
// hint_floats: size the library scratch for at least this much when it has to be (re)allocated.  rows: a call of the row entry points (decode_geometry).
int decode_impl(const float * q, const b200_kv_cache * c, const merge_out & mo, int n_slots, int q_len, const int32_t * pos,
                const int32_t * p0p, int p0, int max_n, int Hq, float scale, int chunk_keys, cudaStream_t s, const char * who,
                size_t hint_floats = 0, bool rows = false) {
    const int chk = decode_check(q, c, mo.out, mo.gate, n_slots, q_len, Hq, who);
    if (chk != B200_OK) return chk;
    if (mo.qbuf && (!mo.out || ((uintptr_t) mo.qbuf & 3))) B200_REFUSE(B200_ERR_SHAPE, "%s: the a16 buffer needs out and 4-byte alignment", who);
    dec_geom gm;
    if (!decode_geometry(gm, c->type, n_slots, q_len, max_n, c->n_ctx, c->Hkv, chunk_keys, tc_eligible(*c, q_len), rows)) B200_REFUSE(B200_ERR_SHAPE, "%s: too many chunks", who);
    scratch * e = scratch_entry(s, gm.part_floats, hint_floats);
    if (!e || !e->p) B200_REFUSE(B200_ERR_ALLOC, "%s: split scratch (%zu floats) could not be allocated", who, gm.part_floats);
    float * scr = e->p + 2 * SCR_PLAN_INTS;
    unsigned * st = device_status_word();
    if (!st) return B200_ERR_CUDA;
    plan_key k;
    k.scr = scr; k.pos = pos; k.p0p = p0p; k.p0 = p0; k.n_slots = n_slots; k.q_len = q_len; k.CH = gm.CH; k.max_chunks = gm.max_chunks;
    k.max_cta = gm.max_cta; k.Hkv = c->Hkv; k.n_ctx = c->n_ctx; k.paged = c->pt != nullptr; k.part_floats = gm.part_floats;
    k.list_cap = gm.list_cap; k.split = gm.split; k.tc = gm.tc;
    const bool in_step = e->step_mode && pos && (const char *) pos >= e->step_lo && (const char *) pos < e->step_hi;
    const bool listed = (gm.split && n_slots > 1) || gm.planned;
    const bool known = !listed || recording_of(s, k.rec);
    const bool reuse = listed && in_step && known && e->plan_valid && k == e->key;
    int * list = reinterpret_cast<int *>(e->p) + (!known || k.rec ? SCR_PLAN_INTS : 0);
    const int rc = decode_launch(q, c, mo, n_slots, q_len, pos, p0p, p0, Hq, scale, gm, scr, list, st, s, who, reuse);
    e->plan_valid = listed && in_step && known && rc == B200_OK;
    e->key = k;
    return rc;
}

// ---- decode / verify without any allocation --------------------------------------------------------------------
// Same kernels as decode_impl, but the split partials live in a fixed array inside the library image instead of a
// buffer obtained from cudaMalloc.  Every GPU that loads the library carries the array (NOALLOC_BYTES) until the
// process exits.
constexpr size_t NOALLOC_FLOATS = (size_t) 4 << 20;                 // 16 MiB of partials
constexpr size_t NOALLOC_BYTES = NOALLOC_FLOATS * sizeof(float);
static __device__ __align__(256) float g_noalloc_partials[NOALLOC_FLOATS];
static __device__ __align__(256) unsigned g_noalloc_status[64];
struct noalloc_dev { bool ready = false; float * partials = nullptr; unsigned * status = nullptr; };
noalloc_dev g_noalloc[64];
std::mutex g_noalloc_mu;

// In host code the two array names above are host-side handles, not device addresses: the addresses the kernels need are
// looked up once per device, with that device current.
int noalloc_setup(noalloc_dev & out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return B200_ERR_CUDA; }
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    noalloc_dev & e = g_noalloc[dev & 63];
    if (!e.ready) {
        void * p = nullptr, * st = nullptr;
        cudaError_t rc = cudaGetSymbolAddress(&p, g_noalloc_partials);
        if (rc == cudaSuccess) rc = cudaGetSymbolAddress(&st, g_noalloc_status);
        if (rc != cudaSuccess) {
            cudaGetLastError();
            fprintf(stderr, "b200attn: attn_decode_slots_noalloc: cudaGetSymbolAddress failed: %s\n", cudaGetErrorString(rc));
            return B200_ERR_CUDA;
        }
        e.partials = (float *) p;
        e.status = (unsigned *) st;
        e.ready = true;
    }
    out = e;
    return B200_OK;
}

int decode_noalloc_impl(const float * q, const b200_kv_cache * c, float * out, const float * gate, int n_slots, int q_len,
                        const int32_t * pos, int max_n, int Hq, float scale, int chunk_keys, cudaStream_t s) {
    const char * who = "attn_decode_slots_noalloc";
    if (!out || !pos) B200_REFUSE(B200_ERR_SHAPE, "%s: null argument", who);
    const int chk = decode_check(q, c, out, gate, n_slots, q_len, Hq, who);
    if (chk != B200_OK) return chk;
    dec_geom gm;
    bool ok = decode_geometry(gm, c->type, n_slots, q_len, max_n, c->n_ctx, c->Hkv, chunk_keys, tc_eligible(*c, q_len));
    if (ok && gm.warp && gm.part_floats + gm.list_ints > NOALLOC_FLOATS)   // decode_part_k takes fewer runs, and with them partials, of q4_0
        ok = decode_geometry(gm, c->type, n_slots, q_len, max_n, c->n_ctx, c->Hkv, chunk_keys, false, false, false);
    // fixed chunks need no plan; beyond that the kv heads go in as many groups as the array needs (their partials are independent of one another)
    if (ok && gm.planned && gm.part_floats <= NOALLOC_FLOATS && gm.part_floats + gm.list_ints > NOALLOC_FLOATS) { gm.planned = false; gm.list_ints = 0; }
    const size_t per_head = ok ? gm.part_floats / c->Hkv : 0;
    int nhk = ok ? c->Hkv : 0;
    if (ok && gm.part_floats + gm.list_ints > NOALLOC_FLOATS)
        nhk = gm.split || gm.list_ints >= NOALLOC_FLOATS ? 0 : (int) ((NOALLOC_FLOATS - gm.list_ints) / per_head);
    if (nhk < 1)
        B200_REFUSE(B200_ERR_SCRATCH, "%s: %zu bytes of split partials needed (slots %d x kv heads %d x chunks %d x rows %d), the built-in array holds %zu for one kv head at "
                    "least; use a larger chunk_keys or attn_decode_slots", who, (gm.part_floats + gm.list_ints) * sizeof(float), n_slots, c->Hkv, ok ? gm.max_chunks : -1,
                    q_len * GQA, NOALLOC_BYTES);
    noalloc_dev e;
    const int src = noalloc_setup(e);
    if (src != B200_OK) return src;
    const merge_out mo = {out, gate, nullptr, nullptr, nullptr, nullptr};
    for (int h0 = 0; h0 < c->Hkv; h0 += nhk) {
        const int rc = decode_launch(q, c, mo, n_slots, q_len, pos, nullptr, 0, Hq, scale, gm, e.partials, nullptr, e.status, s, who, false, h0, std::min(nhk, c->Hkv - h0));
        if (rc != B200_OK) return rc;
    }
    return B200_OK;
}

}  // namespace b200

using namespace b200;

extern "C" {

// Batched decode / verify for callers that must not allocate device memory.  See include/b200attn.h.
int b200_attn_decode_slots_noalloc(const float * q, const b200_kv_cache * c, float * out, const float * gate, int n_slots,
                                   int q_len, const int32_t * pos, int max_n, int Hq, float scale, int chunk_keys, void * stream) {
    return decode_noalloc_impl(q, c, out, gate, n_slots, q_len, pos, max_n, Hq, scale, chunk_keys, (cudaStream_t) stream);
}

// Status word of the allocation-free entry point on the current device: synchronises the stream, reads the word with a
// symbol copy and clears it with another (neither allocates).  0 = no kernel of that entry point recorded an error.
int b200_noalloc_device_status(void * stream) {
    if (cudaStreamSynchronize((cudaStream_t) stream) != cudaSuccess) return -1;
    unsigned h = 0;
    if (cudaMemcpyFromSymbol(&h, g_noalloc_status, sizeof h) != cudaSuccess) { cudaGetLastError(); return -1; }
    if (h) {
        const unsigned z = 0;
        if (cudaMemcpyToSymbol(g_noalloc_status, &z, sizeof z) != cudaSuccess) { cudaGetLastError(); return -1; }
    }
    return (int) h;
}

int b200_attn_chunk_keys(void) { return default_chunk(); }
int b200_attn_fixed_chunk(int n_ctx) { return fixed_chunk(n_ctx); }

int b200_attn_dec2_nsplit(int Hkv) {
    (void) Hkv;   // the reference derives its stream count from the SM count and Hkv; here the split follows the context
    return g_nsplit_override > 0 ? g_nsplit_override : MAX_DEFAULT_CHUNKS;
}
void b200_attn_dec2_set_nsplit(int n) { g_nsplit_override = n > 0 ? n : 0; }
int b200_attn_step_begin(void * stream, const int32_t * positions, size_t bytes) {
    if (!positions || !bytes) B200_REFUSE(B200_ERR_SHAPE, "attn_step_begin: null position array");
    scratch * e = scratch_entry((cudaStream_t) stream, 0, 0);
    if (!e) B200_REFUSE(B200_ERR_ALLOC, "attn_step_begin: too many (device, stream) pairs");
    e->step_mode = true;
    e->plan_valid = false;
    e->step_lo = (const char *) positions;
    e->step_hi = e->step_lo + bytes;
    return B200_OK;
}
int b200_attn_step_end(void * stream) {
    scratch * e = scratch_entry((cudaStream_t) stream, 0, 0);
    if (!e) return B200_OK;
    e->step_mode = false;
    e->plan_valid = false;
    e->step_lo = e->step_hi = nullptr;
    return B200_OK;
}
int b200_attn_dec_tc(void) { return tc_enabled() ? 1 : 0; }
void b200_attn_dec_set_tc(int on) { g_tc = on < 0 ? -1 : on ? 1 : 0; }
int b200_attn_dec2_reload_env(void) {
    const int before = default_chunk();
    const bool before_env = g_chunk_from_env;
    g_chunk = env_chunk(&g_chunk_from_env);
    return (g_chunk != before || g_chunk_from_env != before_env) ? 1 : 0;
}

int b200_attn_reserve(uint32_t kv_type, int max_slots, int q_len, int max_n, int n_ctx, int Hkv, int chunk_keys, void * stream) {
    if (max_slots < 1 || max_slots > 65535 || q_len < 1 || q_len > B200_MAX_QLEN || max_n < 1 || Hkv < 1 ||
        (kv_type != B200_KV_F16 && kv_type != B200_KV_Q8_0 && kv_type != B200_KV_Q4_0))
        B200_REFUSE(B200_ERR_SHAPE, "attn_reserve: unsupported arguments");
    dec_geom gm;
    if (!decode_geometry(gm, kv_type, max_slots, q_len, max_n, n_ctx > 0 ? n_ctx : max_n, Hkv, chunk_keys)) B200_REFUSE(B200_ERR_SHAPE, "attn_reserve: too many chunks");
    size_t need = gm.part_floats;
    dec_geom g1;   // the position grid of the row entry points, and one slot with -1, may take more partials than a small batch of equal chunks or runs
    if (chunk_keys <= 0 && decode_geometry(g1, kv_type, std::min(max_slots, B200_ATTN_MAX_ROWS), q_len, max_n, n_ctx > 0 ? n_ctx : max_n, Hkv, 0, false, true))
        need = std::max(need, g1.part_floats);
    // one slot of any length up to max_n: most chunks where its chunk is about to double, and at the end of single_grid's fine chunks
    for (long long c = 256; chunk_keys < 0 && c <= 4096; c *= 2)
        for (const long long cap : {(long long) max_n, std::min(65536LL, (long long) max_n)}) {
            const int n1 = (int) std::max(1LL, std::min(cap, (c + 1) * 16 * sm_count() / Hkv));
            if (decode_geometry(g1, kv_type, 1, q_len, n1, n1, Hkv, -1)) need = std::max(need, g1.part_floats);
        }
    if (chunk_keys < 0 && max_slots == 1 && decode_geometry(g1, kv_type, 1, q_len, max_n, max_n, Hkv, -1)) need = std::max(need, g1.part_floats);
    if (chunk_keys < 0 && kv_type == B200_KV_Q8_0 && q_len >= 2 && decode_geometry(g1, kv_type, 1, q_len, max_n, max_n, Hkv, -1, true)) need = std::max(need, g1.part_floats);
    if (chunk_keys < 0 && max_slots > 1 && !gm.split) {
        // a fixed chunk chosen from the batch: smaller batches take smaller chunks; their unit count stays under this bound
        const size_t u = 2 * 8 * (size_t) sm_count() + (size_t) max_slots * Hkv;
        need = std::max(need, u * q_len * GQA * (DH + 2));
    }
    if (!scratch_for((cudaStream_t) stream, need, 0)) B200_REFUSE(B200_ERR_ALLOC, "attn_reserve: %zu floats could not be allocated", need);
    return B200_OK;
}

int b200_attn_decode2(const float * q, const b200_kv_cache * c, float * out, int T, int p0, const int32_t * p0_dev, int Hq,
                      float scale, void * stream, const int32_t * pos_rows) {
    if (T < 1 || T > B200_ATTN_MAX_ROWS) B200_REFUSE(B200_ERR_SHAPE, "attn_decode: unsupported row count %d", T);
    if (!out) B200_REFUSE(B200_ERR_SHAPE, "attn_decode: out is null");
    const int n_ctx = c ? std::max(c->n_ctx, 1) : 1;
    // the grid covers the rows' keys when the host knows them, else the cache's capacity
    const int max_n = (!p0_dev && !pos_rows && p0 >= 0) ? std::min(std::max(p0 + T, 1), c && !c->pt ? n_ctx : 0x7fffffff) : n_ctx;
    // the first call per (device, stream) sizes the scratch for the largest call these entry points accept on this cache
    // (B200_ATTN_MAX_ROWS rows over n_ctx keys), as the reference does (src/fast/attn_dec2.cu:503-517)
    size_t hint = 0;
    if (c && c->Hkv > 0) {
        dec_geom gm;
        if (decode_geometry(gm, c->type, B200_ATTN_MAX_ROWS, 1, n_ctx, n_ctx, c->Hkv, 0, false, true)) hint = gm.part_floats;
    }
    const merge_out mo = {out, nullptr, nullptr, nullptr, nullptr, nullptr};
    // rows of one sequence at consecutive positions share the pass over its KV (up to 4 rows per slot)
    if (!pos_rows && T <= B200_MAX_QLEN)
        return decode_impl(q, c, mo, 1, T, nullptr, p0_dev, p0, max_n, Hq, scale, 0, (cudaStream_t) stream, "attn_decode", hint, true);
    return decode_impl(q, c, mo, T, 1, pos_rows, p0_dev, p0, max_n, Hq, scale, 0, (cudaStream_t) stream, "attn_decode", hint, true);
}

int b200_attn_decode(const float * q, const b200_kv_cache * c, float * out, int T, int p0, int Hq, float scale, void * stream) {
    if (c && !c->pt && (p0 < 0 || p0 + T > c->n_ctx)) B200_REFUSE(B200_ERR_SHAPE, "attn_decode: rows %d..%d outside n_ctx %d", p0, p0 + T - 1, c->n_ctx);
    return b200_attn_decode2(q, c, out, T, p0, nullptr, Hq, scale, stream, nullptr);
}
int b200_attn_decode_dev(const float * q, const b200_kv_cache * c, float * out, int T, const int32_t * p0_dev, int max_n, int Hq,
                         float scale, void * stream) {
    if (!p0_dev) B200_REFUSE(B200_ERR_SHAPE, "attn_decode_dev: p0_dev is null");
    if (T < 1 || T > B200_ATTN_MAX_ROWS) B200_REFUSE(B200_ERR_SHAPE, "attn_decode: unsupported row count %d", T);
    if (!out) B200_REFUSE(B200_ERR_SHAPE, "attn_decode_dev: out is null");
    const int n_ctx = c ? std::max(c->n_ctx, 1) : 1;
    if (max_n < 1 || (c && !c->pt && max_n > n_ctx)) max_n = n_ctx;   // the caller's bound on *p0_dev + T sizes the grid
    size_t hint = 0;
    if (c && c->Hkv > 0) {
        dec_geom gm;
        if (decode_geometry(gm, c->type, B200_ATTN_MAX_ROWS, 1, n_ctx, n_ctx, c->Hkv, 0, false, true)) hint = gm.part_floats;
    }
    const merge_out mo = {out, nullptr, nullptr, nullptr, nullptr, nullptr};
    if (T <= B200_MAX_QLEN)
        return decode_impl(q, c, mo, 1, T, nullptr, p0_dev, 0, max_n, Hq, scale, 0, (cudaStream_t) stream, "attn_decode_dev", hint, true);
    return decode_impl(q, c, mo, T, 1, nullptr, p0_dev, 0, max_n, Hq, scale, 0, (cudaStream_t) stream, "attn_decode_dev", hint, true);
}
int b200_attn_decode_rows(const float * q, const b200_kv_cache * c, float * out, int T, const int32_t * pos, int Hq, float scale,
                          void * stream) {
    if (!pos) B200_REFUSE(B200_ERR_SHAPE, "attn_decode_rows: pos is null");
    return b200_attn_decode2(q, c, out, T, 0, nullptr, Hq, scale, stream, pos);
}

int b200_attn_decode_slots(const float * q, const b200_kv_cache * c, float * out, const float * gate, int n_slots, int q_len,
                           const int32_t * pos, int max_n, int Hq, float scale, int chunk_keys, void * stream) {
    if (!pos || !out) B200_REFUSE(B200_ERR_SHAPE, "attn_decode_slots: pos / out is null");
    const merge_out mo = {out, gate, nullptr, nullptr, nullptr, nullptr};
    return decode_impl(q, c, mo, n_slots, q_len, pos, nullptr, 0, max_n, Hq, scale, chunk_keys, (cudaStream_t) stream, "attn_decode_slots");
}

int b200_attn_decode_slots_a16(const float * q, const b200_kv_cache * c, float * out, const float * gate, void * qbuf, int n_slots,
                               int q_len, const int32_t * pos, int max_n, int Hq, float scale, int chunk_keys, void * stream) {
    if (!pos || !out || !qbuf) B200_REFUSE(B200_ERR_SHAPE, "attn_decode_slots_a16: pos / out / qbuf is null");
    const merge_out mo = {out, gate, nullptr, nullptr, nullptr, qbuf};
    return decode_impl(q, c, mo, n_slots, q_len, pos, nullptr, 0, max_n, Hq, scale, chunk_keys, (cudaStream_t) stream, "attn_decode_slots_a16");
}

int b200_attn_decode_slots_partial(const float * q, const b200_kv_cache * c, float * part_o, float * part_m, float * part_l,
                                   int n_slots, int q_len, const int32_t * pos, int max_n, int Hq, float scale, int chunk_keys,
                                   void * stream) {
    if (!pos || !part_o || !part_m || !part_l) B200_REFUSE(B200_ERR_SHAPE, "attn_decode_slots_partial: null argument");
    if (!aligned16(part_o)) B200_REFUSE(B200_ERR_SHAPE, "attn_decode_slots_partial: part_o must be 16-byte aligned");
    const merge_out mo = {nullptr, nullptr, part_o, part_m, part_l, nullptr};
    return decode_impl(q, c, mo, n_slots, q_len, pos, nullptr, 0, max_n, Hq, scale, chunk_keys, (cudaStream_t) stream,
                       "attn_decode_slots_partial");
}

int b200_attn_merge_gate(const float * part_o, const float * part_m, const float * part_l, int nparts, int R, int D,
                         const float * gate, float * out, void * stream) {
    if (!part_o || !part_m || !part_l || !out || nparts < 1 || R < 1 || D % 4 || D < 4 || D > 4096 || !aligned16(part_o) ||
        !aligned16(out) || (gate && !aligned16(gate)))
        B200_REFUSE(B200_ERR_SHAPE, "attn_merge_gate: unsupported arguments");
    launch(merge_parts_k, R, D / 4, 0, (cudaStream_t) stream, part_o, part_m, part_l, nparts, R, D, gate, out, (size_t) R * D, (size_t) R,
                                                          nullptr);
    count_launch();
    return launch_status("attn_merge_gate");
}

// shared by the two exchange entries: optional all-gather over the caller's communicator, then the merge
static int seq_exchange_impl(void * nccl_comm, int n_seq, const float * send, float * recv, int R, int D, const float * gate,
                             float * out, void * qbuf, void * stream, const char * who) {
    using allgather_fn = int (*)(const void *, void *, size_t, int, void *, cudaStream_t);
    static allgather_fn allgather = [] {
        void * f = dlsym(RTLD_DEFAULT, "ncclAllGather");
        if (!f) {
            void * h = dlopen("libnccl.so.2", RTLD_NOW | RTLD_GLOBAL);
            if (h) f = dlsym(h, "ncclAllGather");
        }
        return (allgather_fn) f;
    }();
    const size_t part = (size_t) R * (D + 2);
    if (!send || !recv || !out || n_seq < 1 || R < 1 || D % 4 || D < 4 || D > 4096 || part % 4 || !aligned16(send) || !aligned16(recv) ||
        !aligned16(out) || (gate && !aligned16(gate)))
        B200_REFUSE(B200_ERR_SHAPE, "%s: unsupported arguments (R * (D + 2) must be a multiple of 4, buffers 16-byte aligned)", who);
    if (qbuf && (D % 128 || ((uintptr_t) qbuf & 3)))
        B200_REFUSE(B200_ERR_SHAPE, "%s: the a16 buffer needs D %% 128 == 0 and 4-byte alignment", who);
    cudaStream_t s = (cudaStream_t) stream;
    const float * parts = n_seq > 1 ? recv : send;
    if (n_seq > 1 && nccl_comm) {   // without a communicator the caller has gathered the parts into recv already
        if (!allgather) B200_REFUSE(B200_ERR_CUDA, "%s: no NCCL library is loaded in this process", who);
        const int rc = allgather(send, recv, part, 7 /* ncclFloat32 */, nccl_comm, s);
        if (rc != 0) B200_REFUSE(B200_ERR_CUDA, "%s: ncclAllGather returned %d", who, rc);
    }
    launch(merge_parts_k, R, D / 4, 0, s, parts, parts + (size_t) R * D, parts + (size_t) R * D + R, n_seq, R, D, gate, out, part, part,
                                      (__half2 *) qbuf);
    count_launch();
    return launch_status(who);
}

// The exchange step of the sequence split for a host that drives NCCL itself.  ncclAllGather is taken from the NCCL library
// the process has already loaded (the host's own, or the one bundled with its framework), so the communicator and the
// function come from the same library; nothing here links NCCL.
int b200_seq_exchange_merge(void * nccl_comm, int n_seq, const float * send, float * recv, int R, int D, const float * gate,
                            float * out, void * stream) {
    return seq_exchange_impl(nccl_comm, n_seq, send, recv, R, D, gate, out, nullptr, stream, "seq_exchange_merge");
}
int b200_seq_exchange_merge_a16(void * nccl_comm, int n_seq, const float * send, float * recv, int R, int D, const float * gate,
                                float * out, void * qbuf, void * stream) {
    if (!qbuf) B200_REFUSE(B200_ERR_SHAPE, "seq_exchange_merge_a16: qbuf is null");
    return seq_exchange_impl(nccl_comm, n_seq, send, recv, R, D, gate, out, qbuf, stream, "seq_exchange_merge_a16");
}

// ---- sequence split over peer-mapped buffers ------------------------------------------------------------------
// A buffer other processes of the node can map (cudaMalloc + cudaIpcGetMemHandle): the host passes the 64-byte handle to the
// peers by whatever means it has, they map it with b200_peer_open.  Zero-filled.
int b200_peer_alloc(size_t bytes, void ** ptr, unsigned char * handle) {
    if (!ptr || !handle || !bytes) B200_REFUSE(B200_ERR_SHAPE, "peer_alloc: null argument");
    void * p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) { cudaGetLastError(); B200_REFUSE(B200_ERR_ALLOC, "peer_alloc: cudaMalloc(%zu) failed", bytes); }
    cudaIpcMemHandle_t h;
    if (cudaMemset(p, 0, bytes) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess || cudaIpcGetMemHandle(&h, p) != cudaSuccess) {
        const cudaError_t e = cudaGetLastError();
        cudaFree(p);
        B200_REFUSE(B200_ERR_CUDA, "peer_alloc: %s", cudaGetErrorString(e));
    }
    static_assert(sizeof h == 64, "handle size");
    memcpy(handle, &h, 64);
    *ptr = p;
    return B200_OK;
}
int b200_peer_open(const unsigned char * handle, void ** ptr) {
    if (!ptr || !handle) B200_REFUSE(B200_ERR_SHAPE, "peer_open: null argument");
    cudaIpcMemHandle_t h;
    memcpy(&h, handle, 64);
    void * p = nullptr;
    const cudaError_t e = cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess);
    if (e != cudaSuccess) { cudaGetLastError(); B200_REFUSE(B200_ERR_CUDA, "peer_open: %s", cudaGetErrorString(e)); }
    *ptr = p;
    return B200_OK;
}
int b200_peer_close(void * ptr) { return ptr && cudaIpcCloseMemHandle(ptr) != cudaSuccess ? (cudaGetLastError(), B200_ERR_CUDA) : B200_OK; }
int b200_peer_free(void * ptr) { return ptr && cudaFree(ptr) != cudaSuccess ? (cudaGetLastError(), B200_ERR_CUDA) : B200_OK; }

static int seq_merge_peers_impl(const void * const * parts, void * const * flags, int n_seq, int me, unsigned epoch, int R, int D,
                                const float * gate, float * out, void * qbuf, void * stream, const char * who) {
    if (!parts || !flags || !out || n_seq < 1 || n_seq > MAX_PEERS || me < 0 || me >= n_seq || R < 1 || D % 4 || D < 4 * MAX_PEERS || D > 4096 ||
        !aligned16(out) || (gate && !aligned16(gate)))
        B200_REFUSE(B200_ERR_SHAPE, "%s: unsupported arguments", who);
    if (qbuf && (D % 128 || ((uintptr_t) qbuf & 3))) B200_REFUSE(B200_ERR_SHAPE, "%s: the a16 buffer needs D %% 128 == 0 and 4-byte alignment", who);
    peer_parts pp;
    for (int s = 0; s < MAX_PEERS; ++s) {
        pp.part[s] = s < n_seq ? (const float *) parts[s] : nullptr;
        pp.flag[s] = s < n_seq ? (unsigned *) flags[s] : nullptr;
        if (s < n_seq && (!pp.part[s] || !pp.flag[s] || !aligned16(pp.part[s]) || ((uintptr_t) pp.flag[s] & 3)))
            B200_REFUSE(B200_ERR_SHAPE, "%s: shard %d: buffers must be mapped and 16-byte aligned", who, s);
    }
    unsigned * st = device_status_word();
    if (!st) return B200_ERR_CUDA;
    merge_peers_k<<<R, D / 4, 0, (cudaStream_t) stream>>>(pp, n_seq, me, epoch, R, D, gate, out, (__half2 *) qbuf, st);
    count_launch();
    return launch_status(who);
}
int b200_seq_merge_peers(const void * const * parts, void * const * flags, int n_seq, int me, unsigned epoch, int R, int D,
                         const float * gate, float * out, void * stream) {
    return seq_merge_peers_impl(parts, flags, n_seq, me, epoch, R, D, gate, out, nullptr, stream, "seq_merge_peers");
}
int b200_seq_merge_peers_a16(const void * const * parts, void * const * flags, int n_seq, int me, unsigned epoch, int R, int D,
                             const float * gate, float * out, void * qbuf, void * stream) {
    if (!qbuf) B200_REFUSE(B200_ERR_SHAPE, "seq_merge_peers_a16: qbuf is null");
    return seq_merge_peers_impl(parts, flags, n_seq, me, epoch, R, D, gate, out, qbuf, stream, "seq_merge_peers_a16");
}

}  // extern "C"
