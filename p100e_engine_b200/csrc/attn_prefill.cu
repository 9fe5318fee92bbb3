// Chunked causal prefill attention over the paged f16 / q8_0 / q4_0 cache on the sm_100a tensor cores (tcgen05 + TMEM).
//
// Two or three kernels per call:
//   kv_tiles_k   dequantises the visible keys once into f16 "tile images" in scratch: per (kv head, 64-key tile) a
//                32 KB K image and a 32 KB V image laid out exactly as the tensor core reads them from shared memory
//                (un-swizzled canonical layout, see umma.cuh; 8-key groups 4 KB apart, so two images side by side form
//                one 128-key operand), so the main kernel fetches a tile with one bulk copy.
//   prefill_k    one CTA per (128 query rows of one kv head): rows n = 6 t + hh (token t, head hh of the GQA group) on
//                the MMA M axis, keys in steps of 128 (a pair of images).  Per step: S = Q K^T as 16 MMAs m128n128k16
//                (Q from tensor memory and shared memory, half of the dims each; fp32 S in tensor memory), online softmax in base 2
//                with two threads per row (64 keys each, no shuffles), P to tensor memory as f16, O += P V as 8 MMAs m128n256k16
//                accumulated in tensor memory.  Warp roles: 8 softmax warps, 1 bulk-copy producer warp, 1 MMA-issue warp.  The MMA
//                queue alternates Q K^T of step J+1 and P V of step J, so the tensor pipe has work while the softmax
//                of a step runs; S is single-buffered (the next Q K^T starts when the softmax threads hold S in
//                registers), P is freed and filled in halves of 64 keys.  The running output is rescaled only when a row's maximum
//                grows by more than 2^8 (P stays below 256 in f16).  Epilogue: O / l, optional sigmoid gate.
//                What bounds a step is shared memory (128 bytes per clk): K and V images in and out 256 KB and half of Q out 32 KB are 2304 clk, measured
//                2300 (1.4 us at 1.65 GHz; the MMAs take 2048).  With P in shared memory (64 KB in and out) and all of Q in tensor memory it
//                was 2515; tensor memory is full now: S 128, O 256, Q 64, P 64 columns.
//                A few rows behind a long history are fewer row tiles than SMs: then the steps of all row tiles are cut evenly over
//                the SMs and prefill_merge_k adds up the pieces of a tile (pf_cut, split_ctas).
// f16 operands (int8 * f16 scale is not representable in bf16's 8 significand bits), fp32 accumulation.
// Long contexts run as several passes over consecutive key ranges (as many keys as the scratch holds tile images for):
// a row tile whose keys continue in a later pass leaves its unnormalised O in the output buffer and (max, sum) beside it,
// and the next pass loads them back into tensor memory; the pass that holds a row tile's last key writes the result.
// Q may come as bf16 rows straight from the projection: the partial rotation is then applied while the rows are converted
// for tensor memory (cos / sin per token from a table the append kernel wrote), so no fp32 copy of Q goes through HBM.
//
// Reference counterparts: attn_fold (src/fast/attn_fold.cu:562-649: per chunk dequantise to f16 in scratch, HFMA2 tile
// GEMMs on CUDA cores), attn_prefill (src/fast/attn.cu:457-499, fp32 CUDA cores).
#include "umma.cuh"
#include "grow.h"

#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <mutex>

namespace b200 {
namespace {

constexpr int BM = 128;                 // query rows per CTA
constexpr int BN = 64;                  // keys per tile image
constexpr int BP = 2 * BN;              // keys per step: S tile = 128 rows x 128 keys
constexpr int IMG = BN * DH * 2;        // bytes of one tile image (32 KB)
constexpr int Q_BYTES = BM * DH / 2 * 2;    // 32 KB: half of the dims
constexpr int EPI_STR = DH / 2 + 4;     // floats per row of the epilogue's tiles: 32 rows x 128 dims per softmax warp (+ 4: rows on different banks)
constexpr int EPI_BYTES = 8 * 32 * EPI_STR * 4;
constexpr int NSOFT = 256;              // softmax threads: two per query row (key halves of a tile, dim halves of the output)
constexpr int NTHR_PF = NSOFT + 64;     // 8 softmax warps + producer + MMA issuer
constexpr int W_PROD = NSOFT / 32, W_MMA = W_PROD + 1;
constexpr float LOG2E_PF = 1.4426950408889634f;
constexpr float RESCALE_GAP = 8.0f;     // rescale O when a row maximum grows by more than this (log2 units)

// Two pairs of K images and one pair of V images whose halves are copied and freed by themselves: every copy has 1500 clk or more before it
// is waited for.  One pair of K images left 1024 clk for its 64 KB (48 rows behind 100003 keys, images from HBM: a step 1.84 us, 1.65 with two).
// A ring of single images that frees K by halves needs Q K^T in two m128n64k16, which take longer than half of an m128n128k16: 1.75 us for 1.5.
constexpr int SM_K = 0;
constexpr int SM_V = SM_K + 4 * IMG;
constexpr int SM_Q = SM_V + 2 * IMG;            // dims 128 .. 255 of the query rows
constexpr int SM_EPI = SM_K;                    // the epilogue tiles lie over K and V
constexpr int SM_XCH = SM_Q + Q_BYTES;          // [2][128] floats exchanged between the two threads of a row
constexpr int SM_BAR = SM_XCH + 1024;           // mbarriers + tmem base
constexpr int SM_TOTAL = SM_BAR + 256;
static_assert(SM_TOTAL <= 227 * 1024 && EPI_BYTES <= SM_Q, "prefill_k shared memory");

// ---- pre-pass: cache rows -> f16 tile images -------------------------------------------------------------------
// grid (n_tiles, Hkv), 256 threads; thread = (key, 64 dims).  Image byte of (key, dim) = (key/8)*4096 + (dim/8)*128 +
// (key%8)*16 + (dim%8)*2 for K (K-major B operand) and for V (MN-major B operand) alike.  Keys >= n_keys are zero.
// Bound by HBM: 2 x 272 bytes read (q8_0) and 1 KiB written per key and head.  A thread has all its loads of K and V in flight at
// once, behind one page lookup; eight rounds of 8-byte loads, each behind a lookup of its own, took a call of 48 rows behind 100003 keys
// (four heads, 218 MB of rows in, 410 MB of images out) 423 us instead of 363, one of 512 rows behind 16000 263 us instead of 253.

// 64 values of a head row (the blocks 2 part, 2 part + 1) as f16 pairs, each the stored integer times its block's scale, rounded once
template <uint32_t KT> struct row_part {
    uint4 d[KT == B200_KV_F16 ? 8 : 4];
    uint32_t s[KT == B200_KV_Q4_0 ? 9 : 1];
    __device__ __forceinline__ void load(const unsigned char * row, int part) {
        if constexpr (KT == B200_KV_F16) {
#pragma unroll
            for (int u = 0; u < 8; ++u) d[u] = __ldg(reinterpret_cast<const uint4 *>(row + 128 * part) + u);
        } else if constexpr (KT == B200_KV_Q8_0) {
            s[0] = __ldg(reinterpret_cast<const uint32_t *>(row) + part);
#pragma unroll
            for (int u = 0; u < 4; ++u) d[u] = __ldg(reinterpret_cast<const uint4 *>(row + 16 + 64 * part) + u);
        } else {   // two blocks of {f16 scale, 16 bytes}: 36 bytes from a 4-byte boundary
#pragma unroll
            for (int u = 0; u < 9; ++u) s[u] = __ldg(reinterpret_cast<const uint32_t *>(row + 36 * part) + u);
        }
    }
    // values 8 c .. 8 c + 7
    __device__ __forceinline__ uint4 chunk(int c) const {
        if constexpr (KT == B200_KV_F16) return d[c];
        else if constexpr (KT == B200_KV_Q8_0) {
            const uint32_t d2 = __byte_perm(s[0], 0u, c < 4 ? 0x1010 : 0x3232);
            const uint32_t x = (&d[c >> 1].x)[2 * (c & 1)] ^ 0x80808080u, y = (&d[c >> 1].x)[2 * (c & 1) + 1] ^ 0x80808080u;
            auto pair = [&](uint32_t w, uint32_t sel) { return hmul2_u32(hsub2_u32(__byte_perm(w, 0x64646464u, sel), 0x64806480u), d2); };
            return make_uint4(pair(x, 0x5140), pair(x, 0x7362), pair(y, 0x5140), pair(y, 0x7362));
        } else {
            // block b = c / 4: scale in the low (b = 0) or high (b = 1) half of word 4 b + ..., its 16 bytes on a 2-byte (b = 0) or 4-byte boundary
            const int b = c >> 2, j = c & 3;   // values 8 j .. of the block: bytes 8 (j & 1) .. + 7, low (j < 2) or high nibbles
            const uint32_t d2 = b ? __byte_perm(s[4], 0u, 0x3232) : __byte_perm(s[0], 0u, 0x1010);
            const int o = 2 * (j & 1);
            uint32_t x, y;
            if (b) { x = s[5 + o]; y = s[6 + o]; }
            else { x = __funnelshift_r(s[o], s[o + 1], 16); y = __funnelshift_r(s[o + 1], s[o + 2], 16); }
            if (j >= 2) { x >>= 4; y >>= 4; }
            x &= 0x0f0f0f0fu; y &= 0x0f0f0f0fu;
            auto pair = [&](uint32_t w, uint32_t sel) { return hmul2_u32(hsub2_u32(__byte_perm(w, 0x64646464u, sel), 0x64086408u), d2); };
            return make_uint4(pair(x, 0x5140), pair(x, 0x7362), pair(y, 0x5140), pair(y, 0x7362));
        }
    }
};

template <uint32_t KT>
__global__ void __launch_bounds__(256) kv_tiles_k(kv_view g, int kb, int n_keys, unsigned char * __restrict__ tiles, int n_tiles,
                                                  unsigned * status) {
    pdl_enter();
    const int tile = blockIdx.x, hk = blockIdx.y;   // tile j of the pass holds keys kb + 64 j ..; keys >= n_keys are zero
    const int key = threadIdx.x & (BN - 1), part = threadIdx.x / BN, kk = kb + tile * BN + key;
    unsigned char * kimg = tiles + ((size_t) hk * n_tiles + tile) * (2 * IMG) + (key >> 3) * 4096 + part * 1024 + (key & 7) * 16;
    bool have = kk < n_keys;
    const int32_t * tab = kv_tab(g, 0);
    int pg = 0;
    if (have && tab && (pg = tab[kk >> g.psh]) < 0) { atomicOr(status, ST_BAD_PAGE); have = false; }
    row_part<KT> k, v;
    if (have) {
        const unsigned long long off = (tab ? (unsigned long long) pg * g.pstride + (unsigned long long) (kk & ((1 << g.psh) - 1)) * g.rowb
                                            : (unsigned long long) kk * g.rowb) + (unsigned long long) hk * head_bytes(KT);
        k.load((const unsigned char *) g.k + off, part);
        v.load((const unsigned char *) g.v + off, part);
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4 *>(kimg + c * 128) = have ? k.chunk(c) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4 *>(kimg + IMG + c * 128) = have ? v.chunk(c) : make_uint4(0, 0, 0, 0);
}

struct pf_args {
    const float * q;              // [T][Hq][256] f32, already rotated, or nullptr
    const __nv_bfloat16 * qb;     // [T][Hq][256] bf16, not yet rotated (used when q is null); needs cs
    const float * cs;             // [T][64]: cos of the 32 rotary pairs, then sin (written by the append kernel)
    const float * gate;           // [T][Hq*256] f32 or nullptr
    const __nv_bfloat16 * gate_b; // the gate as bf16 (used when gate is null) or nullptr
    float * out;                  // [T][Hq][256] f32: the result; between passes the running unnormalised O
    __nv_bfloat16 * out_b;        // the result as bf16 (optional; out is then only the carry buffer)
    float * ml;                   // [T*Hq][2] running (maximum in log2 units, sum) between passes
    float * pm, * pl;             // partial form: [T*Hq] maximum (natural-log units) and sum; out keeps the unnormalised O
    __half2 * qbuf;               // a16 copy of the result (optional)
    const int32_t * lim;          // per token: last visible key (device), or nullptr for p0 + t
    const unsigned char * tiles;
    int n_tiles;                  // tile images per head in scratch
    int kb, ke;                   // keys of this pass: kb (a multiple of 128) .. ke - 1
    int T, p0, Hq, Hkv;
    float qscale;                 // softmax scale * log2(e)
    unsigned * status;
    // even split (n_run > 0; one pass, no lim): see pf_cut
    int n_run;                    // CTAs
    int n_mtiles;                 // row tiles of a kv head
    int head_steps;               // 128-key steps of a kv head, all row tiles together
    float * po;                   // [2 n_run][128][256] unnormalised O of the pieces
    float2 * pml;                 // [2 n_run][128] (maximum in log2 units, sum)
};

// Even split: the 128-key steps of all row tiles (kv head by kv head, row tile by row tile) form one sequence of
// Hkv * head_steps; CTA c of n_run takes steps pf_cut(c) .. pf_cut(c + 1) - 1.  A row tile whose steps lie in several CTAs is left
// as pieces, unnormalised, which prefill_merge_k adds up in key order: a CTA's piece that starts a row tile is number 2 c + 1, one that
// continues a row tile number 2 c (a CTA has at most one of each).
__host__ __device__ __forceinline__ int pf_tile_steps(int T, int p0, int m) {
    const int n_last = m * BM + BM < T * GQA ? m * BM + BM - 1 : T * GQA - 1;
    return (p0 + n_last / GQA + BP) / BP;   // ceil(visible keys / 128)
}
__device__ __forceinline__ int pf_cut(const pf_args & a, int c) { return (int) ((long long) a.Hkv * a.head_steps * c / a.n_run); }
// row tile of a kv head that holds step `rem` of the head and the head's steps before that tile; called by a whole warp
__device__ __forceinline__ int pf_find_tile(const pf_args & a, int rem, int & before) {
    const int lane = threadIdx.x & 31;
    int base = 0;
    for (int m0 = 0;; m0 += 32) {
        const int m = m0 + lane, own = m < a.n_mtiles ? pf_tile_steps(a.T, a.p0, m) : 0;
        int x = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
        const unsigned past = __ballot_sync(0xffffffffu, base + x > rem);
        if (past || m0 + 32 >= a.n_mtiles) {
            const int l = past ? __ffs(past) - 1 : 31;
            before = base + __shfl_sync(0xffffffffu, x - own, l);
            return m0 + l;
        }
        base += __shfl_sync(0xffffffffu, x, 31);
    }
}

__device__ __forceinline__ float rcpf(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 1 / (1 + 2^(-g log2 e)) with the hardware exponential and reciprocal (relative error ~1e-7 against expf and an IEEE divide)
__device__ __forceinline__ float fast_sigmoid(float g) { return rcpf(1.0f + ex2f(-g * LOG2E_PF)); }

__device__ __forceinline__ void mbar_arrive(uint64_t * bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void bf16x8_widen(const uint4 u, float (&f)[8]) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) { f[2 * e] = __uint_as_float(w[e] << 16); f[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u); }
}

__global__ void __launch_bounds__(NTHR_PF, 1) prefill_k(const pf_args a) {
    pdl_enter();
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t * bars = reinterpret_cast<uint64_t *>(smem + SM_BAR);
    uint64_t * k_full = bars, * k_free = bars + 2, * v_full = bars + 4, * v_free = bars + 6, * p_full = bars + 8, * pv_done = bars + 10,   // two each
             * s_full = bars + 12, * s_free = bars + 13, * o_done = bars + 14, * q_ready = bars + 15;
    uint32_t * tbase_p = reinterpret_cast<uint32_t *>(bars + 16);

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);     // as a warp-uniform value
    const int R = a.T * GQA;                                    // rows of a kv head
    // the segments of this CTA: one row tile, or (even split) the row tiles of its run of steps
    int hk = blockIdx.y, mtile = (int) gridDim.x - 1 - (int) blockIdx.x;   // one tile per CTA: heaviest (latest rows) first
    int st0 = 0, w = 0, w_end = 0;
    if (a.n_run) {
        w = pf_cut(a, (int) blockIdx.x); w_end = pf_cut(a, (int) blockIdx.x + 1);
        hk = w / a.head_steps;
        int before;
        mtile = pf_find_tile(a, w - hk * a.head_steps, before);
        st0 = w - hk * a.head_steps - before;
    } else {
        // This pass covers keys kb .. ke-1.  A tile whose keys ended in an earlier pass has been written already; a tile
        // whose keys go on past ke leaves its running state behind for the next pass.
        const int t_l = min(mtile * BM + BM - 1, R - 1) / GQA;
        if ((a.lim ? a.lim[t_l] : a.p0 + t_l) < a.kb && a.kb > 0) return;
    }

    if (tid == 0) {
        mbar_init(s_full, 1); mbar_init(s_free, NSOFT);
        for (int b = 0; b < 2; ++b) {
            mbar_init(&k_full[b], 1); mbar_init(&k_free[b], 1); mbar_init(&v_full[b], 1); mbar_init(&v_free[b], 1);
            mbar_init(&p_full[b], NSOFT / 2); mbar_init(&pv_done[b], 1);
        }
        mbar_init(o_done, 1);
        mbar_init(q_ready, 1);
        mbar_fence_init();
    }
    if (warp == 0) umma::tmem_alloc(tbase_p, 512);
    umma::fence_async_smem();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tb = *tbase_p;
    const uint32_t t_S = tb, t_O = tb + BP, t_Q = t_O + DH, t_P = t_Q + DH / 4;   // S at columns 0..127, O at 128..383, Q (dims 0..127 as f16 pairs) at 384.., P (128 keys) at 448..

    // row bookkeeping of the softmax threads, shared by the prologue, the loop and the epilogue: a warp owns the 32 rows of its
    // tensor-memory lanes; for row-wise global accesses 8 lanes cover 128 bytes of one row, a warp instruction touches 4 rows
    const uint32_t lane_off = (uint32_t) ((warp & 3) * 32) << 16;
    const int sub = lane >> 3, col = 4 * (lane & 7);

    // steps of the earlier segments and those of them that had a second V image: the barriers' phases run on from one segment to the next
    int g = 0, g2 = 0;
    for (int seg = 0;; ++seg) {
    const int n0 = mtile * BM;
    const int t_last = min(n0 + BM - 1, R - 1) / GQA;           // last token of the tile
    const int n_keys_vis = (a.lim ? a.lim[t_last] : a.p0 + t_last) + 1;   // keys any row of the tile can see (limits do not decrease with t)
    const bool carry_in = a.kb > 0;
    const bool carry_out = n_keys_vis > a.ke;
    const int n_keys_pass = max(0, min(n_keys_vis, a.ke) - a.kb);
    const int tile_steps = (n_keys_pass + BP - 1) / BP;
    const int st1 = a.n_run ? min(tile_steps, st0 + w_end - w) : tile_steps;
    const int nsteps = st1 - st0;                               // 128-key steps of this segment; a tile's last one may hold a single image
    const int ntiles = min((n_keys_pass + BN - 1) / BN, 2 * st1) - 2 * st0;   // 64-key images of this segment
    const bool piece = nsteps < tile_steps;                     // the tile is shared with other CTAs
    float m_ref = B200_NEG_INF, l = 0.0f;

    if (warp < W_PROD) {
        // Q rows -> f16, scaled by softmax scale * log2(e), into tensor memory as the A operand of Q K^T: lane = row,
        // column c holds dims 2c, 2c+1.  The two threads of a row take 128 dims each.  A warp reads 256 bytes of a row with 16 lanes (all of
        // its half of a bf16 row, half of it of an f32 row), two rows per load and 16 loads in flight, and turns them by way of a tile of its own
        // where the K images of the second step go, chunk c of row i at c ^ (i & 7): with each lane reading along its own row a load touched 32 rows (4.5 us of
        // prologue on a busy chip; as one bulk copy per row 9 us, of which 128 copies took 6 to issue).
        const int r = tid & (BM - 1), hf = tid >> 7, n = n0 + r;
        const int t = n / GQA, hh = n - t * GQA;
        const size_t rowidx = (size_t) t * a.Hq + hk * GQA + hh;
        const float sc = a.qscale;
        unsigned char * qt = smem + SM_K + ((g + 1) & 1) * (2 * IMG) + warp * 8192;
        const int esz = a.q ? 4 : 2;
        const char * qsrc = a.q ? reinterpret_cast<const char *>(a.q) : reinterpret_cast<const char *>(a.qb);
        auto ahead = [&](uint4 (&x)[16], int part) {   // bytes 256 part .. of the warp's half rows
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                const int nr = n0 + (warp & 3) * 32 + 2 * u + (lane >> 4), tr = nr / GQA, hr = nr - tr * GQA;
                x[u] = nr < R ? __ldg(reinterpret_cast<const uint4 *>(qsrc + (((size_t) tr * a.Hq + hk * GQA + hr) * DH + hf * (DH / 2)) * esz + 256 * part) + (lane & 15))
                              : make_uint4(0, 0, 0, 0);
            }
        };
        auto put = [&](const uint4 (&x)[16]) {
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                const int i = 2 * u + (lane >> 4);
                *reinterpret_cast<uint4 *>(qt + i * 256 + (((lane & 15) ^ (i & 7)) << 4)) = x[u];
            }
            __syncwarp();
        };
        auto chunk = [&](int c) { return *reinterpret_cast<const uint4 *>(qt + lane * 256 + ((c ^ (lane & 7)) << 4)); };
        auto put_q = [&](const uint32_t (&w)[32], int part) {   // 64 dims of the thread's row, f16 pairs: to tensor memory, or K-major to shared memory
            if (hf == 0) umma::tmem_st32(t_Q + lane_off + 32 * part, w);
            else
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    *reinterpret_cast<uint4 *>(smem + SM_Q + (8 * part + c) * 2048 + r * 16) = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
        };
        uint4 x[16];
        ahead(x, 0);
        if (a.q) {
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                put(x);
                if (part == 0) ahead(x, 1);
                uint32_t w[32];
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    const uint4 v = chunk(u);
                    w[2 * u] = pack_h2(__uint_as_float(v.x) * sc, __uint_as_float(v.y) * sc);
                    w[2 * u + 1] = pack_h2(__uint_as_float(v.z) * sc, __uint_as_float(v.w) * sc);
                }
                put_q(w, part);
            }
        } else {
            // bf16 rows as the projection wrote them: widen, rotate the 32 pairs (j, j + 32) of the first 64 dims with the
            // token's cos / sin (same expressions and roundings as the append kernel), scale, round to f16
            const float4 * cs4 = reinterpret_cast<const float4 *>(a.cs + (size_t) t * 64);
            put(x);
#pragma unroll 1
            for (int part = 0; part < 2; ++part) {
                float f[64];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    float e8[8];
                    bf16x8_widen(chunk(8 * part + u), e8);
#pragma unroll
                    for (int e = 0; e < 8; ++e) f[8 * u + e] = e8[e];
                }
                if (hf == 0 && part == 0 && n < R) {
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const float4 c4 = __ldg(cs4 + u), s4 = __ldg(cs4 + 8 + u);
                        const float cc[4] = {c4.x, c4.y, c4.z, c4.w}, ss[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) rot_pair(f[4 * u + e], f[32 + 4 * u + e], cc[e], ss[e], f[4 * u + e], f[32 + 4 * u + e]);
                    }
                }
                uint32_t w[32];
#pragma unroll
                for (int u = 0; u < 32; ++u) w[u] = pack_h2(f[2 * u] * sc, f[2 * u + 1] * sc);
                put_q(w, part);
            }
        }
        if (carry_in) {
            // the running O of the earlier passes goes back into tensor memory (read row-wise, handed over through a
            // per-warp tile in the same place), with the row's maximum and sum
            asm volatile("bar.sync 1, %0;" ::"n"(NSOFT) : "memory");   // every warp is done with its tile of query values
            float * tile = reinterpret_cast<float *>(smem + SM_K + ((g + 1) & 1) * (2 * IMG)) + warp * (32 * 33);
            const int c_lo = hf * (DH / 2), c_hi = c_lo + DH / 2;
#pragma unroll 1
            for (int c0 = c_lo; c0 < c_hi; c0 += 32) {
#pragma unroll
                for (int q8 = 0; q8 < 8; ++q8) {
                    const int rl = 4 * q8 + sub, nr = n0 + (warp & 3) * 32 + rl;
                    const int tr = nr / GQA, hr = nr - tr * GQA;
                    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (nr < R) v = *reinterpret_cast<const float4 *>(a.out + ((size_t) tr * a.Hq + hk * GQA + hr) * DH + c0 + col);
                    tile[rl * 33 + col] = v.x; tile[rl * 33 + col + 1] = v.y; tile[rl * 33 + col + 2] = v.z; tile[rl * 33 + col + 3] = v.w;
                }
                __syncwarp();
                uint32_t o[32];
#pragma unroll
                for (int c = 0; c < 32; ++c) o[c] = __float_as_uint(tile[lane * 33 + c]);
                umma::tmem_st32(t_O + lane_off + c0, o);
                __syncwarp();
            }
            if (n < R) {
                m_ref = a.ml[rowidx * 2];
                l = hf == 0 ? a.ml[rowidx * 2 + 1] : 0.0f;
            }
        }
        umma::tmem_st_wait();
        umma::fence_before_sync();
        umma::fence_async_smem();   // K images are copied to where the tiles lay
        asm volatile("bar.sync 1, %0;" ::"n"(NSOFT) : "memory");   // the softmax warps: every Q (and O) row is in place
        if (tid == 0) mbar_arrive(q_ready);
    }
    const bool any_gate = a.gate || a.gate_b;
    if (warp == W_PROD) {
        // ---------------- producer: K in pairs of images (lane 0), V image by image (lane 16) ----------------
        const unsigned char * src = a.tiles + ((size_t) hk * a.n_tiles + 2 * st0) * (2 * IMG);
        if (lane == 0) {
            for (int J = 0; J < nsteps; ++J) {
                const int G = g + J, b = G & 1;
                if (J == 1) mbar_wait(q_ready, (uint32_t) (seg & 1), a.status);   // the query rows have passed through this pair's place
                if (G >= 2) mbar_wait(&k_free[b], (uint32_t) (((G >> 1) - 1) & 1), a.status);   // Q K^T of step J-2 has read the pair
                const int n_img = min(2, ntiles - 2 * J);
                mbar_expect_tx(&k_full[b], (uint32_t) n_img * IMG);
                for (int h = 0; h < n_img; ++h)
                    bulk_g2s(smem + SM_K + (2 * b + h) * IMG, src + (size_t) (2 * J + h) * (2 * IMG), IMG, &k_full[b]);
            }
        } else if (lane == 16) {
            for (int j = 0; j < ntiles; ++j) {
                const int h = j & 1, u = (h ? g2 : g) + (j >> 1);   // earlier uses of the slot
                if (u >= 1) mbar_wait(&v_free[h], (uint32_t) ((u - 1) & 1), a.status);   // P V of the image before has read the slot
                mbar_expect_tx(&v_full[h], IMG);
                bulk_g2s(smem + SM_V + h * IMG, src + (size_t) j * (2 * IMG) + IMG, IMG, &v_full[h]);
            }
        }
    } else if (warp == W_MMA) {
        // ---------------- MMA issuer: Q K^T of step J+1 is queued before P V of step J ----------------
        // All 32 lanes walk the loop and wait, so that addresses and descriptors are warp-uniform values (the MMA takes its
        // operands from uniform registers); one elected lane issues.
        __syncwarp();
        const bool lead = umma::elect_one();
        const uint32_t tb_u = __shfl_sync(0xffffffffu, tb, 0);
        const uint32_t tS_u = tb_u, tO_u = tb_u + BP, tQ_u = tO_u + DH, tP_u = tQ_u + DH / 4;
        const int ns_u = __shfl_sync(0xffffffffu, nsteps, 0), ni_u = __shfl_sync(0xffffffffu, ntiles, 0), g_u = __shfl_sync(0xffffffffu, g, 0);
        const int g2_u = __shfl_sync(0xffffffffu, g2, 0);
        constexpr uint32_t id_qk = umma::idesc_f16(BM, BP, false, false);   // S[128 x 128] = Q (tensor memory) * K^T (K-major)
        constexpr uint32_t id_pv = umma::idesc_f16(BM, DH, false, true);    // O[128 x 256] += P (K-major) * V (MN-major)
        const uint32_t k_s0 = smem_u32(smem + SM_K), v_s0 = smem_u32(smem + SM_V), q_s = smem_u32(smem + SM_Q);
        auto issue_qk = [&](int J) {
            const int G = g_u + J, b = G & 1;
            mbar_wait(&k_full[b], (uint32_t) ((G >> 1) & 1), a.status);
            if (G >= 1) mbar_wait(s_free, (uint32_t) ((G - 1) & 1), a.status);   // the softmax threads hold S of the step before in registers
            umma::fence_after_sync();
            // K pair: K-major, 8-key groups 4096 apart (SBO), 8-dim chunks 128 apart (LBO); 16 dims = 256 bytes per k-step.
            // A step with a single image multiplies whatever the second half of the buffer holds: those keys lie past
            // every row of the tile and are masked.
            if (lead) {
                const uint32_t k_s = k_s0 + b * (2 * IMG);
#pragma unroll
                for (int ks = 0; ks < DH / 32; ++ks)
                    umma::mma_ts(tS_u, tQ_u + ks * 8, umma::smem_desc(k_s + ks * 256, 128, 4096), id_qk, ks > 0);
#pragma unroll
                for (int ks = 0; ks < DH / 32; ++ks)   // Q: 8-row groups 128 apart (SBO), 8-dim chunks 2048 apart (LBO)
                    umma::mma_ss(tS_u, umma::smem_desc(q_s + ks * 2 * 2048, 2048, 128), umma::smem_desc(k_s + (DH / 32 + ks) * 256, 128, 4096), id_qk, 1u);
                umma::commit(s_full);
                umma::commit(&k_free[b]);
            }
        };
        auto issue_pv = [&](int J) {
            const int G = g_u + J, n_img = min(2, ni_u - 2 * J);
            for (int h = 0; h < n_img; ++h) {
                mbar_wait(&p_full[h], (uint32_t) (G & 1), a.status);
                mbar_wait(&v_full[h], (uint32_t) (((h ? g2_u : g_u) + J) & 1), a.status);
                umma::fence_after_sync();
                if (lead) {
                    const uint32_t v_s = v_s0 + h * IMG;
                    const uint32_t acc0 = (carry_in || J > 0 || h > 0) ? 1u : 0u;
#pragma unroll
                    for (int ks = 0; ks < BN / 16; ++ks)   // V: MN-major, 8-key groups 4096 apart (LBO), 8-dim chunks 128 apart (SBO)
                        umma::mma_ts(tO_u, tP_u + 32 * h + ks * 8, umma::smem_desc(v_s + ks * 2 * 4096, 4096, 128), id_pv, ks > 0 ? 1u : acc0);
                    umma::commit(&v_free[h]);
                    umma::commit(&pv_done[h]);
                }
            }
            if (n_img < 2 && lead) umma::commit(&pv_done[1]);   // the half without keys
        };
        mbar_wait(q_ready, (uint32_t) (seg & 1), a.status);
        umma::fence_after_sync();
        if (ns_u > 0) issue_qk(0);
        for (int J = 0; J < ns_u; ++J) {
            if (J + 1 < ns_u) issue_qk(J + 1);
            issue_pv(J);
        }
        if (lead) umma::commit(o_done);
        __syncwarp();
    } else {
        // ---------------- softmax: two threads per row ----------------
        // Thread (row r, half hf) owns keys 64 hf .. 64 hf + 63 of every step and, in the epilogue, output dims 128 hf ..
        // The two warps that share 32 rows (warps w and w + 4, the same tensor-memory lanes) meet once per step at a
        // 64-thread barrier that ORs their "a maximum grew" votes; both keep the same reference maximum in registers.
        const int r = tid & (BM - 1), hf = tid >> 7, n = n0 + r;
        const int t_row = n / GQA;
        const int pos = n < R ? (a.lim ? a.lim[t_row] : a.p0 + t_row) : -1;
        const int pair_bar = 2 + (warp & 3);
        float * xch = reinterpret_cast<float *>(smem + SM_XCH);
        for (int J = 0; J < nsteps; ++J) {
            const int G = g + J;
            mbar_wait(s_full, (uint32_t) (G & 1), a.status);
            umma::fence_after_sync();
            uint32_t sr[2][32];
            umma::tmem_ld32(t_S + lane_off + 64 * hf, sr[0]);
            umma::tmem_ld32(t_S + lane_off + 64 * hf + 32, sr[1]);
            umma::tmem_ld_wait();
            umma::fence_before_sync();
            mbar_arrive(s_free);   // S is in registers: the next Q K^T may overwrite it
            const int k0 = a.kb + (st0 + J) * BP + 64 * hf;
            const bool diag = k0 + 63 > pos;   // some key of this half is masked for this row
            if (__any_sync(0xffffffffu, diag)) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        if (k0 + 32 * h + c > pos) sr[h][c] = __float_as_uint(B200_NEG_INF);
            }
            float mx4[4] = {B200_NEG_INF, B200_NEG_INF, B200_NEG_INF, B200_NEG_INF};   // four chains: the maximum is latency-bound
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int c = 0; c < 32; ++c) mx4[c & 3] = fmaxf(mx4[c & 3], __uint_as_float(sr[h][c]));
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            // lazy rescale: only when some row of the warp pair outgrew its reference maximum
            const int grow_here = mx > m_ref + RESCALE_GAP || (m_ref == B200_NEG_INF && mx != B200_NEG_INF);
            int grow_any;
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 q, %1, 0;\n\tbarrier.red.or.pred p, %2, 64, q;\n\tselp.s32 %0, 1, 0, p;\n\t}"
                         : "=r"(grow_any) : "r"(grow_here), "r"(pair_bar) : "memory");
            if (grow_any) {
                xch[hf * BM + r] = mx;
                asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");
                const float mxr = fmaxf(xch[r], xch[BM + r]);
                asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");   // both have read before the next use of xch
                float f = 1.0f;
                if (mxr > m_ref + RESCALE_GAP || (m_ref == B200_NEG_INF && mxr != B200_NEG_INF)) {
                    f = m_ref == B200_NEG_INF ? 0.0f : ex2f(m_ref - mxr);
                    m_ref = mxr;
                    l *= f;
                }
                if (J > 0 || carry_in) {
                    if (J > 0) mbar_wait(&pv_done[1], (uint32_t) ((G - 1) & 1), a.status);   // P V of step J-1 has landed in O
                    umma::fence_after_sync();
#pragma unroll 1
                    for (int c0 = hf * (DH / 2); c0 < (hf + 1) * (DH / 2); c0 += 32) {
                        uint32_t o[32];
                        umma::tmem_ld32(t_O + lane_off + c0, o);
                        umma::tmem_ld_wait();
#pragma unroll
                        for (int c = 0; c < 32; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * f);
                        umma::tmem_st32(t_O + lane_off + c0, o);
                    }
                    umma::tmem_st_wait();
                    umma::fence_before_sync();
                }
            }
            const float mref_safe = m_ref == B200_NEG_INF ? 0.0f : m_ref;
            if (G >= 1) mbar_wait(&pv_done[hf], (uint32_t) ((G - 1) & 1), a.status);   // this half of P is no longer read
            // P as f16 pairs into tensor memory: lane = row, this thread's 64 keys in columns 32 hf ..
            float l4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t w[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    // ex2(-inf) = 0: masked keys need no special case (mref_safe is finite)
                    const float p0 = ex2f(__uint_as_float(sr[h][2 * e]) - mref_safe);
                    const float p1 = ex2f(__uint_as_float(sr[h][2 * e + 1]) - mref_safe);
                    l4[e & 3] += p0 + p1;
                    w[e] = pack_h2(p0, p1);
                }
                umma::tmem_st16(t_P + lane_off + 32 * hf + 16 * h, w);
            }
            l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
            umma::tmem_st_wait();
            umma::fence_before_sync();
            mbar_arrive(&p_full[hf]);
        }
        // ---------------- epilogue ----------------
        // final:   O / l, gate, store (f32 and / or bf16, a16 copy);  carry_out: unnormalised O, (maximum, sum) for the next pass;
        // partial: unnormalised O with the maximum in natural-log units and the sum, for a merge across sequence shards
        const bool raw = carry_out || a.pm || piece;   // O leaves unnormalised
        const bool gated = any_gate && !raw, gate16 = a.gate == nullptr;
        const size_t slot = 2 * (size_t) blockIdx.x + (st0 == 0 ? 1 : 0);   // number of the piece
        // A warp owns 32 rows x 128 dims.  Its lanes read them back from a private shared-memory tile along the rows: in step i, lane l holds values
        // 4 (l mod 16) .. and 64 + 4 (l mod 16) .. of row 2 i + l / 16.  The gate values go out four steps ahead, raw (a conversion right behind
        // each load made the loads wait for one another: 12 us an epilogue instead of 3).
        const int lr = lane >> 4, lc = 4 * (lane & 15);
        auto row_at = [&](int i) {   // offset of the lane's first values in a result or gate array, or -1 past the last row
            const int nr = n0 + (warp & 3) * 32 + 2 * i + lr;
            const int tr = nr / GQA, hr = nr - tr * GQA;
            return nr < R ? (long long) ((size_t) tr * a.Hq + hk * GQA + hr) * DH + hf * (DH / 2) + lc : -1ll;
        };
        constexpr int AHEAD = 4, STEPS = 16;
        float4 gn[AHEAD][2];
        auto gate_ahead = [&](int i0) {   // rows past the last one: the first values of the array
            if (gate16) {
#pragma unroll
                for (int i = 0; i < AHEAD; ++i) {
                    const __nv_bfloat16 * p = a.gate_b + max(row_at(i0 + i), 0ll);
                    const float2 u = __ldg(reinterpret_cast<const float2 *>(p)), v = __ldg(reinterpret_cast<const float2 *>(p + 64));
                    gn[i][0].x = u.x; gn[i][0].y = u.y; gn[i][1].x = v.x; gn[i][1].y = v.y;
                }
            } else {
#pragma unroll
                for (int i = 0; i < AHEAD; ++i) {
                    const float * p = a.gate + max(row_at(i0 + i), 0ll);
                    gn[i][0] = __ldg(reinterpret_cast<const float4 *>(p)); gn[i][1] = __ldg(reinterpret_cast<const float4 *>(p + 64));
                }
            }
        };
        if (gated) gate_ahead(0);
        xch[hf * BM + r] = l;
        asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");
        l = xch[r] + xch[BM + r];
        mbar_wait(o_done, (uint32_t) (seg & 1), a.status);
        umma::fence_after_sync();
        const bool have_o = nsteps > 0 || carry_in;   // a tile that has seen no key at all (a sequence shard) holds nothing in O
        const float inv = raw ? 1.0f : (l > 0.0f ? 1.0f / l : 0.0f);
        if (n < R && hf == 0) {
            const size_t rowidx = (size_t) t_row * a.Hq + hk * GQA + (n - t_row * GQA);
            if (piece) a.pml[slot * BM + r] = make_float2(m_ref, l);
            else if (carry_out) { a.ml[rowidx * 2] = m_ref; a.ml[rowidx * 2 + 1] = l; }
            else if (a.pm) { a.pm[rowidx] = m_ref * 0.6931471805599453f; a.pl[rowidx] = l; }
        }
        float * tile = reinterpret_cast<float *>(smem + SM_EPI) + warp * (32 * EPI_STR);
#pragma unroll
        for (int c0 = 0; c0 < DH / 2; c0 += 32) {
            uint32_t o[32];
            if (have_o) {
                umma::tmem_ld32(t_O + lane_off + hf * (DH / 2) + c0, o);
                umma::tmem_ld_wait();
            } else {
#pragma unroll
                for (int c = 0; c < 32; ++c) o[c] = 0u;
            }
#pragma unroll
            for (int c = 0; c < 32; c += 4)
                *reinterpret_cast<float4 *>(tile + lane * EPI_STR + c0 + c) = make_float4(__uint_as_float(o[c]) * inv, __uint_as_float(o[c + 1]) * inv,
                                                                                          __uint_as_float(o[c + 2]) * inv, __uint_as_float(o[c + 3]) * inv);
        }
        __syncwarp();
        const size_t n_groups = (size_t) a.T * a.Hq * (DH / 32);
#pragma unroll 1
        for (int i0 = 0; i0 < STEPS; i0 += AHEAD) {
            float4 y[AHEAD][2];
            long long o[AHEAD];
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                o[i] = row_at(i0 + i);
#pragma unroll
                for (int h = 0; h < 2; ++h) y[i][h] = *reinterpret_cast<const float4 *>(tile + (2 * (i0 + i) + lr) * EPI_STR + 64 * h + lc);
            }
            if (gated) {
                float4 gv[AHEAD][2];
#pragma unroll
                for (int i = 0; i < AHEAD; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t u = __float_as_uint(gn[i][h].x), v = __float_as_uint(gn[i][h].y);
                        gv[i][h] = gate16 ? make_float4(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u), __uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u))
                                          : gn[i][h];
                    }
                if (i0 + AHEAD < STEPS) gate_ahead(i0 + AHEAD);
#pragma unroll
                for (int i = 0; i < AHEAD; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        y[i][h].x *= fast_sigmoid(gv[i][h].x); y[i][h].y *= fast_sigmoid(gv[i][h].y);
                        y[i][h].z *= fast_sigmoid(gv[i][h].z); y[i][h].w *= fast_sigmoid(gv[i][h].w);
                    }
            }
            if (!raw && a.out_b) {
#pragma unroll
                for (int i = 0; i < AHEAD; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const __nv_bfloat162 lo = __floats2bfloat162_rn(y[i][h].x, y[i][h].y), hi = __floats2bfloat162_rn(y[i][h].z, y[i][h].w);
                        if (o[i] >= 0) *reinterpret_cast<uint2 *>(a.out_b + o[i] + 64 * h) = make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
                    }
            } else {
                float * const p_out = a.po + (slot * BM + (warp & 3) * 32 + 2 * i0 + lr) * DH + hf * (DH / 2) + lc;
#pragma unroll
                for (int i = 0; i < AHEAD; ++i) {
                    float * dst = piece ? p_out + 2 * i * DH : a.out + o[i];
                    if (o[i] >= 0) { *reinterpret_cast<float4 *>(dst) = y[i][0]; *reinterpret_cast<float4 *>(dst + 64) = y[i][1]; }
                }
            }
            // the a16 copy for the projection that follows: eight lanes of a row hold one 32-value group
            if (a.qbuf && !raw) {
#pragma unroll
                for (int i = 0; i < AHEAD; ++i) {
                    a16_store_lanes8(y[i][0], a.qbuf, (size_t) o[i] / 32, n_groups, o[i] >= 0);
                    a16_store_lanes8(y[i][1], a.qbuf, (size_t) o[i] / 32 + 2, n_groups, o[i] >= 0);
                }
            }
        }
        umma::fence_async_smem();   // the epilogue tiles lie where the next segment's images are copied to
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    g += nsteps; g2 += ntiles >> 1;
    w += nsteps;
    if (w >= w_end) break;
    st0 = 0;
    if (++mtile == a.n_mtiles) { mtile = 0; ++hk; }
    }
    if (warp == 0) umma::tmem_dealloc(tb, 512);
}

// Adds up the pieces of the row tiles that the even split cut, in key order, and finishes them like prefill_k does: 1/l, gate, f32 or
// bf16 result, a16 copy.  grid (row tiles x 16, kv heads), a warp per row, eight values per lane: values 4 l .. 4 l + 3 of both 128-dim halves.  A chain
// of loads with little behind it: the gate and four pieces are asked for before the maximum is known (48 rows behind 10000 keys, two layers, 135 ->
// 124 us; 512 behind 16000 471 -> 463; before, one division and a search per piece's CTA and the loads one after the other).
__global__ void __launch_bounds__(256) prefill_merge_k(const pf_args a) {
    pdl_enter();
    const int m = blockIdx.x >> 4, hk = blockIdx.y, lane = threadIdx.x & 31;
    const int r = (blockIdx.x & 15) * 8 + (threadIdx.x >> 5), n = m * BM + r;
    // the CTAs that hold the tile's first and last step
    int before = 0;
    for (int m0 = 0; m0 < m; m0 += 32) before += m0 + lane < m ? pf_tile_steps(a.T, a.p0, m0 + lane) : 0;
    before = __reduce_add_sync(0xffffffffu, before);
    const long long W = (long long) a.Hkv * a.head_steps;
    const int first = hk * a.head_steps + before, last = first + pf_tile_steps(a.T, a.p0, m) - 1;
    // the CTA whose run holds a step: the largest c with floor(W c / n_run) <= step
    auto cta_of = [&](int step) {
        return W < (1 << 23) ? (int) (((unsigned) (step + 1) * (unsigned) a.n_run - 1u) / (unsigned) W) : (int) (((long long) (step + 1) * a.n_run - 1) / W);
    };
    const int c0 = cta_of(first), c1 = cta_of(last);
    if (c0 == c1 || n >= a.T * GQA) return;   // the whole tile ran in one CTA, which has written the result
    auto piece = [&](int c) { return (size_t) (c == c0 ? 2 * c + 1 : 2 * c) * BM + r; };
    // The gate and four pieces at a time are asked for together, whether they are there or not (a piece past the last is the last again, weight 0).
    const int t = n / GQA;
    const size_t row = ((size_t) t * a.Hq + hk * GQA + (n - t * GQA)) * DH;
    const bool gated = a.gate || a.gate_b;
    float4 gv[2];
    if (a.gate) {
        gv[0] = *reinterpret_cast<const float4 *>(a.gate + row + 4 * lane); gv[1] = *reinterpret_cast<const float4 *>(a.gate + row + 128 + 4 * lane);
    } else if (a.gate_b) {
        const float2 u = *reinterpret_cast<const float2 *>(a.gate_b + row + 4 * lane), v = *reinterpret_cast<const float2 *>(a.gate_b + row + 128 + 4 * lane);
        gv[0] = make_float4(u.x, u.y, 0.0f, 0.0f); gv[1] = make_float4(v.x, v.y, 0.0f, 0.0f);
    }
    constexpr int AHEAD = 4;
    float2 ml[AHEAD];
    float4 u[AHEAD], v[AHEAD];
    auto fetch = [&](int c) {
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            const size_t i = piece(min(c + k, c1));
            ml[k] = a.pml[i];
            u[k] = reinterpret_cast<const float4 *>(a.po + i * DH)[lane]; v[k] = reinterpret_cast<const float4 *>(a.po + i * DH)[32 + lane];
        }
    };
    fetch(c0);
    float M = B200_NEG_INF;
    for (int c = c0 + lane; c <= c1; c += 32) M = fmaxf(M, a.pml[piece(c)].x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    float l = 0.0f;
    float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f), y = x;
    for (int c = c0;;) {
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            if (c + k > c1) break;
            const float f = ml[k].x == B200_NEG_INF ? 0.0f : ex2f(ml[k].x - M);   // -inf: the row saw none of the piece's keys
            l = fmaf(f, ml[k].y, l);
            x.x = fmaf(f, u[k].x, x.x); x.y = fmaf(f, u[k].y, x.y); x.z = fmaf(f, u[k].z, x.z); x.w = fmaf(f, u[k].w, x.w);
            y.x = fmaf(f, v[k].x, y.x); y.y = fmaf(f, v[k].y, y.y); y.z = fmaf(f, v[k].z, y.z); y.w = fmaf(f, v[k].w, y.w);
        }
        if ((c += AHEAD) > c1) break;
        fetch(c);
    }
    const float inv = l > 0.0f ? 1.0f / l : 0.0f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float4 z = h ? y : x;
        const size_t o = row + 128 * h + 4 * lane;
        z.x *= inv; z.y *= inv; z.z *= inv; z.w *= inv;
        if (gated) {
            float4 g = gv[h];
            if (!a.gate) {
                const uint32_t p = __float_as_uint(g.x), q = __float_as_uint(g.y);
                g = make_float4(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u), __uint_as_float(q << 16), __uint_as_float(q & 0xffff0000u));
            }
            z.x *= fast_sigmoid(g.x); z.y *= fast_sigmoid(g.y); z.z *= fast_sigmoid(g.z); z.w *= fast_sigmoid(g.w);
        }
        if (a.out_b) {
            const __nv_bfloat162 lo = __floats2bfloat162_rn(z.x, z.y), hi = __floats2bfloat162_rn(z.z, z.w);
            *reinterpret_cast<uint2 *>(a.out_b + o) = make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
        } else *reinterpret_cast<float4 *>(a.out + o) = z;
        if (a.qbuf) a16_store_lanes8(z, a.qbuf, o / 32, (size_t) a.T * a.Hq * (DH / 32), true);
    }
}

// ------------------------------------------------------------------------------------------------ host side ----
constexpr size_t TILE_BYTES_PER_KEY = 2 * IMG / BN;   // K and V images: 1 KiB per key and kv head
constexpr int DEFAULT_PASS_KEYS = 8192;               // keys per pass that attn_fold_scratch_bytes(T, Hkv, 0, 0) provides for
constexpr size_t OWN_SCRATCH_TILE_CAP = (size_t) 640 << 20;   // library scratch holds tile images for at most this many bytes per pass,
constexpr size_t OWN_SCRATCH_TILE_LOW = (size_t) 256 << 20;   // or this many where that much memory cannot be had
constexpr size_t OWN_SCRATCH_PIECES = (size_t) 40 << 20;      // pieces of the even split: 2 x 148 of 128 rows of 1032 bytes

size_t align256(size_t v) { return (v + 255) & ~(size_t) 255; }
size_t ml_bytes(int T, int Hkv) { return align256((size_t) T * Hkv * GQA * 2 * sizeof(float)); }
size_t tile_bytes(int keys, int Hkv) { return (size_t) ((keys + BP - 1) / BP * BP) * Hkv * TILE_BYTES_PER_KEY; }

// Library scratch of the prefill entry points that take none from the caller: one buffer per (device, stream), sized on
// first use for the call at hand (tile images capped at OWN_SCRATCH_TILE_CAP per pass; longer contexts take more passes).
// A later call that needs more gets a new buffer (grow_buffer); the old one stays allocated until the process exits, so nothing is freed
// under work in flight and no stream is synchronised.
// Launches that share a buffer are queued as one block under its lock: another thread's call on the same stream comes before or after all of
// them.  Calls on other streams and devices do not wait for it (a launch may block on a full queue).
struct own_scratch {
    int dev = -1; cudaStream_t s = nullptr;
    grow_buffer b;
    std::mutex mu;
    unsigned long long user = 0; cudaEvent_t done = nullptr;   // g_pieces: the last stream that used the buffer and its last use
};
struct own_pool { own_scratch e[64]; int n = 0; };
own_pool g_own;      // tile images, carried state and pieces of calls without scratch of their own
own_pool g_pieces;   // pieces of calls with the caller's scratch that has no room for them
std::mutex g_pf_mu;         // the pools' lists

// the buffer of (current device, stream), nullptr if the pool is full
own_scratch * own_entry(own_pool & pool, cudaStream_t s) {
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_pf_mu);
    for (int i = 0; i < pool.n; ++i) if (pool.e[i].dev == dev && pool.e[i].s == s) return &pool.e[i];
    if (pool.n == 64) return nullptr;
    own_scratch * e = &pool.e[pool.n++];
    e->dev = dev; e->s = s;
    return e;
}
// at least `bytes` in the buffer, under its lock
bool own_grow(own_scratch * e, size_t bytes) {
    return e->b.need(bytes, OWN_SCRATCH_TILE_CAP + OWN_SCRATCH_PIECES, [](size_t want) {
        void * p = nullptr;
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;   // no other thread's recording is disturbed
        cudaThreadExchangeStreamCaptureMode(&mode);
        const cudaError_t rc = cudaMalloc(&p, want);
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (rc != cudaSuccess) { cudaGetLastError(); return (void *) nullptr; }
        return p;
    });
}

// Pieces for a call whose scratch is the caller's.  Such a call must not depend on what else runs on the GPU: a recorded one may be replayed
// anywhere, so it gets none; and a stream handle may stand for several streams (cudaStreamPerThread; the handle of a destroyed stream, given out
// again), so the buffer goes from one stream to the next through an event.  On success the buffer is locked and `user` is the stream's id.
own_scratch * pieces_acquire(size_t bytes, cudaStream_t s, std::unique_lock<std::mutex> & lk, unsigned long long & user) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    if (cap != cudaStreamCaptureStatusNone) return nullptr;
    if (cudaStreamGetId(s, &user) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    own_scratch * e = own_entry(g_pieces, s);
    if (!e) return nullptr;
    lk = std::unique_lock<std::mutex>(e->mu);
    bool ok = true;
    if (!e->done) {
        ok = cudaEventCreateWithFlags(&e->done, cudaEventDisableTiming) == cudaSuccess;
        e->user = user;
    } else if (e->user != user) ok = cudaStreamWaitEvent(s, e->done, 0) == cudaSuccess;
    if (!ok) cudaGetLastError();
    if (ok && own_grow(e, bytes)) return e;
    lk.unlock();
    return nullptr;
}
void pieces_release(own_scratch * e, cudaStream_t s, unsigned long long user) {
    if (cudaEventRecord(e->done, s) != cudaSuccess) cudaGetLastError();
    e->user = user;
}

// CTAs of the even split for rows p0 .. p0 + T - 1 (n_mtiles row tiles per kv head); 0 = one row tile per CTA.  Row tiles that are fewer than
// the SMs leave SMs idle for as long as the longest tile takes: they are cut, into at least two steps per CTA, if that is shorter by the
// time model below, in tenths of a microsecond, fitted to 1457 calls (T 5 .. 3000 behind 0 .. 65000 keys, q8_0 and q4_0, 1 / 2 / 4 heads, f32 and bf16
// forms) timed both ways in turn: a step 1.3 us, each further row tile in a CTA's run 8 us (prologue and epilogue), pieces and their merge 1 us and
// 0.06 us a CTA.  Measured, us, one row tile per CTA / cut: 4 heads, T = 48 behind 40000 keys 586 / 124, T = 512 behind 20000 323 / 256, T = 16
// behind 700 (bf16) 38 / 28; but T = 512 behind nothing 28 / 49, 2 heads, T = 1500 behind nothing 39 / 112 (the first runs cross six tiles of one
// step): those are left whole.  The choice is within 5 % of the better one on all but 31 of the calls, 13 % off at worst.
int split_ctas(int T, int p0, int n_mtiles, int Hkv, int sms, size_t image_bytes, int * head_steps) {
    const long long tiles = (long long) n_mtiles * Hkv;
    if (tiles >= sms) return 0;
    long long hs = 0;
    for (int m = 0; m < n_mtiles; ++m) hs += pf_tile_steps(T, p0, m);
    if (hs * Hkv >= 1 << 30) return 0;
    *head_steps = (int) hs;
    long long n = std::min<long long>(sms, hs * Hkv / 2);
    // Images that L2 does not hold (126 MB, shared with everything else) are read from HBM by every row tile that is elsewhere in the keys at
    // the time: the same number of runs for every tile keeps the tiles of a head at the same keys, if that leaves few SMs idle.
    // 48 rows behind 100003 keys (410 MB of images, three tiles a head): 368 -> 300 us.  512 rows behind 16000 (66 MB) would get 96 runs: not taken.
    const long long same = sms / tiles * tiles;
    const bool aligned = image_bytes > ((size_t) 64 << 20) && n == sms && same > tiles && same * 8 >= 7LL * sms;
    if (aligned) n = same;
    if (n <= tiles) return 0;
    // longest tile, longest run, most row tiles in a run
    const long long W = hs * Hkv, longest = pf_tile_steps(T, p0, n_mtiles - 1);
    long long run = 0, segs = 0, end = 0;
    int m = -1;   // row tile that holds the last step looked at; `end`: steps up to its end
    for (long long c = 0; c < n; ++c) {
        const long long a = W * c / n, b = W * (c + 1) / n;
        while (end <= a) { m = m + 1 == n_mtiles ? 0 : m + 1; end += pf_tile_steps(T, p0, m); }
        long long k = 1;
        while (end < b) { m = m + 1 == n_mtiles ? 0 : m + 1; end += pf_tile_steps(T, p0, m); ++k; }
        run = std::max(run, b - a);
        segs = std::max(segs, k);
    }
    // images beyond L2 with the tiles at different keys: every step is read from HBM, 128 KB at 6.5 TB/s (512 rows behind 65000 keys, 4 heads:
    // 948 / 977 us)
    const long long steps_us10 = std::max(13 * run, image_bytes > ((size_t) 144 << 20) && !aligned ? W / 5 : 0);
    return 100 * run <= 86 * longest && 13 * longest > steps_us10 + 80 * (segs - 1) + 10 + 6 * n / 10 ? (int) n : 0;
}

struct pf_io {
    const float * q; const __nv_bfloat16 * qb; const float * cs;
    const float * gate; const __nv_bfloat16 * gate_b;
    float * out; __nv_bfloat16 * out_b; float * pm, * pl; void * qbuf;
    const int32_t * lim;
};

// n_keys: keys the last row sees (p0 + T, or the host's bound on lim[T-1] + 1).  scratch == nullptr: library scratch.
int prefill_run(const pf_io & io, const b200_kv_cache * c, int T, int p0, int n_keys, int Hq, float scale, void * scratch,
                size_t scratch_bytes, cudaStream_t s, const char * who) {
    if (!c || (!io.q && !io.qb) || (!io.out && !io.out_b) || !c->k || !c->v) B200_REFUSE(B200_ERR_SHAPE, "%s: null argument", who);
    if (c->D != DH || Hq != GQA * c->Hkv || c->Hkv <= 0 || T < 1 || p0 < 0 || n_keys < 0)
        B200_REFUSE(B200_ERR_SHAPE, "%s: unsupported shape (D=%d Hq=%d Hkv=%d T=%d p0=%d)", who, c->D, Hq, c->Hkv, T, p0);
    if (c->type != B200_KV_F16 && c->type != B200_KV_Q8_0 && c->type != B200_KV_Q4_0) B200_REFUSE(B200_ERR_SHAPE, "%s: unsupported cache type %u", who, c->type);
    if (!aligned16(c->k) || !aligned16(c->v) || (io.q && !aligned16(io.q)) || (io.qb && !aligned16(io.qb)) || (io.out && !aligned16(io.out)) ||
        (io.out_b && !aligned16(io.out_b)) || (io.gate && !aligned16(io.gate)) || (io.gate_b && !aligned16(io.gate_b)) ||
        (c->pt && c->pstride % 16) || (io.qbuf && ((uintptr_t) io.qbuf & 3)))
        B200_REFUSE(B200_ERR_SHAPE, "%s: cache base, page stride, q, out and gate must be 16-byte aligned", who);
    if (!c->pt && n_keys > c->n_ctx) B200_REFUSE(B200_ERR_SHAPE, "%s: keys 0..%d outside n_ctx %d", who, n_keys - 1, c->n_ctx);
    if (io.pm && (!io.pl || !io.out)) B200_REFUSE(B200_ERR_SHAPE, "%s: the partial form needs part_o, part_m and part_l", who);
    // scratch: [running (max, sum) per row][running O when the result leaves as bf16 only][tile images of one pass]
    const size_t fixed = ml_bytes(T, c->Hkv);
    const size_t carry = io.out ? 0 : align256((size_t) T * Hq * DH * sizeof(float));
    const size_t per_step = (size_t) BP * c->Hkv * TILE_BYTES_PER_KEY;
    const size_t full = tile_bytes(std::max(n_keys, 1), c->Hkv);
    // row tiles cut between n_run CTAs (calls of one pass): pieces behind the images
    int dev = 0, sms = 148, head_steps = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int n_mtiles = (T * GQA + BM - 1) / BM;
    const int n_run = io.lim || io.pm ? 0 : split_ctas(T, p0, n_mtiles, c->Hkv, sms, full, &head_steps);
    const size_t pml_bytes = align256((size_t) 2 * n_run * BM * sizeof(float2)), piece_bytes = n_run ? pml_bytes + (size_t) 2 * n_run * BM * DH * sizeof(float) : 0;
    std::unique_lock<std::mutex> lk;
    const bool own = !scratch;
    if (own) {
        own_scratch * e = own_entry(g_own, s);
        if (e) lk = std::unique_lock<std::mutex>(e->mu);
        size_t want = 0;
        for (const size_t cap : {OWN_SCRATCH_TILE_CAP, OWN_SCRATCH_TILE_LOW}) {
            const size_t images = std::min(full, std::max(cap / per_step, (size_t) 1) * per_step);
            for (const size_t extra : {images == full ? piece_bytes : 0, (size_t) 0}) {
                want = fixed + carry + images + extra + 256;
                if (e && own_grow(e, want)) { scratch = e->b.p; scratch_bytes = e->b.cap; break; }
                if (!extra) break;
            }
            if (scratch) break;
        }
        if (!scratch) B200_REFUSE(B200_ERR_ALLOC, "%s: %zu bytes of scratch could not be allocated", who, want);
    } else if ((uintptr_t) scratch & 255) {
        B200_REFUSE(B200_ERR_SCRATCH, "%s: scratch must be 256-byte aligned", who);
    }
    // one pass if the tile images of every visible key fit (no running O is needed then), else as many keys per pass as fit
    // (of the library's buffer no more than its cap, whatever an earlier call made of it: the passes depend on this call alone)
    const size_t most = own ? std::max(OWN_SCRATCH_TILE_CAP / per_step, (size_t) 1) : (size_t) 1 << 40;
    size_t steps_fit = std::min(most, scratch_bytes > fixed ? (scratch_bytes - fixed) / per_step : 0);
    bool multi = steps_fit * per_step < full;
    if (multi) steps_fit = std::min(most, scratch_bytes > fixed + carry ? (scratch_bytes - fixed - carry) / per_step : 0);
    if (steps_fit < 1)
        B200_REFUSE(B200_ERR_SCRATCH, "%s: scratch too small (%zu bytes given; %zu needed for one 128-key step, %zu for a single pass over %d keys)",
                    who, scratch_bytes, fixed + carry + per_step, fixed + full, n_keys);
    const long long keys_per_pass = (long long) std::min<size_t>(steps_fit, (size_t) 1 << 22) * BP;
    unsigned * st = device_status_word();
    if (!st) return B200_ERR_CUDA;
    static std::atomic<bool> attr_done[64];
    if (!attr_done[dev & 63].load(std::memory_order_acquire)) {
        if (cudaFuncSetAttribute(prefill_k, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_TOTAL) != cudaSuccess)
            return launch_status("attn_prefill (shared memory attribute)");
        attr_done[dev & 63].store(true, std::memory_order_release);
    }
    unsigned char * base = (unsigned char *) scratch;
    pf_args a;
    a.q = io.q; a.qb = io.q ? nullptr : io.qb; a.cs = io.cs;
    a.gate = io.gate; a.gate_b = io.gate ? nullptr : io.gate_b;
    a.ml = reinterpret_cast<float *>(base);
    a.out = io.out ? io.out : multi ? reinterpret_cast<float *>(base + fixed) : nullptr;
    a.out_b = io.out_b; a.pm = io.pm; a.pl = io.pl; a.qbuf = (__half2 *) io.qbuf; a.lim = io.lim;
    unsigned char * tiles = base + fixed + (multi ? carry : 0);
    a.tiles = tiles;
    a.T = T; a.p0 = p0; a.Hq = Hq; a.Hkv = c->Hkv; a.qscale = scale * LOG2E_PF; a.status = st;
    const kv_view g = view_of(*c);
    a.n_run = 0; a.n_mtiles = n_mtiles; a.head_steps = head_steps; a.po = nullptr; a.pml = nullptr;
    own_scratch * lent = nullptr;
    unsigned long long user = 0;
    if (n_run && !multi) {
        unsigned char * pieces = nullptr;
        if (scratch_bytes >= fixed + full + piece_bytes) pieces = base + fixed + full;
        else if (!own && (lent = pieces_acquire(piece_bytes, s, lk, user)) != nullptr) pieces = (unsigned char *) lent->b.p;
        if (pieces) {   // else one row tile per CTA
            a.n_run = n_run;
            a.pml = reinterpret_cast<float2 *>(pieces);
            a.po = reinterpret_cast<float *>(pieces + pml_bytes);
        }
    }
    int launches = 0;
    long long kb = 0;
    do {   // at least one pass, also when no key is visible (a sequence shard that owns nothing yet): it writes the empty result
        const long long ke = std::min<long long>(kb + keys_per_pass, std::max(n_keys, 1));
        const int n_tiles = (int) ((ke - kb + BN - 1) / BN);
        const dim3 tg(n_tiles, c->Hkv);
        if (c->type == B200_KV_F16) launch(kv_tiles_k<B200_KV_F16>, tg, 256, 0, s, g, (int) kb, n_keys, tiles, n_tiles, st);
        else if (c->type == B200_KV_Q8_0) launch(kv_tiles_k<B200_KV_Q8_0>, tg, 256, 0, s, g, (int) kb, n_keys, tiles, n_tiles, st);
        else launch(kv_tiles_k<B200_KV_Q4_0>, tg, 256, 0, s, g, (int) kb, n_keys, tiles, n_tiles, st);
        a.n_tiles = n_tiles; a.kb = (int) kb; a.ke = (int) ke;
        const dim3 pg = a.n_run ? dim3(a.n_run) : dim3(n_mtiles, c->Hkv);
        // few images: early launches (see `launch`) save two gaps, 77 rows behind nothing, four layers 92 -> 77 us; behind a grid of several waves the early
        // CTAs are in the way (512 rows behind 16000 keys, two layers 462 -> 476)
        if ((size_t) tg.x * tg.y < PDL_MAX_CTAS) launch(prefill_k, pg, NTHR_PF, SM_TOTAL, s, a);
        else prefill_k<<<pg, NTHR_PF, SM_TOTAL, s>>>(a);
        launches += 2;
        if (a.n_run) {
            launch(prefill_merge_k, dim3(n_mtiles * (BM / 8), c->Hkv), 256, 0, s, a);
            ++launches;
        }
        kb = ke;
    } while (kb < n_keys);
    if (lent) pieces_release(lent, s, user);
    count_launch(launches);
    return launch_status(who);
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" {

int b200_attn_prefill(const float * q, const b200_kv_cache * c, float * out, int T, int p0, int Hq, float scale, void * stream) {
    const pf_io io = {q, nullptr, nullptr, nullptr, nullptr, out, nullptr, nullptr, nullptr, nullptr, nullptr};
    return prefill_run(io, c, T, p0, p0 + T, Hq, scale, nullptr, 0, (cudaStream_t) stream, "attn_prefill");
}
int b200_attn_prefill_variant(const float * q, const b200_kv_cache * c, float * out, int T, int p0, int Hq, float scale, void * stream,
                              int variant) {
    (void) variant;   // the reference's variants are bitwise-equal schedules of one fp32 algorithm; there is one kernel here
    return b200_attn_prefill(q, c, out, T, p0, Hq, scale, stream);
}
// Scratch for passes of `chunk` keys (chunk <= 0: DEFAULT_PASS_KEYS); any amount from one 128-key step upwards works, a
// context that does not fit takes more passes.  nsplit has no meaning here.
size_t b200_attn_fold_scratch_bytes(int T, int Hkv, int chunk, int nsplit) {
    (void) nsplit;
    if (T < 1 || Hkv < 1) return 0;
    return ml_bytes(T, Hkv) + tile_bytes(chunk > 0 ? chunk : DEFAULT_PASS_KEYS, Hkv);
}
int b200_attn_fold(const float * q, const b200_kv_cache * c, float * out, int T, int p0, int Hq, float scale, void * scratch,
                   size_t scratch_bytes, void * stream, int chunk, int nsplit) {
    (void) nsplit;
    if (!scratch) B200_REFUSE(B200_ERR_SCRATCH, "attn_fold: scratch is null");
    if (chunk > 0 && c && c->Hkv > 0 && T > 0)   // the caller's chunk caps the keys per pass (it may be smaller than the scratch allows)
        scratch_bytes = std::min(scratch_bytes, ml_bytes(T, c->Hkv) + tile_bytes(chunk, c->Hkv));
    const pf_io io = {q, nullptr, nullptr, nullptr, nullptr, out, nullptr, nullptr, nullptr, nullptr, nullptr};
    return prefill_run(io, c, T, p0, p0 + T, Hq, scale, scratch, scratch_bytes, (cudaStream_t) stream, "attn_fold");
}
int b200_attn_prefill_gated(const float * q, const b200_kv_cache * c, float * out, const float * gate, int T, int p0, int Hq,
                            float scale, void * scratch, size_t scratch_bytes, void * stream) {
    const pf_io io = {q, nullptr, nullptr, gate, nullptr, out, nullptr, nullptr, nullptr, nullptr, nullptr};
    return prefill_run(io, c, T, p0, p0 + T, Hq, scale, scratch, scratch_bytes, (cudaStream_t) stream, "attn_prefill_gated");
}
int b200_attn_prefill_gated_a16(const float * q, const b200_kv_cache * c, float * out, const float * gate, void * qbuf, int T, int p0,
                                int Hq, float scale, void * scratch, size_t scratch_bytes, void * stream) {
    if (!qbuf || !out) B200_REFUSE(B200_ERR_SHAPE, "attn_prefill_gated_a16: out / qbuf is null");
    const pf_io io = {q, nullptr, nullptr, gate, nullptr, out, nullptr, nullptr, nullptr, qbuf, nullptr};
    return prefill_run(io, c, T, p0, p0 + T, Hq, scale, scratch, scratch_bytes, (cudaStream_t) stream, "attn_prefill_gated_a16");
}
int b200_attn_prefill_partial(const float * q, const b200_kv_cache * c, float * part_o, float * part_m, float * part_l,
                              const int32_t * last_key, int max_keys, int T, int Hq, float scale, void * scratch, size_t scratch_bytes,
                              void * stream) {
    if (!last_key || !part_o || !part_m || !part_l) B200_REFUSE(B200_ERR_SHAPE, "attn_prefill_partial: null argument");
    const pf_io io = {q, nullptr, nullptr, nullptr, nullptr, part_o, nullptr, part_m, part_l, nullptr, last_key};
    return prefill_run(io, c, T, 0, max_keys, Hq, scale, scratch, scratch_bytes, (cudaStream_t) stream, "attn_prefill_partial");
}

size_t b200_attn_prefill_bf16_scratch_bytes(int T, int Hkv, int pass_keys, int out_is_bf16) {
    if (T < 1 || Hkv < 1) return 0;
    const size_t carry = out_is_bf16 ? align256((size_t) T * Hkv * GQA * DH * sizeof(float)) : 0;
    return align256((size_t) T * 64 * sizeof(float)) + ml_bytes(T, Hkv) + carry + tile_bytes(pass_keys > 0 ? pass_keys : DEFAULT_PASS_KEYS, Hkv);
}
int b200_attn_prefill_bf16(const uint16_t * q, const uint16_t * k, const uint16_t * v, const float * gate_f32,
                           const uint16_t * gate_bf16, float * out_f32, uint16_t * out_bf16, void * qbuf, const b200_kv_cache * c,
                           int p0, int T, int Hq, int n_rot, float freq_base, float scale, void * scratch, size_t scratch_bytes,
                           void * stream) {
    const char * who = "attn_prefill_bf16";
    if (!q || !k || !v || !c || !scratch) B200_REFUSE(B200_ERR_SHAPE, "%s: null argument (scratch is required)", who);
    if (n_rot != 64 || c->D != DH || T < 1) B200_REFUSE(B200_ERR_SHAPE, "%s: needs D = 256 and n_rot = 64 (got D=%d n_rot=%d)", who, c->D, n_rot);
    if (((uintptr_t) scratch & 255)) B200_REFUSE(B200_ERR_SCRATCH, "%s: scratch must be 256-byte aligned", who);
    const size_t cs_bytes = align256((size_t) T * 64 * sizeof(float));
    if (scratch_bytes <= cs_bytes) B200_REFUSE(B200_ERR_SCRATCH, "%s: scratch too small", who);
    float * cs = reinterpret_cast<float *>(scratch);
    // K: rotation + quantise + append, V: quantise + append; the tokens' cos / sin go to the table the attention kernel reads
    const int rc = rope_append_launch(nullptr, k, v, nullptr, cs, c, p0, T, Hq, c->Hkv, DH, n_rot, freq_base, (cudaStream_t) stream, who);
    if (rc != B200_OK) return rc;
    const pf_io io = {nullptr, (const __nv_bfloat16 *) q, cs, gate_f32, (const __nv_bfloat16 *) gate_bf16, out_f32,
                      (__nv_bfloat16 *) out_bf16, nullptr, nullptr, qbuf, nullptr};
    return prefill_run(io, c, T, p0, p0 + T, Hq, scale, (unsigned char *) scratch + cs_bytes, scratch_bytes - cs_bytes,
                       (cudaStream_t) stream, who);
}

}  // extern "C"
