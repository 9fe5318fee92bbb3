// Batched decode of quantised caches with one or two row tiles (q8_0: one row per slot, q4_0: one or two) in the even split of a batch: mma.sync
// with warps that never wait for one another inside a unit of work.  Included by attn_decode.cu inside its namespace.
//
// A run of the plan belongs to two warps; warp w takes keys 32 w .. 32 w + 31 of every 64 and walks them by itself: its own ring of TMA copies (32
// rows of K, 32 rows of V), its own reference maxima, sums and output accumulators.  P never leaves the registers: the accumulator
// fragment of Q K^T, packed to f16, becomes the operand fragment of P V by a transposing register move (movmatrix).  The two warps meet where a
// segment ends and add up their (O, m, l) through shared memory.  A CTA of four warps works on two runs at a time.
//
// What bounds decode_part_k there (four warps sharing each tile of 64 keys, P and the V scales through shared memory, one block barrier and one
// poll per tile) is waiting: q4_0, one row, 57 warp instructions per key and kv head issued at 0.65 of the rate, the largest stall the barrier; a
// fifth fewer instructions in that structure changed nothing (697 -> 694 us, 16 slots of 131072 keys).  Here a warp's tile has 32 keys, so that query fragments,
// waits and refills are paid once per 32 keys instead of per 16, and nothing waits but for its own copies: 700 -> 614 us; q8_0, 16 slots of 65536 keys, two
// layers 885 -> 800; q4_0, 16 slots x 2 rows of 32768 keys, two layers 514 -> 456.  What is left is the integer pipe (0.55 of its rate at 44
// instructions per key, 20 of them on it) and the latency of dependent instructions.
//
// Accumulators: q8_0 keeps O in registers (64 per thread; shared memory holds eight warps' rings only).  q4_0 keeps it in tensor memory, this warp's own 32
// lanes, and passes it through registers 32 dims at a time, once per tile: 16 warps per SM instead of 12 (one row: 620 -> 614 us and, one slot of
// 131000 keys, 297 -> 279).  With three row tiles (q_len 3, 4) tensor memory holds eight warps and this kernel is slower than decode_part_k
// (654 us for 614), so those stay there, and with them all fixed chunks, whose rows are bitwise independent of q_len.
constexpr int WT = 32;                        // keys of a warp's tile
constexpr int WU_THR = 64;                    // threads that share a run
constexpr int WK_THR = 128;                   // threads of a CTA: two runs
constexpr int WK_TAB = 1088;                  // per warp: block scales, of K as floats [key][8] or of V as f16 [block][WK_SD bytes]
constexpr int WK_SD = 68;
constexpr int WK_ML = 128, WK_Q = 384;        // offsets in a unit's shared memory: (m, l) of the two warps [2][2][16], query rows

template <uint32_t KT, int NT> struct wk {
    static constexpr int SLOT = WT * head_bytes(KT);
    static constexpr int QB = WK_Q + NT * 8 * QSTR;                           // block sums of Q
    static constexpr int TAB = QB + NBLK * NT * 4 * 16;
    static constexpr int RING = (TAB + 2 * WK_TAB + 127) / 128 * 128;
    static constexpr bool TM = KT == B200_KV_Q4_0;                             // O in tensor memory
    static constexpr int CTAS = KT == B200_KV_Q8_0 ? 2 : NT == 1 ? 4 : 3;      // per SM
    static constexpr size_t unit_bytes(int nslot) { return RING + (size_t) 2 * nslot * SLOT; }
    static constexpr size_t smem(int nslot) { return 2 * unit_bytes(nslot) + 128; }
    static constexpr int slots() {
        int n = 2;
        while (n < 8 && CTAS * (smem(n + 1) + 1024) <= (size_t) 227 * 1024) ++n;
        return n;
    }
    static_assert(CTAS * (smem(2) + 1024) <= (size_t) 227 * 1024, "two slots fit");
};

__device__ __forceinline__ uint32_t movm_trans(uint32_t x) {
    uint32_t r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}
__device__ __forceinline__ void bar_unit(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(WU_THR) : "memory"); }

// the 8 NT accumulators of one 32-dim block: columns from 8 NT b of the warp's lanes
__device__ __forceinline__ void wk_ld(uint32_t t, float (&o)[2][1][4]) {
    uint32_t r[8];
    umma::tmem_ld8(t, r);
#pragma unroll
    for (int e = 0; e < 8; ++e) (&o[0][0][0])[e] = __uint_as_float(r[e]);
}
__device__ __forceinline__ void wk_ld(uint32_t t, float (&o)[2][2][4]) {
    uint32_t r[16];
    umma::tmem_ld16(t, r);
#pragma unroll
    for (int e = 0; e < 16; ++e) (&o[0][0][0])[e] = __uint_as_float(r[e]);
}
__device__ __forceinline__ void wk_st(uint32_t t, const float (&o)[2][1][4]) {
    uint32_t r[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) r[e] = __float_as_uint((&o[0][0][0])[e]);
    umma::tmem_st8(t, r);
}
__device__ __forceinline__ void wk_st(uint32_t t, const float (&o)[2][2][4]) {
    uint32_t r[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) r[e] = __float_as_uint((&o[0][0][0])[e]);
    umma::tmem_st16(t, r);
}

template <uint32_t KT, int NT>
__global__ void __launch_bounds__(WK_THR, wk<KT, NT>::CTAS)
decode_warp_k(const dec_args a, const int n_runs, const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapV) {
    pdl_enter();
    using W = wk<KT, NT>;
    constexpr int HB = head_bytes(KT), SLOT = W::SLOT, nslot = W::slots();
    constexpr bool Q8 = KT == B200_KV_Q8_0, TM = W::TM;
    constexpr uint32_t TCOLS = 64 * NT;
    static_assert(NT <= 2, "one or two row tiles");
    static_assert(nslot * SLOT >= 4 * 2 * NT * 32 * 16, "the two warps hand each other half of O through their rings");
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, v = warp >> 1, w = warp & 1, ut = tid & (WU_THR - 1), g = lane >> 2, t = lane & 3;
    unsigned char * us = smem + 128 + v * W::unit_bytes(nslot);
    uint64_t * full = reinterpret_cast<uint64_t *>(us) + w * 8;
    float * ml = reinterpret_cast<float *>(us + WK_ML);                       // [2 warps][2][16]
    unsigned char * Qs = us + WK_Q;
    float4 * Qb = reinterpret_cast<float4 *>(us + W::QB);
    unsigned char * tabs = us + W::TAB + w * WK_TAB;
    unsigned char * ring = us + W::RING + (size_t) w * nslot * SLOT, * ring_o = us + W::RING + (size_t) (1 - w) * nslot * SLOT;
    const int bar = 1 + v, R = a.q_len * GQA;

    if (lane == 0) {
        for (int s = 0; s < nslot; ++s) mbar_init(&full[s], 1);
        mbar_fence_init();
    }
    uint32_t t_O = 0;
    if constexpr (TM) {
        uint32_t * t_slot = reinterpret_cast<uint32_t *>(smem);
        if (warp == 0) umma::tmem_alloc(t_slot, TCOLS);
        umma::fence_before_sync();
        __syncthreads();
        umma::fence_after_sync();
        t_O = *t_slot + ((uint32_t) (32 * warp) << 16);
    } else __syncwarp();

    // the run of this pair of warps; kv head = run index mod heads, as in decode_part_k.  n_runs: runs of all heads the grid was made for
    const int vi = (int) blockIdx.x * 2 + v, hl = vi % a.nhk, ui = vi / a.nhk, hk = a.hk0 + hl;
    int s0 = 0, s1 = 0;
    {
        const int c = min(ui, a.max_cta - 1), n = *a.n_cta, c0 = a.cta_seg[c], c1 = a.cta_seg[c + 1];   // loads that do not wait for one another
        if (vi < n_runs && ui < n) { s0 = c0; s1 = c1; }
    }

    int sc = 0;              // ring slot of the next item to be consumed; a segment starts and ends with an empty ring
    uint32_t ph = 0;         // and the parity of its use
    int q_slot_of = -1;      // slot whose query rows are staged
    int n_slot = 0, rmin = 0;
    int rpos[NT][2];
    for (int u = s0; u < s1; ++u) {
        const int4 seg = a.segs[u];
        const int slot = seg.x, k_lo = seg.y;
        const unsigned unit = (unsigned) u * a.nhk + hl;
        if (slot != q_slot_of) {   // visible keys = 1 + the largest row position
            n_slot = 0; rmin = 0x7fffffff;
            for (int j = 0; j < a.q_len; ++j) { const int p = row_pos(a, slot, j); n_slot = max(n_slot, p + 1); rmin = min(rmin, p); }
            const int lim = key_limit(a);
            if (n_slot > lim) { if (ut == 0) atomicOr(a.status, ST_BAD_POS); n_slot = lim; }
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int r = 8 * i + 2 * t + e;
                    rpos[i][e] = r < R ? row_pos(a, slot, r / GQA) : -1;
                }
        }
        const int k_hi = min(seg.z, n_slot);
        if (k_lo >= k_hi) continue;
        const int32_t * tab = a.g.pt ? a.g.pt + (a.g.rtab ? a.g.rtab[slot * a.q_len] : 0) : nullptr;
        {
            const int mine = k_hi - k_lo - WT * w, nt = mine > 0 ? (mine + 63) / 64 : 0;
            // page entries: lane l holds that of page pg0 + l
            const int pg_last = (k_hi - 1) >> a.g.psh;
            int pg0 = (k_lo + WT * w) >> a.g.psh;
            int pgv = tab && nt ? tab[min(pg0 + lane, pg_last)] : 0;
            int qi = 0, si = sc;   // next item (2 tile: K, 2 tile + 1: V) to be fetched and its slot
            int p_t = k_lo + WT * w, z = 0;   // first position of its tile and the page that holds it
            auto issue = [&]() {   // by the whole warp; the slot is empty
                if (qi >= 2 * nt) return;
                unsigned char * dst = ring + si * SLOT;
                if (tab && !(qi & 1)) {
                    int pi = (p_t >> a.g.psh) - pg0;
                    if (pi >= 32) { pg0 += pi; pi = 0; pgv = tab[min(pg0 + lane, pg_last)]; }
                    z = __shfl_sync(0xffffffffu, pgv, pi);
                    if (z < 0) { if (lane == 0) atomicOr(a.status, ST_BAD_PAGE); z = 0; }
                }
                const int y = tab ? p_t & ((1 << a.g.psh) - 1) : p_t;
                if (a.tiled) {
                    if (lane == 0) {
                        mbar_expect_tx(&full[si], (uint32_t) SLOT);
                        tma_box3(dst, (qi & 1) ? &mapV : &mapK, hk * (HB / 2), y, z, &full[si]);
                    }
                } else {   // row by row through registers; rows past the last key are that key's
                    constexpr int CPR = HB / 16;
                    const char * base = ((qi & 1) ? a.g.v : a.g.k) + (unsigned long long) hk * HB;
                    for (int idx = lane; idx < WT * CPR; idx += 32) {
                        const int row = idx / CPR, c = idx - row * CPR, p = min(p_t + row, n_slot - 1);
                        unsigned long long off = (unsigned long long) p * a.g.rowb;
                        if (tab) {
                            const int pg = tab[p >> a.g.psh];
                            if (pg < 0) { atomicOr(a.status, ST_BAD_PAGE); off = 0; }
                            else off = (unsigned long long) pg * a.g.pstride + (unsigned long long) (p & ((1 << a.g.psh) - 1)) * a.g.rowb;
                        }
                        *reinterpret_cast<uint4 *>(dst + row * HB + c * 16) = __ldg(reinterpret_cast<const uint4 *>(base + off) + c);
                    }
                    __syncwarp();
                    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full[si])) : "memory");
                }
                if (qi & 1) p_t += 64;
                ++qi;
                if (++si == nslot) si = 0;
            };
            for (int s = 0; s < nslot; ++s) issue();

            if (slot != q_slot_of) {
                // Q rows -> shared memory as f16, scaled; row r = j * 6 + hh (verify row j, head hh of the group).  The middle two of every four dims
                // are swapped (d0 d2 d1 d3): a 32-bit word of cache bytes then splits into the f16 pairs (byte 0, byte 2) and (byte 1, byte 3)
                // with one mask each.  q4_0: the high nibbles (dims 16 .. 31 of a block) enter the MMA where they stand in the byte, 16 times their
                // value, so their query dims are 1/16.
                if (q_slot_of >= 0) bar_unit(bar);   // the other warp is done with the rows of the slot before
                for (int i = ut; i < NT * 8 * (DH / 4); i += WU_THR) {
                    const int r = i / (DH / 4), d4 = (i - r * (DH / 4)) * 4;
                    float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (r < R) {
                        const int j = r / GQA, hh = r - j * GQA;
                        x = *reinterpret_cast<const float4 *>(a.q + ((size_t) (slot * a.q_len + j) * a.Hq + hk * GQA + hh) * DH + d4);
                    }
                    const float qs = !Q8 && (d4 & 16) ? a.qscale * 0.0625f : a.qscale;
                    *reinterpret_cast<uint2 *>(Qs + r * QSTR + q_slot<KT>(d4) * 2) = make_uint2(pack_h2(x.x * qs, x.z * qs), pack_h2(x.y * qs, x.w * qs));
                }
                bar_unit(bar);
                // The cache integers enter the tensor cores as f16 subnormals u * 2^-24 with u = q + 128 (q8_0) or the nibble itself (q4_0, value =
                // nibble - 8).  The offset is taken out again through the accumulator's starting value: for block b and row r it is
                // -OFFS * 2^-24 * (sum of the block's 32 scaled f16 query values), in the order of an accumulator fragment {row 2t, row 2t+1, row 2t, row 2t+1}.
                constexpr float OFFS = Q8 ? 128.0f : 8.0f;
                for (int i = ut; i < NBLK * NT * 8; i += WU_THR) {
                    const int b = i / (NT * 8), r = i - b * (NT * 8);
                    const __half2 * src = reinterpret_cast<const __half2 *>(Qs + r * QSTR + b * 64);   // a block's dims stay inside its 64 bytes
                    float sum = 0.0f;
#pragma unroll
                    for (int e = 0; e < 16; ++e) { const float2 f = __half22float2(src[e]); sum += (!Q8 && (e & 2) ? 16.0f : 1.0f) * (f.x + f.y); }
                    const float x = -OFFS * 5.9604644775390625e-8f * sum;
                    float * dst = reinterpret_cast<float *>(Qb + (b * NT + (r >> 3)) * 4 + ((r & 7) >> 1));
                    dst[r & 1] = x; dst[2 + (r & 1)] = x;
                }
                bar_unit(bar);
                q_slot_of = slot;
            }

            float m_run[NT][2], l_run[NT][2];
            float O[TM ? 1 : NBLK][2][NT][4];
            uint32_t v_exp = 0;   // nibble b: O of block b is kept times 2^-nibble (see P V)
#pragma unroll
            for (int i = 0; i < NT; ++i) { m_run[i][0] = m_run[i][1] = B200_NEG_INF; l_run[i][0] = l_run[i][1] = 0.0f; }
#pragma unroll
            for (int b = 0; b < (TM ? 1 : NBLK); ++b)
#pragma unroll
                for (int e = 0; e < 8 * NT; ++e) (&O[b][0][0][0])[e] = 0.0f;
            if constexpr (TM) {
                for (int b = 0; b < NBLK; ++b) wk_st(t_O + 8 * NT * b, O[0]);
                umma::tmem_st_wait();
            }
            // multiplies all accumulators of a row by f[row]
            auto scale_O = [&](const float (&f)[NT][2]) {
                auto one = [&](float (&o)[2][NT][4]) {
#pragma unroll
                    for (int x = 0; x < 2; ++x)
#pragma unroll
                        for (int i = 0; i < NT; ++i) { o[x][i][0] *= f[i][0]; o[x][i][1] *= f[i][1]; o[x][i][2] *= f[i][0]; o[x][i][3] *= f[i][1]; }
                };
                if constexpr (TM) {
#pragma unroll 1
                    for (int b = 0; b < NBLK; ++b) {
                        wk_ld(t_O + 8 * NT * b, O[0]);
                        umma::tmem_ld_wait();
                        one(O[0]);
                        wk_st(t_O + 8 * NT * b, O[0]);
                    }
                    umma::tmem_st_wait();
                } else {
#pragma unroll
                    for (int b = 0; b < NBLK; ++b) one(O[b]);
                }
            };
            const int mask_from = min(k_hi, rmin + 1);

            for (int it = 0; it < nt; ++it) {
                const int k_t = k_lo + it * 64 + WT * w;   // first key of the tile
                const unsigned char * Ks = ring + sc * SLOT;
                mbar_wait(&full[sc], ph, a.status);
                if (++sc == nslot) { sc = 0; ph ^= 1u; }
                // ---------------- block scales of K as floats: lane = key ----------------
                {
                    const unsigned char * row = Ks + lane * HB;
                    float f[8];
                    if constexpr (Q8) {
                        const uint4 x = *reinterpret_cast<const uint4 *>(row);
                        const uint32_t xw[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) { const float2 p = __half22float2(*reinterpret_cast<const __half2 *>(&xw[e])); f[2 * e] = p.x; f[2 * e + 1] = p.y; }
                    } else {
#pragma unroll
                        for (int b = 0; b < NBLK; ++b) f[b] = __half2float(*reinterpret_cast<const __half *>(row + 18 * b));
                    }
                    float4 * dst = reinterpret_cast<float4 *>(tabs) + 2 * lane;
                    dst[0] = make_float4(f[0], f[1], f[2], f[3]); dst[1] = make_float4(f[4], f[5], f[6], f[7]);
                    __syncwarp();
                }
                // ---------------- S = K Q^T ----------------
                // Integers -> f16 without arithmetic: a 16-bit lane holding a value u in 0..255 in its low byte IS the f16 subnormal u * 2^-24, and
                // the tensor cores take subnormal operands at full rate.  Products accumulate in fp32, the block scale multiplies the block's sum.
                float S[2][NT][4];
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int i = 0; i < NT; ++i) S[m][i][0] = S[m][i][1] = S[m][i][2] = S[m][i][3] = 0.0f;
                float4 sc4[2][2];   // [key half][key A, key B]: four block scales
#pragma unroll
                for (int b = 0; b < NBLK; ++b) {
                    uint4 qv[NT];
                    float4 q0[NT];
#pragma unroll
                    for (int i = 0; i < NT; ++i) {
                        qv[i] = *reinterpret_cast<const uint4 *>(Qs + (8 * i + g) * QSTR + 64 * b + 16 * t);
                        q0[i] = Qb[(b * NT + i) * 4 + t];
                    }
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        const unsigned char * rowA = Ks + (16 * m + g) * HB, * rowB = rowA + 8 * HB;
                        if ((b & 3) == 0) {
                            sc4[m][0] = reinterpret_cast<const float4 *>(tabs)[2 * (16 * m + g) + (b >> 2)];
                            sc4[m][1] = reinterpret_cast<const float4 *>(tabs)[2 * (16 * m + g + 8) + (b >> 2)];
                        }
                        const float dA = (&sc4[m][0].x)[b & 3], dB = (&sc4[m][1].x)[b & 3];
                        uint32_t a0[4], a1[4];
                        if constexpr (Q8) {
                            const uint2 wa = *reinterpret_cast<const uint2 *>(rowA + 16 + 32 * b + 8 * t);
                            const uint2 wb = *reinterpret_cast<const uint2 *>(rowB + 16 + 32 * b + 8 * t);
                            const uint32_t ax = wa.x ^ 0x80808080u, ay = wa.y ^ 0x80808080u;
                            const uint32_t bx = wb.x ^ 0x80808080u, by = wb.y ^ 0x80808080u;
                            a0[0] = ax & 0x00ff00ffu; a0[1] = bx & 0x00ff00ffu; a0[2] = __byte_perm(ax, 0u, 0x4341); a0[3] = __byte_perm(bx, 0u, 0x4341);
                            a1[0] = ay & 0x00ff00ffu; a1[1] = by & 0x00ff00ffu; a1[2] = __byte_perm(ay, 0u, 0x4341); a1[3] = __byte_perm(by, 0u, 0x4341);
                        } else {
                            // block at byte 18 b: f16 d, then 16 bytes; this lane takes bytes 4t..4t+3 (dims 4t.. low nibbles, 16+4t.. high
                            // nibbles).  The 16 bytes start on a 2-byte boundary for even b.
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
                            // nibble pairs: low nibbles of bytes (0, 2) and (1, 3) feed the first k-step, the high nibbles, times 16, the second
                            const uint32_t qa8 = qa >> 8, qb8 = qb >> 8;
                            a0[0] = qa & 0x000f000fu; a0[1] = qb & 0x000f000fu; a0[2] = qa8 & 0x000f000fu; a0[3] = qb8 & 0x000f000fu;
                            a1[0] = qa & 0x00f000f0u; a1[1] = qb & 0x00f000f0u; a1[2] = qa8 & 0x00f000f0u; a1[3] = qb8 & 0x00f000f0u;
                        }
#pragma unroll
                        for (int i = 0; i < NT; ++i) {
                            float c[4];
                            mma16816_from(c, q0[i], a0, qv[i].x, qv[i].y);
                            mma16816(c, a1, qv[i].z, qv[i].w);
                            S[m][i][0] = fmaf(dA, c[0], S[m][i][0]); S[m][i][1] = fmaf(dA, c[1], S[m][i][1]);
                            S[m][i][2] = fmaf(dB, c[2], S[m][i][2]); S[m][i][3] = fmaf(dB, c[3], S[m][i][3]);
                        }
                    }
                }
                __syncwarp();   // K's slot is read
                issue();
                // ---------------- mask, online softmax ----------------
                constexpr float UNSUB = 16777216.0f;   // 2^24
                bool grow = false;
                const bool masked = k_t + WT > mask_from;
#pragma unroll
                for (int i = 0; i < NT; ++i)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
#pragma unroll
                        for (int m = 0; m < 2; ++m) { S[m][i][e] *= UNSUB; S[m][i][2 + e] *= UNSUB; }
                        if (masked) {
#pragma unroll
                            for (int m = 0; m < 2; ++m) {
                                const int kA = k_t + 16 * m + g, kB = kA + 8;
                                if (kA > rpos[i][e] || kA >= k_hi) S[m][i][e] = B200_NEG_INF;
                                if (kB > rpos[i][e] || kB >= k_hi) S[m][i][2 + e] = B200_NEG_INF;
                            }
                        }
                        grow = grow || fmaxf(fmaxf(S[0][i][e], S[0][i][2 + e]), fmaxf(S[1][i][e], S[1][i][2 + e])) > m_run[i][e] + REF_GAP;
                    }
                // A row's reference maximum m_run trails its true maximum by at most REF_GAP (P = 2^(S - m_run + PSHIFT) <= 2^15 stays inside f16)
                // and moves, with O and l, only in a tile that outgrows it.
                if (__any_sync(0xffffffffu, grow)) {
                    float f[NT][2];
#pragma unroll
                    for (int i = 0; i < NT; ++i)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            float mx = fmaxf(fmaxf(S[0][i][e], S[0][i][2 + e]), fmaxf(S[1][i][e], S[1][i][2 + e]));
                            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                            const float mnew = mx > m_run[i][e] + REF_GAP ? mx : m_run[i][e];
                            f[i][e] = ex2f(m_run[i][e] - (mnew == B200_NEG_INF ? 0.0f : mnew));
                            m_run[i][e] = mnew;
                            l_run[i][e] *= f[i][e];
                        }
                    if (it > 0) scale_O(f);
                }
                // P carries a factor 2^PSHIFT (numerator and denominator alike): keeps small weights out of the f16 subnormal range; 2^(-inf) = 0 for a
                // masked key.  Accumulator fragment (keys g, g + 8; rows 2t, 2t + 1) -> operand fragment (keys 2t, 2t + 1; row g).
                uint32_t pw[2][NT][2];
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    const float o0 = PSHIFT - (m_run[i][0] == B200_NEG_INF ? 0.0f : m_run[i][0]), o1 = PSHIFT - (m_run[i][1] == B200_NEG_INF ? 0.0f : m_run[i][1]);
#pragma unroll
                    for (int m = 0; m < 2; ++m)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint32_t p = pack_h2(ex2f(S[m][i][2 * h] + o0), ex2f(S[m][i][2 * h + 1] + o1));
                            const float2 pf = __half22float2(*reinterpret_cast<const __half2 *>(&p));
                            l_run[i][0] += pf.x; l_run[i][1] += pf.y;
                            pw[m][i][h] = movm_trans(p);
                        }
                }
                // ---------------- V block scales, f16, [block][key], times 2^-exponent; zero for rows past the last key (their bytes may be anything) ----------------
                const unsigned char * Vs = ring + sc * SLOT;
                mbar_wait(&full[sc], ph, a.status);
                if (++sc == nslot) { sc = 0; ph ^= 1u; }
                {
                    const unsigned char * row = Vs + lane * HB;
                    uint32_t d2[4];   // blocks 2 e, 2 e + 1
                    if constexpr (Q8) {
                        const uint4 x = *reinterpret_cast<const uint4 *>(row);
                        d2[0] = x.x; d2[1] = x.y; d2[2] = x.z; d2[3] = x.w;
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e) d2[e] = __byte_perm(*reinterpret_cast<const uint16_t *>(row + 36 * e), *reinterpret_cast<const uint16_t *>(row + 36 * e + 18), 0x5410);
                    }
                    if (k_t + WT > k_hi && k_t + lane >= k_hi) d2[0] = d2[1] = d2[2] = d2[3] = 0u;
                    const uint32_t t2 = hmax2_u32(hmax2_u32(d2[0] & 0x7fff7fffu, d2[1] & 0x7fff7fffu), hmax2_u32(d2[2] & 0x7fff7fffu, d2[3] & 0x7fff7fffu));
                    if (__any_sync(0xffffffffu, v_exp || max(t2 >> 16, t2 & 0xffffu) >= 0x4000u)) {   // some |d| >= 2 (bit patterns of f16 order like their values)
#pragma unroll
                        for (int b = 0; b < NBLK; ++b) {
                            unsigned d = (b & 1 ? d2[b >> 1] >> 16 : d2[b >> 1]) & 0x7fffu;
                            if (d >= 0x7c00u) d = 0;   // infinite or no number: the block's sums are so, whatever the exponent
                            const int was = v_exp >> 4 * b & 15, e = max(was, (int) (__reduce_max_sync(0xffffffffu, d) >> 10) - 15);   // at most 15
                            if (e > was) {
                                const float f = __int_as_float((127 + was - e) << 23);
                                float (&o)[2][NT][4] = O[TM ? 0 : b];
                                if constexpr (TM) { wk_ld(t_O + 8 * NT * b, o); umma::tmem_ld_wait(); }
#pragma unroll
                                for (int x = 0; x < 8 * NT; ++x) (&o[0][0][0])[x] *= f;
                                if constexpr (TM) { wk_st(t_O + 8 * NT * b, o); umma::tmem_st_wait(); }
                                v_exp += (uint32_t) (e - was) << 4 * b;
                            }
                            const uint32_t h = e < 15 ? (uint32_t) (15 - e) << 10 : 1u << 9;   // 2^-e
                            d2[b >> 1] = hmul2_u32(d2[b >> 1], b & 1 ? 0x3c00u | h << 16 : 0x3c000000u | h);
                        }
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        *reinterpret_cast<uint16_t *>(tabs + (2 * e) * WK_SD + 2 * lane) = (uint16_t) d2[e];
                        *reinterpret_cast<uint16_t *>(tabs + (2 * e + 1) * WK_SD + 2 * lane) = (uint16_t) (d2[e] >> 16);
                    }
                    __syncwarp();
                }
                // ---------------- O^T += V^T P^T, 32 dims at a time ----------------
                // V enters as its exact integers; the block scale of each key goes into P: P d is rounded once.  P <= 2^15 and d 2^-v_exp < 2, so the product is
                // finite whatever finite scales there are: a tile with larger scales moves the block's exponent and with it O, by exact powers of two.
                float On[TM ? 2 : 1][2][NT][4];   // tensor memory: this block's accumulators and the next one's, on their way
                if constexpr (TM) wk_ld(t_O, On[0]);
#pragma unroll
                for (int b = 0; b < NBLK; ++b) {
                    if constexpr (TM) {
                        umma::tmem_ld_wait();
                        if (b + 1 < NBLK) wk_ld(t_O + 8 * NT * (b + 1), On[(b + 1) & 1]);
                    }
                    float (&o)[2][NT][4] = TM ? On[TM ? b & 1 : 0] : O[TM ? 0 : b];
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        const unsigned char * v0 = Vs + (16 * m + 2 * t) * HB, * v1 = v0 + HB, * v2 = v0 + 8 * HB, * v3 = v2 + HB;
                        uint32_t ax[4], ay[4];   // m-tiles X and Y of this block
                        if constexpr (Q8) {
                            const int col = 16 + 32 * b + 4 * g;
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
                            const int col = 18 * b + 2 + 2 * g;   // bytes 2g, 2g+1 of the block: dims 2g, 2g+1 | 16+2g, 17+2g
                            const uint32_t h0 = *reinterpret_cast<const uint16_t *>(v0 + col), h1 = *reinterpret_cast<const uint16_t *>(v1 + col);
                            const uint32_t h2 = *reinterpret_cast<const uint16_t *>(v2 + col), h3 = *reinterpret_cast<const uint16_t *>(v3 + col);
                            const uint32_t w01 = __byte_perm(h0, h1, 0x5410), w23 = __byte_perm(h2, h3, 0x5410);   // bytes (k0.B0, k0.B1, k1.B0, k1.B1)
                            const uint32_t x01 = w01 >> 8, x23 = w23 >> 8;
                            // (k0.x, k1.x) pairs: bytes 0 and 2 -> dim 2g (+16), bytes 1 and 3 -> dim 2g+1 (+16); 1024 + nibble and 1024 + 16 nibble are exact
                            // in f16, less 1032 or times 1/16 less 72 they are the stored integers
                            auto lo4 = [](uint32_t x) { return hsub2_u32((x & 0x000f000fu) | 0x64006400u, 0x64086408u); };
                            auto hi4 = [](uint32_t x) { return hfma2_u32((x & 0x00f000f0u) | 0x64006400u, 0x2c002c00u, 0xd480d480u); };
                            ax[0] = lo4(w01); ax[1] = lo4(x01); ax[2] = lo4(w23); ax[3] = lo4(x23);
                            ay[0] = hi4(w01); ay[1] = hi4(x01); ay[2] = hi4(w23); ay[3] = hi4(x23);
                        }
                        const uint32_t sd0 = *reinterpret_cast<const uint32_t *>(tabs + b * WK_SD + (16 * m + 2 * t) * 2);
                        const uint32_t sd1 = *reinterpret_cast<const uint32_t *>(tabs + b * WK_SD + (16 * m + 2 * t + 8) * 2);
#pragma unroll
                        for (int i = 0; i < NT; ++i) {
                            const uint32_t p0 = hmul2_u32(pw[m][i][0], sd0), p1 = hmul2_u32(pw[m][i][1], sd1);
                            mma16816(o[0][i], ax, p0, p1);
                            mma16816(o[1][i], ay, p0, p1);
                        }
                    }
                    if constexpr (TM) wk_st(t_O + 8 * NT * b, o);
                }
                if constexpr (TM) umma::tmem_st_wait();
                __syncwarp();   // V's slot and the scales are read
                issue();
            }

            // ---------------- the segment's partial: the two warps' (O, m, l) ----------------
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float l = l_run[i][e];
                    l += __shfl_xor_sync(0xffffffffu, l, 4);
                    l += __shfl_xor_sync(0xffffffffu, l, 8);
                    l += __shfl_xor_sync(0xffffffffu, l, 16);
                    l_run[i][e] = l;
                    if (g == 0) { ml[w * 32 + 8 * i + 2 * t + e] = m_run[i][e]; ml[w * 32 + 16 + 8 * i + 2 * t + e] = l; }
                }
            // warp w writes dims 128 w .. 128 w + 127 of the partial and hands the other half of its sums to the other warp, through its own ring (empty now)
            auto get = [&](int b, float (&o)[2][NT][4]) {
                if constexpr (TM) { wk_ld(t_O + 8 * NT * b, o); umma::tmem_ld_wait(); }
                else {
#pragma unroll
                    for (int e = 0; e < 8 * NT; ++e) (&o[0][0][0])[e] = (&O[b][0][0][0])[e];
                }
#pragma unroll
                for (int e = 0; e < 8 * NT; ++e) (&o[0][0][0])[e] *= __int_as_float((127 + (v_exp >> 4 * b & 15)) << 23);
            };
            auto give = [&](int b, int k) {
                float o[2][NT][4];
                get(b, o);
#pragma unroll
                for (int e = 0; e < 2 * NT; ++e)
                    reinterpret_cast<float4 *>(ring)[(k * 2 * NT + e) * 32 + lane] = make_float4((&o[0][0][0])[4 * e], (&o[0][0][0])[4 * e + 1], (&o[0][0][0])[4 * e + 2], (&o[0][0][0])[4 * e + 3]);
            };
            if (w == 0) {
#pragma unroll
                for (int k = 0; k < 4; ++k) give(4 + k, k);
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) give(k, k);
            }
            bar_unit(bar);
            float fo[NT][2], fx[NT][2];   // weights of this warp's and the other warp's sums
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int r = 8 * i + 2 * t + e;
                    const float m0 = ml[r], m1 = ml[32 + r], l0 = ml[16 + r], l1 = ml[48 + r], M = fmaxf(m0, m1), Ms = M == B200_NEG_INF ? 0.0f : M;
                    const float f0 = ex2f(m0 - Ms), f1 = ex2f(m1 - Ms);
                    fo[i][e] = w == 0 ? f0 : f1; fx[i][e] = w == 0 ? f1 : f0;
                    if (w == 0 && g == 0 && r < R) {
                        a.pm[(size_t) unit * R + r] = M;
                        a.pl[(size_t) unit * R + r] = fmaf(f1, l1, f0 * l0);
                    }
                }
            auto put = [&](int b, int k) {
                float o[2][NT][4];
                get(b, o);
#pragma unroll
                for (int e = 0; e < 2 * NT; ++e) {
                    const float4 x = reinterpret_cast<const float4 *>(ring_o)[(k * 2 * NT + e) * 32 + lane];
                    const int i = e % NT;
                    float * p = &(&o[0][0][0])[4 * e];
                    const float y[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                    for (int c = 0; c < 4; ++c) {   // warp 0's sums first, whichever warp adds them up
                        const float fa = w == 0 ? fo[i][c & 1] : fx[i][c & 1], fb = w == 0 ? fx[i][c & 1] : fo[i][c & 1];
                        const float oa = w == 0 ? p[c] : y[c], ob = w == 0 ? y[c] : p[c];
                        p[c] = fmaf(fb, ob, __fmul_rn(fa, oa));
                    }
                }
#pragma unroll
                for (int i = 0; i < NT; ++i)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int r = 8 * i + 2 * t + e;
                        if (r >= R) continue;
                        float * dst = a.po + ((size_t) unit * R + r) * DH + 32 * b;
                        if constexpr (Q8) *reinterpret_cast<float4 *>(dst + 4 * g) = make_float4(o[0][i][e], o[0][i][2 + e], o[1][i][e], o[1][i][2 + e]);
                        else {
                            *reinterpret_cast<float2 *>(dst + 2 * g) = make_float2(o[0][i][e], o[0][i][2 + e]);
                            *reinterpret_cast<float2 *>(dst + 16 + 2 * g) = make_float2(o[1][i][e], o[1][i][2 + e]);
                        }
                    }
            };
            if (w == 0) {
#pragma unroll
                for (int k = 0; k < 4; ++k) put(k, k);
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) put(4 + k, k);
            }
            umma::fence_async_smem();   // the next segment's copies go where the sums lay
            bar_unit(bar);
        }
    }
    if constexpr (TM) {
        umma::fence_before_sync();
        __syncthreads();
        if (warp == 0) {
            umma::fence_after_sync();
            umma::tmem_dealloc(t_O, TCOLS);
        }
    }
}
