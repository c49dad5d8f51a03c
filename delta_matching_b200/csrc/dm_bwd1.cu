// Pass 1 of the backward at head_dim 128 (head_dim 256: dm_bwd1_d256.cu): dK and dV per query head, plus the e4m3 dS' code tiles and
// their psi scales for pass 2
// (csrc/mainloop_bwd_sm90_fp8r.hpp:695-952 of the reference, restated for tcgen05).
//
// One work item = one 128-key block of one (batch, query head), walked in tiles of 128 rows (two 64-row m-blocks) from the causal
// start.  The kernel is persistent: one CTA per SM walks its share of the items, every
// role keeps its own place in the list, and the next item starts under the tail of the current one.  896 threads:
//   warps 0..15  softmax: P-hat, dS', the tile maxima, psi and both code tiles
//   warps 16..23 fold: thread = (key, 64 d columns); dK in registers, and dV's accumulator kept in the unit of the next dO block
//   warps 24..27 service, one per scheduler: the S / dP MMAs, the dK / dV MMAs and the dS' store, the TMA loads, the row constants
// Per tile:
//   S = Q K^T, dP = dO V^T   M128 N128 K32 x 4 each, tensor-memory lane = row, as soon as the softmax warps hold
//                            the previous pair
//   softmax warps            codes P-hat8 = e4m3(P-hat), dS'8 = e4m3(dS' / psi), psi by the F2 / F2b rules from the tile maxima
//   X = dS'8(m0)^T Q8        fold: dK += X * (psi 2^-8 q8sc)
//   dV += P-hat8^T dO8       into the accumulator itself (tensor memory), which is in units of this block's dO scale
//   X = dS'8(m1)^T Q8        fold: dK += X * (psi 2^-8 q8sc); then dV's accumulator times (this block's / the next one's dO scale)
// Q8 / dO8 tiles serve twice: K-major as the A operand of S / dP and MN-major as the B operand of dK / dV.
//
// Why this shape.  The kernel before this one held S^T / dP^T (lane = key) for one 64-row m-block at a time: N = 64 MMAs run the
// tensor pipe at half rate, the row constants came from shared memory in every thread (8 x 16 bytes per 16 elements), and each of
// the two m-blocks of 128 rows was a serial chain of its own (products, exponentials, maximum over a barrier, psi, codes:
// about 2600 clocks).  Here a chain of about 3800 clocks, which is what bounds the kernel, serves 128 x 128.  S / dP are read in the
// matrix-fragment layout (tcgen05.ld 16x256b): a thread has four rows and eight keys of each, so the row constants are registers, and
// a fragment of four codes is what stmatrix stores transposed, so the [key][row] code tiles (A operand of dK / dV, and the tile pass 2
// reads) still leave as whole 16-byte chunks.  With both m-blocks in one step dV's product would be a third use of the one product
// buffer X (tensor memory is full: S 128, dP 128, X 128, dV 128 columns), and X's round trip (MMA, commit, fold, release) sets the
// pace then; so dV accumulates in place and only its unit is moved, off that path.
// Measured at B4 N4096 H32 causal: 1235 us before; 1290 with dV through X; 1206 with dV in place; 1037 with the unit moved in
// 16-column pieces (fewer spills in the fold warps, which need 64 accumulators and two 16-register pieces); 960 with 72 / 96 / 24
// registers per role and a maximum barrier per row half; 900 with the hardware warps in the order service, fold, softmax; 875 with
// the unit moved in 8-column pieces (28 instead of 88 bytes spilled).
#include "dm_attn_common.cuh"
#include "dm_host.h"

namespace dm {

struct Bwd1Params {
    const float* q8s;
    const float* k8s;
    const float* v8s;
    const float* do8s;
    const float* lse;
    const float* delta;
    __nv_bfloat16* dk;
    __nv_bfloat16* dv;
    uint8_t* ds_ws;
    float* psi;
    int H, Hk, N, h0, hcount, causal;
    int* status;
    RowMap rm;                                    // which rows of the sequence the Q-side tensors hold
    int out_fp32;                                 // dK / dV leave as fp32 (partials that another rank's are added to)
    int n_heads;                                  // batch * hcount: (batch, query head) pairs of this call
    FastDiv fd_heads, fd_hcount, fd_rep;          // divisions by n_heads, hcount and H / Hk
};

// The work list: one item = one 128-key block J of one (batch, query head), ordered by
// key block, i.e. heaviest first when causal, and walked as walk_index says.
struct Bwd1Item {
    HeadCoord hc;
    int J, m_lo, n_it, bhl;                   // m_lo, n_it: first 64-row m-block and their count, both even
    bool valid;
};
template <class Walk>
__device__ __forceinline__ Bwd1Item bwd1_item(const Bwd1Params& p, const Walk& walk, int round) {
    Bwd1Item w;
    const int nbn = p.N / 128;
    const int idx = walk_index(walk, round);
    w.valid = idx < p.n_heads * nbn;
    w.J = (int)fdiv((uint32_t)idx, p.fd_heads);
    w.hc = head_coord(idx - w.J * p.n_heads, p.h0, p.fd_hcount, p.H, p.Hk, p.fd_rep);
    w.bhl = w.hc.b * p.hcount + (w.hc.h - p.h0);
    // m-blocks are counted in the local rows; global position grows with the local index, and both chunks of a row map
    // start on a 128-row pair, so local and global m-block parity agree.  Causal: start at the first local m-block that is
    // not wholly above the diagonal of key block J; a rank may hold none (n_it == 0: dK = dV = 0 for this block).
    const int nq_blk = p.rm.nq / 128, nbm = p.rm.nq / 64;
    w.m_lo = 0;
    if (p.causal) {
        const int rest = nq_blk - p.rm.half;
        if (w.J < p.rm.off0 + p.rm.half) w.m_lo = 2 * max(w.J - p.rm.off0, 0);
        else if (w.J < p.rm.off1 + rest) w.m_lo = 2 * (p.rm.half + max(w.J - p.rm.off1, 0));
        else w.m_lo = nbm;
    }
    w.n_it = nbm - w.m_lo;
    return w;
}

}  // namespace dm


namespace {

constexpr int kTile = 128 * 128;
constexpr int kSoftmaxThreads = 512;
constexpr int kFoldWarp = 16, kServiceWarp = 24;
constexpr int kThreads = 896;
constexpr int kRegSoftmax = 72, kRegFold = 96, kRegService = 24;     // per thread after setmaxnreg: the sum is the launch pool
constexpr int kRows = 3;               // ring of row constants
constexpr int kGf = 4;                 // ring of product scales between softmax and fold warps
// Tiles that dV's accumulator sums by itself.  The tensor pipe's fp32 additions drop what does not fit (they round towards zero), so the
// sum of a long walk drifts: by 8.7e-7 of its size over 32 tiles, 3.5e-6 over 128, 1.9e-5 over 512, where rounded additions stay below
// 2e-7; a drift of 1.9e-5 moves one bf16 value in two hundred.  So a walk of more than kWindow tiles moves the accumulator into an fp32
// sum in memory every kWindow tiles, and starts it again: 1.6e-6 over 512 tiles.  Shorter windows drift less and cost more (pass 1 at
// B1 N16384 H8, us: none 763, 64 tiles 769, 32 tiles 795); a shape of up to 64 row blocks never gets there.
constexpr int kWindow = 64;

// Named barriers.  Warp-to-warp hand-offs cost a quarter of an mbarrier's; an arriving side is never a whole round ahead, because
// its next arrival on the same barrier needs a product that is issued behind the synchronising side's.
constexpr int kBarSpFree = 1;          // (S | dP) is in registers                          512 + 32
constexpr int kBarAmax = 2;            // + m-block: its warps' maxima are in shared memory  256
constexpr int kBarCodes = 6;           // + tile parity: the tile's codes are               512 + 32
constexpr int kBarXFree = 8;           // the fold warps hold the dK product                256 + 32
constexpr int kBarDvFree = 9;          // dV's accumulator is in the next block's unit      256 + 32

constexpr int kStages = 3;             // ring of Q / dO tiles
constexpr int kStgCols = 32;           // columns of the output staging

struct Smem {
    alignas(1024) uint8_t k[kTile];
    alignas(1024) uint8_t v[kTile];
    alignas(1024) uint8_t q[kStages][kTile];
    alignas(1024) uint8_t dO[kStages][kTile];
    alignas(1024) uint8_t pt[2][kTile];       // P-hat codes, [key][row], by tile parity
    alignas(1024) uint8_t ds[2][kTile];       // dS' codes, same layout
    alignas(16) uint8_t stg[8][32 * 2 * kStgCols];  // per fold warp: 32 keys of bf16 columns on their way out (chunks XOR-swizzled)
    alignas(16) float2 rd[kRows][128];        // per row: 8 - lse * log2e, -delta
    alignas(16) float sc[kRows][4];           // q8sc, do8sc, what dV's accumulator is multiplied by before the tile, dV's unit
    float gf[kGf][2];                         // dK scale of m-block m
    float fv[kGf];                            // dV's unit after the tile
    float psi[kGf][2];                        // psi of m-block m, on its way to pass 2
    float amax[2][16];                        // [tile parity][m-block, warp of it]
    uint64_t bar_kv, bar_kv_free, bar_qdo[kStages], bar_qdo_free[kStages], bar_sp_full, bar_x_full, bar_done[2], bar_ds_free[2], bar_rows_full[kRows], bar_rows_free[kRows];
    uint32_t tmem_base;
    int abort_flag;
};

template <class Walk>
__global__ void __launch_bounds__(kThreads, 1)
bwd1_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
            const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
            const __grid_constant__ CUtensorMap tm_ds, const dm::Bwd1Params p, const __grid_constant__ Walk walk) {
    extern __shared__ uint8_t smem_raw[];
    Smem& s = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    // The hardware warps are taken in the order service, fold, softmax (the role numbers below keep their tensor-memory quarter,
    // warp mod 4): 949 -> 900 us against softmax first (B4 N4096 H32 causal).
    const int tid = threadIdx.x, lane = tid & 31, hw_warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int warp = hw_warp < 4 ? hw_warp + kServiceWarp : (hw_warp < 12 ? hw_warp + kFoldWarp - 4 : hw_warp - 12);
    const int nbn = p.N / 128, nq_blk = p.rm.nq / 128;
    // `t` counts the CTA's tiles (128 rows each) over its items, so ring stages, buffer parities and mbarrier phases run on across
    // items.  `kvn` counts the items that loaded K / V (those with tiles).
    dm::WaitCtx wc{&s.abort_flag, p.status};

    if (tid == 0) {
        s.abort_flag = 0;
        dm::mbar_init(&s.bar_kv, 1);
        dm::mbar_init(&s.bar_kv_free, 1);
        dm::mbar_init(&s.bar_sp_full, 1);
        dm::mbar_init(&s.bar_x_full, 1);
        for (int i = 0; i < kStages; ++i) {
            dm::mbar_init(&s.bar_qdo[i], 1);
            dm::mbar_init(&s.bar_qdo_free[i], 1);
        }
        for (int i = 0; i < kRows; ++i) {
            dm::mbar_init(&s.bar_rows_full[i], 1);
            dm::mbar_init(&s.bar_rows_free[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            dm::mbar_init(&s.bar_done[i], 1);
            dm::mbar_init(&s.bar_ds_free[i], 1);
        }
        dm::fence_mbar_init();
    }
    if (warp == 0) dm::tmem_alloc(&s.tmem_base, 512);
    dm::tc_fence_before();
    __syncthreads();
    dm::tc_fence_after();
    dm::pdl_wait();
    // tensor memory: S [0, 128) | dP [128, 256) (lane = row), product X [256, 384), dV accumulator [384, 512) (lane = key)
    const uint32_t tmem = s.tmem_base;
    const uint32_t t_x = tmem + 256, t_dva = tmem + 384;
    const uint32_t lane_base = (uint32_t)(warp & 3) * 32;

    if (warp >= kServiceWarp) {
        // =============================================================== service warps: loops converged, one elected lane issues
        dm::reg_dec<kRegService>();
        constexpr uint32_t kSub = kTile >> 4;
        if (warp == kServiceWarp) {
            // ---- S = Q K^T and dP = dO V^T of every tile
            constexpr uint32_t idesc_sp = dm::idesc_e4m3(128, 128, false, false);
            const uint32_t k_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.k)), v_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.v));
            const uint32_t q_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.q[0])), do_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.dO[0]));
            int t = 0, kvn = 0;
            for (int r = 0;; ++r) {
                const dm::Bwd1Item w = dm::bwd1_item(p, walk, r);
                if (!w.valid) break;
                const int n = w.n_it >> 1;
                if (n > 0) dm::mbar_wait(&s.bar_kv, kvn++ & 1, wc);
                for (int it = 0; it < n; ++it, ++t) {
                    const int st = t % kStages;
                    dm::mbar_wait(&s.bar_qdo[st], (t / kStages) & 1, wc);
                    // The softmax warps rewrite the code tiles of tile t - 2: its products and its dS' store must be done.  Gating the
                    // products gates the softmax warps.
                    if (t >= 2) {
                        dm::mbar_wait(&s.bar_done[t & 1], ((t - 2) >> 1) & 1, wc);
                        dm::mbar_wait(&s.bar_ds_free[t & 1], ((t - 2) >> 1) & 1, wc);
                    }
                    dm::mbar_wait(&s.bar_rows_full[t % kRows], (t / kRows) & 1, wc);      // saves the softmax warps a wait of their own
                    if (t >= 1) dm::named_bar_sync(kBarSpFree, kSoftmaxThreads + 32);
                    dm::tc_fence_after();
                    if (dm::elect_one()) {
#pragma unroll
                        for (int m = 0; m < 2; ++m) {              // S, then dP
                            const uint32_t a = (m ? do_lo : q_lo) + st * kSub, b = m ? v_lo : k_lo, d = tmem + 128 * m;
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                if (k == 0) dm::umma_e4m3_lo<false>(d, a, b, idesc_sp);
                                else dm::umma_e4m3_lo<true>(d, a + 2 * k, b + 2 * k, idesc_sp);
                            }
                        }
                        dm::umma_commit(&s.bar_sp_full);
                        if (it == n - 1) dm::umma_commit(&s.bar_kv_free);     // the loader may bring the next item's K / V
                    }
                    __syncwarp();
                }
            }
            if (t > 0) dm::named_bar_sync(kBarSpFree, kSoftmaxThreads + 32);      // the last release: no arrival is left over
        } else if (warp == kServiceWarp + 1) {
            // ---- dK's two products of a tile through X, dV's into its accumulator; the dS' store
            constexpr uint32_t idesc_x = dm::idesc_e4m3(128, 128, false, true);
            const uint32_t q_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.q[0])), do_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.dO[0]));
            const uint32_t pt_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.pt[0])), ds_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.ds[0]));
            int t = 0;
            for (int r = 0;; ++r) {
                const dm::Bwd1Item w = dm::bwd1_item(p, walk, r);
                if (!w.valid) break;
                int ds_row = (int)((((int64_t)w.bhl * nq_blk + (w.m_lo >> 1)) * nbn + w.J) * 128);   // dS' tile of the first row block
                float* psi_out = p.psi + ((int64_t)w.bhl * (2 * nq_blk) + w.m_lo + lane) * nbn + w.J;
                for (int it = 0; it < w.n_it; it += 2, ++t, ds_row += nbn * 128) {
                    const int par = t & 1, st = t % kStages;
                    const uint32_t qs = q_lo + st * kSub, dos = do_lo + st * kSub, da = ds_lo + par * kSub, pa = pt_lo + par * kSub;
                    if (t >= 1 && dm::elect_one()) {       // the previous tile has left shared memory
                        dm::tma_store_wait_read0();
                        dm::mbar_arrive(&s.bar_ds_free[par ^ 1]);
                    }
                    __syncwarp();
                    dm::named_bar_sync(kBarCodes + par, kSoftmaxThreads + 32);
#pragma unroll
                    for (int m = 0; m < 2; ++m) {          // the two m-blocks
                        // dK_tmp
                        if (t > 0 || m > 0) dm::named_bar_sync(kBarXFree, 256 + 32);
                        dm::tc_fence_after();
                        if (dm::elect_one()) {
                            dm::umma_e4m3_lo<false>(t_x, da + 4 * m, qs + 512 * m, idesc_x);
                            dm::umma_e4m3_lo<true>(t_x, da + 4 * m + 2, qs + 512 * m + 256, idesc_x);
                            dm::umma_commit(&s.bar_x_full);
                            if (m == 0) {
                                dm::tma_store_2d(&tm_ds, 0, ds_row, s.ds[par]);
                                dm::tma_store_commit();
                            } else {
                                dm::umma_commit(&s.bar_qdo_free[st]);       // the stage's Q / dO have been read for the last time
                                dm::umma_commit(&s.bar_done[par]);
                            }
                        }
                        __syncwarp();
                        if (m == 0 && lane < 2) psi_out[(int64_t)it * nbn] = s.psi[t % kGf][lane];
                        // dV += P-hat8^T dO8 of a whole dO scale block, in the accumulator itself
                        if (m == 0) {
                            if (t > 0) dm::named_bar_sync(kBarDvFree, 256 + 32);
                            dm::tc_fence_after();
                            if (dm::elect_one()) {
                                dm::umma_e4m3_lo_rt(t_dva, pa, dos, idesc_x, (it >> 1) % kWindow != 0);
#pragma unroll
                                for (int k = 1; k < 4; ++k) dm::umma_e4m3_lo<true>(t_dva, pa + 2 * k, dos + 256 * k, idesc_x);
                                dm::mbar_arrive(&s.bar_rows_free[t % kRows]);
                            }
                            __syncwarp();
                        }
                    }
                }
            }
            if (t > 0) {
                dm::named_bar_sync(kBarXFree, 256 + 32);           // the last products: shared memory has been read
                dm::named_bar_sync(kBarDvFree, 256 + 32);
                if (dm::elect_one()) dm::tma_store_wait_all0();
                __syncwarp();
            }
        } else if (warp == kServiceWarp + 2) {
            // ---- TMA loads: an item's K / V once the previous item's last S / dP have read theirs, then the Q8 / dO8 tiles as far
            // ahead as the ring allows
            int t = 0, kvn = 0;
            for (int r = 0;; ++r) {
                const dm::Bwd1Item w = dm::bwd1_item(p, walk, r);
                if (!w.valid) break;
                const int n = w.n_it >> 1;
                const int kv_row0 = w.hc.bhk * p.N + w.J * 128;
                const int q_row0 = w.hc.bh * p.rm.nq + w.m_lo * 64;
                if (n > 0) {
                    if (kvn >= 1) dm::mbar_wait(&s.bar_kv_free, (kvn - 1) & 1, wc);
                    if (dm::elect_one()) {
                        dm::mbar_expect_tx(&s.bar_kv, 2 * kTile);
                        dm::tma_load_2d(s.k, &tm_k, 0, kv_row0, &s.bar_kv);
                        dm::tma_load_2d(s.v, &tm_v, 0, kv_row0, &s.bar_kv);
                    }
                    __syncwarp();
                    ++kvn;
                }
                for (int it = 0; it < n; ++it, ++t) {
                    const int st = t % kStages;
                    if (t >= kStages) dm::mbar_wait(&s.bar_qdo_free[st], (t / kStages - 1) & 1, wc);
                    if (dm::elect_one()) {
                        dm::mbar_expect_tx(&s.bar_qdo[st], 2 * kTile);
                        dm::tma_load_2d(s.q[st], &tm_q, 0, q_row0 + it * 128, &s.bar_qdo[st]);
                        dm::tma_load_2d(s.dO[st], &tm_do, 0, q_row0 + it * 128, &s.bar_qdo[st]);
                    }
                    __syncwarp();
                }
            }
        } else {
            // ---- the rows' constants (four per lane) and the Q / dO scales of the tile, kRows ahead
            int t = 0;
            for (int r = 0;; ++r) {
                const dm::Bwd1Item w = dm::bwd1_item(p, walk, r);
                if (!w.valid) break;
                float unit = 0.f, top = 0.f;
                for (int it = 0; it < w.n_it; it += 2, ++t) {
                    const int slot = t % kRows, li = (w.m_lo + it) >> 1;
                    const int64_t gi = (int64_t)w.hc.bh * p.rm.nq + (int64_t)li * 128 + 4 * lane;
                    float l4[4], d4[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        l4[i] = p.lse[gi + i];
                        d4[i] = p.delta[gi + i];
                    }
                    const int64_t sq = (int64_t)w.hc.bh * nq_blk + li;
                    const float q8sc = p.q8s[sq], do8sc = p.do8s[sq];
                    // dV's accumulator is kept in units of the current dO scale block's scale, so that the MMAs add to it directly.
                    // A block more than 2^-80 below the item's largest so far (an all-zero one) takes the unit at that bound: the
                    // accumulator stays finite, and zero codes add nothing whatever the unit is.
                    top = fmaxf(top, do8sc);
                    const float unit_new = fmaxf(do8sc, top * 0x1p-80f);
                    const float mult = unit / unit_new;
                    unit = unit_new;
                    if (t >= kRows) dm::mbar_wait(&s.bar_rows_free[slot], (t / kRows - 1) & 1, wc);
#pragma unroll
                    for (int i = 0; i < 4; i += 2)
                        *reinterpret_cast<float4*>(&s.rd[slot][4 * lane + i]) =
                            make_float4(dm::phat_row_const(l4[i]), -d4[i], dm::phat_row_const(l4[i + 1]), -d4[i + 1]);
                    if (lane == 0) *reinterpret_cast<float4*>(s.sc[slot]) = make_float4(q8sc, do8sc, mult, dm::kMoInv * unit);
                    __syncwarp();
                    if (dm::elect_one()) dm::mbar_arrive(&s.bar_rows_full[slot]);
                }
            }
        }
    } else if (warp >= kFoldWarp) {
        // =============================================================== fold warps: thread = (key, 64 d columns)
        dm::reg_inc<kRegFold>();
        const int key = (warp & 3) * 32 + lane, half = (warp >> 2) & 1;
        const uint32_t x_src = dm::tmem_addr(t_x, lane_base, 64 * half), dva = dm::tmem_addr(t_dva, lane_base, 64 * half);
        int t = 0;
        for (int r = 0;; ++r) {
            int n_it;                                  // all that the tile loop keeps of the item: it has no registers to spare
            float ik;                                  // for the epilogue; read early
            {
                const dm::Bwd1Item w = dm::bwd1_item(p, walk, r);
                if (!w.valid) break;
                n_it = w.n_it;
                ik = 1.0f / p.k8s[(int64_t)w.hc.bhk * (p.N / 64) + 2 * w.J + key / 64];
            }
            float dk_acc[64];
#pragma unroll
            for (int i = 0; i < 64; ++i) dk_acc[i] = 0.f;
            auto fold_dk = [&](const float* g, int m) {             // two products a tile
                dm::mbar_wait(&s.bar_x_full, m, wc);                // also orders the ring slot written before the codes
                dm::tc_fence_after();
                // four 16-column pieces, two in flight
                uint32_t sa[16], sb[16];
                dm::tmem_ld16(x_src, sa);
                dm::tmem_ld16(x_src + 16, sb);
                const float gk = g[m];
                auto add16 = [&](int pc, const uint32_t* x) {
#pragma unroll
                    for (int i = 0; i < 16; i += 2)
                        dm::fma2(dk_acc[16 * pc + i], dk_acc[16 * pc + i + 1], __uint_as_float(x[i]), __uint_as_float(x[i + 1]), gk,
                                 dk_acc[16 * pc + i], dk_acc[16 * pc + i + 1]);
                };
                dm::tmem_ld_wait();
                add16(0, sa);
                dm::tmem_ld16(x_src + 32, sa);
                add16(1, sb);
                dm::tmem_ld16(x_src + 48, sb);
                dm::tmem_ld_wait();
                dm::tc_fence_before();
                dm::named_bar_arrive(kBarXFree, 256 + 32);
                add16(2, sa);
                add16(3, sb);
            };
            auto rescale_dv = [&](float mult) {                     // dV's accumulator into the unit of the next dO scale block
#pragma unroll
                for (int pc = 0; pc < 8; ++pc) {
                    uint32_t sa[8];
                    dm::tmem_ld8(dva + 8 * pc, sa);
                    dm::tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 8; i += 2) {
                        float y0, y1;
                        dm::mul2(y0, y1, __uint_as_float(sa[i]), __uint_as_float(sa[i + 1]), mult, mult);
                        sa[i] = __float_as_uint(y0);
                        sa[i + 1] = __float_as_uint(y1);
                    }
                    dm::tmem_st8(dva + 8 * pc, sa);
                }
                dm::tmem_st_wait();
                dm::tc_fence_before();
                dm::named_bar_arrive(kBarDvFree, 256 + 32);
            };
            // The fp32 sum of dV's earlier windows lives in the item's own outputs, which are written at its end: a warp's 32 keys x 64
            // columns of dK and dV are 8 KB, its share of the sum.  Unit u (16 columns) is in dV's (u even) or dK's half rows, at 64 bytes
            // times u / 2: the epilogue's stores of a unit's columns then cover only what has been read.  (fp32 outputs: in dV itself.)  A
            // slot is one thread's own; the lanes of a warp take whole 64-byte pieces.
            struct DvSum {
                uint8_t* at;                           // unit 0's slot of this lane
                int64_t odd, even;                     // from there to units 1 and 2
                int64_t step;                          // eight keys
            };
            auto dv_sum = [&]() {
                int r_again = r;                       // (looked up again: the tile loop has no registers for it)
                asm volatile("" : "+r"(r_again));
                const dm::Bwd1Item v = dm::bwd1_item(p, walk, r_again);
                const int64_t at = (((int64_t)v.hc.b * p.N + v.J * 128 + lane_base + (lane >> 2)) * p.H + v.hc.h) * 128 + 64 * half;
                const int64_t keys8 = (int64_t)p.H * (8 * 128);
                uint8_t* dv = reinterpret_cast<uint8_t*>(p.dv) + 16 * (lane & 3);
                if (p.out_fp32) return DvSum{dv + 4 * at, 64, 128, 4 * keys8};
                return DvSum{dv + 2 * at, reinterpret_cast<uint8_t*>(p.dk) - reinterpret_cast<uint8_t*>(p.dv), 64, 2 * keys8};
            };
            auto flush_dv = [&](float unit, bool first) {
                DvSum m = dv_sum();
#pragma unroll 1
                for (int u = 0; u < 4; ++u) {
                    uint8_t* to = m.at + ((u & 1) ? m.odd : 0) + ((u & 2) ? m.even : 0);
#pragma unroll
                    for (int c = 0; c < 16; c += 8) {
                        uint32_t sa[8];
                        dm::tmem_ld8(dva + 16 * u + c, sa);
                        dm::tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 8; e += 4, to += m.step) {
                            const float4 y = make_float4(__uint_as_float(sa[e]) * unit, __uint_as_float(sa[e + 1]) * unit,
                                                         __uint_as_float(sa[e + 2]) * unit, __uint_as_float(sa[e + 3]) * unit);
                            if (first) *reinterpret_cast<float4*>(to) = y;
                            else dm::red_add_f32x4(to, y);
                        }
                    }
                }
                dm::tc_fence_before();
                dm::named_bar_arrive(kBarDvFree, 256 + 32);
            };
            for (int it = 0; it < n_it;) {
                const int end = min(n_it, it + 2 * kWindow);
                for (; it < end; it += 2, ++t) {
                    const float* g = s.gf[t % kGf];
                    fold_dk(g, 0);
                    fold_dk(g, 1);                                       // (its product was committed behind the tile's dV)
                    if (it + 2 < end) {
                        const int slot = (t + 1) % kRows;
                        dm::mbar_wait(&s.bar_rows_full[slot], ((t + 1) / kRows) & 1, wc);
                        rescale_dv(s.sc[slot][2]);
                    }
                }
                if (n_it > 2 * kWindow) flush_dv(s.fv[(t + kGf - 1) % kGf], it == 2 * kWindow);
            }

            // ---- epilogue: dK *= 1 / k8s, dV from its accumulator, per query head.  After a long walk dV's accumulator has joined the sum of
            // the windows, and dV leaves first: dK's rows hold a part of that sum.
            const bool have_dv = n_it > 0, have_sum = (n_it >> 1) > kWindow;
            int r_again = r;
            asm volatile("" : "+r"(r_again));
            const dm::Bwd1Item w = dm::bwd1_item(p, walk, r_again);
            const float fv = have_dv ? s.fv[(t + kGf - 1) % kGf] : 0.f;      // dV's last unit
            const int64_t row_stride = (int64_t)p.H * 128;           // elements between consecutive keys
            const int64_t off = (((int64_t)w.hc.b * p.N + w.J * 128) * p.H + w.hc.h) * 128 + 64 * half;   // key 0 of the block
            auto dv16 = [&](int pc, float* y) {
                if (have_dv) {
                    dm::tmem_ld16(dva + 16 * pc, reinterpret_cast<uint32_t*>(y));
                    dm::tmem_ld_wait();
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) y[i] = 0.f;
                }
            };
            auto sum16 = [&](const DvSum& m, int u, float* y) {
                const uint8_t* from = m.at + ((u & 1) ? m.odd : 0) + ((u & 2) ? m.even : 0);
#pragma unroll
                for (int j = 0; j < 4; ++j, from += m.step) *reinterpret_cast<float4*>(y + 4 * j) = __ldcg(reinterpret_cast<const float4*>(from));
                __syncwarp();                                        // the warp has read the unit: its place may be written
            };
            if (p.out_fp32) {
                float4* ok = reinterpret_cast<float4*>(reinterpret_cast<float*>(p.dk) + off + key * row_stride);
                float4* ov = reinterpret_cast<float4*>(reinterpret_cast<float*>(p.dv) + off + key * row_stride);
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    ok[c] = make_float4(dk_acc[4 * c] * ik, dk_acc[4 * c + 1] * ik, dk_acc[4 * c + 2] * ik, dk_acc[4 * c + 3] * ik);
                const DvSum m = dv_sum();
#pragma unroll 1
                for (int pc = 0; pc < 4; ++pc) {
                    float y[16];
                    if (have_sum) sum16(m, pc, y);
                    else dv16(pc, y);
                    const float f = have_sum ? 1.0f : fv;
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        ov[4 * pc + c] = make_float4(y[4 * c] * f, y[4 * c + 1] * f, y[4 * c + 2] * f, y[4 * c + 3] * f);
                }
            } else {
                // The bf16 rows leave through the warp's own staging slice, kStgCols columns at a time: a thread holds one key, so
                // stored directly every 16-byte store instruction would touch 32 rows; from the slice it writes 8 pieces of 64 bytes.
                constexpr int kCh = kStgCols / 8;                   // 16-byte chunks per key
                uint8_t* stg = s.stg[warp & 7];
                auto chunk = [&](int row, int c) { return stg + row * (16 * kCh) + ((c ^ ((row >> 1) & (kCh - 1))) << 4); };
                auto put8 = [&](int c, const float* y, float f) {      // 8 columns = one 16-byte chunk
                    uint32_t w4[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        __nv_bfloat162 a = __floats2bfloat162_rn(y[2 * e] * f, y[2 * e + 1] * f);
                        w4[e] = *reinterpret_cast<uint32_t*>(&a);
                    }
                    *reinterpret_cast<uint4*>(chunk(lane, c)) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                };
                auto out = [&](__nv_bfloat16* dst, int h) {            // 32 keys from the slice
                    __syncwarp();
                    const int c = lane & (kCh - 1);
#pragma unroll
                    for (int i = 0; i < kCh; ++i) {
                        const int row = (32 / kCh) * i + lane / kCh;
                        const uint4 val = *reinterpret_cast<const uint4*>(chunk(row, c));
                        *reinterpret_cast<uint4*>(dst + off + (lane_base + row) * row_stride + kStgCols * h + 8 * c) = val;
                    }
                    __syncwarp();
                };
                if (have_sum) {
                    const DvSum m = dv_sum();
#pragma unroll 1
                    for (int h = 0; h < 64 / kStgCols; ++h) {
#pragma unroll
                        for (int pc = 0; pc < kCh / 2; ++pc) {
                            float y[16];
                            sum16(m, (kCh / 2) * h + pc, y);
                            put8(2 * pc, y, 1.0f);
                            put8(2 * pc + 1, y + 8, 1.0f);
                        }
                        out(p.dv, h);
                    }
                }
#pragma unroll
                for (int h = 0; h < 64 / kStgCols; ++h) {
#pragma unroll
                    for (int c = 0; c < kCh; ++c) put8(c, dk_acc + kStgCols * h + 8 * c, ik);
                    out(p.dk, h);
                }
                if (!have_sum) {
#pragma unroll
                    for (int h = 0; h < 64 / kStgCols; ++h) {
#pragma unroll
                        for (int pc = 0; pc < kCh / 2; ++pc) {
                            float y[16];
                            dv16((kCh / 2) * h + pc, y);
                            put8(2 * pc, y, fv);
                            put8(2 * pc + 1, y + 8, fv);
                        }
                        out(p.dv, h);
                    }
                }
            }
            if (have_dv && !have_sum) {
                dm::tc_fence_before();
                dm::named_bar_arrive(kBarDvFree, 256 + 32);
            }
        }
    } else {
        // =============================================================== softmax warps
        dm::reg_dec<kRegSoftmax>();
        const int rq = warp & 3, kq = warp >> 2;      // rows [32 rq, +32) and keys [32 kq, +32) of the tile
        const int rhalf = rq >> 1;                    // the 64-row m-block
        const bool leader = (warp & 13) == 0;         // one warp of each m-block
        const int row_t = 32 * rq + (lane >> 2);      // the thread's rows: row_t + {0, 8, 16, 24}
        const int key_t = 32 * kq + 2 * (lane & 3);   // its keys: key_t + 8 j + {0, 1}
        const uint32_t t_s = dm::tmem_addr(tmem, lane_base, 32 * kq);
        // this lane's line of the transposed stores: key 32 kq + lane, the 16-byte chunk of rows [32 rq, +16) (the next chunk: ^ 16)
        const uint32_t st_addr = dm::smem_u32(s.pt[0]) + (32 * kq + lane) * 128 + (((2 * rq) ^ (lane & 7)) << 4);
        const uint32_t ds_off = dm::smem_u32(s.ds[0]) - dm::smem_u32(s.pt[0]);
        int t = 0, rb = 0;                            // tiles so far; ring slot of the row constants
        for (int r = 0;; ++r) {
            const dm::Bwd1Item w = dm::bwd1_item(p, walk, r);
            if (!w.valid) break;
            const int n_it = w.n_it >> 1;
            const float k8s_t = p.k8s[(int64_t)w.hc.bhk * (p.N / 64) + 2 * w.J + (kq >> 1)];
            const float v8s_t = p.v8s[(int64_t)w.hc.bhk * (p.N / 64) + 2 * w.J + (kq >> 1)];
            const bool diag_item = p.causal && n_it > 0 && dm::global_block(p.rm, w.m_lo >> 1) == w.J;
            float g_max = 0.f;

            for (int it = 0; it < n_it; ++it, ++t, rb = rb == kRows - 1 ? 0 : rb + 1) {
                const int par = t & 1;
                dm::mbar_wait(&s.bar_sp_full, par, wc);
                const float q8sc = s.sc[rb][0], do8sc = s.sc[rb][1];
                const float dsc = dm::descale_log2(q8sc, k8s_t);
                const float dpk = do8sc * v8s_t * k8s_t;
                const float2* rd = &s.rd[rb][row_t];
                const uint32_t addr = st_addr + par * kTile, ds_addr = st_addr + ds_off + par * kTile;
                dm::tc_fence_after();

                // ---- phase 1: P-hat, dS', tile amax; P-hat codes to shared memory.  Two halves of 16 rows; S first: the
                // exponentials run while dP is still on its way from tensor memory.
                float ds[32], am0 = 0.f, am1 = 0.f;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float sv[16], *dp = ds + 16 * h;
                    dm::tmem_ld16x256_x4(t_s + (16u << 16) * h, reinterpret_cast<uint32_t*>(sv));
                    const float2 ra = rd[16 * h], rb2 = rd[16 * h + 8];
                    dm::tmem_ld_wait();
                    dm::tmem_ld16x256_x4(t_s + 128 + (16u << 16) * h, reinterpret_cast<uint32_t*>(dp));
#pragma unroll
                    for (int j = 0; j < 16; j += 4) {           // P-hat = 2^min(S dsc + rc, 12), the exponent two at a time
                        dm::fma2(sv[j], sv[j + 1], sv[j], sv[j + 1], dsc, ra.x, ra.x);
                        dm::fma2(sv[j + 2], sv[j + 3], sv[j + 2], sv[j + 3], dsc, rb2.x, rb2.x);
#pragma unroll
                        for (int e = 0; e < 4; ++e) sv[j + e] = dm::ex2(fminf(sv[j + e], dm::kMoE + 4.0f));
                    }
                    if (diag_item && it == 0) {                 // the diagonal 128 x 128 block only: keys above the row
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (key_t + 2 * (j & ~3) + (j & 1) > row_t + 16 * h + 4 * (j & 2)) sv[j] = 0.f;
                    }
                    dm::tmem_ld_wait();
                    if (h == 1) {
                        dm::tc_fence_before();
                        dm::named_bar_arrive(kBarSpFree, kSoftmaxThreads + 32);     // (S | dP) may be overwritten
                    }
                    const float da = ra.y * k8s_t, db = rb2.y * k8s_t;              // -delta * k8s
#pragma unroll
                    for (int j = 0; j < 16; j += 4) {
                        dm::fma2(dp[j], dp[j + 1], dp[j], dp[j + 1], dpk, da, da);
                        dm::fma2(dp[j + 2], dp[j + 3], dp[j + 2], dp[j + 3], dpk, db, db);
                        dm::mul2(dp[j], dp[j + 1], dp[j], dp[j + 1], sv[j], sv[j + 1]);
                        dm::mul2(dp[j + 2], dp[j + 3], dp[j + 2], dp[j + 3], sv[j + 2], sv[j + 3]);
                        am0 = dm::fmax3_abs(am0, dp[j], dp[j + 1]);
                        am1 = dm::fmax3_abs(am1, dp[j + 2], dp[j + 3]);
                    }
                    uint32_t c4[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) c4[j] = dm::cvt_e4m3x4(sv[4 * j], sv[4 * j + 1], sv[4 * j + 2], sv[4 * j + 3]);
                    dm::stmatrix_t_b8_x4(addr ^ (16 * h), c4);
                }
                // the warp's maximum in one instruction: non-negative floats order like their bit patterns
                const float am = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(am0, am1))));
                if (lane == 0) s.amax[par][8 * rhalf + 2 * kq + (rq & 1)] = am;
                dm::named_bar_sync(kBarAmax + rhalf, 256);
                // psi of the tile: psi = max(psi_raw, g_max * 256e-8 / q8sc); the quotient can only win when its numerator
                // exceeds psi_raw * q8sc, so the division is formed only then (the 1 % margin covers the rounding of both sides).
                // g_max runs over the psi tiles of this row half: the floor acts only on a tile whose maximum lies eight decades
                // below an earlier one's, and one barrier for both halves and both psi in every thread cost 3 %.
                float psi_my;
                {
                    const float mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(s.amax[par][8 * rhalf + (lane & 7)])));
                    const float amx = mx * (1.0f / 448.0f);
                    psi_my = fmaxf(amx, 1e-30f);
                    const float fl_num = g_max * (256.0f * 1e-8f);
                    if (fl_num > psi_my * q8sc * 0.99f) psi_my = fmaxf(psi_my, fl_num / q8sc);
                    if (amx < 1e-30f) psi_my = 0.f;                          // a zero tile
                }
                const float g_my = psi_my * dm::kMoInv * q8sc;
                g_max = fmaxf(g_max, g_my);
                const float psi_inv = psi_my == 0.f ? 0.f : __frcp_rn(psi_my);   // the correctly rounded reciprocal, as 1 / psi

                // ---- phase 2: dS' codes, to shared memory for dK and for the tile that leaves to pass 2
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t c4[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float a0, a1, a2, a3;
                        dm::mul2(a0, a1, ds[16 * h + 4 * j], ds[16 * h + 4 * j + 1], psi_inv, psi_inv);
                        dm::mul2(a2, a3, ds[16 * h + 4 * j + 2], ds[16 * h + 4 * j + 3], psi_inv, psi_inv);
                        c4[j] = dm::cvt_e4m3x4(a0, a1, a2, a3);
                    }
                    dm::stmatrix_t_b8_x4((ds_addr ^ (16 * h)), c4);
                }
                // the scales of this tile's products for the fold warps (the ring slot was last read four tiles ago; S of this tile
                // waited for the products of two tiles ago) and psi, which the product warp takes to global memory
                if (leader && lane == 0) {
                    s.gf[t % kGf][rhalf] = g_my;
                    s.psi[t % kGf][rhalf] = psi_my;
                    if (warp == 0) s.fv[t % kGf] = s.sc[rb][3];
                }
                dm::fence_proxy_async_smem();
                dm::named_bar_arrive(kBarCodes + par, kSoftmaxThreads + 32);
            }
        }
    }
    dm::tc_fence_before();
    __syncthreads();
    if (warp == 0) dm::tmem_dealloc(tmem, 512);
}

}  // namespace

namespace dmh {
int check_shape(const DmShape& s, int h0, int hcount, char* err, size_t errlen);
int check_cp(const DmShape& s, const DmCp& cp, char* err, size_t errlen);
}

namespace dmh {
int prepare_bwd1(char* err, size_t errlen) {
    static DeviceOnce once;
    return device_once(once, err, errlen, [&]() -> int {
        constexpr int kPool = kSoftmaxThreads * kRegSoftmax + 256 * kRegFold + 128 * kRegService;
        static_assert(kPool == kThreads * 72, "the roles' register requests must add up to the launch pool");
        for (auto kernel : {(const void*)bwd1_kernel<dm::SnakeWalk>, (const void*)bwd1_kernel<dm::PackedWalk>}) {
            DM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem) + 1024));
            if (int rc = check_register_pool(kernel, kThreads, kPool, err, errlen)) return rc;
        }
        return DM_OK;
    });
}
}  // namespace dmh

namespace dmh {
int launch_bwd1_d256(const void* q8, const void* k8, const void* v8, const void* do8, const float* q8s, const float* k8s, const float* v8s,
                     const float* do8s, const float* lse, const float* delta, DmShape sh, int h0, int hcount, void* dk, void* dv, void* ds8_ws,
                     float* psi_ws, void* stream, char* err, size_t errlen);
}

extern "C" int dm_bwd_workspace_bytes(DmShape sh, int32_t hcount, size_t* ds8_bytes, size_t* psi_bytes) {
    if (!ds8_bytes || !psi_bytes || sh.N <= 0 || sh.N % 128 || sh.B <= 0 || hcount <= 0) return DM_ERR_ARG;
    const size_t kb = sh.D == 128 ? 128 : 64;
    *ds8_bytes = (size_t)sh.B * hcount * sh.N * sh.N;
    *psi_bytes = (size_t)sh.B * hcount * (sh.N / 64) * (sh.N / kb) * sizeof(float);
    return DM_OK;
}

extern "C" int dm_bwd_workspace_bytes_cp(DmShape sh, DmCp cp, int32_t hcount, size_t* ds8_bytes, size_t* psi_bytes) {
    if (!ds8_bytes || !psi_bytes || sh.N <= 0 || sh.N % 128 || sh.B <= 0 || hcount <= 0 || sh.D != 128) return DM_ERR_ARG;
    if (cp.nq <= 0 || cp.nq % 128 || cp.nq > sh.N) return DM_ERR_ARG;
    *ds8_bytes = (size_t)sh.B * hcount * cp.nq * sh.N;
    *psi_bytes = (size_t)sh.B * hcount * (cp.nq / 64) * (sh.N / 128) * sizeof(float);
    return DM_OK;
}

extern "C" int dm_bwd_fp8_pass1(const void* q8, const void* k8, const void* v8, const void* do8, const float* q8s, const float* k8s,
                                const float* v8s, const float* do8s, const float* lse, const float* delta, DmShape sh, int32_t h0,
                                int32_t hcount, void* dk, void* dv, void* ds8_ws, float* psi_ws, void* stream, char* err, size_t errlen) {
    DmCp cp{sh.N, sh.N / 128, 0, 0};
    return dm_bwd_fp8_pass1_cp(q8, k8, v8, do8, q8s, k8s, v8s, do8s, lse, delta, sh, cp, h0, hcount, 0, dk, dv, ds8_ws, psi_ws, stream, err,
                               errlen);
}

extern "C" int dm_bwd_fp8_pass1_cp(const void* q8, const void* k8, const void* v8, const void* do8, const float* q8s, const float* k8s,
                                   const float* v8s, const float* do8s, const float* lse, const float* delta, DmShape sh, DmCp cp,
                                   int32_t h0, int32_t hcount, int32_t out_fp32, void* dk, void* dv, void* ds8_ws, float* psi_ws,
                                   void* stream, char* err, size_t errlen) {
    int rc = dmh::check_shape(sh, h0, hcount, err, errlen);
    if (rc) return rc;
    const bool plain = cp.nq == sh.N && cp.half_blocks == sh.N / 128 && cp.off0 == 0;
    if (!plain && (rc = dmh::check_cp(sh, cp, err, errlen))) return rc;
    DM_REQUIRE(!out_fp32 || sh.D == 128, DM_ERR_UNSUPPORTED, "fp32 dK / dV partials are built for head_dim 128 only");
    const void* ptrs[] = {q8, k8, v8, do8, q8s, k8s, v8s, do8s, lse, delta, dk, dv, ds8_ws, psi_ws};
    const char* names[] = {"q8", "k8", "v8", "do8", "q8s", "k8s", "v8s", "do8s", "lse", "delta", "dk", "dv", "ds8_ws", "psi_ws"};
    for (int i = 0; i < 14; ++i)
        if ((rc = dmh::check_device_ptr(ptrs[i], names[i], err, errlen))) return rc;
    DM_REQUIRE(dmh::aligned16(dk) && dmh::aligned16(dv) && dmh::aligned16(ds8_ws), DM_ERR_ARG, "outputs and workspace must be 16-byte aligned");
    const uint64_t ntiles = (uint64_t)sh.B * hcount * (cp.nq / 128) * (sh.N / 128);
    DM_REQUIRE(ntiles * 128 < ((uint64_t)1 << 31), DM_ERR_ARG, "dS' workspace too large for one call: split the heads (got %llu tiles)",
               (unsigned long long)ntiles);
    if (sh.D == 256)
        return dmh::launch_bwd1_d256(q8, k8, v8, do8, q8s, k8s, v8s, do8s, lse, delta, sh, h0, hcount, dk, dv, ds8_ws, psi_ws, stream, err, errlen);
    CUtensorMap tq, td, tk, tv, ts;
    if ((rc = dmh::make_tmap_u8(&tq, q8, sh.D, (uint64_t)sh.B * sh.H * cp.nq, 128, err, errlen))) return rc;
    if ((rc = dmh::make_tmap_u8(&td, do8, sh.D, (uint64_t)sh.B * sh.H * cp.nq, 128, err, errlen))) return rc;
    if ((rc = dmh::make_tmap_u8(&tk, k8, sh.D, (uint64_t)sh.B * sh.Hk * sh.N, 128, err, errlen))) return rc;
    if ((rc = dmh::make_tmap_u8(&tv, v8, sh.D, (uint64_t)sh.B * sh.Hk * sh.N, 128, err, errlen))) return rc;
    if ((rc = dmh::make_tmap_u8(&ts, ds8_ws, 128, ntiles * 128, 128, err, errlen))) return rc;
    int* status = dmh::device_status_word(err, errlen);
    if (!status) return DM_ERR_CUDA;
    dm::Bwd1Params p{q8s, k8s, v8s, do8s, lse, delta, static_cast<__nv_bfloat16*>(dk), static_cast<__nv_bfloat16*>(dv), static_cast<uint8_t*>(ds8_ws), psi_ws,
                 sh.H, sh.Hk, sh.N, h0, hcount, sh.causal, status, dm::RowMap{cp.nq, cp.half_blocks, cp.off0, cp.off1}, out_fp32,
                 sh.B * hcount, dm::make_fastdiv(sh.B * hcount), dm::make_fastdiv(hcount), dm::make_fastdiv(sh.H / sh.Hk)};
    // persistent: one CTA per SM walks the (key block, head) items, heaviest first
    if ((rc = dmh::prepare_bwd1(err, errlen))) return rc;
    int sms = 0;
    if ((rc = dmh::sm_count(&sms, err, errlen))) return rc;
    const int64_t items = (int64_t)sh.B * hcount * (sh.N / 128);
    const int grid = (int)(items < sms ? items : sms);
    dm::PackedWalk walk;
    if (sh.causal && plain && dmh::plan_walk(sh.B * hcount, sh.N / 128, grid, &walk)) {
        DM_CUDA(dmh::launch_pdl(bwd1_kernel<dm::PackedWalk>, grid, kThreads, sizeof(Smem) + 1024, stream, tq, td, tk, tv, ts, p, walk));
    } else {
        DM_CUDA(dmh::launch_pdl(bwd1_kernel<dm::SnakeWalk>, grid, kThreads, sizeof(Smem) + 1024, stream, tq, td, tk, tv, ts, p, dm::SnakeWalk{}));
    }
    return DM_OK;
}
