// Pass 1 of the backward at head_dim 256 (csrc/mainloop_bwd_sm90_fp8v10.hpp:1674-1761 of the reference): dK and dV per query head, the e4m3
// dS' code tiles and their psi scales (64 rows x 64 keys) for pass 2.  The arithmetic is that of dm_bwd1.cu with K / V scales per 32 keys
// and Q / dO scales per 64-row m-block; the division of the work is another.
//
// One work item = 64 keys (half a key block) of one (batch, query head) with all 256 columns of d, walked in tiles of 128 rows from the causal
// start; persistent, one CTA per SM.  896 threads, as in dm_bwd1.cu:
//   warps 0..15  softmax: P-hat, dS', the tile maxima, psi and both code tiles; warp = 32 rows x 16 keys
//   warps 16..23 fold: thread = (d column, 64 keys); dK in registers, and dV's accumulator kept in the unit of the next dO block
//   warps 24..27 service: the S / dP MMAs, the dK / dV MMAs and the dS' store, the TMA loads, the row constants
// Per tile:
//   S = Q K^T, dP = dO V^T   M128 N64 K32 x 8 each (tensor-memory lane = row), two buffers of each, S as soon as Q is there
//   softmax warps            codes P-hat8, dS'8 in [key][row] tiles, psi by the F2 / F2b rules
//   per m-block m, d half h  X_h = Q8_h(m)^T dS'8(m) (lane = d column, column = key): fold: dK += X (psi 2^-8 q8sc)
//                            dV_h += dO8_h(m)^T P-hat8(m), into the accumulator itself, whose unit is moved after every m-block
// Q8 / dO8 tiles serve twice: K-major as the A operand of S / dP, MN-major as the A operand of dK / dV.
//
// Why this shape.  128 keys x 256 columns of dK and dV do not fit tensor memory and the fold warps.  The kernel before this one gave two work
// items the two d halves of 128 keys, and both formed S / dP, P-hat and the codes of all of them; two items with all of d and half
// the keys each form their own scores only.  The price is that every MMA is N = 64 wide, which takes as long as 128 (2100 clocks of
// tensor pipe a tile), but of the softmax warps' work, which bounded that kernel, each item has half.  Q and dO share a ring of five 32 KB
// units, so that Q (and S) run half a tile further ahead than dO; Q is released behind dK's last product, dO behind dV's.
// Measured, us at B2 N4096 H16 full / causal / B1 N1920 H8 causal: 1056 / 625 / 68.7 with the d halves, 840 / 455 / 36.0 with this.  What bounds
// it: two chains of about 3400 clocks a tile, the fold's (each product's wait, loads and additions, twice; the unit moved twice) and the one
// dS' tile's (codes, both products, free again); shared memory is half busy with operands (280 KB a tile).  On the way: 72 / 96 / 24
// registers for softmax, fold and service 864, 56 / 128 / 24 906 (the service warps spill at 24); the m-blocks'
// loops unrolled 862 (the instruction cache missed one request in nine); two X buffers and one of S / dP instead 855.
#include "dm_attn_common.cuh"
#include "dm_host.h"

namespace {

constexpr int kTile = 128 * 128;               // 128 rows x one 128-byte d half
constexpr int kHalfTile = 64 * 128;            // 64 keys x one 128-byte d half, or x 128 rows of codes
constexpr int kSoftmaxThreads = 512;
constexpr int kFoldWarp = 16, kServiceWarp = 24;
constexpr int kThreads = 896;
constexpr int kRegSoftmax = 56, kRegFold = 120, kRegService = 40;     // per thread after setmaxnreg: the sum is the launch pool
constexpr int kUnits = 5;              // ring of Q and dO tiles (both d halves each): unit 2 t is Q of tile t, 2 t + 1 its dO
constexpr int kRows = 3;               // ring of row constants
constexpr int kGf = 4;                 // ring of product scales between softmax and fold warps
constexpr int kWindow = 64;            // tiles that dV's accumulator sums by itself (dm_bwd1.cu)

// Named barriers (see dm_bwd1.cu).
constexpr int kBarSpFree = 1;          // + tile parity: (S | dP) is in registers            512 + 32
constexpr int kBarAmax = 3;            // + m-block: its warps' maxima are in shared memory  256
constexpr int kBarCodes = 5;           // + tile parity: the tile's codes are                512 + 32
constexpr int kBarXFree = 7;           // the fold warps hold the dK product                 256 + 32
constexpr int kBarDvFree = 8;          // dV's accumulator is in the next m-block's unit     256 + 32

struct Params {
    const float* q8s;
    const float* k8s;
    const float* v8s;
    const float* do8s;
    const float* lse;
    const float* delta;
    __nv_bfloat16* dk;
    __nv_bfloat16* dv;
    float* psi;
    int H, Hk, N, h0, hcount, causal;
    int* status;
    int n_heads;                                  // batch * hcount: (batch, query head) pairs of this call
    dm::FastDiv fd_heads, fd_hcount, fd_rep;      // divisions by n_heads, hcount and H / Hk
};

// The work list: one item = 64 keys `zh` of one 128-key block J of one (batch, query head), ordered by key block, i.e. heaviest first when
// causal, and walked in a snake over the rounds (dm::SnakeWalk).
struct Item {
    dm::HeadCoord hc;
    int J, zh, t_lo, n, bhl;                      // first 128-row tile and their count
    bool valid;
};
__device__ __forceinline__ Item item(const Params& p, int round) {
    Item w;
    const int nbn = p.N / 128;
    const int idx = dm::walk_index(dm::SnakeWalk{}, round);
    w.valid = idx < 2 * p.n_heads * nbn;
    const int jz = (int)dm::fdiv((uint32_t)idx, p.fd_heads);
    w.hc = dm::head_coord(idx - jz * p.n_heads, p.h0, p.fd_hcount, p.H, p.Hk, p.fd_rep);
    w.bhl = w.hc.b * p.hcount + (w.hc.h - p.h0);
    w.J = jz >> 1;
    w.zh = jz & 1;
    w.t_lo = p.causal ? w.J : 0;
    w.n = nbn - w.t_lo;
    return w;
}

struct Smem {
    alignas(1024) uint8_t k[2][kHalfTile];    // [d half][key]
    alignas(1024) uint8_t v[2][kHalfTile];
    alignas(1024) uint8_t qdo[kUnits][2][kTile];   // [unit][d half][row]
    alignas(1024) uint8_t pt[2][kHalfTile];   // P-hat codes, [key][row], by tile parity
    alignas(1024) uint8_t ds[kHalfTile];      // dS' codes, same layout
    alignas(16) float2 rd[kRows][128];        // per row: 8 - lse * log2e, -delta
    alignas(16) float sc[kRows][8];           // of m-block m: [m] q8sc, [2 + m] do8sc, [4 + m] what dV's accumulator is multiplied by before it,
                                              // [6 + m] dV's unit
    float gf[kGf][2];                         // dK scale of m-block m
    float fv[kGf];                            // dV's unit after the tile
    float psi[kGf][2];                        // psi of m-block m, on its way to pass 2
    float amax[2][16];                        // [tile parity][m-block, warp of it]
    uint64_t bar_kv, bar_kv_free, bar_unit[kUnits], bar_unit_free[kUnits], bar_s[2], bar_dp[2], bar_x, bar_dv, bar_pt_free[2], bar_ds_free,
        bar_rows[kRows], bar_rows_free[kRows];
    uint32_t tmem_base;
    int abort_flag;
};

__global__ void __launch_bounds__(kThreads, 1)
bwd1_d256_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_ds, const Params p) {
    extern __shared__ uint8_t smem_raw[];
    Smem& s = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    // The hardware warps are taken in the order service, fold, softmax (the role numbers below keep their tensor-memory quarter).
    const int tid = threadIdx.x, lane = tid & 31, hw_warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int warp = hw_warp < 4 ? hw_warp + kServiceWarp : (hw_warp < 12 ? hw_warp + kFoldWarp - 4 : hw_warp - 12);
    const int nbn = p.N / 128;
    // `t` counts the CTA's tiles over its items, so ring places, buffer parities and mbarrier phases run on across items.
    dm::WaitCtx wc{&s.abort_flag, p.status};

    if (tid == 0) {
        s.abort_flag = 0;
        dm::mbar_init(&s.bar_kv, 1);
        dm::mbar_init(&s.bar_kv_free, 1);
        dm::mbar_init(&s.bar_x, 1);
        dm::mbar_init(&s.bar_dv, 1);
        dm::mbar_init(&s.bar_ds_free, 2);
        for (int i = 0; i < kUnits; ++i) {
            dm::mbar_init(&s.bar_unit[i], 1);
            dm::mbar_init(&s.bar_unit_free[i], 1);
        }
        for (int i = 0; i < kRows; ++i) {
            dm::mbar_init(&s.bar_rows[i], 1);
            dm::mbar_init(&s.bar_rows_free[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            dm::mbar_init(&s.bar_s[i], 1);
            dm::mbar_init(&s.bar_dp[i], 1);
            dm::mbar_init(&s.bar_pt_free[i], 1);
        }
        dm::fence_mbar_init();
        dm::tma_prefetch_desc(&tm_q);
        dm::tma_prefetch_desc(&tm_do);
        dm::tma_prefetch_desc(&tm_k);
        dm::tma_prefetch_desc(&tm_v);
    }
    if (warp == 0) dm::tmem_alloc(&s.tmem_base, 512);
    dm::tc_fence_before();
    __syncthreads();
    dm::tc_fence_after();
    dm::pdl_wait();
    // tensor memory: by tile parity S [0, 64) | dP [64, 128) and S [128, 192) | dP [192, 256) (lane = row); the product X [256, 384) and dV's
    // accumulator [384, 512), 64 keys per d half (lane = d column)
    const uint32_t tmem = s.tmem_base;
    const uint32_t t_x = tmem + 256, t_dva = tmem + 384;
    const uint32_t lane_base = (uint32_t)(warp & 3) * 32;

    if (warp >= kServiceWarp) {
        // =============================================================== service warps: loops converged, one elected lane issues
        dm::reg_dec<kRegService>();
        constexpr uint32_t kSub = kTile >> 4, kHalf = kHalfTile >> 4;
        if (warp == kServiceWarp) {
            // ---- S = Q K^T and dP = dO V^T of every tile, into the buffers of its parity, once the softmax warps have read tile t - 2's
            constexpr uint32_t idesc_sp = dm::idesc_e4m3(128, 64, false, false);
            const uint32_t k_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.k[0])), v_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.v[0]));
            const uint32_t u_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.qdo[0][0]));
            int t = 0, kvn = 0, u = 0, up = 0;             // the unit's place in the ring and its phase
            for (int r = 0;; ++r) {
                const Item w = item(p, r);
                if (!w.valid) break;
                dm::mbar_wait(&s.bar_kv, kvn++ & 1, wc);
                for (int it = 0; it < w.n; ++it, ++t) {
                    const int par = t & 1;
                    dm::mbar_wait(&s.bar_rows[t % kRows], (t / kRows) & 1, wc);       // saves the softmax warps a wait of their own
                    if (t >= 2) dm::named_bar_sync(kBarSpFree + par, kSoftmaxThreads + 32);
#pragma unroll 1
                    for (int m = 0; m < 2; ++m) {          // S, then dP
                        dm::mbar_wait(&s.bar_unit[u], up, wc);
                        // the softmax warps write their P-hat codes behind dP, over those of tile t - 2
                        if (m == 1 && t >= 2) dm::mbar_wait(&s.bar_pt_free[par], ((t - 2) >> 1) & 1, wc);
                        dm::tc_fence_after();
                        const uint32_t a = u_lo + 2 * u * kSub, b = m ? v_lo : k_lo, d = tmem + 128 * par + 64 * m;
                        if (dm::elect_one()) {
#pragma unroll
                            for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    if ((hh | k) == 0) dm::umma_e4m3_lo<false>(d, a, b, idesc_sp);
                                    else dm::umma_e4m3_lo<true>(d, a + hh * kSub + 2 * k, b + hh * kHalf + 2 * k, idesc_sp);
                                }
                            dm::umma_commit(m ? &s.bar_dp[par] : &s.bar_s[par]);
                            if (m == 1 && it == w.n - 1) dm::umma_commit(&s.bar_kv_free);     // the loader may bring the next item's K / V
                        }
                        __syncwarp();
                        if (++u == kUnits) {
                            u = 0;
                            up ^= 1;
                        }
                    }
                }
            }
            // the last releases: no arrival is left over
            if (t > 0) dm::named_bar_sync(kBarSpFree + ((t - 1) & 1), kSoftmaxThreads + 32);
            if (t > 1) dm::named_bar_sync(kBarSpFree + (t & 1), kSoftmaxThreads + 32);
        } else if (warp == kServiceWarp + 1) {
            // ---- dK's products of a tile through X, dV's into its accumulator, m-block by m-block; the dS' store
            constexpr uint32_t idesc_x = dm::idesc_e4m3(128, 64, true, false);
            const uint32_t u_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.qdo[0][0]));
            const uint32_t pt_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.pt[0])), ds_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.ds));
            int t = 0, u = 0;
            for (int r = 0;; ++r) {
                const Item w = item(p, r);
                if (!w.valid) break;
                int ds_row = (int)((((int64_t)w.bhl * nbn + w.t_lo) * nbn + w.J) * 128) + 64 * w.zh;   // dS' tile of the first row block
                const int psi_stride = 2 * nbn;
                float* psi_out = p.psi + ((int64_t)w.bhl * (2 * nbn) + 2 * w.t_lo + lane) * psi_stride + 2 * w.J + w.zh;
                for (int it = 0; it < w.n; ++it, ++t, ds_row += nbn * 128) {
                    const int par = t & 1, uq = u, ud = u + 1 == kUnits ? 0 : u + 1;
                    u = ud + 1 == kUnits ? 0 : ud + 1;
                    dm::named_bar_sync(kBarCodes + par, kSoftmaxThreads + 32);
#pragma unroll 1
                    for (int m = 0; m < 2; ++m) {          // the two m-blocks
                        if (t > 0 || m > 0) dm::named_bar_sync(kBarXFree, 256 + 32);
                        dm::tc_fence_after();
                        if (dm::elect_one()) {
#pragma unroll
                            for (int hh = 0; hh < 2; ++hh) {
                                const uint32_t a = u_lo + (2 * uq + hh) * kSub + 512 * m, b = ds_lo + 4 * m;
                                dm::umma_e4m3_lo<false>(t_x + 64 * hh, a, b, idesc_x);
                                dm::umma_e4m3_lo<true>(t_x + 64 * hh, a + 256, b + 2, idesc_x);
                            }
                            dm::umma_commit(&s.bar_x);
                            if (m == 0) {
                                dm::tma_store_2d(&tm_ds, 0, ds_row, s.ds);
                                dm::tma_store_commit();
                            } else {                       // Q has been read for the last time; the dS' tile by both products, and it has left
                                dm::umma_commit(&s.bar_unit_free[uq]);
                                dm::umma_commit(&s.bar_ds_free);
                                dm::tma_store_wait_read0();
                                dm::mbar_arrive(&s.bar_ds_free);
                            }
                        }
                        __syncwarp();
                        if (m == 0 && lane < 2) psi_out[(int64_t)(2 * it) * psi_stride] = s.psi[t % kGf][lane];
                        if (t > 0 || m > 0) dm::named_bar_sync(kBarDvFree, 256 + 32);
                        dm::tc_fence_after();
                        if (dm::elect_one()) {
#pragma unroll
                            for (int hh = 0; hh < 2; ++hh) {
                                const uint32_t a = u_lo + (2 * ud + hh) * kSub + 512 * m, b = pt_lo + par * kHalf + 4 * m;
                                dm::umma_e4m3_lo_rt(t_dva + 64 * hh, a, b, idesc_x, it % kWindow != 0 || m > 0);
                                dm::umma_e4m3_lo<true>(t_dva + 64 * hh, a + 256, b + 2, idesc_x);
                            }
                            dm::umma_commit(&s.bar_dv);
                            if (m == 1) {
                                dm::umma_commit(&s.bar_unit_free[ud]);
                                dm::umma_commit(&s.bar_pt_free[par]);
                                dm::mbar_arrive(&s.bar_rows_free[t % kRows]);
                            }
                        }
                        __syncwarp();
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
            // ---- TMA loads: an item's K / V once the previous item's last S / dP have read theirs, then its Q8 / dO8 tiles as far ahead as the
            // ring allows
            int kvn = 0, u = 0, n = 0;                     // n: units so far
            for (int r = 0;; ++r) {
                const Item w = item(p, r);
                if (!w.valid) break;
                const int kv_row0 = w.hc.bhk * p.N + w.J * 128 + 64 * w.zh;
                const int q_row0 = w.hc.bh * p.N + w.t_lo * 128;
                for (int i = 0; i < 2 * w.n; ++i, ++n) {
                    if (n >= kUnits) dm::mbar_wait(&s.bar_unit_free[u], (n / kUnits - 1) & 1, wc);
                    if (dm::elect_one()) {
                        const CUtensorMap* tm = (i & 1) ? &tm_do : &tm_q;
                        const int row = q_row0 + (i >> 1) * 128;
                        dm::mbar_expect_tx(&s.bar_unit[u], 2 * kTile);
                        dm::tma_load_2d(s.qdo[u][0], tm, 0, row, &s.bar_unit[u]);
                        dm::tma_load_2d(s.qdo[u][1], tm, 128, row, &s.bar_unit[u]);
                    }
                    __syncwarp();
                    if (++u == kUnits) u = 0;
                    if (i == 0) {                          // behind the first Q, whose place has long been free
                        if (kvn >= 1) dm::mbar_wait(&s.bar_kv_free, (kvn - 1) & 1, wc);
                        if (dm::elect_one()) {
                            dm::mbar_expect_tx(&s.bar_kv, 4 * kHalfTile);
#pragma unroll
                            for (int hh = 0; hh < 2; ++hh) {
                                dm::tma_load_2d(s.k[hh], &tm_k, 128 * hh, kv_row0, &s.bar_kv);
                                dm::tma_load_2d(s.v[hh], &tm_v, 128 * hh, kv_row0, &s.bar_kv);
                            }
                        }
                        __syncwarp();
                        ++kvn;
                    }
                }
            }
        } else {
            // ---- the rows' constants (four per lane) and the Q / dO scales of the tile's m-blocks, kRows ahead
            int t = 0;
            for (int r = 0;; ++r) {
                const Item w = item(p, r);
                if (!w.valid) break;
                float unit = 0.f, top = 0.f;
                for (int it = 0; it < w.n; ++it, ++t) {
                    const int slot = t % kRows, li = w.t_lo + it;
                    const int64_t gi = (int64_t)w.hc.bh * p.N + (int64_t)li * 128 + 4 * lane;
                    float l4[4], d4[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        l4[i] = p.lse[gi + i];
                        d4[i] = p.delta[gi + i];
                    }
                    const int64_t sq = ((int64_t)w.hc.bh * nbn + li) * 2;
                    float q8sc[2], do8sc[2], mult[2], un[2];
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        q8sc[m] = p.q8s[sq + m];
                        do8sc[m] = p.do8s[sq + m];
                        // dV's accumulator is kept in units of the current dO scale block's scale, so that the MMAs add to it directly.
                        // A block more than 2^-80 below the item's largest so far (an all-zero one) takes the unit at that bound: the
                        // accumulator stays finite, and zero codes add nothing whatever the unit is.
                        top = fmaxf(top, do8sc[m]);
                        const float unit_new = fmaxf(do8sc[m], top * 0x1p-80f);
                        mult[m] = unit / unit_new;
                        unit = unit_new;
                        un[m] = dm::kMoInv * unit;
                    }
                    if (t >= kRows) dm::mbar_wait(&s.bar_rows_free[slot], (t / kRows - 1) & 1, wc);
#pragma unroll
                    for (int i = 0; i < 4; i += 2)
                        *reinterpret_cast<float4*>(&s.rd[slot][4 * lane + i]) =
                            make_float4(dm::phat_row_const(l4[i]), -d4[i], dm::phat_row_const(l4[i + 1]), -d4[i + 1]);
                    if (lane == 0) {
                        *reinterpret_cast<float4*>(s.sc[slot]) = make_float4(q8sc[0], q8sc[1], do8sc[0], do8sc[1]);
                        *reinterpret_cast<float4*>(s.sc[slot] + 4) = make_float4(mult[0], mult[1], un[0], un[1]);
                    }
                    __syncwarp();
                    if (dm::elect_one()) dm::mbar_arrive(&s.bar_rows[slot]);
                }
            }
        }
    } else if (warp >= kFoldWarp) {
        // =============================================================== fold warps: thread = (d column, 64 keys)
        dm::reg_inc<kRegFold>();
        const int half = (warp >> 2) & 1;
        const uint32_t x_src = dm::tmem_addr(t_x, lane_base, 64 * half), dva = dm::tmem_addr(t_dva, lane_base, 64 * half);
        int t = 0;
        for (int r = 0;; ++r) {
            int n;                                     // all that the tile loop keeps of the item: it has no registers to spare
            {
                const Item w = item(p, r);
                if (!w.valid) break;
                n = w.n;
            }
            float dk_acc[64];
#pragma unroll
            for (int i = 0; i < 64; ++i) dk_acc[i] = 0.f;
            auto fold_dk = [&](int m) {                             // two products a tile
                dm::mbar_wait(&s.bar_x, m, wc);                     // also orders the ring slot written before the codes
                dm::tc_fence_after();
                // four 16-column pieces, two in flight
                uint32_t sa[16], sb[16];
                dm::tmem_ld16(x_src, sa);
                dm::tmem_ld16(x_src + 16, sb);
                const float gk = s.gf[t % kGf][m];
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
                for (int pc = 0; pc < 64; pc += 32) {
                    uint32_t sa[16], sb[16];
                    dm::tmem_ld16(dva + pc, sa);
                    dm::tmem_ld16(dva + pc + 16, sb);
                    dm::tmem_ld_wait();
                    auto mul16 = [&](uint32_t* x) {
#pragma unroll
                        for (int i = 0; i < 16; i += 2) {
                            float y0, y1;
                            dm::mul2(y0, y1, __uint_as_float(x[i]), __uint_as_float(x[i + 1]), mult, mult);
                            x[i] = __float_as_uint(y0);
                            x[i + 1] = __float_as_uint(y1);
                        }
                    };
                    mul16(sa);
                    dm::tmem_st16(dva + pc, sa);
                    mul16(sb);
                    dm::tmem_st16(dva + pc + 16, sb);
                }
                dm::tmem_st_wait();
                dm::tc_fence_before();
                dm::named_bar_arrive(kBarDvFree, 256 + 32);
            };
            // The thread's place in dK and dV: its column of the item's first key.  (Looked up again: the tile loop has no registers for it.)
            auto out_offset = [&]() {
                int r_again = r;
                asm volatile("" : "+r"(r_again));
                const Item v = item(p, r_again);
                return (((int64_t)v.hc.b * p.N + v.J * 128 + 64 * v.zh) * p.H + v.hc.h) * 256 + 128 * half + lane_base + lane;
            };
            const int64_t key_stride = (int64_t)p.H * 256;          // elements between consecutive keys
            // The fp32 sum of dV's earlier windows lives in the item's own outputs, which are written at its end: a warp's 32 columns x 64 keys
            // of dK and dV are 8 KB, its share of the sum.  Unit u (16 keys) is in dV's (u even) or dK's half of 32 keys u / 2, lane l's
            // sixteen numbers in the 64 bytes of the warp's columns of key 32 (u / 2) + l: the epilogue's stores of a unit's keys to dV then
            // cover only what has been read.  A slot is one thread's own.
            auto sum_at = [&](int64_t off, int u) {
                return reinterpret_cast<float4*>(((u & 1) ? p.dk : p.dv) + (off - lane) + (32 * (u >> 1) + lane) * key_stride);
            };
            auto flush_dv = [&](float unit, bool first) {
                const int64_t off = out_offset();
#pragma unroll 1
                for (int u = 0; u < 4; ++u) {
                    float4* to = sum_at(off, u);
#pragma unroll
                    for (int c = 0; c < 16; c += 8) {
                        uint32_t sa[8];
                        dm::tmem_ld8(dva + 16 * u + c, sa);
                        dm::tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 8; e += 4, ++to) {
                            const float4 y = make_float4(__uint_as_float(sa[e]) * unit, __uint_as_float(sa[e + 1]) * unit,
                                                         __uint_as_float(sa[e + 2]) * unit, __uint_as_float(sa[e + 3]) * unit);
                            if (first) *to = y;
                            else dm::red_add_f32x4(to, y);
                        }
                    }
                }
                dm::tc_fence_before();
                dm::named_bar_arrive(kBarDvFree, 256 + 32);
            };
            for (int it = 0; it < n;) {
                const int end = min(n, it + kWindow);
                for (; it < end; ++it, ++t) {
#pragma unroll 1
                    for (int m = 0; m < 2; ++m) {
                        fold_dk(m);
                        dm::mbar_wait(&s.bar_dv, m, wc);            // two commits a tile, as for X
                        dm::tc_fence_after();
                        if (m == 1 && it + 1 == end) break;         // (the flush or the epilogue releases the accumulator)
                        const int slot = (t + m) % kRows;
                        if (m == 1) dm::mbar_wait(&s.bar_rows[slot], ((t + 1) / kRows) & 1, wc);
                        rescale_dv(s.sc[slot][5 - m]);
                    }
                }
                if (n > kWindow) flush_dv(s.fv[(t + kGf - 1) % kGf], it == kWindow);
            }

            // ---- epilogue: dK *= 1 / k8s, dV from its accumulator (after a long walk from the sum of the windows, before dK: dK's rows hold a part
            // of it), per query head.  A key's 32 columns of a warp are one whole 64-byte piece, so the values are stored as they lie.
            const bool have_sum = n > kWindow;
            const float fv = s.fv[(t + kGf - 1) % kGf];             // dV's last unit
            const int64_t off = out_offset();
            float ik[2];
            {
                int r_again = r;
                asm volatile("" : "+r"(r_again));
                const Item w = item(p, r_again);
#pragma unroll
                for (int i = 0; i < 2; ++i) ik[i] = 1.0f / p.k8s[(int64_t)w.hc.bhk * (p.N / 32) + 4 * w.J + 2 * w.zh + i];
            }
#pragma unroll 1
            for (int u = 0; u < 4; ++u) {
                float y[16];
                if (have_sum) {
                    const float4* from = sum_at(off, u);
#pragma unroll
                    for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(y + 4 * j) = __ldcg(from + j);
                    __syncwarp();                                   // the warp has read the unit: its place may be written
                } else {
                    dm::tmem_ld16(dva + 16 * u, reinterpret_cast<uint32_t*>(y));
                    dm::tmem_ld_wait();
                }
                const float f = have_sum ? 1.0f : fv;
#pragma unroll
                for (int i = 0; i < 16; ++i) p.dv[off + (16 * u + i) * key_stride] = __float2bfloat16_rn(y[i] * f);
            }
            if (!have_sum) {
                dm::tc_fence_before();
                dm::named_bar_arrive(kBarDvFree, 256 + 32);
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 64; ++i) p.dk[off + i * key_stride] = __float2bfloat16_rn(dk_acc[i] * ik[i >> 5]);
        }
    } else {
        // =============================================================== softmax warps: 32 rows x 16 keys
        dm::reg_dec<kRegSoftmax>();
        const int rq = warp & 3, kq = warp >> 2;      // rows [32 rq, +32) and keys [16 kq, +16) of the tile
        const int rhalf = rq >> 1;                    // the 64-row m-block
        const bool leader = (warp & 13) == 0;         // one warp of each m-block
        const int row_t = 32 * rq + (lane >> 2);      // the thread's rows: row_t + {0, 8, 16, 24}
        const uint32_t t_s = dm::tmem_addr(tmem, lane_base, 16 * kq);
        // this lane's line of the transposed stores: fragment (16 rows h, 8 keys j) = lane / 8 = 2 h + j; key 16 kq + 8 j + lane % 8, chunk 2 rq + h
        const uint32_t st_addr = dm::smem_u32(s.pt[0]) + (16 * kq + (lane & 15)) * 128 + (((2 * rq + (lane >> 4)) ^ (lane & 7)) << 4);
        const uint32_t ds_addr = st_addr + (dm::smem_u32(s.ds) - dm::smem_u32(s.pt[0]));
        int t = 0, rb = 0;                            // tiles so far; ring slot of the row constants
        for (int r = 0;; ++r) {
            const Item w = item(p, r);
            if (!w.valid) break;
            const int n = w.n;
            const int64_t si = (int64_t)w.hc.bhk * (p.N / 32) + 4 * w.J + 2 * w.zh + (kq >> 1);
            const float k8s_t = p.k8s[si], v8s_t = p.v8s[si];
            const int ahead = row_t - (64 * w.zh + 16 * kq + 2 * (lane & 3));        // on the diagonal block: the thread's row minus its key
            float g_max = 0.f;

            for (int it = 0; it < n; ++it, ++t, rb = rb == kRows - 1 ? 0 : rb + 1) {
                const int par = t & 1;
                dm::mbar_wait(&s.bar_s[par], (t >> 1) & 1, wc);
                dm::tc_fence_after();
                // ---- phase 1: P-hat, dS', tile amax; P-hat codes to shared memory.  Element 8 h + 4 j + 2 a + e: row row_t + 16 h + 8 a, key
                // 2 (lane % 4) + 8 j + e
                float sv[16], ds[16];
                dm::tmem_ld16x256_x2(t_s + 128 * par, reinterpret_cast<uint32_t*>(sv));
                dm::tmem_ld16x256_x2(t_s + 128 * par + (16u << 16), reinterpret_cast<uint32_t*>(sv + 8));
                const float q8sc = s.sc[rb][rhalf], do8sc = s.sc[rb][2 + rhalf];
                const float dsc = dm::descale_log2(q8sc, k8s_t);
                const float dpk = do8sc * v8s_t * k8s_t;
                float2 rd[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) rd[i] = s.rd[rb][row_t + 8 * i];
                dm::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; j += 2) {               // P-hat = 2^min(S dsc + rc, 12), the exponent two at a time
                    const float rc = rd[2 * (j >> 3) + ((j >> 1) & 1)].x;
                    dm::fma2(sv[j], sv[j + 1], sv[j], sv[j + 1], dsc, rc, rc);
                    sv[j] = dm::ex2(fminf(sv[j], dm::kMoE + 4.0f));
                    sv[j + 1] = dm::ex2(fminf(sv[j + 1], dm::kMoE + 4.0f));
                }
                if (p.causal && it == 0) {                      // the diagonal block only: keys above the row
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (2 * (j & 4) + (j & 1) - 2 * (j & 8) - 4 * (j & 2) > ahead) sv[j] = 0.f;
                }
                dm::mbar_wait(&s.bar_dp[par], (t >> 1) & 1, wc);
                dm::tc_fence_after();
                dm::tmem_ld16x256_x2(t_s + 128 * par + 64, reinterpret_cast<uint32_t*>(ds));
                dm::tmem_ld16x256_x2(t_s + 128 * par + 64 + (16u << 16), reinterpret_cast<uint32_t*>(ds + 8));
                dm::tmem_ld_wait();
                dm::tc_fence_before();
                dm::named_bar_arrive(kBarSpFree + par, kSoftmaxThreads + 32);       // (S | dP) may be overwritten
                float am0 = 0.f, am1 = 0.f;
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    const float da = rd[2 * (j >> 3)].y * k8s_t, db = rd[2 * (j >> 3) + 1].y * k8s_t;      // -delta * k8s
                    dm::fma2(ds[j], ds[j + 1], ds[j], ds[j + 1], dpk, da, da);
                    dm::fma2(ds[j + 2], ds[j + 3], ds[j + 2], ds[j + 3], dpk, db, db);
                    dm::mul2(ds[j], ds[j + 1], ds[j], ds[j + 1], sv[j], sv[j + 1]);
                    dm::mul2(ds[j + 2], ds[j + 3], ds[j + 2], ds[j + 3], sv[j + 2], sv[j + 3]);
                    am0 = dm::fmax3_abs(am0, ds[j], ds[j + 1]);
                    am1 = dm::fmax3_abs(am1, ds[j + 2], ds[j + 3]);
                }
                uint32_t c4[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) c4[j] = dm::cvt_e4m3x4(sv[4 * j], sv[4 * j + 1], sv[4 * j + 2], sv[4 * j + 3]);
                dm::stmatrix_t_b8_x4(st_addr + par * kHalfTile, c4);
                // the warp's maximum in one instruction: non-negative floats order like their bit patterns
                const float am = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(am0, am1))));
                if (lane == 0) s.amax[par][8 * rhalf + 2 * kq + (rq & 1)] = am;
                if (leader && t >= 1) dm::mbar_wait(&s.bar_ds_free, (t - 1) & 1, wc);       // the dS' tile is free
                dm::named_bar_sync(kBarAmax + rhalf, 256);
                // psi = max(psi_raw, g_max * 256e-8 / q8sc), as in dm_bwd1.cu
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
                for (int j = 0; j < 4; ++j) {
                    float a0, a1, a2, a3;
                    dm::mul2(a0, a1, ds[4 * j], ds[4 * j + 1], psi_inv, psi_inv);
                    dm::mul2(a2, a3, ds[4 * j + 2], ds[4 * j + 3], psi_inv, psi_inv);
                    c4[j] = dm::cvt_e4m3x4(a0, a1, a2, a3);
                }
                dm::stmatrix_t_b8_x4(ds_addr, c4);
                // the scales of this tile's products for the fold warps (the ring slot was last read four tiles ago; the P-hat codes of this
                // tile waited for the products of two tiles ago) and psi, which the product warp takes to global memory
                if (leader && lane == 0) {
                    s.gf[t % kGf][rhalf] = g_my;
                    s.psi[t % kGf][rhalf] = psi_my;
                    if (warp == 0) s.fv[t % kGf] = s.sc[rb][7];
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
int prepare_bwd1_d256(char* err, size_t errlen) {
    static DeviceOnce once;
    return device_once(once, err, errlen, [&]() -> int {
        DM_CUDA(cudaFuncSetAttribute(bwd1_d256_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem) + 1024));
        constexpr int kPool = kSoftmaxThreads * kRegSoftmax + 256 * kRegFold + 128 * kRegService;
        static_assert(kPool == kThreads * 72, "the roles' register requests must add up to the launch pool");
        return check_register_pool((const void*)bwd1_d256_kernel, kThreads, kPool, err, errlen);
    });
}

int launch_bwd1_d256(const void* q8, const void* k8, const void* v8, const void* do8, const float* q8s, const float* k8s, const float* v8s,
                     const float* do8s, const float* lse, const float* delta, DmShape sh, int h0, int hcount, void* dk, void* dv, void* ds8_ws,
                     float* psi_ws, void* stream, char* err, size_t errlen) {
    int rc;
    CUtensorMap tq, td, tk, tv, ts;
    const uint64_t tiles = (uint64_t)sh.B * hcount * (sh.N / 128) * (sh.N / 128);
    if ((rc = make_tmap_u8(&tq, q8, 256, (uint64_t)sh.B * sh.H * sh.N, 128, err, errlen))) return rc;
    if ((rc = make_tmap_u8(&td, do8, 256, (uint64_t)sh.B * sh.H * sh.N, 128, err, errlen))) return rc;
    if ((rc = make_tmap_u8(&tk, k8, 256, (uint64_t)sh.B * sh.Hk * sh.N, 64, err, errlen))) return rc;
    if ((rc = make_tmap_u8(&tv, v8, 256, (uint64_t)sh.B * sh.Hk * sh.N, 64, err, errlen))) return rc;
    if ((rc = make_tmap_u8(&ts, ds8_ws, 128, tiles * 128, 64, err, errlen))) return rc;
    int* status = device_status_word(err, errlen);
    if (!status) return DM_ERR_CUDA;
    Params p{q8s, k8s, v8s, do8s, lse, delta, static_cast<__nv_bfloat16*>(dk), static_cast<__nv_bfloat16*>(dv), psi_ws, sh.H, sh.Hk, sh.N, h0, hcount,
             sh.causal, status, sh.B * hcount, dm::make_fastdiv(sh.B * hcount), dm::make_fastdiv(hcount), dm::make_fastdiv(sh.H / sh.Hk)};
    if ((rc = prepare_bwd1_d256(err, errlen))) return rc;
    int sms = 0;
    if ((rc = sm_count(&sms, err, errlen))) return rc;
    // persistent: one CTA per SM walks the (key half block, head) items, heaviest first
    const int64_t items = (int64_t)sh.B * hcount * (sh.N / 128) * 2;
    const int grid = (int)(items < sms ? items : sms);
    DM_CUDA(launch_pdl(bwd1_d256_kernel, grid, kThreads, sizeof(Smem) + 1024, stream, tq, td, tk, tv, ts, p));
    return DM_OK;
}
}  // namespace dmh
