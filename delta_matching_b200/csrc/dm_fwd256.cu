// Forward kernel, head_dim 256: the head_dim-128 design (dm_fwd.cu) in the head_dim-256 geometry of the reference
// (csrc/flash_fwd_fp8f_launch.h:40, csrc/softmax_fq8f.h kGroups = 4): Q scales per 64 rows, K / V scales per 32 keys,
// key tiles of 128 keys = FOUR 32-key P groups, each with its own per-row basis.
//
// One work item = 128 query rows of one (batch, head); the kernel is persistent, one CTA per SM walks its items (dm::SnakeWalk),
// and every role keeps its own place in the list.  A code row is 256 bytes = two 128-byte swizzled sub-tiles (d 0..127 and d 128..255).
// 512 threads:
//   warps 0..3   service (one elected lane issues): S; the products; the loads of Q and K; the loads of V
//   warps 4..11  fold: thread = (row, d half), 128 of O's columns in registers
//   warps 12..15 softmax: thread = row, with all four P groups of the tile; nothing is exchanged
// Per tile:
//   S = Q K^T        8 x tcgen05.mma (M128 N128 K32) into the one S buffer, as soon as the softmax warps have read the previous tile's
//   softmax          the group maxima, the row's running maximum (and with it alpha, the groups' bases and weights); codes to shared memory
//                    (the products' A operand)
//   D = C_g V_g      one M128 N128 K32 MMA per group and d half into one of three product buffers in turn: the next two are formed while
//                    the fold warps add one up
//   fold             O = O alpha (the tile's first group), O += D (v8sc sigma) in group order; O / l at the item's end
// Every mbarrier wait is bounded.
//
// Why this shape.  O's 128 x 256 accumulators are half the register file, so eight fold warps hold 128 each and what is left serves one
// softmax warp per scheduler; four groups of 32 keys mean four products of 128 x 256 per tile, i.e. 1024 clocks of tensor-memory loads and
// about 1600 of multiply-adds a tile, beside 1024 of exponentials.  One thread for scores and O (255 registers, eight warps,
// everything in turn) took 5900 clocks a tile; this takes 3700, and is bound by the fold warps' chain (a product's wait, loads and
// additions: about 900 clocks a unit, four units a tile) with the softmax warps close behind.  us at B2 N4096 H16 full / causal / B1 N1920 H8
// causal: 641 / 352 / 46.7 before, 430 / 238 / 35.6 now.  On the way: eight softmax warps, the fold in 8-column pieces (160 registers)
// 484; this split with the roles taken by hardware warp number 460, by role number 430 (below); S behind the products of two tiles
// ago: the same; both halves' warps on every product 611, that unrolled over the tile 768 (instruction cache misses: two fifths of
// its requests).
#include "dm_attn_common.cuh"
#include "dm_host.h"

namespace dmh {
int check_shape(const DmShape& s, int h0, int hcount, char* err, size_t errlen);
}

namespace {

constexpr int kTile = 128 * 128;
constexpr int kThreads = 512;
constexpr int kFoldWarp = 4, kSoftmaxWarp = 12;                        // (role numbers)
constexpr int kFoldThreads = 256, kSoftmaxThreads = 128;
constexpr int kRegSoftmax = 120, kRegFold = 184, kRegService = 24;      // per thread after setmaxnreg; the sum is the launch pool
constexpr int kBufs = 3;           // product buffers
constexpr int kRing = 3;           // tiles of row constants between softmax and fold warps
// Named barriers (see dm_fwd.cu).
constexpr int kBarSFree = 1;       // S has been read                                            128 + 32
constexpr int kBarCodes = 2;       // + 2 * tile parity + half: two groups' codes are in shared memory   128 + 32
constexpr int kBarDFree = 6;       // + product unit % 6: its d half's fold warps hold it               128 + 32

struct Fwd256Smem {
    alignas(1024) uint8_t q[2][kTile];          // [d half][128 rows x 128 bytes]
    alignas(1024) uint8_t k[2][2][kTile];       // [stage][d half]
    alignas(1024) uint8_t v[2][2][kTile];
    alignas(1024) uint8_t c[2][kTile];          // P codes by tile parity: [row][key]
    alignas(16) uint8_t stg[8][32 * 64];        // per fold warp: 32 bf16 columns of its 32 rows on their way out (chunks XOR-swizzled)
    alignas(16) float4 w[kRing][128];           // [tile % kRing][row]: the groups' weights
    float alpha[kRing][128];
    float2 ml[kRing][128];                      // an item's last tile: the row's maximum and denominator
    uint64_t bar_q, bar_q_free, bar_k[2], bar_k_free[2], bar_v[2], bar_pv[2], bar_s, bar_d[2 * kBufs];
    uint32_t tmem_base;
    int abort_flag;
};

struct Fwd256Params {
    const float* q8s;
    const float* k8s;
    const float* v8s;
    __nv_bfloat16* o;
    float* lse;
    int H, Hk, N, h0, hcount, causal;
    int* status;
    int n_heads;                      // B * hcount: work items are (head, row block), heaviest row blocks first
    dm::FastDiv fd_heads, fd_hcount, fd_rep;   // divisions by n_heads, hcount and H / Hk
};

struct Fwd256Item {
    dm::HeadCoord hc;
    int I, n_tiles;
    bool valid;
};
__device__ __forceinline__ Fwd256Item fwd256_item(const Fwd256Params& p, int round) {
    Fwd256Item w;
    const int nblk = p.N / 128;
    const int idx = dm::walk_index(dm::SnakeWalk{}, round);
    w.valid = idx < p.n_heads * nblk;
    const int rank = (int)dm::fdiv((uint32_t)idx, p.fd_heads);
    w.hc = dm::head_coord(idx - rank * p.n_heads, p.h0, p.fd_hcount, p.H, p.Hk, p.fd_rep);
    w.I = nblk - 1 - rank;
    w.n_tiles = p.causal ? w.I + 1 : nblk;
    return w;
}

__global__ void __launch_bounds__(kThreads, 1)
fwd_d256_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const Fwd256Params p) {
    extern __shared__ uint8_t smem_raw[];
    Fwd256Smem& s = *reinterpret_cast<Fwd256Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    // The hardware warps are taken in the order softmax, service, fold (the role numbers below keep their tensor-memory quarter, warp mod 4):
    // 460 -> 430 us at B2 N4096 H16 full; service, softmax, fold 435; fold or service before both others 462 to 470.
    const int tid = threadIdx.x, lane = tid & 31, hw_warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int warp = hw_warp < 4 ? hw_warp + kSoftmaxWarp : hw_warp - 4;
    dm::WaitCtx wc{&s.abort_flag, p.status};
    // Every role walks the same list of work items; `t` counts the CTA's key tiles over its items, so that ring stages, buffer
    // parities and mbarrier phases run on across items.  Product unit u = 8 t + 2 group + d half: buffer u % 3, barriers u % 6.

    if (tid == 0) {
        s.abort_flag = 0;
        dm::mbar_init(&s.bar_q, 1);
        dm::mbar_init(&s.bar_q_free, 1);
        dm::mbar_init(&s.bar_s, 1);
        for (int i = 0; i < 2; ++i) {
            dm::mbar_init(&s.bar_k[i], 1);
            dm::mbar_init(&s.bar_k_free[i], 1);
            dm::mbar_init(&s.bar_v[i], 1);
            dm::mbar_init(&s.bar_pv[i], 1);
        }
        for (int i = 0; i < 2 * kBufs; ++i) dm::mbar_init(&s.bar_d[i], 1);
        dm::fence_mbar_init();
        dm::tma_prefetch_desc(&tm_q);
        dm::tma_prefetch_desc(&tm_k);
        dm::tma_prefetch_desc(&tm_v);
    }
    if (warp == 0) dm::tmem_alloc(&s.tmem_base, 512);
    dm::tc_fence_before();
    __syncthreads();
    dm::tc_fence_after();
    dm::pdl_wait();
    const uint32_t tmem = s.tmem_base;
    const uint32_t t_d = tmem + 128;                       // S: columns [0, 128); the product buffers behind it
    const uint32_t lane_base = (uint32_t)(warp & 3) * 32;

    if (warp < kFoldWarp) {
        // =============================================================== service warps
        dm::reg_dec<kRegService>();
        constexpr uint32_t kSub = kTile >> 4;
        if (warp == 0) {
            // ---- S = Q K^T of tile t, once the softmax warps have read the scores of tile t - 1
            constexpr uint32_t idesc_s = dm::idesc_e4m3(128, 128, false, false);
            const uint32_t q_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.q[0])), k_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.k[0][0]));
            int t = 0;
            for (int r = 0;; ++r) {
                const Fwd256Item w = fwd256_item(p, r);
                if (!w.valid) break;
                dm::mbar_wait(&s.bar_q, r & 1, wc);
                for (int it = 0; it < w.n_tiles; ++it, ++t) {
                    const int st = t & 1;
                    dm::mbar_wait(&s.bar_k[st], (t >> 1) & 1, wc);
                    if (t >= 1) dm::named_bar_sync(kBarSFree, kSoftmaxThreads + 32);
                    dm::tc_fence_after();
                    const uint32_t ks = k_lo + 2 * st * kSub;
                    if (dm::elect_one()) {
#pragma unroll
                        for (int hh = 0; hh < 2; ++hh) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                if ((hh | k) == 0) dm::umma_e4m3_lo<false>(tmem, q_lo, ks, idesc_s);
                                else dm::umma_e4m3_lo<true>(tmem, q_lo + hh * kSub + 2 * k, ks + hh * kSub + 2 * k, idesc_s);
                            }
                        }
                        dm::umma_commit(&s.bar_s);
                        dm::umma_commit(&s.bar_k_free[st]);
                        if (it == w.n_tiles - 1) dm::umma_commit(&s.bar_q_free);   // the item's Q tile has been read
                    }
                    __syncwarp();
                }
            }
            if (t > 0) dm::named_bar_sync(kBarSFree, kSoftmaxThreads + 32);      // the last release: no arrival is left over
        } else if (warp == 1) {
            // ---- D = C_g V_g, group by group, d half by d half, each into the buffer that was released three units ago
            constexpr uint32_t idesc_pv = dm::idesc_e4m3(128, 128, false, true);
            const uint32_t c_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.c[0])), v_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.v[0][0]));
            int t = 0, u6 = 0;
            for (int r = 0;; ++r) {
                const Fwd256Item w = fwd256_item(p, r);
                if (!w.valid) break;
                for (int it = 0; it < w.n_tiles; ++it, ++t) {
                    const int st = t & 1;
                    const uint32_t ca = c_lo + st * kSub, va = v_lo + 2 * st * kSub;
                    dm::mbar_wait(&s.bar_v[st], (t >> 1) & 1, wc);
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const int other = u6 >= kBufs ? u6 - kBufs : u6 + kBufs, buf = u6 >= kBufs ? u6 - kBufs : u6;
                        if ((u & 3) == 0) dm::named_bar_sync(kBarCodes + 2 * st + (u >> 2), kSoftmaxThreads + 32);
                        if (t > 0 || u >= kBufs) dm::named_bar_sync(kBarDFree + other, 128 + 32);
                        dm::tc_fence_after();
                        if (dm::elect_one()) {
                            dm::umma_e4m3_lo<false>(t_d + 128 * buf, ca + 2 * (u >> 1), va + (u & 1) * kSub + 256 * (u >> 1), idesc_pv);
                            dm::umma_commit(&s.bar_d[u6]);
                            if (u == 7) dm::umma_commit(&s.bar_pv[st]);    // the tile's V and codes have been read
                        }
                        __syncwarp();
                        u6 = u6 == 2 * kBufs - 1 ? 0 : u6 + 1;
                    }
                }
            }
            if (t > 0)                                     // the last releases: no arrival is left over
                for (int i = 0; i < kBufs; ++i) {
                    dm::named_bar_sync(kBarDFree + (u6 >= kBufs ? u6 - kBufs : u6 + kBufs), 128 + 32);
                    u6 = u6 == 2 * kBufs - 1 ? 0 : u6 + 1;
                }
        } else if (warp == 2) {
            // ---- TMA loads: every item's Q once the previous item's last S has read its own, and the K tiles, a stage ahead
            int t = 0;
            for (int r = 0;; ++r) {
                const Fwd256Item w = fwd256_item(p, r);
                if (!w.valid) break;
                const int q_row0 = w.hc.bh * p.N + w.I * 128, kv_row0 = w.hc.bhk * p.N;
                auto load_k = [&](int it) {
                    const int st = (t + it) & 1, row = kv_row0 + (w.n_tiles - 1 - it) * 128;
                    if (t + it >= 2) dm::mbar_wait(&s.bar_k_free[st], (((t + it) >> 1) - 1) & 1, wc);
                    if (dm::elect_one()) {
                        dm::mbar_expect_tx(&s.bar_k[st], 2 * kTile);
                        dm::tma_load_2d(s.k[st][0], &tm_k, 0, row, &s.bar_k[st]);
                        dm::tma_load_2d(s.k[st][1], &tm_k, 128, row, &s.bar_k[st]);
                    }
                    __syncwarp();
                };
                load_k(0);                                 // (its stage is free before Q's place is)
                if (r >= 1) dm::mbar_wait(&s.bar_q_free, (r - 1) & 1, wc);
                if (dm::elect_one()) {
                    dm::mbar_expect_tx(&s.bar_q, 2 * kTile);
                    dm::tma_load_2d(s.q[0], &tm_q, 0, q_row0, &s.bar_q);
                    dm::tma_load_2d(s.q[1], &tm_q, 128, q_row0, &s.bar_q);
                }
                __syncwarp();
                for (int it = 1; it < w.n_tiles; ++it) load_k(it);
                t += w.n_tiles;
            }
        } else {
            // ---- TMA loads: the V tiles, a stage ahead
            int t = 0;
            for (int r = 0;; ++r) {
                const Fwd256Item w = fwd256_item(p, r);
                if (!w.valid) break;
                const int kv_row0 = w.hc.bhk * p.N;
                for (int it = 0; it < w.n_tiles; ++it, ++t) {
                    const int st = t & 1, row = kv_row0 + (w.n_tiles - 1 - it) * 128;
                    if (t >= 2) dm::mbar_wait(&s.bar_pv[st], ((t >> 1) - 1) & 1, wc);
                    if (dm::elect_one()) {
                        dm::mbar_expect_tx(&s.bar_v[st], 2 * kTile);
                        dm::tma_load_2d(s.v[st][0], &tm_v, 0, row, &s.bar_v[st]);
                        dm::tma_load_2d(s.v[st][1], &tm_v, 128, row, &s.bar_v[st]);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp < kSoftmaxWarp) {
        // =============================================================== fold warps: thread = (row, d half)
        dm::reg_inc<kRegFold>();
        const int row = (warp & 3) * 32 + lane, half = (warp >> 2) - 1;
        const uint32_t src0 = dm::tmem_addr(t_d, lane_base, 0);
        int sl = 0, u6 = half, ph = 0;                     // ring slot of the tile's constants; the unit's barriers and their phase
        for (int r = 0;; ++r) {
            int n_tiles;                                   // all that the tile loop keeps of the item: it has no registers to spare
            {
                const Fwd256Item w = fwd256_item(p, r);
                if (!w.valid) break;
                n_tiles = w.n_tiles;
            }
            float o_acc[128];
#pragma unroll
            for (int i = 0; i < 128; ++i) o_acc[i] = 0.f;
            for (int it = 0; it < n_tiles; ++it) {
                const float* wp = reinterpret_cast<const float*>(&s.w[sl][row]);
#pragma unroll 1
                for (int grp = 0; grp < 4; ++grp) {
                    dm::mbar_wait(&s.bar_d[u6], ph, wc);   // also orders the ring slot, written before the codes
                    dm::tc_fence_after();
                    const uint32_t src = src0 + 128 * (u6 >= kBufs ? u6 - kBufs : u6);
                    // eight 16-column pieces, two in flight
                    uint32_t sa[16], sb[16];
                    dm::tmem_ld16(src, sa);
                    dm::tmem_ld16(src + 16, sb);
                    const float w = wp[grp];
                    if (grp == 0) {
                        const float alpha = s.alpha[sl][row];
                        if (__any_sync(0xffffffffu, alpha != 1.0f)) {
#pragma unroll
                            for (int i = 0; i < 128; i += 2) dm::mul2(o_acc[i], o_acc[i + 1], o_acc[i], o_acc[i + 1], alpha, alpha);
                        }
                    }
                    auto add16 = [&](int pc, const uint32_t* x) {
#pragma unroll
                        for (int i = 0; i < 16; i += 2)
                            dm::fma2(o_acc[16 * pc + i], o_acc[16 * pc + i + 1], __uint_as_float(x[i]), __uint_as_float(x[i + 1]), w,
                                     o_acc[16 * pc + i], o_acc[16 * pc + i + 1]);
                    };
#pragma unroll
                    for (int pc = 0; pc < 6; pc += 2) {
                        dm::tmem_ld_wait();
                        add16(pc, sa);
                        dm::tmem_ld16(src + 16 * pc + 32, sa);
                        add16(pc + 1, sb);
                        dm::tmem_ld16(src + 16 * pc + 48, sb);
                    }
                    dm::tmem_ld_wait();
                    dm::tc_fence_before();
                    dm::named_bar_arrive(kBarDFree + u6, 128 + 32);
                    add16(6, sa);
                    add16(7, sb);
                    u6 += 2;
                    if (u6 >= 2 * kBufs) {
                        u6 -= 2 * kBufs;
                        ph ^= 1;
                    }
                }
                if (it + 1 < n_tiles) sl = sl == kRing - 1 ? 0 : sl + 1;
            }
            // ---- the item's epilogue
            int r_again = r;
            asm volatile("" : "+r"(r_again));
            const Fwd256Item w = fwd256_item(p, r_again);
            const float2 ml = s.ml[sl][row];
            const float l = ml.y;
            const bool dead = (l == 0.f) || (l != l);
            const float inv = dead ? 0.f : 1.0f / l;
            if (half == 0) p.lse[(int64_t)w.hc.bh * p.N + w.I * 128 + row] = dead ? -INFINITY : ml.x + logf(l);
            sl = sl == kRing - 1 ? 0 : sl + 1;
            // the bf16 rows leave through the warp's own staging slice, 32 columns at a time: eight whole 64-byte pieces per instruction
            uint8_t* stg = s.stg[warp - kFoldWarp];
            uint8_t* obase = reinterpret_cast<uint8_t*>(p.o + (((int64_t)w.hc.b * p.N + w.I * 128 + (warp & 3) * 32) * p.H + w.hc.h) * 256) + 256 * half;
            const int64_t row_bytes = (int64_t)p.H * 512;
            auto chunk = [&](int rr, int c) { return stg + rr * 64 + ((c ^ ((rr >> 1) & 3)) << 4); };
#pragma unroll
            for (int h = 0; h < 4; ++h) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t w4[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int i = 32 * h + 8 * c + 2 * e;
                        __nv_bfloat162 tt = __floats2bfloat162_rn(o_acc[i] * inv, o_acc[i + 1] * inv);
                        w4[e] = *reinterpret_cast<uint32_t*>(&tt);
                    }
                    *reinterpret_cast<uint4*>(chunk(lane, c)) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int rr = 8 * i + (lane >> 2);
                    const uint4 val = *reinterpret_cast<const uint4*>(chunk(rr, lane & 3));
                    *reinterpret_cast<uint4*>(obase + rr * row_bytes + 64 * h + ((lane & 3) << 4)) = val;
                }
                __syncwarp();
            }
        }
    } else {
        // =============================================================== softmax warps: thread = row, all four P groups
        dm::reg_dec<kRegSoftmax>();
        const int row = (warp & 3) * 32 + lane;            // query row inside the block = tensor-memory lane
        const uint32_t t_s = dm::tmem_addr(tmem, lane_base, 0);
        const uint32_t c_row = dm::smem_u32(s.c[0]) + row * 128;
        int t = 0, sl = 0;
        // What an item's first tile needs from global memory is read one item ahead, a tile's K scales one tile ahead: read in place they
        // would be exposed loads.  The four scales of a tile are read one by one: a caller's scale tensor may start at any multiple of 4 bytes.
        auto scales4 = [](const float* at) { return make_float4(at[0], at[1], at[2], at[3]); };
        float q8sc_nx = 0.f;
        float4 ks_nx = make_float4(0.f, 0.f, 0.f, 0.f);
        auto first_scales = [&](const Fwd256Item& wi) {
            if (!wi.valid) return;
            q8sc_nx = p.q8s[(int64_t)wi.hc.bh * (p.N / 64) + 2 * wi.I + (row >> 6)];
            ks_nx = scales4(p.k8s + (int64_t)wi.hc.bhk * (p.N / 32) + 4 * (wi.n_tiles - 1));
        };
        Fwd256Item w = fwd256_item(p, 0);
        first_scales(w);
        for (int r = 0; w.valid; ++r) {
            const int n_tiles = w.n_tiles, I = w.I;
            const float q8sc = q8sc_nx;
            const float* ksp = p.k8s + (int64_t)w.hc.bhk * (p.N / 32);
            const float* vsp = p.v8s + (int64_t)w.hc.bhk * (p.N / 32);
            float m_run = -INFINITY, l0 = 0.f, l1 = 0.f;   // the running maximum, the denominator's part per 64-key half
            float4 ks_n = ks_nx;
            w = fwd256_item(p, r + 1);
            first_scales(w);
            for (int it = 0; it < n_tiles; ++it, ++t, sl = sl == kRing - 1 ? 0 : sl + 1) {
                const int j = n_tiles - 1 - it;
                const float dsc[4] = {q8sc * ks_n.x, q8sc * ks_n.y, q8sc * ks_n.z, q8sc * ks_n.w};
                const float4 vs4 = scales4(vsp + 4 * j);
                if (it + 1 < n_tiles) ks_n = scales4(ksp + 4 * (j - 1));
                const bool diag = p.causal && j == I;

                dm::mbar_wait(&s.bar_s, t & 1, wc);
                dm::tc_fence_after();
                float sa[32], sb[32];
                auto load = [&](int gg, float* sv) { dm::tmem_ld32(t_s + 32 * gg, reinterpret_cast<uint32_t*>(sv)); };
                auto mask = [&](int gg, float* sv) {       // the diagonal tile only, where the 32 keys lie on or above the warp's 32 rows
                    if (diag && gg >= (warp & 3)) {
                        const int last = gg == (warp & 3) ? lane : -1;
#pragma unroll
                        for (int c = 0; c < 32; ++c)
                            if (c > last) sv[c] = -INFINITY;
                    }
                };
                // ---- the groups' maxima.  Groups 0 and 1 stay in registers, the last two are read again.
                float gm[4];
                auto maximum = [&](int gg, const float* sv) {
                    float m0 = fmaxf(sv[0], sv[1]), m1 = fmaxf(sv[2], sv[3]);
#pragma unroll
                    for (int c = 4; c < 32; c += 4) {
                        m0 = dm::fmax3(m0, sv[c], sv[c + 1]);
                        m1 = dm::fmax3(m1, sv[c + 2], sv[c + 3]);
                    }
                    gm[gg] = fmaxf(m0, m1) * dsc[gg];
                };
#pragma unroll
                for (int gg = 2; gg >= 0; gg -= 2) {
                    load(gg, sa);
                    load(gg + 1, sb);
                    dm::tmem_ld_wait();
                    mask(gg, sa);
                    mask(gg + 1, sb);
                    maximum(gg, sa);
                    maximum(gg + 1, sb);
                }
                const float m_new = fmaxf(m_run, fmaxf(fmaxf(gm[0], gm[1]), fmaxf(gm[2], gm[3])));
                const float m_cur = (m_new == -INFINITY) ? 0.f : m_new;
                const float alpha = dm::ex2((m_run - m_cur) * dm::kLog2e);
                m_run = m_new;
                // ---- codes and the denominator.  The products of tile t - 2 are complete: its codes may be overwritten, and the constants of tile
                // t - 3 (whose folds were over before the last products of tile t - 2 were issued).
                if (t >= 2) dm::mbar_wait(&s.bar_pv[t & 1], ((t - 2) >> 1) & 1, wc);
                const uint32_t c_at = c_row + (t & 1) * kTile;
                float wgt[4];
                auto codes32 = [&](int gg, const float* sv, float& lacc) {
                    const float ms = fmaxf(gm[gg] * dm::kLog2e, fmaf(m_cur, dm::kLog2e, -dm::kPhatFloorB)) - dm::kLog2_448;
                    const float dl2 = dsc[gg] * dm::kLog2e;
                    float acc[4] = {0.f, 0.f, 0.f, 0.f};
                    const float nms = -ms;
#pragma unroll
                    for (int c = 0; c < 32; c += 16) {
                        uint32_t codes[4];
#pragma unroll
                        for (int e = 0; e < 16; e += 4) {
                            float x0, x1, x2, x3;
                            dm::fma2(x0, x1, sv[c + e], sv[c + e + 1], dl2, nms, nms);
                            dm::fma2(x2, x3, sv[c + e + 2], sv[c + e + 3], dl2, nms, nms);
                            const float p0 = dm::ex2(x0), p1 = dm::ex2(x1), p2 = dm::ex2(x2), p3 = dm::ex2(x3);
                            dm::add2(acc[0], acc[1], p0, p1);
                            dm::add2(acc[2], acc[3], p2, p3);
                            codes[e >> 2] = dm::cvt_e4m3x4(p0, p1, p2, p3);
                        }
                        // 16 codes = one 16-byte chunk of the row's swizzled 128 bytes (eight rows of a store phase: eight chunks)
                        const uint32_t at = c_at + (((2 * gg + (c >> 4)) ^ (lane & 7)) << 4);
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(codes[0]), "r"(codes[1]), "r"(codes[2]), "r"(codes[3])
                                     : "memory");
                    }
                    const float sigma = dm::ex2(fmaf(-m_cur, dm::kLog2e, ms));
                    lacc = fmaf(sigma, (acc[0] + acc[1]) + (acc[2] + acc[3]), lacc);
                    wgt[gg] = (gg == 0 ? vs4.x : gg == 1 ? vs4.y : gg == 2 ? vs4.z : vs4.w) * sigma;
                };
                float lacc0 = 0.f, lacc1 = 0.f;
                codes32(0, sa, lacc0);
                load(2, sa);
                codes32(1, sb, lacc0);
                load(3, sb);
                l0 = fmaf(l0, alpha, lacc0);
                *reinterpret_cast<float2*>(&s.w[sl][row]) = make_float2(wgt[0], wgt[1]);
                s.alpha[sl][row] = alpha;
                dm::fence_proxy_async_smem();
                dm::named_bar_arrive(kBarCodes + 2 * (t & 1), kSoftmaxThreads + 32);
                dm::tmem_ld_wait();
                dm::tc_fence_before();
                dm::named_bar_arrive(kBarSFree, kSoftmaxThreads + 32);      // S may be overwritten
                mask(2, sa);
                codes32(2, sa, lacc1);
                mask(3, sb);
                codes32(3, sb, lacc1);
                l1 = fmaf(l1, alpha, lacc1);
                *(reinterpret_cast<float2*>(&s.w[sl][row]) + 1) = make_float2(wgt[2], wgt[3]);
                if (it == n_tiles - 1) s.ml[sl][row] = make_float2(m_run, l0 + l1);
                dm::fence_proxy_async_smem();
                dm::named_bar_arrive(kBarCodes + 2 * (t & 1) + 1, kSoftmaxThreads + 32);
            }
        }
    }
    dm::tc_fence_before();
    __syncthreads();
    if (warp == 0) dm::tmem_dealloc(tmem, 512);
}

}  // namespace

namespace dmh {
constexpr int kFwd256RegPool = kSoftmaxThreads * kRegSoftmax + kFoldThreads * kRegFold + 128 * kRegService;
static_assert(kFwd256RegPool == kThreads * 128, "the roles' register requests must add up to the launch pool");

int prepare_fwd256(char* err, size_t errlen) {
    static DeviceOnce once;
    return device_once(once, err, errlen, [&]() -> int {
        DM_CUDA(cudaFuncSetAttribute(fwd_d256_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Fwd256Smem) + 1024));
        return check_register_pool((const void*)fwd_d256_kernel, kThreads, kFwd256RegPool, err, errlen);
    });
}

int launch_fwd_d256(const void* q8, const void* k8, const void* v8, const float* q8s, const float* k8s, const float* v8s, DmShape sh,
                    int h0, int hcount, void* o, float* lse, void* stream, char* err, size_t errlen) {
    int rc;
    CUtensorMap tq, tk, tv;
    if ((rc = make_tmap_u8(&tq, q8, 256, (uint64_t)sh.B * sh.H * sh.N, 128, err, errlen))) return rc;
    if ((rc = make_tmap_u8(&tk, k8, 256, (uint64_t)sh.B * sh.Hk * sh.N, 128, err, errlen))) return rc;
    if ((rc = make_tmap_u8(&tv, v8, 256, (uint64_t)sh.B * sh.Hk * sh.N, 128, err, errlen))) return rc;
    int* status = device_status_word(err, errlen);
    if (!status) return DM_ERR_CUDA;
    Fwd256Params p{q8s, k8s, v8s, static_cast<__nv_bfloat16*>(o), lse, sh.H, sh.Hk, sh.N, h0, hcount, sh.causal, status,
                   sh.B * hcount, dm::make_fastdiv(sh.B * hcount), dm::make_fastdiv(hcount), dm::make_fastdiv(sh.H / sh.Hk)};
    if ((rc = prepare_fwd256(err, errlen))) return rc;
    int sms = 0;
    if ((rc = sm_count(&sms, err, errlen))) return rc;
    // persistent: one CTA per SM walks the (head, row block) items, heaviest first
    const int64_t items = (int64_t)sh.B * hcount * (sh.N / 128);
    const int grid = (int)(items < sms ? items : sms);
    DM_CUDA(launch_pdl(fwd_d256_kernel, grid, kThreads, sizeof(Fwd256Smem) + 1024, stream, tq, tk, tv, p));
    return DM_OK;
}
}  // namespace dmh
