// Forward kernel, head_dim 128: O and LSE from e4m3 Q / K / V codes and their block scales, with the reference's
// faithful P basis (per row, per 64-key group) -- csrc/softmax_fq8f.h and csrc/mainloop_fwd_sm90_fp8f.hpp of the
// reference, restated for tcgen05.
//
// One work item = 128 query rows of one (batch, head); the kernel is persistent, one CTA per SM walks a list of items, and since
// every role keeps its own place in the list, the loads and S of the next item start while the current one is finished.  896 threads:
//   warps 0..15   softmax, two teams of eight on alternating key tiles: thread = (row, 64-key group of its team's tiles)
//   warps 16..23  fold: thread = (row, 64 of O's 128 columns); they own O, the LSE and nothing else
//   warps 24..27  service (converged loops, one elected lane issues): S; the products of key group 0; of key group 1; the TMA loads
// Key tiles of 128 keys (two 64-key groups) are visited from the diagonal tile downwards.  Per tile:
//   S = Q K^T            4 x tcgen05.mma (M128 N128 K32) into the tensor-memory buffer of the tile's parity, i.e. of its team
//   softmax              basis ms_g = max(gm_g*l2, m*l2 - 12) - log2(448) (gm: the group's maximum in this tile, m: the thread's own
//                        running one), codes = e4m3(2^(S*l2 - ms_g)) written back into tensor memory over the scores they came from
//                        (four codes per column, lane = row).  ms_g, gm_g and the sum of the unrounded p go to a ring; nothing is
//                        exchanged between softmax threads
//   D_g = C_g V_g        2 x tcgen05.mma per group (A = the codes in tensor memory, B = the V tile) into zero-initialised
//                        tensor-memory temporaries, issued when the codes are stored and the previous product has been read
//   fold                 the row's softmax in tile order: M = max(M, gm_0, gm_1), alpha = 2^((M_before - M)*l2), s_g = 2^(ms_g - M*l2),
//                        l_g = l_g alpha + s_g sum_g, O = O alpha + D_0 (v8sc_0 s_0) + D_1 (v8sc_1 s_1); O / (l_0 + l_1) at the end
// K / V tiles arrive by TMA into a 3-stage ring.  Every mbarrier wait is bounded.
//
// Why this shape.  A 128 x 128 tile holds 1024 clocks of exponentials and 512 of MMAs; with one set of softmax warps the wait for
// S, the maxima, the exchange of the running maximum and the codes (about 1200 clocks a tile) ran with the exponential unit idle.  Two
// teams half a tile apart overlap them, which needs the running maximum handed from tile to tile gone from the softmax warps (a serial
// chain through both teams: measured slower than one set).  It lives in the fold warps, which see the tiles in order: a running
// maximum of the softmax thread's own only lowers the 12-binade floor of a group's basis (never the precision of its codes).
// Why O and l are kept against the row's maximum of the moment and not in a basis that moves only now and then: in a row of few keys
// O is a code times a V scale, and where the scale has few significant bits (the block's maximum / 448, a maximum whose significand is a
// multiple of 7) up to half of these products lie exactly half way between two bf16 values: the last bit of a weight decides dozens of
// elements of O at once, and through rowsum(dO * O) a visible part of the row's dQ.  Both forms are equally accurate; this one
// rounds as a plain row softmax does, and it costs nothing: the softmax warps lose their share of the denominator and the fold its
// epilogue, which pays for the multiplications of O (lazy basis -> this, us: B4 N4096 H32 causal 508 -> 506, B1 N16384 H32
// 1788 -> 1792, B2 N2048 H16 49.2 -> 47.2, B4 N768 H12 22.5 -> 20.6, B64 N256 H16 59.5 -> 53.3).
// What bounds it: the issue rate more than any pipe (ncu at B1 N4096 H32 causal: issue slots 70 % active, MUFU 54 %, tensor pipe 26 %).  Of
// the lazy form's 531 us at B4 N4096 H32 (on a slower clock) 526 were left without the exponentials, 508 without three quarters of the
// fold's loads and 497 without the second read of the scores.
#include "dm_attn_common.cuh"
#include "dm_host.h"

namespace {

constexpr int kTile = 128 * 128;   // bytes of one e4m3 tile (128 rows x 128 bytes)
constexpr int kStages = 3;
constexpr int kThreads = 896;
constexpr int kSoftmaxThreads = 512;
constexpr int kFoldWarp = 16, kServiceWarp = 24;
constexpr int kRegSoftmax = 64, kRegFold = 104, kRegService = 40;      // per thread after setmaxnreg; the sum is the launch pool
// Named barriers (a warp-to-warp hand-off costs a quarter of an mbarrier's; an arriving side is never a whole round ahead, because
// its next arrival on the same barrier needs a product that is issued behind the synchronising side's).
constexpr int kBarCodes = 1;       // + 2 * team + key group: the group's codes are in tensor memory     128 + 32
constexpr int kBarDFree = 5;       // + key group: the fold warps hold the group's product              256 + 32
constexpr int kRing = 4;           // depth of the per-tile row-constant ring between softmax and fold warps

struct FwdSmem {
    alignas(1024) uint8_t q[2][kTile];             // by work item parity: the next item's Q arrives under this item's tail
    alignas(1024) uint8_t k[kStages][kTile];
    alignas(1024) uint8_t v[kStages][kTile];
    float ms[kRing][2][128];          // [tile % kRing][key group][row]: the basis of the row's codes, log2 units
    float2 gp[kRing][2][128];         // the group's maximum and the sum of its exponentials against ms
    float vs[kRing][2];               // the group's V scale
    alignas(16) uint8_t stg[8][32 * 128];   // per fold warp: its 32 bf16 half rows of O on their way out (16-byte chunks XOR-swizzled by the row)
    uint64_t bar_q[2], bar_q_free[2], bar_kv[kStages], bar_kv_free[kStages], bar_s_full[2], bar_d_full[2][2];   // bar_d_full: [tile parity][key group]
    uint32_t tmem_base;
    int abort_flag;
};

struct FwdParams {
    const float* q8s;
    const float* k8s;
    const float* v8s;
    __nv_bfloat16* o;
    float* lse;
    int H, Hk, N, h0, hcount, causal;
    int* status;
    dm::RowMap rm;
    int n_heads;                      // B * hcount: work items are (head, row block), heaviest row blocks first
    dm::FastDiv fd_heads, fd_hcount, fd_rep;   // divisions by n_heads, hcount and H / Hk
};

// One work item of a persistent CTA.  Items are numbered rank-major (rank 0 = the row blocks with the most key tiles, all
// heads, then rank 1, ...) and walked as dm::walk_index says.
struct FwdItem {
    dm::HeadCoord hc;
    int li, I, n_tiles;
    bool valid;
};
template <class Walk>
__device__ __forceinline__ FwdItem fwd_item(const FwdParams& p, const Walk& walk, int round) {
    FwdItem w;
    const int nq_blk = p.rm.nq / 128;
    const int idx = dm::walk_index(walk, round);
    w.valid = idx < p.n_heads * nq_blk;
    const int rank = (int)dm::fdiv((uint32_t)idx, p.fd_heads);
    w.hc = dm::head_coord(idx - rank * p.n_heads, p.h0, p.fd_hcount, p.H, p.Hk, p.fd_rep);
    w.li = nq_blk - 1 - rank;
    w.I = dm::global_block(p.rm, w.li);
    w.n_tiles = p.causal ? w.I + 1 : p.N / 128;
    return w;
}

template <class Walk>
__global__ void __launch_bounds__(kThreads, 1)
fwd_d128_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const FwdParams p, const __grid_constant__ Walk walk) {
    extern __shared__ uint8_t smem_raw[];
    FwdSmem& s = *reinterpret_cast<FwdSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int nq_blk = p.rm.nq / 128;
    dm::WaitCtx wc{&s.abort_flag, p.status};
    // Every role walks the same list of work items; `gt` counts the key tiles of the items before the current one, so
    // that ring stages, buffer parities and mbarrier phases run on across items (t = gt + it below).

    if (tid == 0) {
        s.abort_flag = 0;
        for (int i = 0; i < kStages; ++i) {
            dm::mbar_init(&s.bar_kv[i], 1);
            dm::mbar_init(&s.bar_kv_free[i], 2);
        }
        for (int i = 0; i < 2; ++i) {
            dm::mbar_init(&s.bar_s_full[i], 1);
            dm::mbar_init(&s.bar_d_full[i][0], 1);
            dm::mbar_init(&s.bar_d_full[i][1], 1);
            dm::mbar_init(&s.bar_q[i], 1);
            dm::mbar_init(&s.bar_q_free[i], 1);
        }
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
    const uint32_t t_d0 = tmem + 256, t_d1 = tmem + 384;      // S buffers at columns [0, 128) and [128, 256)
    const uint32_t lane_base = (uint32_t)(warp & 3) * 32;

    if (warp >= kServiceWarp) {
        // =============================================================== service warps
        dm::reg_dec<kRegService>();
        constexpr uint32_t kSub = kTile >> 4;
        if (warp == kServiceWarp) {
            // ---- S = Q K^T of tile t into buffer t & 1, once the products of tile t - 2 are complete: they read their codes from
            // that buffer, and their codes came after the softmax warps had read its scores.
            constexpr uint32_t idesc_s = dm::idesc_e4m3(128, 128, false, false);
            const uint32_t q_lo0 = dm::smem_desc_lo_sw128(dm::smem_u32(s.q[0])), k_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.k[0]));
            int gt = 0;
            for (int r = 0;; ++r) {
                const FwdItem w = fwd_item(p, walk, r);
                if (!w.valid) break;
                const int qb = r & 1;
                const uint32_t q_lo = q_lo0 + qb * kSub;
                dm::mbar_wait(&s.bar_q[qb], (r >> 1) & 1, wc);
                for (int it = 0; it < w.n_tiles; ++it) {
                    const int t = gt + it, st = t % kStages, b = t & 1;
                    dm::mbar_wait(&s.bar_kv[st], (t / kStages) & 1, wc);
                    if (t >= 2) {
                        dm::mbar_wait(&s.bar_d_full[b][0], ((t - 2) >> 1) & 1, wc);
                        dm::mbar_wait(&s.bar_d_full[b][1], ((t - 2) >> 1) & 1, wc);
                    }
                    dm::tc_fence_after();
                    const uint32_t ks = k_lo + st * kSub, ts = tmem + b * 128;
                    if (dm::elect_one()) {
                        dm::umma_e4m3_lo<false>(ts, q_lo, ks, idesc_s);
#pragma unroll
                        for (int k = 1; k < 4; ++k) dm::umma_e4m3_lo<true>(ts, q_lo + 2 * k, ks + 2 * k, idesc_s);
                        dm::umma_commit(&s.bar_s_full[b]);
                        if (it == w.n_tiles - 1) dm::umma_commit(&s.bar_q_free[qb]);   // the item's Q tile has been read
                    }
                    __syncwarp();
                }
                gt += w.n_tiles;
            }
        } else if (warp <= kServiceWarp + 2) {
            // ---- D_g = C_g V_g, one warp per key group, once the group's codes are in tensor memory and the fold warps hold its product
            // of the tile before
            const int g = warp - kServiceWarp - 1;
            constexpr uint32_t idesc_pv = dm::idesc_e4m3(128, 128, false, true);
            const uint32_t v_lo = dm::smem_desc_lo_sw128(dm::smem_u32(s.v[0])) + 512 * g;      // V rows of the group (MN-major: 32 rows = +256)
            const uint32_t t_d = g ? t_d1 : t_d0;
            int t = 0, st = 0;
            for (int r = 0;; ++r) {
                const FwdItem w = fwd_item(p, walk, r);
                if (!w.valid) break;
                for (int it = 0; it < w.n_tiles; ++it, ++t) {
                    const int b = t & 1;
                    const uint32_t pa = tmem + b * 128 + 64 * g, va = v_lo + st * kSub;     // codes: columns [64 g, 64 g + 16) of S buffer b
                    if (t >= 1) dm::named_bar_sync(kBarDFree + g, 256 + 32);
                    dm::named_bar_sync(kBarCodes + 2 * b + g, 128 + 32);       // (V came with the K that S was made of)
                    dm::tc_fence_after();
                    if (dm::elect_one()) {
                        dm::umma_e4m3_ts<false>(t_d, pa, va, idesc_pv);
                        dm::umma_e4m3_ts<true>(t_d, pa + 8, va + 256, idesc_pv);
                        dm::umma_commit(&s.bar_d_full[b][g]);
                        dm::umma_commit(&s.bar_kv_free[st]);       // K was read by S long ago, V just now
                    }
                    __syncwarp();
                    if (++st == kStages) st = 0;
                }
            }
            if (t > 0) dm::named_bar_sync(kBarDFree + g, 256 + 32);      // the last release: no arrival is left over
        } else {
            // ---- TMA loads: every item's Q, then its K / V tiles, as far ahead as the rings allow (across items too)
            int gt = 0;
            for (int r = 0;; ++r) {
                const FwdItem w = fwd_item(p, walk, r);
                if (!w.valid) break;
                const int qb = r & 1;
                const int q_row0 = w.hc.bh * p.rm.nq + w.li * 128, kv_row0 = w.hc.bhk * p.N;
                if (r >= 2) dm::mbar_wait(&s.bar_q_free[qb], ((r - 2) >> 1) & 1, wc);
                if (dm::elect_one()) {
                    dm::mbar_expect_tx(&s.bar_q[qb], kTile);
                    dm::tma_load_2d(s.q[qb], &tm_q, 0, q_row0, &s.bar_q[qb]);
                }
                for (int it = 0; it < w.n_tiles; ++it) {
                    const int t = gt + it, st = t % kStages, j = w.n_tiles - 1 - it;
                    if (t >= kStages) dm::mbar_wait(&s.bar_kv_free[st], (t / kStages - 1) & 1, wc);
                    if (dm::elect_one()) {
                        dm::mbar_expect_tx(&s.bar_kv[st], 2 * kTile);
                        dm::tma_load_2d(s.k[st], &tm_k, 0, kv_row0 + j * 128, &s.bar_kv[st]);
                        dm::tma_load_2d(s.v[st], &tm_v, 0, kv_row0 + j * 128, &s.bar_kv[st]);
                    }
                    __syncwarp();
                }
                gt += w.n_tiles;
            }
        }
    } else if (warp >= kFoldWarp) {
        // =============================================================== fold warps: thread = (row, 64 of O's 128 columns)
        dm::reg_inc<kRegFold>();
        const int row = (warp & 3) * 32 + lane, half = (warp >> 2) & 1;
        const uint32_t src = dm::tmem_addr(t_d0, lane_base, 64 * half);      // group 1's products: + 128
        int gt = 0;
        for (int r = 0;; ++r) {
            int n_tiles;                               // all that the tile loop keeps of the item: it has no registers to spare
            {
                const FwdItem w = fwd_item(p, walk, r);
                if (!w.valid) break;
                n_tiles = w.n_tiles;
            }
            float o_acc[64];
#pragma unroll
            for (int i = 0; i < 64; ++i) o_acc[i] = 0.f;
            float m_run = -INFINITY, l0 = 0.f, l1 = 0.f;        // the row's running maximum, the denominator's part per key group
            for (int it = 0; it < n_tiles; ++it) {
                const int t = gt + it, b = t & 1, rg = t % kRing;
                dm::mbar_wait(&s.bar_d_full[b][0], (t >> 1) & 1, wc);      // also order the ring slot, written before the codes
                dm::mbar_wait(&s.bar_d_full[b][1], (t >> 1) & 1, wc);
                dm::tc_fence_after();
                // sixteen 8-column pieces, two in flight (16-column pieces spill beside the 64 accumulators: 1904 against 1832 us at
                // B1 N16384 H32); the first pair arrives while the weights are worked out, and group 1's under group 0's last additions
                uint32_t sa[8], sb[8];
                auto ld8 = [&](int pc, uint32_t* x) { dm::tmem_ld8(src + 8 * pc, x); };
                ld8(0, sa);
                ld8(1, sb);
                float w0, w1;
                {
                    const float2 g0 = s.gp[rg][0][row], g1 = s.gp[rg][1][row];
                    const float m_new = fmaxf(m_run, fmaxf(g0.x, g1.x));
                    const float m_cur = (m_new == -INFINITY) ? 0.f : m_new;
                    const float alpha = dm::ex2((m_run - m_cur) * dm::kLog2e);
                    // M * l2 is not rounded on its own here (fma): the weight is the power of two of the basis' true distance
                    const float s0 = dm::ex2(fmaf(-m_cur, dm::kLog2e, s.ms[rg][0][row]));
                    const float s1 = dm::ex2(fmaf(-m_cur, dm::kLog2e, s.ms[rg][1][row]));
                    l0 = fmaf(l0, alpha, __fmul_rn(s0, g0.y));
                    l1 = fmaf(l1, alpha, __fmul_rn(s1, g1.y));
                    w0 = s.vs[rg][0] * s0;
                    w1 = s.vs[rg][1] * s1;
                    m_run = m_new;
                    if (__any_sync(0xffffffffu, alpha != 1.0f)) {
#pragma unroll
                        for (int i = 0; i < 64; i += 2) dm::mul2(o_acc[i], o_acc[i + 1], o_acc[i], o_acc[i + 1], alpha, alpha);
                    }
                }
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    const float wg = g ? w1 : w0;
                    auto add8 = [&](int pc, const uint32_t* x) {
#pragma unroll
                        for (int i = 0; i < 8; i += 2)
                            dm::fma2(o_acc[8 * pc + i], o_acc[8 * pc + i + 1], __uint_as_float(x[i]), __uint_as_float(x[i + 1]), wg,
                                     o_acc[8 * pc + i], o_acc[8 * pc + i + 1]);
                    };
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        dm::tmem_ld_wait();
                        add8(2 * q, sa);
                        ld8(16 * g + 2 * q + 2, sa);
                        add8(2 * q + 1, sb);
                        ld8(16 * g + 2 * q + 3, sb);
                    }
                    dm::tmem_ld_wait();
                    dm::tc_fence_before();
                    dm::named_bar_arrive(kBarDFree + g, 256 + 32);
                    add8(6, sa);
                    if (g == 0) ld8(16, sa);
                    add8(7, sb);
                    if (g == 0) ld8(17, sb);
                }
            }
            gt += n_tiles;
            int r_again = r;
            asm volatile("" : "+r"(r_again));
            const FwdItem w = fwd_item(p, walk, r_again);
            // ---- the item's epilogue
            const float l = l0 + l1;
            const bool dead = (l == 0.f) || (l != l);
            const float inv = dead ? 0.f : 1.0f / l;
            if (half == 0) p.lse[(int64_t)w.hc.bh * p.rm.nq + w.li * 128 + row] = dead ? -INFINITY : m_run + logf(l);
            // The bf16 half rows leave through shared memory: stored directly every 16-byte store instruction would touch 32 different
            // rows; from the warp's staging slice each instruction writes four whole 128-byte half rows.  A warp's slice is its own, so
            // the hand-over needs no more than the warp.
            uint8_t* stg = s.stg[warp & 7];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                uint32_t w4[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    __nv_bfloat162 tt = __floats2bfloat162_rn(o_acc[8 * c + 2 * e] * inv, o_acc[8 * c + 2 * e + 1] * inv);
                    w4[e] = *reinterpret_cast<uint32_t*>(&tt);
                }
                *reinterpret_cast<uint4*>(stg + lane * 128 + ((c ^ (lane & 7)) << 4)) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
            }
            __syncwarp();
            {
                const int row0 = w.li * 128 + (warp & 3) * 32;          // first of the warp's rows inside the (local) Q-side tensors
                uint8_t* obase = reinterpret_cast<uint8_t*>(p.o + (((int64_t)w.hc.b * p.rm.nq + row0) * p.H + w.hc.h) * 128) + 128 * half;
                const int64_t row_bytes = (int64_t)p.H * 128 * 2;
                const int j = lane & 7;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int rr = 4 * i + (lane >> 3);
                    const uint4 val = *reinterpret_cast<const uint4*>(stg + rr * 128 + ((j ^ (rr & 7)) << 4));
                    *reinterpret_cast<uint4*>(obase + rr * row_bytes + (j << 4)) = val;
                }
            }
            __syncwarp();                                  // the slice may take the next item's rows
        }
    } else {
        // =============================================================== softmax warps
        dm::reg_dec<kRegSoftmax>();
        const int team = warp >> 3, g = (warp >> 2) & 1;      // parity of the tiles (= the S buffer), 64-key group of the tile
        const int row = (warp & 3) * 32 + lane;   // query row inside the block = tensor-memory lane
        const uint32_t t_s = dm::tmem_addr(tmem + team * 128, lane_base, g * 64);
        int gt = 0;
        // What an item's first tile needs from global memory is read one item ahead: read at the item's start it would be three
        // exposed loads.
        float q8sc_nx = 0.f, ks_nx = 0.f, vs_nx = 0.f;
        auto first_scales = [&](const FwdItem& wi, int gt_at) {
            if (!wi.valid) return;
            q8sc_nx = p.q8s[(int64_t)wi.hc.bh * nq_blk + wi.li];
            const int first = (gt_at ^ team) & 1;
            if (first < wi.n_tiles) {
                const int64_t ko = (int64_t)wi.hc.bhk * (p.N / 64) + g + 2 * (wi.n_tiles - 1 - first);
                ks_nx = p.k8s[ko];
                vs_nx = p.v8s[ko];
            }
        };
        FwdItem w = fwd_item(p, walk, 0);
        first_scales(w, 0);
        for (int r = 0; w.valid; ++r) {
            const int n_tiles = w.n_tiles, I = w.I;
            const float q8sc = q8sc_nx;
            const float* ksp = p.k8s + (int64_t)w.hc.bhk * (p.N / 64) + g;
            const float* vsp = p.v8s + (int64_t)w.hc.bhk * (p.N / 64) + g;
            // The thread's own running maximum (its group, its team's tiles): it only places the floor of the basis, 12 binades below it.
            float m_run = -INFINITY;
            float ks_n = ks_nx, vs_n = vs_nx;
            w = fwd_item(p, walk, r + 1);
            first_scales(w, gt + n_tiles);
            for (int it = (gt ^ team) & 1; it < n_tiles; it += 2) {
                const int t = gt + it, j = n_tiles - 1 - it, rg = t % kRing;
                const float ks = ks_n, vs = vs_n;
                if (it + 2 < n_tiles) {
                    ks_n = ksp[2 * (j - 2)];
                    vs_n = vsp[2 * (j - 2)];
                }
                // The group maximum is taken on the raw products: the group's scale is positive, so scaling the maximum gives the
                // maximum of the scaled scores bit for bit, and the scores themselves are scaled inside the exponent's one
                // multiply-add below (x = raw * (dsc * log2 e) - ms).  The scale is kept a normal number (it underflows only when a Q
                // block and a K group are both all zero, where every product is zero anyway), so that a masked -inf stays -inf.
                const float dsc = fmaxf(q8sc * ks, 1.2e-38f);
                const bool diag = p.causal && j == I;

                // ---- S for this thread's (row, key group): 64 fp32 values, 32 at a time.  The first half stays in registers from its
                // maximum to its codes, the second is read again.
                dm::mbar_wait(&s.bar_s_full[team], (t >> 1) & 1, wc);
                dm::tc_fence_after();
                float sv[32];
                float m0 = -INFINITY, m1 = -INFINITY;
                auto load = [&](int h) {
                    dm::tmem_ld32(t_s + 32 * h, reinterpret_cast<uint32_t*>(sv));
                    dm::tmem_ld_wait();
                    // The mask: only where the 32 keys lie on or above the warp's 32 rows (10 of a diagonal tile's 16 pieces), against a
                    // limit that is worked out once (502 -> 495 us at B4 N4096 H32).
                    if (diag && 2 * g + h >= (warp & 3)) {
                        const int last = 2 * g + h == (warp & 3) ? lane : -1;
#pragma unroll
                        for (int c = 0; c < 32; ++c)
                            if (c > last) sv[c] = -INFINITY;
                    }
                };
#pragma unroll
                for (int h = 1; h >= 0; --h) {
                    load(h);
#pragma unroll
                    for (int c = 0; c < 32; c += 4) {
                        m0 = dm::fmax3(m0, sv[c], sv[c + 1]);
                        m1 = dm::fmax3(m1, sv[c + 2], sv[c + 3]);
                    }
                }
                const float gm = fmaxf(m0, m1) * dsc;
                m_run = fmaxf(m_run, gm);
                const bool some = m_run != -INFINITY;              // a key has been visible
                const float ms = fmaxf(gm * dm::kLog2e, (some ? m_run * dm::kLog2e : 0.f) - dm::kPhatFloorB) - dm::kLog2_448;
                // the ring slot of tile t - kRing has been read: its fold released the group's product before the product of tile t - 3,
                // and S of this tile waited for the product of tile t - 2.  A group without a visible key weighs nothing (2^-inf).
                s.ms[rg][g][row] = some ? ms : -INFINITY;
                if (lane == 0) s.vs[rg][g] = vs;
                float part0 = 0.f, part1 = 0.f;
                uint32_t codes[16];
                const float nms = -ms, cl = __fmul_rn(dsc, dm::kLog2e);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (h == 1) load(1);
#pragma unroll
                    for (int c = 0; c < 32; c += 4) {
                        float x0, x1, x2, x3;
                        dm::fma2(x0, x1, sv[c], sv[c + 1], cl, nms, nms);
                        dm::fma2(x2, x3, sv[c + 2], sv[c + 3], cl, nms, nms);
                        const float p0 = dm::ex2(x0), p1 = dm::ex2(x1), p2 = dm::ex2(x2), p3 = dm::ex2(x3);
                        dm::add2(part0, part1, p0, p1);
                        dm::add2(part0, part1, p2, p3);
                        codes[8 * h + (c >> 2)] = dm::cvt_e4m3x4(p0, p1, p2, p3);
                    }
                }
                s.gp[rg][g][row] = make_float2(gm, part0 + part1);
                // the codes go back into tensor memory, over the first 16 columns of this thread's own 64 scores (all read by now): the
                // P V products take them from there as their A operand, four e4m3 per column, lane = row
                dm::tmem_st16(t_s, codes);
                dm::tmem_st_wait();
                dm::tc_fence_before();
                dm::named_bar_arrive(kBarCodes + 2 * team + g, 128 + 32);
            }
            gt += n_tiles;
        }
    }
    dm::tc_fence_before();
    __syncthreads();
    if (warp == 0) dm::tmem_dealloc(tmem, 512);
}


}  // namespace

namespace dmh {
int check_shape(const DmShape& s, int h0, int hcount, char* err, size_t errlen) {
    DM_REQUIRE(s.D == 128 || s.D == 256, DM_ERR_ARG, "head_dim must be 128 or 256 (got %d)", s.D);
    const int mult = s.D == 128 ? 256 : 128;
    DM_REQUIRE(s.N > 0 && s.N % mult == 0, DM_ERR_ARG, "seqlen must be a positive multiple of %d at head_dim %d (got %d)", mult, s.D, s.N);
    DM_REQUIRE(s.B > 0, DM_ERR_ARG, "empty batch");
    DM_REQUIRE(s.Hk > 0 && s.H > 0 && s.H % s.Hk == 0, DM_ERR_ARG, "nheads (%d) must be a positive multiple of nheads_k (%d)", s.H, s.Hk);
    DM_REQUIRE((int64_t)s.B * s.H <= 65535, DM_ERR_ARG, "batch * nheads must be at most 65535 (got %lld)", (long long)s.B * s.H);
    DM_REQUIRE(h0 >= 0 && hcount > 0 && h0 + hcount <= s.H, DM_ERR_ARG, "head range [%d, %d) is outside [0, %d)", h0, h0 + hcount, s.H);
    DM_REQUIRE((int64_t)s.B * s.H * s.N < (int64_t)1 << 31, DM_ERR_ARG, "batch * nheads * seqlen must be below 2^31");
    return DM_OK;
}
}  // namespace dmh

namespace dmh {
int launch_fwd_d256(const void* q8, const void* k8, const void* v8, const float* q8s, const float* k8s, const float* v8s, DmShape sh,
                    int h0, int hcount, void* o, float* lse, void* stream, char* err, size_t errlen);
}

namespace dmh {
constexpr int kFwdRegPool = kSoftmaxThreads * kRegSoftmax + 256 * kRegFold + 128 * kRegService;
static_assert(kFwdRegPool == kThreads * 72, "the roles' register requests must add up to the launch pool");

int prepare_fwd(char* err, size_t errlen) {
    static DeviceOnce once;
    return device_once(once, err, errlen, [&]() -> int {
        for (auto kernel : {(const void*)fwd_d128_kernel<dm::SnakeWalk>, (const void*)fwd_d128_kernel<dm::PackedWalk>}) {
            DM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FwdSmem) + 1024));
            if (int rc = check_register_pool(kernel, kThreads, kFwdRegPool, err, errlen)) return rc;
        }
        return DM_OK;
    });
}

int check_cp(const DmShape& s, const DmCp& cp, char* err, size_t errlen) {
    DM_REQUIRE(s.D == 128, DM_ERR_UNSUPPORTED, "context-parallel row maps are built for head_dim 128 only");
    DM_REQUIRE(cp.nq > 0 && cp.nq % 256 == 0 && cp.nq <= s.N, DM_ERR_ARG, "local seqlen must be a positive multiple of 256 (got %d)", cp.nq);
    DM_REQUIRE(cp.half_blocks > 0 && cp.half_blocks % 2 == 0 && cp.half_blocks * 128 <= cp.nq, DM_ERR_ARG, "bad first-chunk size %d blocks", cp.half_blocks);
    DM_REQUIRE(cp.off0 >= 0 && cp.off0 % 2 == 0 && (cp.off0 + cp.half_blocks) * 128 <= s.N, DM_ERR_ARG, "first chunk lies outside the sequence");
    const int rest = cp.nq / 128 - cp.half_blocks;
    DM_REQUIRE(rest == 0 || (cp.off1 % 2 == 0 && cp.off1 >= cp.off0 + cp.half_blocks && (cp.off1 + rest) * 128 <= s.N), DM_ERR_ARG,
               "second chunk must follow the first and lie inside the sequence");
    return DM_OK;
}
}  // namespace dmh

extern "C" int dm_fwd_fp8(const void* q8, const void* k8, const void* v8, const float* q8s, const float* k8s, const float* v8s,
                          DmShape sh, int32_t h0, int32_t hcount, void* o, float* lse, void* stream, char* err, size_t errlen) {
    if (sh.D == 256) {
        int rc = dmh::check_shape(sh, h0, hcount, err, errlen);
        if (rc) return rc;
        const void* ptrs[] = {q8, k8, v8, q8s, k8s, v8s, o, lse};
        const char* names[] = {"q8", "k8", "v8", "q8s", "k8s", "v8s", "o", "lse"};
        for (int i = 0; i < 8; ++i)
            if ((rc = dmh::check_device_ptr(ptrs[i], names[i], err, errlen))) return rc;
        DM_REQUIRE(dmh::aligned16(q8) && dmh::aligned16(k8) && dmh::aligned16(v8) && dmh::aligned16(o), DM_ERR_ARG,
                   "code and output pointers must be 16-byte aligned");
        return dmh::launch_fwd_d256(q8, k8, v8, q8s, k8s, v8s, sh, h0, hcount, o, lse, stream, err, errlen);
    }
    DmCp cp{sh.N, sh.N / 128, 0, 0};
    return dm_fwd_fp8_cp(q8, k8, v8, q8s, k8s, v8s, sh, cp, h0, hcount, o, lse, stream, err, errlen);
}

extern "C" int dm_fwd_fp8_cp(const void* q8, const void* k8, const void* v8, const float* q8s, const float* k8s, const float* v8s,
                          DmShape sh, DmCp cp, int32_t h0, int32_t hcount, void* o, float* lse, void* stream, char* err, size_t errlen) {
    int rc = dmh::check_shape(sh, h0, hcount, err, errlen);
    if (rc) return rc;
    if ((rc = dmh::check_cp(sh, cp, err, errlen))) return rc;
    const void* ptrs[] = {q8, k8, v8, q8s, k8s, v8s, o, lse};
    const char* names[] = {"q8", "k8", "v8", "q8s", "k8s", "v8s", "o", "lse"};
    for (int i = 0; i < 8; ++i)
        if ((rc = dmh::check_device_ptr(ptrs[i], names[i], err, errlen))) return rc;
    DM_REQUIRE(dmh::aligned16(q8) && dmh::aligned16(k8) && dmh::aligned16(v8) && dmh::aligned16(o), DM_ERR_ARG,
               "code and output pointers must be 16-byte aligned");
    CUtensorMap tq, tk, tv;
    if ((rc = dmh::make_tmap_u8(&tq, q8, 128, (uint64_t)sh.B * sh.H * cp.nq, 128, err, errlen))) return rc;
    if ((rc = dmh::make_tmap_u8(&tk, k8, 128, (uint64_t)sh.B * sh.Hk * sh.N, 128, err, errlen))) return rc;
    if ((rc = dmh::make_tmap_u8(&tv, v8, 128, (uint64_t)sh.B * sh.Hk * sh.N, 128, err, errlen))) return rc;
    int* status = dmh::device_status_word(err, errlen);
    if (!status) return DM_ERR_CUDA;
    FwdParams p{q8s, k8s, v8s, static_cast<__nv_bfloat16*>(o), lse, sh.H, sh.Hk, sh.N, h0, hcount, sh.causal, status,
                dm::RowMap{cp.nq, cp.half_blocks, cp.off0, cp.off1}, sh.B * hcount, dm::make_fastdiv(sh.B * hcount), dm::make_fastdiv(hcount),
                dm::make_fastdiv(sh.H / sh.Hk)};
    if ((rc = dmh::prepare_fwd(err, errlen))) return rc;
    const int smem = (int)sizeof(FwdSmem) + 1024;
    int sms = 0;
    if ((rc = dmh::sm_count(&sms, err, errlen))) return rc;
    // persistent: one CTA per SM walks the (head, row block) items, heaviest first
    const int64_t items = (int64_t)sh.B * hcount * (cp.nq / 128);
    const int grid = (int)(items < sms ? items : sms);
    dm::PackedWalk walk;
    if (sh.causal && cp.nq == sh.N && dmh::plan_walk(sh.B * hcount, sh.N / 128, grid, &walk)) {
        DM_CUDA(dmh::launch_pdl(fwd_d128_kernel<dm::PackedWalk>, grid, kThreads, smem, stream, tq, tk, tv, p, walk));
    } else {
        DM_CUDA(dmh::launch_pdl(fwd_d128_kernel<dm::SnakeWalk>, grid, kThreads, smem, stream, tq, tk, tv, p, dm::SnakeWalk{}));
    }
    return DM_OK;
}
