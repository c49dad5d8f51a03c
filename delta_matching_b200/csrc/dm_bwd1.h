// What the two pass 1 kernels (dm_bwd1_d128.cu, dm_bwd1.cu for head_dim 256) share: the launch parameters, the work list.
#pragma once
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
    FastDiv fd_heads, fd_hcount, fd_rep, fd_nbn;  // divisions by n_heads, hcount, H / Hk and N / 128
};

// The work list: one item = one 128-key block J of one (batch, query head) (and one d half at head_dim 256), ordered by
// key block, i.e. heaviest first when causal.  CTA c takes position c of the even rounds and G - 1 - c of the odd ones
// (a snake), so the long and the short items of a round pair up.
struct Bwd1Item {
    HeadCoord hc;
    int J, zh, m_lo, n_it, bhl;                   // m_lo, n_it: first 64-row m-block and their count, both even
    bool valid;
};
template <int kD>
__device__ __forceinline__ Bwd1Item bwd1_item(const Bwd1Params& p, int round) {
    Bwd1Item w;
    const int G = gridDim.x, c = blockIdx.x;
    const int nbn = p.N / 128;
    const int idx = round * G + ((round & 1) ? G - 1 - c : c);
    w.valid = idx < p.n_heads * nbn * (kD / 128);
    const int jz = (int)fdiv((uint32_t)idx, p.fd_heads);
    w.hc = head_coord(idx - jz * p.n_heads, p.h0, p.fd_hcount, p.H, p.Hk, p.fd_rep);
    w.bhl = w.hc.b * p.hcount + (w.hc.h - p.h0);
    w.zh = kD == 128 ? 0 : (int)fdiv((uint32_t)jz, p.fd_nbn);   // d half whose dK / dV columns the item keeps
    w.J = jz - w.zh * nbn;
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
