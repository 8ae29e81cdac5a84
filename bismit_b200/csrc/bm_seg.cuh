// bm_seg.cuh -- one tuft's stages for tufts the fused tuft kernel does not
// take: dendrites whose length is no power of two in 16..512 (one synapse, 8,
// 12, 24, ...), dendrite counts that are no power of two, and, of tufts whose
// synapses do not start on a 16-byte boundary, those the tiled kernel's
// unaligned form does not serve.
//
// A block takes whole cells, in pieces of whole dendrites of at most
// kSegSyns synapses, in three steps:
//  1. Threads take W-byte windows of the synapse arrays on the arrays' own
//     alignment, whatever the tuft's: vector loads and stores, byte stores
//     only for the windows that straddle the piece's ends. Each synapse's
//     axon comes through L1 (a cell's neighbourhood spans a few lines). New
//     states, and the same bytes where the strength is not negative, go to
//     shared memory.
//  2. A thread per dendrite sums its bytes there, a masked word at a time.
//  3. A thread per cell reduces its dendrites' results (pyramidal layers).
// The gathers with their source extraction and bounds checks bound it. A
// thread per cell, the form it replaces, walked the cell's synapses one by
// one: the 16 x 64 tuft of a 150 x 150 x 3 layer (69 M synapses, 8 bytes off
// alignment) took 3.43 ms and 0.236 ms this way (the tiled kernel's unaligned
// form: 0.092); 27,648 cells of 4 x 8 dendrites
// 23.2 us, now 10.1; 30,000 cells of 4 x 12 with nonspatial sources 44 us,
// now 15.3 (cold, ncu).
#pragma once
#include "bm_items.cuh"

namespace bm {

constexpr uint32_t kSegBlock = 128;
constexpr uint32_t kSegSyns = 4096;   // synapses of a piece: the longest dendrite a plan allows
constexpr uint32_t kSegDens = 2048;   // dendrites of a block: kSegBlock * 16 one-synapse ones, or one cell's 256

struct SegSmem {
    uint32_t ns[kSegSyns / 4 + 8], ps[kSegSyns / 4 + 8];
    uint8_t draw[kSegDens], dst[kSegDens];
    uint32_t sx[256];
};

// Cells a block takes, for windows of W bytes.
__host__ __device__ __forceinline__ uint32_t seg_cells(uint32_t spt, uint32_t W) {
    const uint32_t n = kSegBlock * W / spt;
    return n ? n : 1u;
}

// Bytes of a thread's window for launches of n synapses: 16, or 4 where 16
// would leave SMs without eight blocks.
__host__ __device__ __forceinline__ uint32_t seg_window(uint64_t n, int sms) {
    return n >= (uint64_t)sms * 8 * kSegBlock * 16 ? 16u : 4u;
}

template <int W> struct SegVec;
template <> struct SegVec<16> { using T = uint4; };
template <> struct SegVec<4> { using T = uint32_t; };

struct SegBlockSync {
    static __device__ __forceinline__ void sync() { __syncthreads(); }
};

// Cells [c0, c0 + nc) of tuft t (at most seg_cells of them), by NT threads
// (threadIdx.x < NT) that Sync::sync() joins.
template <int W, uint32_t NT = kSegBlock, class Sync = SegBlockSync>
__device__ __forceinline__ void tuft_seg_block(const uint8_t* __restrict__ axns, const SliceRec* __restrict__ slices,
                                               const DevLayer& L, uint32_t t, int32_t rnd, uint32_t c0, uint32_t nc,
                                               bool soma, SegSmem& S) {
    using V = typename SegVec<W>::T;
    const DevTuft& T = L.tft[t];
    const uint32_t tid = threadIdx.x;
    const uint32_t spt = T.spt, spd = T.spd, dpt = T.dpt;
    const uint32_t usz = L.u_size, cols = L.v_size * usz;
    // Slices that share the first source's geometry (and are spatial, where
    // the scalar and vec4 index forms agree) are gathered from by their first
    // axon alone; any other slice id takes the general index.
    const SliceRec r0 = slices[T.src_slc];
    const uint32_t sv = r0.y & 0xFFFFu, su = r0.y >> 16, vs = r0.z & 0xFFu, us = (r0.z >> 8) & 0xFFu;
    for (uint32_t k = tid; k < 256; k += NT) {
        uint32_t x = 0xFFFFFFFFu;
        if (k < L.n_slices) {
            const SliceRec r = slices[k];
            if (r.y == r0.y && r.z == r0.z && (r.z >> 16) == 0) x = r.x;
        }
        S.sx[k] = x;
    }
    Sync::sync();
    const uint8_t* a_slc = L.buf[BM_BUF_SYN_SRC_SLC_IDS];
    const uint8_t* a_vo = L.buf[BM_BUF_SYN_SRC_COL_V_OFFS];
    const uint8_t* a_uo = L.buf[BM_BUF_SYN_SRC_COL_U_OFFS];
    const uint8_t* a_str = L.buf[BM_BUF_SYN_STRENGTHS];
    uint8_t* a_st = L.buf[BM_BUF_SYN_STATES];
    uint8_t* a_fl = L.buf[BM_BUF_SYN_FLAG_SETS];
    const uint32_t d_first = c0 * dpt, d_end = (c0 + nc) * dpt;
    const uint32_t d_step = min(d_end - d_first, max(kSegSyns / spd, 1u));
    for (uint32_t d0 = d_first; d0 < d_end; d0 += d_step) {
        const uint32_t nd = min(d_step, d_end - d0);
        const uint64_t lo = T.syn_idz + (uint64_t)d0 * spd, hi = lo + (uint64_t)nd * spd;
        const uint64_t base = lo & ~15ull;
        for (uint64_t g = base + (uint64_t)tid * W; g < hi; g += (uint64_t)NT * W) {
            if (W < 16 && g + W <= lo) continue;
            const V slc_v = *(const V*)(a_slc + g), vo_v = *(const V*)(a_vo + g), uo_v = *(const V*)(a_uo + g);
            const V str_v = *(const V*)(a_str + g), st_v = *(const V*)(a_st + g), fl_v = *(const V*)(a_fl + g);
            const uint32_t* slc_w = (const uint32_t*)&slc_v;
            const uint32_t* vo_w = (const uint32_t*)&vo_v;
            const uint32_t* uo_w = (const uint32_t*)&uo_v;
            const uint32_t* str_w = (const uint32_t*)&str_v;
            const uint32_t* st_w = (const uint32_t*)&st_v;
            const uint32_t* fl_w = (const uint32_t*)&fl_v;
            const bool full = g >= lo && g + W <= hi;
            // The cell of the window's first synapse inside the piece; `left`
            // counts down to the next cell from the window's first byte (bytes
            // before or past the piece gather from some cell, in bounds, and
            // are dropped).
            const uint32_t skip = g < lo ? (uint32_t)(lo - g) : 0u;
            const uint32_t rel = (uint32_t)(g + skip - T.syn_idz);
            const uint32_t cell = rel / spt;
            uint32_t left = spt - (rel - cell * spt) + skip;
            const uint32_t rem = cell % cols;
            uint32_t v = rem / usz, u = rem - v * usz;
            int32_t vsc = (int32_t)((v * vs) >> kSlcSclCoeffL2), usc = (int32_t)((u * us) >> kSlcSclCoeffL2);
            V nst_v, nfl_v;
            uint32_t* nst_w = (uint32_t*)&nst_v;
            uint32_t* nfl_w = (uint32_t*)&nfl_v;
#pragma unroll
            for (int w = 0; w < W / 4; w++) {
                uint32_t a[4];
#pragma unroll
                for (int b = 0; b < 4; b++) {
                    const uint32_t slc = (slc_w[w] >> (8 * b)) & 0xFFu;
                    const int vo = (int)(int8_t)(vo_w[w] >> (8 * b)), uo = (int)(int8_t)(uo_w[w] >> (8 * b));
                    const uint32_t x = S.sx[slc];
                    a[b] = 0;
                    if (x != 0xFFFFFFFFu) {
                        const int32_t vt = vsc + vo, ut = usc + uo;
                        if ((uint32_t)vt < sv && (uint32_t)ut < su) a[b] = __ldg(axns + (x + (uint32_t)vt * su + (uint32_t)ut));
                    } else {
                        bool safe;
                        const uint32_t ai = axn_idx(slices[slc], v, vo, u, uo, (spt & 3) == 0, safe);
                        if (safe) a[b] = __ldg(axns + ai);
                    }
                    if (--left == 0) {   // the next synapse is the next cell's
                        left = spt;
                        if (++u == usz) {
                            u = 0;
                            if (++v == L.v_size) v = 0;
                        }
                        vsc = (int32_t)((v * vs) >> kSlcSclCoeffL2);
                        usc = (int32_t)((u * us) >> kSlcSclCoeffL2);
                    }
                }
                const uint32_t x4 = __byte_perm(__byte_perm(a[0], a[1], 0x0040), __byte_perm(a[2], a[3], 0x0040), 0x5410);
                // syn_fire (cl/syns.cl:2-4) of four bytes; the flags of
                // tft_set_syn_flags (cl/syns.cl:23-33) from the states before.
                nst_w[w] = nz_bytes(x4) | ((x4 >> 1) & 0x7F7F7F7Fu);
                nfl_w[w] = (fl_w[w] & 0xEFEFEFEFu) | (nz_bytes(st_w[w]) >> 3);
                const uint32_t at = (uint32_t)(g - base) / 4 + w;
                S.ns[at] = nst_w[w];
                S.ps[at] = nst_w[w] & ~neg_bytes(str_w[w]);
            }
            if (full) {
                *(V*)(a_st + g) = nst_v;
                *(V*)(a_fl + g) = nfl_v;
            } else {
#pragma unroll
                for (int k = 0; k < W; k++)
                    if (g + k >= lo && g + k < hi) {
                        a_st[g + k] = (uint8_t)(nst_w[k / 4] >> (8 * (k & 3)));
                        a_fl[g + k] = (uint8_t)(nfl_w[k / 4] >> (8 * (k & 3)));
                    }
            }
        }
        Sync::sync();
        // den_cycle_tft, cl/bismit.cl:695-747.
        for (uint32_t k = tid; k < nd; k += NT) {
            const uint32_t d = d0 + k;
            const uint64_t di = T.den_idz + d;
            const uint8_t act0 = L.buf[BM_BUF_DEN_ACTIVITIES][di];
            const uint32_t s0 = (uint32_t)(lo - base) + k * spd, s1 = s0 + spd - 1;
            const uint32_t w0 = s0 >> 2, nw = (s1 >> 2) - w0 + 1;
            const uint32_t m0 = 0xFFFFFFFFu << (8 * (s0 & 3)), m1 = 0xFFFFFFFFu >> (8 * (3 - (s1 & 3)));
            uint32_t sum = 0, raw = 0;
            uint32_t q = k % nw;   // threads start at different words: fewer bank conflicts
            for (uint32_t j = 0; j < nw; j++) {
                const uint32_t m = (q == 0 ? m0 : 0xFFFFFFFFu) & (q + 1 == nw ? m1 : 0xFFFFFFFFu);
                raw = __dp4a(S.ns[w0 + q] & m, 0x01010101u, raw);
                sum = __dp4a(S.ps[w0 + q] & m, 0x01010101u, sum);
                if (++q == nw) q = 0;
            }
            const int active = sum > T.thresh;
            if (!active) sum = 0;
            const uint32_t seed = (raw + T.thresh) | (uint32_t)di;
            L.buf[BM_BUF_DEN_ACTIVITIES][di] =
                update_activity(act0, active, rnd, (int32_t)seed, kDendriteActivityDecay);
            const uint32_t d_raw = min(raw >> 4, 255u);
            uint32_t d_st = min(sum >> 4, 255u);
            L.buf[BM_BUF_DEN_STATES_RAW][di] = (uint8_t)d_raw;
            if (soma) d_st = ssc_soma(L.buf[BM_BUF_CEL_ENERGIES], d, L.buf[BM_BUF_CEL_ENERGIES][d], d_st);
            L.buf[BM_BUF_DEN_STATES][di] = (uint8_t)d_st;
            S.draw[d - d_first] = (uint8_t)d_raw;
            S.dst[d - d_first] = (uint8_t)d_st;
        }
        Sync::sync();
    }
    if (L.kind != BM_LYR_PYRAMIDAL) return;
    for (uint32_t k = tid; k < nc; k += NT) tft_cycle_of(L, T, c0 + k, S.draw + k * dpt, S.dst + k * dpt);
}

}  // namespace bm
