// bm_plain.cu -- the plain CUDA form of bismit's cycle: one kernel per
// reference stage, one area per launch, same stage order as the reference host.
// Each kernel restates the bismit OpenCL kernel it names; the fused stage
// kernels (bm_fused.cu) must produce identical bytes.
#include "bm_items.cuh"
#include "bm_kernels.h"
#include "bm_seg.cuh"

namespace bm {

namespace {

__device__ __forceinline__ uint64_t gtid() { return (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; }

// tft_set_syn_flags, cl/syns.cl:23-33, 16 synapses per thread.
__global__ void k_set_syn_flags(const uint8_t* __restrict__ states, uint8_t* __restrict__ flags, uint64_t n) {
    pdl_begin();
    uint64_t i = gtid() * 16;
    if (i + 16 <= n && ((((uintptr_t)states) | ((uintptr_t)flags)) & 15) == 0) {
        uint4 s = *(const uint4*)(states + i);
        uint4 f = *(const uint4*)(flags + i);
        uint32_t* sp = (uint32_t*)&s;
        uint32_t* fp = (uint32_t*)&f;
#pragma unroll
        for (int w = 0; w < 4; w++) {
            uint32_t x = sp[w];
            uint32_t nz = (((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x) & 0x80808080u;  // 0x80 per nonzero byte
            fp[w] = (fp[w] & 0xEFEFEFEFu) | (nz >> 3);
        }
        *(uint4*)(flags + i) = f;
    } else {
        for (uint64_t k = i; k < n && k < i + 16; k++)
            flags[k] = (uint8_t)((flags[k] & ~kSynPrevActiveFlag) | (states[k] ? kSynPrevActiveFlag : 0));
    }
}

// The per-item bodies are in bm_items.cuh; each kernel below is one area's
// stage, one thread per item.
__global__ void k_syn_cycle(const uint8_t* __restrict__ axns, const SliceRec* __restrict__ slices,
                            DevLayer L, uint32_t t) {
    pdl_begin();
    uint64_t i = gtid();
    if (i >= (uint64_t)L.cells * L.tft[t].spt) return;
    syn_cycle_item(axns, slices, L, t, i);
}

__global__ void k_den_cycle(DevLayer L, uint32_t t, const AreaCtl* ctl) {
    pdl_begin();
    uint64_t d = gtid();
    if (d >= (uint64_t)L.cells * L.tft[t].dpt) return;
    den_cycle_item(L, t, rnd_at(L.tft[t].rnd_key_den, ctl->cycle), d);
}

__global__ void k_tft_cycle(DevLayer L, uint32_t t) {
    pdl_begin();
    uint32_t c = (uint32_t)gtid();
    if (c < L.cells) tft_cycle_item(L, t, c);
}

__global__ void k_ssc_cycle(DevLayer L) {
    pdl_begin();
    uint32_t c = (uint32_t)gtid();
    if (c < L.cells) ssc_cycle_item(L, c);
}

__global__ void k_inhib_simple(uint8_t* __restrict__ axns, const SliceRec* __restrict__ slices, DevLayer L,
                               int radius, uint64_t rnd_key, const AreaCtl* ctl) {
    pdl_begin();
    uint32_t c = (uint32_t)gtid();
    if (c < L.cells) inhib_simple_item(axns, slices, L, radius, rnd_at(rnd_key, ctl->cycle), c);
}

__global__ void k_inhib_passthrough(uint8_t* __restrict__ axns, const SliceRec* __restrict__ slices, DevLayer L) {
    pdl_begin();
    uint32_t c = (uint32_t)gtid();
    if (c < L.cells) inhib_passthrough_item(axns, slices, L, c);
}

__global__ void k_ssc_mtp_simple(const uint8_t* __restrict__ axns, DevLayer L, const AreaCtl* ctl) {
    pdl_begin();
    uint32_t c = (uint32_t)gtid();
    if (c < L.cells) ssc_mtp_item(axns, L, rnd_at(L.rnd_key_ssc_mtp, ctl->cycle), c);
}

__global__ void k_pyr_cycle(DevLayer L) {
    pdl_begin();
    uint32_t c = (uint32_t)gtid();
    if (c < L.cells) pyr_cycle_item(L, c);
}

__global__ void k_pyr_output(uint8_t* __restrict__ axns, const SliceRec* __restrict__ slices, DevLayer L) {
    pdl_begin();
    uint32_t c = (uint32_t)gtid();
    if (c < L.cells) pyr_output_item(axns, slices, L, c);
}

__global__ void k_inhib_intra_column(uint8_t* __restrict__ axns, const SliceRec* __restrict__ slices, DevLayer L) {
    pdl_begin();
    uint32_t col = (uint32_t)gtid();
    if (col < L.v_size * L.u_size) intra_column_item(axns, slices, L, col);
}

__global__ void k_tft_dst_mtp(const uint8_t* __restrict__ axns, DevLayer L, uint32_t t, const AreaCtl* ctl) {
    pdl_begin();
    uint32_t c = (uint32_t)gtid();
    if (c < L.cells) tft_dst_mtp_item(axns, L, t, rnd_at(L.tft[t].rnd_key_mtp, ctl->cycle), c);
}

// Tufts of at most kCellTuftSyns synapses a cell, a thread per cell: 28,800
// one-synapse cells take 4.7 us cold, in k_tuft_seg's blocks 15.6 us (57 of
// them, each walking four cells a thread through its three steps).
__global__ void k_tuft_cells(const uint8_t* __restrict__ axns, const SliceRec* __restrict__ slices, DevLayer L,
                             uint32_t t, const AreaCtl* ctl) {
    pdl_begin();
    uint32_t c = (uint32_t)gtid();
    if (c < L.cells) tuft_cells_item(axns, slices, L, t, rnd_at(L.tft[t].rnd_key_den, ctl->cycle), c);
}

// W: bytes of each thread's window (bm_seg.cuh). 16 while that still gives
// every SM several blocks, else 4.
template <int W>
__global__ void __launch_bounds__(kSegBlock) k_tuft_seg(const uint8_t* __restrict__ axns,
                                                        const SliceRec* __restrict__ slices, DevLayer L, uint32_t t,
                                                        const AreaCtl* ctl, uint32_t per, int soma,
                                                        long long host_cycle) {
    pdl_begin();
    __shared__ SegSmem S;
    const uint32_t c0 = blockIdx.x * per;
    const unsigned long long cyc = host_cycle >= 0 ? (unsigned long long)host_cycle : ctl->cycle;
    tuft_seg_block<W>(axns, slices, L, t, rnd_at(L.tft[t].rnd_key_den, cyc), c0, min(per, L.cells - c0), soma != 0, S);
}

// Warp-cooperative: no thread leaves before the warp's shared part. With
// host_cycle >= 0 the cycle number comes from the host (a launch on the
// area's front stream, which may run ahead of the area's counter).
__global__ void __launch_bounds__(128) k_inhib_mtp(uint8_t* __restrict__ axns, const SliceRec* __restrict__ slices,
                                                   DevLayer L, int radius, uint64_t key, int learn,
                                                   const AreaCtl* ctl, long long host_cycle) {
    pdl_begin();
    uint32_t c = (uint32_t)gtid();
    const unsigned long long cyc = host_cycle >= 0 ? (unsigned long long)host_cycle : ctl->cycle;
    inhib_mtp_warp(axns, slices, L, radius, rnd_at(key, cyc), rnd_at(L.rnd_key_ssc_mtp, cyc), learn != 0, c,
                   c < L.cells);
}

// With end_cycle, the last block to finish also ends the cycle (the cycle-end
// launch folded in): every block has read the cycle number by then. Twelve
// blocks of 128 per SM (40 registers): area_256's 262,144 cells then need 1.15
// waves of warps instead of the 1.54 that 54 registers allowed. With folded
// tufts there are few cells: six, and nothing spilled.
template <int FOLD>
__global__ void __launch_bounds__(128, FOLD == FOLD_NONE ? 12 : 6)
    k_pyr_tail(uint8_t* __restrict__ axns, const SliceRec* __restrict__ slices, DevLayer L, int ctrl, int learn,
               AreaCtl* ctl, uint32_t tufts, int end) {
    pdl_begin();
    const uint64_t i = gtid();
    pyr_tail_warp<FOLD>(axns, slices, L, ctrl, learn != 0, ctl, (uint32_t)i, i < tail_items(L.depth, L.v_size * L.u_size),
                  tufts);
    if (!end) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1) {
            ctl->blocks_done = 0;
            end_cycle(ctl);
        }
    }
}

inline unsigned nblk(uint64_t n, unsigned b) { return (unsigned)((n + b - 1) / b); }

}  // namespace

// ------------------------------------------------------------ launchers ---
void launch_set_syn_flags(const DevLayer& L, cudaStream_t s) {
    uint64_t n = L.n_syns;
    if (!n) return;
    launch_pdl(k_set_syn_flags, nblk((n + 15) / 16, 256), 256, 0, s, L.buf[BM_BUF_SYN_STATES], L.buf[BM_BUF_SYN_FLAG_SETS], n);
}
void launch_set_syn_flags_tuft(const DevLayer& L, uint32_t t, cudaStream_t s) {
    const DevTuft& T = L.tft[t];
    uint64_t n = (uint64_t)L.cells * T.spt;
    if (!n) return;
    launch_pdl(k_set_syn_flags, nblk((n + 15) / 16, 256), 256, 0, s, L.buf[BM_BUF_SYN_STATES] + T.syn_idz,
                                                              L.buf[BM_BUF_SYN_FLAG_SETS] + T.syn_idz, n);
}
void launch_syn_cycle_plain(const uint8_t* axns, const SliceRec* slices, const DevLayer& L, uint32_t t,
                            cudaStream_t s) {
    uint64_t n = (uint64_t)L.cells * L.tft[t].spt;
    launch_pdl(k_syn_cycle, nblk(n, 256), 256, 0, s, axns, slices, L, t);
}
void launch_den_cycle_plain(const DevLayer& L, uint32_t t, const AreaCtl* ctl, cudaStream_t s) {
    uint64_t n = (uint64_t)L.cells * L.tft[t].dpt;
    launch_pdl(k_den_cycle, nblk(n, 256), 256, 0, s, L, t, ctl);
}
void launch_tft_cycle_plain(const DevLayer& L, uint32_t t, cudaStream_t s) {
    launch_pdl(k_tft_cycle, nblk(L.cells, 256), 256, 0, s, L, t);
}
void launch_ssc_cycle(const DevLayer& L, cudaStream_t s) {
    launch_pdl(k_ssc_cycle, nblk(L.cells, 256), 256, 0, s, L);
}
void launch_inhib_simple(uint8_t* axns, const SliceRec* slices, const DevLayer& L, int radius, uint64_t key,
                         const AreaCtl* ctl, cudaStream_t s) {
    launch_pdl(k_inhib_simple, nblk(L.cells, 128), 128, 0, s, axns, slices, L, radius, key, ctl);
}
void launch_inhib_passthrough(uint8_t* axns, const SliceRec* slices, const DevLayer& L, cudaStream_t s) {
    launch_pdl(k_inhib_passthrough, nblk(L.cells, 256), 256, 0, s, axns, slices, L);
}
void launch_ssc_mtp_plain(const uint8_t* axns, const DevLayer& L, const AreaCtl* ctl, cudaStream_t s) {
    launch_pdl(k_ssc_mtp_simple, nblk(L.cells, 128), 128, 0, s, axns, L, ctl);
}
void launch_pyr_cycle_plain(const DevLayer& L, cudaStream_t s) {
    launch_pdl(k_pyr_cycle, nblk(L.cells, 256), 256, 0, s, L);
}
void launch_pyr_output(uint8_t* axns, const SliceRec* slices, const DevLayer& L, cudaStream_t s) {
    launch_pdl(k_pyr_output, nblk(L.cells, 256), 256, 0, s, axns, slices, L);
}
// smooth_activity (cl/control.cl:227-295). Each group center scans the hexagon
// of side r around it over every slice of the host layer (slice, then v
// offset, then u offset, as the reference loops), finds the least active cell
// (ties: the later one) and the most active (ties: the later one), and raises
// the least active cell's energy by one and lowers the most active's by one,
// each within 0..255 and only when they differ. Six lattices of centers act
// one after the other; within a lattice the hexagons are disjoint.
//
// Activities do not change while the smoother runs, so every lattice's finds
// run at once (a warp per center), each leaving a bit per lattice at the cells
// it picked: bit k, raise; bit 8 + k, lower. A second launch applies a cell's
// bits in lattice order, which is what six launches one after the other do.
// Latency-bound (a hexagon's loads, then a warp's reduction): a 120 x 120 layer
// with r = 3 took six launches of a thread per center, 7.0 us each; the two
// launches take 4.9 and 3.6 us (cold, ncu).
struct SmoothRange {
    uint32_t off[7];   // lattice k: centers off[k] .. off[k + 1] - 1
};

__global__ void __launch_bounds__(128) k_smooth_find(DevLayer L, const int32_t* __restrict__ centers, SmoothRange R,
                                                     int32_t r, uint32_t* __restrict__ ops) {
    pdl_begin();
    const uint32_t i = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= R.off[6]) return;
    const int32_t cv = centers[i] >> 16, cu = (int32_t)(int16_t)(centers[i] & 0xFFFF);
    const uint8_t* act = L.buf[BM_BUF_CEL_ACTIVITIES];
    const int32_t vs = (int32_t)L.v_size, us = (int32_t)L.u_size;
    const uint32_t side = 2 * (uint32_t)r + 1, sq = side * side;   // at most 255; sq * depth < 2^24
    // Keys order cells by activity, then by place in the scan.
    uint32_t least = 0xFFFFFFFFu, most = 0;
    bool any = false;
    auto place = [&](uint32_t p, int32_t& v, int32_t& u) {   // the p-th cell of the square around the hexagon
        const int32_t vo = (int32_t)(p / side) - r, uo = (int32_t)(p % side) - r;
        v = cv + vo;
        u = cu + uo;
        return uo >= max(-r, -vo - r) && uo <= min(r, -vo + r) && v >= 0 && v < vs && u >= 0 && u < us;
    };
    for (uint32_t slc = 0; slc < L.depth; slc++)
        for (uint32_t p = lane; p < sq; p += 32) {
            int32_t v, u;
            if (!place(p, v, u)) continue;
            const uint32_t a = act[slc * (uint32_t)(vs * us) + (uint32_t)(v * us + u)], ord = slc * sq + p;
            least = min(least, (a << 24) | (0xFFFFFFu - ord));
            most = max(most, (a << 24) | ord);
            any = true;
        }
    least = __reduce_min_sync(0xFFFFFFFFu, least);
    most = __reduce_max_sync(0xFFFFFFFFu, most);
    // A hexagon wholly outside the layer changes nothing, nor does one whose
    // two cells are the same.
    if (!__any_sync(0xFFFFFFFFu, any) || lane) return;
    const uint32_t lo = 0xFFFFFFu - (least & 0xFFFFFFu), mo = most & 0xFFFFFFu, most_act = most >> 24;
    if (lo == mo) return;
    uint32_t k = 0;
    while (i >= R.off[k + 1]) k++;
    auto cell = [&](uint32_t ord) {
        int32_t v, u;
        const uint32_t slc = ord / sq;
        place(ord - slc * sq, v, u);
        return slc * (uint32_t)(vs * us) + (uint32_t)(v * us + u);
    };
    if (most_act < 255) atomicOr(&ops[cell(lo)], 1u << k);
    if (most_act > 0) atomicOr(&ops[cell(mo)], 256u << k);
}

__global__ void __launch_bounds__(128) k_smooth_apply(uint8_t* __restrict__ en, uint32_t* __restrict__ ops, uint32_t n) {
    pdl_begin();
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const uint32_t o = ops[c];
    if (!o) return;
    uint32_t e = en[c];
#pragma unroll
    for (int k = 0; k < 6; k++) {
        e += (uint32_t)(((o >> k) & 1) && e < 255);
        e -= (uint32_t)(((o >> (8 + k)) & 1) && e > 0);
    }
    en[c] = (uint8_t)e;
    ops[c] = 0;
}

void launch_smooth(const DevLayer& L, const int32_t* centers, const uint32_t off[7], int32_t radius, uint32_t* ops,
                   cudaStream_t s) {
    SmoothRange R;
    for (int k = 0; k < 7; k++) R.off[k] = off[k];
    if (!R.off[6]) return;
    launch_pdl(k_smooth_find, nblk(R.off[6], 4), 128, 0, s, L, centers, R, radius, ops);
    launch_pdl(k_smooth_apply, nblk(L.cells, 128), 128, 0, s, L.buf[BM_BUF_CEL_ENERGIES], ops, L.cells);
}

// retina (cl/filters.cl:34-100), one input filter over a (depth, v, u) grid
// of input bytes. Cell i (its index in the grid) is an off-center cell when
// bit 0 of i is set and a large one when bits 1 and 0 differ; it averages the
// hexagon of radius 5 (large) or 3 (small) around it in its own slice,
// counting cells outside the grid as zero but still dividing by the full
// hexagon (get_neighbors_avg, :8-31). The output is how far the average
// exceeds the cell by more than RETNAL_THRESHOLD (48, cl/bismit.cl:19) for an
// off-center cell, or the cell the average, else 0. It goes to slice
// base_slc + slice of the output at that slice's first axon (the slice
// table's x), the cell's (v, u) place within the slice.
//
// Bound by latency: 91 dependent byte loads a cell, each an L1 or L2 trip, and
// both radii in every warp. So a block takes 4 rows of 32 cells, brings them
// and the 5 cells around into shared memory with a few independent loads a
// thread, and every lane sums both hexagons in one pass without a branch
// (96 x 96: 8.8 us cold with a thread reading global memory, now 3.8).
constexpr int kRetU = 32, kRetV = 4, kRetR = 5, kRetPitch = kRetU + 2 * kRetR;

__global__ void __launch_bounds__(kRetU * kRetV)
    k_retina(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, const SliceRec* __restrict__ slices,
             uint32_t base_slc, uint32_t vs, uint32_t us, uint32_t tiles_u, uint32_t tiles_v) {
    constexpr int kTile = kRetPitch * (kRetV + 2 * kRetR);
    __shared__ uint8_t tile[kTile];
    pdl_begin();
    const uint32_t tu = blockIdx.x % tiles_u, tv = blockIdx.x / tiles_u % tiles_v, slc = blockIdx.x / tiles_u / tiles_v;
    const uint32_t cols = vs * us;
    const int32_t v0 = (int32_t)(tv * kRetV), u0 = (int32_t)(tu * kRetU);
    const uint8_t* plane = in + (uint64_t)slc * cols;
#pragma unroll
    for (int k0 = 0; k0 < kTile; k0 += kRetU * kRetV) {
        const int k = k0 + (int)threadIdx.x;
        const int32_t v = v0 - kRetR + k / kRetPitch, u = u0 - kRetR + k % kRetPitch;
        const bool inside = k < kTile && v >= 0 && v < (int32_t)vs && u >= 0 && u < (int32_t)us;
        const uint8_t x = inside ? plane[(uint32_t)v * us + u] : 0;
        if (k < kTile) tile[k] = x;
    }
    __syncthreads();
    const int tx = threadIdx.x % kRetU, ty = threadIdx.x / kRetU;
    const uint32_t v = v0 + ty, u = u0 + tx;
    if (v >= vs || u >= us) return;
    const uint8_t* mid = tile + (ty + kRetR) * kRetPitch + tx + kRetR;
    int32_t small = 0, ring = 0;   // radius 3, and what radius 5 adds
#pragma unroll
    for (int vo = -5; vo <= 5; vo++)
#pragma unroll
        for (int uo = -5; uo <= 5; uo++) {
            const int w = vo + uo;
            if (w < -5 || w > 5) continue;
            const bool in3 = vo >= -3 && vo <= 3 && uo >= -3 && uo <= 3 && w >= -3 && w <= 3;
            (in3 ? small : ring) += mid[vo * kRetPitch + uo];
        }
    const uint32_t col = v * us + u, i = slc * cols + col;
    const uint32_t off_cen = i & 1, large = ((i & 3) >> 1) ^ off_cen;
    const int32_t avg = large ? (small + ring) / 91 : small / 37;
    const int32_t center = mid[0];
    int32_t st;
    if (off_cen) {
        const int32_t cst = center + kRetinalThreshold;
        st = avg > cst ? avg - cst : 0;
    } else {
        const int32_t nat = avg + kRetinalThreshold;
        st = center > nat ? center - nat : 0;
    }
    out[slices[(base_slc + slc) & 0xFF].x + col] = (uint8_t)st;
}

void launch_retina(const uint8_t* in, uint8_t* out, const SliceRec* slices, uint32_t base_slc, uint32_t depth,
                   uint32_t v_size, uint32_t u_size, cudaStream_t s) {
    const uint32_t tu = nblk(u_size, kRetU), tv = nblk(v_size, kRetV);
    if (depth * v_size * u_size)
        launch_pdl(k_retina, tu * tv * depth, kRetU * kRetV, 0, s, in, out, slices, base_slc, v_size, u_size, tu, tv);
}

void launch_inhib_intra_column_plain(uint8_t* axns, const SliceRec* slices, const DevLayer& L, cudaStream_t s) {
    launch_pdl(k_inhib_intra_column, nblk((uint64_t)L.v_size * L.u_size, 256), 256, 0, s, axns, slices, L);
}
void launch_tuft_seg(const uint8_t* axns, const SliceRec* slices, const DevLayer& L, uint32_t t, const AreaCtl* ctl,
                     int sms, bool soma, cudaStream_t s, int64_t host_cycle) {
    if (L.tft[t].spt <= kCellTuftSyns && !soma && host_cycle < 0) {
        launch_pdl(k_tuft_cells, nblk(L.cells, 128), 128, 0, s, axns, slices, L, t, ctl);
        return;
    }
    const uint32_t W = seg_window((uint64_t)L.cells * L.tft[t].spt, sms), per = seg_cells(L.tft[t].spt, W);
    launch_pdl(W == 16 ? k_tuft_seg<16> : k_tuft_seg<4>, nblk(L.cells, per), kSegBlock, 0, s, axns, slices, L, t, ctl,
               per, soma ? 1 : 0, (long long)host_cycle);
}
void launch_inhib_mtp(uint8_t* axns, const SliceRec* slices, const DevLayer& L, int radius, uint64_t key,
                      bool learn, const AreaCtl* ctl, cudaStream_t s, int64_t host_cycle) {
    launch_pdl(k_inhib_mtp, nblk(L.cells, 128), 128, 0, s, axns, slices, L, radius, key, learn ? 1 : 0, ctl,
               (long long)host_cycle);
}
void launch_pyr_tail(uint8_t* axns, const SliceRec* slices, const DevLayer& L, int ctrl, bool learn, AreaCtl* ctl,
                     cudaStream_t s, uint32_t tufts, bool end) {
    const TailFold f = tail_fold(L, tufts);
    auto kern = f == FOLD_NONE ? k_pyr_tail<FOLD_NONE> : f == FOLD_ONE ? k_pyr_tail<FOLD_ONE> : k_pyr_tail<FOLD_ANY>;
    launch_pdl(kern, nblk(tail_items(L.depth, L.v_size * L.u_size), 128), 128, 0, s, axns, slices, L, ctrl,
               learn ? 1 : 0, ctl, tufts, end ? 1 : 0);
}
void launch_tft_dst_mtp_plain(const uint8_t* axns, const DevLayer& L, uint32_t t, const AreaCtl* ctl,
                              cudaStream_t s) {
    launch_pdl(k_tft_dst_mtp, nblk(L.cells, 128), 128, 0, s, axns, L, t, ctl);
}

}  // namespace bm
