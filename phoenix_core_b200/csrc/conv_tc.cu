// General quaternion convolution on the tensor cores (tcgen05 / TMEM / TMA): any filter size, stride 1 or 2,
// any TF-style padding, any channel count; forward, backward-data and backward-filter.
//
// The reference layout (NCHW, components stacked on the batch axis) cannot feed tap-shifted TMA boxes: the
// innermost TMA coordinate must be a multiple of 16 bytes, and a filter tap shifts the pixel axis by single
// elements. So a convolution with taps first stages two small-or-cheap things in the caller's workspace:
//   * the activations, channels-last:  xp[comp][img][h][w][c16]   (stage_compact, mostly)
//   * the filters as the signed, permuted real matrix of the Hamilton product, one slab per tap:
//       Wexp[tap][(d,co)][(l,ci)] = s(l,d) * w[l^d][co][ci][tap]                    (pack_filters_tile)
//     (reference sign table src/algebras.cc:28-49; for backward-data the transposed block with flipped taps)
// and then runs ONE implicit-GEMM kernel: D[(d,co), pixel] = sum over (tap, l, ci). With channels innermost a
// tap is a shift of the *outer* TMA coordinates (free), stride 2 is the tensor map's element stride, and
// padding is TMA out-of-bounds fill. This replaces the 8/16 cuDNN calls and their
// crop / insert / accumulate kernels (src/conv2d.hpp:167-275, :433-562; src/backend/cudnn/conv2d.hpp:280-309,
// :447-488; src/backend/cudnn/kernels.cu:39-156).
//
// Kernel: persistent, one CTA per SM, or a pair of SMs per tile of 256 rows. Tile = 128 rows (d,co) x 256 pixels (a PW x PH x PN box);
// K slice per stage = one tap, one input component, KS channels; A and B both K-major, both by TMA;
// tcgen05.mma M=128 N=256 K=16; the accumulator is double-buffered in TMEM (2 x 256 columns) so the epilogue
// (8 warps: TMEM -> bias -> cast -> NCHW stores) of tile i overlaps the main loop of tile i+1.
// All mbarrier waits are bounded.
#include "tc_common.cuh"
#include "tensor_path.cuh"

namespace pcb {
namespace {

using namespace umma;
using namespace tc;

constexpr int GM = 128, GN = 256;
constexpr int G_THREADS = 320;                       // warp 0 TMA, warp 1 MMA, warps 2..9 epilogue
constexpr int ST_G_PRODUCER = 0x100, ST_G_MMA = 0x200, ST_G_EPILOGUE = 0x400;

struct GParams {
    int Nb, Mvalid, Cout;        // quaternion batch; valid GEMM rows (4*Cout); channels per output component
    int HO, WO;                  // output plane
    int Cp;                      // padded channels per input component (multiple of 16)
    int KH, KW, SH, SW, DH, DW;
    int PW, PH, PN;              // output tile box, PW*PH*PN == 256
    int tiles_w, tiles_h, tiles_n, tiles_m;
    int fmt, has_bias;
    int LK;                      // input components along K: 4, or 1 for a real-valued (type-0) input
    int store_vec;               // output pixels per store: largest power of two <= 16 dividing WO (and the pointer alignment)
    int n_cols;                  // columns of the tile in use (256, or 8 * PH in halo mode)
    int lw, lh;                  // log2(PW), log2(PH) (lh = -1: PH is not a power of two, and then PN == 1)
    int n_stages;                // operand stages in shared memory
    int plane_mode;              // the tile box covers whole output planes and 128 rows are 128 channels of one component:
                                 // the tile leaves through shared memory as one contiguous bulk copy per image
    // halo mode
    int Wt, Ht;
    int a_slots, a_taps;         // filter slices in flight, and the taps of one (a filter row, or one tap)
    uint32_t halo_bytes;         // shared-memory pitch of one halo tile (n_stages of them)
    uint32_t stage_bytes;        // the other forms: one stage of both operands
    int off_w, off_h;            // added to the pixel coordinates of every activation box: minus the padding (out-of-range coordinates
                                 // read zeros); 0 for a zero-inserted copy, which holds its padding
    int o_generic;               // the output is addressed through the element strides below (channels-last tensors, channel
    int o_p, o_c, o_h, o_w;      // slices of grouped layers, boxes narrower than 8 pixels): one 16-bit store per element
    int o_cl32;                  // channels-last output whose channel count is a multiple of 32: a warp transposes its 32 rows x 32
                                 // columns through shared memory and stores 16-byte runs of channels
    int bias_ld;                 // bias is [components][bias_ld]
    int exact;                   // plane mode with a tile box of exactly PN whole planes (WO x HO x PN pixels, any plane size up to
                                 // 256 pixels): the MMAs are n_cols = PN * WO * HO rounded up to 16 columns wide
    uint32_t b_tx;               // bytes one activation box brings (plain and DUAL forms)
    int split_w, split_h, split_n;   // PAIR: pixels, pixel rows and images from the even CTA's half of the tile box to the odd one's
    int half_valid;              // PAIR, exact: pixels of a half (its columns are rounded up to 8)
    int rows_epi;                // NCHW output whose image rows are not 16-byte aligned: stored through shared memory (store_rows)
    int PT, PL;                  // DUAL form: padding of the strided layer
};
constexpr uint32_t G_PLANE_BYTES = GM * GN * 2;      // staging buffer of the plane-mode epilogue

// K-major operand tile whose rows hold KS 16-bit elements (KS*2 bytes, swizzle span == row size):
// 8-row groups are 8*KS*2 bytes apart. KS = 64 -> 128-byte swizzle, KS = 32 -> 64-byte, KS = 16 -> 32-byte.
template <int KS>
__device__ __forceinline__ uint64_t make_desc_kmajor_rows(uint32_t smem_addr) {
    constexpr uint64_t layout = (KS == 64 ? 2ull : (KS == 32 ? 4ull : 6ull)) << 61;
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)((8 * KS * 2) >> 4) << 32) | DESC_VERSION_SM100 | layout;
}

// The same rows with the 8-row groups `group_bytes` apart: the halo tile, where a group is 8 consecutive pixels of one
// tile row and the next group is one halo-row pitch further. The swizzle is a function of the absolute shared-memory
// address (TMA writes it that way and the MMA reads it that way), so the start address may sit anywhere on a pixel.
__device__ __forceinline__ uint64_t make_desc_kmajor_sw64_groups(uint32_t smem_addr, uint32_t group_bytes) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)((group_bytes >> 4) & 0x3FFFu) << 32) | DESC_VERSION_SM100 |
           (4ull << 61);
}

// Plane-mode epilogue, one thread's 32 accumulator columns (32 >> LW rows of the tile box, PW = 1 << LW pixels each): the
// valid pixels go to the thread's channel plane in the staging buffer. The box row is decoded once per row, the pixel
// index is a compile-time constant: the epilogue warps are few (two per scheduler), so every instruction saved per
// element shortens the tile by its issue latency.
template <int LW>
__device__ __forceinline__ void plane_pack(const uint32_t (&v)[32], int col0, const GParams& p, uint16_t* mine, int HWo, float badd) {
    constexpr int PWc = 1 << LW, ROWS = 32 >> LW;
    const bool pairs = ((HWo | p.WO) & 1) == 0;          // even planes and rows: 4-byte stores of two pixels
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const int jr = (col0 >> LW) + r;
        const int hl = jr & (p.PH - 1), nl = jr >> p.lh;
        if (hl >= p.HO) continue;                         // warp-uniform
        uint16_t* dst = mine + (size_t)nl * GM * HWo + hl * p.WO;
#pragma unroll
        for (int wl = 0; wl < PWc; wl += 2) {
            const float f0 = __uint_as_float(v[r * PWc + wl]) + badd, f1 = __uint_as_float(v[r * PWc + wl + 1]) + badd;
            uint32_t both;
            if (p.fmt == 0) { const __half2 h = __floats2half2_rn(f0, f1); both = *reinterpret_cast<const uint32_t*>(&h); }
            else { const __nv_bfloat162 h = __floats2bfloat162_rn(f0, f1); both = *reinterpret_cast<const uint32_t*>(&h); }
            if (pairs) {
                if (wl < p.WO) *reinterpret_cast<uint32_t*>(dst + wl) = both;
            } else {
                if (wl < p.WO) dst[wl] = (uint16_t)(both & 0xffffu);
                if (wl + 1 < p.WO) dst[wl + 1] = (uint16_t)(both >> 16);
            }
        }
    }
}

// The same for a box of exactly PN whole planes: column j is pixel j % (HO * WO) of image j / (HO * WO) of the tile, in the
// order the plane is stored, so a thread's columns are runs of consecutive elements of its channel plane.
// PAIR: the second half of the columns starts with pixel half_valid.
// EVEN: planes of an even number of pixels, two of which are stored at a time.
template <bool PAIR, bool EVEN>
__device__ __forceinline__ void plane_pack_exact(const uint32_t (&v)[32], int col0, const GParams& p, uint16_t* mine, int HWo, float badd) {
    constexpr int S = EVEN ? 2 : 1;
    const int half_cols = p.n_cols / 2;
    int at = col0;                                       // pixel of the tile; `left`: columns until the padding of the half (or of the tile)
    int left = PAIR ? p.half_valid - col0 : p.PN * HWo - col0;
    if (PAIR && col0 >= half_cols) { at = p.half_valid + col0 - half_cols; left = 2 * p.half_valid - at; }
    const int edge = PAIR ? half_cols - col0 : -1;       // (a multiple of 8)
    int nl = at / HWo, pix = at - nl * HWo;
    uint16_t* dst = mine + (size_t)nl * GM * HWo + pix;
#pragma unroll
    for (int e = 0; e < 32; e += S) {
        if (PAIR && e % 8 == 0 && e > 0 && e == edge) {
            left = p.half_valid + e;
            nl = p.half_valid / HWo; pix = p.half_valid - nl * HWo;
            dst = mine + (size_t)nl * GM * HWo + pix;
        }
        if (e < left) {
            const float f0 = __uint_as_float(v[e]) + badd;
            if (EVEN) {
                const float f1 = __uint_as_float(v[e + 1]) + badd;
                uint32_t both;
                if (p.fmt == 0) { const __half2 h = __floats2half2_rn(f0, f1); both = *reinterpret_cast<const uint32_t*>(&h); }
                else { const __nv_bfloat162 h = __floats2bfloat162_rn(f0, f1); both = *reinterpret_cast<const uint32_t*>(&h); }
                *reinterpret_cast<uint32_t*>(dst) = both;
            } else {
                *dst = p.fmt == 0 ? __half_as_ushort(__float2half_rn(f0)) : __bfloat16_as_ushort(__float2bfloat16_rn(f0));
            }
        }
        dst += S;
        if ((pix += S) == HWo) { pix = 0; dst += (size_t)(GM - 1) * HWo; }
    }
}

// 192 KB of operand stages, at most 12. HALVES: DUAL and PAIR each halve the pixels of a stage
constexpr int H_MAX_SLOTS = 22, H_MAX_TILES = 3;               // halo form: filter slices and halo tiles in flight
template <int KS, int HALVES> constexpr int G_MAX_STAGES = KS == 64 ? (HALVES == 2 ? 8 : (HALVES == 1 ? 6 : 4)) : (KS == 32 ? (HALVES ? 12 : 8) : 12);

// HALO (KS == 32, stride-1 correlation, tile = 8 x PH pixels of one image): for every 32-channel slice of one component the halo
// tile [Ht][Wt][32 channels] of the output tile is loaded once, and every tap's MMAs read it at a shifted start address; the filter
// slices stream beside it. Per MMA the kernel then moves 5 KB from L2 instead of 12 KB, which is what bounds the plain form (an SM
// takes in about 64 bytes per clock). The two operands have rings of their own: 2 or 3 halo tiles of some 20 KB, and as many filter
// slices of one filter row (or tap) as fit; with both operands of all taps in one of two 90 KB stages the loads were exposed. Channels-last
// 3x3, 64 -> 64, 56 x 56, batch 128, forward: 373 -> 356 us (first 20 launches), 424 -> 410 us under the power limit. Also open to 5x5
// and larger filters, whose slices did not fit a stage. What bounds it now is the power limit: 1155 TFLOP/s at 990 W.
//
// DUAL (backward-data of a layer with strides 2 x 2): the input pixels fall into four classes by the parity of row and column,
// and with r = (a + PT) mod 2, c = (a + PT) div 2 the gradient of row class a is dx[2 i + a] = sum over k of dy[i + c - k] w[r + 2 k]
// (columns alike) -- every class takes its own taps of the same dy and filters. A tile is one row class and BOTH column
// classes of 128 x 128 class pixels: a tap kw belongs to column class (kw + PL) mod 2 and its MMAs go to that class's accumulator,
// and the epilogue interleaves the two accumulators into runs of neighbouring pixels of dx. The layer's FLOPs are executed once
// (a convolution of a zero-inserted dy executes four times as many) from one compact copy of dy, in one launch. Bound by the
// operand traffic from L2: 32 KB per four MMAs of 128 x 128 x 16.
//
// PAIR: a cluster of two CTAs takes two neighbouring row tiles and half of the pixels of the tile box each (cta_group::2): per SM
// 32 KB instead of 48 KB from L2 for four MMAs of 128 x 256 x 16, and 7.5 instead of 11 KB of operands from shared memory per MMA of the halo
// form. Without / with, under the power limit: 1x1 256 at 14, bf16, forward 94 / 82 us; 3x3 stride 2, 128 at 28, forward 184 / 157; forward +
// backward of 3x3 64 at 56 1471 / 1362, channels-last 1164 / 1116.
template <int KS, bool HALO, bool DUAL, bool PAIR>
__global__ void __launch_bounds__(G_THREADS, 1)
qconv_general_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, GParams p,
                        const uint16_t* bias, uint16_t* __restrict__ out, int* __restrict__ status) {
    constexpr uint32_t A_BYTES = GM * KS * 2, B_BYTES = GN / ((DUAL ? 2 : 1) * (PAIR ? 2 : 1)) * KS * 2;
    constexpr int MAX_STAGES = HALO ? H_MAX_SLOTS : G_MAX_STAGES<KS, DUAL + PAIR>;
    const int rank = PAIR ? (int)cluster_ctarank() : 0, first = PAIR ? blockIdx.x / 2 : blockIdx.x, step = PAIR ? gridDim.x / 2 : gridDim.x;
    const uint32_t STAGE = HALO ? A_BYTES * p.a_taps : A_BYTES + B_BYTES;      // HALO: one slot of the filter ring
    const int STAGES = HALO ? p.a_slots : p.n_stages;
    const int taps = p.KH * p.KW;
    extern __shared__ uint8_t smem_raw[];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t operand_bytes = STAGES * STAGE + (HALO ? p.n_stages * p.halo_bytes : 0u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + operand_bytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * MAX_STAGES + 5 + 2 * H_MAX_TILES);
    const uint32_t tiles_addr = smem_u32(base), halo_addr = tiles_addr + STAGES * STAGE;
    const uint32_t full_bar = smem_u32(bars), empty_bar = smem_u32(bars + MAX_STAGES);
    const uint32_t tmem_full = smem_u32(bars + 2 * MAX_STAGES), tmem_empty = smem_u32(bars + 2 * MAX_STAGES + 2);
    const uint32_t epi_bar = smem_u32(bars + 2 * MAX_STAGES + 4);
    const uint32_t halo_full = smem_u32(bars + 2 * MAX_STAGES + 5), halo_empty = halo_full + 8 * H_MAX_TILES;      // HALO
    uint8_t* plane_buf = base + operand_bytes + 512;               // plane mode only: [image][128 rows][HO * WO]

    const int tiles_px = p.tiles_w * p.tiles_h * p.tiles_n;
    const int tiles_m = PAIR ? p.tiles_m / 2 : p.tiles_m;
    const int n_tiles = tiles_px * tiles_m * (DUAL ? 2 : 1);
    const int c_steps = p.Cp / KS;
    // DUAL: the row class with more taps comes first in the tile order
    const int first_class = p.PT & 1;               // (a + PT) mod 2 == 0: taps 0, 2, ...
    const int n_k = (HALO ? 1 : taps) * p.LK * c_steps;           // stages per tile

    if (t == 0) {
        for (int s = 0; s < MAX_STAGES; ++s) { mbar_init(full_bar + 8 * s, 1); mbar_init(empty_bar + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(tmem_full + 8 * b, 1); mbar_init(tmem_empty + 8 * b, PAIR ? 16 : 8); }
        mbar_init(epi_bar, 8);
        if (HALO)
            for (int s = 0; s < H_MAX_TILES; ++s) { mbar_init(halo_full + 8 * s, 1); mbar_init(halo_empty + 8 * s, 1); }
        fence_barrier_init();
    }
    if (warp == 1) { if (PAIR) tmem_alloc_pair(smem_u32(tmem_slot), 512); else tmem_alloc(smem_u32(tmem_slot), 512); }
    tc_fence_before_sync();
    __syncthreads();
    if (PAIR) cluster_sync_all();                     // both CTAs' barriers exist before anything signals them
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    chain_wait();
    chain_next();

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        {
            const bool el = elect_one();
            int s = 0, phase = 1;                  // ring position and the parity its `empty` barrier is waited with
            int hs = 0, hphase = 1;                // the same of the halo tiles
            bool ok = true;
            for (int tile = first; tile < n_tiles && ok; tile += step) {
                const int tm = PAIR ? 2 * (tile % tiles_m) + rank : tile % tiles_m;
                int rest = tile / tiles_m;
                const int tw = rest % p.tiles_w; rest /= p.tiles_w;
                const int th = rest % p.tiles_h;
                const int tn = rest / p.tiles_h;
                if (DUAL) {
                    const int cls = tn / p.tiles_n, a = first_class ^ cls, n0 = (tn - cls * p.tiles_n) * p.PN + rank * p.split_n, m0 = tm * GM;
                    for (int kh = (a + p.PT) & 1; kh < p.KH && ok; kh += 2) {
                        const int row = th * p.PH + rank * p.split_h + ((a + p.PT) >> 1) - (kh >> 1);
                        for (int kw = 0; kw < p.KW && ok; ++kw) {
                            const int b = (kw + p.PL) & 1, col = tw * p.PW + ((b + p.PL) >> 1) - (kw >> 1);
                            const int tap = taps - 1 - (kh * p.KW + kw);             // the packed filters hold the taps flipped
                            for (int l = 0; l < p.LK && ok; ++l) {
                                for (int cs = 0; cs < c_steps; ++cs) {
                                    ok = warp_wait_bounded(empty_bar + 8 * s, phase, status, ST_G_PRODUCER);
                                    if (!ok) break;
                                    const uint32_t a_dst = tiles_addr + s * STAGE, bar = full_bar + 8 * s;
                                    if (el && PAIR) {
                                        const uint32_t lead = map_to_cta(bar, 0);
                                        if (rank == 0) mbar_arrive_expect_tx(bar, 2 * (A_BYTES + p.b_tx));
                                        tma_load_3d_pair(a_dst, &map_w, l * p.Cp + cs * KS, m0, tap, lead);
                                        tma_load_5d_pair(a_dst + A_BYTES, &map_x, cs * KS, col, row, n0, l, lead);
                                    } else if (el) {
                                        mbar_arrive_expect_tx(bar, A_BYTES + p.b_tx);
                                        tma_load_3d(a_dst, &map_w, l * p.Cp + cs * KS, m0, tap, bar);
                                        tma_load_5d(a_dst + A_BYTES, &map_x, cs * KS, col, row, n0, l, bar);
                                    }
                                    if (++s == STAGES) { s = 0; phase ^= 1; }
                                }
                            }
                        }
                    }
                    continue;
                }
                const int m0 = tm * GM, ow0 = tw * p.PW + rank * p.split_w, oh0 = th * p.PH + rank * p.split_h, n0 = tn * p.PN + rank * p.split_n;
                if (HALO) {
                    for (int l = 0; l < p.LK && ok; ++l) {
                        for (int cs = 0; cs < c_steps && ok; ++cs) {
                            ok = warp_wait_bounded(halo_empty + 8 * hs, hphase, status, ST_G_PRODUCER);
                            if (!ok) break;
                            if (el && PAIR) {
                                if (rank == 0) mbar_arrive_expect_tx(halo_full + 8 * hs, 2 * (uint32_t)p.Wt * p.Ht * KS * 2);
                                tma_load_5d_pair(halo_addr + hs * p.halo_bytes, &map_x, cs * KS, ow0 + p.off_w, oh0 + p.off_h, n0, l, map_to_cta(halo_full + 8 * hs, 0));
                            } else if (el) {
                                mbar_arrive_expect_tx(halo_full + 8 * hs, (uint32_t)p.Wt * p.Ht * KS * 2);
                                tma_load_5d(halo_addr + hs * p.halo_bytes, &map_x, cs * KS, ow0 + p.off_w, oh0 + p.off_h, n0, l, halo_full + 8 * hs);   // [Ht][Wt][32 channels]
                            }
                            if (++hs == p.n_stages) { hs = 0; hphase ^= 1; }
                            for (int tap = 0; tap < taps; tap += p.a_taps) {
                                ok = warp_wait_bounded(empty_bar + 8 * s, phase, status, ST_G_PRODUCER);
                                if (!ok) break;
                                if (el && PAIR) {
                                    if (rank == 0) mbar_arrive_expect_tx(full_bar + 8 * s, 2 * STAGE);
                                    tma_load_3d_pair(tiles_addr + s * STAGE, &map_w, l * p.Cp + cs * KS, m0, tap, map_to_cta(full_bar + 8 * s, 0));
                                } else if (el) {
                                    mbar_arrive_expect_tx(full_bar + 8 * s, STAGE);
                                    tma_load_3d(tiles_addr + s * STAGE, &map_w, l * p.Cp + cs * KS, m0, tap, full_bar + 8 * s);   // [taps][128 rows][32 channels]
                                }
                                if (++s == STAGES) { s = 0; phase ^= 1; }
                            }
                        }
                    }
                    continue;
                }
                for (int tap = 0; tap < p.KH * p.KW && ok; ++tap) {
                    const int kh = tap / p.KW, kw = tap - kh * p.KW;
                    const int wp0 = ow0 * p.SW + kw * p.DW + p.off_w, hp0 = oh0 * p.SH + kh * p.DH + p.off_h;
                    for (int l = 0; l < p.LK && ok; ++l) {
                        for (int cs = 0; cs < c_steps; ++cs) {
                            ok = warp_wait_bounded(empty_bar + 8 * s, phase, status, ST_G_PRODUCER);
                            if (!ok) break;
                            const uint32_t a_dst = tiles_addr + s * STAGE, bar = full_bar + 8 * s;
                            if (el && PAIR) {
                                const uint32_t lead = map_to_cta(bar, 0);
                                if (rank == 0) mbar_arrive_expect_tx(bar, 2 * (A_BYTES + p.b_tx));
                                tma_load_3d_pair(a_dst, &map_w, l * p.Cp + cs * KS, m0, tap, lead);
                                tma_load_5d_pair(a_dst + A_BYTES, &map_x, cs * KS, wp0, hp0, n0, l, lead);
                            } else if (el) {
                                mbar_arrive_expect_tx(bar, A_BYTES + p.b_tx);
                                tma_load_3d(a_dst, &map_w, l * p.Cp + cs * KS, m0, tap, bar);
                                tma_load_5d(a_dst + A_BYTES, &map_x, cs * KS, wp0, hp0, n0, l, bar);
                            }
                            if (++s == STAGES) { s = 0; phase ^= 1; }
                        }
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        // One elected lane issues (umma.cuh: elect_one); a stage's two descriptors are built once and stepped by adding to the address
        // field of their low words (16-byte units, never carrying out of the field).
        if (rank == 0) {                              // PAIR: the even CTA issues the MMAs of both
            const bool el = elect_one();
            auto mma = [](uint32_t d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t id, uint32_t acc) {
                if (PAIR) mma_f16_pair(d, a_lo, a_hi, b_lo, b_hi, id, acc);
                else mma_f16_ss_words(d, a_lo, a_hi, b_lo, b_hi, id, acc);
            };
            auto commit = [](uint32_t bar) {          // in both CTAs
                if (PAIR) { mma_commit_pair(bar); mma_commit_pair(map_to_cta(bar, 1)); }
                else mma_commit(bar);
            };
            const uint32_t idesc = make_idesc_f16(p.fmt, PAIR ? 2 * GM : GM, DUAL ? GN / 2 : ((HALO || p.exact) ? p.n_cols : GN), false, false);
            int s = 0, phase = 0, hs = 0, hphase = 0, local_tile = 0;
            bool ok = true;
            for (int tile = first; tile < n_tiles && ok; tile += step, ++local_tile) {
                const int buf = local_tile & 1, use = local_tile >> 1;       // use-th time this accumulator buffer is filled
                if (use > 0) {
                    ok = warp_wait_bounded(tmem_empty + 8 * buf, (use - 1) & 1, status, ST_G_MMA);
                    if (!ok) break;
                    tc_fence_after_sync();
                }
                const uint32_t d_tmem = tmem_base + buf * GN;
                if (DUAL) {
                    const int a = first_class ^ (tile / (tiles_px * tiles_m)), kh0 = (a + p.PT) & 1;
                    const int inner = p.LK * c_steps, steps = (p.KH - kh0 + 1) / 2 * p.KW * inner;
                    int kw = 0, left = inner, b = p.PL & 1;
                    uint32_t started = 0;                              // bit b: column class b's accumulator has been written
                    for (int k = 0; k < steps; ++k) {
                        ok = warp_wait_bounded(full_bar + 8 * s, phase, status, ST_G_MMA);
                        if (!ok) break;
                        tc_fence_after_sync();
                        const uint32_t a_addr = tiles_addr + s * STAGE;
                        const uint64_t ad = make_desc_kmajor_rows<KS>(a_addr), bd = make_desc_kmajor_rows<KS>(a_addr + A_BYTES);
                        if (el) {
#pragma unroll
                            for (int j = 0; j < KS / 16; ++j)
                                mma(d_tmem + b * (GN / 2), (uint32_t)ad + 2 * j, (uint32_t)(ad >> 32), (uint32_t)bd + 2 * j, (uint32_t)(bd >> 32),
                                                 idesc, (j > 0 || ((started >> b) & 1u)) ? 1u : 0u);
                            commit(empty_bar + 8 * s);
                            if (k == steps - 1) commit(tmem_full + 8 * buf);
                        }
                        started |= 1u << b;
                        if (++s == STAGES) { s = 0; phase ^= 1; }
                        if (--left == 0) { left = inner; b ^= 1; if (++kw == p.KW) { kw = 0; b = p.PL & 1; } }
                    }
                    continue;
                }
                if (HALO) {
                    const uint32_t row_step = (uint32_t)(p.DH * p.Wt * KS * 2) >> 4, col_step = (uint32_t)(p.DW * KS * 2) >> 4;
                    for (int k = 0; k < n_k && ok; ++k) {
                        ok = warp_wait_bounded(halo_full + 8 * hs, hphase, status, ST_G_MMA);
                        if (!ok) break;
                        const uint64_t bd = make_desc_kmajor_sw64_groups(halo_addr + hs * p.halo_bytes, p.Wt * KS * 2);
                        const uint32_t b_hi = (uint32_t)(bd >> 32);
                        uint32_t b_row = (uint32_t)bd, b_tap = b_row;
                        int kw = 0;
                        for (int tap = 0; tap < taps && ok; tap += p.a_taps) {
                            ok = warp_wait_bounded(full_bar + 8 * s, phase, status, ST_G_MMA);
                            if (!ok) break;
                            tc_fence_after_sync();
                            const uint64_t ad = make_desc_kmajor_rows<KS>(tiles_addr + s * STAGE);
                            if (el) {
                                uint32_t a_lo = (uint32_t)ad, b_lo = b_tap;
                                const uint32_t a_hi = (uint32_t)(ad >> 32);
                                for (int i = 0; i < p.a_taps; ++i) {
#pragma unroll
                                    for (int j = 0; j < KS / 16; ++j)
                                        mma(d_tmem, a_lo + 2 * j, a_hi, b_lo + 2 * j, b_hi, idesc, (k > 0 || tap + i > 0 || j > 0) ? 1u : 0u);
                                    a_lo += A_BYTES >> 4;
                                    b_lo += col_step;
                                }
                                commit(empty_bar + 8 * s);
                            }
                            // (a slot's taps lie in one filter row)
                            if ((kw += p.a_taps) == p.KW) { kw = 0; b_row += row_step; b_tap = b_row; } else b_tap += col_step;
                            if (++s == STAGES) { s = 0; phase ^= 1; }
                        }
                        if (el) {
                            commit(halo_empty + 8 * hs);
                            if (k == n_k - 1) commit(tmem_full + 8 * buf);
                        }
                        if (++hs == p.n_stages) { hs = 0; hphase ^= 1; }
                    }
                    continue;
                }
                for (int k = 0; k < n_k && ok; ++k) {
                    ok = warp_wait_bounded(full_bar + 8 * s, phase, status, ST_G_MMA);
                    if (!ok) break;
                    tc_fence_after_sync();
                    const uint32_t a_addr = tiles_addr + s * STAGE;
                    const uint64_t ad = make_desc_kmajor_rows<KS>(a_addr), bd = make_desc_kmajor_rows<KS>(a_addr + A_BYTES);
                    const uint32_t a_lo = (uint32_t)ad, a_hi = (uint32_t)(ad >> 32), b_lo = (uint32_t)bd, b_hi = (uint32_t)(bd >> 32);
                    if (el) {
#pragma unroll
                        for (int j = 0; j < KS / 16; ++j)
                            mma(d_tmem, a_lo + 2 * j, a_hi, b_lo + 2 * j, b_hi, idesc, (k > 0 || j > 0) ? 1u : 0u);
                        commit(empty_bar + 8 * s);
                        if (k == n_k - 1) commit(tmem_full + 8 * buf);
                    }
                    if (++s == STAGES) { s = 0; phase ^= 1; }
                }
            }
        }
        __syncwarp();
    } else {
        // ---------------------------------------------------------------- epilogue (warps 2..9)
        const int q = warp & 3;                    // TMEM lane quadrant
        const int chalf = (warp - 2) >> 2;         // which 128 of the 256 columns
        const int sv = p.store_vec;                // pixels per store instruction: 16, 8, 4, 2 or 1
        const bool issuer = warp == 2 && lane == 0;
        const int HWo = p.HO * p.WO;
        const int ePW = DUAL ? 2 * p.PW : p.PW, eLW = DUAL ? p.lw + 1 : p.lw;
        constexpr int ROW_STEP = DUAL ? 2 : 1;
        int local_tile = 0, epi_phase = 0;
        bool ok = true;
        // all eight warps meet; bounded like every other wait of the kernel
        auto epi_sync = [&]() {
            __syncwarp();
            if (lane == 0) mbar_arrive(epi_bar);
            const bool done = mbar_wait_bounded(epi_bar, epi_phase & 1, status, ST_G_EPILOGUE);
            ++epi_phase;
            return __all_sync(0xffffffffu, done);
        };
        for (int tile = first; tile < n_tiles && ok; tile += step, ++local_tile) {
            const int buf = local_tile & 1, use = local_tile >> 1;
            const int tm = PAIR ? 2 * (tile % tiles_m) + rank : tile % tiles_m;
            int rest = tile / tiles_m;
            const int tw = rest % p.tiles_w; rest /= p.tiles_w;
            const int th = rest % p.tiles_h;
            int tn = rest / p.tiles_h, cls = 0;
            if (DUAL) { cls = tn / p.tiles_n; tn -= cls * p.tiles_n; }
            // DUAL: the two accumulators interleave to rows of 2 PW output pixels, two output rows apart
            const int ow0 = tw * ePW, oh0 = DUAL ? 2 * th * p.PH + (first_class ^ cls) : th * p.PH, n0 = tn * p.PN;
            const int m = tm * GM + q * 32 + lane;
            const bool row_ok = m < p.Mvalid;
            const int d = row_ok ? m / p.Cout : 0, co = m - d * p.Cout;
            float badd = 0.f;
            if (row_ok && p.has_bias) {
                const uint16_t raw = ld_chained(bias + d * p.bias_ld + co);
                badd = p.fmt == 0 ? __half2float(__ushort_as_half(raw)) : __bfloat162float(__ushort_as_bfloat16(raw));
            }
            const int seen = read_status(status);
            ok = mbar_wait_bounded(tmem_full + 8 * buf, use & 1, status, ST_G_EPILOGUE);
            ok = warp_may_store(ok, seen);
            if (!ok) break;
            tc_fence_after_sync();
            if (p.plane_mode) {
                // Small planes (14 x 14, 7 x 7): a thread's 32 columns are a few short runs of its channel's plane, and
                // 32 lanes scatter them over 32 planes -- stores of 2 to 8 bytes that cost more than the tile's MMAs.
                // The valid pixels are packed [image][row][plane] in shared memory instead; the 128 rows of a tile are 128
                // consecutive channels of one component, so each image of the tile is ONE contiguous range of the output.
                if (issuer) bulk_wait_read_all();                  // the previous tile has left the staging buffer
                ok = epi_sync();
                if (!ok) break;
                uint16_t* mine = reinterpret_cast<uint16_t*>(plane_buf) + (size_t)(q * 32 + lane) * HWo;
#pragma unroll 1
                for (int cb = 0; cb < 4; ++cb) {
                    uint32_t v[32];
                    const int col0 = chalf * 128 + cb * 32;
                    tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + buf * GN + col0, v);
                    tmem_ld_wait();
                    if (p.exact) {
                        if (col0 >= p.n_cols) continue;
                        if ((HWo & 1) == 0 && (!PAIR || (p.half_valid & 1) == 0)) plane_pack_exact<PAIR, true>(v, col0, p, mine, HWo, badd);
                        else plane_pack_exact<PAIR, false>(v, col0, p, mine, HWo, badd);
                    }
                    else if (p.lw == 3) plane_pack<3>(v, col0, p, mine, HWo, badd);
                    else plane_pack<4>(v, col0, p, mine, HWo, badd);
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) { if (PAIR) mbar_arrive_cluster(map_to_cta(tmem_empty + 8 * buf, 0)); else mbar_arrive(tmem_empty + 8 * buf); }
                fence_proxy_async_smem();
                ok = epi_sync();
                if (!ok) break;
                if (issuer) {
                    const int m0 = tm * GM, d0 = m0 / p.Cout, co0 = m0 - d0 * p.Cout;
                    for (int nl = 0; nl < p.PN; ++nl)
                        if (n0 + nl < p.Nb)
                            bulk_store_1d(out + ((size_t)(d0 * p.Nb + n0 + nl) * p.Cout + co0) * HWo,
                                          smem_u32(plane_buf) + (uint32_t)nl * GM * HWo * 2, (uint32_t)GM * HWo * 2);
                    bulk_commit_group();
                }
                continue;
            }
#pragma unroll 1
            for (int cb = 0; cb < 4; ++cb) {
                uint32_t v[32];
                const int col0 = chalf * 128 + cb * 32;
                if (DUAL) {
                    uint32_t even[16], odd[16];
                    const uint32_t at = tmem_base + ((uint32_t)(q * 32) << 16) + buf * GN + col0 / 2;
                    tmem_ld_32x32b_x16(at, even);
                    tmem_ld_32x32b_x16(at + GN / 2, odd);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e) { v[2 * e] = even[e]; v[2 * e + 1] = odd[e]; }
                } else {
                    tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + buf * GN + col0, v);
                    tmem_ld_wait();
                }
                if (!row_ok && !p.rows_epi) continue;
                // convert the 32 columns once, then store runs of 16 pixels (32 bytes) where a run stays inside one
                // output row and rows are 32-byte aligned, runs of 8 pixels (16 bytes) where rows are 16-byte aligned,
                // single elements otherwise
                uint32_t packed[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float f0 = __uint_as_float(v[2 * e]) + badd, f1 = __uint_as_float(v[2 * e + 1]) + badd;
                    if (p.fmt == 0) { const __half2 h = __floats2half2_rn(f0, f1); packed[e] = *reinterpret_cast<const uint32_t*>(&h); }
                    else { const __nv_bfloat162 h = __floats2bfloat162_rn(f0, f1); packed[e] = *reinterpret_cast<const uint32_t*>(&h); }
                }
                if (p.rows_epi) {
                    const uint32_t tbuf = smem_u32(plane_buf) + (uint32_t)(warp - 2) * EPI_ROWS_BYTES;
                    const int row_off = row_ok ? (d * p.Nb * p.Cout + co) * HWo : -1;
                    const int je = col0 + (sv == 1 ? lane : (sv == 2 ? (lane & 15) * 2 : (lane & 7) * 4));
                    const int wl = je & (ePW - 1), hl = p.lh >= 0 ? ((je >> eLW) & (p.PH - 1)) : (je >> eLW), nl = p.lh >= 0 ? (je >> (eLW + p.lh)) : 0;
                    const int ow = ow0 + wl, oh = oh0 + hl * ROW_STEP, img = n0 + nl;
                    const int pix_off = (je < p.n_cols && ow < p.WO && oh < p.HO && img < p.Nb) ? (img * p.Cout * p.HO + oh) * p.WO + ow : -1;
                    if (sv == 1) store_rows<1>(tbuf, packed, out, row_off, pix_off, lane);
                    else if (sv == 2) store_rows<2>(tbuf, packed, out, row_off, pix_off, lane);
                    else store_rows<4>(tbuf, packed, out, row_off, pix_off, lane);
                    continue;
                }
                if (p.o_cl32) {
                    // channels-last output, 32 consecutive channels per warp: the 32 x 32 block goes through 2 KB of shared memory
                    // ([pixel][32 channels]) and leaves as 16-byte stores, 64 contiguous bytes per pixel (the strided path below
                    // writes one 2-byte element per store instruction)
                    const uint32_t tbuf = smem_u32(plane_buf) + (uint32_t)(warp - 2) * 2048u;
                    __syncwarp();
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        st_shared_u16(tbuf + (2 * e) * 64 + lane * 2, (uint16_t)(packed[e] & 0xffffu));
                        st_shared_u16(tbuf + (2 * e + 1) * 64 + lane * 2, (uint16_t)(packed[e] >> 16));
                    }
                    __syncwarp();
                    const int row0 = tm * GM + q * 32, d0 = row0 / p.Cout, cch = row0 - d0 * p.Cout + (lane & 3) * 8;
#pragma unroll
                    for (int it = 0; it < 4; ++it) {
                        const int px = it * 8 + (lane >> 2), je = col0 + px;
                        if (je >= p.n_cols) continue;
                        const int wl = je & (ePW - 1), hl = p.lh >= 0 ? ((je >> eLW) & (p.PH - 1)) : (je >> eLW), nl = p.lh >= 0 ? (je >> (eLW + p.lh)) : 0;
                        const int ow = ow0 + wl, oh = oh0 + hl * ROW_STEP, img = n0 + nl;
                        if (ow >= p.WO || oh >= p.HO || img >= p.Nb) continue;
                        const uint4 val = ld_shared_v4(tbuf + px * 64 + (lane & 3) * 16);
                        *reinterpret_cast<uint4*>(out + (size_t)(d0 * p.Nb + img) * p.o_p + (size_t)oh * p.o_h + (size_t)ow * p.o_w + cch) = val;
                    }
                    continue;
                }
                const bool wide = !p.o_generic && sv >= 16 && (ePW % 16) == 0;
#pragma unroll
                for (int g8 = 0; g8 < 4; ++g8) {
                    if (wide && (g8 & 1)) continue;                      // the odd groups were written with their even neighbours
                    const int j = col0 + g8 * 8;                         // column -> (image, row, pixel) of the tile box
                    if (j >= p.n_cols) continue;
                    if (p.o_generic) {
                        // Output addressed through element strides: channels-last tensors (consecutive lanes hold consecutive
                        // channels, so a warp's stores of one pixel are contiguous), channel slices of grouped layers, and boxes
                        // narrower than 8 pixels (dense layers are 1 x 1 images: the columns are batch rows). Every column is
                        // decoded on its own.
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const int je = j + e;
                            if (je >= p.n_cols) continue;
                            const int wl = je & (ePW - 1), hl = p.lh >= 0 ? ((je >> eLW) & (p.PH - 1)) : (je >> eLW), nl = p.lh >= 0 ? (je >> (eLW + p.lh)) : 0;
                            const int ow = ow0 + wl, oh = oh0 + hl * ROW_STEP, img = n0 + nl;
                            if (ow >= p.WO || oh >= p.HO || img >= p.Nb) continue;
                            out[(size_t)(d * p.Nb + img) * p.o_p + (size_t)co * p.o_c + (size_t)oh * p.o_h + (size_t)ow * p.o_w] =
                                (uint16_t)((packed[4 * g8 + (e >> 1)] >> ((e & 1) * 16)) & 0xffffu);
                        }
                        continue;
                    }
                    // PW is a power of two; PH too unless the tile is one image tall (PN == 1, halo mode)
                    const int wl = j & (ePW - 1), hl = p.lh >= 0 ? ((j >> eLW) & (p.PH - 1)) : (j >> eLW), nl = p.lh >= 0 ? (j >> (eLW + p.lh)) : 0;
                    const int ow = ow0 + wl, oh = oh0 + hl * ROW_STEP, img = n0 + nl;
                    if (ow >= p.WO || oh >= p.HO || img >= p.Nb) continue;
                    uint16_t* dst = out + (((size_t)(d * p.Nb + img) * p.Cout + co) * p.HO + oh) * p.WO + ow;
                    if (wide) {
                        st_global_v8(dst, &packed[4 * g8]);
                    } else {                       // rows are 16-byte aligned (all others: store_rows)
                        *reinterpret_cast<uint4*>(dst) = make_uint4(packed[4 * g8], packed[4 * g8 + 1], packed[4 * g8 + 2], packed[4 * g8 + 3]);
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) { if (PAIR) mbar_arrive_cluster(map_to_cta(tmem_empty + 8 * buf, 0)); else mbar_arrive(tmem_empty + 8 * buf); }
        }
        if (issuer) bulk_wait_read_all();                           // shared memory must outlive the last bulk store's reads
    }

    tc_fence_before_sync();
    __syncthreads();
    if (PAIR) cluster_sync_all();                     // nobody leaves while its peer may still signal its barriers or read its shared memory
    if (warp == 1) { if (PAIR) tmem_dealloc_pair(tmem_base, 512); else tmem_dealloc(tmem_base, 512); }
}

// ---- staging kernels ------------------------------------------------------------------------------
// xp[comp][img][hp][wp][c] = x[comp][img][c][hp - pad_top][wp - pad_left] (zero outside, zero for c >= C).
// One thread per (pixel, 8-channel group): reads are coalesced along w, writes are 16-byte vectors.
// The source is addressed through element strides (plane, channel, row, pixel), so it may be NCHW, channels-last, or a
// channel slice of a wider tensor (one group of a grouped layer).
struct SrcStrides { long long p, c, h, w; };
template <typename T>
__global__ void pack_activations_kernel(const T* __restrict__ x, T* __restrict__ xp, int planes /*4*Nb*/, int C, int H, int W,
                                        int Hp, int Wp, int Cp, int pad_top, int pad_left, int ins_h, int ins_w, int cb, int Nb, SrcStrides ss) {
    const int groups = Cp / 8;
    const unsigned total = (unsigned)planes * Hp * Wp * groups;       // 32-bit indices: the staged copy is capped at 8 GB
    for (unsigned idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
        // wp fastest so that a warp reads consecutive pixels of one channel
        const int wp = (int)(idx % Wp);
        unsigned rest = idx / Wp;
        const int grp = (int)(rest % groups); rest /= groups;
        const int hp = (int)(rest % Hp);
        const int plane = (int)(rest / Hp);
        // ins_h / ins_w > 1 spread the source pixels ins apart with zeros between them (the zero-insertion that
        // turns the backward-data pass of a strided convolution into a stride-1 correlation)
        int ih = hp - pad_top, iw = wp - pad_left;
        bool inside = ih >= 0 && iw >= 0;
        if (inside && (ins_h > 1 || ins_w > 1)) {
            inside = (ih % ins_h == 0) && (iw % ins_w == 0);
            ih /= ins_h; iw /= ins_w;
        }
        inside = inside && ih < H && iw < W;
        alignas(16) T vals[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int c = grp * 8 + e;
            T v = T(0.f);
            if (c < C && inside) v = x[(long long)plane * ss.p + (long long)c * ss.c + (long long)ih * ss.h + (long long)iw * ss.w];
            vals[e] = v;
        }
        T* dst = xp + (((size_t)plane * Hp + hp) * Wp + wp) * Cp + grp * 8;
        if (cb > 0) {   // blocks of cb channels, block index outermost: xp[comp * (Cp / cb) + c / cb][img][hp][wp][cb]
            const int comp = plane / Nb, img = plane - comp * Nb, b = (grp * 8) / cb;
            dst = xp + (((((size_t)comp * (Cp / cb) + b) * Nb + img) * Hp + hp) * Wp + wp) * cb + (grp * 8 - b * cb);
        }
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(vals);
    }
}

// The general staging through shared memory for dense NCHW sources whose plane (all channels of one image and component,
// one contiguous block of C * H * W elements) fits there: the block is read once with coalesced 16-byte loads, and the
// padded / zero-inserted / channel-blocked copy is written from it with the channel groups of a pixel on neighbouring
// threads, so that a warp writes whole pixels (Cp * 2 contiguous bytes each). One CTA per plane. The general kernel above
// reads 2-byte elements H * W apart, which on 7 x 7 planes and on zero-inserted copies runs at a quarter of this.
constexpr int PACK_SMEM_THREADS = 256;
constexpr size_t PACK_SMEM_MAX_BYTES = 96 * 1024;               // two CTAs per SM
template <typename T>
__global__ void __launch_bounds__(PACK_SMEM_THREADS)
pack_activations_smem_kernel(const T* __restrict__ x, T* __restrict__ xp, int C, int H, int W, int Hp, int Wp, int Cp, int pad_top, int pad_left,
                             int ins_h, int ins_w, int cb, int Nb, int scatter) {
    extern __shared__ __align__(16) uint8_t pack_smem[];
    T* tile = reinterpret_cast<T*>(pack_smem);                   // [C][H * W]
    const int plane = blockIdx.x, HW = H * W, n = C * HW;
    const T* src = x + (size_t)plane * n;
    if ((n & 7) == 0) {                                          // every plane starts on a 16-byte boundary (the tensor does)
        for (int i = threadIdx.x; i < n / 8; i += PACK_SMEM_THREADS)
            reinterpret_cast<uint4*>(tile)[i] = __ldg(reinterpret_cast<const uint4*>(src) + i);
    } else {
        for (int i = threadIdx.x; i < n; i += PACK_SMEM_THREADS) tile[i] = src[i];
    }
    __syncthreads();
    // scatter: the copy was zeroed beforehand (zero-inserted copies are three quarters zeros) and only the source pixels are
    // visited and written to their places; otherwise every element of the copy is visited and written
    const int groups = Cp / 8, items = (scatter ? H * W : Hp * Wp) * groups;
    const int comp = plane / Nb, img = plane - comp * Nb;
    for (int idx = threadIdx.x; idx < items; idx += PACK_SMEM_THREADS) {
        const int grp = idx % groups, pix = idx / groups;
        int hp, wp, ih, iw;
        bool inside;
        if (scatter) {
            ih = pix / W; iw = pix - ih * W;
            hp = pad_top + ih * ins_h; wp = pad_left + iw * ins_w;
            if (hp < 0 || hp >= Hp || wp < 0 || wp >= Wp) continue;
            inside = true;
        } else {
            hp = pix / Wp; wp = pix - hp * Wp;
            ih = hp - pad_top; iw = wp - pad_left;
            inside = ih >= 0 && iw >= 0;
            if (inside && (ins_h > 1 || ins_w > 1)) {
                inside = (ih % ins_h == 0) && (iw % ins_w == 0);
                ih /= ins_h; iw /= ins_w;
            }
            inside = inside && ih < H && iw < W;
        }
        alignas(16) T vals[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int c = grp * 8 + e;
            vals[e] = (inside && c < C) ? tile[c * HW + ih * W + iw] : T(0.f);
        }
        T* dst = xp + (((size_t)plane * Hp + hp) * Wp + wp) * Cp + grp * 8;
        if (cb > 0) {
            const int b = (grp * 8) / cb;
            dst = xp + (((((size_t)comp * (Cp / cb) + b) * Nb + img) * Hp + hp) * Wp + wp) * cb + (grp * 8 - b * cb);
        }
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(vals);
    }
}

// The staging of dense NCHW tensors: x[plane][C][HW] -> xp[plane][HW][Cp] (blocked == 0) or blocks of 8 U channels with the block
// index outermost, xp[comp * nblk + block][img][HW][8 U] -- a batched transposition without padding (the tensor maps supply it as
// zero fill). A CTA takes 1024 / U consecutive pixels (across planes) of one block of 8 U channels: a thread loads V pixels of
// 8 channels (coalesced along the pixels; V divides HW, so the pixels lie in one plane and the address is aligned), turns them in
// registers into V 16-byte units of 8 channels, and the units leave through shared memory, 16 U contiguous bytes per
// pixel. Bound by memory: 51 MB of
// 14 x 14 planes 38 -> 18 us, 28 x 28 planes of 128 channels (103 MB) 56 -> 36 us against a thread per pixel group and 8 channels that
// wrote its units itself.
struct StageJob {
    const void* x;
    void* xp;
    unsigned total_px, HW, Nb;      // pixels of all planes, of one plane; images per component
    size_t plane;                   // elements between the planes of x (more than C * HW: a channel slice of a wider tensor)
    int C, nblk, U, V;              // channels, blocks of 8 U channels, pixels per load (0: a channels-last source, -1: tiny planes)
    int blocked;
    unsigned bx, blocks;            // CTAs along the pixels; all CTAs
};
template <int V, int U>
__device__ __forceinline__ void stage_compact(const StageJob& p, unsigned block, uint4* tile /*[STAGE_UNITS]*/) {
    constexpr int TPX = STAGE_UNITS / U;
    const uint16_t* x = static_cast<const uint16_t*>(p.x);
    uint4* __restrict__ xp = static_cast<uint4*>(p.xp);
    const unsigned total_px = p.total_px, HW = p.HW, by = block / p.bx;
    const int C = p.C, nblk = p.nblk;
    const unsigned px0 = (block - by * p.bx) * TPX;
    const int c0 = by * 8 * U;
#pragma unroll
    for (int it = 0; it < STAGE_UNITS / V / STAGE_THREADS; ++it) {
        const int item = threadIdx.x + it * STAGE_THREADS, l = item % (TPX / V), g = item / (TPX / V);
        const unsigned P = px0 + l * V;
        uint32_t raw[8][V == 4 ? 2 : 1];
        const unsigned plane = P / HW;
        const uint16_t* src = x + plane * p.plane + (size_t)(c0 + 8 * g) * HW + (P - plane * HW);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const bool ok = P < total_px && c0 + 8 * g + e < C;
            if (V == 4) {
                const uint2 w = ld_chained(reinterpret_cast<const uint2*>(src + (size_t)e * HW), ok);
                raw[e][0] = w.x; raw[e][V == 4 ? 1 : 0] = w.y;
            } else if (V == 2) {
                raw[e][0] = ld_chained(reinterpret_cast<const uint32_t*>(src + (size_t)e * HW), ok);
            } else {
                raw[e][0] = ld_chained(src + (size_t)e * HW, ok);
            }
        }
#pragma unroll
        for (int j = 0; j < V; ++j) {
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = __byte_perm(raw[2 * i][j / 2], raw[2 * i + 1][j / 2], (j & 1) ? 0x7632 : 0x5410);
            tile[stage_unit<V, U>(l * V + j, g)] = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < STAGE_UNITS / STAGE_THREADS; ++it) {
        const int i = threadIdx.x + it * STAGE_THREADS, px = i / U, g = i % U;
        const unsigned P = px0 + px;
        if (P >= total_px) continue;
        size_t unit;
        if (p.blocked) {
            const unsigned comp = P / HW / p.Nb;                     // pixel of plane (comp * nblk + block) * Nb + img
            unit = ((size_t)P + (size_t)(comp * (unsigned)(nblk - 1) + by) * p.Nb * HW) * U + g;
        } else {
            unit = ((size_t)P * nblk + by) * U + g;
        }
        xp[unit] = tile[stage_unit<V, U>(px, g)];
    }
}
template <int U>
__device__ __forceinline__ void stage_compact(const StageJob& p, unsigned block, uint4* tile) {
    if (p.V == 4) stage_compact<4, U>(p, block, tile);
    else if (p.V == 2) stage_compact<2, U>(p, block, tile);
    else stage_compact<1, U>(p, block, tile);
}
// Channels are taken in slices of 64, 32 or 16, and their number is padded to whole slices (zeros in the filter matrix, and in the
// staged copy or by the zero fill of the tensor map). A TMA copy costs about the same whatever its size and moves rows of one slice,
// so 16-channel slices are kept for layers of at most 16 channels: 48 channels as one slice of 64 instead of three of 16 take a
// 3x3 forward pass (44 images of 39 x 47, 40 output channels) from 164 to 105 us although a quarter of the products are zeros.
// `tight` (see Geom): the fewest channels, a multiple of 16.
int padded_channels(int c, bool tight) { return round_up(c, c <= 16 || tight ? 16 : (round_up(c, 32) % 64 == 0 ? 64 : 32)); }
int channel_slice(int c, bool tight) { const int p = padded_channels(c, tight); return p % 64 == 0 ? 64 : (p % 32 == 0 ? 32 : 16); }

// Channels-last sources that have to be copied (padded to slices, or cut into blocks of 8 U channels for the filter gradient): 16-byte
// units, C a multiple of 8. Destination as for stage_compact.
__device__ __forceinline__ void repack_channels_last(const StageJob& p, unsigned block) {
    const uint4* x = static_cast<const uint4*>(p.x);
    uint4* __restrict__ xp = static_cast<uint4*>(p.xp);
    const unsigned per_px = (unsigned)(p.nblk * p.U), src_units = (unsigned)p.C / 8;
    const size_t total = (size_t)p.total_px * per_px;
    for (size_t i = (size_t)block * STAGE_THREADS + threadIdx.x; i < total; i += (size_t)p.blocks * STAGE_THREADS) {
        const unsigned P = (unsigned)(i / per_px), u = (unsigned)(i - (size_t)P * per_px);
        const uint4 v = ld_chained(x + (size_t)P * src_units + u, u < src_units);
        size_t dst = i;
        if (p.blocked) {
            const unsigned comp = P / p.HW / p.Nb, b = u / p.U;
            dst = ((size_t)P + (size_t)(comp * (unsigned)(p.nblk - 1) + b) * p.Nb * p.HW) * p.U + (u - b * p.U);
        }
        xp[dst] = v;
    }
}

// NCHW planes of fewer than 16 pixels: a thread per pixel and 8 channels, consecutive threads along the pixels of a plane and then its
// channel groups. (The batched transposition loads along the pixels, of which there are too few.)
__device__ __forceinline__ void stage_tiny(const StageJob& p, unsigned block) {
    const uint16_t* x = static_cast<const uint16_t*>(p.x);
    uint4* __restrict__ xp = static_cast<uint4*>(p.xp);
    const unsigned groups = (unsigned)(p.nblk * p.U), HW = p.HW;
    const size_t total = (size_t)p.total_px * groups;
    for (size_t i = (size_t)block * STAGE_THREADS + threadIdx.x; i < total; i += (size_t)p.blocks * STAGE_THREADS) {
        const unsigned px = (unsigned)(i % HW), grp = (unsigned)(i / HW % groups), plane = (unsigned)(i / HW / groups);
        const uint16_t* src = x + plane * p.plane + (size_t)(8 * grp) * HW + px;
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
            w[e] = (uint32_t)ld_chained(src + (size_t)(2 * e) * HW, (int)(8 * grp) + 2 * e < p.C) |
                   (uint32_t)ld_chained(src + (size_t)(2 * e + 1) * HW, (int)(8 * grp) + 2 * e + 1 < p.C) << 16;
        const size_t P = (size_t)plane * HW + px;
        size_t dst = P * groups + grp;
        if (p.blocked) {
            const unsigned comp = plane / p.Nb, b = grp / p.U;
            dst = (P + (size_t)(comp * (unsigned)(p.nblk - 1) + b) * p.Nb * HW) * p.U + (grp - b * p.U);
        }
        xp[dst] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Forward:       Wexp[tap][m = d*Co + co][k = l*Cp + ci]  = s(l,d) * w[l^d][co][ci][tap]
// Backward-data: Wexp[tap][m = l*Ci + ci][k = d*Cop + co] = s(l,d) * w[l^d][co][ci][taps-1-tap]   (flipped taps)
// The filters are addressed through element strides (component, output channel, input channel, tap row, tap column): OIHW, OHWI,
// HWIO, the input-major dense layout, or the slice of one group.
struct FilterStrides { long long r, o, i, h, w; int KW; };
struct FilterJob {
    const uint16_t* w;
    uint16_t* wexp;
    int Co, Ci, taps, Mp, Kp, Cp /*padded channels of the reduced side*/, transposed, nc, ga;
    unsigned long long neg;
    FilterStrides fs;
    int tiled, tap_split;          // the tiled form below: CTAs per (tile, component)
    unsigned bx, by, blocks;
};
// 16-bit elements are moved as raw bits; a negative coefficient flips the sign bit.
__device__ __forceinline__ void pack_filters_rows(const FilterJob& p, unsigned block) {
    // one row (tap, m) of the expanded matrix per wx threads; the row is decoded once, its threads walk k
    const int Cm = p.transposed ? p.Ci : p.Co;     // channels on the M side
    const int Ck = p.transposed ? p.Co : p.Ci;     // channels on the K side
    const int wx = p.Cp >= 64 ? 64 : 32, tx = threadIdx.x % wx, ty = threadIdx.x / wx, wy = STAGE_THREADS / wx;
    const int rows = p.taps * p.Mp;
    for (int row = block * wy + ty; row < rows; row += p.blocks * wy) {
        const int tap = row / p.Mp, m = row - tap * p.Mp;
        const int cm_comp = m / Cm, cm = m - cm_comp * Cm;
        const int src_tap = p.transposed ? p.taps - 1 - tap : tap;
        uint16_t* dst = p.wexp + (size_t)row * p.Kp;
        for (int ck_comp = 0, k0 = 0; k0 < p.Kp; ++ck_comp, k0 += p.Cp) {
            const int d = p.transposed ? ck_comp : cm_comp, l = p.transposed ? cm_comp : ck_comp;
            const bool comp_ok = cm_comp < p.nc && ck_comp < p.nc;
            const uint16_t flip = (comp_ok && alg_negative(p.neg, l, d)) ? 0x8000u : 0u;
            // forward: w[r][co = cm][ci = ck][tap]; backward-data: w[r][co = ck][ci = cm][tap]
            const uint16_t* src = nullptr;
            const long long ck_stride = p.transposed ? p.fs.o : p.fs.i;
            if (comp_ok) {
                const int kh = src_tap / p.fs.KW, kw = src_tap - kh * p.fs.KW;
                src = p.w + (long long)alg_pair(p.ga, l, d) * p.fs.r + (long long)kh * p.fs.h + (long long)kw * p.fs.w + (long long)cm * (p.transposed ? p.fs.i : p.fs.o);
            }
            for (int ck = tx; ck < p.Cp; ck += wx) dst[k0 + ck] = (comp_ok && ck < Ck) ? (uint16_t)(ld_chained(src + ck * ck_stride) ^ flip) : (uint16_t)0;
        }
    }
}

// The same matrix for filters whose (input channel, tap) run is contiguous (OIHW), tile by tile through shared memory: a block
// takes one filter component r and a 32 x 64 block of (M-side, K-side) channels with all its taps, reads it as whole runs
// (coalesced, where the row-per-thread kernel above strides by a whole output channel in the transposed case), and writes, for
// every (l, d) pair whose product component is r, 64 consecutive K columns per row. Requires taps <= PACK_TILE_MAX_TAPS and no
// padded rows beyond the last component (Mp == nc * Cm).
constexpr int PACK_TM = 32, PACK_TK = 64;   // rows (M-side channels) and K columns of a tile
constexpr int PACK_TILE_MAX_TAPS = 9;     // 37 KB of shared memory at 9 taps
// (every thread writes 8 consecutive K columns with one 16-byte store)
__device__ __forceinline__ void pack_filters_tile(const FilterJob& p, unsigned block, uint16_t* tile) {
    const uint16_t* w = p.w;
    uint16_t* __restrict__ wexp = p.wexp;
    const int Co = p.Co, Ci = p.Ci, taps = p.taps, Mp = p.Mp, Kp = p.Kp, Cp = p.Cp, transposed = p.transposed, nc = p.nc, ga = p.ga, tap_split = p.tap_split;
    const unsigned long long neg = p.neg;
    const FilterStrides& fs = p.fs;
    const int Cm = transposed ? Ci : Co, Ck = transposed ? Co : Ci;
    // small layers have few tiles: then the last block index also splits the taps a block WRITES (every block still reads whole runs)
    const int bx = block % p.bx, by = block / p.bx % p.by, bz = block / p.bx / p.by;
    const int ck0 = bx * PACK_TK, cm0 = by * PACK_TM, r = bz / tap_split, tpart = bz - r * tap_split;
    const int taps_per = (taps + tap_split - 1) / tap_split, tap_beg = tpart * taps_per, tap_end = min(taps, tap_beg + taps_per);
    const int co0 = transposed ? ck0 : cm0, ci0 = transposed ? cm0 : ck0;
    const int n_co = transposed ? PACK_TK : PACK_TM, n_ci = transposed ? PACK_TM : PACK_TK;
    const int run = n_ci * taps;               // elements of the tile's input channels x all taps of one output channel
    const int pitch = run + 2;                 // an odd number of 32-bit words
    {   // load: a warp takes whole runs (one output channel each); a run is a multiple of 32 elements, so the loop unrolls into
        // independent loads
        const int e_limit = min(run, max(0, (Ci - ci0) * taps));      // elements of a run that belong to existing input channels
        const uint16_t* src = w + (long long)r * fs.r + (long long)co0 * fs.o + (long long)ci0 * fs.i;
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        for (int co = warp; co < n_co; co += 8) {
            const uint16_t* row = src + (long long)co * fs.o;
            const int limit = co0 + co < Co ? e_limit : 0;
            uint16_t* trow = tile + co * pitch;
#pragma unroll 9
            for (int e = lane; e < run; e += 32) trow[e] = ld_chained(row + e, e < limit);
        }
    }
    __syncthreads();
    // write: a thread keeps its row cm and its 8 K columns for every tap and every (l, d) pair
    const int j = threadIdx.x & (PACK_TK / 8 - 1), cm = threadIdx.x >> 3;
    const int ck = ck0 + 8 * j;
    if (cm0 + cm >= Cm || ck >= Cp) return;
    const uint16_t* src0 = transposed ? tile + (8 * j) * pitch + cm * taps : tile + cm * pitch + (8 * j) * taps;
    const int step = transposed ? pitch : taps;
    uint32_t keep[4];                     // columns beyond the K-side channel count are zero
#pragma unroll
    for (int t = 0; t < 4; ++t) keep[t] = (ck + 2 * t < Ck ? 0xFFFFu : 0u) | (ck + 2 * t + 1 < Ck ? 0xFFFF0000u : 0u);
    for (int l = 0; l < nc; ++l) {
        int d = -1;
        for (int dd = 0; dd < nc; ++dd)
            if (alg_pair(ga, l, dd) == r) d = dd;
        if (d < 0) continue;
        if ((transposed ? d : l) * Cp >= Kp) continue;      // a real-valued input has one component along K
        const uint32_t flip = alg_negative(neg, l, d) ? 0x80008000u : 0u;
        const int m_comp = transposed ? l : d, k_comp = transposed ? d : l;
        uint16_t* dst = wexp + ((size_t)m_comp * Cm + cm0 + cm) * Kp + (size_t)k_comp * Cp + ck;
        for (int tap = tap_beg; tap < tap_end; ++tap) {
            const uint16_t* src = src0 + (transposed ? taps - 1 - tap : tap);
            uint32_t q[4];
#pragma unroll
            for (int t = 0; t < 4; ++t)
                q[t] = (((uint32_t)src[(2 * t) * step] | ((uint32_t)src[(2 * t + 1) * step] << 16)) ^ flip) & keep[t];
            *reinterpret_cast<uint4*>(dst + (size_t)tap * Mp * Kp) = make_uint4(q[0], q[1], q[2], q[3]);
        }
    }
}

// Everything a convolution needs before its main kernel, in one launch: the device status word of the call, the filter matrix, the
// staged copies, the zeroed accumulator. The jobs are independent and share the machine (the packing is bound by latency, the copies
// by memory). As launches of their own, the packing on a side stream, these cost a small layer more than its convolution:
// 1x1 160 -> 24 channels, 14 x 14, batch 33, bf16, forward + backward: 78 -> 69 us; QResNet-18 step 5478 -> 5210 us.
struct Prologue {
    int* status = nullptr;
    FilterJob filter;
    StageJob stage[2];
    uint4* zero = nullptr;
    unsigned zero_units = 0, filter_blocks = 0, stage_blocks[2] = {0, 0}, zero_blocks = 0;
    int n_stages = 0;
};
__global__ void __launch_bounds__(STAGE_THREADS) prologue_kernel(const __grid_constant__ Prologue p) {
    extern __shared__ __align__(16) uint8_t pack_smem[];
    unsigned block = blockIdx.x;
    chain_wait();
    chain_next();
    if (block == 0 && threadIdx.x == 0 && p.status) *p.status = 0;
    if (block < p.filter_blocks) {
        if (p.filter.tiled) pack_filters_tile(p.filter, block, reinterpret_cast<uint16_t*>(pack_smem));
        else pack_filters_rows(p.filter, block);
        return;
    }
    block -= p.filter_blocks;
    if (block < p.zero_blocks) {
        for (unsigned i = block * STAGE_THREADS + threadIdx.x; i < p.zero_units; i += p.zero_blocks * STAGE_THREADS) p.zero[i] = make_uint4(0u, 0u, 0u, 0u);
        return;
    }
    block -= p.zero_blocks;
    const bool second = block >= p.stage_blocks[0];
    const StageJob& job = second ? p.stage[1] : p.stage[0];
    if (second) block -= p.stage_blocks[0];
    uint4* tile = reinterpret_cast<uint4*>(pack_smem);
    if (job.V == 0) repack_channels_last(job, block);
    else if (job.V < 0) stage_tiny(job, block);
    else if (job.U == 8) stage_compact<8>(job, block, tile);
    else if (job.U == 4) stage_compact<4>(job, block, tile);
    else stage_compact<2>(job, block, tile);
}
void add_filter_job(Prologue& pro, const void* w, void* wexp, int Co, int Ci, int taps, int Mp, int Kp, int Cp, int transposed, int nc, int ga,
                    unsigned long long neg, const FilterStrides& fs) {
    FilterJob& f = pro.filter;
    f.w = static_cast<const uint16_t*>(w); f.wexp = static_cast<uint16_t*>(wexp);
    f.Co = Co; f.Ci = Ci; f.taps = taps; f.Mp = Mp; f.Kp = Kp; f.Cp = Cp; f.transposed = transposed; f.nc = nc; f.ga = ga; f.neg = neg; f.fs = fs;
    const int Cm = transposed ? Ci : Co;
    const bool runs = fs.w == 1 && fs.h == fs.KW && fs.i == taps;
    f.tiled = runs && taps <= PACK_TILE_MAX_TAPS && Mp == nc * Cm && Cm >= PACK_TM && (reinterpret_cast<uintptr_t>(wexp) & 15u) == 0;
    if (f.tiled) {
        f.bx = (Cp + PACK_TK - 1) / PACK_TK; f.by = (Cm + PACK_TM - 1) / PACK_TM;
        f.tap_split = (int)(f.bx * f.by * nc) < sm_count() / 2 ? taps : 1;
        f.blocks = f.bx * f.by * nc * f.tap_split;
    } else {
        f.tap_split = 1;
        f.blocks = grid_cap((size_t)taps * Mp, STAGE_THREADS / (Cp >= 64 ? 64 : 32), 32);
    }
    pro.filter_blocks = f.blocks;
}
void add_zero_job(Prologue& pro, void* p, size_t bytes) {          // a multiple of 16 bytes
    pro.zero = static_cast<uint4*>(p);
    pro.zero_units = (unsigned)(bytes / 16);
    pro.zero_blocks = grid_cap(pro.zero_units, 4 * STAGE_THREADS, 1);
}
// `sc`: the pending reset of the status word, done by this launch.
// `chain`: whether the main kernel may be chained to this launch.
int launch_prologue(Prologue& pro, StatusClear* sc, cudaStream_t stream, bool* chain) {
    const unsigned blocks = pro.filter_blocks + pro.zero_blocks + pro.stage_blocks[0] + pro.stage_blocks[1];
    *chain = chain_behind(blocks, 8);
    if (blocks == 0) return PCB_OK;                                // (nothing to prepare: the caller's status reset stays pending)
    if (sc && sc->pending) { pro.status = sc->word; sc->pending = false; }
    const FilterJob& f = pro.filter;
    size_t smem = pro.n_stages ? STAGE_UNITS * sizeof(uint4) : 0;
    const size_t tile = pro.filter_blocks && f.tiled ? (size_t)(f.transposed ? PACK_TK * (PACK_TM * f.taps + 2) : PACK_TM * (PACK_TK * f.taps + 2)) * 2 : 0;
    if (tile > smem) smem = tile;
    // Not chained where a large filter matrix is gathered element by element (conv_tf32.cu): 14 x 14, batch 16, 256 channels, 5 x 5, fp16,
    // backward-data 333 us chained, 285 not; channels-last 7 x 7, 512 channels, 3 x 3 278 / 258; 256 channels, 3 x 3 (19 MB) 98.5 / 98.5.
    const bool gathers = pro.filter_blocks && !f.tiled && (f.transposed ? f.fs.o : f.fs.i) != 1 && (size_t)f.taps * f.Mp * f.Kp * 2 > (size_t)32 << 20;
    PCB_CUDA_TRY(launch_chained_if(!gathers, prologue_kernel, blocks, STAGE_THREADS, smem, stream, pro));
    PCB_CUDA_TRY(cudaGetLastError());
    return PCB_OK;
}

// Host dispatch of the activation staging: a job of the prologue launch where that form applies, a kernel of its own otherwise. cb > 0 selects the channel-block layout of the filter-gradient kernels (Nb images per
// component). `ss` = nullptr: a dense NCHW source (the fast forms apply); otherwise its element strides.
void stage_activations(Prologue& pro, int fmt, const void* src, void* dst, int planes, int C, int H, int W, int Hp, int Wp, int Cp, int pad_top, int pad_left,
                       int ins_h, int ins_w, int block, cudaStream_t stream, int cb = 0, int Nb = 1, const SrcStrides* ss = nullptr) {
    const size_t total = (size_t)planes * Hp * Wp * (Cp / 8);
    const SrcStrides dense = {(long long)C * H * W, (long long)H * W, (long long)W, 1};
    const SrcStrides st = ss ? *ss : dense;
    const bool compact = Hp == H && Wp == W && pad_top == 0 && pad_left == 0 && ins_h == 1 && ins_w == 1;
    const uintptr_t at = reinterpret_cast<uintptr_t>(src);
    const bool last = (ss ? ss->c == 1 && ss->w == C && ss->h == (long long)W * C && ss->p == (long long)H * W * C : H * W == 1) && C % 8 == 0 && at % 16 == 0;
    // NCHW planes: the whole tensor, or the channel slice of a group (as a thread per pixel and 8 channels, bf16 72 -> 6 channels of two groups,
    // 105 x 105, batch 7, 1 x 1, forward took 198 us instead of 156). Tiny planes up to 16 MB; larger ones are copied faster through
    // shared memory, by a kernel of their own (2 -> 40 channels, 1 x 5, batch 69, filter gradient 31 us with two of those, 21 without).
    const bool nchw = st.w == 1 && st.h == W && st.c == (long long)H * W;
    if (compact && (last || (nchw && (H * W >= 16 || total <= (size_t)1 << 20)))) {
        StageJob& j = pro.stage[pro.n_stages];
        j.x = src; j.xp = dst; j.total_px = (unsigned)planes * H * W; j.HW = H * W; j.Nb = Nb; j.plane = (size_t)st.p;
        j.C = C; j.U = block / 8; j.nblk = Cp / block; j.blocked = cb > 0;
        j.V = last ? 0 : (H * W < 16 ? -1 : (j.HW % 4 == 0 && at % 8 == 0 ? 4 : (j.HW % 2 == 0 && at % 4 == 0 ? 2 : 1)));
        j.bx = (j.total_px + STAGE_UNITS / j.U - 1) / (STAGE_UNITS / j.U);
        j.blocks = j.V <= 0 ? (unsigned)grid_cap(total, STAGE_THREADS, 16) : j.bx * j.nblk;
        pro.stage_blocks[pro.n_stages++] = j.blocks;
    } else if (!ss && (size_t)C * H * W * 2 <= PACK_SMEM_MAX_BYTES && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
        const size_t smem = ((size_t)C * H * W * 2 + 15) / 16 * 16;
        const int scatter = (ins_h > 1 || ins_w > 1) ? 1 : 0;
        if (scatter) cudaMemsetAsync(dst, 0, (size_t)planes * Hp * Wp * Cp * 2, stream);
        if (fmt == 0) {
            cudaFuncSetAttribute(pack_activations_smem_kernel<__half>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PACK_SMEM_MAX_BYTES);
            pack_activations_smem_kernel<__half><<<planes, PACK_SMEM_THREADS, smem, stream>>>((const __half*)src, (__half*)dst, C, H, W, Hp, Wp, Cp, pad_top, pad_left,
                                                                                           ins_h, ins_w, cb, Nb, scatter);
        } else {
            cudaFuncSetAttribute(pack_activations_smem_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PACK_SMEM_MAX_BYTES);
            pack_activations_smem_kernel<__nv_bfloat16><<<planes, PACK_SMEM_THREADS, smem, stream>>>((const __nv_bfloat16*)src, (__nv_bfloat16*)dst, C, H, W, Hp, Wp, Cp,
                                                                                                  pad_top, pad_left, ins_h, ins_w, cb, Nb, scatter);
        }
    } else {
        const int blocks = grid_cap(total, 256, 16);
        if (fmt == 0) pack_activations_kernel<__half><<<blocks, 256, 0, stream>>>((const __half*)src, (__half*)dst, planes, C, H, W, Hp, Wp, Cp, pad_top, pad_left, ins_h, ins_w, cb, Nb, st);
        else pack_activations_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>((const __nv_bfloat16*)src, (__nv_bfloat16*)dst, planes, C, H, W, Hp, Wp, Cp, pad_top, pad_left, ins_h, ins_w, cb, Nb, st);
    }
}

// ===================================================================================================
// General backward-filter. Both operands come from channels-last staged copies (dy unpadded, x padded as for
// the forward pass) and are MN-major: K = output pixels, M = (d, co), N = (l, ci). One work item = one
// filter tap, one 128-row M tile, one <=256-column N tile and one slice of the pixels; its accumulator is
// the real-valued gradient block G[(d,co),(l,ci)] which the epilogue folds through the quaternion table,
//   dw[l^d][co][ci][tap] += s(l,d) * G[(d,co),(l,ci)],
// into an fp32 scratch laid out [tap][r][co][ci] with vector reductions; a last kernel transposes and casts.
// (replaces the 8/16 cudnnConvolutionBackwardFilter calls and accumulate passes of src/conv2d.hpp:433-562.)
// ===================================================================================================
constexpr int FK = 64;                               // pixels per stage
constexpr int F_STAGES = 4;
constexpr uint32_t F_STAGE = (GM + GN) * FK * 2;     // 48 KB
constexpr size_t FG_SMEM = 1024 + F_STAGES * F_STAGE + 512;
constexpr int FP_STAGES = 6;                         // pairs of SMs: half of the N columns in each CTA
constexpr uint32_t FP_STAGE = (GM + GN / 2) * FK * 2;

struct FGParams {
    int Nb, Co, Ci, HO, WO;
    int Cop, Cip;                 // padded channels per component of dy / x
    int cbA, cbB;                 // channel-block width (elements) of the two operands: 64, 32 or 16
    int KH, KW, SH, SW, DH, DW;
    int PW, PH, PN;               // pixel box per stage, PW*PH*PN == FK
    int tiles_w, tiles_h, tiles_n;
    int m_tiles, n_tiles, n_tile_cols;   // N columns per tile (multiple of 16, <= 256)
    int splits, steps_per_split;
    int fmt;
    int LK;                       // components of x (1 for a real-valued input)
    int TPG;                      // x-major variant: taps stacked along M per work item
    int nc, ga;                   // algebra: components, GA(3,0,0) component order
    unsigned long long neg;       // negative entries of the block, bit (8*l + d)
    int off_w, off_h;             // added to the pixel coordinates of every x box: minus the padding (out-of-range coordinates read zeros)
    int flat;                     // pointwise layers: the copies are [component][pixel of all images][channels], the tensor maps (channel of a block,
                                  // pixel, block, component), and a tile's blocks are whole components or a part of one
};

__device__ __forceinline__ uint64_t make_desc_mn_blocks(uint32_t smem_addr, int cb, uint32_t block_bytes) {
    // MN-major tile made of blocks of `cb` elements: K-rows of cb*2 bytes, 8-row groups contiguous.
    const uint64_t layout = cb == 64 ? 2ull : (cb == 32 ? 4ull : 6ull);
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)((block_bytes >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)(((8u * cb * 2u) >> 4) & 0x3FFFu) << 32) | DESC_VERSION_SM100 | (layout << 61);
}

// PAIR: a cluster of two CTAs takes a 256-row M tile (128 rows each) and half of the N columns each; per SM 32 KB instead of 48 KB come
// from L2 for every four MMAs of 512 clocks (an SM takes in about 64 bytes per clock). Forward + backward, before / after: 3x3 64 at 56,
// channels-last, batch 128 1199 / 1164 us; 3x3 stride 2, 128 at 28 578 / 565; 1x1 256 at 14 304 / 295.
template <bool PAIR>
__global__ void __launch_bounds__(G_THREADS, 1)
qconv_filter_general_tc_kernel(const __grid_constant__ CUtensorMap map_dy, const __grid_constant__ CUtensorMap map_x, FGParams p,
                               float* __restrict__ dw32, int* __restrict__ status) {
    constexpr int STAGES = PAIR ? FP_STAGES : F_STAGES;
    constexpr uint32_t STAGE = PAIR ? FP_STAGE : F_STAGE;
    extern __shared__ uint8_t smem_raw[];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int rank = PAIR ? (int)cluster_ctarank() : 0;
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + STAGES * STAGE);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 1);
    const uint32_t tiles_addr = smem_u32(base);
    const uint32_t full_bar = smem_u32(bars), empty_bar = smem_u32(bars + STAGES), tmem_full = smem_u32(bars + 2 * STAGES);

    // work item of this CTA (pair)
    // items (tap, tiles) vary fastest so that the CTAs running at the same time read the same pixel slice (L2 reuse)
    const int m_tiles = PAIR ? p.m_tiles / 2 : p.m_tiles;
    const int n_items = m_tiles * p.n_tiles * p.KH * p.KW, id = PAIR ? blockIdx.x / 2 : blockIdx.x;
    int item = id % n_items;
    const int split = id / n_items;
    const int mt = PAIR ? 2 * (item % m_tiles) + rank : item % m_tiles; item /= m_tiles;
    const int nt = item % p.n_tiles;
    const int tap = item / p.n_tiles;
    const int kh = tap / p.KW, kw = tap - kh * p.KW;
    const int steps_total = p.tiles_w * p.tiles_h * p.tiles_n;
    const int step_beg = split * p.steps_per_split;
    const int n_steps = max(0, min(steps_total, step_beg + p.steps_per_split) - step_beg);

    const int nblkA = GM / p.cbA, nblkB = p.n_tile_cols / p.cbB / (PAIR ? 2 : 1);        // blocks of this CTA's shared memory
    const int bpcA = p.Cop / p.cbA, bpcB = p.Cip / p.cbB;               // channel blocks per component
    const uint32_t blkA_bytes = FK * p.cbA * 2, blkB_bytes = FK * p.cbB * 2;
    const uint32_t a_bytes = nblkA * blkA_bytes, b_bytes = nblkB * blkB_bytes;
    const int blockA0 = mt * nblkA, blockB0 = nt * (GN / p.cbB);

    if (t == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar + 8 * s, 1); mbar_init(empty_bar + 8 * s, 1); }
        mbar_init(tmem_full, 1);
        fence_barrier_init();
    }
    if (warp == 1) { if (PAIR) tmem_alloc_pair(smem_u32(tmem_slot), 512); else tmem_alloc(smem_u32(tmem_slot), 512); }
    tc_fence_before_sync();
    __syncthreads();
    if (PAIR) cluster_sync_all();                     // both CTAs' barriers exist before anything signals them
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    chain_wait();
    chain_next();

    if (warp == 0) {
        // one copy per operand and stage (the staged tensors keep the channel-block index outermost, so the blocks of
        // a tile are one box even across components), and a running (tw, th, tn) of the pixel box: the thread that
        // issues the copies runs no division in this loop -- at a few hundred cycles per copy it used to bound the kernel
        const bool el = elect_one();
        const int myB0 = blockB0 + rank * nblkB;
        const int compA = blockA0 / bpcA, flatA = blockA0 - compA * bpcA, compB = myB0 / bpcB, flatB = myB0 - compB * bpcB;
        int tw = step_beg % p.tiles_w, th = (step_beg / p.tiles_w) % p.tiles_h, tn = step_beg / (p.tiles_w * p.tiles_h);
        int s = 0, phase = 1;
        bool ok = true;
        for (int it = 0; it < n_steps; ++it) {
            ok = warp_wait_bounded(empty_bar + 8 * s, phase, status, ST_G_PRODUCER);
            if (!ok) break;
            if (el) {
                const int ow0 = tw * p.PW, oh0 = th * p.PH, n0 = tn * p.PN;
                const int wx = ow0 * p.SW + kw * p.DW + p.off_w, hx = oh0 * p.SH + kh * p.DH + p.off_h;
                const uint32_t a_dst = tiles_addr + s * STAGE, b_dst = a_dst + GM * FK * 2, bar = full_bar + 8 * s;
                const int a2 = p.flat ? flatA : oh0, a3 = p.flat ? compA : n0, a4 = p.flat ? 0 : blockA0;
                const int b2 = p.flat ? flatB : hx, b3 = p.flat ? compB : n0, b4 = p.flat ? 0 : myB0;
                if (PAIR) {
                    const uint32_t lead = map_to_cta(bar, 0);
                    if (rank == 0) mbar_arrive_expect_tx(bar, 2 * (a_bytes + b_bytes));
                    tma_load_5d_pair(a_dst, &map_dy, 0, ow0, a2, a3, a4, lead);
                    tma_load_5d_pair(b_dst, &map_x, 0, wx, b2, b3, b4, lead);
                } else {
                    mbar_arrive_expect_tx(bar, a_bytes + b_bytes);
                    tma_load_5d(a_dst, &map_dy, 0, ow0, a2, a3, a4, bar);
                    tma_load_5d(b_dst, &map_x, 0, wx, b2, b3, b4, bar);
                }
            }
            if (++tw == p.tiles_w) { tw = 0; if (++th == p.tiles_h) { th = 0; ++tn; } }
            if (++s == STAGES) { s = 0; phase ^= 1; }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t idesc = make_idesc_f16(p.fmt, PAIR ? 2 * GM : GM, p.n_tile_cols, true, true);
            const uint32_t peer_empty = PAIR ? map_to_cta(empty_bar, 1) : 0u, peer_full = PAIR ? map_to_cta(tmem_full, 1) : 0u;
            const bool el = elect_one();
            int s = 0, phase = 0;
            for (int it = 0; it < n_steps; ++it) {
                if (!warp_wait_bounded(full_bar + 8 * s, phase, status, ST_G_MMA)) break;
                tc_fence_after_sync();
                if (el) {
                    const uint32_t a_addr = tiles_addr + s * STAGE;
                    const uint64_t ad = make_desc_mn_blocks(a_addr, p.cbA, blkA_bytes), bd = make_desc_mn_blocks(a_addr + GM * FK * 2, p.cbB, blkB_bytes);
                    const uint32_t a_step = (16u * p.cbA * 2u) >> 4, b_step = (16u * p.cbB * 2u) >> 4;
#pragma unroll
                    for (int j = 0; j < FK / 16; ++j) {
                        // two accumulators in turn: an MMA truncates when it adds (conv_tf32.cu), so half as many in each is half the error
                        const uint32_t al = (uint32_t)ad + j * a_step, bl = (uint32_t)bd + j * b_step, acc = (it > 0 || j > 1) ? 1u : 0u, dst = tmem_base + (j & 1) * GN;
                        if (PAIR) mma_f16_pair(dst, al, (uint32_t)(ad >> 32), bl, (uint32_t)(bd >> 32), idesc, acc);
                        else mma_f16_ss_words(dst, al, (uint32_t)(ad >> 32), bl, (uint32_t)(bd >> 32), idesc, acc);
                    }
                    if (PAIR) {
                        mma_commit_pair(empty_bar + 8 * s);
                        mma_commit_pair(peer_empty + 8 * s);
                        if (it == n_steps - 1) { mma_commit_pair(tmem_full); mma_commit_pair(peer_full); }
                    } else {
                        mma_commit(empty_bar + 8 * s);
                        if (it == n_steps - 1) mma_commit(tmem_full);
                    }
                }
                if (++s == STAGES) { s = 0; phase ^= 1; }
            }
            if (n_steps == 0 && el) { mbar_arrive(tmem_full); if (PAIR) mbar_arrive_cluster(peer_full); }
        }
        __syncwarp();
    } else {
        const int q = warp & 3, chalf = (warp - 2) >> 2;
        const int seen = read_status(status);
        bool ok = mbar_wait_bounded(tmem_full, 0, status, ST_G_EPILOGUE);
        ok = warp_may_store(ok, seen);
        tc_fence_after_sync();
        if (ok && n_steps > 0) {
            // row of the tile -> (output component d, channel co)
            const int row = q * 32 + lane;
            const int blk = blockA0 + row / p.cbA;
            const int d = blk / bpcA, co = (blk % bpcA) * p.cbA + row % p.cbA;
            const bool row_ok = d < p.nc && co < p.Co;
            const bool any_row = __any_sync(0xffffffffu, row_ok);
            const size_t comp_stride = (size_t)p.Co * p.Ci;
            const uint32_t rbuf = tiles_addr + (uint32_t)(warp - 2) * ADD_ROWS_BYTES<32>;      // the operand ring: all MMAs have read it
            float* tap_base = dw32 + (size_t)tap * p.nc * comp_stride;
#pragma unroll 1
            for (int cb = 0; cb < 4; ++cb) {
                const int col0 = chalf * 128 + cb * 32;
                if (col0 >= p.n_tile_cols || !any_row) break;                         // warp-uniform
                uint32_t v[32], u[32];
                tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + col0, v);
                tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + GN + col0, u);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) + __uint_as_float(u[e]));
                auto add = [&](auto quads) {
                    constexpr bool Q = decltype(quads)::value;
                    const int col = col0 + add_rows_column<32, Q>(lane), nblk = blockB0 + col / p.cbB;      // (l, ci) of this lane's columns
                    const int l = nblk / bpcB, ci = (nblk % bpcB) * p.cbB + col % p.cbB;
                    const bool col_ok = col < p.n_tile_cols && l < p.LK && ci < p.Ci;
                    add_rows<32, Q>(rbuf, v, lane, [&](int r, float& sgn) -> float* {
                        const int rd = __shfl_sync(0xffffffffu, row_ok ? d : -1, r), rco = __shfl_sync(0xffffffffu, co, r);
                        if (rd < 0 || !col_ok) return nullptr;
                        if (alg_negative(p.neg, l, rd)) sgn = -1.f;
                        return tap_base + (size_t)alg_pair(p.ga, l, rd) * comp_stride + (size_t)rco * p.Ci + ci;
                    });
                };
                if ((p.Ci & 3) == 0) add(Bool<true>()); else add(Bool<false>());
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (PAIR) cluster_sync_all();                     // nobody leaves while its peer may still signal its barriers or read its shared memory
    if (warp == 1) { if (PAIR) tmem_dealloc_pair(tmem_base, 512); else tmem_dealloc(tmem_base, 512); }
}

// ---------------------------------------------------------------------------------------------------
// Backward-filter for narrow layers, "x-major": the M side is the *input* with several filter taps stacked
// (rows = (tap, l, ci), one tap-shifted TMA box per tap), the N side is dy (columns = (d, co)). One dy tile
// then serves up to 8 taps instead of being re-read for every tap, which is what bounds the layers with 16
// or 32 quaternion channels and the 49-tap stem. Used when 4*Cop <= 256 and one x box per tap fits in M.
// ---------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(G_THREADS, 1)
qconv_filter_xmajor_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_dy, FGParams p,
                              float* __restrict__ dw32, int* __restrict__ status) {
    extern __shared__ uint8_t smem_raw[];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + F_STAGES * F_STAGE);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * F_STAGES + 1);
    const uint32_t tiles_addr = smem_u32(base);
    const uint32_t full_bar = smem_u32(bars), empty_bar = smem_u32(bars + F_STAGES), tmem_full = smem_u32(bars + 2 * F_STAGES);

    const int taps = p.KH * p.KW;
    const int n_groups = (taps + p.TPG - 1) / p.TPG;
    const int tg = blockIdx.x % n_groups, split = blockIdx.x / n_groups;
    const int steps_total = p.tiles_w * p.tiles_h * p.tiles_n;
    const int step_beg = split * p.steps_per_split;
    const int n_steps = max(0, min(steps_total, step_beg + p.steps_per_split) - step_beg);
    const uint32_t tap_bytes = p.LK * FK * p.cbB * 2;          // one tap's x box: LK components of cbB channels
    const uint32_t blkX_bytes = FK * p.cbB * 2, blkY_bytes = FK * p.cbA * 2;
    const int n_cols = p.nc * p.cbA;                            // (d, co) with co padded to the channel block
    const uint32_t a_bytes = p.TPG * tap_bytes, b_bytes = p.nc * blkY_bytes;

    if (t == 0) {
        for (int s = 0; s < F_STAGES; ++s) { mbar_init(full_bar + 8 * s, 1); mbar_init(empty_bar + 8 * s, 1); }
        mbar_init(tmem_full, 1);
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 512);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    chain_wait();
    chain_next();

    if (warp == 0) {
        {
            const bool el = elect_one();
            // per-tap offsets of the x boxes and the running (tw, th, tn) of the pixel box: no division in the loop
            int w_ofs[8], h_ofs[8], comp[8];
            for (int tl = 0; tl < p.TPG && tl < 8; ++tl) {
                const int tap = tg * p.TPG + tl;
                const int kh = tap / p.KW, kw = tap - kh * p.KW;
                w_ofs[tl] = kw * p.DW; h_ofs[tl] = kh * p.DH;
                comp[tl] = tap < taps ? 0 : p.LK;     // a tap past the end is loaded from component LK: entirely out of range, i.e. zeros
            }
            int tw = step_beg % p.tiles_w, th = (step_beg / p.tiles_w) % p.tiles_h, tn = step_beg / (p.tiles_w * p.tiles_h);
            int s = 0, phase = 1;
            bool ok = true;
            for (int it = 0; it < n_steps && ok; ++it) {
                ok = warp_wait_bounded(empty_bar + 8 * s, phase, status, ST_G_PRODUCER);
                if (!ok) break;
                const int ow0 = tw * p.PW, oh0 = th * p.PH, n0 = tn * p.PN;
                const uint32_t a_dst = tiles_addr + s * F_STAGE, b_dst = a_dst + GM * FK * 2, bar = full_bar + 8 * s;
                if (++tw == p.tiles_w) { tw = 0; if (++th == p.tiles_h) { th = 0; ++tn; } }
                if (++s == F_STAGES) { s = 0; phase ^= 1; }
                if (el) {
                    mbar_arrive_expect_tx(bar, a_bytes + b_bytes);
                    for (int tl = 0; tl < p.TPG; ++tl)
                        tma_load_5d(a_dst + tl * tap_bytes, &map_x, 0, ow0 * p.SW + w_ofs[tl] + p.off_w, oh0 * p.SH + h_ofs[tl] + p.off_h, n0, comp[tl], bar);
                    tma_load_5d(b_dst, &map_dy, 0, ow0, oh0, n0, 0, bar);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        const uint32_t idesc = make_idesc_f16(p.fmt, GM, n_cols, true, true);
        bool ok = true;
        const bool el = elect_one();
        for (int it = 0; it < n_steps && ok; ++it) {
            const int s = it % F_STAGES;
            ok = warp_wait_bounded(full_bar + 8 * s, (it / F_STAGES) & 1, status, ST_G_MMA);
            if (!ok) break;
            tc_fence_after_sync();
            if (el) {
                const uint32_t a_addr = tiles_addr + s * F_STAGE, b_addr = a_addr + GM * FK * 2;
#pragma unroll
                for (int j = 0; j < FK / 16; ++j)           // two accumulators in turn, as in the general kernel
                    mma_f16_ss(tmem_base + (j & 1) * GN, make_desc_mn_blocks(a_addr + j * 16 * p.cbB * 2, p.cbB, blkX_bytes),
                               make_desc_mn_blocks(b_addr + j * 16 * p.cbA * 2, p.cbA, blkY_bytes), idesc, (it > 0 || j > 1) ? 1u : 0u);
                mma_commit(empty_bar + 8 * s);
                if (it == n_steps - 1) mma_commit(tmem_full);
            }
            __syncwarp();
        }
        if (n_steps == 0 && lane == 0) mbar_arrive(tmem_full);
        __syncwarp();
    } else {
        const int q = warp & 3, chalf = (warp - 2) >> 2;
        const int seen = read_status(status);
        bool ok = mbar_wait_bounded(tmem_full, 0, status, ST_G_EPILOGUE);
        ok = warp_may_store(ok, seen);
        tc_fence_after_sync();
        if (ok && n_steps > 0) {
            const int row = q * 32 + lane;                       // row -> (tap, input component l, channel ci)
            const int blk = row / p.cbB;
            const int tap = tg * p.TPG + blk / p.LK, l = blk % p.LK, ci = row % p.cbB;
            const bool row_ok = tap < taps && ci < p.Ci;
            const size_t comp_stride = (size_t)p.Co * p.Ci;
            float* tap_base = dw32 + (size_t)tap * p.nc * comp_stride + ci;
#pragma unroll 1
            for (int cb = 0; cb < 4; ++cb) {
                const int col0 = chalf * 128 + cb * 32;
                if (col0 >= n_cols) break;
                uint32_t v[32], u[32];
                tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + col0, v);
                tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + GN + col0, u);
                tmem_ld_wait();
                if (!row_ok) continue;
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    const int col = col0 + e;
                    const int d = col / p.cbA, co = col - d * p.cbA;
                    if (col < n_cols && co < p.Co) {
                        const float val = __uint_as_float(v[e]) + __uint_as_float(u[e]);
                        atomicAdd(tap_base + (size_t)alg_pair(p.ga, l, d) * comp_stride + (size_t)co * p.Ci, alg_negative(p.neg, l, d) ? -val : val);
                    }
                }
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, 512);
}

// scratch [tap][r][co][ci] fp32 -> dw in the tensor type. `dense_oihw`: dw is [r][co][ci][tap] and the threads walk the
// destination (coalesced stores); otherwise the destination is addressed through the filter-gradient strides (OHWI, HWIO,
// the input-major dense gradient, the slice of one group) and the threads walk the source.
template <typename T>
__global__ void unpack_filter_grad_kernel(const float* src, T* __restrict__ dw, int taps, size_t per_tap, int dense_oihw,
                                          int Co, int Ci, FilterStrides ds) {
    const size_t total = per_tap * taps;
    chain_wait();
    chain_next();
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        if (dense_oihw) {
            const int tap = (int)(idx % taps);
            const size_t e = idx / taps;
            DType<T>::store(dw + idx, ld_chained(src + (size_t)tap * per_tap + e));
            continue;
        }
        const int ci = (int)(idx % Ci);
        size_t rest = idx / Ci;
        const int co = (int)(rest % Co); rest /= Co;
        const size_t comps = per_tap / ((size_t)Co * Ci);
        const int r = (int)(rest % comps), tap = (int)(rest / comps);
        const int kh = tap / ds.KW, kw = tap - kh * ds.KW;
        DType<T>::store(dw + (long long)r * ds.r + (long long)co * ds.o + (long long)ci * ds.i + (long long)kh * ds.h + (long long)kw * ds.w, ld_chained(src + idx));
    }
}

// Geometry of one launch of the implicit-GEMM kernel: "input" is the tensor being convolved (x forward,
// dy backward-data), "output" the tensor produced.
struct Plan {
    int Cin, Cout;                 // channels per component of the convolved / produced tensor
    int Hin, Win, Hout, Wout;
    int pad_top, pad_left;         // zero padding: materialised in a zero-inserted copy, the tensor map's zero fill otherwise
    int SH, SW;
    int ins_h, ins_w;              // zero-insertion factors of the staged copy (strided backward-data)
    int Cp, Hp, Wp, Mp, Kp;
    int LK;                        // components of the convolved tensor (1 for a real-valued input)
    int KS;
    int dual;                      // backward-data with strides 2 x 2 by pixel classes (the kernel's DUAL form)
    bool tight;                    // see Geom
    size_t xp_bytes, w_bytes;
};

// Both row and column classes need taps of their own.
bool dual_classes(Pass pass, const Geom& g) {
    return pass == PASS_BWD_DATA && g.SH == 2 && g.SW == 2 && g.DH == 1 && g.DW == 1 && g.KH >= 2 && g.KW >= 2;
}

Plan make_plan(Pass pass, const Geom& g, bool tight) {
    Plan pl;
    pl.tight = tight;
    if (pass == PASS_FWD) {
        pl.Cin = g.Ci; pl.Cout = g.Co; pl.Hin = g.H; pl.Win = g.W; pl.Hout = g.HO; pl.Wout = g.WO;
        pl.pad_top = g.PT; pl.pad_left = g.PL; pl.SH = g.SH; pl.SW = g.SW; pl.ins_h = pl.ins_w = 1;
    } else {   // backward-data: stride-1 correlation of dy (zero-inserted by the stride, padded by k-1-pad) with the
               // flipped, transposed filters
        pl.Cin = g.Co; pl.Cout = g.Ci; pl.Hin = g.HO; pl.Win = g.WO; pl.Hout = g.H; pl.Wout = g.W;
        pl.pad_top = (g.KH - 1) * g.DH - g.PT; pl.pad_left = (g.KW - 1) * g.DW - g.PL; pl.SH = 1; pl.SW = 1;
        pl.ins_h = g.SH; pl.ins_w = g.SW;
    }
    pl.dual = dual_classes(pass, g) ? 1 : 0;
    if (pl.dual) { pl.ins_h = pl.ins_w = 1; pl.pad_top = pl.pad_left = 0; }   // (the kernel places the taps itself)
    pl.LK = (pass == PASS_FWD && g.real_in) ? 1 : g.nc;
    pl.KS = channel_slice(pl.Cin, tight);
    pl.Cp = padded_channels(pl.Cin, tight);
    pl.Hp = (pl.Hout - 1) * pl.SH + (g.KH - 1) * g.DH + 1;
    pl.Wp = (pl.Wout - 1) * pl.SW + (g.KW - 1) * g.DW + 1;
    if (pl.ins_h == 1 && pl.ins_w == 1) {                              // the copy is not padded: the tensor map's zero fill is the padding
        pl.Hp = tight && !pl.dual ? reached(pl.Hin, pl.Hout, pl.SH, g.KH, g.DH, pl.pad_top) : pl.Hin;
        pl.Wp = tight && !pl.dual ? reached(pl.Win, pl.Wout, pl.SW, g.KW, g.DW, pl.pad_left) : pl.Win;
    }
    pl.Mp = round_up(g.nc * pl.Cout, GM);
    pl.Kp = pl.LK * pl.Cp;
    pl.xp_bytes = ((size_t)pl.LK * g.Nb * pl.Hp * pl.Wp * pl.Cp * 2 + 1023) / 1024 * 1024;
    pl.w_bytes = ((size_t)g.KH * g.KW * pl.Mp * pl.Kp * 2 + 1023) / 1024 * 1024;
    return pl;
}

constexpr size_t MAX_COPY = (size_t)8 << 30;
Plan make_plan(Pass pass, const Geom& g) {
    const Plan pl = make_plan(pass, g, g.tight != 0);
    return pl.xp_bytes <= MAX_COPY ? pl : make_plan(pass, g, true);
}

}  // namespace

bool conv_tc_dual_classes(Pass pass, const Geom& g) { return dual_classes(pass, g); }

bool conv_tc_supported(Pass pass, int dtype, int variant, const Geom& g) {
    if (pass != PASS_FWD && pass != PASS_BWD_DATA) return false;
    if (dtype != PCB_F16 && dtype != PCB_BF16) return false;
    if (variant != PCB_VARIANT_16_PRODUCT) return false;
    if (g.w_io && g.KH * g.KW != 1) return false;                       // input-major filters: dense layers (1x1 images, one tap)
    if (g.real_in && pass != PASS_FWD) return false;
    if (g.SH > 2 || g.SW > 2) return false;
    if (pass == PASS_BWD_DATA) {
        if ((g.KH - 1) * g.DH < g.PT || (g.KW - 1) * g.DW < g.PL) return false;
    }
    const Plan pl = make_plan(pass, g);
    if ((long long)(pl.Hout - 1) * pl.SH + (long long)(g.KH - 1) * g.DH > 65534 || (long long)(pl.Wout - 1) * pl.SW + (long long)(g.KW - 1) * g.DW > 65534) return false;
    if ((long long)pl.Wp * pl.Cp * 2 > (1ll << 31) || pl.xp_bytes > MAX_COPY) return false;
    return true;
}

size_t conv_tc_scratch_bytes(Pass pass, const Geom& g) {
    const Plan pl = make_plan(pass, g);
    return pl.xp_bytes + pl.w_bytes;
}

int conv_tc_launch(Pass pass, int dtype, const Geom& layer, const void* w, const void* act, const void* bias, void* out,
                   void* scratch, int* status, cudaStream_t stream, StatusClear* sc) {
    EncodeTiledFn encode = encode_fn();
    if (!encode) { set_error("cuTensorMapEncodeTiled is not available from the driver"); return PCB_ERR_CUDA; }
    const int fmt = dtype == PCB_F16 ? 0 : 1;
    // (planes that leave whole, see the plane mode below, stay planes)
    const bool planes = layer.H * layer.W <= 256 && (pass == PASS_FWD ? layer.Co : layer.Ci) % GM == 0;
    const Geom g = planes ? layer : flat_pixels(layer);
    const Plan pl = make_plan(pass, g);
    const int taps = g.KH * g.KW;
    uint8_t* xp = static_cast<uint8_t*>(scratch);
    uint8_t* wexp = xp + pl.xp_bytes;
    // element strides of the convolved tensor (x forward, dy backward-data) and of the produced one
    const SrcStrides sa = pass == PASS_FWD ? SrcStrides{g.xp, g.xc, g.xh, g.xw} : SrcStrides{g.yp, g.yc, g.yh, g.yw};
    const SrcStrides so = pass == PASS_FWD ? SrcStrides{g.yp, g.yc, g.yh, g.yw} : SrcStrides{g.xp, g.xc, g.xh, g.xw};
    // A channels-last tensor whose channel count is a multiple of 16 already IS the staged layout: it is read in place, the
    // padding (of the image and of the last channel slice) comes from the zero fill of out-of-range TMA coordinates, and no copy of
    // the activations is made at all. (Other multiples of 8 are copied to padded pixels: a 5x5 layer of 56 channels, 45 x 45, batch 105, takes
    // 1506 us forward + backward with its 112-byte pixels read in place and 1309 us from a copy with 128-byte pixels.)
    // (Not for zero-inserted gradients, channel slices of grouped layers, or images smaller than a tile box.)
    bool direct = !g.plain && sa.c == 1 && sa.w == pl.Cin && sa.h == (long long)pl.Win * pl.Cin && sa.p == (long long)pl.Hin * pl.Win * pl.Cin &&
                  pl.Cin % 16 == 0 && pl.ins_h == 1 && pl.ins_w == 1 && (reinterpret_cast<uintptr_t>(act) & 15u) == 0;
    // The strided backward-data pass reads a copy of dy where dx shares its memory.
    if (pl.dual && direct)
        direct = !overlaps(out, (size_t)g.nc * g.Nb * pl.Cout * pl.Hout * pl.Wout * 2, act, (size_t)pl.LK * g.Nb * pl.Cin * pl.Hin * pl.Win * 2);

    const bool inserted = pl.ins_h != 1 || pl.ins_w != 1;
    bool chain = false;

    // stage the operands
    {
        Prologue pro;
        if (!direct)
            stage_activations(pro, fmt, act, xp, pl.LK * g.Nb, pl.Cin, pl.Hin, pl.Win, pl.Hp, pl.Wp, pl.Cp, inserted ? pl.pad_top : 0, inserted ? pl.pad_left : 0,
                              pl.ins_h, pl.ins_w, pl.KS, stream, 0, 1, g.plain ? nullptr : &sa);
        const FilterStrides fs = {g.wr, g.wo, g.wi, g.wh, g.ww, g.KW};
        add_filter_job(pro, w, wexp, g.Co, g.Ci, taps, pl.Mp, pl.Kp, pl.Cp, pass == PASS_BWD_DATA ? 1 : 0, g.nc, g.ga, g.neg, fs);
        const int rc = launch_prologue(pro, sc, stream, &chain);
        if (rc != PCB_OK) return rc;
        PCB_CUDA_TRY(cudaGetLastError());
    }

    GParams p;
    p.store_vec = 1;
    while (p.store_vec < 16 && pl.Wout % (p.store_vec * 2) == 0 && (reinterpret_cast<uintptr_t>(out) % (size_t)(p.store_vec * 4)) == 0) p.store_vec *= 2;
    // pick the output tile box (PW x PH x PN = 256 pixels, DUAL: 128 pixels of a class) that wastes the fewest MMA columns
    const int Wc = pl.dual ? (pl.Wout + 1) / 2 : pl.Wout, Hc = pl.dual ? (pl.Hout + 1) / 2 : pl.Hout;
    if (pl.dual) {
        long long best = -1;
        for (int pw = 4; pw <= 64; pw *= 2)
            for (int ph = 1; ph * pw <= GN / 2; ph *= 2) {
                const int pn = GN / 2 / (pw * ph);
                const long long vol = (long long)round_up(Wc, pw) * round_up(Hc, ph) * round_up(g.Nb, pn);
                if (best < 0 || vol < best || (vol == best && pw > p.PW)) { best = vol; p.PW = pw; p.PH = ph; p.PN = pn; }
            }
    } else {
        long long best = -1;
        // (dense layers are 1 x 1 images: their box is 1 x 1 x 256, so that the columns of a tile are batch rows and none is wasted)
        const bool dense_like = pl.Wout == 1 && pl.Hout == 1;
        for (int pw = dense_like ? 1 : 8; pw <= 256; pw *= 2)
            for (int ph = 1; ph * pw <= 256; ph *= 2) {
                const int pn = 256 / (pw * ph);
                if (pw * pl.SW > 256 || ph * pl.SH > 256) continue;
                const long long vol = (long long)round_up(pl.Wout, pw) * round_up(pl.Hout, ph) * round_up(g.Nb, pn);
                if (best < 0 || vol < best || (vol == best && pw > p.PW)) { best = vol; p.PW = pw; p.PH = ph; p.PN = pn; }
            }
    }
    // Planes that fit one tile box and 128-channel row tiles: take whole planes per tile even if that wastes a few more
    // columns, because the tile then leaves as bulk copies (plane mode, see the epilogue) instead of 2..8-byte stores
    // scattered over 128 planes, which saturate the store path long before the tensor pipe.
    {
        int pw = 8, ph = 1;
        while (pw < pl.Wout) pw *= 2;
        while (ph < pl.Hout) ph *= 2;
        if (!pl.dual && pw * ph <= 256 && pl.Cout % GM == 0 && pl.Wout % 8 != 0 && !(pl.Wout == 1 && pl.Hout == 1)) { p.PW = pw; p.PH = ph; p.PN = 256 / (pw * ph); }
    }
    // Halo mode (see the kernel): stride-1 correlation, 32-channel slices, several taps, and an image tall enough for
    // tiles of 8 x PH >= 192 pixels (smaller tiles re-read the filter slices too often to gain anything).
    // channels-last output with a multiple of 32 channels and 16-byte aligned pixels: the transposing epilogue (16 KB of shared memory)
    const bool cl32 = !g.plain && so.c == 1 && pl.Cout % 32 == 0 && so.w % 8 == 0 && so.h % 8 == 0 && so.p % 8 == 0 &&
                      (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
    constexpr int CL32_BYTES = 8 * 2048, ROWS_BYTES = 8 * EPI_ROWS_BYTES;
    // shared memory of the epilogue beside the operand stages (plane mode has its own)
    const bool unaligned_rows = g.plain && p.store_vec < 8;
    const int epi_bytes = cl32 ? CL32_BYTES : (unaligned_rows ? ROWS_BYTES : 0);
    bool halo = false;
    // pairs of SMs: two row tiles at a time
    bool pair = (pl.Mp / GM) % 2 == 0 && worth_pairs((double)g.Nb * Hc * Wc / 256 * (pl.Mp / GM) * taps * pl.LK * (pl.Cp / 16));
    p.split_w = p.split_h = p.split_n = p.half_valid = 0;
    p.n_cols = 256; p.Wt = p.Ht = 0; p.n_stages = 0; p.stage_bytes = 0; p.a_slots = 0; p.a_taps = 1; p.halo_bytes = 0;
    if (!pl.dual && pl.Cp % 32 == 0 && pl.SH == 1 && pl.SW == 1 && taps >= 4 && pl.Wout >= 8) {
        const int rows = (pl.Hout + 31) / 32;
        const int ph = (((pl.Hout + rows - 1) / rows) + 1) & ~1;
        // (a pair splits the rows of the tile in two; even the halves of 24 to 32 rows are 8 x PH / 2 >= 96 columns, a multiple of 8)
        const int wt = 8 + (g.KW - 1) * g.DW, ht = (pair ? ph / 2 : ph) + (g.KH - 1) * g.DH;
        const uint32_t tile = ((uint32_t)wt * ht * 64 + 1023) / 1024 * 1024, tap_bytes = GM * 32 * 2;
        const int room = 227 * 1024 - 1024 - 512 - epi_bytes;
        // a slot of the filter ring holds a filter row where at least four of those fit beside two halo tiles, one tap otherwise
        p.a_taps = room >= (int)(2 * tile + 4 * g.KW * tap_bytes) ? g.KW : 1;
        const int slot = p.a_taps * (int)tap_bytes;
        if (ph >= 24 && wt <= 256 && ht <= 256 && room >= (int)(2 * tile) + 4 * slot) {
            halo = true;
            p.PW = 8; p.PH = ph; p.PN = 1; p.n_cols = 8 * ph; p.Wt = wt; p.Ht = ht;
            p.split_h = pair ? ph / 2 : 0;
            p.halo_bytes = tile;
            p.n_stages = room >= (int)(H_MAX_TILES * tile) + 6 * slot ? H_MAX_TILES : 2;
            p.a_slots = (room - p.n_stages * (int)tile) / slot;
            if (p.a_slots > H_MAX_SLOTS) p.a_slots = H_MAX_SLOTS;
            p.stage_bytes = 0;
        }
    }
    {
        auto log2i = [](int v) { int l = 0; while ((1 << l) < v) ++l; return (1 << l) == v ? l : -1; };
        p.lw = log2i(p.PW); p.lh = log2i(p.PH);
    }
    // plane mode (see the epilogue): whole output planes per tile, 128 rows = 128 consecutive channels of one component
    // strided output: anything but a dense NCHW tensor, and the narrow boxes of dense layers
    p.o_generic = (!g.plain || p.lw + pl.dual < 3) ? 1 : 0;
    p.o_cl32 = (cl32 && p.o_generic && p.lw >= 0) ? 1 : 0;
    p.o_p = (int)so.p; p.o_c = (int)so.c; p.o_h = (int)so.h; p.o_w = (int)so.w;
    p.bias_ld = g.bias_ld;
    p.off_w = inserted ? 0 : -pl.pad_left; p.off_h = inserted ? 0 : -pl.pad_top;
    p.plane_mode = (!p.o_generic && !halo && !pl.dual && p.PW >= pl.Wout && p.PH >= pl.Hout && pl.Cout % GM == 0 && p.lh >= 0 && (p.lw == 3 || p.lw == 4) &&
                    (reinterpret_cast<uintptr_t>(out) & 15u) == 0) ? 1 : 0;
    // Planes of at most 256 pixels: the box is exactly PN whole planes (7 x 7 x 5 = 245 of 256 columns instead of 8 x 8 x 4 with
    // 49 of every 64 in use; 14 x 14 x 1 = 196 columns in MMAs 208 wide instead of 256), and the tile still leaves as one bulk
    // copy per image.
    p.exact = 0;
    if (!p.o_generic && !halo && !pl.dual && pl.Cout % GM == 0 && pl.Hout * pl.Wout <= 256 && pl.Wout <= 256 && pl.Hout <= 256 &&
        (pl.Wout - 1) * pl.SW + 1 <= 256 && (pl.Hout - 1) * pl.SH + 1 <= 256 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
        const int HWo = pl.Hout * pl.Wout;
        int pn = 256 / HWo;
        if (pn > g.Nb) pn = g.Nb;
        // only where it puts more pixels into a tile than the power-of-two box does (measured: a 14 x 14 plane gains nothing
        // from MMAs 208 instead of 256 columns wide)
        const int pow2_valid = p.plane_mode ? HWo * p.PN : 0;
        if (pn * HWo > pow2_valid) {
            p.exact = 1; p.plane_mode = 1;
            p.PW = pl.Wout; p.PH = pl.Hout; p.PN = pn;
            p.n_cols = round_up(p.PW * p.PH * p.PN, 16);
            p.lw = p.lh = 0;
        }
        // a pair: as many whole planes in each half, or half a plane of an even number of rows
        if (pair && (HWo <= 128 || (pl.Hout % 2 == 0 && HWo <= 256))) {
            const int planes = HWo <= 128 ? 128 / HWo : 1;
            p.exact = 1; p.plane_mode = 1;
            p.PW = pl.Wout; p.PH = pl.Hout; p.PN = HWo <= 128 ? 2 * planes : 1;
            p.split_n = HWo <= 128 ? planes : 0;
            p.split_h = HWo <= 128 ? 0 : pl.Hout / 2;
            p.half_valid = HWo <= 128 ? planes * HWo : HWo / 2;
            p.n_cols = 2 * round_up(p.half_valid, 8);
            p.lw = p.lh = 0;
        } else if (p.exact) {
            pair = false;
        }
    }
    if (pair && !halo && !p.exact) {               // halves of the power-of-two box, in the order of its columns
        if (p.PN >= 2) p.split_n = p.PN / 2;
        else if (p.PH >= 2) p.split_h = p.PH / 2;
        else p.split_w = p.PW / 2;
    }
    p.rows_epi = (unaligned_rows && !p.o_generic && !p.plane_mode) ? 1 : 0;
    const int halves = pl.dual + (pair ? 1 : 0), b_rows = GN >> halves;
    p.b_tx = (uint32_t)(p.exact ? (pair ? p.half_valid : p.PW * p.PH * p.PN) : b_rows) * (uint32_t)pl.KS * 2u;
    const int tail_bytes = p.plane_mode ? (int)G_PLANE_BYTES : (p.o_cl32 ? CL32_BYTES : (p.rows_epi ? ROWS_BYTES : 0));
    if (!halo) {
        const int max_stages = pl.KS == 64 ? G_MAX_STAGES<64, 0> + 2 * halves : (pl.KS == 32 && !halves ? G_MAX_STAGES<32, 0> : G_MAX_STAGES<16, 0>);
        const int fit = (int)((227 * 1024 - 1024 - 512 - tail_bytes) / ((GM + b_rows) * pl.KS * 2));
        p.n_stages = fit < max_stages ? fit : max_stages;
        p.stage_bytes = (uint32_t)(GM + b_rows) * pl.KS * 2;
    }
    p.Nb = g.Nb; p.Cout = pl.Cout; p.Mvalid = g.nc * pl.Cout; p.HO = pl.Hout; p.WO = pl.Wout; p.Cp = pl.Cp;
    p.KH = g.KH; p.KW = g.KW; p.SH = pl.SH; p.SW = pl.SW; p.DH = g.DH; p.DW = g.DW;
    p.tiles_w = (Wc + p.PW - 1) / p.PW; p.tiles_h = (Hc + p.PH - 1) / p.PH; p.tiles_n = (g.Nb + p.PN - 1) / p.PN;
    p.tiles_m = pl.Mp / GM;
    p.PT = g.PT; p.PL = g.PL;
    p.fmt = fmt; p.has_bias = (pass == PASS_FWD && g.has_bias) ? 1 : 0;
    p.LK = pl.LK;

    const CUtensorMapDataType dt = fmt == 0 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const int ks = halo ? 32 : pl.KS;
    const CUtensorMapSwizzle sw = ks == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : (ks == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    alignas(64) CUtensorMap map_w, map_x;
    {
        const cuuint64_t dims[3] = {(cuuint64_t)pl.Kp, (cuuint64_t)pl.Mp, (cuuint64_t)taps};
        const cuuint64_t strides[2] = {(cuuint64_t)pl.Kp * 2, (cuuint64_t)pl.Mp * pl.Kp * 2};
        const cuuint32_t box[3] = {(cuuint32_t)ks, GM, (cuuint32_t)(halo ? p.a_taps : 1)};
        const cuuint32_t es[3] = {1, 1, 1};
        const CUresult r = encode(&map_w, dt, 3, wexp, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled (filters) failed with code %d", (int)r); return PCB_ERR_CUDA; }
    }
    {
        // staged copy [comp][img][Hp][Wp][Cp], or the caller's channels-last tensor (the same without padding) read in place
        const int Wd = direct ? pl.Win : pl.Wp, Hd = direct ? pl.Hin : pl.Hp, Cd = direct ? pl.Cin : pl.Cp;
        const cuuint64_t dims[5] = {(cuuint64_t)Cd, (cuuint64_t)Wd, (cuuint64_t)Hd, (cuuint64_t)g.Nb, (cuuint64_t)pl.LK};
        const cuuint64_t strides[4] = {(cuuint64_t)Cd * 2, (cuuint64_t)Wd * Cd * 2, (cuuint64_t)Hd * Wd * Cd * 2, (cuuint64_t)g.Nb * Hd * Wd * Cd * 2};
        // with an element stride s the box extent is given in input elements: s * (pixels - 1) + 1 of them hold the pixels loaded
        const int rows = p.split_h > 0 ? p.split_h : p.PH, width = p.split_w > 0 ? p.split_w : p.PW;
        const cuuint32_t box[5] = {(cuuint32_t)ks, (cuuint32_t)(halo ? p.Wt : (width - 1) * pl.SW + 1), (cuuint32_t)(halo ? p.Ht : (rows - 1) * pl.SH + 1),
                                   (cuuint32_t)(p.split_n > 0 ? p.split_n : p.PN), 1};
        const cuuint32_t es[5] = {1, (cuuint32_t)pl.SW, (cuuint32_t)pl.SH, 1, 1};
        const CUresult r = encode(&map_x, dt, 5, direct ? const_cast<void*>(act) : static_cast<void*>(xp), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled (activations) failed with code %d", (int)r); return PCB_ERR_CUDA; }
    }

    const int n_tiles = p.tiles_w * p.tiles_h * p.tiles_n * p.tiles_m * (pl.dual ? 2 : 1) / (pair ? 2 : 1);
    const int most = pair ? sm_pairs() : sm_count(), grid = (n_tiles < most ? n_tiles : most) * (pair ? 2 : 1);
    const size_t operand_bytes = halo ? (size_t)p.a_slots * p.a_taps * GM * 64 + (size_t)p.n_stages * p.halo_bytes : (size_t)p.n_stages * p.stage_bytes;
    size_t smem = 1024 + operand_bytes + 512 + tail_bytes;
    if (smem < ONE_CTA_SMEM) smem = ONE_CTA_SMEM;
    auto run = [&](auto* kernel) -> int {
        PCB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_CTA_SMEM));
        PCB_CUDA_TRY(launch_clusters(pair ? 2 : 1, chain, kernel, grid, G_THREADS, smem, stream, map_w, map_x, p, (const uint16_t*)bias, (uint16_t*)out, status));
        return PCB_OK;
    };
    auto by_slice = [&](auto* k64, auto* k32, auto* k16) -> int { return pl.KS == 64 ? run(k64) : (pl.KS == 32 ? run(k32) : run(k16)); };
    int rc;
    if (pl.dual && pair) rc = by_slice(qconv_general_tc_kernel<64, false, true, true>, qconv_general_tc_kernel<32, false, true, true>, qconv_general_tc_kernel<16, false, true, true>);
    else if (pl.dual) rc = by_slice(qconv_general_tc_kernel<64, false, true, false>, qconv_general_tc_kernel<32, false, true, false>, qconv_general_tc_kernel<16, false, true, false>);
    else if (halo) rc = pair ? run(qconv_general_tc_kernel<32, true, false, true>) : run(qconv_general_tc_kernel<32, true, false, false>);
    else if (pair) rc = by_slice(qconv_general_tc_kernel<64, false, false, true>, qconv_general_tc_kernel<32, false, false, true>, qconv_general_tc_kernel<16, false, false, true>);
    else rc = by_slice(qconv_general_tc_kernel<64, false, false, false>, qconv_general_tc_kernel<32, false, false, false>, qconv_general_tc_kernel<16, false, false, false>);
    if (rc != PCB_OK) return rc;
    PCB_CUDA_TRY(cudaGetLastError());
    return PCB_OK;
}

namespace {
struct FilterPlan {
    int Cop, Cip, cbx, cby;        // padded channels and the width of their blocks
    int H, W;                      // extents of the copy of x
    bool tight;                    // see Geom
    size_t xp_bytes, dyp_bytes, acc_bytes;
};

FilterPlan make_filter_plan(const Geom& g, bool tight) {
    FilterPlan f;
    f.tight = tight;
    f.Cop = padded_channels(g.Co, tight); f.cby = channel_slice(g.Co, tight);
    f.Cip = padded_channels(g.Ci, tight); f.cbx = channel_slice(g.Ci, tight);
    f.H = tight ? reached(g.H, g.HO, g.SH, g.KH, g.DH, g.PT) : g.H;
    f.W = tight ? reached(g.W, g.WO, g.SW, g.KW, g.DW, g.PL) : g.W;
    f.xp_bytes = ((size_t)(g.real_in ? 1 : g.nc) * g.Nb * f.H * f.W * f.Cip * 2 + 1023) / 1024 * 1024;
    f.dyp_bytes = ((size_t)g.nc * g.Nb * g.HO * g.WO * f.Cop * 2 + 1023) / 1024 * 1024;
    f.acc_bytes = ((size_t)g.nc * g.Co * g.Ci * g.KH * g.KW * sizeof(float) + 1023) / 1024 * 1024;
    return f;
}
constexpr size_t MAX_COPIES = (size_t)12 << 30;
FilterPlan make_filter_plan(const Geom& g) {
    const FilterPlan f = make_filter_plan(g, g.tight != 0);
    return f.xp_bytes + f.dyp_bytes <= MAX_COPIES ? f : make_filter_plan(g, true);
}
}  // namespace

namespace {
// x-major variant: one x box per tap must tile M = 128 exactly and dy's (d, co) columns must fit one MMA.
bool filter_xmajor(const Geom& g, const FilterPlan& f) {
    const int lk = g.real_in ? 1 : g.nc;
    return f.Cip == f.cbx && f.Cop == f.cby && lk * f.cbx <= 64 && g.nc * f.cby <= 256;
}
}  // namespace

namespace {
// At most 64 channels that fill a block of 16, 32 or 64 to its last 16 (not 33 .. 48, which are padded by more).
bool one_block(int c) { const int p16 = round_up(c, 16); return p16 == 16 || p16 == 32 || p16 == 64; }
}  // namespace

// Whether the filter gradient takes the layer as rows of pixels that run on over the images, from copies laid out as those of the other
// passes: pointwise layers whose row and column tiles hold whole components or lie inside one. No pixel of a box is padding then, and
// backward-data's copy of dy serves both passes: 256 -> 256 channels, 14 x 14, batch 32, forward + backward in bf16 253 us, with a
// blocked copy of its own 270.
bool conv_filter_tc_flat(const Geom& g) {
    if (!g.plain || g.KH != 1 || g.KW != 1 || g.SH != 1 || g.SW != 1 || g.PT != 0 || g.PL != 0 || g.HO != g.H || g.WO != g.W || g.H * g.W == 1) return false;
    const FilterPlan f = make_filter_plan(g);
    if (f.tight || filter_xmajor(g, f)) return false;
    auto fits = [](int blocks, int per) { return blocks % per == 0 || per % blocks == 0; };
    const int per_b = f.Cip / f.cbx, cols = (g.real_in ? 1 : g.nc) * f.Cip, tile_b = (cols < GN ? cols : GN) / f.cbx;
    return fits(GM / f.cby, f.Cop / f.cby) && fits(tile_b, per_b) && (tile_b % 2 != 0 || fits(tile_b / 2, per_b));
}

bool conv_filter_tc_supported(int dtype, int variant, const Geom& g) {
    if (dtype != PCB_F16 && dtype != PCB_BF16) return false;
    if (variant != PCB_VARIANT_16_PRODUCT) return false;
    if (g.dw_io && g.KH * g.KW != 1) return false;                      // input-major gradient: dense layers
    if (g.real_in && !(one_block(g.Ci) && one_block(g.Co) && filter_xmajor(g, make_filter_plan(g)))) return false;
    if (g.SH > 2 || g.SW > 2) return false;
    const FilterPlan f = make_filter_plan(g);
    if ((long long)(g.HO - 1) * g.SH + (long long)(g.KH - 1) * g.DH > 65534 || (long long)(g.WO - 1) * g.SW + (long long)(g.KW - 1) * g.DW > 65534 ||
        f.xp_bytes + f.dyp_bytes > MAX_COPIES) return false;
    return true;
}

size_t conv_filter_tc_scratch_bytes(const Geom& g) {
    const FilterPlan f = make_filter_plan(g);
    return f.xp_bytes + f.dyp_bytes + f.acc_bytes;
}

bool conv_filter_tc_stages_like_forward(const Geom& g) {
    const FilterPlan f = make_filter_plan(g);
    const Plan pl = make_plan(PASS_FWD, g);
    return g.plain && one_block(g.Ci) && !f.tight && !pl.tight && f.xp_bytes == pl.xp_bytes;
}

bool conv_tc_staged_dy_view(const Geom& g, StagedView* view, size_t* bytes) {
    const Plan pl = make_plan(PASS_BWD_DATA, g);
    if (!g.plain || pl.ins_h != 1 || pl.ins_w != 1) return false;   // backward-data reads a zero-inserted copy
    const FilterPlan f = make_filter_plan(g);
    if (f.cby != f.Cop && !conv_filter_tc_flat(g)) return false;      // the filter gradient would block the channels
    if (pl.Cp != f.Cop || pl.tight || f.tight) return false;
    view->Hp = pl.Hp; view->Wp = pl.Wp; view->pad_top = view->pad_left = 0;
    *bytes = pl.xp_bytes;
    return true;
}

int conv_filter_tc_launch(int dtype, const Geom& layer, const void* dy, const void* x, void* dw, void* scratch, int* status,
                          cudaStream_t stream, const void* kept_x, const StagedView* kept_dy, StatusClear* sc) {
    EncodeTiledFn encode = encode_fn();
    if (!encode) { set_error("cuTensorMapEncodeTiled is not available from the driver"); return PCB_ERR_CUDA; }
    const int fmt = dtype == PCB_F16 ? 0 : 1;
    const Geom g = flat_pixels(layer);
    const FilterPlan f = make_filter_plan(g);
    const int taps = g.KH * g.KW;
    // with one channel block per component the staged x is the forward pass's: a copy it kept is read in place
    uint8_t* xp = kept_x ? static_cast<uint8_t*>(const_cast<void*>(kept_x)) : static_cast<uint8_t*>(scratch);
    uint8_t* dyp = static_cast<uint8_t*>(scratch) + f.xp_bytes;
    float* acc = reinterpret_cast<float*>(dyp + f.dyp_bytes);

    // A channels-last tensor with one channel block per component (at most 64 channels, a multiple of 16) already is the staged layout
    // [component][image][h][w][channels]: it is read in place, its padding supplied by out-of-range TMA coordinates.
    const bool direct_x = !g.plain && g.xc == 1 && g.xw == g.Ci && g.xh == g.W * g.Ci && (long long)g.xp == (long long)g.H * g.W * g.Ci &&
                          f.cbx == f.Cip && g.Ci % 16 == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    const bool direct_dy = !g.plain && g.yc == 1 && g.yw == g.Co && g.yh == g.WO * g.Co && (long long)g.yp == (long long)g.HO * g.WO * g.Co &&
                           f.cby == f.Cop && g.Co % 16 == 0 && (reinterpret_cast<uintptr_t>(dy) & 15u) == 0;
    const bool flat = conv_filter_tc_flat(layer);
    bool chain = false;
    {   // stage both activations channels-last, clear the accumulator
        Prologue pro;
        const int lk = g.real_in ? 1 : g.nc;
        const SrcStrides sx = {g.xp, g.xc, g.xh, g.xw}, sy = {g.yp, g.yc, g.yh, g.yw};
        if (!direct_x && !kept_x)
            stage_activations(pro, fmt, x, xp, lk * g.Nb, g.Ci, g.H, g.W, f.H, f.W, f.Cip, 0, 0, 1, 1, f.cbx, stream, flat ? 0 : f.cbx, g.Nb, g.plain ? nullptr : &sx);
        if (!direct_dy && !kept_dy)
            stage_activations(pro, fmt, dy, dyp, g.nc * g.Nb, g.Co, g.HO, g.WO, g.HO, g.WO, f.Cop, 0, 0, 1, 1, f.cby, stream, flat ? 0 : f.cby, g.Nb, g.plain ? nullptr : &sy);
        PCB_CUDA_TRY(cudaGetLastError());
        add_zero_job(pro, acc, f.acc_bytes);
        const int rc = launch_prologue(pro, sc, stream, &chain);
        if (rc != PCB_OK) return rc;
    }

    FGParams p;
    p.nc = g.nc; p.ga = g.ga; p.neg = g.neg;
    p.Nb = g.Nb; p.Co = g.Co; p.Ci = g.Ci; p.HO = g.HO; p.WO = g.WO; p.Cop = f.Cop; p.Cip = f.Cip;
    p.cbA = f.cby; p.cbB = f.cbx;
    p.KH = g.KH; p.KW = g.KW; p.SH = g.SH; p.SW = g.SW; p.DH = g.DH; p.DW = g.DW; p.fmt = fmt;
    {   // pixel box of FK pixels wasting the fewest K rows (boxes of less than four pixels side by side are slow to load: conv_tf32.cu)
        long long best = -1;
        for (int pw = 1; pw <= FK; pw *= 2)
            for (int ph = 1; ph * pw <= FK; ph *= 2) {
                const int pn = FK / (pw * ph);
                const long long vol = (long long)round_up(g.WO, pw) * round_up(g.HO, ph) * round_up(g.Nb, pn) * (pw >= 4 ? 16 : (pw == 2 ? 17 : 19));
                if (best < 0 || vol < best || (vol == best && pw > p.PW)) { best = vol; p.PW = pw; p.PH = ph; p.PN = pn; }
            }
    }
    p.tiles_w = (g.WO + p.PW - 1) / p.PW; p.tiles_h = (g.HO + p.PH - 1) / p.PH; p.tiles_n = (g.Nb + p.PN - 1) / p.PN;
    p.flat = flat ? 1 : 0;
    const cuuint64_t pixels = (cuuint64_t)g.Nb * g.HO * g.WO;
    if (flat) { p.PW = FK; p.PH = p.PN = 1; p.tiles_w = (int)((pixels + FK - 1) / FK); p.tiles_h = p.tiles_n = 1; }
    const int m_cols = g.nc * f.Cop, n_cols = g.nc * f.Cip;
    p.m_tiles = (m_cols + GM - 1) / GM;
    p.n_tiles = (n_cols + GN - 1) / GN;
    p.n_tile_cols = n_cols < GN ? n_cols : GN;           // 4*Cip is a multiple of 64; tiles of a multi-tile problem are full or padded by zero blocks
    p.LK = g.real_in ? 1 : g.nc;
    p.off_w = -g.PL; p.off_h = -g.PT;
    const bool xmajor = filter_xmajor(g, f);
    p.TPG = xmajor ? GM / (p.LK * p.cbB) : 1;
    const int steps_total = p.tiles_w * p.tiles_h * p.tiles_n;
    const bool pair = !xmajor && p.m_tiles % 2 == 0 && (p.n_tile_cols / p.cbB) % 2 == 0 &&
                      worth_pairs((double)taps * p.m_tiles * p.n_tiles * steps_total * (FK / 16) * p.n_tile_cols / GN);
    const int items = xmajor ? (taps + p.TPG - 1) / p.TPG : taps * p.m_tiles * p.n_tiles / (pair ? 2 : 1);
    const int splits = split_count(items, pair ? sm_pairs() : sm_count(), steps_total, 24);
    p.steps_per_split = (steps_total + splits - 1) / splits;
    p.splits = (steps_total + p.steps_per_split - 1) / p.steps_per_split;

    const CUtensorMapDataType dt = fmt == 0 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    auto swz = [](int cb) { return cb == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : (cb == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B); };
    alignas(64) CUtensorMap map_dy, map_x;
    if (flat) {
        auto encode_flat = [&](CUtensorMap* map, const void* base, int C, int cb, int comps, int blocks, const char* what) {
            const int per = C / cb;
            const cuuint64_t dims[5] = {(cuuint64_t)cb, pixels, (cuuint64_t)per, (cuuint64_t)comps, 1};
            const cuuint64_t strides[4] = {(cuuint64_t)C * 2, (cuuint64_t)cb * 2, pixels * C * 2, pixels * C * 2 * comps};
            const cuuint32_t box[5] = {(cuuint32_t)cb, FK, (cuuint32_t)(blocks < per ? blocks : per), (cuuint32_t)(blocks < per ? 1 : blocks / per), 1};
            return make_tensor_map(map, dt, base, 5, dims, strides, box, nullptr, swz(cb), what);
        };
        int rc = encode_flat(&map_dy, kept_dy ? kept_dy->base : dyp, f.Cop, p.cbA, g.nc, GM / p.cbA, "dy");
        if (rc == PCB_OK) rc = encode_flat(&map_x, xp, f.Cip, p.cbB, p.LK, p.n_tile_cols / p.cbB / (pair ? 2 : 1), "x");
        if (rc != PCB_OK) return rc;
    }
    // staged tensors: [component * blocks per component + channel block][image][h][w][cb channels]; the last box extent is
    // the number of channel blocks one tile takes (blocks past the end read as zeros)
    if (!flat) {
        const int Cd = direct_dy ? g.Co : p.cbA;
        const cuuint64_t dims[5] = {(cuuint64_t)Cd, (cuuint64_t)g.WO, (cuuint64_t)g.HO, (cuuint64_t)g.Nb, (cuuint64_t)(g.nc * (f.Cop / p.cbA))};
        cuuint64_t strides[4] = {(cuuint64_t)Cd * 2, (cuuint64_t)g.WO * Cd * 2, (cuuint64_t)g.HO * g.WO * Cd * 2,
                                 (cuuint64_t)g.Nb * g.HO * g.WO * Cd * 2};
        void* dy_base = direct_dy ? const_cast<void*>(dy) : static_cast<void*>(dyp);
        if (kept_dy) {
            // the copy backward-data staged: [d][img][Hp][Wp][Cop] with pixel (0, 0) at (pad_top, pad_left); the map covers the
            // HO x WO pixels only, so the padding is never read and pixels past the end read as zeros, as in the compact copy
            const size_t px = (size_t)f.Cop * 2, plane = (size_t)kept_dy->Hp * kept_dy->Wp * px;
            strides[0] = px; strides[1] = (cuuint64_t)kept_dy->Wp * px; strides[2] = plane; strides[3] = (cuuint64_t)g.Nb * plane;
            dy_base = static_cast<uint8_t*>(const_cast<void*>(kept_dy->base)) + ((size_t)kept_dy->pad_top * kept_dy->Wp + kept_dy->pad_left) * px;
        }
        const cuuint32_t box[5] = {(cuuint32_t)p.cbA, (cuuint32_t)p.PW, (cuuint32_t)p.PH, (cuuint32_t)p.PN, (cuuint32_t)(xmajor ? g.nc : GM / p.cbA)};
        const cuuint32_t es[5] = {1, 1, 1, 1, 1};
        const CUresult r = encode(&map_dy, dt, 5, dy_base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swz(p.cbA),
                                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled (dy) failed with code %d", (int)r); return PCB_ERR_CUDA; }
    }
    if (!flat) {
        const int Wd = direct_x ? g.W : f.W, Hd = direct_x ? g.H : f.H, Cd = direct_x ? g.Ci : p.cbB;
        const cuuint64_t dims[5] = {(cuuint64_t)Cd, (cuuint64_t)Wd, (cuuint64_t)Hd, (cuuint64_t)g.Nb, (cuuint64_t)(p.LK * (f.Cip / p.cbB))};
        const cuuint64_t strides[4] = {(cuuint64_t)Cd * 2, (cuuint64_t)Wd * Cd * 2, (cuuint64_t)Hd * Wd * Cd * 2,
                                       (cuuint64_t)g.Nb * Hd * Wd * Cd * 2};
        const cuuint32_t box[5] = {(cuuint32_t)p.cbB, (cuuint32_t)((p.PW - 1) * g.SW + 1), (cuuint32_t)((p.PH - 1) * g.SH + 1), (cuuint32_t)p.PN,
                                   (cuuint32_t)(xmajor ? p.LK : p.n_tile_cols / p.cbB / (pair ? 2 : 1))};
        const cuuint32_t es[5] = {1, (cuuint32_t)g.SW, (cuuint32_t)g.SH, 1, 1};
        const CUresult r = encode(&map_x, dt, 5, direct_x ? const_cast<void*>(x) : static_cast<void*>(xp), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swz(p.cbB),
                                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled (x) failed with code %d", (int)r); return PCB_ERR_CUDA; }
    }
    if (xmajor) {
        PCB_CUDA_TRY(cudaFuncSetAttribute(qconv_filter_xmajor_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FG_SMEM));
        PCB_CUDA_TRY(launch_chained_if(chain, qconv_filter_xmajor_tc_kernel, items * p.splits, G_THREADS, FG_SMEM, stream, map_x, map_dy, p, acc, status));
    } else {
        auto* kernel = pair ? qconv_filter_general_tc_kernel<true> : qconv_filter_general_tc_kernel<false>;
        PCB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FG_SMEM));
        PCB_CUDA_TRY(launch_clusters(pair ? 2 : 1, chain, kernel, items * p.splits * (pair ? 2 : 1), G_THREADS, FG_SMEM, stream, map_dy, map_x, p, acc, status));
    }
    PCB_CUDA_TRY(cudaGetLastError());
    const size_t per_tap = (size_t)g.nc * g.Co * g.Ci, total = per_tap * taps;
    const int blocks = (int)((total + 255) / 256 < 2368 ? (total + 255) / 256 : 2368);
    const FilterStrides ds = {g.dr, g.dco, g.dci, g.dkh, g.dkw, g.KW};
    const int dense_oihw = (g.dci == taps && g.dco == g.Ci * taps && (long long)g.dr == (long long)g.Co * g.Ci * taps && g.dkh == g.KW && g.dkw == 1) ? 1 : 0;
    if (fmt == 0) PCB_CUDA_TRY(launch_chained(unpack_filter_grad_kernel<__half>, blocks, 256, 0, stream, acc, (__half*)dw, taps, per_tap, dense_oihw, g.Co, g.Ci, ds));
    else PCB_CUDA_TRY(launch_chained(unpack_filter_grad_kernel<__nv_bfloat16>, blocks, 256, 0, stream, acc, (__nv_bfloat16*)dw, taps, per_tap, dense_oihw, g.Co, g.Ci, ds));
    PCB_CUDA_TRY(cudaGetLastError());
    return PCB_OK;
}

}  // namespace pcb
