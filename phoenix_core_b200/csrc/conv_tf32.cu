// fp32 quaternion convolution and dense on the tensor cores with error-compensated TF32 (three products).
//
// tcgen05.mma.kind::tf32 keeps 10 mantissa bits of each fp32 operand, far from the 1e-5 parity the fp32 path
// owes. Every operand is therefore split while it is staged into hi, x rounded to a TF32 number, and lo = x - hi
// (exact in fp32, at most 2^-11 of x), and a product is hi*hi + lo*hi + hi*lo. What is dropped is lo*lo (2^-22) and the last bit of each lo that TF32
// does not hold (2^-23): at most 2^-21 of a product, 4.8e-7. Against 64 bits,
// 2-norm of the difference over that of the result, forward: one product 8e-8; 1x1, 16 and 32 channels 2.0e-7 and 3.4e-7; 3x3, 16 channels 7.0e-7, 128
// channels 7.9e-7; all filter gradients below 9.3e-7. Constant planes, whose errors all have one sign: 1.4e-6 at most. (With the cross terms in
// bf16, four fifths of the time where the MMAs bound: one product 6.5e-7, 7.0e-7, 7.3e-7, 9.7e-7, 1.38e-6, 1.39e-6, constant planes 3.3e-6.)
//
// Structure as in conv_tc.cu: channels-last activations (not padded: the zero fill of the tensor maps is
// the padding) and the signed/permuted filter matrix
// Wexp[tap][(d,co)][(l,ci)] (reference sign table src/algebras.cc:28-49) are staged in the workspace, here in fp32
// and twice (hi, lo); the implicit-GEMM kernel is TMA-fed, 128 x 256 tile.
// Dense layers are the 1x1 convolution of 1x1 images (pixels = batch); input-major dense filters and the
// input-major dense filter gradient are handled while staging / unstaging. Replaces, for fp32 tensors, the scalar
// fp32 library calls of src/backend/cudnn/conv2d.hpp:280-309, :447-488 and src/backend/cudnn/dense.hpp:102-133, :181-216.
#include "column_halves.h"
#include "tc_common.cuh"
#include "tensor_path.cuh"

namespace pcb {
namespace {

using namespace umma;
using namespace tc;

constexpr int TM = 128, TN = 256, TKS = 16;                 // tile, channels (fp32) per K slice: 64-byte rows
constexpr int T_THREADS = 320;
constexpr uint32_t TA_BYTES = TM * TKS * 4, TB_BYTES = TN * TKS * 4;
constexpr uint32_t T_STAGE = 2 * (TA_BYTES + TB_BYTES);     // hi and lo of both operands: 48 KB
constexpr int T_STAGES = 4, TP_STAGES = 6;                  // PAIR: half of the pixels in each CTA, 32 KB
constexpr int T_MAX_SLOTS = 10, T_HALO_TILES = 2;           // halo form: filter slices and halo tiles in flight
constexpr size_t T_SMEM = 1024 + T_STAGES * T_STAGE + 512;
constexpr int ST_T_PRODUCER = 0x1000, ST_T_MMA = 0x2000, ST_T_EPILOGUE = 0x4000;

struct TParams {
    int Nb, Mvalid, Cout, HO, WO, Cp;
    int KH, KW, SH, SW, DH, DW;
    int PW, PH, PN;
    int tiles_w, tiles_h, tiles_n, tiles_m;
    int has_bias, LK, store_vec;
    int n_cols;                       // pixels of a tile: 256, 128 where few tiles leave most SMs idle, 8 * PH in halo form
    int apart;                        // column of a buffer where the cross terms are summed: 128, or 0 with hi * hi
    int n_chunks, chunk_len;          // a work item's K range runs in n_chunks pieces of at most chunk_len stages
    int off_w, off_h;                 // added to the pixel coordinates of every activation box: minus the padding; 0 for a zero-inserted copy
    int rows_epi;                     // image rows not a multiple of 8 pixels: stored through shared memory (store_rows_f32)
    int splits, k_per_split;          // the K loop of a tile is cut into `splits` work items of k_per_split stages; with more than one
                                      // the partial results meet in the (zeroed) output by fp32 reductions
    int Wt, Ht, a_slots;              // halo form: halo tile, filter slices in flight
    int split_w, split_h, split_n;    // PAIR: pixels, pixel rows and images from the even CTA's half of the tile box to the odd one's
    uint32_t halo_bytes;              // halo form: shared-memory pitch of the hi (and of the lo) part of a halo tile
};

// K-major tile with 64-byte rows, 64-byte swizzle, groups of 8 rows `group_bytes` apart (512, or the row pitch of a halo tile).
__device__ __forceinline__ uint64_t desc_k64(uint32_t addr, uint32_t group_bytes = 512) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)((group_bytes >> 4) & 0x3FFFu) << 32) | DESC_VERSION_SM100 | (4ull << 61);
}

// Each MMA truncates when it adds into the TMEM accumulator, so the error of one accumulator grows with the number
// of MMAs it takes (measured: about 3e-8 of the largest output per MMA). K loops are therefore cut into chunks; chunks alternate between
// the two TMEM buffers (as whole tiles do when one chunk is enough) and the epilogue warps add them up in registers, rounding to nearest.
// A buffer has 256 columns. Tiles of up to 128 sum the cross terms, 2^-11 of the size, in the other half of them: a chunk is T_CHUNK_APART stages,
// 64 MMAs of hi * hi. In wider tiles the three products share the accumulator and a chunk is T_CHUNK stages, 42 MMAs.
constexpr int T_SPLIT = 16;           // fewest stages of a work item
constexpr int T_CHUNK = 7, T_CHUNK_APART = 32;

// HALO (stride-1 correlation, tile = 8 x PH pixels of one image): as in conv_tc.cu, the halo tile of 16 channels is loaded once and every
// tap's MMAs read it at a shifted start address; the filter slices have a ring of their own. 20 KB instead of 48 KB from L2 per six MMAs of
// 128 x 224, which take 672 clocks (an SM takes in about 64 bytes per clock). Forward, us, without / with: 3x3, 32 channels, 56 x 52, batch 40 225 / 205;
// 3x3, 128 channels, 28 x 28, batch 128, where the MMAs bound at the power limit, the same within the spread (2.10 / 2.13 ms).
// PAIR: a cluster of two CTAs takes two neighbouring row tiles and half of the pixels each, as in conv_tc.cu. Forward, us, without / with: 3x3, 128 channels,
// 28 x 28, batch 128 2272 / 2158; 64 channels, 56 x 56, batch 32 578 / 546.
template <bool CHUNKED, bool HALO, bool PAIR>
__global__ void __launch_bounds__(T_THREADS, 1)
qconv_general_tf32_kernel(const __grid_constant__ CUtensorMap map_w_hi, const __grid_constant__ CUtensorMap map_w_lo,
                          const __grid_constant__ CUtensorMap map_x_hi, const __grid_constant__ CUtensorMap map_x_lo, TParams p,
                          const float* bias, float* __restrict__ out, int* __restrict__ status) {
    constexpr int MAX_SLOTS = HALO ? T_MAX_SLOTS : (PAIR ? TP_STAGES : T_STAGES);
    constexpr uint32_t B_PART = PAIR ? TB_BYTES / 2 : TB_BYTES, SLOT = HALO ? 2 * TA_BYTES : 2 * (TA_BYTES + B_PART);
    const int slots = HALO ? p.a_slots : MAX_SLOTS;
    const int rank = PAIR ? (int)cluster_ctarank() : 0, first = PAIR ? blockIdx.x / 2 : blockIdx.x, step = PAIR ? gridDim.x / 2 : gridDim.x;
    extern __shared__ uint8_t smem_raw[];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t operand_bytes = slots * SLOT + (HALO ? T_HALO_TILES * 2 * p.halo_bytes : 0u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + operand_bytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * MAX_SLOTS + 4 + 2 * T_HALO_TILES);
    const uint32_t tiles_addr = smem_u32(base), halo_addr = tiles_addr + slots * SLOT;
    const uint32_t full_bar = smem_u32(bars), empty_bar = smem_u32(bars + MAX_SLOTS);
    const uint32_t tmem_full = smem_u32(bars + 2 * MAX_SLOTS), tmem_empty = smem_u32(bars + 2 * MAX_SLOTS + 2);
    const uint32_t halo_full = smem_u32(bars + 2 * MAX_SLOTS + 4), halo_empty = halo_full + 8 * T_HALO_TILES;

    const int tiles_m = PAIR ? p.tiles_m / 2 : p.tiles_m, n_items = p.tiles_w * p.tiles_h * p.tiles_n * tiles_m * p.splits;
    const int c_steps = p.Cp / TKS, taps = p.KH * p.KW;
    const int n_k = taps * p.LK * c_steps;

    if (t == 0) {
        for (int s = 0; s < MAX_SLOTS; ++s) { mbar_init(full_bar + 8 * s, 1); mbar_init(empty_bar + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(tmem_full + 8 * b, 1); mbar_init(tmem_empty + 8 * b, PAIR ? 16 : 8); }
        for (int s = 0; s < T_HALO_TILES; ++s) { mbar_init(halo_full + 8 * s, 1); mbar_init(halo_empty + 8 * s, 1); }
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
        const bool el = elect_one();
        int s = 0, phase = 1, hs = 0, hphase = 1;
        bool ok = true;
        for (int item = first; item < n_items && ok; item += step) {
            const int tile = item / p.splits, split = item - tile * p.splits;
            const int tm = PAIR ? 2 * (tile % tiles_m) + rank : tile % tiles_m;
            int rest = tile / tiles_m;
            const int tw = rest % p.tiles_w; rest /= p.tiles_w;
            const int th = rest % p.tiles_h;
            const int tn = rest / p.tiles_h;
            const int m0 = tm * TM, ow0 = tw * p.PW + rank * p.split_w, oh0 = th * p.PH + rank * p.split_h, n0 = tn * p.PN + rank * p.split_n;
            const int k0 = split * p.k_per_split, k1 = min(n_k, k0 + p.k_per_split);
            if (HALO) {                                  // stage k = (l * c_steps + cs) * taps + tap
                for (int l = 0; l < p.LK && ok; ++l)
                    for (int cs = 0; cs < c_steps && ok; ++cs) {
                        ok = warp_wait_bounded(halo_empty + 8 * hs, hphase, status, ST_T_PRODUCER);
                        if (!ok) break;
                        if (el && PAIR) {
                            const uint32_t dst = halo_addr + hs * 2 * p.halo_bytes, lead = map_to_cta(halo_full + 8 * hs, 0);
                            if (rank == 0) mbar_arrive_expect_tx(halo_full + 8 * hs, 4 * (uint32_t)p.Wt * p.Ht * TKS * 4);
                            tma_load_5d_pair(dst, &map_x_hi, cs * TKS, ow0 + p.off_w, oh0 + p.off_h, n0, l, lead);
                            tma_load_5d_pair(dst + p.halo_bytes, &map_x_lo, cs * TKS, ow0 + p.off_w, oh0 + p.off_h, n0, l, lead);
                        } else if (el) {
                            const uint32_t dst = halo_addr + hs * 2 * p.halo_bytes, bar = halo_full + 8 * hs;
                            mbar_arrive_expect_tx(bar, 2 * (uint32_t)p.Wt * p.Ht * TKS * 4);
                            tma_load_5d(dst, &map_x_hi, cs * TKS, ow0 + p.off_w, oh0 + p.off_h, n0, l, bar);              // [Ht][Wt][16 channels]
                            tma_load_5d(dst + p.halo_bytes, &map_x_lo, cs * TKS, ow0 + p.off_w, oh0 + p.off_h, n0, l, bar);
                        }
                        if (++hs == T_HALO_TILES) { hs = 0; hphase ^= 1; }
                        for (int tap = 0; tap < taps; ++tap) {
                            ok = warp_wait_bounded(empty_bar + 8 * s, phase, status, ST_T_PRODUCER);
                            if (!ok) break;
                            if (el && PAIR) {
                                const uint32_t dst = tiles_addr + s * SLOT, lead = map_to_cta(full_bar + 8 * s, 0);
                                if (rank == 0) mbar_arrive_expect_tx(full_bar + 8 * s, 2 * SLOT);
                                tma_load_3d_pair(dst, &map_w_hi, l * p.Cp + cs * TKS, m0, tap, lead);
                                tma_load_3d_pair(dst + TA_BYTES, &map_w_lo, l * p.Cp + cs * TKS, m0, tap, lead);
                            } else if (el) {
                                const uint32_t dst = tiles_addr + s * SLOT, bar = full_bar + 8 * s;
                                mbar_arrive_expect_tx(bar, SLOT);
                                tma_load_3d(dst, &map_w_hi, l * p.Cp + cs * TKS, m0, tap, bar);
                                tma_load_3d(dst + TA_BYTES, &map_w_lo, l * p.Cp + cs * TKS, m0, tap, bar);
                            }
                            if (++s == slots) { s = 0; phase ^= 1; }
                        }
                    }
                continue;
            }
            // stage k = (tap * LK + l) * c_steps + cs
            int cs = k0 % c_steps, l = (k0 / c_steps) % p.LK, tap = k0 / (c_steps * p.LK);
            for (int k = k0; k < k1; ++k) {
                const int kh = tap / p.KW, kw = tap - kh * p.KW;
                const int wp0 = ow0 * p.SW + kw * p.DW + p.off_w, hp0 = oh0 * p.SH + kh * p.DH + p.off_h;
                ok = warp_wait_bounded(empty_bar + 8 * s, phase, status, ST_T_PRODUCER);
                if (!ok) break;
                if (el && PAIR) {
                    const uint32_t dst = tiles_addr + s * SLOT, lead = map_to_cta(full_bar + 8 * s, 0);
                    if (rank == 0) mbar_arrive_expect_tx(full_bar + 8 * s, 2 * SLOT);
                    tma_load_3d_pair(dst, &map_w_hi, l * p.Cp + cs * TKS, m0, tap, lead);
                    tma_load_3d_pair(dst + TA_BYTES, &map_w_lo, l * p.Cp + cs * TKS, m0, tap, lead);
                    tma_load_5d_pair(dst + 2 * TA_BYTES, &map_x_hi, cs * TKS, wp0, hp0, n0, l, lead);
                    tma_load_5d_pair(dst + 2 * TA_BYTES + B_PART, &map_x_lo, cs * TKS, wp0, hp0, n0, l, lead);
                } else if (el) {
                    const uint32_t dst = tiles_addr + s * SLOT, bar = full_bar + 8 * s;
                    mbar_arrive_expect_tx(bar, 2 * (TA_BYTES + (uint32_t)p.n_cols * TKS * 4));
                    tma_load_3d(dst, &map_w_hi, l * p.Cp + cs * TKS, m0, tap, bar);
                    tma_load_3d(dst + TA_BYTES, &map_w_lo, l * p.Cp + cs * TKS, m0, tap, bar);
                    tma_load_5d(dst + 2 * TA_BYTES, &map_x_hi, cs * TKS, wp0, hp0, n0, l, bar);
                    tma_load_5d(dst + 2 * TA_BYTES + TB_BYTES, &map_x_lo, cs * TKS, wp0, hp0, n0, l, bar);
                }
                if (++s == slots) { s = 0; phase ^= 1; }
                if (++cs == c_steps) { cs = 0; if (++l == p.LK) { l = 0; ++tap; } }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        const bool el = elect_one();
        constexpr int M = PAIR ? 2 * TM : TM;
        const uint32_t idesc = make_idesc_f16(2, M, p.n_cols, false, false);
        auto mma = [&](uint32_t d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t acc) {
            if (PAIR) mma_tf32_pair(d, a_lo, a_hi, b_lo, b_hi, idesc, acc);
            else mma_tf32_ss_words(d, a_lo, a_hi, b_lo, b_hi, idesc, acc);
        };
        auto commit = [](uint32_t bar) {              // in both CTAs
            if (PAIR) { mma_commit_pair(bar); mma_commit_pair(map_to_cta(bar, 1)); }
            else mma_commit(bar);
        };
        const uint32_t row_step = (uint32_t)(p.DH * p.Wt * TKS * 4) >> 4, col_step = (uint32_t)(p.DW * TKS * 4) >> 4;      // HALO
        int s = 0, phase = 0, hs = 0, hphase = 0, unit = 0;      // unit = one accumulator's worth of work: a chunk of a tile
        bool ok = rank == 0;                          // PAIR: the even CTA issues the MMAs of both
        for (int item = first; item < n_items && ok; item += step) {
            const int split = item % p.splits;
            const int k0 = split * p.k_per_split, k1 = min(n_k, k0 + p.k_per_split);
            int tap = 0, kw = 0;
            uint32_t b_row = 0;                                    // HALO: start-address offset of the tap's filter row
            for (int c = 0; c < p.n_chunks && ok; ++c, ++unit) {
                const int buf = unit & 1, use = unit >> 1;
                if (use > 0) {
                    ok = warp_wait_bounded(tmem_empty + 8 * buf, (use - 1) & 1, status, ST_T_MMA);
                    if (!ok) break;
                    tc_fence_after_sync();
                }
                const uint32_t d = tmem_base + buf * TN, d_cross = d + p.apart;
                const int k_beg = k0 + c * p.chunk_len, k_end = min(k1, k_beg + p.chunk_len);
                for (int k = k_beg; k < k_end; ++k) {
                    if (HALO && tap == 0) {
                        ok = warp_wait_bounded(halo_full + 8 * hs, hphase, status, ST_T_MMA);
                        if (!ok) break;
                    }
                    ok = warp_wait_bounded(full_bar + 8 * s, phase, status, ST_T_MMA);
                    if (!ok) break;
                    tc_fence_after_sync();
                    if (el) {
                        const uint32_t a_hi = tiles_addr + s * SLOT, b_hi = HALO ? halo_addr + hs * 2 * p.halo_bytes : a_hi + 2 * TA_BYTES;
                        const uint64_t ad = desc_k64(a_hi), bd = desc_k64(b_hi, HALO ? p.Wt * TKS * 4 : 512);
                        const uint32_t a0 = (uint32_t)ad, ah = (uint32_t)(ad >> 32), b0 = (uint32_t)bd + (HALO ? b_row + kw * col_step : 0u), bh = (uint32_t)(bd >> 32);
                        const uint32_t a1 = a0 + (TA_BYTES >> 4), b1 = b0 + ((HALO ? p.halo_bytes : B_PART) >> 4);
#pragma unroll
                        for (int j = 0; j < 2; ++j) {                   // 8 fp32 = 32 bytes per MMA along a row
                            const uint32_t acc = (k > k_beg || j > 0) ? 1u : 0u;
                            mma(d_cross, a1 + 2 * j, ah, b0 + 2 * j, bh, acc);                          // small terms first
                            mma(d_cross, a0 + 2 * j, ah, b1 + 2 * j, bh, 1u);
                            mma(d, a0 + 2 * j, ah, b0 + 2 * j, bh, p.apart ? acc : 1u);
                        }
                        commit(empty_bar + 8 * s);
                        if (HALO && tap == taps - 1) commit(halo_empty + 8 * hs);
                        if (k == k_end - 1) commit(tmem_full + 8 * buf);
                    }
                    if (++s == slots) { s = 0; phase ^= 1; }
                    if (HALO) {
                        if (++kw == p.KW) { kw = 0; b_row += row_step; }
                        if (++tap == taps) { tap = 0; kw = 0; b_row = 0; if (++hs == T_HALO_TILES) { hs = 0; hphase ^= 1; } }
                    }
                }
            }
        }
        __syncwarp();
    } else {
        const int q = warp & 3, chalf = (warp - 2) >> 2;
        const int sv = p.store_vec;                  // pixels per store: 8, 4, 2 or 1
        const int half = columns_per_half(p.n_cols);                // columns of a warp: chalf * half and on
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + chalf * half;
        int unit = 0;
        bool ok = true;
        const bool reduce = p.splits > 1;            // partial sums of a tile meet in the zeroed output
        for (int item = first; item < n_items && ok; item += step) {
            const int tile = item / p.splits, split = item - tile * p.splits;
            const int tm = PAIR ? 2 * (tile % tiles_m) + rank : tile % tiles_m;
            int rest = tile / tiles_m;
            const int tw = rest % p.tiles_w; rest /= p.tiles_w;
            const int th = rest % p.tiles_h;
            const int tn = rest / p.tiles_h;
            const int ow0 = tw * p.PW, oh0 = th * p.PH, n0 = tn * p.PN;
            const int m = tm * TM + q * 32 + lane;
            const bool row_ok = m < p.Mvalid;
            const int d = row_ok ? m / p.Cout : 0, co = m - d * p.Cout;
            const float badd = (row_ok && p.has_bias && split == 0) ? ld_chained(bias + d * p.Cout + co) : 0.f;
            uint32_t part[CHUNKED ? 4 : 1][32];                     // this thread's 128 columns, summed over the chunks so far
            if (CHUNKED) {
#pragma unroll
                for (int cb = 0; cb < 4; ++cb)
#pragma unroll
                    for (int e = 0; e < 32; ++e) part[CHUNKED ? cb : 0][e] = 0u;
                // 16 columns at a time: with 32 the kernel spills, and what it spilled waits behind the stores of the tile
                auto add = [&](int cb, int h, uint32_t at) {
                    uint32_t v[16];
                    tmem_ld_32x32b_x16(at, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        part[CHUNKED ? cb : 0][16 * h + e] = __float_as_uint(__uint_as_float(part[CHUNKED ? cb : 0][16 * h + e]) + __uint_as_float(v[e]));
                };
                const int seen = read_status(status);               // (once per tile: in front of every chunk it would wait behind the stores of the last tile)
                // (the last chunk too: its buffer is free for the next tile while this one is stored)
                for (int c = 0; c < p.n_chunks && ok; ++c, ++unit) {
                    const int buf = unit & 1, use = unit >> 1;
                    ok = mbar_wait_bounded(tmem_full + 8 * buf, use & 1, status, ST_T_EPILOGUE);
                    ok = warp_may_store(ok, seen);
                    if (!ok) break;
                    tc_fence_after_sync();
#pragma unroll
                    for (int cb = 0; cb < 4; ++cb) {
                        if (cb * 32 >= half || chalf * half + cb * 32 >= p.n_cols) break;
                        const uint32_t at = lane_addr + buf * TN + cb * 32;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            add(cb, h, at + 16 * h);
                            if (p.apart) add(cb, h, at + 16 * h + p.apart);
                        }
                    }
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) { if (PAIR) mbar_arrive_cluster(map_to_cta(tmem_empty + 8 * buf, 0)); else mbar_arrive(tmem_empty + 8 * buf); }
                }
                if (!ok) break;
            }
            const int buf = unit & 1, use = unit >> 1;
            if (!CHUNKED) {
                ++unit;
                const int seen = read_status(status);
                ok = mbar_wait_bounded(tmem_full + 8 * buf, use & 1, status, ST_T_EPILOGUE);
                ok = warp_may_store(ok, seen);
                if (!ok) break;
                tc_fence_after_sync();
            }
#pragma unroll(CHUNKED ? 4 : 1)
            for (int cb = 0; cb < 4; ++cb) {
                uint32_t(&v)[32] = part[CHUNKED ? cb : 0];
                const int col0 = chalf * half + cb * 32;
                if (cb * 32 >= half || col0 >= p.n_cols) break;
                if (!CHUNKED) {
                    tmem_ld_32x32b_x32(lane_addr + buf * TN + cb * 32, v);
                    tmem_ld_wait();
                    if (p.apart) {
                        uint32_t u[32];
                        tmem_ld_32x32b_x32(lane_addr + buf * TN + p.apart + cb * 32, u);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) + __uint_as_float(u[e]));
                    }
                }
#pragma unroll
                for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) + badd);
                if (!row_ok && !p.rows_epi) continue;
                if (p.rows_epi) {
                    const uint32_t rbuf = smem_u32(base) + operand_bytes + 512 + (uint32_t)(warp - 2) * EPI_ROWS_F32_BYTES;
                    const int HWo = p.HO * p.WO, je = col0 + (sv == 1 ? lane : (sv == 2 ? (lane & 15) * 2 : (lane & 7) * 4));
                    const int wl = je % p.PW, hl = (je / p.PW) % p.PH, nl = je / (p.PW * p.PH);
                    const int ow = ow0 + wl, oh = oh0 + hl, img = n0 + nl;
                    const int pix_off = (je < p.n_cols && ow < p.WO && oh < p.HO && img < p.Nb) ? (img * p.Cout * p.HO + oh) * p.WO + ow : -1;
                    const int row_off = row_ok ? (d * p.Nb * p.Cout + co) * HWo : -1;
                    if (p.Mvalid <= 64) {
                        if (tm * TM + q * 32 >= p.Mvalid) continue;         // (a warp without rows)
                        if (sv == 1) store_rows_f32_few<1>(rbuf, v, out, row_off, pix_off, lane, reduce);
                        else if (sv == 2) store_rows_f32_few<2>(rbuf, v, out, row_off, pix_off, lane, reduce);
                        else store_rows_f32_few<4>(rbuf, v, out, row_off, pix_off, lane, reduce);
                    } else if (sv == 1) store_rows_f32<1>(rbuf, v, out, row_off, pix_off, lane, reduce);
                    else if (sv == 2) store_rows_f32<2>(rbuf, v, out, row_off, pix_off, lane, reduce);
                    else store_rows_f32<4>(rbuf, v, out, row_off, pix_off, lane, reduce);
                    continue;
                }
#pragma unroll
                for (int g8 = 0; g8 < 4; ++g8) {
                    const int j = col0 + g8 * 8;
                    if (j >= p.n_cols) continue;
                    const int wl = j % p.PW, hl = (j / p.PW) % p.PH, nl = j / (p.PW * p.PH);
                    const int ow = ow0 + wl, oh = oh0 + hl, img = n0 + nl;
                    if (p.PW >= 8) {
                        if (ow >= p.WO || oh >= p.HO || img >= p.Nb) continue;
                        float* dst = out + (((size_t)(d * p.Nb + img) * p.Cout + co) * p.HO + oh) * p.WO + ow;
                        if (reduce) {                      // rows of whole 8-pixel runs (all others: store_rows_f32)
#pragma unroll
                            for (int h = 0; h < 2; ++h)
                                red_add_f32x4(dst + 4 * h, __uint_as_float(v[8 * g8 + 4 * h]), __uint_as_float(v[8 * g8 + 4 * h + 1]),
                                              __uint_as_float(v[8 * g8 + 4 * h + 2]), __uint_as_float(v[8 * g8 + 4 * h + 3]));
                        } else {
                            st_global_v8(dst, &v[8 * g8]);
                        }
                    } else {
                        // narrow boxes (dense layers: one pixel per image): every column is its own (image, row, pixel)
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const int je = j + e;
                            const int w2 = je % p.PW, h2 = (je / p.PW) % p.PH, n2 = je / (p.PW * p.PH);
                            if (ow0 + w2 < p.WO && oh0 + h2 < p.HO && n0 + n2 < p.Nb) {
                                float* dst = out + (((size_t)(d * p.Nb + n0 + n2) * p.Cout + co) * p.HO + oh0 + h2) * p.WO + ow0 + w2;
                                if (reduce) atomicAdd(dst, __uint_as_float(v[8 * g8 + e]));
                                else *dst = __uint_as_float(v[8 * g8 + e]);
                            }
                        }
                    }
                }
            }
            if (!CHUNKED) {
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) { if (PAIR) mbar_arrive_cluster(map_to_cta(tmem_empty + 8 * buf, 0)); else mbar_arrive(tmem_empty + 8 * buf); }
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (PAIR) cluster_sync_all();                     // nobody leaves while its peer may still signal its barriers or read its shared memory
    if (warp == 1) { if (PAIR) tmem_dealloc_pair(tmem_base, 512); else tmem_dealloc(tmem_base, 512); }
}

// ---- staging: fp32 -> (hi, lo) ------------------------------------------------------------------------
// hi: x rounded to a TF32 number, or cut off where rounding a finite x would overflow; lo: x - hi (exact). Infinities and NaN make lo a NaN.
__device__ __forceinline__ void split_f32(float x, float& hi, float& lo) {
    const uint32_t u = __float_as_uint(x);
    uint32_t h = (u + 0x1000u) & 0xFFFFE000u;
    if ((h & 0x7F800000u) == 0x7F800000u) h = u & 0xFFFFE000u;
    hi = __uint_as_float(h);
    lo = x - hi;
}
// N (4 or 8) channels of a pixel, aligned to 16 bytes.
template <int N>
__device__ __forceinline__ void store_split(const float (&f)[N], float* hi, float* lo) {
    float h[N], l[N];
#pragma unroll
    for (int e = 0; e < N; ++e) split_f32(f[e], h[e], l[e]);
    if (N == 8) {
        uint32_t w[8], v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) { w[e] = __float_as_uint(h[e < N ? e : 0]); v[e] = __float_as_uint(l[e < N ? e : 0]); }
        if (((reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo)) & 31u) == 0) {      // (whole sectors)
            st_global_v8(hi, w);
            st_global_v8(lo, v);
        } else {                                     // the workspace is only 16-byte aligned
#pragma unroll
            for (int e = 0; e < 8; e += 4) {
                *reinterpret_cast<uint4*>(hi + e) = make_uint4(w[e], w[e + 1], w[e + 2], w[e + 3]);
                *reinterpret_cast<uint4*>(lo + e) = make_uint4(v[e], v[e + 1], v[e + 2], v[e + 3]);
            }
        }
    } else {
        *reinterpret_cast<float4*>(hi) = make_float4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<float4*>(lo) = make_float4(l[0], l[1], l[2], l[3]);
    }
}

// A block takes 32 consecutive padded pixels of one plane and up to 64 channels at a time through shared memory: the NCHW reads
// run along the pixels of one channel (coalesced), the channels-last writes along the channel groups of one pixel (coalesced;
// a thread per (pixel, 4 channels) writes one float4 of hi and one of lo).
__global__ void __launch_bounds__(256)
pack_activations_f32_kernel(const float* __restrict__ x, float* __restrict__ hi, float* __restrict__ lo, int planes, int C,
                            int H, int W, int Hp, int Wp, int Cp, int pad_top, int pad_left, int ins_h, int ins_w,
                            int cb, int Nb) {
    __shared__ float tile[64][33];
    const int PP = Hp * Wp, tiles_pp = (PP + 31) / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long n_tiles = (long long)planes * tiles_pp;
    for (long long t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        const int plane = (int)(t / tiles_pp), pp0 = (int)(t - (long long)plane * tiles_pp) * 32;
        const int pp = pp0 + lane;
        const int hp = pp / Wp, wp = pp - hp * Wp;
        int ih = hp - pad_top, iw = wp - pad_left;
        bool inside = pp < PP && ih >= 0 && iw >= 0;
        if (inside && (ins_h > 1 || ins_w > 1)) {
            inside = (ih % ins_h == 0) && (iw % ins_w == 0);
            ih /= ins_h; iw /= ins_w;
        }
        inside = inside && ih < H && iw < W;
        const float* src = x + ((size_t)plane * C * H + ih) * W + iw;      // + c * H * W
        for (int c0 = 0; c0 < Cp; c0 += 64) {
            const int c_pass = min(64, Cp - c0);
            for (int c = warp; c < c_pass; c += 8) tile[c][lane] = (inside && c0 + c < C) ? __ldg(src + (size_t)(c0 + c) * H * W) : 0.f;
            __syncthreads();
            const int groups = c_pass / 4;
            for (int idx = threadIdx.x; idx < 32 * groups; idx += 256) {
                const int g = idx % groups, px = idx / groups;
                if (pp0 + px >= PP) continue;
                const float f[4] = {tile[4 * g][px], tile[4 * g + 1][px], tile[4 * g + 2][px], tile[4 * g + 3][px]};
                const int ch = c0 + 4 * g;
                size_t o = ((size_t)plane * PP + pp0 + px) * Cp + ch;
                if (cb > 0) {   // blocks of cb channels, block index outermost: [comp * (Cp / cb) + c / cb][img][hp][wp][cb]
                    const int comp = plane / Nb, img = plane - comp * Nb, bl = ch / cb;
                    o = ((((size_t)comp * (Cp / cb) + bl) * Nb + img) * PP + pp0 + px) * cb + (ch - bl * cb);
                }
                store_split(f, hi + o, lo + o);
            }
            __syncthreads();
        }
    }
}

// The same staging, one thread per (pixel, 4 channels), for planes of fewer than 32 padded pixels (dense layers are 1 x 1 images:
// consecutive threads then walk the channel groups of one row, and both sides are contiguous).
__global__ void pack_activations_f32_small_kernel(const float* __restrict__ x, float* __restrict__ hi, float* __restrict__ lo, int planes, int C,
                                                  int H, int W, int Hp, int Wp, int Cp, int pad_top, int pad_left, int ins_h, int ins_w,
                                                  int cb, int Nb) {
    const int groups = Cp / 4;
    const size_t total = (size_t)planes * Hp * Wp * groups;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        const int wp = (int)(idx % Wp);
        size_t rest = idx / Wp;
        const int grp = (int)(rest % groups); rest /= groups;
        const int hp = (int)(rest % Hp);
        const int plane = (int)(rest / Hp);
        int ih = hp - pad_top, iw = wp - pad_left;
        bool inside = ih >= 0 && iw >= 0;
        if (inside && (ins_h > 1 || ins_w > 1)) {
            inside = (ih % ins_h == 0) && (iw % ins_w == 0);
            ih /= ins_h; iw /= ins_w;
        }
        inside = inside && ih < H && iw < W;
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int c = grp * 4 + e;
            v[e] = (c < C && inside) ? __ldg(x + (((size_t)plane * C + c) * H + ih) * W + iw) : 0.f;
        }
        size_t o = (((size_t)plane * Hp + hp) * Wp + wp) * Cp + grp * 4;
        if (cb > 0) {
            const int comp = plane / Nb, img = plane - comp * Nb, b = (grp * 4) / cb;
            o = (((((size_t)comp * (Cp / cb) + b) * Nb + img) * Hp + hp) * Wp + wp) * cb + (grp * 4 - b * cb);
        }
        store_split(v, hi + o, lo + o);
    }
}

// ---- everything a call needs before its main kernel, in one launch (as in conv_tc.cu): status word, filters, copies, zeroed output ----
// Staging of dense NCHW tensors without padding, x[plane][C][HW] -> hi, lo [plane][HW][Cp] (blocked == 0) or blocks of 4 U channels
// with the block index outermost: the transposition of conv_tc.cu's stage_compact with units of four channels, split into hi and lo
// where the units leave shared memory. Blocks of 64 channels wherever there are more than 32 (the last one may hold fewer): a CTA writes
// 256 bytes per pixel. 112 channels of 67 x 67, batch 125, 2 x 1 taps, forward 691 us, with blocks of 16 channels 811; 48 channels of
// 56 x 56, batch 32, 1 x 1, 99 / 120.
struct StageJob32 {
    const float* x;
    float *hi, *lo;
    unsigned total_px, HW, Nb;
    int C, nblk, U, V, blocked;
    unsigned units;                   // units of a pixel (all blocks)
    unsigned bx, blocks;
};
// Units g .. g + N / 4 (of U) of block `by` of pixel P (counted over all planes) of component `comp`.
template <int N>
__device__ __forceinline__ void store_units(const StageJob32& p, unsigned P, unsigned comp, unsigned by, unsigned g, unsigned U, const float (&f)[N]) {
    size_t unit;
    if (p.blocked) unit = ((size_t)P + (size_t)(comp * (unsigned)(p.nblk - 1) + by) * p.Nb * p.HW) * U + g;
    else unit = (size_t)P * p.units + by * U + g;
    store_split(f, p.hi + 4 * unit, p.lo + 4 * unit);
}
template <int V, int U>
__device__ __forceinline__ void stage_compact_f32(const StageJob32& p, unsigned block, float4* tile /*[STAGE_UNITS]*/) {
    constexpr int TPX = STAGE_UNITS / U;
    const unsigned by = block / p.bx, px0 = (block - by * p.bx) * TPX, HW = p.HW;
    const int c0 = by * 4 * U;
#pragma unroll
    for (int it = 0; it < STAGE_UNITS / V / STAGE_THREADS; ++it) {
        const int item = threadIdx.x + it * STAGE_THREADS, l = item % (TPX / V), g = item / (TPX / V);
        const unsigned P = px0 + l * V, plane = P / HW;
        const float* src = p.x + ((size_t)plane * p.C + c0 + 4 * g) * HW + (P - plane * HW);
        float raw[4][V];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const bool ok = P < p.total_px && c0 + 4 * g + e < p.C;
            const float* q = src + (size_t)e * HW;
            if (V == 4) { const float4 f = ld_chained(reinterpret_cast<const float4*>(q), ok); raw[e][0] = f.x; raw[e][V > 1 ? 1 : 0] = f.y; raw[e][V > 2 ? 2 : 0] = f.z; raw[e][V > 3 ? 3 : 0] = f.w; }
            else if (V == 2) { const float2 f = ld_chained(reinterpret_cast<const float2*>(q), ok); raw[e][0] = f.x; raw[e][V > 1 ? 1 : 0] = f.y; }
            else raw[e][0] = ld_chained(q, ok);
        }
#pragma unroll
        for (int j = 0; j < V; ++j) tile[stage_unit<V, U>(l * V + j, g)] = make_float4(raw[0][j], raw[1][j], raw[2][j], raw[3][j]);
    }
    __syncthreads();
    // (two units, eight channels, per step: whole sectors of either part)
#pragma unroll
    for (int it = 0; it < STAGE_UNITS / 2 / STAGE_THREADS; ++it) {
        const int i = threadIdx.x + it * STAGE_THREADS, px = i / (U / 2), g = i % (U / 2) * 2;
        const unsigned P = px0 + px;
        if (P >= p.total_px || by * U + g >= p.units) continue;
        // (half of each eight lanes read their second unit first: eight units of different banks)
        const bool late = (threadIdx.x & 4) != 0;
        const float4 a = tile[stage_unit<V, U>(px, g + late)], b = tile[stage_unit<V, U>(px, g + !late)];
        const float f[8] = {late ? b.x : a.x, late ? b.y : a.y, late ? b.z : a.z, late ? b.w : a.w, late ? a.x : b.x, late ? a.y : b.y, late ? a.z : b.z, late ? a.w : b.w};
        store_units(p, P, P / HW / p.Nb, by, g, U, f);
    }
}
template <int U>
__device__ __forceinline__ void stage_compact_f32(const StageJob32& p, unsigned block, float4* tile) {
    if (p.V == 4) stage_compact_f32<4, U>(p, block, tile);
    else if (p.V == 2) stage_compact_f32<2, U>(p, block, tile);
    else stage_compact_f32<1, U>(p, block, tile);
}
// The same copy for planes of fewer than 16 pixels (dense layers are 1 x 1 images), where consecutive pixels of a channel are few: one
// thread per pixel and 4 channels, consecutive threads along the pixels of a plane and then its channel groups.
__device__ __forceinline__ void stage_tiny_f32(const StageJob32& p, unsigned block) {
    const unsigned groups = p.units, HW = p.HW;
    const size_t total = (size_t)p.total_px * groups;
    for (size_t i = (size_t)block * STAGE_THREADS + threadIdx.x; i < total; i += (size_t)p.blocks * STAGE_THREADS) {
        const unsigned px = (unsigned)(i % HW), grp = (unsigned)(i / HW % groups), plane = (unsigned)(i / HW / groups);
        const float* src = p.x + ((size_t)plane * p.C + 4 * grp) * HW + px;
        float f[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) f[e] = ld_chained(src + (size_t)e * HW, (int)(4 * grp) + e < p.C);
        const unsigned b = grp / p.U;
        store_units(p, plane * HW + px, plane / p.Nb, b, grp - b * p.U, p.U, f);
    }
}
struct FilterJob32 {
    const float* w;
    float *hi, *lo;
    int Co, Ci, taps, Mp, Kp, Cp, transposed, w_io, nc, ga;
    unsigned long long neg;
};
// Forward:       Wexp[tap][m = d*Co + co][k = l*Cp + ci]  = s(l,d) * w[l^d](co, ci, tap)
// Backward-data: Wexp[tap][m = l*Ci + ci][k = d*Cop + co] = s(l,d) * w[l^d](co, ci, taps-1-tap)
// w_io: the filters are stored [r][ci][co] (dense input-major layout, one tap).
// Threads per row: short rows share a CTA (8 -> 275 channels, 6 x 7, batch 16, 5 x 5, forward 43 us, 62 with a CTA per row).
__host__ __device__ __forceinline__ int pack_threads_f32(int Kp) { return Kp > 128 ? 256 : (Kp > 64 ? 128 : 64); }
__device__ __forceinline__ void pack_filters_f32(const FilterJob32& p, unsigned block, unsigned blocks) {
    // one row (tap, m) of the expanded matrix per `wx` threads; the row is decoded once and its threads walk k
    const float* w = p.w;
    float* __restrict__ hi = p.hi;
    float* __restrict__ lo = p.lo;
    const int Co = p.Co, Ci = p.Ci, taps = p.taps, Mp = p.Mp, Kp = p.Kp, Cp = p.Cp, transposed = p.transposed, w_io = p.w_io, nc = p.nc, ga = p.ga;
    const unsigned long long neg = p.neg;
    const int Cm = transposed ? Ci : Co, Ck = transposed ? Co : Ci;
    const int rows = taps * Mp;
    const int wx = pack_threads_f32(Kp), tx = threadIdx.x % wx, per = STAGE_THREADS / wx;
    for (int row = block * per + threadIdx.x / wx; row < rows; row += blocks * per) {
        const int tap = row / Mp, m = row - tap * Mp;
        const int cm_comp = m / Cm, cm = m - cm_comp * Cm;
        const int src_tap = transposed ? taps - 1 - tap : tap;
        float* hrow = hi + (size_t)row * Kp;
        float* lrow = lo + (size_t)row * Kp;
        for (int k = tx; k < Kp; k += wx) {
            const int ck_comp = k / Cp, ck = k - ck_comp * Cp;
            float v = 0.f;
            if (cm_comp < nc && ck_comp < nc && ck < Ck) {
                const int d = transposed ? ck_comp : cm_comp, l = transposed ? cm_comp : ck_comp;
                const int co = transposed ? ck : cm, ci = transposed ? cm : ck;
                const int r = alg_pair(ga, l, d);
                const size_t src = w_io ? ((size_t)r * Ci + ci) * Co + co : ((size_t)(r * Co + co) * Ci + ci) * taps + src_tap;
                v = ld_chained(w + src);
                if (alg_negative(neg, l, d)) v = -v;
            }
            float h, l32;
            split_f32(v, h, l32);
            hrow[k] = h;
            lrow[k] = l32;
        }
    }
}

struct Prologue32 {
    int* status = nullptr;
    FilterJob32 filter;
    StageJob32 stage[2];
    float4* zero = nullptr;
    unsigned zero_units = 0, filter_blocks = 0, stage_blocks[2] = {0, 0}, zero_blocks = 0;
    int n_stages = 0;
};
__device__ __forceinline__ void zero_f32(const Prologue32& p, unsigned block) {
    for (unsigned i = block * STAGE_THREADS + threadIdx.x; i < p.zero_units; i += p.zero_blocks * STAGE_THREADS) p.zero[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}
__global__ void __launch_bounds__(STAGE_THREADS) prologue_f32_kernel(const __grid_constant__ Prologue32 p) {
    __shared__ float4 tile[STAGE_UNITS];
    unsigned block = blockIdx.x;
    chain_wait();
    chain_next();
    if (block == 0 && threadIdx.x == 0 && p.status) *p.status = 0;
    if (block < p.filter_blocks) { pack_filters_f32(p.filter, block, p.filter_blocks); return; }
    block -= p.filter_blocks;
    if (block < p.zero_blocks) { zero_f32(p, block); return; }
    block -= p.zero_blocks;
    const bool second = block >= p.stage_blocks[0];
    const StageJob32& job = second ? p.stage[1] : p.stage[0];
    if (second) block -= p.stage_blocks[0];
    if (job.V == 0) stage_tiny_f32(job, block);
    else if (job.U == 16) stage_compact_f32<16>(job, block, tile);
    else if (job.U == 8) stage_compact_f32<8>(job, block, tile);
    else stage_compact_f32<4>(job, block, tile);
}
// Without the copies: fewer registers and no shared memory, eight CTAs per SM instead of five.
__global__ void __launch_bounds__(STAGE_THREADS) filter_prologue_f32_kernel(const __grid_constant__ Prologue32 p) {
    const unsigned block = blockIdx.x;
    chain_wait();
    chain_next();
    if (block == 0 && threadIdx.x == 0 && p.status) *p.status = 0;
    if (block < p.filter_blocks) pack_filters_f32(p.filter, block, p.filter_blocks);
    else zero_f32(p, block - p.filter_blocks);
}
// 16-byte aligned, a multiple of 16 bytes; false otherwise (the caller clears it).
bool add_zero_job(Prologue32& pro, void* p, size_t bytes) {
    if ((bytes | reinterpret_cast<uintptr_t>(p)) % 16 != 0 || bytes / 16 > 0x7fffffffull) return false;
    pro.zero = static_cast<float4*>(p);
    pro.zero_units = (unsigned)(bytes / 16);
    pro.zero_blocks = grid_cap(pro.zero_units, 4 * STAGE_THREADS, 4);
    return true;
}
// `chain`: whether the main kernel may be chained to this launch.
int launch_prologue(Prologue32& pro, StatusClear* sc, cudaStream_t stream, bool* chain) {
    unsigned blocks = pro.filter_blocks + pro.zero_blocks + pro.stage_blocks[0] + pro.stage_blocks[1];
    *chain = chain_behind(blocks, 8);
    if (blocks == 0) return PCB_OK;
    if (sc && sc->pending) { pro.status = sc->word; sc->pending = false; }
    // A large filter matrix that is gathered across its storage order (backward-data of OIHW filters, forward of input-major ones or of many
    // taps), one sector per element, is bound by the loads in flight, and by rows that lie side by side being packed at the same time, when they share
    // what they fetch. It is packed by a launch of its own, which is not chained: CTAs that start on a few SMs beside the tail of the kernel
    // in front fall out of step with the rest. Backward-data, one chained launch / this: 7 x 7, batch 4, 512 channels (302 MB)
    // 551 / 306 us; 14 x 14, batch 4, 256 channels (75 MB) 180 / 154; batch 8, 128 channels (19 MB) 68 / 72; dense 1024 x 2048 x 2048
    // forward (537 MB) 1206 / 1036.
    const FilterJob32& f = pro.filter;
    const bool gathers = f.transposed != f.w_io || f.taps >= 16;        // (elements 64 and more bytes apart)
    if (pro.filter_blocks > 0 && gathers && (size_t)f.taps * f.Mp * f.Kp * 8 > (size_t)64 << 20) {
        PCB_CUDA_TRY(launch_chained_if(false, filter_prologue_f32_kernel, pro.filter_blocks + pro.zero_blocks, STAGE_THREADS, 0, stream, pro));
        blocks -= pro.filter_blocks + pro.zero_blocks;
        if (blocks == 0) return PCB_OK;
        pro.status = nullptr;
        pro.filter_blocks = pro.zero_blocks = 0;
    }
    PCB_CUDA_TRY(launch_chained(prologue_f32_kernel, blocks, STAGE_THREADS, 0, stream, pro));
    PCB_CUDA_TRY(cudaGetLastError());
    return PCB_OK;
}

// A job of the prologue launch for unpadded copies, a kernel of its own otherwise (zero-inserted gradients). As kernels of their own in
// front of the prologue, with the filters packed behind them, the copies of planes of a few pixels cost a dense layer 1024 -> 1024 at
// batch 3000 728 us forward and 552 us for the filter gradient instead of 709 and 508.
void stage_activations_f32(Prologue32& pro, const float* x, float* hi, float* lo, int planes, int C, int H, int W, int Hp, int Wp, int Cp, int pad_top,
                           int pad_left, int ins_h, int ins_w, int cb, int Nb, cudaStream_t stream) {
    if (Hp == H && Wp == W && pad_top == 0 && pad_left == 0 && ins_h == 1 && ins_w == 1) {
        const int block = cb > 0 ? cb : (Cp > 32 ? 64 : (Cp > 16 ? 32 : 16));       // (cb is 0 or 32, and then Cp a multiple of 32)
        const uintptr_t at = reinterpret_cast<uintptr_t>(x);
        StageJob32& j = pro.stage[pro.n_stages];
        j.x = x; j.hi = hi; j.lo = lo; j.total_px = (unsigned)planes * H * W; j.HW = H * W; j.Nb = Nb;
        j.C = C; j.U = block / 4; j.nblk = (Cp + block - 1) / block; j.units = Cp / 4; j.blocked = cb > 0;
        j.V = H * W < 16 ? 0 : (j.HW % 4 == 0 && at % 16 == 0 ? 4 : (j.HW % 2 == 0 && at % 8 == 0 ? 2 : 1));
        j.bx = (j.total_px + STAGE_UNITS / j.U - 1) / (STAGE_UNITS / j.U);
        j.blocks = j.V ? j.bx * j.nblk : (unsigned)grid_cap((size_t)j.total_px * (Cp / 4), STAGE_THREADS, 16);
        pro.stage_blocks[pro.n_stages++] = j.blocks;
    } else if (Hp * Wp < 32) {
        pack_activations_f32_small_kernel<<<grid_cap((size_t)planes * Hp * Wp * (Cp / 4), 256, 16), 256, 0, stream>>>(
            x, hi, lo, planes, C, H, W, Hp, Wp, Cp, pad_top, pad_left, ins_h, ins_w, cb, Nb);
    } else {
        const size_t tiles = (size_t)planes * ((Hp * Wp + 31) / 32);
        pack_activations_f32_kernel<<<grid_cap(tiles, 1, 16), 256, 0, stream>>>(x, hi, lo, planes, C, H, W, Hp, Wp, Cp, pad_top, pad_left, ins_h,
                                                                                 ins_w, cb, Nb);
    }
}

// ---- backward-filter ------------------------------------------------------------------------------------
// Both staged tensors MN-major (K = pixels, 16 per stage), M = (d, co), N = (l, ci); per K step of 8 pixels three
// TF32 MMAs; the epilogue folds G[(d,co),(l,ci)] through the quaternion table into fp32 scratch [tap][r][co][ci].
// 32-bit MN-major operands exist in one shared-memory layout only: 128-byte rows (32 channels) swizzled in 32-byte
// units over groups of 4 rows (descriptor layout type 1, TMA swizzle 128B_ATOM_32B), so channels are padded to 32.
constexpr int TFK = 16;
constexpr int TF_CHUNK = 8;                                 // stages of a chunk: 48 MMAs of the three products
constexpr uint32_t TF_STAGE = 2 * (TM + TN) * TFK * 4;      // 48 KB
constexpr int TFP_STAGES = 6;                               // pairs of SMs: half of the N columns in each CTA, 32 KB
constexpr uint32_t TFP_STAGE = 2 * (TM + TN / 2) * TFK * 4;
struct TFParams {
    int Nb, Co, Ci, HO, WO, Cop, Cip, cbA, cbB;             // channel-block width in fp32 elements: 32
    int KH, KW, SH, SW, DH, DW, PW, PH, PN, tiles_w, tiles_h, tiles_n;
    int m_tiles, n_tiles, n_tile_cols, splits, steps_per_split;
    int off_w, off_h;             // added to the pixel coordinates of every x box: minus the padding (out-of-range coordinates read zeros)
    int nc, ga;                                              // algebra: components, GA(3,0,0) component order
    unsigned long long neg;                                  // negative entries of the block, bit (8*l + d)
};

// leading offset = distance between 32-channel blocks, stride offset = distance between groups of 4 pixel rows
__device__ __forceinline__ uint64_t desc_mn_f32(uint32_t addr, int cb, uint32_t block_bytes) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((block_bytes >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)(((4u * cb * 4u) >> 4) & 0x3FFFu) << 32) | DESC_VERSION_SM100 | (1ull << 61);
}

// PAIR: as in conv_tc.cu, a cluster of two CTAs takes 256 rows and half of the N columns each: 32 instead of 48 KB per SM and stage. (Forward + backward of
// the layers above within the spread of the same with single SMs: the MMAs bound both.)
template <bool PAIR>
__global__ void __launch_bounds__(T_THREADS, 1)
qconv_filter_tf32_kernel(const __grid_constant__ CUtensorMap map_dy_hi, const __grid_constant__ CUtensorMap map_dy_lo,
                         const __grid_constant__ CUtensorMap map_x_hi, const __grid_constant__ CUtensorMap map_x_lo, TFParams p,
                         float* __restrict__ dw32, int* __restrict__ status) {
    constexpr int STAGES = PAIR ? TFP_STAGES : T_STAGES;
    constexpr uint32_t STAGE = PAIR ? TFP_STAGE : TF_STAGE;
    extern __shared__ uint8_t smem_raw[];
    const int rank = PAIR ? (int)cluster_ctarank() : 0;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + STAGES * STAGE);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
    const uint32_t tiles_addr = smem_u32(base);
    const uint32_t full_bar = smem_u32(bars), empty_bar = smem_u32(bars + STAGES);
    const uint32_t tmem_full = smem_u32(bars + 2 * STAGES), tmem_empty = smem_u32(bars + 2 * STAGES + 2);

    const int m_tiles = PAIR ? p.m_tiles / 2 : p.m_tiles, id = PAIR ? blockIdx.x / 2 : blockIdx.x;
    const int n_items = m_tiles * p.n_tiles * p.KH * p.KW;
    int item = id % n_items;
    const int split = id / n_items;
    const int mt = PAIR ? 2 * (item % m_tiles) + rank : item % m_tiles; item /= m_tiles;
    const int nt = item % p.n_tiles;
    const int tap = item / p.n_tiles;
    const int kh = tap / p.KW, kw = tap - kh * p.KW;
    const int steps_total = p.tiles_w * p.tiles_h * p.tiles_n;
    const int step_beg = split * p.steps_per_split;
    const int n_steps = max(0, min(steps_total, step_beg + p.steps_per_split) - step_beg);
    const int n_chunks = (n_steps + TF_CHUNK - 1) / TF_CHUNK;       // chunks alternate between the two TMEM buffers

    const int nblkA = TM / p.cbA, nblkB = p.n_tile_cols / p.cbB / (PAIR ? 2 : 1);      // blocks of this CTA's shared memory
    const int bpcA = p.Cop / p.cbA, bpcB = p.Cip / p.cbB;
    const uint32_t blkA_bytes = TFK * p.cbA * 4, blkB_bytes = TFK * p.cbB * 4;
    const uint32_t a_bytes = nblkA * blkA_bytes, b_bytes = nblkB * blkB_bytes;
    const uint32_t A_REGION = TM * TFK * 4, B_REGION = (PAIR ? TN / 2 : TN) * TFK * 4;      // 8 KB, 16 (8) KB
    const int blockA0 = mt * nblkA, blockB0 = nt * (TN / p.cbB);

    if (t == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar + 8 * s, 1); mbar_init(empty_bar + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(tmem_full + 8 * b, 1); mbar_init(tmem_empty + 8 * b, PAIR ? 16 : 8); }
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
        {
            const bool el = elect_one();
            // one copy per operand half and stage (the staged tensors keep the channel-block index outermost, so the blocks
            // of a tile are one box even across components) and a running (tw, th, tn) of the pixel box: no division in
            // this loop -- a division per copy used to bound the kernel
            int tw = step_beg % p.tiles_w, th = (step_beg / p.tiles_w) % p.tiles_h, tn = step_beg / (p.tiles_w * p.tiles_h);
            int s = 0, phase = 1;
            bool ok = true;
            for (int it = 0; it < n_steps && ok; ++it) {
                ok = warp_wait_bounded(empty_bar + 8 * s, phase, status, ST_T_PRODUCER);
                if (!ok) break;
                const int ow0 = tw * p.PW, oh0 = th * p.PH, n0 = tn * p.PN;
                const uint32_t a_hi = tiles_addr + s * STAGE, a_lo = a_hi + A_REGION, b_hi = a_hi + 2 * A_REGION, b_lo = b_hi + B_REGION;
                const uint32_t bar = full_bar + 8 * s;
                if (++tw == p.tiles_w) { tw = 0; if (++th == p.tiles_h) { th = 0; ++tn; } }
                if (++s == STAGES) { s = 0; phase ^= 1; }
                const int wp0 = ow0 * p.SW + kw * p.DW + p.off_w, hp0 = oh0 * p.SH + kh * p.DH + p.off_h;
                if (el && PAIR) {
                    const uint32_t lead = map_to_cta(bar, 0);
                    if (rank == 0) mbar_arrive_expect_tx(bar, 4 * (a_bytes + b_bytes));
                    tma_load_5d_pair(a_hi, &map_dy_hi, 0, ow0, oh0, n0, blockA0, lead);
                    tma_load_5d_pair(a_lo, &map_dy_lo, 0, ow0, oh0, n0, blockA0, lead);
                    tma_load_5d_pair(b_hi, &map_x_hi, 0, wp0, hp0, n0, blockB0 + rank * nblkB, lead);
                    tma_load_5d_pair(b_lo, &map_x_lo, 0, wp0, hp0, n0, blockB0 + rank * nblkB, lead);
                } else if (el) {
                    mbar_arrive_expect_tx(bar, 2 * (a_bytes + b_bytes));
                    tma_load_5d(a_hi, &map_dy_hi, 0, ow0, oh0, n0, blockA0, bar);
                    tma_load_5d(a_lo, &map_dy_lo, 0, ow0, oh0, n0, blockA0, bar);
                    tma_load_5d(b_hi, &map_x_hi, 0, wp0, hp0, n0, blockB0, bar);
                    tma_load_5d(b_lo, &map_x_lo, 0, wp0, hp0, n0, blockB0, bar);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (rank == 0) {
            constexpr int M = PAIR ? 2 * TM : TM;
            const uint32_t idesc = make_idesc_f16(2, M, p.n_tile_cols, true, true);
            const uint32_t peer_empty = PAIR ? map_to_cta(empty_bar, 1) : 0u, peer_full = PAIR ? map_to_cta(tmem_full, 1) : 0u;
            const bool el = elect_one();
            bool ok = true;
            int s = 0, phase = 0;
            for (int c = 0; c < n_chunks && ok; ++c) {
                const int buf = c & 1, use = c >> 1;
                if (use > 0) {
                    ok = warp_wait_bounded(tmem_empty + 8 * buf, (use - 1) & 1, status, ST_T_MMA);
                    if (!ok) break;
                    tc_fence_after_sync();
                }
                const int k_beg = c * TF_CHUNK, k_end = min(n_steps, k_beg + TF_CHUNK);
                const uint32_t d = tmem_base + buf * TN;
                for (int it = k_beg; it < k_end; ++it) {
                    ok = warp_wait_bounded(full_bar + 8 * s, phase, status, ST_T_MMA);
                    if (!ok) break;
                    tc_fence_after_sync();
                    if (el) {
                        const uint32_t a_hi = tiles_addr + s * STAGE, a_lo = a_hi + A_REGION, b_hi = a_hi + 2 * A_REGION, b_lo = b_hi + B_REGION;
                        auto mma = [&](uint64_t ad, uint64_t bd, uint32_t acc) {
                            if (PAIR) mma_tf32_pair(d, (uint32_t)ad, (uint32_t)(ad >> 32), (uint32_t)bd, (uint32_t)(bd >> 32), idesc, acc);
                            else mma_tf32_ss(d, ad, bd, idesc, acc);
                        };
#pragma unroll
                        for (int j = 0; j < TFK / 8; ++j) {                   // 8 pixels (K rows) per MMA
                            const uint32_t ao = j * 8 * p.cbA * 4, bo = j * 8 * p.cbB * 4;
                            const uint64_t ah = desc_mn_f32(a_hi + ao, p.cbA, blkA_bytes), bh = desc_mn_f32(b_hi + bo, p.cbB, blkB_bytes);
                            mma(desc_mn_f32(a_lo + ao, p.cbA, blkA_bytes), bh, (it > k_beg || j > 0) ? 1u : 0u);
                            mma(ah, desc_mn_f32(b_lo + bo, p.cbB, blkB_bytes), 1u);
                            mma(ah, bh, 1u);
                        }
                        if (PAIR) {
                            mma_commit_pair(empty_bar + 8 * s);
                            mma_commit_pair(peer_empty + 8 * s);
                            if (it == k_end - 1) { mma_commit_pair(tmem_full + 8 * buf); mma_commit_pair(peer_full + 8 * buf); }
                        } else {
                            mma_commit(empty_bar + 8 * s);
                            if (it == k_end - 1) mma_commit(tmem_full + 8 * buf);
                        }
                    }
                    if (++s == STAGES) { s = 0; phase ^= 1; }
                }
            }
        }
        __syncwarp();
    } else {
        const int q = warp & 3, chalf = (warp - 2) >> 2;
        uint32_t part[4][32];                                        // this thread's 128 columns, summed over the chunks so far
#pragma unroll
        for (int cb = 0; cb < 4; ++cb)
#pragma unroll
            for (int e = 0; e < 32; ++e) part[cb][e] = 0u;
        bool ok = true;
        for (int c = 0; c < n_chunks && ok; ++c) {
            const int buf = c & 1, use = c >> 1;
            const int seen = read_status(status);
            ok = mbar_wait_bounded(tmem_full + 8 * buf, use & 1, status, ST_T_EPILOGUE);
            ok = warp_may_store(ok, seen);
            if (!ok) break;
            tc_fence_after_sync();
#pragma unroll
            for (int cb = 0; cb < 4; ++cb) {
                if (chalf * 128 + cb * 32 < p.n_tile_cols) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {                         // (16 columns at a time: with 32 the kernel spills)
                        uint32_t v[16];
                        tmem_ld_32x32b_x16(tmem_base + ((uint32_t)(q * 32) << 16) + buf * TN + chalf * 128 + cb * 32 + 16 * h, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 16; ++e) part[cb][16 * h + e] = __float_as_uint(__uint_as_float(part[cb][16 * h + e]) + __uint_as_float(v[e]));
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) { if (PAIR) mbar_arrive_cluster(map_to_cta(tmem_empty + 8 * buf, 0)); else mbar_arrive(tmem_empty + 8 * buf); }
        }
        if (ok && n_steps > 0) {
            const int row = q * 32 + lane;
            const int blk = blockA0 + row / p.cbA;
            const int d = blk / bpcA, co = (blk % bpcA) * p.cbA + row % p.cbA;
            const bool row_ok = d < p.nc && co < p.Co;
            const bool any_row = __any_sync(0xffffffffu, row_ok);
            const size_t comp_stride = (size_t)p.Co * p.Ci;
            const uint32_t rbuf = tiles_addr + (uint32_t)(warp - 2) * ADD_ROWS_BYTES<32>;      // the operand ring: all MMAs have read it
            float* tap_base = dw32 + (size_t)tap * p.nc * comp_stride;
#pragma unroll
            for (int cb = 0; cb < 4; ++cb) {
                const int col0 = chalf * 128 + cb * 32;
                if (col0 >= p.n_tile_cols || !any_row) break;
                auto add = [&](auto quads) {
                    constexpr bool Q = decltype(quads)::value;
                    const int col = col0 + add_rows_column<32, Q>(lane), nblk = blockB0 + col / p.cbB;      // (l, ci) of this lane's columns
                    const int l = nblk / bpcB, ci = (nblk % bpcB) * p.cbB + col % p.cbB;
                    const bool col_ok = col < p.n_tile_cols && l < p.nc && ci < p.Ci;
                    add_rows<32, Q>(rbuf, part[cb], lane, [&](int r, float& sgn) -> float* {
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

// scratch [tap][r][co][ci] -> dw [r][co][ci][tap], or [r][ci][co] for dense layers (input-major, one tap)
__global__ void unpack_filter_grad_f32_kernel(const float* src, float* __restrict__ dw, int taps, int Co, int Ci, int dw_io, int nc) {
    const size_t per_tap = (size_t)nc * Co * Ci, total = per_tap * taps;
    chain_wait();
    chain_next();
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        if (dw_io) {
            const int co = (int)(idx % Co);
            const int ci = (int)((idx / Co) % Ci);
            const int r = (int)(idx / ((size_t)Co * Ci));
            dw[idx] = ld_chained(src + ((size_t)r * Co + co) * Ci + ci);
        } else {
            const int tap = (int)(idx % taps);
            dw[idx] = ld_chained(src + (size_t)tap * per_tap + idx / taps);
        }
    }
}

struct Plan32 {
    int Cin, Cout, Hin, Win, Hout, Wout, pad_top, pad_left, SH, SW, ins_h, ins_w, Cp, Hp, Wp, Mp, Kp, LK;
    size_t xp_bytes, w_bytes;      // one of (hi, lo)
};

Plan32 make_plan32(Pass pass, const Geom& g, bool tight) {
    Plan32 pl;
    if (pass == PASS_FWD) {
        pl.Cin = g.Ci; pl.Cout = g.Co; pl.Hin = g.H; pl.Win = g.W; pl.Hout = g.HO; pl.Wout = g.WO;
        pl.pad_top = g.PT; pl.pad_left = g.PL; pl.SH = g.SH; pl.SW = g.SW; pl.ins_h = pl.ins_w = 1;
    } else {
        pl.Cin = g.Co; pl.Cout = g.Ci; pl.Hin = g.HO; pl.Win = g.WO; pl.Hout = g.H; pl.Wout = g.W;
        pl.pad_top = (g.KH - 1) * g.DH - g.PT; pl.pad_left = (g.KW - 1) * g.DW - g.PL; pl.SH = 1; pl.SW = 1;
        pl.ins_h = g.SH; pl.ins_w = g.SW;
    }
    pl.LK = (pass == PASS_FWD && g.real_in) ? 1 : g.nc;
    pl.Cp = round_up(pl.Cin, 16);
    pl.Hp = (pl.Hout - 1) * pl.SH + (g.KH - 1) * g.DH + 1;
    pl.Wp = (pl.Wout - 1) * pl.SW + (g.KW - 1) * g.DW + 1;
    if (pl.ins_h == 1 && pl.ins_w == 1) {                              // the copy is not padded: the tensor map's zero fill is the padding
        pl.Hp = tight ? reached(pl.Hin, pl.Hout, pl.SH, g.KH, g.DH, pl.pad_top) : pl.Hin;
        pl.Wp = tight ? reached(pl.Win, pl.Wout, pl.SW, g.KW, g.DW, pl.pad_left) : pl.Win;
    }
    pl.Mp = round_up(g.nc * pl.Cout, TM);
    pl.Kp = pl.LK * pl.Cp;
    pl.xp_bytes = ((size_t)pl.LK * g.Nb * pl.Hp * pl.Wp * pl.Cp * 4 + 1023) / 1024 * 1024;
    pl.w_bytes = ((size_t)g.KH * g.KW * pl.Mp * pl.Kp * 4 + 1023) / 1024 * 1024;
    return pl;
}

constexpr size_t MAX_COPIES = (size_t)16 << 30;               // hi and lo
Plan32 make_plan32(Pass pass, const Geom& g) {
    const Plan32 pl = make_plan32(pass, g, g.tight != 0);
    return 2 * pl.xp_bytes <= MAX_COPIES ? pl : make_plan32(pass, g, true);
}

struct FilterPlan32 {
    int Cop, Cip;
    int H, W;                      // extents of the copy of x
    size_t xp_bytes, dyp_bytes, acc_bytes;
};

FilterPlan32 make_filter_plan32(const Geom& g, bool tight) {
    FilterPlan32 f;
    f.H = tight ? reached(g.H, g.HO, g.SH, g.KH, g.DH, g.PT) : g.H;
    f.W = tight ? reached(g.W, g.WO, g.SW, g.KW, g.DW, g.PL) : g.W;
    f.Cop = round_up(g.Co, 32);
    f.Cip = round_up(g.Ci, 32);
    f.xp_bytes = ((size_t)g.nc * g.Nb * f.H * f.W * f.Cip * 4 + 1023) / 1024 * 1024;
    f.dyp_bytes = ((size_t)g.nc * g.Nb * g.HO * g.WO * f.Cop * 4 + 1023) / 1024 * 1024;
    f.acc_bytes = ((size_t)g.nc * g.Co * g.Ci * g.KH * g.KW * 4 + 1023) / 1024 * 1024;
    return f;
}

FilterPlan32 make_filter_plan32(const Geom& g) {
    const FilterPlan32 f = make_filter_plan32(g, g.tight != 0);
    return 2 * (f.xp_bytes + f.dyp_bytes) <= MAX_COPIES ? f : make_filter_plan32(g, true);
}

// Extents of the padded image, which the tensor-map coordinates span.
bool extents_ok(const Geom& g, int Hout, int Wout, int SH, int SW) {
    return (long long)(Hout - 1) * SH + (long long)(g.KH - 1) * g.DH <= 65534 && (long long)(Wout - 1) * SW + (long long)(g.KW - 1) * g.DW <= 65534;
}

bool common_ok(int dtype, int variant, const Geom& g) {
    if (dtype != PCB_F32 || variant != PCB_VARIANT_16_PRODUCT) return false;
    if (g.SH > 2 || g.SW > 2) return false;
    if (g.w_io && g.KH * g.KW != 1) return false;
    return true;
}

}  // namespace

bool conv_tf32_supported(Pass pass, int dtype, int variant, const Geom& g) {
    if (!common_ok(dtype, variant, g)) return false;
    if (pass == PASS_BWD_FILTER) {
        if (g.real_in) return false;
        const FilterPlan32 f = make_filter_plan32(g);
        return extents_ok(g, g.HO, g.WO, g.SH, g.SW) && 2 * (f.xp_bytes + f.dyp_bytes) <= MAX_COPIES;
    }
    if (g.real_in && pass != PASS_FWD) return false;
    if (pass == PASS_BWD_DATA && ((g.KH - 1) * g.DH < g.PT || (g.KW - 1) * g.DW < g.PL)) return false;
    const Plan32 pl = make_plan32(pass, g);
    return extents_ok(g, pl.Hout, pl.Wout, pl.SH, pl.SW) && 2 * pl.xp_bytes <= MAX_COPIES;
}

size_t conv_tf32_scratch_bytes(Pass pass, const Geom& g) {
    if (pass == PASS_BWD_FILTER) {
        const FilterPlan32 f = make_filter_plan32(g);
        return 2 * (f.xp_bytes + f.dyp_bytes) + f.acc_bytes;
    }
    const Plan32 pl = make_plan32(pass, g);
    return 2 * (pl.xp_bytes + pl.w_bytes);
}

static int conv_tf32_filter_launch(const Geom& layer, const float* dy, const float* x, float* dw, void* scratch, int* status, cudaStream_t stream, StatusClear* sc) {
    const Geom g = flat_pixels(layer);
    const FilterPlan32 f = make_filter_plan32(g);
    const int taps = g.KH * g.KW;
    uint8_t* s8 = static_cast<uint8_t*>(scratch);
    float* x_hi = reinterpret_cast<float*>(s8);
    float* x_lo = reinterpret_cast<float*>(s8 + f.xp_bytes);
    float* y_hi = reinterpret_cast<float*>(s8 + 2 * f.xp_bytes);
    float* y_lo = reinterpret_cast<float*>(s8 + 2 * f.xp_bytes + f.dyp_bytes);
    float* acc = reinterpret_cast<float*>(s8 + 2 * f.xp_bytes + 2 * f.dyp_bytes);
    bool chain = false;
    Prologue32 pro;
    stage_activations_f32(pro, x, x_hi, x_lo, g.nc * g.Nb, g.Ci, g.H, g.W, f.H, f.W, f.Cip, 0, 0, 1, 1, 32, g.Nb, stream);
    stage_activations_f32(pro, dy, y_hi, y_lo, g.nc * g.Nb, g.Co, g.HO, g.WO, g.HO, g.WO, f.Cop, 0, 0, 1, 1, 32, g.Nb, stream);
    PCB_CUDA_TRY(cudaGetLastError());
    add_zero_job(pro, acc, f.acc_bytes);                             // (rounded up to 1 KB: always whole units)
    {
        const int rc = launch_prologue(pro, sc, stream, &chain);
        if (rc != PCB_OK) return rc;
    }

    TFParams p;
    p.nc = g.nc; p.ga = g.ga; p.neg = g.neg;
    p.Nb = g.Nb; p.Co = g.Co; p.Ci = g.Ci; p.HO = g.HO; p.WO = g.WO; p.Cop = f.Cop; p.Cip = f.Cip;
    p.cbA = 32; p.cbB = 32;
    p.KH = g.KH; p.KW = g.KW; p.SH = g.SH; p.SW = g.SW; p.DH = g.DH; p.DW = g.DW;
    p.off_w = -g.PL; p.off_h = -g.PT;
    {
        long long best = -1;
        for (int pw = 1; pw <= TFK; pw *= 2)
            for (int ph = 1; ph * pw <= TFK; ph *= 2) {
                const int pn = TFK / (pw * ph);
                // (boxes of less than four pixels side by side are slow to load. 3x3, 16 -> 24 channels, 101 x 101, batch 32, forward + backward: 1862 us
                // with the 1 x 1 x 16 boxes that waste nothing, 1419 with these)
                const long long vol = (long long)round_up(g.WO, pw) * round_up(g.HO, ph) * round_up(g.Nb, pn) * (pw >= 4 ? 16 : (pw == 2 ? 17 : 19));
                if (best < 0 || vol < best || (vol == best && pw > p.PW)) { best = vol; p.PW = pw; p.PH = ph; p.PN = pn; }
            }
    }
    p.tiles_w = (g.WO + p.PW - 1) / p.PW; p.tiles_h = (g.HO + p.PH - 1) / p.PH; p.tiles_n = (g.Nb + p.PN - 1) / p.PN;
    const int m_cols = g.nc * f.Cop, n_cols = g.nc * f.Cip;
    p.m_tiles = (m_cols + TM - 1) / TM;
    p.n_tiles = (n_cols + TN - 1) / TN;
    p.n_tile_cols = n_cols < TN ? n_cols : TN;
    const int steps_total = p.tiles_w * p.tiles_h * p.tiles_n;
    const bool pair = p.m_tiles % 2 == 0 && (p.n_tile_cols / p.cbB) % 2 == 0 && worth_pairs((double)taps * p.m_tiles * p.n_tiles * steps_total * 6 * p.n_tile_cols / TN);
    const int items = taps * p.m_tiles * p.n_tiles / (pair ? 2 : 1);
    const int splits = split_count(items, pair ? sm_pairs() : sm_count(), steps_total, 16);
    p.steps_per_split = (steps_total + splits - 1) / splits;
    p.splits = (steps_total + p.steps_per_split - 1) / p.steps_per_split;

    auto swz = [](int) { return CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B; };
    alignas(64) CUtensorMap m_dy_hi, m_dy_lo, m_x_hi, m_x_lo;
    {
        // staged tensors: [component * blocks per component + channel block][image][h][w][32 channels]; the last box extent
        // is the number of channel blocks of a tile (blocks past the end read as zeros)
        const cuuint64_t dims[5] = {(cuuint64_t)p.cbA, (cuuint64_t)g.WO, (cuuint64_t)g.HO, (cuuint64_t)g.Nb, (cuuint64_t)(g.nc * (f.Cop / p.cbA))};
        const cuuint64_t strides[4] = {(cuuint64_t)p.cbA * 4, (cuuint64_t)g.WO * p.cbA * 4, (cuuint64_t)g.HO * g.WO * p.cbA * 4,
                                       (cuuint64_t)g.Nb * g.HO * g.WO * p.cbA * 4};
        const cuuint32_t box[5] = {(cuuint32_t)p.cbA, (cuuint32_t)p.PW, (cuuint32_t)p.PH, (cuuint32_t)p.PN, (cuuint32_t)(TM / p.cbA)};
        int rc = make_tensor_map(&m_dy_hi, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, y_hi, 5, dims, strides, box, nullptr, swz(p.cbA), "dy hi");
        if (rc == PCB_OK) rc = make_tensor_map(&m_dy_lo, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, y_lo, 5, dims, strides, box, nullptr, swz(p.cbA), "dy lo");
        if (rc != PCB_OK) return rc;
    }
    {
        const cuuint64_t dims[5] = {(cuuint64_t)p.cbB, (cuuint64_t)f.W, (cuuint64_t)f.H, (cuuint64_t)g.Nb, (cuuint64_t)(g.nc * (f.Cip / p.cbB))};
        const cuuint64_t strides[4] = {(cuuint64_t)p.cbB * 4, (cuuint64_t)f.W * p.cbB * 4, (cuuint64_t)f.H * f.W * p.cbB * 4,
                                       (cuuint64_t)g.Nb * f.H * f.W * p.cbB * 4};
        const cuuint32_t box[5] = {(cuuint32_t)p.cbB, (cuuint32_t)((p.PW - 1) * g.SW + 1), (cuuint32_t)((p.PH - 1) * g.SH + 1), (cuuint32_t)p.PN,
                                   (cuuint32_t)(p.n_tile_cols / p.cbB / (pair ? 2 : 1))};
        const cuuint32_t es[5] = {1, (cuuint32_t)g.SW, (cuuint32_t)g.SH, 1, 1};
        int rc = make_tensor_map(&m_x_hi, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, x_hi, 5, dims, strides, box, es, swz(p.cbB), "x hi");
        if (rc == PCB_OK) rc = make_tensor_map(&m_x_lo, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, x_lo, 5, dims, strides, box, es, swz(p.cbB), "x lo");
        if (rc != PCB_OK) return rc;
    }
    constexpr size_t smem = 1024 + T_STAGES * TF_STAGE + 512;
    auto* kernel = pair ? qconv_filter_tf32_kernel<true> : qconv_filter_tf32_kernel<false>;
    PCB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PCB_CUDA_TRY(launch_clusters(pair ? 2 : 1, chain, kernel, items * p.splits * (pair ? 2 : 1), T_THREADS, smem, stream, m_dy_hi, m_dy_lo, m_x_hi, m_x_lo, p, acc, status));
    PCB_CUDA_TRY(cudaGetLastError());
    PCB_CUDA_TRY(launch_chained(unpack_filter_grad_f32_kernel, grid_cap((size_t)g.nc * g.Co * g.Ci * taps, 256, 16), 256, 0, stream, acc, dw, taps, g.Co, g.Ci, g.dw_io, g.nc));
    PCB_CUDA_TRY(cudaGetLastError());
    return PCB_OK;
}

int conv_tf32_launch(Pass pass, const Geom& layer, const void* a, const void* b, const void* bias, void* out, void* scratch, int* status,
                     cudaStream_t stream, StatusClear* sc) {
    // operand roles as for the other launchers: forward/backward-data a = filters, b = activations; backward-filter a = dy, b = x
    if (pass == PASS_BWD_FILTER) return conv_tf32_filter_launch(layer, (const float*)a, (const float*)b, (float*)out, scratch, status, stream, sc);
    const Geom g = flat_pixels(layer);
    const Plan32 pl = make_plan32(pass, g);
    const int taps = g.KH * g.KW;
    uint8_t* s8 = static_cast<uint8_t*>(scratch);
    float* x_hi = reinterpret_cast<float*>(s8);
    float* x_lo = reinterpret_cast<float*>(s8 + pl.xp_bytes);
    float* w_hi = reinterpret_cast<float*>(s8 + 2 * pl.xp_bytes);
    float* w_lo = reinterpret_cast<float*>(s8 + 2 * pl.xp_bytes + pl.w_bytes);
    const bool inserted = pl.ins_h != 1 || pl.ins_w != 1;
    bool chain = false;
    Prologue32 pro;
    stage_activations_f32(pro, (const float*)b, x_hi, x_lo, pl.LK * g.Nb, pl.Cin, pl.Hin, pl.Win, pl.Hp, pl.Wp, pl.Cp, inserted ? pl.pad_top : 0,
                          inserted ? pl.pad_left : 0, pl.ins_h, pl.ins_w, 0, 1, stream);
    PCB_CUDA_TRY(cudaGetLastError());
    pro.filter = FilterJob32{(const float*)a, w_hi, w_lo, g.Co, g.Ci, taps, pl.Mp, pl.Kp, pl.Cp, pass == PASS_BWD_DATA ? 1 : 0, g.w_io, g.nc, g.ga, g.neg};
    pro.filter_blocks = grid_cap((size_t)taps * pl.Mp, STAGE_THREADS / pack_threads_f32(pl.Kp), 8);

    TParams p;
    const int n_k = taps * pl.LK * (pl.Cp / TKS);
    p.store_vec = 1;
    while (p.store_vec < 8 && pl.Wout % (p.store_vec * 2) == 0 && (reinterpret_cast<uintptr_t>(out) % (size_t)(p.store_vec * 8)) == 0) p.store_vec *= 2;
    const bool deep = worth_pairs((double)g.Nb * pl.Hout * pl.Wout / 256 * (pl.Mp / TM) * n_k * 6);
    // Clocks of a form, from which the fastest is taken. Of a stage: 680 with tiles of 256 pixels, 610 with 128, in halo form 22 per row of up to 32 or
    // 525. Of storing 256 pixels of 128 rows: aligned rows, and rows that go through shared memory, 4, 2 or 1 pixels per lane. A tile is stored
    // beside the stages of the next one, a tile of 256 in several chunks beside two of those at most, and the chunks cost 3000 more, 8000 where rows are aligned
    // (1x1, 24 -> 16, 112 x 112, batch 20, tiles of 256 / 128 135.3 / 129.7 us; 64 -> 64, 28 x 28, batch 40 60.1 / 53.4). Constants with
    // which the choice lost 0.7 % on average over the forms of 32 forward layers, each timed in every form, us, 256 / 128 / halo of 32 / of 16: 3x3, 16
    // channels, 32 x 32, batch 8 26.1 / 18.4 / 31.7 / 23.6; 16 -> 24, 101 x 101, batch 32 296 / 315 / 349 / 342; 24 -> 40, 30 x 30, batch 60 173 / 201 / 175 / 160;
    // 64 -> 64, 56 x 56, batch 32 523 / 658 / 541 / 578; 1x1, 24 -> 16, 112 x 112, batch 10 82 / 69.
    long long epilogue = p.store_vec == 8 ? 5000 : (p.store_vec == 4 ? 15000 : (p.store_vec == 2 ? 24000 : 20000));
    if (g.nc * pl.Cout <= 64 && p.store_vec < 8) epilogue /= 3;          // (store_rows_f32_few)
    if (pl.Wout < 8) epilogue = 32000;                                   // (an element of 32 planes per store)
    auto wide_clocks = [&](long long rounds, long long stages, long long stage) {
        if (stages <= T_CHUNK) return rounds * (stages * stage > epilogue ? stages * stage : epilogue) + epilogue;
        const long long hidden = (stages < 2 * T_CHUNK ? stages : 2 * T_CHUNK) * stage;
        return rounds * (stages * stage + (epilogue > hidden ? epilogue - hidden : 0) + (p.store_vec == 8 ? 8000 : 3000)) + epilogue;
    };
    auto narrow_clocks = [&](long long rounds, long long stages, long long stage) {
        return rounds * (stages * stage > epilogue / 2 ? stages * stage : epilogue / 2) + epilogue / 2;
    };
    // Box of `cols` pixels that wastes the fewest columns, and the cut of its K loop. Too few tiles for the SMs (dense layers, small
    // planes): the K loop of every tile is cut into work items of at least one chunk each; their partial sums meet in the output, zeroed
    // first, by fp32 reductions (the order of which is not fixed).
    auto plan_tiles = [&](int cols) -> long long {
        long long best = -1;
        p.n_cols = cols;
        for (int pw = 1; pw <= cols; pw *= 2)
            for (int ph = 1; ph * pw <= cols; ph *= 2) {
                const int pn = cols / (pw * ph);
                if (pn > 256 || (pw - 1) * pl.SW + 1 > 256 || (ph - 1) * pl.SH + 1 > 256) continue;
                if (pw < 8 && pl.Wout >= 8) continue;                      // narrow boxes only for narrow planes
                const long long vol = (long long)round_up(pl.Wout, pw) * round_up(pl.Hout, ph) * round_up(g.Nb, pn);
                if (best < 0 || vol < best || (vol == best && pw > p.PW)) { best = vol; p.PW = pw; p.PH = ph; p.PN = pn; }
            }
        p.tiles_w = (pl.Wout + p.PW - 1) / p.PW; p.tiles_h = (pl.Hout + p.PH - 1) / p.PH; p.tiles_n = (g.Nb + p.PN - 1) / p.PN;
        p.tiles_m = pl.Mp / TM;
        const long long tiles = (long long)p.tiles_w * p.tiles_h * p.tiles_n * p.tiles_m;
        p.splits = 1;
        if (2 * tiles <= sm_count() && n_k >= 2 * T_SPLIT) {
            p.splits = sm_count() / (int)tiles;
            if (p.splits > n_k / T_SPLIT) p.splits = n_k / T_SPLIT;
            while (n_k % p.splits != 0) --p.splits;                  // equal work items: every chunk of every item holds stages
        }
        p.k_per_split = n_k / p.splits;
        const long long rounds = (tiles * p.splits + sm_count() - 1) / sm_count();
        return cols == 256 ? wide_clocks(rounds, p.k_per_split, 680) : narrow_clocks(rounds, p.k_per_split, 610);
    };
    const long long narrow_cost = plan_tiles(128);
    long long cost = plan_tiles(256);
    if (narrow_cost < cost) { cost = narrow_cost; plan_tiles(128); }
    // Halo tiles of up to 32 rows, or of up to 16.
    bool halo = false;
    p.Wt = p.Ht = p.a_slots = 0; p.halo_bytes = 0;
    for (int cap = 32; cap >= 16 && pl.SH == 1 && pl.SW == 1 && taps >= 4 && pl.Wout >= 8; cap -= 16) {
        const int rows = (pl.Hout + cap - 1) / cap;
        const int ph = (((pl.Hout + rows - 1) / rows) + 1) & ~1;
        const bool two = pl.Mp / TM % 2 == 0 && deep;
        const int wt = 8 + (g.KW - 1) * g.DW, ht = (two ? ph / 2 : ph) + (g.KH - 1) * g.DH;
        const uint32_t part = ((uint32_t)wt * ht * TKS * 4 + 1023) / 1024 * 1024;
        const int room = 227 * 1024 - 1024 - 512 - (p.store_vec < 8 ? 8 * EPI_ROWS_F32_BYTES : 0) - (int)(T_HALO_TILES * 2 * part);
        const long long tiles = (long long)((pl.Wout + 7) / 8) * ((pl.Hout + ph - 1) / ph) * g.Nb * (pl.Mp / TM);
        const long long rounds = (tiles + sm_count() - 1) / sm_count();
        const long long halo_cost = cap == 32 ? wide_clocks(rounds, n_k, 22 * ph) : narrow_clocks(rounds, n_k, 525);
        if (ph >= cap * 3 / 4 && wt <= 256 && ht <= 256 && room >= 6 * (int)(2 * TA_BYTES) && halo_cost < cost) {
            halo = true;
            cost = halo_cost;
            p.PW = 8; p.PH = ph; p.PN = 1; p.n_cols = 8 * ph; p.Wt = wt; p.Ht = ht;
            p.tiles_w = (pl.Wout + 7) / 8; p.tiles_h = (pl.Hout + ph - 1) / ph; p.tiles_n = g.Nb;
            p.splits = 1; p.k_per_split = n_k;
            p.halo_bytes = part;
            p.a_slots = room / (int)(2 * TA_BYTES);
            if (p.a_slots > T_MAX_SLOTS) p.a_slots = T_MAX_SLOTS;
        }
    }
    p.Nb = g.Nb; p.Cout = pl.Cout; p.Mvalid = g.nc * pl.Cout; p.HO = pl.Hout; p.WO = pl.Wout; p.Cp = pl.Cp;
    p.KH = g.KH; p.KW = g.KW; p.SH = pl.SH; p.SW = pl.SW; p.DH = g.DH; p.DW = g.DW;
    p.has_bias = (pass == PASS_FWD && g.has_bias) ? 1 : 0;
    p.LK = pl.LK;
    const bool pair = p.tiles_m % 2 == 0 && deep && (halo || p.n_cols == 256);
    p.split_w = p.split_h = p.split_n = 0;
    if (pair) { if (p.PN >= 2) p.split_n = p.PN / 2; else if (p.PH >= 2) p.split_h = p.PH / 2; else p.split_w = p.PW / 2; }
    p.rows_epi = (p.PW >= 8 && p.store_vec < 8) ? 1 : 0;
    p.off_w = inserted ? 0 : -pl.pad_left; p.off_h = inserted ? 0 : -pl.pad_top;

    alignas(64) CUtensorMap m_w_hi, m_w_lo, m_x_hi, m_x_lo;
    {
        const cuuint64_t dims[3] = {(cuuint64_t)pl.Kp, (cuuint64_t)pl.Mp, (cuuint64_t)taps};
        const cuuint64_t strides[2] = {(cuuint64_t)pl.Kp * 4, (cuuint64_t)pl.Mp * pl.Kp * 4};
        const cuuint32_t box[3] = {TKS, TM, 1};
        int rc = make_tensor_map(&m_w_hi, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, w_hi, 3, dims, strides, box, nullptr, CU_TENSOR_MAP_SWIZZLE_64B, "filters hi");
        if (rc == PCB_OK) rc = make_tensor_map(&m_w_lo, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, w_lo, 3, dims, strides, box, nullptr, CU_TENSOR_MAP_SWIZZLE_64B, "filters lo");
        if (rc != PCB_OK) return rc;
    }
    {
        const cuuint64_t dims[5] = {(cuuint64_t)pl.Cp, (cuuint64_t)pl.Wp, (cuuint64_t)pl.Hp, (cuuint64_t)g.Nb, (cuuint64_t)pl.LK};
        const cuuint64_t strides[4] = {(cuuint64_t)pl.Cp * 4, (cuuint64_t)pl.Wp * pl.Cp * 4, (cuuint64_t)pl.Hp * pl.Wp * pl.Cp * 4,
                                       (cuuint64_t)g.Nb * pl.Hp * pl.Wp * pl.Cp * 4};
        const cuuint32_t box[5] = {TKS, (cuuint32_t)(halo ? p.Wt : ((p.split_w ? p.split_w : p.PW) - 1) * pl.SW + 1), (cuuint32_t)(halo ? p.Ht : ((p.split_h ? p.split_h : p.PH) - 1) * pl.SH + 1), (cuuint32_t)(p.split_n ? p.split_n : p.PN), 1};
        const cuuint32_t es[5] = {1, (cuuint32_t)pl.SW, (cuuint32_t)pl.SH, 1, 1};
        int rc = make_tensor_map(&m_x_hi, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, x_hi, 5, dims, strides, box, es, CU_TENSOR_MAP_SWIZZLE_64B, "activations hi");
        if (rc == PCB_OK) rc = make_tensor_map(&m_x_lo, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, x_lo, 5, dims, strides, box, es, CU_TENSOR_MAP_SWIZZLE_64B, "activations lo");
        if (rc != PCB_OK) return rc;
    }
    const int n_tiles = p.tiles_w * p.tiles_h * p.tiles_n * p.tiles_m;
    {
        // the output is cleared beside the staging of the operands, unless it shares memory with one of them
        const size_t out_bytes = (size_t)g.nc * g.Nb * pl.Cout * pl.Hout * pl.Wout * sizeof(float);
        const bool apart = !overlaps(out, out_bytes, b, (size_t)pl.LK * g.Nb * pl.Cin * pl.Hin * pl.Win * sizeof(float)) &&
                           !overlaps(out, out_bytes, a, (size_t)g.nc * g.Co * g.Ci * taps * sizeof(float));
        const bool cleared = p.splits > 1 && apart && add_zero_job(pro, out, out_bytes);
        const int rc = launch_prologue(pro, sc, stream, &chain);
        if (rc != PCB_OK) return rc;
        if (p.splits > 1 && !cleared) PCB_CUDA_TRY(cudaMemsetAsync(out, 0, out_bytes, stream));
    }
    const int n_items = n_tiles * p.splits / (pair ? 2 : 1), most = pair ? sm_pairs() : sm_count();
    const int grid = (n_items < most ? n_items : most) * (pair ? 2 : 1);
    p.apart = p.n_cols <= TN / 2 ? TN / 2 : 0;
    const int chunk = p.apart ? T_CHUNK_APART : T_CHUNK;
    p.n_chunks = (p.k_per_split + chunk - 1) / chunk;
    p.chunk_len = (p.k_per_split + p.n_chunks - 1) / p.n_chunks;
    size_t smem = (halo ? 1024 + 512 + (size_t)p.a_slots * 2 * TA_BYTES + T_HALO_TILES * 2 * (size_t)p.halo_bytes : T_SMEM) + (p.rows_epi ? 8 * EPI_ROWS_F32_BYTES : 0);
    if (smem < ONE_CTA_SMEM) smem = ONE_CTA_SMEM;
    auto run = [&](auto* kernel) -> int {
        PCB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_CTA_SMEM));
        PCB_CUDA_TRY(launch_clusters(pair ? 2 : 1, chain, kernel, grid, T_THREADS, smem, stream, m_w_hi, m_w_lo, m_x_hi, m_x_lo, p, (const float*)bias, (float*)out, status));
        return PCB_OK;
    };
    int rc;
    if (p.n_chunks > 1) rc = halo ? (pair ? run(qconv_general_tf32_kernel<true, true, true>) : run(qconv_general_tf32_kernel<true, true, false>))
                                  : (pair ? run(qconv_general_tf32_kernel<true, false, true>) : run(qconv_general_tf32_kernel<true, false, false>));
    else rc = halo ? (pair ? run(qconv_general_tf32_kernel<false, true, true>) : run(qconv_general_tf32_kernel<false, true, false>))
                   : (pair ? run(qconv_general_tf32_kernel<false, false, true>) : run(qconv_general_tf32_kernel<false, false, false>));
    if (rc != PCB_OK) return rc;
    PCB_CUDA_TRY(cudaGetLastError());
    return PCB_OK;
}

}  // namespace pcb
