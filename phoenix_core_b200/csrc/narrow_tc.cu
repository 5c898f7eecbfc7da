// tcgen05 kernels for NARROW layers: at most 16 channels per component on the reduced side, stride-1 correlation
// (forward of a stride-1 layer, backward-data of any layer this file's geometry covers, filter gradient of a
// stride-1 layer), 16-bit tensors.
//
// Why a separate family. With 16 channels a pixel is 32 bytes, and the general implicit-GEMM kernels (conv_tc.cu)
// fetch, for every filter tap, a fresh box of such 32-byte rows: per MMA of 128 x 256 x 16 they move 12 KB from L2
// to shared memory and run at 1/7 of the tensor rate; the filter-gradient kernel fares worse. Here every pixel is
// fetched ONCE per tile and all taps read it from shared memory:
//
//   * Staged activations are "planar": xp[comp][img][plane = c / 8][hp][wp][8 channels] (zero padded as in
//     conv_tc.cu), so that pixels of one plane are 16 bytes apart. A tile of 8 x PH output pixels needs the halo
//     tile (8 + (KW-1)*DW) x (PH + (KH-1)*DH), which one TMA box brings in as [plane][row][pixel][8].
//   * That halo tile IS a tcgen05 operand in the layout without swizzle for every tap at once: 8 consecutive pixels
//     of a row are one 128-byte core matrix, the next row of the tile is one halo-row pitch further (the stride
//     offset), the second 8-channel half is one plane further (the leading offset), and tap (kh, kw) is nothing but
//     a different start address, (kh*DH*Wt + kw*DW) * 16 bytes. The same holds for the MN-major view that the filter
//     gradient needs (K = pixels).
//   * The signed/permuted filter matrix Wexp[tap][(d,co)][(l,ci)] (reference sign tables src/algebras.cc:5-145) of such
//     a layer is small (3x3 quaternion: 144 KB) and stays resident in shared memory for the life of the CTA.
//
// Replaces, for these layers, the 8/16 scalar library convolutions and accumulate passes of src/conv2d.hpp:167-275
// (forward), :433-562 (backward).
#include "tc_common.cuh"
#include "tensor_path.cuh"

namespace pcb {
namespace {

using namespace umma;
using namespace tc;

constexpr int NM = 128;                  // MMA M: (d, co) rows, padded
constexpr int N_THREADS = 320;           // filter gradient: warp 0 TMA, warp 1 MMA, warps 2..9 epilogue
// Forward / backward-data: warps 2..17 epilogue, four per TMEM lane quadrant. Layers of this file have few rows (16 quaternion channels:
// 64 of the 128 lanes), so half of the epilogue warps have none, and with two warps per quadrant the drain of a tile took twice as
// long as its MMAs.
constexpr int N_EPI_WARPS = 16, NW_THREADS = 64 + 32 * N_EPI_WARPS;
constexpr int NB_STAGES = 4;             // halo tiles in flight (one per input component)
constexpr uint32_t NA_BYTES = NM * 16 * 2;   // one (tap, component) slice of the filter matrix: [2 planes][128 rows][8]
constexpr int ST_N_PRODUCER = 0x10000, ST_N_MMA = 0x20000, ST_N_EPILOGUE = 0x40000;

struct NParams {
    int Nb, Mvalid, Cout, HO, WO;        // batch; valid rows (components x Cout); output plane
    int KH, KW, DH, DW;
    int PH;                              // output tile = 8 x PH pixels of one image (PH even, <= 32), 16 x PH (PH <= 16) in the wide form
    int Wt, Ht;                          // halo tile
    int tiles_w, tiles_h;
    int LK, taps;
    int fmt, has_bias, store_vec;
    int rows_epi;                        // image rows that are not 16-byte aligned leave through shared memory (store_rows)
    uint32_t stage_bytes;                // shared-memory pitch of one halo stage
    uint32_t plane_bytes;                // Ht * Wt * 16
};

// Operand without swizzle: core matrices of 8 rows x 16 bytes; `lead` = distance between the two 8-element halves of
// the 16 K elements (K-major) or between 8-row K groups (MN-major); `stride` = distance between 8-row groups
// (K-major) or between 8-element MN chunks (MN-major).
__device__ __forceinline__ uint64_t desc_plain(uint32_t smem_addr, uint32_t lead, uint32_t stride) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)((lead >> 4) & 0x3FFFu) << 16) | ((uint64_t)((stride >> 4) & 0x3FFFu) << 32) |
           DESC_VERSION_SM100;
}

// K-major operand with 64-byte rows, 64-byte swizzle.
__device__ __forceinline__ uint64_t desc_rows64(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | DESC_VERSION_SM100 | (4ull << 61);
}

// ===================================================================================================
// Forward / backward-data: D[(d,co), pixel] = sum over (tap, l, ci) of Wexp * x, tile 128 x (8 x PH pixels).
// WIDE: the tile is two such blocks of 8 pixels side by side, an MMA each per tap, so that a lane stores runs of 16 pixels (whole 32-byte
// sectors): taken where image rows are whole runs. The 16-byte runs of single blocks
// bound the 7x7/2 stem (112 x 112 outputs): forward 158 -> 111 us at batch 128.
// ===================================================================================================
template <bool WIDE>
__global__ void __launch_bounds__(NW_THREADS, 1)
qconv_narrow_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, NParams p,
                       const uint16_t* bias, uint16_t* __restrict__ out, int* __restrict__ status) {
    extern __shared__ uint8_t smem_raw[];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t a_bytes = (uint32_t)p.taps * p.LK * NA_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + a_bytes + NB_STAGES * p.stage_bytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * NB_STAGES + 5);
    const uint32_t a_addr = smem_u32(base), b_addr = a_addr + a_bytes;
    const uint32_t full_bar = smem_u32(bars), empty_bar = smem_u32(bars + NB_STAGES);
    const uint32_t tmem_full = smem_u32(bars + 2 * NB_STAGES), tmem_empty = smem_u32(bars + 2 * NB_STAGES + 2);
    const uint32_t a_full = smem_u32(bars + 2 * NB_STAGES + 4);

    const int tiles_img = p.tiles_w * p.tiles_h;
    const int n_tiles = tiles_img * p.Nb;
    const int n_block = 8 * p.PH, n_cols = WIDE ? 2 * n_block : n_block;      // columns of an MMA, of the tile

    if (t == 0) {
        for (int s = 0; s < NB_STAGES; ++s) { mbar_init(full_bar + 8 * s, 1); mbar_init(empty_bar + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(tmem_full + 8 * b, 1); mbar_init(tmem_empty + 8 * b, N_EPI_WARPS); }
        mbar_init(a_full, 1);
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
        // ---------------------------------------------------------------- TMA producer
        if (blockIdx.x < n_tiles) {
            const bool el = elect_one();
            if (el) {
                mbar_arrive_expect_tx(a_full, a_bytes);
                for (int tap = 0; tap < p.taps; ++tap)
                    for (int l = 0; l < p.LK; ++l)
                        tma_load_4d(a_addr + (tap * p.LK + l) * NA_BYTES, &map_w, 0, 0, 2 * l, tap, a_full);   // [2 planes][128 rows][8]
            }
            int it = 0;
            bool ok = true;
            const uint32_t tx = (uint32_t)p.Wt * p.Ht * 32;
            for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
                const int img = tile / tiles_img, r = tile - img * tiles_img;
                const int th = r / p.tiles_w, tw = r - th * p.tiles_w;
                for (int l = 0; l < p.LK; ++l, ++it) {
                    const int s = it % NB_STAGES;
                    ok = warp_wait_bounded(empty_bar + 8 * s, ((it / NB_STAGES) & 1) ^ 1, status, ST_N_PRODUCER);
                    if (!ok) break;
                    if (el) {
                        mbar_arrive_expect_tx(full_bar + 8 * s, tx);
                        tma_load_5d(b_addr + s * p.stage_bytes, &map_x, tw * (WIDE ? 128 : 64), th * p.PH, 0, img, l, full_bar + 8 * s);   // [2 planes][Ht][Wt][8]
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        const uint32_t idesc = make_idesc_f16(p.fmt, NM, n_block, false, false);
        int it = 0, local_tile = 0;
        const bool el = elect_one();
        bool ok = blockIdx.x >= n_tiles || warp_wait_bounded(a_full, 0, status, ST_N_MMA);
        for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++local_tile) {
            const int buf = local_tile & 1, use = local_tile >> 1;
            if (use > 0) {
                ok = warp_wait_bounded(tmem_empty + 8 * buf, (use - 1) & 1, status, ST_N_MMA);
                if (!ok) break;
                tc_fence_after_sync();
            }
            for (int l = 0; l < p.LK && ok; ++l, ++it) {
                const int s = it % NB_STAGES;
                ok = warp_wait_bounded(full_bar + 8 * s, (it / NB_STAGES) & 1, status, ST_N_MMA);
                if (!ok) break;
                tc_fence_after_sync();
                if (el) {
                    const uint64_t ad = desc_plain(a_addr + l * NA_BYTES, NM * 16, 128), bd = desc_plain(b_addr + s * p.stage_bytes, p.plane_bytes, p.Wt * 16);
                    const uint32_t a_step = (uint32_t)(p.LK * NA_BYTES) >> 4, a_hi = (uint32_t)(ad >> 32), b_hi = (uint32_t)(bd >> 32);
                    uint32_t a_lo = (uint32_t)ad, b_row = (uint32_t)bd;
                    for (int kh = 0; kh < p.KH; ++kh) {
                        uint32_t b_lo = b_row;
                        for (int kw = 0; kw < p.KW; ++kw) {
                            const uint32_t acc = (l > 0 || kh > 0 || kw > 0) ? 1u : 0u;
                            mma_f16_ss_words(tmem_base + buf * 256, a_lo, a_hi, b_lo, b_hi, idesc, acc);
                            if (WIDE) mma_f16_ss_words(tmem_base + buf * 256 + n_block, a_lo, a_hi, b_lo + 8, b_hi, idesc, acc);
                            a_lo += a_step;
                            b_lo += p.DW;
                        }
                        b_row += p.DH * p.Wt;
                    }
                    mma_commit(empty_bar + 8 * s);
                    if (l == p.LK - 1) mma_commit(tmem_full + 8 * buf);
                }
                __syncwarp();
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue (warps 2..17)
        const int q = warp & 3;                    // TMEM lane quadrant
        const int part = (warp - 2) >> 2;          // takes the 32-column blocks part, part + 4
        const bool some_rows = q * 32 < p.Mvalid;  // warp-uniform
        const uint32_t rbuf = smem_u32(bars) + 256 + (uint32_t)(warp - 2) * EPI_ROWS_BYTES;
        const int sv = p.store_vec;                // output pixels per store: 8, 4, 2 or 1
        int local_tile = 0;
        bool ok = true;
        const int m = q * 32 + lane;
        const bool row_ok = m < p.Mvalid;
        const int d = row_ok ? m / p.Cout : 0, co = m - d * p.Cout;
        float badd = 0.f;
        if (row_ok && p.has_bias) {
            const uint16_t raw = ld_chained(bias + d * p.Cout + co);
            badd = p.fmt == 0 ? __half2float(__ushort_as_half(raw)) : __bfloat162float(__ushort_as_bfloat16(raw));
        }
        for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++local_tile) {
            const int buf = local_tile & 1, use = local_tile >> 1;
            const int img = tile / tiles_img, r = tile - img * tiles_img;
            const int th = r / p.tiles_w, tw = r - th * p.tiles_w;
            const int ow0 = tw * (WIDE ? 16 : 8), oh0 = th * p.PH;
            // (no read of the status word here: 16 warps that all ask for it at every tile cost the 7x7/2 stem 3 to 6 %. Whoever gives up
            // a wait stops signalling, so a tile behind an expired wait is never announced.)
            ok = mbar_wait_bounded(tmem_full + 8 * buf, use & 1, status, ST_N_EPILOGUE);
            ok = warp_may_store(ok, 0);
            if (!ok) break;
            tc_fence_after_sync();
#pragma unroll 1
            for (int col0 = part * 32; col0 < n_cols && some_rows; col0 += 128) {
                uint32_t v[32];
                if (WIDE) {                                              // two rows: eight pixels of each from either block
                    uint32_t left[16], right[16];
                    const uint32_t at = tmem_base + ((uint32_t)(q * 32) << 16) + buf * 256 + col0 / 2;
                    tmem_ld_32x32b_x16(at, left);
                    tmem_ld_32x32b_x16(at + n_block, right);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 8; ++e) { v[e] = left[e]; v[8 + e] = right[e]; v[16 + e] = left[8 + e]; v[24 + e] = right[8 + e]; }
                } else {
                    tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + buf * 256 + col0, v);
                    tmem_ld_wait();
                }
                if (!row_ok && !p.rows_epi) continue;
                uint32_t packed[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float f0 = __uint_as_float(v[2 * e]) + badd, f1 = __uint_as_float(v[2 * e + 1]) + badd;
                    if (p.fmt == 0) { const __half2 h = __floats2half2_rn(f0, f1); packed[e] = *reinterpret_cast<const uint32_t*>(&h); }
                    else { const __nv_bfloat162 h = __floats2bfloat162_rn(f0, f1); packed[e] = *reinterpret_cast<const uint32_t*>(&h); }
                }
                if (p.rows_epi) {
                    const int je = col0 + (sv == 1 ? lane : (sv == 2 ? (lane & 15) * 2 : (lane & 7) * 4));
                    const int ow = ow0 + (je & 7), oh = oh0 + (je >> 3);
                    const int pix_off = (je < n_cols && ow < p.WO && oh < p.HO) ? (img * p.Cout * p.HO + oh) * p.WO + ow : -1;
                    const int row_off = row_ok ? (d * p.Nb * p.Cout + co) * p.HO * p.WO : -1;
                    if (sv == 1) store_rows<1>(rbuf, packed, out, row_off, pix_off, lane);
                    else if (sv == 2) store_rows<2>(rbuf, packed, out, row_off, pix_off, lane);
                    else store_rows<4>(rbuf, packed, out, row_off, pix_off, lane);
                    continue;
                }
                if (WIDE) {
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const int oh = oh0 + (col0 >> 4) + r;
                        if (col0 + r * 16 >= n_cols || oh >= p.HO) continue;
                        st_global_v8(out + (((size_t)(d * p.Nb + img) * p.Cout + co) * p.HO + oh) * p.WO + ow0, &packed[8 * r]);
                    }
                    continue;
                }
#pragma unroll
                for (int g8 = 0; g8 < 4; ++g8) {                         // 8 columns = one row of the tile
                    const int oh = oh0 + (col0 >> 3) + g8;
                    if (col0 + g8 * 8 >= n_cols || oh >= p.HO || ow0 >= p.WO) continue;
                    uint16_t* dst = out + (((size_t)(d * p.Nb + img) * p.Cout + co) * p.HO + oh) * p.WO + ow0;
                    if (sv >= 8) {
                        *reinterpret_cast<uint4*>(dst) = make_uint4(packed[4 * g8], packed[4 * g8 + 1], packed[4 * g8 + 2], packed[4 * g8 + 3]);
                    } else if (sv == 4) {
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            if (ow0 + 4 * h < p.WO) *reinterpret_cast<uint2*>(dst + 4 * h) = make_uint2(packed[4 * g8 + 2 * h], packed[4 * g8 + 2 * h + 1]);
                    } else if (sv == 2) {
#pragma unroll
                        for (int h = 0; h < 4; ++h)
                            if (ow0 + 2 * h < p.WO) *reinterpret_cast<uint32_t*>(dst + 2 * h) = packed[4 * g8 + h];
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            if (ow0 + e < p.WO) dst[e] = (uint16_t)((packed[4 * g8 + (e >> 1)] >> ((e & 1) * 16)) & 0xffffu);
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(tmem_empty + 8 * buf);
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, 512);
}

// ---- staging: everything a call needs before its main kernel, in one launch (as in conv_tc.cu) -----------------------------------
// xp[plane_in = comp*Nb + img][c / 8 (`groups` planes)][hp][wp][8] = x[plane_in][c][hp - pad_top][wp - pad_left], zero outside and for
// c >= C; ins > 1 spreads the source pixels `ins` apart (the zero insertion of a strided backward-data pass).
// s2d ("space to depth", stride-2 layers with at most 4 channels): staged channel c' = (dy, dx, c) of staged pixel
// (hp, wp) is source channel c at padded position (2*hp + dy, 2*wp + dx); the stride-2 convolution of the source
// is then a stride-1 convolution of the staged tensor with ceil(K/2) taps per axis and 4*C channels.
// 16-bit elements are moved as raw bits.
enum { PLANAR_NONE = -1, PLANAR_ANY = 0, PLANAR_ROWS = 1, PLANAR_S2D_PAIRS = 2 };
struct PlanarJob {
    const uint16_t* x;
    uint16_t* xp;
    int form, planes_in, C, H, W, Hp, Wp, groups /*8-channel planes per component*/, pad_top, pad_left, ins_h, ins_w, s2d;
    unsigned blocks;
};
constexpr int NP_THREADS = 256;

__device__ __forceinline__ void pack_planar_any(const PlanarJob& p, unsigned block) {
    const size_t total = (size_t)p.planes_in * p.groups * p.Hp * p.Wp;
    for (size_t idx = (size_t)block * NP_THREADS + threadIdx.x; idx < total; idx += (size_t)p.blocks * NP_THREADS) {
        const int wp = (int)(idx % p.Wp);
        size_t rest = idx / p.Wp;
        const int hp = (int)(rest % p.Hp); rest /= p.Hp;
        const int grp = (int)(rest % p.groups);
        const int plane = (int)(rest / p.groups);
        int ih = hp - p.pad_top, iw = wp - p.pad_left;
        bool inside = ih >= 0 && iw >= 0;
        if (inside && (p.ins_h > 1 || p.ins_w > 1)) {
            inside = (ih % p.ins_h == 0) && (iw % p.ins_w == 0);
            ih /= p.ins_h; iw /= p.ins_w;
        }
        inside = inside && ih < p.H && iw < p.W;
        alignas(16) uint16_t vals[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int c = grp * 8 + e;
            uint16_t v = 0;
            if (p.s2d) {
                const int sub = c / p.C, cs = c - sub * p.C;             // sub = dy * 2 + dx
                const int sh = 2 * hp + (sub >> 1) - p.pad_top, sw = 2 * wp + (sub & 1) - p.pad_left;
                if (sub < 4 && sh >= 0 && sw >= 0 && sh < p.H && sw < p.W) v = ld_chained(p.x + (((size_t)plane * p.C + cs) * p.H + sh) * p.W + sw);
            } else if (c < p.C && inside) {
                v = ld_chained(p.x + (((size_t)plane * p.C + c) * p.H + ih) * p.W + iw);
            }
            vals[e] = v;
        }
        *reinterpret_cast<uint4*>(p.xp + idx * 8) = *reinterpret_cast<const uint4*>(vals);
    }
}

// No zero insertion, W a multiple of 4 and rows aligned to 8 bytes: one thread moves 8 channels x 4 pixels -- eight loads of 8 bytes and
// four 16-byte stores. The channel group runs fastest across threads. The threads at the ends of a row also write the padding columns.
__device__ __forceinline__ void pack_planar_rows(const PlanarJob& p, unsigned block) {
    const int Wq = p.W / 4;
    const unsigned total = (unsigned)p.planes_in * p.groups * p.Hp * Wq;   // 32-bit indices: staged copies stay below 2^32 / 8 threads
    for (unsigned idx = block * NP_THREADS + threadIdx.x; idx < total; idx += p.blocks * NP_THREADS) {
        const int grp = (int)(idx % p.groups);
        unsigned rest = idx / p.groups;
        const int q = (int)(rest % Wq); rest /= Wq;
        const int hp = (int)(rest % p.Hp);
        const int plane = (int)(rest / p.Hp);
        const int ih = hp - p.pad_top;
        const bool row_in = ih >= 0 && ih < p.H;
        alignas(8) uint16_t v[8][4];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int c = grp * 8 + e;
            const uint2 raw = ld_chained(reinterpret_cast<const uint2*>(p.x + (((size_t)plane * p.C + c) * p.H + ih) * p.W + 4 * q), row_in && c < p.C);
            *reinterpret_cast<uint2*>(v[e]) = raw;
        }
        uint16_t* row = p.xp + (((size_t)plane * p.groups + grp) * p.Hp + hp) * (size_t)p.Wp * 8;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            alignas(16) uint16_t o[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = v[e][j];
            *reinterpret_cast<uint4*>(row + (size_t)(p.pad_left + 4 * q + j) * 8) = *reinterpret_cast<const uint4*>(o);
        }
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        if (q == 0)
            for (int wp = 0; wp < p.pad_left && wp < p.Wp; ++wp) *reinterpret_cast<uint4*>(row + (size_t)wp * 8) = zero;
        if (q == Wq - 1)
            for (int wp = p.pad_left + p.W; wp < p.Wp; ++wp) *reinterpret_cast<uint4*>(row + (size_t)wp * 8) = zero;
    }
}

// The space-to-depth copy for an even left padding and an even line length: a staged pixel's two source columns (dx = 0, 1)
// are one aligned 32-bit word, so a thread makes BOTH 8-channel planes of one staged pixel from 2 * C coalesced 4-byte loads
// (2 source lines x C channels) instead of 16 scattered 2-byte loads.
template <int C>
__device__ __forceinline__ void pack_planar_s2d_pairs(const PlanarJob& p, unsigned block) {
    const size_t total = (size_t)p.planes_in * p.Hp * p.Wp;
    const size_t plane_pitch = (size_t)p.Hp * p.Wp * 8;           // elements between the two 8-channel planes
    for (size_t idx = (size_t)block * NP_THREADS + threadIdx.x; idx < total; idx += (size_t)p.blocks * NP_THREADS) {
        const int wp = (int)(idx % p.Wp);
        size_t rest = idx / p.Wp;
        const int hp = (int)(rest % p.Hp);
        const int plane = (int)(rest / p.Hp);
        alignas(16) uint16_t vals[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) vals[e] = 0;
        const int sw = 2 * wp - p.pad_left;                      // even: the pair (sw, sw + 1) is one aligned word
#pragma unroll
        for (int dy = 0; dy < 2; ++dy) {
            const int sh = 2 * hp + dy - p.pad_top;
            if (sh < 0 || sh >= p.H || sw < 0 || sw >= p.W) continue;   // W is even, so sw + 1 < W as well
#pragma unroll
            for (int cs = 0; cs < C; ++cs) {
                const uint32_t pair = ld_chained(reinterpret_cast<const uint32_t*>(p.x + (((size_t)plane * C + cs) * p.H + sh) * p.W + sw));
                vals[(dy * 2 + 0) * C + cs] = (uint16_t)(pair & 0xffffu);             // staged channel (dy, dx, c)
                vals[(dy * 2 + 1) * C + cs] = (uint16_t)(pair >> 16);
            }
        }
        uint16_t* dst = p.xp + (((size_t)plane * 2) * p.Hp + hp) * (size_t)p.Wp * 8 + (size_t)wp * 8;
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(vals);
        *reinterpret_cast<uint4*>(dst + plane_pitch) = *reinterpret_cast<const uint4*>(vals + 8);
    }
}

// Wexp[tap][k / 8][m][k % 8] with m = (d, co) or (l, ci), k = (l, ci) or (d, co) as in conv_tc.cu; 128 rows, K = LK * 16.
// s2d: staged tap (a, b) of staged channel c' = (dy, dx, ci) is source tap (2a + dy, 2b + dx) of channel ci (zero past the
// filter edge); `taps` counts staged taps, KH x KW is the source filter, KWe the staged filter width.
struct PlanarFilterJob {
    const uint16_t* w;
    uint16_t* wexp;
    int Co, Ci, taps, Kp, transposed, nc, ga;
    unsigned long long neg;
    int s2d, KH, KW, KWe;
};
__device__ __forceinline__ void pack_filters_planar(const PlanarFilterJob& p, unsigned block, unsigned blocks) {
    const size_t total = (size_t)p.taps * NM * p.Kp;
    const int Cm = p.transposed ? p.Ci : p.Co, Ck = p.transposed ? p.Co : p.Ci;
    for (size_t idx = (size_t)block * NP_THREADS + threadIdx.x; idx < total; idx += (size_t)blocks * NP_THREADS) {
        const int k = (int)(idx % p.Kp);
        const int m = (int)((idx / p.Kp) % NM);
        const int tap = (int)(idx / ((size_t)p.Kp * NM));
        const int cm_comp = m / Cm, cm = m - cm_comp * Cm;
        const int ck_comp = k / 16, ck = k - ck_comp * 16;
        uint16_t v = 0;
        if (p.s2d) {                                 // forward only: m = (d, co), k = (l, c')
            const int sub = ck / p.Ci, ci = ck - sub * p.Ci;
            const int kh = 2 * (tap / p.KWe) + (sub >> 1), kw = 2 * (tap % p.KWe) + (sub & 1);
            if (cm_comp < p.nc && ck_comp < p.nc && sub < 4 && kh < p.KH && kw < p.KW) {
                v = ld_chained(p.w + ((size_t)(alg_pair(p.ga, ck_comp, cm_comp) * p.Co + cm) * p.Ci + ci) * (p.KH * p.KW) + kh * p.KW + kw);
                if (alg_negative(p.neg, ck_comp, cm_comp)) v ^= 0x8000u;
            }
        } else if (cm_comp < p.nc && ck_comp < p.nc && ck < Ck) {
            const int d = p.transposed ? ck_comp : cm_comp, l = p.transposed ? cm_comp : ck_comp;
            const int co = p.transposed ? ck : cm, ci = p.transposed ? cm : ck;
            const int src_tap = p.transposed ? p.taps - 1 - tap : tap;
            v = ld_chained(p.w + ((size_t)(alg_pair(p.ga, l, d) * p.Co + co) * p.Ci + ci) * p.taps + src_tap);
            if (alg_negative(p.neg, l, d)) v ^= 0x8000u;
        }
        p.wexp[(((size_t)tap * (p.Kp / 8) + k / 8) * NM + m) * 8 + (k & 7)] = v;
    }
}

// The status word of the call, the filter matrix, the zeroed accumulator and up to two staged copies. As launches of their own (the
// filter matrix on a side stream, two memsets) they cost a 3x3/2 stem of 64 x 64 images, batch 81, fp16, forward + backward 13 of 54 us.
struct PlanarPrologue {
    int* status = nullptr;
    PlanarFilterJob filter;
    PlanarJob stage[2];
    uint4* zero = nullptr;
    unsigned zero_units = 0, filter_blocks = 0, zero_blocks = 0;
    int n_stages = 0;
};
// One instance per pair of staging forms (a stage that is not there: PLANAR_NONE), each with the registers of its own forms: the copies
// live on the number of loads in flight.
template <int FORM>
__device__ __forceinline__ void pack_planar(const PlanarJob& job, unsigned block) {
    if (FORM == PLANAR_ROWS) pack_planar_rows(job, block);
    else if (FORM == PLANAR_ANY) pack_planar_any(job, block);
    else if (FORM == PLANAR_S2D_PAIRS) {
        if (job.C == 3) pack_planar_s2d_pairs<3>(job, block);
        else if (job.C == 1) pack_planar_s2d_pairs<1>(job, block);
        else if (job.C == 2) pack_planar_s2d_pairs<2>(job, block);
        else pack_planar_s2d_pairs<4>(job, block);
    }
}
template <int FORM0, int FORM1>
__global__ void __launch_bounds__(NP_THREADS) planar_prologue_kernel(const __grid_constant__ PlanarPrologue p) {
    chain_wait();
    chain_next();
    unsigned block = blockIdx.x;
    if (block == 0 && threadIdx.x == 0 && p.status) *p.status = 0;
    if (block < p.filter_blocks) { pack_filters_planar(p.filter, block, p.filter_blocks); return; }
    block -= p.filter_blocks;
    if (block < p.zero_blocks) {
        for (unsigned i = block * NP_THREADS + threadIdx.x; i < p.zero_units; i += p.zero_blocks * NP_THREADS) p.zero[i] = make_uint4(0u, 0u, 0u, 0u);
        return;
    }
    block -= p.zero_blocks;
    if (block < p.stage[0].blocks) pack_planar<FORM0>(p.stage[0], block);
    else pack_planar<FORM1>(p.stage[1], block - p.stage[0].blocks);
}
void add_planar_job(PlanarPrologue& pro, const void* src, void* dst, int planes_in, int C, int H, int W, int Hp, int Wp, int groups, int pad_top, int pad_left,
                    int ins_h, int ins_w, int s2d) {
    PlanarJob& j = pro.stage[pro.n_stages++];
    j.x = static_cast<const uint16_t*>(src); j.xp = static_cast<uint16_t*>(dst);
    j.planes_in = planes_in; j.C = C; j.H = H; j.W = W; j.Hp = Hp; j.Wp = Wp; j.groups = groups; j.pad_top = pad_top; j.pad_left = pad_left;
    j.ins_h = ins_h; j.ins_w = ins_w; j.s2d = s2d;
    const uintptr_t at = reinterpret_cast<uintptr_t>(src), to = reinterpret_cast<uintptr_t>(dst);
    const size_t units = (size_t)planes_in * groups * Hp * Wp;
    if (!s2d && ins_h == 1 && ins_w == 1 && pad_left >= 0 && pad_left + W <= Wp && W % 4 == 0 && at % 8 == 0) {
        j.form = PLANAR_ROWS;
        j.blocks = grid_cap(units / 4 + 1, NP_THREADS, 16);
    } else if (s2d && groups == 2 && C >= 1 && C <= 4 && pad_left % 2 == 0 && W % 2 == 0 && at % 4 == 0 && to % 16 == 0) {
        j.form = PLANAR_S2D_PAIRS;
        j.blocks = grid_cap((size_t)planes_in * Hp * Wp, NP_THREADS, 16);
    } else {
        j.form = PLANAR_ANY;
        j.blocks = grid_cap(units, NP_THREADS, 16);
    }
}
// `chain`: whether the main kernel may be chained to this launch (the copies' CTAs are capped at 16 per SM: a capped one is a long one.
// Chained / not, us: 16 -> 16, 32 x 32, 3x3, forward, batch 256, below the cap 45.8 / 49.5, batch 16 12.8 / 14.8; above it 112 x 112, batch 64, both
// gradients 350 / 340, the 7x7/2 stem at batch 128 350 / 245).
int launch_prologue(PlanarPrologue& pro, StatusClear* sc, cudaStream_t stream, bool* chain) {
    unsigned copies = 0;
    for (int i = 0; i < pro.n_stages; ++i) copies += pro.stage[i].blocks;
    const unsigned blocks = pro.filter_blocks + pro.zero_blocks + copies;
    if (pro.n_stages == 0) pro.stage[0].blocks = 0;
    *chain = copies < 16u * (unsigned)sm_count();
    if (sc && sc->pending) { pro.status = sc->word; sc->pending = false; }
    auto run = [&](void (*kernel)(PlanarPrologue)) -> int {
        PCB_CUDA_TRY(launch_chained(kernel, blocks, NP_THREADS, 0, stream, pro));
        return PCB_OK;
    };
    const int f0 = pro.n_stages > 0 ? pro.stage[0].form : PLANAR_NONE, f1 = pro.n_stages > 1 ? pro.stage[1].form : PLANAR_NONE;
    if (f0 == PLANAR_NONE) return run(planar_prologue_kernel<PLANAR_NONE, PLANAR_NONE>);
#define PCB_PLANAR_PAIR(F0)                                                                   \
    if (f0 == F0) {                                                                           \
        if (f1 == PLANAR_NONE) return run(planar_prologue_kernel<F0, PLANAR_NONE>);           \
        if (f1 == PLANAR_ROWS) return run(planar_prologue_kernel<F0, PLANAR_ROWS>);           \
        return run(planar_prologue_kernel<F0, PLANAR_ANY>);                                   \
    }
    PCB_PLANAR_PAIR(PLANAR_ROWS)
    PCB_PLANAR_PAIR(PLANAR_ANY)
    PCB_PLANAR_PAIR(PLANAR_S2D_PAIRS)
#undef PCB_PLANAR_PAIR
    return PCB_ERR_INVALID_ARGUMENT;
}

// ===================================================================================================
// Filter gradient: G_tap[(d,co), (l,ci)] = sum over pixels of dy[(d,co), pixel] * x[(l,ci), pixel + tap], then
// dw[pair(l,d)][co][ci][tap] += sign(l,d) * G_tap. Both operands MN-major (K = pixels) in the layout without swizzle:
// dy tile [d][plane][PH][8 px][8], x halo tile [l][plane][Ht][Wt][8]; 8 consecutive pixels are one core matrix, the
// next tile row is the leading offset, the next 8 channels the stride offset, a tap is a start address. One CTA owns
// a group of taps (as many accumulators of N = LK*16 columns as fit the 512 TMEM columns) and a range of pixel
// tiles; its accumulators stay in TMEM for the whole range and are folded into fp32 scratch at the end.
// M is always 128: with fewer (d, plane) chunks than 16 the upper rows multiply whatever follows the dy tile in
// shared memory and are never read back.
// Folded form (p.fold = KW > 1): an MMA costs about the same whether it is 16 or 128 columns wide, so the kw taps of one
// filter row become columns of ONE MMA. The x tensor map gets the tap as a dimension of its own with a stride of one pixel
// (16 bytes) over the same staged copy -- overlapping views -- so that one box brings the tile shifted by every kw:
// [kw][l][plane][Ht][8 px][8], planes at one uniform pitch, N = KW * LK * 16 columns, one MMA per filter row and 16 pixels.
// A real-valued x (one component) leaves a map dimension free for the filter rows as well (stride: one staged row): the
// box is then [kw][kh][plane][Ht][8 px][8] and one MMA of N = fold_h * KW * 16 columns serves fold_h filter rows: all of them (no halo
// rows), or half of them from four rows up.
// DIRECT: dy is read in place. Pixels are contiguous in NCHW, so a box of 32 pixels x all channels of all components x PH rows is a K-major
// operand, 64-byte rows [row][(d, co)][32 pixels]; x boxes are 32 pixels wide too, and 16 pixels of one image row are the K of an MMA.
// Layers whose dy nobody stages for another pass (no input gradient: the stem), where tiles of 32 pixels exceed the rows by a quarter at
// most. Backward of the 7x7/2 stem, 224 x 224, batch 128: 209 -> 133 us, of which 70 us were the copy of dy.
// ===================================================================================================
constexpr int NF_STAGES = 2;
constexpr int NF_MAX_GROUPS = 16;        // tap groups that can be given CTA shares of their own

struct NFParams {
    int Nb, Co, Ci, nc, ga;
    unsigned long long neg;
    int KH, KW, DH, DW;
    int PH, Wt, Ht, tiles_w, tiles_h;
    int LK, taps, taps_per_group, n_groups;
    int fold, fold_h, LKr;               // kw (and, for one-component x, kh) taps folded into the columns of one MMA (1 = none); components of x
    int y_planes;                        // 8-channel planes of dy per component
    int steps_total, steps_per_split;
    // uneven != 0: group g owns the CTAs [cta_begin[g], cta_begin[g + 1]) and walks group_steps[g] pixel tiles per CTA -- a
    // last group with fewer taps gets fewer CTAs, so that every CTA issues about the same number of MMAs
    int uneven, cta_begin[NF_MAX_GROUPS + 1], group_steps[NF_MAX_GROUPS];
    int fmt;
    uint32_t y_bytes, x_bytes, stage_bytes, plane_bytes;
};
constexpr int ND_W = 32;                 // pixels across a tile of the DIRECT form

template <bool DIRECT>
__global__ void __launch_bounds__(N_THREADS, 1)
qconv_narrow_filter_tc_kernel(const __grid_constant__ CUtensorMap map_dy, const __grid_constant__ CUtensorMap map_x, NFParams p,
                              float* __restrict__ dw32, int* __restrict__ status) {
    extern __shared__ uint8_t smem_raw[];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    // barriers first: the operand region is followed by slack that the M = 128 operand may read
    uint64_t* bars = reinterpret_cast<uint64_t*>(base);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * NF_STAGES + 1);
    const uint32_t tiles_addr = smem_u32(base) + 1024;
    const uint32_t full_bar = smem_u32(bars), empty_bar = smem_u32(bars + NF_STAGES), tmem_full = smem_u32(bars + 2 * NF_STAGES);

    int group = blockIdx.x % p.n_groups, split = blockIdx.x / p.n_groups, steps_per_split = p.steps_per_split;
    if (p.uneven) {
        group = 0;
        while (group + 1 < p.n_groups && (int)blockIdx.x >= p.cta_begin[group + 1]) ++group;
        split = blockIdx.x - p.cta_begin[group];
        steps_per_split = p.group_steps[group];
    }
    const int tap0 = group * p.taps_per_group;
    const int n_taps = min(p.taps_per_group, p.taps - tap0);
    const int step_beg = split * steps_per_split;
    const int n_steps = max(0, min(p.steps_total, step_beg + steps_per_split) - step_beg);
    const int tiles_img = p.tiles_w * p.tiles_h;
    const int ncols = p.LK * 16;

    if (t == 0) {
        for (int s = 0; s < NF_STAGES; ++s) { mbar_init(full_bar + 8 * s, 1); mbar_init(empty_bar + 8 * s, 1); }
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
            bool ok = true;
            int img = step_beg / tiles_img, th = (step_beg - img * tiles_img) / p.tiles_w, tw = step_beg - img * tiles_img - th * p.tiles_w;
            for (int it = 0; it < n_steps && ok; ++it) {
                const int s = it % NF_STAGES;
                ok = warp_wait_bounded(empty_bar + 8 * s, ((it / NF_STAGES) & 1) ^ 1, status, ST_N_PRODUCER);
                if (!ok) break;
                const uint32_t dst = tiles_addr + s * p.stage_bytes, bar = full_bar + 8 * s;
                if (el) {
                    mbar_arrive_expect_tx(bar, p.y_bytes + p.x_bytes);
                    if (DIRECT) {
                        tma_load_5d(dst, &map_dy, tw * ND_W, 0, 0, th * p.PH, img, bar);                            // [PH][d][co][32 px]
                        tma_load_5d(dst + p.y_bytes, &map_x, tw * ND_W * 8, th * p.PH, img * 2, 0, 0, bar);         // [kw][l][plane][Ht][32][8]
                    } else tma_load_5d(dst, &map_dy, tw * 64, th * p.PH, 0, img, 0, bar);                 // [d][plane][PH][8 px][8]
                    if (DIRECT) {
                    } else if (p.fold > 1) tma_load_5d(dst + p.y_bytes, &map_x, tw * 64, th * p.PH, img * 2, 0, 0, bar);   // [kw][l][plane][Ht][8][8]
                    else tma_load_5d(dst + p.y_bytes, &map_x, tw * 64, th * p.PH, 0, img, 0, bar);                  // [l][plane][Ht][Wt][8]
                }
                if (++tw == p.tiles_w) { tw = 0; if (++th == p.tiles_h) { th = 0; ++img; } }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        const uint32_t idesc = make_idesc_f16(p.fmt, NM, ncols, !DIRECT, true);
        const bool el = elect_one();
        bool ok = true;
        for (int it = 0; it < n_steps && ok; ++it) {
            const int s = it % NF_STAGES;
            ok = warp_wait_bounded(full_bar + 8 * s, (it / NF_STAGES) & 1, status, ST_N_MMA);
            if (!ok) break;
            tc_fence_after_sync();
            if (el) {
                const uint32_t y0 = tiles_addr + s * p.stage_bytes, x0 = y0 + p.y_bytes;
                int kh = tap0 / p.KW, kw = tap0 - kh * p.KW;
                for (int tl = 0; tl < n_taps; ++tl) {
                    const uint32_t shift = (uint32_t)(kh * p.DH * p.Wt + kw * p.DW) * 16;
                    if (++kw == p.KW) { kw = 0; ++kh; }
                    if (DIRECT) {
                        const uint64_t ad = desc_rows64(y0), bd = desc_plain(x0 + shift, 128, p.plane_bytes);
                        uint32_t a_lo = (uint32_t)ad, b_lo = (uint32_t)bd;
                        const uint32_t a_row = (uint32_t)(p.nc * p.Co * ND_W * 2) >> 4;
                        for (int r = 0; r < p.PH; ++r) {
#pragma unroll
                            for (int j = 0; j < ND_W / 16; ++j)
                                mma_f16_ss_words(tmem_base + tl * ncols, a_lo + 2 * j, (uint32_t)(ad >> 32), b_lo + 16 * j, (uint32_t)(bd >> 32), idesc,
                                                 (it > 0 || r > 0 || j > 0) ? 1u : 0u);
                            a_lo += a_row;
                            b_lo += ND_W;
                        }
                        continue;
                    }
                    const uint64_t ad = desc_plain(y0, 128, p.PH * 128), bd = desc_plain(x0 + shift, p.Wt * 16, p.plane_bytes);
                    uint32_t a_lo = (uint32_t)ad, b_lo = (uint32_t)bd;
                    for (int kk = 0; kk < p.PH / 2; ++kk) {             // 16 pixels = two rows of the tile per MMA
                        mma_f16_ss_words(tmem_base + tl * ncols, a_lo, (uint32_t)(ad >> 32), b_lo, (uint32_t)(bd >> 32), idesc, (it > 0 || kk > 0) ? 1u : 0u);
                        a_lo += 256 >> 4;
                        b_lo += 2 * p.Wt;
                    }
                }
                mma_commit(empty_bar + 8 * s);
                if (it == n_steps - 1) mma_commit(tmem_full);
            }
            __syncwarp();
        }
        if (n_steps == 0 && lane == 0) mbar_arrive(tmem_full);
        __syncwarp();
    } else {
        const int q = warp & 3, tsel = (warp - 2) >> 2;                // two warps per lane quadrant share the taps
        const int seen = read_status(status);
        bool ok = mbar_wait_bounded(tmem_full, 0, status, ST_N_EPILOGUE);
        ok = warp_may_store(ok, seen);
        tc_fence_after_sync();
        if (ok && n_steps > 0) {
            const int m = q * 32 + lane;                                // row -> (d, plane, channel within the plane)
            const int chunk = m >> 3, d = DIRECT ? m / p.Co : chunk / p.y_planes, co = DIRECT ? m - d * p.Co : (chunk - d * p.y_planes) * 8 + (m & 7);
            const bool row_ok = d < p.nc && co < p.Co;
            const size_t comp_stride = (size_t)p.Co * p.Ci;
            for (int tl = tsel; tl < n_taps; tl += 2) {
                for (int c0 = 0; c0 < ncols; c0 += 16) {                // 16 columns = the channels of one input component (of one kw tap)
                    uint32_t v[16];
                    tmem_ld_32x32b_x16(tmem_base + ((uint32_t)(q * 32) << 16) + tl * ncols + c0, v);
                    tmem_ld_wait();
                    if (!row_ok) continue;
                    int kwf, l, tap;
                    if (p.fold_h > 1) { kwf = (c0 >> 4) / p.fold_h; l = 0; tap = ((tap0 + tl) * p.fold_h + (c0 >> 4) - kwf * p.fold_h) * p.fold + kwf; }
                    else { kwf = (c0 >> 4) / p.LKr; l = (c0 >> 4) - kwf * p.LKr; tap = (tap0 + tl) * p.fold + kwf; }
                    float* tap_base = dw32 + (size_t)tap * p.nc * comp_stride;
                    const float sgn = alg_negative(p.neg, l, d) ? -1.f : 1.f;
                    float* dst = tap_base + (size_t)alg_pair(p.ga, l, d) * comp_stride + (size_t)co * p.Ci;
#pragma unroll
                    for (int g4 = 0; g4 < 4; ++g4) {
                        if ((p.Ci & 3) == 0) {
                            if (4 * g4 < p.Ci)
                                red_add_f32x4(dst + 4 * g4, sgn * __uint_as_float(v[4 * g4]), sgn * __uint_as_float(v[4 * g4 + 1]),
                                              sgn * __uint_as_float(v[4 * g4 + 2]), sgn * __uint_as_float(v[4 * g4 + 3]));
                        } else {
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (4 * g4 + e < p.Ci) atomicAdd(dst + 4 * g4 + e, sgn * __uint_as_float(v[4 * g4 + e]));
                        }
                    }
                }
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, 512);
}

// scratch [tap][r][co][ci] fp32 -> dw [r][co][ci][tap] in the tensor type
template <typename T>
__global__ void unpack_narrow_filter_grad_kernel(const float* src, T* __restrict__ dw, int taps, size_t per_tap) {
    const size_t total = per_tap * taps;
    chain_wait();
    chain_next();
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        const int tap = (int)(idx % taps);
        DType<T>::store(dw + idx, ld_chained(src + (size_t)tap * per_tap + idx / taps));
    }
}
// s2d: scratch [staged tap][r][co][c' = (dy, dx, ci)] -> dw [r][co][ci][kh][kw]
template <typename T>
__global__ void unpack_narrow_filter_grad_s2d_kernel(const float* src, T* __restrict__ dw, int rows /*nc*Co*/, int Ci, int KH, int KW,
                                                     int KWe, int taps_e) {
    const size_t total = (size_t)rows * Ci * KH * KW;
    chain_wait();
    chain_next();
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        const int kw = (int)(idx % KW);
        size_t rest = idx / KW;
        const int kh = (int)(rest % KH); rest /= KH;
        const int ci = (int)(rest % Ci);
        const size_t row = rest / Ci;
        const int tap = (kh >> 1) * KWe + (kw >> 1), cp = ((kh & 1) * 2 + (kw & 1)) * Ci + ci;
        DType<T>::store(dw + idx, ld_chained(src + ((size_t)tap * rows + row) * (4 * Ci) + cp));
    }
}

// Stride-2 layers with at most 4 channels and no dilation run as stride-1 layers of a space-to-depth copy.
bool s2d_layer(const Geom& g) { return g.SH == 2 && g.SW == 2 && g.DH == 1 && g.DW == 1 && 4 * g.Ci <= 16; }

struct NPlan {
    int Cin, Cout, Hin, Win, Hout, Wout, pad_top, pad_left, ins_h, ins_w;
    int s2d, KHe, KWe, DHe, DWe;         // effective (staged) filter
    int wide;
    int LK, Hp, Wp, PH, Wt, Ht, tiles_w, tiles_h;
    uint32_t stage_bytes;
    size_t xp_bytes, w_bytes, smem;
};

NPlan make_nplan(Pass pass, const Geom& g, bool may_be_wide = true) {
    NPlan pl;
    if (pass == PASS_FWD) {
        pl.Cin = g.Ci; pl.Cout = g.Co; pl.Hin = g.H; pl.Win = g.W; pl.Hout = g.HO; pl.Wout = g.WO;
        pl.pad_top = g.PT; pl.pad_left = g.PL; pl.ins_h = pl.ins_w = 1;
    } else {
        pl.Cin = g.Co; pl.Cout = g.Ci; pl.Hin = g.HO; pl.Win = g.WO; pl.Hout = g.H; pl.Wout = g.W;
        pl.pad_top = (g.KH - 1) * g.DH - g.PT; pl.pad_left = (g.KW - 1) * g.DW - g.PL;
        pl.ins_h = g.SH; pl.ins_w = g.SW;
    }
    pl.LK = (pass == PASS_FWD && g.real_in) ? 1 : g.nc;
    pl.s2d = (pass == PASS_FWD && s2d_layer(g)) ? 1 : 0;
    pl.KHe = pl.s2d ? (g.KH + 1) / 2 : g.KH; pl.KWe = pl.s2d ? (g.KW + 1) / 2 : g.KW;
    pl.DHe = pl.s2d ? 1 : g.DH; pl.DWe = pl.s2d ? 1 : g.DW;
    if (pl.s2d) pl.Cin = 4 * g.Ci;
    const int rows = (pl.Hout + 31) / 32;                      // tile rows per image, then the smallest even height that covers them
    pl.PH = (((pl.Hout + rows - 1) / rows) + 1) & ~1;
    pl.tiles_h = (pl.Hout + pl.PH - 1) / pl.PH;
    pl.tiles_w = (pl.Wout + 7) / 8;
    pl.Wt = 8 + (pl.KWe - 1) * pl.DWe;
    pl.Ht = pl.PH + (pl.KHe - 1) * pl.DHe;
    pl.Hp = pl.tiles_h * pl.PH + (pl.KHe - 1) * pl.DHe;         // staged plane covers every halo tile completely
    pl.Wp = pl.tiles_w * 8 + (pl.KWe - 1) * pl.DWe;
    pl.stage_bytes = ((uint32_t)pl.Wt * pl.Ht * 32 + 1023) / 1024 * 1024;
    pl.xp_bytes = ((size_t)pl.LK * g.Nb * 2 * pl.Hp * pl.Wp * 16 + 1023) / 1024 * 1024;
    pl.w_bytes = ((size_t)pl.KHe * pl.KWe * pl.LK * NA_BYTES + 1023) / 1024 * 1024;
    pl.smem = 1024 + (size_t)pl.KHe * pl.KWe * pl.LK * NA_BYTES + (size_t)NB_STAGES * pl.stage_bytes + 256;
    // the wide form on the same staged copy (rows past it read as zeros through the tensor map)
    pl.wide = 0;
    const int rows16 = (pl.Hout + 15) / 16, ph16 = (((pl.Hout + rows16 - 1) / rows16) + 1) & ~1;
    const int wt16 = 16 + (pl.KWe - 1) * pl.DWe, ht16 = ph16 + (pl.KHe - 1) * pl.DHe;
    const uint32_t stage16 = ((uint32_t)wt16 * ht16 * 32 + 1023) / 1024 * 1024;
    const size_t smem16 = pl.smem - (size_t)NB_STAGES * pl.stage_bytes + (size_t)NB_STAGES * stage16;
    if (may_be_wide && pl.Wout % 16 == 0 && wt16 <= 32 && ht16 <= 255 && smem16 <= 226 * 1024) {
        pl.wide = 1;
        pl.PH = ph16; pl.Wt = wt16; pl.Ht = ht16; pl.stage_bytes = stage16; pl.smem = smem16;
        pl.tiles_h = (pl.Hout + ph16 - 1) / ph16; pl.tiles_w = pl.Wout / 16;
    }
    return pl;
}

}  // namespace

bool narrow_tc_supported(Pass pass, int dtype, int variant, const Geom& g) {
    if (pass != PASS_FWD && pass != PASS_BWD_DATA) return false;
    if (dtype != PCB_F16 && dtype != PCB_BF16) return false;
    if (variant != PCB_VARIANT_16_PRODUCT || g.w_io || g.dw_io) return false;
    if (g.real_in && pass != PASS_FWD) return false;
    if (g.H * g.W == 1) return false;
    if (pass == PASS_FWD && (g.SH != 1 || g.SW != 1) && !s2d_layer(g)) return false;   // backward-data is a stride-1 correlation of the zero-inserted dy
    if (pass == PASS_BWD_DATA && (g.SH > 2 || g.SW > 2)) return false;
    if (pass == PASS_BWD_DATA && ((g.KH - 1) * g.DH < g.PT || (g.KW - 1) * g.DW < g.PL)) return false;
    // (the tile of 8 pixels has to fit: outputs that are not 32-byte aligned take it. Where only the tile of 16 does -- quaternion 2x6, 19 rows,
    // 230 656 bytes of shared memory against 234 752 -- the layer is the general kernel's.)
    const NPlan pl = make_nplan(pass, g, false);
    if (pl.Cin > 16 || g.nc * pl.Cout > NM) return false;
    if (pl.Wt > 32 || pl.Ht > 255 || pl.smem > 226 * 1024) return false;
    if (pl.Wout < 8 || pl.Hout < 8) return false;                             // tiny images: the general kernel packs several per tile
    if (pl.xp_bytes > (size_t)8 << 30) return false;
    return true;
}

size_t narrow_tc_scratch_bytes(Pass pass, const Geom& g) {
    const NPlan pl = make_nplan(pass, g);
    return pl.xp_bytes + pl.w_bytes;
}

int narrow_tc_launch(Pass pass, int dtype, const Geom& g, const void* w, const void* act, const void* bias, void* out, void* scratch,
                     int* status, cudaStream_t stream, StatusClear* sc) {
    const int fmt = dtype == PCB_F16 ? 0 : 1;
    const NPlan pl = make_nplan(pass, g, reinterpret_cast<uintptr_t>(out) % 32 == 0);
    const int taps = pl.KHe * pl.KWe, Kp = pl.LK * 16;
    const int src_c = pl.s2d ? g.Ci : pl.Cin;            // channels of the tensor being staged
    uint8_t* xp = static_cast<uint8_t*>(scratch);
    uint8_t* wexp = xp + pl.xp_bytes;
    bool chain = false;
    {
        PlanarPrologue pro;
        add_planar_job(pro, act, xp, pl.LK * g.Nb, src_c, pl.Hin, pl.Win, pl.Hp, pl.Wp, 2, pl.pad_top, pl.pad_left, pl.ins_h, pl.ins_w, pl.s2d);
        pro.filter = PlanarFilterJob{(const uint16_t*)w, (uint16_t*)wexp, g.Co, g.Ci, taps, Kp, pass == PASS_BWD_DATA ? 1 : 0, g.nc, g.ga, g.neg,
                                     pl.s2d, g.KH, g.KW, pl.KWe};
        pro.filter_blocks = grid_cap((size_t)taps * NM * Kp, NP_THREADS, 8);
        const int rc = launch_prologue(pro, sc, stream, &chain);
        if (rc != PCB_OK) return rc;
    }
    NParams p;
    p.Nb = g.Nb; p.Cout = pl.Cout; p.Mvalid = g.nc * pl.Cout; p.HO = pl.Hout; p.WO = pl.Wout;
    p.KH = pl.KHe; p.KW = pl.KWe; p.DH = pl.DHe; p.DW = pl.DWe;
    p.PH = pl.PH; p.Wt = pl.Wt; p.Ht = pl.Ht; p.tiles_w = pl.tiles_w; p.tiles_h = pl.tiles_h;
    p.LK = pl.LK; p.taps = taps; p.fmt = fmt; p.has_bias = (pass == PASS_FWD && g.has_bias) ? 1 : 0;
    p.stage_bytes = pl.stage_bytes; p.plane_bytes = (uint32_t)pl.Ht * pl.Wt * 16;
    p.store_vec = 1;
    while (p.store_vec < 8 && pl.Wout % (p.store_vec * 2) == 0 && (reinterpret_cast<uintptr_t>(out) % (size_t)(p.store_vec * 4)) == 0) p.store_vec *= 2;

    const CUtensorMapDataType dt = fmt == 0 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    alignas(64) CUtensorMap map_w, map_x;
    {   // Wexp[tap][k / 8][128][8] seen as (32 rows x 8, 4, k / 8, tap); box = 2 planes of 128 rows
        const cuuint64_t dims[4] = {256, NM / 32, (cuuint64_t)Kp / 8, (cuuint64_t)taps};
        const cuuint64_t strides[3] = {512, (cuuint64_t)NM * 16, (cuuint64_t)(Kp / 8) * NM * 16};
        const cuuint32_t box[4] = {256, NM / 32, 2, 1};
        const int rc = make_tensor_map(&map_w, dt, wexp, 4, dims, strides, box, nullptr, CU_TENSOR_MAP_SWIZZLE_NONE, "narrow filters");
        if (rc != PCB_OK) return rc;
    }
    {   // xp[comp][img][plane][hp][wp][8] seen as (wp x 8, hp, plane, img, comp); box = the halo tile of one component
        const cuuint64_t dims[5] = {(cuuint64_t)pl.Wp * 8, (cuuint64_t)pl.Hp, 2, (cuuint64_t)g.Nb, (cuuint64_t)pl.LK};
        const cuuint64_t strides[4] = {(cuuint64_t)pl.Wp * 16, (cuuint64_t)pl.Hp * pl.Wp * 16, (cuuint64_t)2 * pl.Hp * pl.Wp * 16,
                                       (cuuint64_t)g.Nb * 2 * pl.Hp * pl.Wp * 16};
        const cuuint32_t box[5] = {(cuuint32_t)pl.Wt * 8, (cuuint32_t)pl.Ht, 2, 1, 1};
        const int rc = make_tensor_map(&map_x, dt, xp, 5, dims, strides, box, nullptr, CU_TENSOR_MAP_SWIZZLE_NONE, "narrow activations");
        if (rc != PCB_OK) return rc;
    }
    const int n_tiles = pl.tiles_w * pl.tiles_h * g.Nb;
    const int grid = n_tiles < sm_count() ? n_tiles : sm_count();
    // (the largest filter matrices leave no room for the row buffers: those layers store from the registers)
    p.rows_epi = p.store_vec < 8 && pl.smem + N_EPI_WARPS * EPI_ROWS_BYTES <= 227 * 1024;
    size_t smem = pl.smem + (p.rows_epi ? N_EPI_WARPS * EPI_ROWS_BYTES : 0);
    if (smem < ONE_CTA_SMEM) smem = ONE_CTA_SMEM;
    auto* kernel = pl.wide ? qconv_narrow_tc_kernel<true> : qconv_narrow_tc_kernel<false>;
    PCB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_CTA_SMEM));
    PCB_CUDA_TRY(launch_chained_if(chain, kernel, grid, NW_THREADS, smem, stream, map_w, map_x, p, (const uint16_t*)bias, (uint16_t*)out, status));
    PCB_CUDA_TRY(cudaGetLastError());
    return PCB_OK;
}

namespace {

struct NFPlan {
    int s2d, KHe, KWe, DHe, DWe, Cie;    // effective (staged) filter and channels
    int LK, PH, Wt, Ht, tiles_w, tiles_h, Hp, Wp, HOp, WOp, y_planes, taps_per_group, n_groups;
    int direct_ph;                       // tile height of the DIRECT form (0: not for this layer)
    int fold, fold_h, LKe, taps;         // kw / kh taps folded into one MMA (1 = none), columns / 16 of one MMA, MMAs per 16 pixels
    uint32_t y_bytes, x_bytes, stage_bytes;
    size_t xp_bytes, dyp_bytes, acc_bytes, smem;
};

NFPlan make_nfplan(const Geom& g) {
    NFPlan f;
    f.LK = g.real_in ? 1 : g.nc;
    f.s2d = s2d_layer(g) ? 1 : 0;
    f.KHe = f.s2d ? (g.KH + 1) / 2 : g.KH; f.KWe = f.s2d ? (g.KW + 1) / 2 : g.KW;
    f.DHe = f.s2d ? 1 : g.DH; f.DWe = f.s2d ? 1 : g.DW;
    f.Cie = f.s2d ? 4 * g.Ci : g.Ci;
    // the staged copies (shared with the forward pass, see forward_keeps_staged_input) follow the standard tile height
    const int rows = (g.HO + 31) / 32;
    const int ph_std = (((g.HO + rows - 1) / rows) + 1) & ~1;
    f.tiles_w = (g.WO + 7) / 8;
    f.HOp = ((g.HO + ph_std - 1) / ph_std) * ph_std; f.WOp = f.tiles_w * 8;
    f.Hp = f.HOp + (f.KHe - 1) * f.DHe; f.Wp = f.WOp + (f.KWe - 1) * f.DWe;
    f.y_planes = (g.Co + 7) / 8;
    // folded form: all kw taps of a filter row in the columns of one MMA, if those fit one MMA (N <= 256)
    f.fold = (f.KWe > 1 && f.KWe * f.LK * 16 <= 256) ? f.KWe : 1;
    // ... and the filter rows too for a one-component x (the tensor map has a dimension to spare)
    f.fold_h = (f.fold > 1 && f.LK == 1 && f.KHe > 1 && f.KHe * f.KWe * 16 <= 256) ? f.KHe : 1;
    // From four filter rows up only half of them: the box holds every folded row and column once more, 80 KB per 8 x 16 pixels at
    // 4 x 4 taps, and the kernel is bound by that traffic from L2 (117 us for the 7x7/2 stem at batch 128). Two of the four rows in the
    // columns of an MMA and the other two as a shifted start address move half of it.
    if (f.fold_h >= 4 && f.fold_h % 2 == 0) f.fold_h /= 2;
    f.LKe = f.LK * f.fold * f.fold_h;
    f.taps = f.fold_h > 1 ? f.KHe / f.fold_h : (f.fold > 1 ? f.KHe : f.KHe * f.KWe);
    f.Wt = f.fold > 1 ? 8 : 8 + (f.KWe - 1) * f.DWe;
    const int ncols = f.LKe * 16;
    // as many taps per group as the 512 accumulator columns hold whole (ncols <= 256), spread evenly over the fewest groups; three taps
    // of 192 columns -- five or seven rows of a 3-wide filter -- would need 576 columns
    const int fit = 512 / ncols;
    f.n_groups = (f.taps + fit - 1) / fit;
    f.taps_per_group = (f.taps + f.n_groups - 1) / f.n_groups;
    f.n_groups = (f.taps + f.taps_per_group - 1) / f.taps_per_group;
    // the kernel's own tile height: the standard one, lowered until two stages fit the shared memory (rows past the staged
    // planes read as zeros through the tensor maps)
    for (int r = rows;; ++r) {
        f.PH = (((g.HO + r - 1) / r) + 1) & ~1;
        f.tiles_h = (g.HO + f.PH - 1) / f.PH;
        f.Ht = f.PH + (f.KHe - f.fold_h) * f.DHe;                   // (all rows folded: no halo)
        f.y_bytes = (uint32_t)g.nc * f.y_planes * f.PH * 128;
        f.x_bytes = (uint32_t)f.LKe * 2 * f.Ht * f.Wt * 16;
        f.stage_bytes = (f.y_bytes + f.x_bytes + 1023) / 1024 * 1024;
        // the M = 128 operand spans 16 chunks of PH * 128 bytes from the start of a dy tile
        const size_t slack = (size_t)16 * f.PH * 128;
        f.smem = 1024 + 1024 + (size_t)NF_STAGES * f.stage_bytes + slack;
        if (f.smem <= 226 * 1024 || f.PH <= 2) break;
    }
    // the DIRECT form: the tile height that two stages leave room for, and where 32-pixel tiles waste little of the rows
    f.direct_ph = 0;
    const int rows_m = g.nc * g.Co;
    if (f.fold > 1 && g.plain && g.WO % 8 == 0 && rows_m % 8 == 0 && rows_m <= NM && g.Co <= 256 && 4 * round_up(g.WO, ND_W) <= 5 * g.WO) {
        const uint32_t y_row = (uint32_t)rows_m * ND_W * 2, x_row = (uint32_t)f.LKe * 2 * ND_W * 16, halo = (f.KHe - f.fold_h) * f.DHe;
        // (the M = 128 operand reads up to 8 KB from the start of a row of dy)
        const int fit = ((226 * 1024 - 2048 - 8192) / NF_STAGES / 1024 * 1024 - (int)(halo * x_row)) / (int)(y_row + x_row);
        if (fit >= 2) {
            const int r = (g.HO + fit - 1) / fit;
            f.direct_ph = (g.HO + r - 1) / r;
        }
    }
    f.xp_bytes = ((size_t)f.LK * g.Nb * 2 * f.Hp * f.Wp * 16 + 1023) / 1024 * 1024;
    f.dyp_bytes = ((size_t)g.nc * g.Nb * f.y_planes * f.HOp * f.WOp * 16 + 1023) / 1024 * 1024;
    f.acc_bytes = ((size_t)g.nc * g.Co * f.Cie * f.KHe * f.KWe * sizeof(float) + 1023) / 1024 * 1024;
    return f;
}

// Number of slices to cut each of `items` work items into when every CTA occupies a whole SM: the CTAs must fill
// one, two or three rounds of the machine as exactly as possible (one CTA more than a round costs a whole round). A further
// round also costs every CTA's fixed part again (tensor-memory allocation, pipeline fill, the atomic fold of its
// accumulator), so it has to fill the machine at least 5 % better to be taken. (A step of
// these kernels takes too different times for the rule by clocks, split_count: 24 -> 16 channels, 5x5, 49 x 52, batch 26 256.8 us, by that rule
// 258.3.)
inline int fill_rounds(int items, int sms) {
    int best = 1;
    double best_util = 0.0;
    for (int waves = 1; waves <= 3; ++waves) {
        const int splits = waves * sms / items;
        if (splits < 1) continue;
        const double util = (double)items * splits / ((double)waves * sms);
        if (util > best_util + (best_util > 0.0 ? 0.05 : 0.0)) { best_util = util; best = splits; }
    }
    return best;
}
}  // namespace

bool narrow_filter_tc_supported(int dtype, int variant, const Geom& g) {
    if (dtype != PCB_F16 && dtype != PCB_BF16) return false;
    if (variant != PCB_VARIANT_16_PRODUCT || g.w_io || g.dw_io) return false;
    if (g.H * g.W == 1 || ((g.SH != 1 || g.SW != 1) && !s2d_layer(g))) return false;
    if ((s2d_layer(g) ? 4 * g.Ci : g.Ci) > 16 || g.nc * ((g.Co + 7) / 8) > 16) return false;   // x: two planes; dy: at most 16 chunks of 8 rows
    if (g.WO < 8 || g.HO < 8) return false;
    const NFPlan f = make_nfplan(g);
    if (f.Wt > 32 || f.Ht > 255 || f.smem > 226 * 1024) return false;
    if (f.xp_bytes + f.dyp_bytes > (size_t)12 << 30) return false;
    return true;
}

size_t narrow_filter_tc_scratch_bytes(const Geom& g) {
    const NFPlan f = make_nfplan(g);
    return f.xp_bytes + f.dyp_bytes + f.acc_bytes;
}

bool narrow_tc_staged_dy_view(const Geom& g, StagedView* view, size_t* bytes) {
    if (g.SH != 1 || g.SW != 1) return false;                   // strided layers: backward-data reads a zero-inserted copy
    const NPlan pl = make_nplan(PASS_BWD_DATA, g);
    view->Hp = pl.Hp; view->Wp = pl.Wp; view->pad_top = pl.pad_top; view->pad_left = pl.pad_left;
    *bytes = pl.xp_bytes;
    return pl.pad_top >= 0 && pl.pad_left >= 0;
}

int narrow_filter_tc_launch(int dtype, const Geom& g, const void* dy, const void* x, void* dw, void* scratch, int* status, cudaStream_t stream,
                            const void* kept_x, const StagedView* kept_dy, StatusClear* sc) {
    const int fmt = dtype == PCB_F16 ? 0 : 1;
    NFPlan f = make_nfplan(g);
    // dy in place, unless backward-data has staged it
    const bool direct = !kept_dy && f.direct_ph > 0 && (reinterpret_cast<uintptr_t>(dy) & 15u) == 0;
    if (direct) {
        f.PH = f.direct_ph; f.tiles_h = (g.HO + f.PH - 1) / f.PH; f.tiles_w = (g.WO + ND_W - 1) / ND_W;
        f.Ht = f.PH + (f.KHe - f.fold_h) * f.DHe; f.Wt = ND_W;
        f.y_bytes = (uint32_t)g.nc * g.Co * ND_W * 2 * f.PH;
        f.x_bytes = (uint32_t)f.LKe * 2 * f.Ht * ND_W * 16;
        f.stage_bytes = (f.y_bytes + f.x_bytes + 1023) / 1024 * 1024;
        f.smem = 1024 + 1024 + (size_t)NF_STAGES * f.stage_bytes + 8192;
    }
    const int taps = f.KHe * f.KWe;                 // filter taps of the staged problem (the folded form issues KHe MMAs per 16 pixels)
    // the forward pass of a narrow layer stages x exactly as this one does: a copy it kept is read in place
    uint8_t* xp = kept_x ? static_cast<uint8_t*>(const_cast<void*>(kept_x)) : static_cast<uint8_t*>(scratch);
    uint8_t* dyp = static_cast<uint8_t*>(scratch) + f.xp_bytes;
    float* acc = reinterpret_cast<float*>(dyp + f.dyp_bytes);
    bool chain = false;
    {
        // x: padded planar copy (space-to-depth for the stride-2 stem); dy: planar copy rounded up to whole tiles
        PlanarPrologue pro;
        if (!kept_x) add_planar_job(pro, x, xp, f.LK * g.Nb, g.Ci, g.H, g.W, f.Hp, f.Wp, 2, g.PT, g.PL, 1, 1, f.s2d);
        if (!kept_dy && !direct) add_planar_job(pro, dy, dyp, g.nc * g.Nb, g.Co, g.HO, g.WO, f.HOp, f.WOp, f.y_planes, 0, 0, 1, 1, 0);
        pro.zero = reinterpret_cast<uint4*>(acc);
        pro.zero_units = (unsigned)(f.acc_bytes / 16);
        pro.zero_blocks = grid_cap(pro.zero_units, 4 * NP_THREADS, 1);
        const int rc = launch_prologue(pro, sc, stream, &chain);
        if (rc != PCB_OK) return rc;
    }
    NFParams p;
    p.Nb = g.Nb; p.Co = g.Co; p.Ci = f.Cie; p.nc = g.nc; p.ga = g.ga; p.neg = g.neg;
    p.KH = f.KHe; p.KW = f.fold > 1 ? 1 : f.KWe; p.DH = f.DHe * f.fold_h; p.DW = f.DWe;
    p.PH = f.PH; p.Wt = f.Wt; p.Ht = f.Ht; p.tiles_w = f.tiles_w; p.tiles_h = f.tiles_h;
    p.LK = f.LKe; p.LKr = f.LK; p.fold = f.fold; p.fold_h = f.fold_h;
    p.taps = f.taps; p.taps_per_group = f.taps_per_group; p.n_groups = f.n_groups; p.y_planes = f.y_planes;
    p.fmt = fmt; p.y_bytes = f.y_bytes; p.x_bytes = f.x_bytes; p.stage_bytes = f.stage_bytes; p.plane_bytes = (uint32_t)f.Ht * f.Wt * 16;
    p.steps_total = f.tiles_w * f.tiles_h * g.Nb;
    int splits = fill_rounds(f.n_groups, sm_count());
    if (splits > p.steps_total) splits = p.steps_total;
    if (splits < 1) splits = 1;
    p.steps_per_split = (p.steps_total + splits - 1) / splits;
    splits = (p.steps_total + p.steps_per_split - 1) / p.steps_per_split;
    int grid = f.n_groups * splits;
    p.uneven = 0;
    const int last_taps = f.taps - (f.n_groups - 1) * f.taps_per_group;
    if (f.n_groups > 1 && f.n_groups <= NF_MAX_GROUPS && last_taps < f.taps_per_group) {
        // CTA shares in proportion to the taps of each group (one wave of CTAs)
        const int sms = sm_count();
        int begin = 0;
        for (int gi = 0; gi < f.n_groups; ++gi) {
            const int taps_g = gi + 1 < f.n_groups ? f.taps_per_group : last_taps;
            int share = (int)((long long)sms * taps_g / f.taps);
            if (share < 1) share = 1;
            if (share > p.steps_total) share = p.steps_total;
            p.group_steps[gi] = (p.steps_total + share - 1) / share;
            share = (p.steps_total + p.group_steps[gi] - 1) / p.group_steps[gi];
            p.cta_begin[gi] = begin;
            begin += share;
        }
        p.cta_begin[f.n_groups] = begin;
        p.uneven = 1;
        grid = begin;
    }

    const CUtensorMapDataType dt = fmt == 0 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    alignas(64) CUtensorMap map_dy, map_x;
    {   // dyp[d][img][plane][HOp][WOp][8] seen as (w x 8, h, plane, img, d); box = the tile of all components
        const cuuint64_t dims[5] = {(cuuint64_t)f.WOp * 8, (cuuint64_t)f.HOp, (cuuint64_t)f.y_planes, (cuuint64_t)g.Nb, (cuuint64_t)g.nc};
        const cuuint64_t strides[4] = {(cuuint64_t)f.WOp * 16, (cuuint64_t)f.HOp * f.WOp * 16, (cuuint64_t)f.y_planes * f.HOp * f.WOp * 16,
                                       (cuuint64_t)g.Nb * f.y_planes * f.HOp * f.WOp * 16};
        const cuuint32_t box[5] = {64, (cuuint32_t)f.PH, (cuuint32_t)f.y_planes, 1, (cuuint32_t)g.nc};
        int rc;
        if (direct) {   // (w, co, d, h, image) of the caller's tensor
            const size_t plane = (size_t)g.HO * g.WO * 2;
            const cuuint64_t ddims[5] = {(cuuint64_t)g.WO, (cuuint64_t)g.Co, (cuuint64_t)g.nc, (cuuint64_t)g.HO, (cuuint64_t)g.Nb};
            const cuuint64_t dstrides[4] = {plane, (cuuint64_t)g.Nb * g.Co * plane, (cuuint64_t)g.WO * 2, (cuuint64_t)g.Co * plane};
            const cuuint32_t dbox[5] = {ND_W, (cuuint32_t)g.Co, (cuuint32_t)g.nc, (cuuint32_t)f.PH, 1};
            rc = make_tensor_map(&map_dy, dt, dy, 5, ddims, dstrides, dbox, nullptr, CU_TENSOR_MAP_SWIZZLE_64B, "narrow dy (in place)");
        } else if (kept_dy) {
            // the copy backward-data staged: [d][img][2 planes][Hp][Wp][8] with pixel (0, 0) at (pad_top, pad_left); only the
            // HO x WO pixels are inside the map, so whatever a tile box takes beyond them reads as zeros
            const size_t plane = (size_t)kept_dy->Hp * kept_dy->Wp * 16;
            const cuuint64_t kdims[5] = {(cuuint64_t)g.WO * 8, (cuuint64_t)g.HO, (cuuint64_t)f.y_planes, (cuuint64_t)g.Nb, (cuuint64_t)g.nc};
            const cuuint64_t kstrides[4] = {(cuuint64_t)kept_dy->Wp * 16, plane, 2 * plane, (cuuint64_t)g.Nb * 2 * plane};
            uint8_t* origin = static_cast<uint8_t*>(const_cast<void*>(kept_dy->base)) + ((size_t)kept_dy->pad_top * kept_dy->Wp + kept_dy->pad_left) * 16;
            rc = make_tensor_map(&map_dy, dt, origin, 5, kdims, kstrides, box, nullptr, CU_TENSOR_MAP_SWIZZLE_NONE, "narrow dy (shared)");
        } else {
            rc = make_tensor_map(&map_dy, dt, dyp, 5, dims, strides, box, nullptr, CU_TENSOR_MAP_SWIZZLE_NONE, "narrow dy");
        }
        if (rc != PCB_OK) return rc;
    }
    if (f.fold > 1) {
        // the same copy with the kw tap as a dimension of its own, one pixel (16 bytes) apart: (w x 8, h, image and plane, l, kw);
        // box = the tile, 8 pixels wide, of every component at every kw shift. The first extent stops short of the halo columns so
        // that the shifted views stay inside their rows.
        // With the filter rows folded as well the fourth dimension is kh (one staged row apart) instead of the component, and
        // the second extent stops short of the halo rows for the same reason.
        const size_t plane = (size_t)f.Hp * f.Wp * 16;
        const bool fh = f.fold_h > 1;
        const cuuint64_t dims[5] = {(cuuint64_t)f.WOp * 8, (cuuint64_t)(f.Hp - (f.fold_h - 1) * f.DHe), (cuuint64_t)2 * g.Nb, (cuuint64_t)(fh ? f.fold_h : f.LK),
                                    (cuuint64_t)f.fold};
        const cuuint64_t strides[4] = {(cuuint64_t)f.Wp * 16, plane, fh ? (cuuint64_t)f.DHe * f.Wp * 16 : (cuuint64_t)g.Nb * 2 * plane,
                                       (cuuint64_t)f.DWe * 16};
        const cuuint32_t box[5] = {(cuuint32_t)(direct ? ND_W * 8 : 64), (cuuint32_t)f.Ht, 2, (cuuint32_t)(fh ? f.fold_h : f.LK), (cuuint32_t)f.fold};
        const int rc = make_tensor_map(&map_x, dt, xp, 5, dims, strides, box, nullptr, CU_TENSOR_MAP_SWIZZLE_NONE, "narrow x (folded)");
        if (rc != PCB_OK) return rc;
    } else {   // xp[l][img][plane][Hp][Wp][8]; box = the halo tile of all components
        const cuuint64_t dims[5] = {(cuuint64_t)f.Wp * 8, (cuuint64_t)f.Hp, 2, (cuuint64_t)g.Nb, (cuuint64_t)f.LK};
        const cuuint64_t strides[4] = {(cuuint64_t)f.Wp * 16, (cuuint64_t)f.Hp * f.Wp * 16, (cuuint64_t)2 * f.Hp * f.Wp * 16,
                                       (cuuint64_t)g.Nb * 2 * f.Hp * f.Wp * 16};
        const cuuint32_t box[5] = {(cuuint32_t)f.Wt * 8, (cuuint32_t)f.Ht, 2, 1, (cuuint32_t)f.LK};
        const int rc = make_tensor_map(&map_x, dt, xp, 5, dims, strides, box, nullptr, CU_TENSOR_MAP_SWIZZLE_NONE, "narrow x");
        if (rc != PCB_OK) return rc;
    }
    const size_t fsmem = f.smem < ONE_CTA_SMEM ? ONE_CTA_SMEM : f.smem;
    auto* kernel = direct ? qconv_narrow_filter_tc_kernel<true> : qconv_narrow_filter_tc_kernel<false>;
    PCB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_CTA_SMEM));
    PCB_CUDA_TRY(launch_chained_if(chain, kernel, grid, N_THREADS, fsmem, stream, map_dy, map_x, p, acc, status));
    PCB_CUDA_TRY(cudaGetLastError());
    const size_t per_tap = (size_t)g.nc * g.Co * g.Ci;
    const int blocks = grid_cap(per_tap * g.KH * g.KW, 256, 16);
    if (f.s2d) {
        if (fmt == 0) PCB_CUDA_TRY(launch_chained(unpack_narrow_filter_grad_s2d_kernel<__half>, blocks, 256, 0, stream, acc, (__half*)dw, g.nc * g.Co, g.Ci, g.KH, g.KW, f.KWe, taps));
        else PCB_CUDA_TRY(launch_chained(unpack_narrow_filter_grad_s2d_kernel<__nv_bfloat16>, blocks, 256, 0, stream, acc, (__nv_bfloat16*)dw, g.nc * g.Co, g.Ci, g.KH, g.KW, f.KWe, taps));
    } else if (fmt == 0) PCB_CUDA_TRY(launch_chained(unpack_narrow_filter_grad_kernel<__half>, blocks, 256, 0, stream, acc, (__half*)dw, taps, per_tap));
    else PCB_CUDA_TRY(launch_chained(unpack_narrow_filter_grad_kernel<__nv_bfloat16>, blocks, 256, 0, stream, acc, (__nv_bfloat16*)dw, taps, per_tap));
    PCB_CUDA_TRY(cudaGetLastError());
    return PCB_OK;
}

}  // namespace pcb
