// Interface of the tcgen05 (tensor-core) kernel family towards the C ABI dispatcher.
#pragma once
#include "common.cuh"

namespace pcb {

// True when a tensor-core kernel exists for this pass / dtype / variant / geometry.
bool tensor_path_supported(Pass pass, int dtype, int variant, const Geom& g);
// Scratch bytes (beyond the workspace header) the tensor-core kernel of this problem needs.
size_t tensor_scratch_bytes(Pass pass, int dtype, int variant, int engine, const Geom& g);
// Operand roles as for simt_launch. `status` is the device status word of the workspace header.
// A staged tensor that another pass already made: where it lies and how it is padded (copies for the narrow kernels are).
struct StagedView {
    const void* base = nullptr;
    int Hp = 0, Wp = 0, pad_top = 0, pad_left = 0;   // padded plane and the position of pixel (0, 0) inside it
};
// What a filter-gradient pass may take over from other passes instead of staging it again:
// `kept_x`: the staged copy of x that the forward call of the same layer left in ITS workspace scratch (see
//           forward_keeps_staged_input);
// `dy`:     the copy of dy that the backward-data pass of the same call staged (see backward_shares_staged_dy);
// `scratch_offset`: bytes of the workspace scratch to leave alone (they hold that copy).
struct PassExtras {
    const void* kept_x = nullptr;
    StagedView dy;
    size_t scratch_offset = 0;
};
// The reset of the device status word that an API call owes its workspace before its first kernel. Launches that have a kernel in
// front of the waiting ones let that kernel do it; everything else calls now() first.
int clear_status_word(int* word, cudaStream_t stream);    // defined in api.cu
struct StatusClear {
    int* word = nullptr;
    bool pending = false;
    int now(cudaStream_t stream) {
        if (!pending) return PCB_OK;
        pending = false;
        return clear_status_word(word, stream);
    }
};
// `sc` (may be null: nothing is owed) is settled before any kernel of the pass can wait.
int tensor_launch(Pass pass, int dtype, int variant, const Geom& g, const void* a, const void* b, const void* bias,
                  void* out, float* scratch, int* status, cudaStream_t stream, const PassExtras* extras = nullptr, StatusClear* sc = nullptr);
// True when the backward-data pass of this layer stages dy (at the start of its scratch, `bytes` long) in a layout its
// filter gradient can read through a tensor map: the narrow pair of kernels (stride 1), or the general pair with one channel block per
// component (stride 1, or 2 x 2 by pixel classes). `view` receives the padded geometry (its base is left null).
bool backward_shares_staged_dy(int dtype, int variant, const Geom& g, StagedView* view, size_t* bytes);
// True when the forward pass of this layer stages x, at the start of its scratch, in exactly the layout its filter
// gradient reads: a narrow forward with a narrow filter gradient, or the general pair with one channel block per component.
bool forward_keeps_staged_input(int dtype, int variant, const Geom& g);

// A pointwise layer of NCHW tensors is the same layer on images one pixel tall: the runs of pixels that tiles load and store are then as long
// as the plane, and aligned where the plane is a round number of pixels although its rows are not. Pointwise, forward or
// forward + backward, us: fp16 24 -> 56, 36 x 36, batch 48 27.1 -> 19.8; fp16 48 -> 48, 46 x 41, batch 48 179 -> 155; bf16 24 -> 40, 63 x 71,
// batch 88 178 -> 148; fp32 16 -> 71, 25 x 25, batch 26 36 -> 30.
inline Geom flat_pixels(const Geom& g) {
    Geom s = g;
    if (g.KH == 1 && g.KW == 1 && g.SH == 1 && g.SW == 1 && g.PT == 0 && g.PL == 0 && g.HO == g.H && g.WO == g.W && g.H > 1 && g.plain &&
        (long long)g.H * g.W <= 32768) {
        s.W = s.WO = g.H * g.W; s.H = s.HO = 1;
        s.xh = s.yh = s.W;
    }
    return s;
}

// Persistent TMA-fed kernel for wide pointwise layers (forward and backward-data); see pointwise_tc.cu.
bool pointwise_tc_supported(Pass pass, int dtype, int variant, const Geom& g);
int pointwise_tc_launch(Pass pass, int dtype, const Geom& g, const void* w, const void* act, const void* bias, void* out,
                        int* status, cudaStream_t stream);

// The forward kernel on pairs of SMs (cta_group::2 MMAs) for layers with a multiple of 256 output channels; see pointwise2_tc.cu.
bool pointwise_pair_tc_supported(Pass pass, int dtype, int variant, const Geom& g);
int pointwise_pair_tc_launch(int dtype, const Geom& g, const void* w, const void* x, const void* bias, void* y, int* status, cudaStream_t stream);
bool pointwise_filter_pair_tc_supported(const Geom& g);
int pointwise_filter_pair_tc_launch(int fmt, const Geom& g, const void* dy, const void* x, float* scratch, int* status, cudaStream_t stream);

bool pointwise_filter_tc_supported(int dtype, int variant, const Geom& g);
int pointwise_filter_tc_launch(int dtype, const Geom& g, const void* dy, const void* x, void* dw, float* scratch, int* status,
                               cudaStream_t stream);

// The factorised 8-product form of pointwise layers (all three passes) with the lane sums formed in shared memory and the
// recombination in the epilogue; see pointwise8_tc.cu.
bool pointwise8_tc_supported(Pass pass, int dtype, int variant, const Geom& g);
size_t pointwise8_tc_scratch_bytes(Pass pass, const Geom& g);
int pointwise8_tc_launch(Pass pass, int dtype, const Geom& g, const void* a, const void* b, const void* bias, void* out,
                         float* scratch, int* status, cudaStream_t stream);

// General implicit-GEMM convolution (any taps / stride <= 2 / padding) on staged operands; see conv_tc.cu.
bool conv_tc_supported(Pass pass, int dtype, int variant, const Geom& g);
size_t conv_tc_scratch_bytes(Pass pass, const Geom& g);
// Backward-data of a layer with strides 2 x 2 whose pixel classes the kernel takes in one launch (no zero insertion).
bool conv_tc_dual_classes(Pass pass, const Geom& g);
int conv_tc_launch(Pass pass, int dtype, const Geom& g, const void* w, const void* act, const void* bias, void* out,
                   void* scratch, int* status, cudaStream_t stream, StatusClear* sc = nullptr);

bool conv_filter_tc_supported(int dtype, int variant, const Geom& g);
size_t conv_filter_tc_scratch_bytes(const Geom& g);
int conv_filter_tc_launch(int dtype, const Geom& g, const void* dy, const void* x, void* dw, void* scratch, int* status,
                          cudaStream_t stream, const void* kept_x = nullptr, const StagedView* kept_dy = nullptr, StatusClear* sc = nullptr);
// Geometry of the copy of dy that the general backward-data kernel stages; false when it inserts zeros (strided layers) or
// the filter gradient would block its channels.
bool conv_filter_tc_flat(const Geom& g);
bool conv_tc_staged_dy_view(const Geom& g, StagedView* view, size_t* bytes);
// The filter gradient stages x as [component][image][h][w][channels], the layout of the forward pass.
bool conv_filter_tc_stages_like_forward(const Geom& g);

// Narrow layers (<= 16 reduced channels, stride-1 correlation): halo tiles in shared memory serve every tap; see narrow_tc.cu.
bool narrow_tc_supported(Pass pass, int dtype, int variant, const Geom& g);
size_t narrow_tc_scratch_bytes(Pass pass, const Geom& g);
int narrow_tc_launch(Pass pass, int dtype, const Geom& g, const void* w, const void* act, const void* bias, void* out, void* scratch,
                     int* status, cudaStream_t stream, StatusClear* sc = nullptr);

bool narrow_filter_tc_supported(int dtype, int variant, const Geom& g);
size_t narrow_filter_tc_scratch_bytes(const Geom& g);
int narrow_filter_tc_launch(int dtype, const Geom& g, const void* dy, const void* x, void* dw, void* scratch, int* status, cudaStream_t stream,
                            const void* kept_x = nullptr, const StagedView* kept_dy = nullptr, StatusClear* sc = nullptr);
bool narrow_tc_staged_dy_view(const Geom& g, StagedView* view, size_t* bytes);

// fp32 tensors on the tensor cores with error-compensated TF32 (convolution and dense); see conv_tf32.cu.
bool conv_tf32_supported(Pass pass, int dtype, int variant, const Geom& g);
size_t conv_tf32_scratch_bytes(Pass pass, const Geom& g);
int conv_tf32_launch(Pass pass, const Geom& g, const void* a, const void* b, const void* bias, void* out, void* scratch, int* status,
                     cudaStream_t stream, StatusClear* sc = nullptr);

// Dense layers of quaternions without staging, both gradients in one launch; see qgemm_tc.cu. Any feature counts; every
// tensor 16-byte aligned. Nothing but the status word of the workspace is used.
bool dense_tc_supported(int dtype, int variant, const Geom& g);
// Which kernels a call takes of those: all of its results, dw alone (dx by the staged kernels), or none -- where the staged kernels are
// faster, where the launch cannot be cut to fit the machine, or where it would not leave the SMs free that it should.
enum DenseRoute { DENSE_STAGED, DENSE_DIRECT, DENSE_FILTER_DIRECT };
DenseRoute dense_tc_route(int dtype, const Geom& g, bool backward, bool need_dx);
// (`sc`: the pending reset of the status word, done by the launch)
int dense_tc_fwd(int dtype, const Geom& g, const void* x, const void* w, const void* bias, void* y, int* status, cudaStream_t stream, StatusClear& sc);
int dense_tc_bwd(int dtype, const Geom& g, const void* x, const void* w, const void* dy, void* dw, void* dx /*or null*/, int* status, cudaStream_t stream,
                 StatusClear& sc);

}  // namespace pcb
