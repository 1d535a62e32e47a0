// Linear projection y = x . W.  The reference reserves this header as an empty
// namespace (kuiper/include/op/matmul.h:1-11) and the LayerMatmul tag (op/layer.h:14).
//
// Quantised (is_quant_layer): INT4-AWQ.  weight slot 0 = qweight Int32 [K, N/8],
// slot 1 = qzeros Int32 [K/group, N/8], set_scales() = Fp16 [K/group, N],
// set_group_size(128); input [M, K], output [M, N].
// Plain: weight slot 0 = Bf16 [N, K] (one row per output, the lm_head layout).
//
// Optional residual: with set_residual(true) the layer takes a second input [M, N] and
// writes output = input2 + x . W in the same kernel (the output may be that tensor).
#ifndef KUIPER_INCLUDE_OP_MATMUL_H
#define KUIPER_INCLUDE_OP_MATMUL_H

#include "base/cuda_config.h"
#include "op/layer.h"

namespace op {
class MatmulLayer : public LayerParam {
public:
    // dim0 = output width N, dim1 = input width K
    explicit MatmulLayer(base::DeviceType device_type, int32_t dim0, int32_t dim1, bool is_quant_layer = false);

    base::Status check() const override;
    using Layer::forward;  // keep the N-ary overloads visible next to the override
    base::Status forward() override;

    void set_residual(bool has_residual);
    // accumulate mode (quantised layers): output += x . W, the output tensor already holds the addend
    // (residual stream or zeros); no workspace, unordered fp32 summation
    void set_accumulate(bool accumulate) { accumulate_ = accumulate; }
    // accumulate mode only: the input is an un-normalised row and the layer applies RMSNorm(input; weight, eps)
    // inside the matmul kernel (weight bf16 [dim1]); saves the separate norm launch
    void set_input_norm(const tensor::Tensor& weight, float eps) {
        input_norm_ = weight;
        input_norm_eps_ = eps;
    }
    // accumulate mode only: the input is a gate|up row [M, 2*dim1] and the layer applies SwiGLU inside the matmul
    // kernel (operand = silu(gate) * up); saves the separate activation launch.  The input is only read.
    void set_input_swiglu(bool on) { input_swiglu_ = on; }
    // where RMSNorm(input) / SwiGLU(input) is written when the row count takes the tensor-core path, which has
    // no fused prologue ([max rows, dim1] fp32)
    void set_norm_scratch(const tensor::Tensor& scratch) { norm_scratch_ = scratch; }
    // quantised layers, fp16-operand mode: inputs of at least this many rows go to the GEMM entry (packed-word kernel up to
    // 32 rows, tcgen05 tiles beyond) instead of the GEMV (0 = never).  Unless this is called the number is 16, and 3 where the
    // layer loses nothing by it: it accumulates (the GEMM entry adds with reductions, the GEMV of a layer that does not
    // accumulate sums in a fixed order), the GEMM workspace holds the rows, and N % 32 == 0 (other widths would
    // round the weight, which the GEMV does not).  Below three rows one pass of the accumulating GEMV, which also runs the input
    // norm / SwiGLU itself and so saves four launches a layer, is as fast: Qwen3-8B decode of two sequences
    // takes the same time either way (1.82 ms a step, 0.6B 0.71 against 0.82), of three 1.97 against 2.13, of five
    // 2.00 against 3.35.
    void set_gemm_min_rows(int32_t rows) { gemm_min_rows_ = rows < 0 ? 0 : rows; }
    // accumulate mode: passes of at least this many rows overwrite the output instead (0 = never), so that nobody has to
    // zero it; the engine sets it for the projections whose addend is zero.  Clearing gate|up before and reading it back for
    // the addition cost a 2048-row chunk of the Qwen3-8B shape 150 us a layer.
    void set_overwrite_rows(int32_t rows) { overwrite_rows_ = rows; }
    bool overwrites(int32_t rows) const {
        return is_quant_layer_ && act_mode_ != 0 && overwrite_rows_ > 0 && gemm_min_rows_ != 0 && rows >= overwrite_from();
    }
    // fewest rows of a pass that overwrites (where passes do): the GEMV, which serves what the GEMM entry does not, only adds
    int32_t overwrite_from() const {
        const int32_t gemm_from = gemm_min_rows_ < 0 ? kGemmRows : gemm_min_rows_;
        return overwrite_rows_ > gemm_from ? overwrite_rows_ : gemm_from;
    }
    // scratch of the split-K kernel: kernel::matmul_quant_workspace_bytes(M, K, N) bytes, zero-initialised once
    void set_workspace(const tensor::Tensor& workspace);
    // scratch of the tensor-core path: kernel::matmul_quant_gemm_workspace_bytes(max rows, dim1) bytes, no
    // initialisation needed
    void set_gemm_workspace(const tensor::Tensor& workspace) { gemm_workspace_ = workspace; }
    // accumulate mode: kernel::matmul_quant_ticket_bytes() zeroed bytes owned by this layer (its balance counters);
    // without them the kernel deals its work out statically
    void set_tickets(const tensor::Tensor& tickets) { tickets_ = tickets; }
    // how the INT4 kernel rounds x: 1 = fp16 operand (default), 0 = fp32 operand, 2 = block-scaled 16-bit integers for
    // single-row passes (the fastest decode kernel) and fp16 for passes of several rows
    void set_act_mode(int32_t act_mode) { act_mode_ = act_mode; }

    int32_t out_features() const { return dim0_; }
    int32_t in_features() const { return dim1_; }

protected:
    base::DataType weight_data_type(int32_t idx) const override;

private:
    static constexpr int32_t kGemmRows = 16, kGemmRowsAccumulating = 3;
    bool takes_gemm(int32_t rows) const;

    int32_t dim0_ = 0;
    int32_t dim1_ = 0;
    bool has_residual_ = false;
    bool accumulate_ = false;
    bool input_swiglu_ = false;
    tensor::Tensor input_norm_;
    float input_norm_eps_ = 1e-6f;
    int32_t act_mode_ = 1;
    tensor::Tensor workspace_;
    tensor::Tensor gemm_workspace_;
    tensor::Tensor norm_scratch_;
    tensor::Tensor tickets_;
    int32_t gemm_min_rows_ = -1;  // -1: the layer's own rule
    int32_t overwrite_rows_ = 0;
};
}  // namespace op

#endif  // KUIPER_INCLUDE_OP_MATMUL_H
