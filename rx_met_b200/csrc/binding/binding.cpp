// Torch side of the hot entry points: argument checks, output allocation, workspace and stream lookup, the call into
// the C ABI of librxmet_b200.so and the autograd node of the learned-grid quantize-dequantize.
//
// In Python with ctypes these took 60 to 180 us a call (qdq 4096 x 4096 with its gradients 160 us against 67 us of
// kernels, one GRU inference 92 us against 72), so that the small calls were bound by the interpreter.  The C ABI is
// not linked: the package loads the library globally first, so that an overridden library path reaches this module too.
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/utils/pybind.h>

#include <array>
#include <cstring>
#include <map>
#include <mutex>
#include <optional>
#include <vector>

#include "rxmet_b200.h"
#include "rxmet_b200_lstm.h"

namespace {

using at::Tensor;
using MaybeTensor = std::optional<Tensor>;
using Shape = std::vector<int64_t>;

void *streamOf(const Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// Null for an absent or empty tensor, as the C ABI expects.
template <class T>
T *pointer(const Tensor &t) {
    return t.defined() && t.numel() > 0 ? static_cast<T *>(t.data_ptr()) : nullptr;
}

std::string listText(at::IntArrayRef sizes) {
    std::string text = "[";
    for (size_t i = 0; i < sizes.size(); ++i) text += (i ? ", " : "") + std::to_string(sizes[i]);
    return text + "]";
}

Tensor emptyLike(const Tensor &like, at::IntArrayRef shape, at::ScalarType type = at::kFloat) {
    return at::empty(shape, at::TensorOptions().dtype(type).device(like.device()));
}

// Tensors of the given shapes over ONE allocation, each on a 16-byte boundary: a forward returns sixteen small tensors,
// and an allocator round trip for each is host time on the critical path of a training step.
std::vector<Tensor> carve(const Tensor &like, at::ScalarType type, const std::vector<Shape> &shapes) {
    const int64_t per = 16 / static_cast<int64_t>(c10::elementSize(type));
    std::vector<int64_t> offsets;
    int64_t total = 0;
    for (const Shape &shape : shapes) {
        int64_t n = 1;
        for (int64_t d : shape) n *= d;
        offsets.push_back(total);
        total += (n + per - 1) / per * per;
    }
    const Tensor pool = emptyLike(like, {std::max<int64_t>(total, 1)}, type);
    std::vector<Tensor> out;
    out.reserve(shapes.size());
    for (size_t i = 0; i < shapes.size(); ++i) {
        Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(pool.storage()), pool.key_set(), pool.dtype());
        t.unsafeGetTensorImpl()->set_storage_offset(pool.storage_offset() + offsets[i]);
        t.unsafeGetTensorImpl()->set_sizes_contiguous(shapes[i]);
        out.push_back(std::move(t));
    }
    return out;
}

// One growing scratch buffer per device and stream, reused across calls (calls on one stream follow one another).
Tensor workspace(const c10::Device &device, int64_t bytes) {
    static std::mutex mutex;
    static auto &buffers = *new std::map<std::pair<int, void *>, Tensor>;   // outlives the CUDA context's teardown
    void *stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    std::lock_guard<std::mutex> lock(mutex);
    Tensor &have = buffers[{device.index(), stream}];
    if (!have.defined() || have.numel() < bytes) {
        have = Tensor();
        have = at::empty({std::max<int64_t>(bytes, 1 << 20)}, at::TensorOptions().dtype(at::kByte).device(device));
    }
    return have;
}

// ---- GRU ----------------------------------------------------------------------------------------------------------

Tensor floatCuda(const Tensor &t, const char *name, at::IntArrayRef shape) {
    if (!t.is_cuda() || t.scalar_type() != at::kFloat) TORCH_CHECK(false, name, " must be CUDA float32 tensor");
    if (t.sizes() != shape) TORCH_CHECK(false, name, " must have shape ", listText(shape));
    return t.contiguous();
}

// Status of the library and the 18 tensors of the interface: h, v, five code tensors, eleven masks.
std::pair<int, std::vector<Tensor>> gruForwardQuant(bool training, int T, int B, int I, int H, Tensor W, Tensor R, Tensor bw,
                                                    Tensor br, Tensor x, const MaybeTensor &h0, uintptr_t paramsAddress,
                                                    bool floatCarrier) {
    const int64_t C = 3 * static_cast<int64_t>(H);
    W = floatCuda(W, "W", {I, C});
    R = floatCuda(R, "R", {H, C});
    bw = floatCuda(bw, "bw", {C});
    br = floatCuda(br, "br", {C});
    x = floatCuda(x, "x", {T, B, I});
    Tensor h0v;
    if (h0 && h0->numel() > 0) h0v = floatCuda(*h0, "h0", {B, H});
    const c10::cuda::CUDAGuard guard(x.device());
    std::vector<Tensor> out{emptyLike(x, {T + 1, B, H}), emptyLike(x, {T, B, 4 * static_cast<int64_t>(H)})};
    for (Tensor &t : carve(x, at::kInt, {{I, C}, {H, C}, {C}, {C}, {T, B, I}})) out.push_back(std::move(t));
    rxmet_gru_masks masks{};
    if (training) {
        uint8_t **const fields[] = {&masks.x, &masks.h0, &masks.W, &masks.R, &masks.bw, &masks.br, &masks.weight_ih_linear,
                                    &masks.weight_hh_linear, &masks.gate_input, &masks.gate_output, &masks.h};
        std::vector<Shape> shapes{{T, B, I}, {B, H}, {I, C}, {H, C}, {C}, {C}, {T, B, C}, {T, B, C}, {T, B, C}, {T, B, C}, {T, B, H}};
        if (!h0v.defined()) shapes[1] = {0};
        size_t k = 0;
        for (Tensor &t : carve(x, at::kByte, shapes)) {
            *fields[k++] = pointer<uint8_t>(t);
            out.push_back(std::move(t));
        }
    } else {
        const Tensor none = emptyLike(x, {0}, at::kByte);
        out.resize(18, none);
    }
    const Tensor ws = workspace(x.device(), static_cast<int64_t>(rxmet_gru_workspace_bytes(1, T, B, I, H)));
    const auto *params = reinterpret_cast<const rxmet_gru_quant_params *>(paramsAddress);
    const auto entry = floatCarrier ? rxmet_gru_forward_quant_fp_carrier : rxmet_gru_forward_quant;
    const pybind11::gil_scoped_release release;
    const int status = entry(training, T, B, I, H, pointer<float>(W), pointer<float>(R), pointer<float>(bw), pointer<float>(br),
                             pointer<float>(x), pointer<float>(h0v), params, pointer<float>(out[0]), pointer<float>(out[1]),
                             pointer<int32_t>(out[2]), pointer<int32_t>(out[3]), pointer<int32_t>(out[4]),
                             pointer<int32_t>(out[5]), pointer<int32_t>(out[6]), nullptr, nullptr, training ? &masks : nullptr,
                             ws.data_ptr(), static_cast<size_t>(ws.numel()), streamOf(x));
    return {status, std::move(out)};
}

std::pair<int, std::vector<Tensor>> gruBackwardQuant(int T, int B, int I, int H, const std::array<Tensor, 5> &cached, Tensor dh,
                                                     Tensor h, Tensor v, uintptr_t paramsAddress,
                                                     const std::array<MaybeTensor, 11> &flags) {
    const int64_t C = 3 * static_cast<int64_t>(H);
    const char *const names[] = {"W_q", "R_q", "bw_q", "br_q", "x_q"};
    const Shape shapes[] = {{I, C}, {H, C}, {C}, {C}, {T, B, I}};
    std::array<Tensor, 5> codes;
    for (int k = 0; k < 5; ++k) {
        if (!cached[k].is_cuda() || cached[k].sizes() != at::IntArrayRef(shapes[k]))
            TORCH_CHECK(false, names[k], " must be a CUDA tensor of shape ", listText(shapes[k]));
        codes[k] = (cached[k].scalar_type() == at::kInt ? cached[k] : cached[k].to(at::kInt)).contiguous();
    }
    dh = floatCuda(dh, "dh_new", {T + 1, B, H});
    h = floatCuda(h, "h", {T + 1, B, H});
    v = floatCuda(v, "v", {T, B, 4 * static_cast<int64_t>(H)});
    rxmet_gru_masks masks{};
    uint8_t **const fields[] = {&masks.x, &masks.h0, &masks.W, &masks.R, &masks.bw, &masks.br, &masks.weight_ih_linear,
                                &masks.weight_hh_linear, &masks.gate_input, &masks.gate_output, &masks.h};
    std::array<Tensor, 11> live;
    for (int k = 0; k < 11; ++k) {
        if (!flags[k] || flags[k]->numel() == 0) continue;
        live[k] = flags[k]->contiguous();
        *fields[k] = static_cast<uint8_t *>(live[k].data_ptr());
    }
    const c10::cuda::CUDAGuard guard(h.device());
    std::vector<Tensor> out = carve(h, at::kFloat, {{T, B, I}, {I, C}, {H, C}, {C}, {C}, {B, H}});
    const auto *params = reinterpret_cast<const rxmet_gru_quant_params *>(paramsAddress);
    const int8_t *bits = params->config.bits;
    const bool tensorCores = bits[RXMET_GRU_W] <= 8 && bits[RXMET_GRU_R] <= 8 && bits[RXMET_GRU_X] <= 16 && bits[RXMET_GRU_H] <= 16;
    const Tensor ws = workspace(h.device(), static_cast<int64_t>(rxmet_gru_workspace_bytes(tensorCores ? 2 : 4, T, B, I, H)));
    const pybind11::gil_scoped_release release;
    const int status = rxmet_gru_backward_quant(
        T, B, I, H, pointer<int32_t>(codes[0]), pointer<int32_t>(codes[1]), pointer<int32_t>(codes[2]), pointer<int32_t>(codes[3]),
        pointer<int32_t>(codes[4]), pointer<float>(dh), pointer<float>(h), pointer<float>(v), params, &masks,
        pointer<float>(out[0]), pointer<float>(out[1]), pointer<float>(out[2]), pointer<float>(out[3]), pointer<float>(out[4]),
        pointer<float>(out[5]), ws.data_ptr(), static_cast<size_t>(ws.numel()), streamOf(h));
    return {status, std::move(out)};
}

// ---- LSTM ---------------------------------------------------------------------------------------------------------

constexpr int kMasters = 7, kTrace = 7;

Tensor lstmFloat(const Tensor &t, const char *name) {
    if (t.scalar_type() != at::kFloat) TORCH_CHECK(false, name, " must be a float32 tensor");
    if (!t.is_cuda()) TORCH_CHECK(false, name, " must be a CUDA tensor");
    return t.contiguous();
}

// Checked, contiguous arguments of a forward or backward call (absent ones stay undefined).
struct LstmInputs {
    Tensor x, wIh, wHh, bIh, bHh, h0, c0;
    int T, B, I, H;
    LstmInputs(const Tensor &input, const Tensor &weightIh, const Tensor &weightHh, const MaybeTensor &biasIh,
               const MaybeTensor &biasHh, const MaybeTensor &hidden, const MaybeTensor &cell, bool batchFirst) {
        x = lstmFloat(input, "input");
        TORCH_CHECK(x.dim() == 3, "input must have 3 dimensions");
        if (batchFirst) x = x.transpose(0, 1).contiguous();
        T = static_cast<int>(x.size(0)); B = static_cast<int>(x.size(1)); I = static_cast<int>(x.size(2));
        wIh = lstmFloat(weightIh, "weight_ih");
        wHh = lstmFloat(weightHh, "weight_hh");
        TORCH_CHECK(wIh.dim() == 2 && wHh.dim() == 2 && wIh.size(0) % 4 == 0, "weights must be [4H, I] and [4H, H]");
        H = static_cast<int>(wIh.size(0) / 4);
        TORCH_CHECK(wIh.size(1) == I && wHh.size(0) == 4 * static_cast<int64_t>(H) && wHh.size(1) == H,
                    "weight shapes do not match input_size / hidden_size");
        TORCH_CHECK(biasIh.has_value() == biasHh.has_value(), "bias_ih and bias_hh must be given together");
        if (biasIh) {
            bIh = lstmFloat(*biasIh, "bias_ih");
            bHh = lstmFloat(*biasHh, "bias_hh");
            for (const Tensor *b : {&bIh, &bHh}) TORCH_CHECK(b->dim() == 1 && b->size(0) == 4 * static_cast<int64_t>(H), "bias must be [4H]");
        }
        TORCH_CHECK(hidden.has_value() == cell.has_value(), "initial_hidden and initial_cell must be given together");
        if (hidden) {
            h0 = lstmFloat(*hidden, "initial_hidden").reshape({B, H});
            c0 = lstmFloat(*cell, "initial_cell").reshape({B, H});
        }
    }
};

using LstmForward = std::tuple<int, Tensor, Tensor, Tensor, std::vector<Tensor>, std::vector<Tensor>, std::vector<Tensor>, std::vector<Tensor>>;

LstmForward lstmForwardQuant(const Tensor &input, const Tensor &weightIh, const Tensor &weightHh, const MaybeTensor &biasIh,
                             const MaybeTensor &biasHh, const MaybeTensor &hidden, const MaybeTensor &cell, bool batchFirst,
                             uintptr_t paramsAddress, bool requireExact, bool checkpoints) {
    const LstmInputs p(input, weightIh, weightHh, biasIh, biasHh, hidden, cell, batchFirst);
    const auto *params = reinterpret_cast<const rxmet_lstm_quant_params *>(paramsAddress);
    const int64_t T = p.T, B = p.B, H = p.H;
    TORCH_CHECK(params->input_size == p.I && params->hidden_size == p.H,
                "quantization parameters do not match input_size / hidden_size of the module");
    TORCH_CHECK((params->bias_enabled != 0) == p.bIh.defined(), "quantization parameters do not match the bias setting of the module");
    const c10::cuda::CUDAGuard guard(p.x.device());
    const Tensor out = emptyLike(p.x, {T, B, H}), hn = emptyLike(p.x, {1, B, H}), cn = emptyLike(p.x, {1, B, H});
    std::vector<Tensor> values, clamped, masters, masterClamped;
    rxmet_lstm_trace trace{};
    rxmet_lstm_masters saved{};
    static_assert(sizeof(trace) == 2 * kTrace * sizeof(void *) && sizeof(saved) == 2 * kMasters * sizeof(void *), "pointer tables");
    if (checkpoints) {
        std::array<void *, 2 * kTrace> table{};
        for (int k = 0; k < kTrace; ++k) {   // large tensors: an allocation each, so that a user can drop them one by one
            const int64_t width = k < 4 ? 4 * H : H;
            values.push_back(emptyLike(p.x, {T, B, width}));
            clamped.push_back(emptyLike(p.x, {T, B, width}, at::kByte));
            table[k] = pointer<void>(values.back());
            table[kTrace + k] = pointer<void>(clamped.back());
        }
        std::memcpy(&trace, table.data(), sizeof(trace));
        const int64_t bias = p.bIh.defined() ? 4 * H : 0;
        const std::vector<Shape> shapes{p.wIh.sizes().vec(), p.wHh.sizes().vec(), {bias}, {bias}, {1, B, H}, {1, B, H}};
        masters.push_back(emptyLike(p.x, p.x.sizes()));
        masterClamped.push_back(emptyLike(p.x, p.x.sizes(), at::kBool));
        for (Tensor &t : carve(p.x, at::kFloat, shapes)) masters.push_back(std::move(t));
        for (Tensor &t : carve(p.x, at::kBool, shapes)) masterClamped.push_back(std::move(t));   // every flag is written
        for (int k = 0; k < kMasters; ++k) {
            table[k] = pointer<void>(masters[k]);
            table[kMasters + k] = pointer<void>(masterClamped[k]);
        }
        std::memcpy(&saved, table.data(), sizeof(saved));
    }
    const Tensor ws = emptyLike(p.x, {static_cast<int64_t>(rxmet_lstm_workspace_bytes(1, p.T, p.B, p.I, p.H))}, at::kByte);
    int status;
    {
        const pybind11::gil_scoped_release release;
        status = rxmet_lstm_forward_quantized(
            p.T, p.B, p.I, p.H, pointer<float>(p.wIh), pointer<float>(p.wHh), pointer<float>(p.bIh), pointer<float>(p.bHh),
            pointer<float>(p.x), pointer<float>(p.h0), pointer<float>(p.c0), params, requireExact, pointer<float>(out),
            pointer<float>(hn), pointer<float>(cn), checkpoints ? &trace : nullptr, checkpoints ? &saved : nullptr, ws.data_ptr(),
            static_cast<size_t>(ws.numel()), streamOf(p.x));
    }
    return {status, out, hn, cn, std::move(values), std::move(clamped), std::move(masters), std::move(masterClamped)};
}

Tensor maskTensor(const Tensor &t, const char *name, at::IntArrayRef shape, const c10::Device &device, bool allowEmpty = false) {
    TORCH_CHECK(t.scalar_type() == at::kBool || t.scalar_type() == at::kByte, name, " must be a bool or uint8 tensor");
    TORCH_CHECK(t.device() == device, name, " is on another device");
    if (allowEmpty && t.numel() == 0) return Tensor();
    TORCH_CHECK(t.sizes() == shape, name, " shape mismatch");
    return t.contiguous();
}

std::pair<int, std::vector<Tensor>> lstmBackwardQat(const std::vector<Tensor> &masters, bool batchFirst, uintptr_t paramsAddress,
                                                    const std::vector<Tensor> &trace, const Tensor &gradOutput,
                                                    const Tensor &gradHidden, const Tensor &gradCell,
                                                    const std::vector<Tensor> &masterMasks, const std::vector<Tensor> &traceMasks) {
    const auto *params = reinterpret_cast<const rxmet_lstm_quant_params *>(paramsAddress);
    const bool bias = params->bias_enabled != 0;
    const LstmInputs p(masters[0], masters[1], masters[2], bias ? MaybeTensor(masters[3]) : MaybeTensor(),
                       bias ? MaybeTensor(masters[4]) : MaybeTensor(), masters[5], masters[6], batchFirst);
    const int64_t T = p.T, B = p.B, H = p.H, C = 4 * H;
    auto shaped = [](const Tensor &given, const char *name, at::IntArrayRef shape) {
        Tensor t = lstmFloat(given, name);
        TORCH_CHECK(t.sizes() == shape, name, " shape mismatch");
        return t;
    };
    const Tensor gates = shaped(trace[0], "gate_outputs", {T, B, C}), cells = shaped(trace[1], "cell_states", {T, B, H});
    const Tensor tanhs = shaped(trace[2], "cell_tanh_outputs", {T, B, H}), hiddens = shaped(trace[3], "hidden_outputs", {T, B, H});
    const Tensor gOut = shaped(gradOutput, "grad_output", {T, B, H}), gH = shaped(gradHidden, "grad_final_hidden", {B, H});
    const Tensor gC = shaped(gradCell, "grad_final_cell", {B, H});
    TORCH_CHECK(masterMasks.empty() == traceMasks.empty(), "master_masks and checkpoint_masks must be given together");
    rxmet_lstm_backward_masks flags{};
    static_assert(sizeof(flags) == (kMasters + kTrace) * sizeof(void *), "pointer table");
    std::vector<Tensor> keep;
    const c10::Device device = p.x.device();
    const c10::cuda::CUDAGuard guard(device);
    if (!masterMasks.empty()) {
        TORCH_CHECK(masterMasks.size() == kMasters && traceMasks.size() == kTrace,
                    "master_masks and checkpoint_masks must hold 7 tensors each");
        const char *const traceNames[] = {"weight_ih_linear_mask", "weight_hh_linear_mask", "gate_inputs_mask", "gate_outputs_mask",
                                          "cell_states_mask", "cell_tanh_outputs_mask", "hidden_outputs_mask"};
        Tensor first = maskTensor(masterMasks[0], "input_mask", masters[0].sizes(), device);
        keep.push_back(batchFirst ? first.transpose(0, 1).contiguous() : first);
        keep.push_back(maskTensor(masterMasks[1], "weight_ih_mask", p.wIh.sizes(), device));
        keep.push_back(maskTensor(masterMasks[2], "weight_hh_mask", p.wHh.sizes(), device));
        keep.push_back(maskTensor(masterMasks[3], "bias_ih_mask", {C}, device, true));
        keep.push_back(maskTensor(masterMasks[4], "bias_hh_mask", {C}, device, true));
        keep.push_back(maskTensor(masterMasks[5], "initial_hidden_mask", {1, B, H}, device));
        keep.push_back(maskTensor(masterMasks[6], "initial_cell_mask", {1, B, H}, device));
        for (int k = 0; k < kTrace; ++k) keep.push_back(maskTensor(traceMasks[k], traceNames[k], {T, B, k < 4 ? C : H}, device));
        std::array<void *, kMasters + kTrace> table;
        for (size_t k = 0; k < table.size(); ++k) table[k] = keep[k].defined() ? keep[k].data_ptr() : nullptr;
        std::memcpy(&flags, table.data(), sizeof(flags));
    }
    std::vector<Tensor> grads{emptyLike(p.x, {T, B, p.I})};
    for (Tensor &t : carve(p.x, at::kFloat, {p.wIh.sizes().vec(), p.wHh.sizes().vec(), {C}, {C}, {B, H}, {B, H}}))
        grads.push_back(std::move(t));
    rxmet_lstm_gradients out{};
    static_assert(sizeof(out) == kMasters * sizeof(void *), "pointer table");
    std::array<void *, kMasters> table;
    for (int k = 0; k < kMasters; ++k) table[k] = grads[k].data_ptr();
    std::memcpy(&out, table.data(), sizeof(out));
    const auto *bits = params->config.bitwidth;
    const bool tensorCores = bits[RXMET_LSTM_WEIGHT_IH] <= 8 && bits[RXMET_LSTM_WEIGHT_HH] <= 8 && bits[RXMET_LSTM_INPUT] <= 16 &&
                             bits[RXMET_LSTM_OUTPUT] <= 16;
    const Tensor ws = emptyLike(p.x, {static_cast<int64_t>(rxmet_lstm_workspace_bytes(tensorCores ? 2 : 4, p.T, p.B, p.I, p.H))}, at::kByte);
    int status;
    {
        const pybind11::gil_scoped_release release;
        status = rxmet_lstm_backward_qat(
            p.T, p.B, p.I, p.H, params, pointer<float>(p.wIh), pointer<float>(p.wHh), pointer<float>(p.x), pointer<float>(p.h0),
            pointer<float>(p.c0), pointer<float>(gates), pointer<float>(cells), pointer<float>(tanhs), pointer<float>(hiddens),
            pointer<float>(gOut), pointer<float>(gH), pointer<float>(gC), masterMasks.empty() ? nullptr : &flags, &out,
            ws.data_ptr(), static_cast<size_t>(ws.numel()), streamOf(p.x));
    }
    if (batchFirst) grads[0] = grads[0].transpose(0, 1);
    return {status, std::move(grads)};
}

// ---- learned-grid quantize-dequantize -----------------------------------------------------------------------------

void checkQdq(int status, const char *what) {
    if (status == RXMET_OK) return;
    const std::string message = std::string(what) + ": " + rxmet_last_error();
    if (status == RXMET_ERR_INVALID_ARGUMENT) throw pybind11::value_error(message);
    TORCH_CHECK(false, message, " (status ", status, ")");
}

Tensor gridValues(const Tensor &t) { return (t.scalar_type() == at::kFloat ? t : t.to(at::kFloat)).contiguous(); }

// Saves the input itself instead of a mask: the backward recomputes the flags in the pass that reads it anyway.
struct QuantDequant : torch::autograd::Function<QuantDequant> {
    static Tensor forward(torch::autograd::AutogradContext *ctx, const Tensor &tensor, const Tensor &scale, const Tensor &offset,
                          int64_t qmin, int64_t qmax, bool reciprocal, int64_t outer, int64_t channels, int64_t inner) {
        const c10::cuda::CUDAGuard guard(tensor.device());   // launch on the tensor's device, whatever device is current
        const Tensor x = tensor.contiguous(), s = gridValues(scale), o = gridValues(offset);
        Tensor y = at::empty_like(x);
        checkQdq(rxmet_affine_qdq_forward(x.const_data_ptr<float>(), outer, channels, inner, s.const_data_ptr<float>(),
                                          o.const_data_ptr<float>(), static_cast<int>(qmin), static_cast<int>(qmax), reciprocal,
                                          y.mutable_data_ptr<float>(), nullptr, streamOf(x)),
                 "affine_qdq.forward");
        ctx->save_for_backward({tensor, scale, offset});
        ctx->saved_data["plan"] = std::vector<int64_t>{qmin, qmax, reciprocal, outer, channels, inner};
        return y;
    }

    static torch::autograd::variable_list backward(torch::autograd::AutogradContext *ctx, torch::autograd::variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const auto plan = ctx->saved_data["plan"].toIntVector();
        const uint64_t outer = plan[3], channels = plan[4], inner = plan[5];
        torch::autograd::variable_list out(9);
        if (!grads[0].defined()) return out;
        const at::NoGradGuard noGrad;
        const c10::cuda::CUDAGuard guard(saved[0].device());
        const Tensor x = saved[0].contiguous(), s = gridValues(saved[1]), o = gridValues(saved[2]), g = gridValues(grads[0]);
        const bool wantScale = ctx->needs_input_grad(1), wantOffset = ctx->needs_input_grad(2);
        Tensor ws;
        size_t bytes = 0;
        if (ctx->needs_input_grad(0)) out[0] = at::empty_like(x);
        if (wantScale) out[1] = emptyLike(x, saved[1].sizes());
        if (wantOffset) out[2] = emptyLike(x, saved[2].sizes());
        if (wantScale || wantOffset) {
            bytes = rxmet_affine_qdq_backward_workspace_bytes(outer, channels, inner);
            if (bytes > 0) ws = emptyLike(x, {static_cast<int64_t>(bytes)}, at::kByte);
        }
        auto raw = [](const Tensor &t) { return t.defined() ? static_cast<float *>(t.data_ptr()) : nullptr; };
        checkQdq(rxmet_affine_qdq_backward(raw(g), raw(x), outer, channels, inner, raw(s), raw(o), static_cast<int>(plan[0]),
                                           static_cast<int>(plan[1]), static_cast<int>(plan[2]), raw(out[0]), raw(out[1]),
                                           raw(out[2]), ws.defined() ? ws.data_ptr() : nullptr, bytes, streamOf(x)),
                 "affine_qdq.backward");
        return out;
    }
};

Tensor quantizeDequantize(const Tensor &tensor, const Tensor &scale, const Tensor &offset, int64_t qmin, int64_t qmax,
                          bool reciprocal, int64_t outer, int64_t channels, int64_t inner) {
    return QuantDequant::apply(tensor, scale, offset, qmin, qmax, reciprocal, outer, channels, inner);
}

}  // namespace

PYBIND11_MODULE(_binding, m) {
    m.def("workspace", [](int device, int64_t bytes) { return workspace(c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(device)), bytes); });
    m.def("gru_forward_quant", &gruForwardQuant);
    m.def("gru_backward_quant", &gruBackwardQuant);
    m.def("lstm_forward_quant", &lstmForwardQuant);
    m.def("lstm_backward_qat", &lstmBackwardQat);
    m.def("quantize_dequantize", &quantizeDequantize, pybind11::call_guard<pybind11::gil_scoped_release>());
}
