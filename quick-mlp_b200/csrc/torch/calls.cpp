// Native call path of the Python package: the tensor-facing half of qmlp/bindings.py, qmlp/ops.py and qmlp/trainer.py.
//
// A small batch is bound by what the host does per call (a thousand points through a 64-wide network are 8 us of kernel).
// Argument checks, tensor views, output allocation, stream lookup and the autograd nodes therefore live here; Python only
// picks the object and makes one call. Measured against ctypes and Python autograd nodes: 29 -> 10 us for that batch,
// forward + mse_loss + backward of 64 000 points 264 -> 136 us.
//
// The entry points of libqmlp_b200.so are resolved at run time from the very library object qmlp/_capi.py has loaded
// (`load`), so this module has no second copy of its state and can be built before it.
#include <dlfcn.h>

#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>
#include <torch/library.h>

#include <qmlp_b200.h>

namespace {

using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// ---- the C ABI -------------------------------------------------------------------------------------------------------
#define QMLP_CALLS(X)                                                                                                     \
    X(last_error) X(network_num_encodings) X(network_channels_in) X(network_channels_out) X(network_encoding)             \
    X(network_destroy) X(network_set_parameter) X(network_inference_memory) X(network_inference_with_memory) X(network_inference_host) X(network_forward_memory)  \
    X(network_forward) X(network_adjoint_memory) X(network_adjoint) X(network_recompute_memory) X(network_forward_recompute) X(network_adjoint_recompute) X(network_parameter_count) X(encoding_create)         \
    X(encoding_num_output_channels) X(encoding_has_parameters) X(encoding_set_parameter) X(encoding_forward_memory) X(encoding_forward_with_memory)              \
    X(encoding_adjoint_memory) X(encoding_adjoint_with_memory) X(activation_create) X(activation_forward) X(activation_adjoint) X(trainer_workspace_bytes)       \
    X(trainer_gradients_part) X(trainer_update) X(convert_half)

struct Api {
#define QMLP_MEMBER(name) decltype(&qmlp_##name) name = nullptr;
    QMLP_CALLS(QMLP_MEMBER)
#undef QMLP_MEMBER
} api;

PyObject* errorType = nullptr;          // qmlp._capi.QmlpError
PyObject* configurationErrorType = nullptr;

// raises a Python exception from any thread, with or without the interpreter lock
[[noreturn]] void raise(PyObject* type, const std::string& message)
{
    py::gil_scoped_acquire gil;
    PyErr_SetString(type ? type : PyExc_RuntimeError, message.c_str());
    python_error e;
    e.persist();
    throw e;
}
[[noreturn]] void raiseError(const std::string& message) { raise(errorType, message); }
void check(int status)
{
    if (status != QMLP_OK) raise(status == QMLP_ERROR_CONFIGURATION ? configurationErrorType : errorType, api.last_error());
}

// non-owning view of a tensor (role of qmlp::wrap, src_cpp/pytorch-bindings/src/bindings.cpp:25-60)
qmlp_tensor_t wrap(const Tensor& t)
{
    qmlp_tensor_t v{};
    if (!t.defined()) return v;
    if (!t.is_cuda()) raiseError("tensor must live on a CUDA device");
    switch (t.scalar_type()) {
    case torch::kFloat32: v.precision = QMLP_FLOAT; break;
    case torch::kFloat16: v.precision = QMLP_HALF; break;
    case torch::kFloat64: v.precision = QMLP_DOUBLE; break;
    default: raiseError(std::string("unsupported dtype ") + c10::toString(t.scalar_type()));
    }
    if (t.dim() < 1 || t.dim() > 2) raiseError("only 1-D and 2-D tensors are supported");
    v.data = t.data_ptr();
    v.ndim = static_cast<int>(t.dim());
    for (int i = 0; i < v.ndim; ++i) {
        v.sizes[i] = t.size(i);
        v.strides[i] = t.stride(i);
    }
    return v;
}

qmlp_stream_t currentStream() { return c10::cuda::getCurrentCUDAStream().stream(); }

Tensor zeros(at::IntArrayRef sizes, const at::TensorOptions& options)
{
    // a plain memset instead of a fill kernel
    Tensor t = at::empty(sizes, options.memory_format(c10::MemoryFormat::Contiguous));
    if (t.numel() > 0) C10_CUDA_CHECK(cudaMemsetAsync(t.data_ptr(), 0, t.nbytes(), c10::cuda::getCurrentCUDAStream().stream()));
    return t;
}
Tensor zerosLike(const Tensor& t) { return t.is_contiguous() ? zeros(t.sizes(), t.options()) : at::zeros_like(t); }
at::TensorOptions floatLike(const Tensor& t) { return at::TensorOptions().dtype(torch::kFloat32).device(t.device()); }

Tensor toHalf(const Tensor& p)
{
    if (p.scalar_type() == torch::kFloat16) return p;
    if (p.scalar_type() != torch::kFloat32 || !p.is_cuda() || p.dim() != 1 || !p.is_contiguous()) return p.to(torch::kFloat16);
    Tensor h = at::empty(p.sizes(), p.options().dtype(torch::kFloat16));
    check(api.convert_half(static_cast<const float*>(p.data_ptr()), static_cast<uint16_t*>(h.data_ptr()), p.numel(), currentStream()));
    return h;
}

// ---- networks --------------------------------------------------------------------------------------------------------
// Owns a network handle. The parameter pointers bound to it are state of the network, so binding and launching happen
// under one mutex (taken without the interpreter lock).
struct NetworkCalls : torch::CustomClassHolder {
    qmlp_network_t* handle;
    std::vector<qmlp_encoding_t*> encodings;
    std::vector<bool> hasParameters;
    int64_t channelsIn, channelsOut, parameterCount;
    std::mutex mutex;

    explicit NetworkCalls(intptr_t h) : handle(reinterpret_cast<qmlp_network_t*>(h))
    {
        const int n = api.network_num_encodings(handle);
        for (int i = 0; i < n; ++i) {
            qmlp_encoding_t* e = nullptr;
            check(api.network_encoding(handle, i, &e));
            encodings.push_back(e);
            hasParameters.push_back(api.encoding_has_parameters(e) != 0);
        }
        channelsIn = api.network_channels_in(handle);
        channelsOut = api.network_channels_out(handle);
        parameterCount = api.network_parameter_count(handle);
    }
    ~NetworkCalls() override { api.network_destroy(handle); }

    void bind(const Tensor& half, const std::vector<OptTensor>& encodingParameters)
    {
        if (half.defined()) {
            const qmlp_tensor_t v = wrap(half);
            check(api.network_set_parameter(handle, &v, QMLP_INFERENCE));
        }
        for (size_t i = 0; i < encodingParameters.size() && i < encodings.size(); ++i)
            if (encodingParameters[i].has_value() && encodingParameters[i]->defined()) {
                const qmlp_tensor_t v = wrap(*encodingParameters[i]);
                check(api.encoding_set_parameter(encodings[i], &v, QMLP_INFERENCE));
            }
    }
};
using NetworkCalls_ptr = c10::intrusive_ptr<NetworkCalls>;

void networkBind(const NetworkCalls_ptr& self, const OptTensor& parameters, const std::vector<OptTensor>& encodingParameters)
{
    std::lock_guard<std::mutex> lock(self->mutex);
    self->bind(parameters.value_or(Tensor()), encodingParameters);
}

Tensor networkInference(const NetworkCalls_ptr& self, const Tensor& input, const Tensor& parameters, const std::vector<OptTensor>& encodingParameters)
{
    const qmlp_tensor_t in = wrap(input);
    Tensor output = at::empty({input.size(0), self->channelsOut}, floatLike(input));
    qmlp_tensor_t out = wrap(output);
    const Tensor half = toHalf(parameters);
    std::lock_guard<std::mutex> lock(self->mutex);
    self->bind(half, encodingParameters);
    size_t bytes = 0;   // feature planes of large grid batches
    check(api.network_inference_memory(self->handle, input.size(0), &bytes));
    const Tensor tmp = bytes > 0 ? at::empty({static_cast<int64_t>(bytes)}, floatLike(input).dtype(torch::kUInt8)) : Tensor();
    check(api.network_inference_with_memory(self->handle, &in, &out, currentStream(), bytes > 0 ? tmp.data_ptr() : nullptr, bytes));
    return output;
}

void networkInferenceHost(const NetworkCalls_ptr& self, const Tensor& input, const Tensor& parameters,
                          const std::vector<OptTensor>& encodingParameters, const Tensor& output, int64_t chunkPoints)
{
    const Tensor half = toHalf(parameters);
    std::lock_guard<std::mutex> lock(self->mutex);
    self->bind(half, encodingParameters);
    check(api.network_inference_host(self->handle, static_cast<const float*>(input.data_ptr()), static_cast<float*>(output.data_ptr()),
                                     input.size(0), chunkPoints, currentStream()));
}

// Autograd node of a network call (NetworkBindings::forward, src_cpp/pytorch-bindings/src/bind_network.cpp:120-321).
// Tensor arguments in order: input, network parameters, and the parameters of the encodings listed in `slots`.
struct NetworkFunction : torch::autograd::Function<NetworkFunction> {
    static std::vector<OptTensor> bySlot(const NetworkCalls& self, const std::vector<int64_t>& slots, at::ArrayRef<Tensor> list)
    {
        std::vector<OptTensor> v(self.encodings.size());
        for (size_t i = 0; i < slots.size(); ++i) v[slots[i]] = list[i];
        return v;
    }
    static Tensor forward(AutogradContext* ctx, const NetworkCalls_ptr& self, int64_t flags, const std::vector<int64_t>& slots, const Tensor& input,
                          const Tensor& parameters, at::TensorList encodingList)
    {
        const qmlp_tensor_t in = wrap(input);
        const Tensor half = toHalf(parameters);
        Tensor output = at::empty({input.size(0), self->channelsOut}, floatLike(input));
        qmlp_tensor_t out = wrap(output);
        Tensor tmp;
        size_t bytes = 0, adjointBytes = 0;
        bool recompute;
        {
            std::lock_guard<std::mutex> lock(self->mutex);
            self->bind(half, bySlot(*self, slots, encodingList));
            check(api.network_recompute_memory(self->handle, input.size(0), static_cast<int>(flags), &bytes, &adjointBytes));
            recompute = bytes > 0;
            if (!recompute) {
                check(api.network_forward_memory(self->handle, input.size(0), static_cast<int>(flags), &bytes));
                check(api.network_adjoint_memory(self->handle, input.size(0), static_cast<int>(flags), &adjointBytes));
            }
            tmp = at::empty({static_cast<int64_t>(std::max<size_t>(bytes, 16))}, floatLike(input).dtype(torch::kUInt8));
            check((recompute ? api.network_forward_recompute : api.network_forward)(self->handle, &in, &out, tmp.data_ptr(), currentStream()));
        }
        ctx->saved_data["recompute"] = recompute;
        ctx->saved_data["adjoint_bytes"] = static_cast<int64_t>(adjointBytes);
        ctx->saved_data["self"] = c10::IValue::make_capsule(self);
        ctx->saved_data["flags"] = flags;
        ctx->saved_data["slots"] = slots;
        ctx->saved_data["param_dtype"] = static_cast<int64_t>(parameters.scalar_type());
        variable_list saved = {input, half, tmp};
        for (const auto& p : encodingList) saved.push_back(p);
        ctx->save_for_backward(std::move(saved));
        return output;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grad)
    {
        const auto self = c10::static_intrusive_pointer_cast<NetworkCalls>(ctx->saved_data["self"].toCapsule());
        const int flags = static_cast<int>(ctx->saved_data["flags"].toInt());
        const auto saved = ctx->get_saved_variables();
        const Tensor &input = saved[0], &half = saved[1], &tmp = saved[2];
        const std::vector<int64_t> slots = ctx->saved_data["slots"].toIntVector();
        const Tensor gradOutput = grad[0].contiguous();
        const qmlp_tensor_t in = wrap(input), go = wrap(gradOutput);
        // the kernels add to their gradient buffers
        Tensor adjInput = (flags & QMLP_GRADIENTS_INPUT) ? zerosLike(input) : Tensor();
        Tensor adjParams = (flags & QMLP_GRADIENTS_NETWORK_WEIGHTS) ? zeros(half.sizes(), floatLike(half)) : Tensor();
        std::vector<Tensor> adjEncodings(slots.size());
        const bool recompute = ctx->saved_data["recompute"].toBool();
        Tensor adjTmp = at::empty({std::max<int64_t>(ctx->saved_data["adjoint_bytes"].toInt(), 16)}, floatLike(input).dtype(torch::kUInt8));
        {
            std::lock_guard<std::mutex> lock(self->mutex);
            self->bind(half, bySlot(*self, slots, at::ArrayRef<Tensor>(saved).slice(3)));
            if (adjParams.defined()) {
                const qmlp_tensor_t v = wrap(adjParams);
                check(api.network_set_parameter(self->handle, &v, QMLP_GRADIENTS));
            }
            if (flags & QMLP_GRADIENTS_INPUT_ENCODINGS) {
                std::vector<qmlp_tensor_t> bound(self->encodings.size(), qmlp_tensor_t{});
                for (size_t i = 0; i < slots.size(); ++i) {
                    const Tensor& p = saved[3 + i];
                    if (!p.requires_grad()) continue;
                    adjEncodings[i] = zeros(p.sizes(), floatLike(p));
                    bound[slots[i]] = wrap(adjEncodings[i]);
                }
                for (size_t i = 0; i < bound.size(); ++i)
                    if (self->hasParameters[i]) check(api.encoding_set_parameter(self->encodings[i], &bound[i], QMLP_GRADIENTS));
            }
            qmlp_tensor_t ai = wrap(adjInput);
            check((recompute ? api.network_adjoint_recompute : api.network_adjoint)(self->handle, &in, &go, flags, &ai, tmp.data_ptr(), adjTmp.data_ptr(),
                                                                                   currentStream()));
        }
        if (adjParams.defined()) adjParams = adjParams.to(static_cast<c10::ScalarType>(ctx->saved_data["param_dtype"].toInt()));
        variable_list out = {Tensor(), Tensor(), Tensor(), adjInput, adjParams};
        for (auto& g : adjEncodings) out.push_back(std::move(g));
        return out;
    }
};

Tensor networkForward(const NetworkCalls_ptr& self, const Tensor& input, const Tensor& parameters, const std::vector<OptTensor>& encodingParameters)
{
    int64_t flags = 0;
    if (torch::GradMode::is_enabled()) {
        if (input.requires_grad()) flags |= QMLP_GRADIENTS_INPUT;
        if (parameters.requires_grad()) flags |= QMLP_GRADIENTS_NETWORK_WEIGHTS;
        for (const auto& p : encodingParameters)
            if (p.has_value() && p->requires_grad()) flags |= QMLP_GRADIENTS_INPUT_ENCODINGS;
    }
    if (flags == 0) return networkInference(self, input, parameters, encodingParameters);
    std::vector<Tensor> list;
    std::vector<int64_t> slots;
    for (size_t i = 0; i < encodingParameters.size() && i < self->encodings.size(); ++i)
        if (encodingParameters[i].has_value() && encodingParameters[i]->defined()) {
            list.push_back(*encodingParameters[i]);
            slots.push_back(static_cast<int64_t>(i));
        }
    return NetworkFunction::apply(self, flags, slots, input, parameters, at::TensorList(list));
}

// ---- stand-alone encodings and activations: torch.ops.qmlp_b200.* -----------------------------------------------------
// The operators are keyed by the configuration text, so that a traced graph holds a string constant and an operator name
// (the reference registers TorchScript classes for this, src_cpp/pytorch-bindings/src/bind_encoding.cpp:167-197,
// bind_activation.cpp:82-98). The compiled objects are looked up by that text and live as long as the process.
struct EncodingEntry {
    qmlp_encoding_t* handle = nullptr;
    int64_t channels = 0;
    std::mutex mutex;   // a call with explicit parameters binds them for its duration
};
template <class Entry, class Make>
Entry& lookup(std::string_view cfg, Make make)
{
    static std::mutex mutex;
    static std::unordered_map<std::string, std::unique_ptr<Entry>> entries;
    std::lock_guard<std::mutex> lock(mutex);
    std::unique_ptr<Entry>& e = entries[std::string(cfg)];
    if (!e) {
        auto fresh = std::make_unique<Entry>();
        make(*fresh, std::string(cfg));
        e = std::move(fresh);
    }
    return *e;
}
EncodingEntry& encodingOf(std::string_view cfg)
{
    return lookup<EncodingEntry>(cfg, [](EncodingEntry& e, const std::string& text) {
        check(api.encoding_create(text.c_str(), &e.handle));
        e.channels = api.encoding_num_output_channels(e.handle);
    });
}
struct ActivationEntry { qmlp_activation_t* handle = nullptr; };
qmlp_activation_t* activationOf(std::string_view cfg)
{
    return lookup<ActivationEntry>(cfg, [](ActivationEntry& e, const std::string& text) { check(api.activation_create(text.c_str(), &e.handle)); }).handle;
}

Tensor encodingForward(const Tensor& input, const OptTensor& parameters, std::string_view cfg)
{
    EncodingEntry& e = encodingOf(cfg);
    const qmlp_tensor_t in = wrap(input), p = parameters.has_value() ? wrap(*parameters) : qmlp_tensor_t{};
    Tensor output = at::empty({input.size(0), e.channels}, floatLike(input));
    qmlp_tensor_t out = wrap(output);
    const qmlp_tensor_t* bound = parameters.has_value() ? &p : nullptr;
    size_t bytes = 0;   // copies of small levels by cell
    check(api.encoding_forward_memory(e.handle, input.size(0), bound, &bytes));
    const Tensor tmp = bytes > 0 ? at::empty({static_cast<int64_t>(bytes)}, floatLike(input).dtype(torch::kUInt8)) : Tensor();
    std::lock_guard<std::mutex> lock(e.mutex);
    check(api.encoding_forward_with_memory(e.handle, &in, &out, currentStream(), bound, bytes > 0 ? tmp.data_ptr() : nullptr, bytes));
    return output;
}
// what is not asked for is returned as an empty tensor
std::tuple<Tensor, Tensor> encodingAdjoint(const Tensor& input, const OptTensor& parameters, const Tensor& adjOutput, bool wantInput,
                                           bool wantParameters, std::string_view cfg)
{
    EncodingEntry& e = encodingOf(cfg);
    const bool param = wantParameters && parameters.has_value();
    const Tensor go = adjOutput.contiguous();
    Tensor adjInput = wantInput ? zerosLike(input) : at::empty({0}, input.options());
    Tensor adjParam = param ? zeros(parameters->sizes(), floatLike(*parameters)) : at::empty({0}, input.options());
    const qmlp_tensor_t in = wrap(input), ao = wrap(go), p = parameters.has_value() ? wrap(*parameters) : qmlp_tensor_t{};
    qmlp_tensor_t ai = wantInput ? wrap(adjInput) : qmlp_tensor_t{}, ap = param ? wrap(adjParam) : qmlp_tensor_t{};
    const int mode = (wantInput ? QMLP_ENCODING_INPUT_GRADIENTS : 0) | (param ? QMLP_ENCODING_PARAM_GRADIENTS : 0);
    size_t bytes = 0;
    check(api.encoding_adjoint_memory(e.handle, input.size(0), mode, &bytes));
    const Tensor tmp = bytes > 0 ? at::empty({static_cast<int64_t>(bytes)}, floatLike(input).dtype(torch::kUInt8)) : Tensor();
    std::lock_guard<std::mutex> lock(e.mutex);
    check(api.encoding_adjoint_with_memory(e.handle, &in, &ao, &ai, currentStream(), parameters.has_value() ? &p : nullptr, param ? &ap : nullptr, mode,
                                           bytes > 0 ? tmp.data_ptr() : nullptr, bytes));
    return {adjInput, adjParam};
}
Tensor activationForward(const Tensor& input, std::string_view cfg)
{
    qmlp_activation_t* a = activationOf(cfg);
    Tensor output = at::empty_like(input, input.options(), c10::MemoryFormat::Contiguous);
    const qmlp_tensor_t in = wrap(input);
    qmlp_tensor_t out = wrap(output);
    check(api.activation_forward(a, &in, &out, currentStream()));
    return output;
}
Tensor activationAdjoint(const Tensor& input, const Tensor& adjOutput, std::string_view cfg)
{
    qmlp_activation_t* a = activationOf(cfg);
    Tensor adjInput = at::empty_like(input, input.options(), c10::MemoryFormat::Contiguous);
    const qmlp_tensor_t in = wrap(input), ao = wrap(adjOutput);
    qmlp_tensor_t ai = wrap(adjInput);
    check(api.activation_adjoint(a, &in, &ao, &ai, currentStream()));
    return adjInput;
}

struct EncodingFunction : torch::autograd::Function<EncodingFunction> {
    static Tensor forward(AutogradContext* ctx, const Tensor& input, const OptTensor& parameters, const std::string& cfg)
    {
        at::AutoDispatchBelowADInplaceOrView below;
        ctx->saved_data["cfg"] = cfg;
        ctx->save_for_backward({input, parameters.value_or(Tensor())});
        static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("qmlp_b200::encoding_forward", "").typed<decltype(encodingForward)>();
        return op.call(input, parameters, cfg);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grad)
    {
        const auto saved = ctx->get_saved_variables();
        const Tensor& parameters = saved[1];
        const bool wantInput = ctx->needs_input_grad(0), wantParameters = parameters.defined() && ctx->needs_input_grad(1);
        static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("qmlp_b200::encoding_adjoint", "").typed<decltype(encodingAdjoint)>();
        auto g = op.call(saved[0], parameters.defined() ? OptTensor(parameters) : OptTensor(), grad[0], wantInput, wantParameters,
                         ctx->saved_data["cfg"].toStringRef());
        return {wantInput ? std::get<0>(g) : Tensor(), wantParameters ? std::get<1>(g).to(parameters.scalar_type()) : Tensor(), Tensor()};
    }
};
struct ActivationFunction : torch::autograd::Function<ActivationFunction> {
    static Tensor forward(AutogradContext* ctx, const Tensor& input, const std::string& cfg)
    {
        at::AutoDispatchBelowADInplaceOrView below;
        ctx->saved_data["cfg"] = cfg;
        ctx->save_for_backward({input});
        static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("qmlp_b200::activation_forward", "").typed<decltype(activationForward)>();
        return op.call(input, cfg);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grad)
    {
        static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("qmlp_b200::activation_adjoint", "").typed<decltype(activationAdjoint)>();
        return {op.call(ctx->get_saved_variables()[0], grad[0].contiguous(), ctx->saved_data["cfg"].toStringRef()), Tensor()};
    }
};
// The kernels write into fresh tensors: without a node of their own the results of the adjoint operators would count as
// constants in a second differentiation (create_graph), and a gradient term of a loss would drop out unnoticed.
[[noreturn]] void raiseNotTwice(const char* op)
{
    throw std::runtime_error(std::string("qmlp_b200::") + op + " is not differentiable: the operators can be differentiated once only");
}
struct EncodingAdjointFunction : torch::autograd::Function<EncodingAdjointFunction> {
    static variable_list forward(AutogradContext* ctx, const Tensor& input, const OptTensor& parameters, const Tensor& adjOutput, bool wantInput,
                                 bool wantParameters, const std::string& cfg)
    {
        at::AutoDispatchBelowADInplaceOrView below;
        static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("qmlp_b200::encoding_adjoint", "").typed<decltype(encodingAdjoint)>();
        auto g = op.call(input, parameters, adjOutput, wantInput, wantParameters, cfg);
        return {std::get<0>(g), std::get<1>(g)};
    }
    static variable_list backward(AutogradContext*, variable_list) { raiseNotTwice("encoding_adjoint"); }
};
struct ActivationAdjointFunction : torch::autograd::Function<ActivationAdjointFunction> {
    static Tensor forward(AutogradContext*, const Tensor& input, const Tensor& adjOutput, const std::string& cfg)
    {
        at::AutoDispatchBelowADInplaceOrView below;
        static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("qmlp_b200::activation_adjoint", "").typed<decltype(activationAdjoint)>();
        return op.call(input, adjOutput, cfg);
    }
    static variable_list backward(AutogradContext*, variable_list) { raiseNotTwice("activation_adjoint"); }
};

// Nodes are made only where a gradient can be asked for. Otherwise the operator runs below autograd, as operators without a
// forward-mode formula do: a dual tensor that requires no gradient is taken for its primal value.
bool differentiable(const Tensor& t) { return t.defined() && t.requires_grad(); }
bool differentiable(const OptTensor& t) { return t.has_value() && differentiable(*t); }
template <class... T>
bool wantsNode(const T&... tensors) { return torch::GradMode::is_enabled() && (differentiable(tensors) || ...); }

Tensor encodingForwardAutograd(const Tensor& input, const OptTensor& parameters, std::string_view cfg)
{
    if (wantsNode(input, parameters)) return EncodingFunction::apply(input, parameters, std::string(cfg));
    at::AutoDispatchBelowADInplaceOrView below;
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("qmlp_b200::encoding_forward", "").typed<decltype(encodingForward)>();
    return op.call(input, parameters, cfg);
}
Tensor activationForwardAutograd(const Tensor& input, std::string_view cfg)
{
    if (wantsNode(input)) return ActivationFunction::apply(input, std::string(cfg));
    at::AutoDispatchBelowADInplaceOrView below;
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("qmlp_b200::activation_forward", "").typed<decltype(activationForward)>();
    return op.call(input, cfg);
}
std::tuple<Tensor, Tensor> encodingAdjointAutograd(const Tensor& input, const OptTensor& parameters, const Tensor& adjOutput, bool wantInput,
                                                   bool wantParameters, std::string_view cfg)
{
    if (wantsNode(input, parameters, adjOutput)) {
        auto g = EncodingAdjointFunction::apply(input, parameters, adjOutput, wantInput, wantParameters, std::string(cfg));
        return {g[0], g[1]};
    }
    at::AutoDispatchBelowADInplaceOrView below;
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("qmlp_b200::encoding_adjoint", "").typed<decltype(encodingAdjoint)>();
    return op.call(input, parameters, adjOutput, wantInput, wantParameters, cfg);
}
Tensor activationAdjointAutograd(const Tensor& input, const Tensor& adjOutput, std::string_view cfg)
{
    if (wantsNode(input, adjOutput)) return ActivationAdjointFunction::apply(input, adjOutput, std::string(cfg));
    at::AutoDispatchBelowADInplaceOrView below;
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("qmlp_b200::activation_adjoint", "").typed<decltype(activationAdjoint)>();
    return op.call(input, adjOutput, cfg);
}

Tensor encodingForwardMeta(const Tensor& input, const OptTensor&, std::string_view cfg)
{
    return at::empty_symint({input.sym_size(0), encodingOf(cfg).channels}, input.options());
}
std::tuple<Tensor, Tensor> encodingAdjointMeta(const Tensor& input, const OptTensor& parameters, const Tensor&, bool wantInput, bool wantParameters, std::string_view)
{
    return {wantInput ? at::empty_like(input) : at::empty({0}, input.options()),
            wantParameters && parameters.has_value() ? at::empty_like(*parameters, at::kFloat) : at::empty({0}, input.options())};
}
Tensor activationForwardMeta(const Tensor& input, std::string_view) { return at::empty_like(input, input.options(), c10::MemoryFormat::Contiguous); }
Tensor activationAdjointMeta(const Tensor& input, const Tensor&, std::string_view) { return activationForwardMeta(input, ""); }

// ---- training step ---------------------------------------------------------------------------------------------------
// workspace the step needs for a batch, in bytes
int64_t trainerWorkspaceBytes(intptr_t trainer, int64_t points)
{
    size_t bytes = 0;
    check(api.trainer_workspace_bytes(reinterpret_cast<qmlp_trainer_t*>(trainer), points, &bytes));
    return static_cast<int64_t>(bytes);
}
void trainerGradients(intptr_t trainer, const Tensor& x, const Tensor& target, int64_t globalPoints, const Tensor& workspace, const OptTensor& lossSum,
                      int64_t parts)
{
    const qmlp_tensor_t in = wrap(x), t = wrap(target);
    check(api.trainer_gradients_part(reinterpret_cast<qmlp_trainer_t*>(trainer), &in, &t, globalPoints, workspace.data_ptr(),
                                     static_cast<size_t>(workspace.numel()),
                                     lossSum.has_value() ? static_cast<float*>(lossSum->data_ptr()) : nullptr, static_cast<int>(parts), currentStream()));
}
void trainerUpdate(intptr_t trainer, int64_t step, double gradScale)
{
    check(api.trainer_update(reinterpret_cast<qmlp_trainer_t*>(trainer), step, static_cast<float>(gradScale), currentStream()));
}

// Resolves the C ABI, then registers the kernels of the operators that qmlp/ops.py defines (in this order: another thread may
// call an operator as soon as it is registered). The devices' own autograd keys are used: the alias key holds the entry that
// loads this module.
void load(const std::string& path, py::object error, py::object configurationError)
{
    void* h = ::dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
    if (!h) throw std::runtime_error(std::string("dlopen: ") + ::dlerror());
#define QMLP_RESOLVE(name)                                                                                                \
    api.name = reinterpret_cast<decltype(&qmlp_##name)>(::dlsym(h, "qmlp_" #name));                                       \
    if (!api.name) throw std::runtime_error("qmlp_" #name " not found in " + path);
    QMLP_CALLS(QMLP_RESOLVE)
#undef QMLP_RESOLVE
    errorType = error.release().ptr();
    configurationErrorType = configurationError.release().ptr();
    auto kernels = [](c10::DispatchKey key, auto encodingForwardK, auto encodingAdjointK, auto activationForwardK, auto activationAdjointK) {
        auto* m = new torch::Library(torch::Library::IMPL, "qmlp_b200", key, __FILE__, __LINE__);   // (lives as long as the process)
        m->impl("encoding_forward", encodingForwardK);
        m->impl("encoding_adjoint", encodingAdjointK);
        m->impl("activation_forward", activationForwardK);
        m->impl("activation_adjoint", activationAdjointK);
    };
    static bool registered = false;
    if (registered) return;
    registered = true;
    kernels(c10::DispatchKey::CUDA, encodingForward, encodingAdjoint, activationForward, activationAdjoint);
    kernels(c10::DispatchKey::Meta, encodingForwardMeta, encodingAdjointMeta, activationForwardMeta, activationAdjointMeta);
    for (auto key : {c10::DispatchKey::AutogradCUDA, c10::DispatchKey::AutogradMeta, c10::DispatchKey::AutogradOther})   // (Other: functorch)
        kernels(key, encodingForwardAutograd, encodingAdjointAutograd, activationForwardAutograd, activationAdjointAutograd);
}

} // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m)
{
    using torch::wrap_pybind_function;
    using torch::wrap_pybind_function_no_gil;
    m.def("load", load);
    py::class_<NetworkCalls, NetworkCalls_ptr>(m, "NetworkCalls")
        .def(py::init([](intptr_t handle) { return c10::make_intrusive<NetworkCalls>(handle); }))
        .def_readonly("channels_out", &NetworkCalls::channelsOut);
    m.def("network_bind", wrap_pybind_function_no_gil(networkBind));
    m.def("network_inference", wrap_pybind_function_no_gil(networkInference));
    m.def("network_inference_host", wrap_pybind_function_no_gil(networkInferenceHost));
    m.def("network_forward", wrap_pybind_function_no_gil(networkForward));
    m.def("trainer_workspace_bytes", wrap_pybind_function_no_gil(trainerWorkspaceBytes));
    m.def("trainer_gradients", wrap_pybind_function_no_gil(trainerGradients));
    m.def("trainer_update", wrap_pybind_function_no_gil(trainerUpdate));
}
