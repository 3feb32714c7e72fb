// The PyTorch side of the calls that are short enough for the interpreter to be what they cost: the
// engine functions of brokefish_b200/env.py and the device-resident evaluator calls of
// brokefish_b200/nn/cuda_impl.py.  Argument checks, output tensors, the current stream and the call
// into the C ABI (include/brokefish_b200.h) in one native function each; the kernels live in
// libbrokefish_b200, which `bind` opens.
//
// One ply of 4096 games (step with moves and key, repetition ring, game-end rules) took 148 us
// through Python and ctypes, of which its kernels needed 45: eleven small tensor operations
// (zero fills of buffers that the kernels fill anyway, clones, conversions between bool and bytes)
// and about 40 us of attribute look-ups, shape tuples and argument boxing.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/utils/pybind.h>

#include <sstream>
#include <string>

#include "../../include/brokefish_b200.h"

namespace py = pybind11;
using at::Tensor;

namespace {

constexpr int64_t kMaxHistory = 100;

#define BF_FUNCTIONS(X)                                                                       \
    X(bf_movegen) X(bf_step) X(bf_hash) X(bf_history_push_to) X(bf_repetition_count) X(bf_terminal) \
    X(bf_terminal_history) X(bf_forward) X(bf_forward_priors) X(bf_forward_leaves) X(bf_forward_host) \
    X(bf_forward_priors_host)
struct Api {
#define X(name) decltype(&::name) name = nullptr;
    BF_FUNCTIONS(X)
#undef X
};
Api g_api;
PyObject* g_check = nullptr;        // _native.check(rc, what), kept for the life of the process

void bind(const std::string& path, py::object check) {
    void* lib = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
    if (lib == nullptr) throw std::runtime_error(std::string("cannot open ") + path + ": " + dlerror());
#define X(name)                                                                      \
    g_api.name = reinterpret_cast<decltype(&::name)>(dlsym(lib, #name));              \
    if (g_api.name == nullptr) throw std::runtime_error(std::string(#name) + " is missing from " + path);
    BF_FUNCTIONS(X)
#undef X
    g_check = check.release().ptr();
}

// Runs a C-ABI call without the interpreter lock (a launch waits when the GPU's queue is full) and
// turns a failure into the exception that the Python layer raises for it.
template <class F>
void call(const char* what, F&& f) {
    int rc;
    {
        py::gil_scoped_release release;
        rc = f();
    }
    if (rc != 0) py::reinterpret_borrow<py::object>(g_check)(rc, what);
}

std::string shape_text(const Tensor& t) {
    std::ostringstream s;
    s << "(";
    for (int64_t i = 0; i < t.dim(); ++i) s << (i ? ", " : "") << t.size(i);
    s << (t.dim() == 1 ? ",)" : ")");
    return s.str();
}
std::string dtype_text(const Tensor& t) {
    return py::str(py::cast(t).attr("dtype")).cast<std::string>();
}
std::string device_text(const Tensor& t) { return t.device().str(); }

template <class T = void>
T* ptr(const Tensor& t) {
    return t.defined() && t.numel() ? static_cast<T*>(t.data_ptr()) : nullptr;
}
void* stream_of(c10::Device d) { return c10::cuda::getCurrentCUDAStream(d.index()).stream(); }
// An output on the inputs' device.  Straight from the allocator: through the dispatcher, `at::empty`, one takes 0.73 us
// instead of 0.52, and a ply of games makes ten of them in 20 us.  (So dispatch modes do not see it, and
// `torch.utils.deterministic.fill_uninitialized_memory` does not fill it; the kernels write every element.)
Tensor output(at::IntArrayRef size, at::ScalarType type, const Tensor& like) {
    return at::detail::empty_cuda(size, type, like.device(), std::nullopt);
}
bool is_vector(const Tensor& t, int64_t n) { return t.dim() == 1 && t.size(0) == n; }

// ---- the engine ----
int64_t check_position(const Tensor& boards, const Tensor& control, const char* no_cpu) {
    const int64_t n = boards.dim() ? boards.size(0) : 0;
    if (boards.dim() != 2 || boards.size(1) != 32 || boards.scalar_type() != at::kShort)
        throw py::value_error("boards must be [n, 32] int16, got " + shape_text(boards) + " " + dtype_text(boards));
    if (!is_vector(control, n) || control.scalar_type() != at::kShort)
        throw py::value_error("control must be [" + std::to_string(n) + "] int16, got " + shape_text(control) + " " + dtype_text(control));
    if (!boards.is_cuda() || !control.is_cuda() || boards.device() != control.device()) throw py::value_error(no_cpu);
    return n;
}
constexpr const char* kNoCpu = "the engine kernels take CUDA tensors on one device; there is no CPU path";

py::tuple movegen(const Tensor& boards, const Tensor& control) {
    const int64_t n = check_position(boards, control, "movegen takes CUDA tensors on one device; there is no CPU path");
    Tensor mask = output({n, 32}, at::kLong, boards), check = output({n}, at::kBool, boards);
    if (n) {
        const Tensor b = boards.contiguous(), c = control.contiguous();
        call("bf_movegen", [&] {
            return g_api.bf_movegen(b.device().index(), ptr<uint16_t>(b), ptr<int16_t>(c), static_cast<int>(n),
                                    ptr<uint64_t>(mask), ptr<unsigned char>(check), stream_of(b.device()));
        });
    }
    return py::make_tuple(mask, check);
}

// (boards, control, key or None, irreversible[, legal words, check flag])
py::tuple step(const Tensor& boards, const Tensor& control, const Tensor& move, const std::optional<Tensor>& promo,
               bool with_moves, bool with_hash) {
    const int64_t n = check_position(boards, control, kNoCpu);
    if (!is_vector(move, n) || !move.is_cuda())
        throw py::value_error("move must be a CUDA tensor of shape [" + std::to_string(n) + "]");
    const auto o = boards.options();
    const Tensor mv = move.to(at::kInt).contiguous();
    Tensor pr;
    if (promo) {
        pr = promo->to(o.dtype(at::kChar)).contiguous();
        if (!is_vector(pr, n)) throw py::value_error("promo must have shape [" + std::to_string(n) + "]");
    }
    Tensor nb = output({n, 32}, at::kShort, boards), nc = output({n}, at::kShort, boards), irr = output({n}, at::kBool, boards);
    Tensor mask, check, key;
    if (with_moves) {
        mask = output({n, 32}, at::kLong, boards);
        check = output({n}, at::kBool, boards);
    }
    if (with_hash) key = output({n}, at::kLong, boards);
    if (n) {
        const Tensor b = boards.contiguous(), c = control.contiguous();
        call("bf_step", [&] {
            return g_api.bf_step(b.device().index(), ptr<uint16_t>(b), ptr<int16_t>(c), ptr<int>(mv), ptr<signed char>(pr),
                                 static_cast<int>(n), ptr<uint16_t>(nb), ptr<int16_t>(nc), ptr<unsigned char>(irr),
                                 ptr<uint64_t>(mask), ptr<unsigned char>(check), ptr<uint64_t>(key), stream_of(b.device()));
        });
    }
    const py::object k = with_hash ? py::cast(key) : py::none();
    return with_moves ? py::make_tuple(nb, nc, k, irr, mask, check) : py::make_tuple(nb, nc, k, irr);
}

Tensor hash_position(const Tensor& boards, const Tensor& control) {
    const int64_t n = check_position(boards, control, kNoCpu);
    Tensor key = output({n}, at::kLong, boards);
    if (n) {
        const Tensor b = boards.contiguous(), c = control.contiguous();
        call("bf_hash", [&] {
            return g_api.bf_hash(b.device().index(), ptr<uint16_t>(b), ptr<int16_t>(c), static_cast<int>(n),
                                 ptr<uint64_t>(key), stream_of(b.device()));
        });
    }
    return key;
}

// A flag tensor as bytes: bools are bytes already, anything else is converted.
Tensor bytes_of(const Tensor& flags) {
    return flags.scalar_type() == at::kBool ? flags.contiguous() : flags.to(at::kByte).contiguous();
}

py::tuple push_history(const Tensor& ring, const Tensor& length, const Tensor& hash, const Tensor& irreversible) {
    const int64_t n = ring.dim() ? ring.size(0) : 0;
    if (ring.dim() != 2 || ring.size(1) != kMaxHistory || ring.scalar_type() != at::kLong || !ring.is_cuda())
        throw py::value_error("ring must be a CUDA int64 tensor [n, 100]");
    if (!is_vector(length, n) || length.scalar_type() != at::kLong || !is_vector(hash, n) ||
        hash.scalar_type() != at::kLong || !is_vector(irreversible, n))
        throw py::value_error("length, hash [n] int64 and irreversible [n] are needed");
    if (length.device() != ring.device() || hash.device() != ring.device() || irreversible.device() != ring.device())
        throw py::value_error("ring, length, hash and irreversible must live on one device");
    Tensor new_ring = output({n, kMaxHistory}, at::kLong, ring), new_length = output({n}, at::kLong, ring);
    if (n) {
        const Tensor r = ring.contiguous(), l = length.contiguous(), h = hash.contiguous(), irr = bytes_of(irreversible);
        call("bf_history_push_to", [&] {
            return g_api.bf_history_push_to(r.device().index(), ptr<uint64_t>(r), reinterpret_cast<long long*>(ptr<int64_t>(l)),
                                            ptr<uint64_t>(h), ptr<unsigned char>(irr), static_cast<int>(n), ptr<uint64_t>(new_ring),
                                            reinterpret_cast<long long*>(ptr<int64_t>(new_length)), stream_of(r.device()));
        });
    }
    return py::make_tuple(new_ring, new_length);
}

void check_history(const Tensor& hash, const Tensor& ring, const Tensor& length, int64_t n) {
    if (ring.dim() != 2 || ring.size(0) != n || ring.size(1) != kMaxHistory || ring.scalar_type() != at::kLong || !ring.is_cuda())
        throw py::value_error("ring must be a CUDA int64 tensor [n, 100]");
    if (!is_vector(hash, n) || hash.scalar_type() != at::kLong || hash.device() != ring.device() || !is_vector(length, n) ||
        length.scalar_type() != at::kLong || length.device() != ring.device())
        throw py::value_error("hash and length must be [n] int64 tensors on the ring's device");
}

Tensor repetition_count(const Tensor& hash, const Tensor& ring, const Tensor& length) {
    const int64_t n = ring.dim() ? ring.size(0) : 0;
    check_history(hash, ring, length, n);
    Tensor count = output({n}, at::kInt, ring);
    if (n) {
        const Tensor h = hash.contiguous(), r = ring.contiguous(), l = length.contiguous();
        call("bf_repetition_count", [&] {
            return g_api.bf_repetition_count(r.device().index(), ptr<uint64_t>(h), ptr<uint64_t>(r),
                                             reinterpret_cast<long long*>(ptr<int64_t>(l)), static_cast<int>(n), ptr<int>(count),
                                             stream_of(r.device()));
        });
    }
    return count.to(at::kLong);
}

py::tuple terminal(const Tensor& mask, const Tensor& in_check, const Tensor& control, const Tensor& boards,
                   const std::optional<Tensor>& hash, const std::optional<Tensor>& ring, const std::optional<Tensor>& length) {
    const int64_t n = check_position(boards, control, kNoCpu);
    const bool history = hash && ring && length;
    if (history) check_history(*hash, *ring, *length, n);
    if (mask.dim() != 2 || mask.size(0) != n || mask.size(1) != 32 || mask.scalar_type() != at::kLong || !mask.is_cuda())
        throw py::value_error("mask must be a CUDA int64 tensor of shape [" + std::to_string(n) + ", 32]");
    if (!is_vector(in_check, n) || !in_check.is_cuda())
        throw py::value_error("in_check must be a CUDA tensor of shape [" + std::to_string(n) + "]");
    Tensor code = output({n}, at::kByte, boards), result = output({n}, at::kChar, boards);
    if (n) {
        const Tensor m = mask.contiguous(), chk = bytes_of(in_check), c = control.contiguous(), b = boards.contiguous();
        const int dev = b.device().index(), count = static_cast<int>(n);
        if (history) {
            const Tensor h = hash->contiguous(), r = ring->contiguous(), l = length->contiguous();
            call("bf_terminal_history", [&] {
                return g_api.bf_terminal_history(dev, ptr<uint64_t>(m), ptr<unsigned char>(chk), ptr<int16_t>(c), ptr<uint16_t>(b),
                                                 ptr<uint64_t>(h), ptr<uint64_t>(r), reinterpret_cast<long long*>(ptr<int64_t>(l)),
                                                 count, ptr<unsigned char>(code), ptr<signed char>(result), stream_of(b.device()));
            });
        } else {
            call("bf_terminal", [&] {
                return g_api.bf_terminal(dev, ptr<uint64_t>(m), ptr<unsigned char>(chk), ptr<int16_t>(c), ptr<uint16_t>(b), nullptr,
                                         count, ptr<unsigned char>(code), ptr<signed char>(result), stream_of(b.device()));
            });
        }
    }
    return py::make_tuple(code, result);
}

// ---- the evaluator's device-resident calls; outputs are the caller's buffers ----
int64_t check_inputs(const Tensor& boards, const Tensor& control, const Tensor& rep) {
    const int64_t n = boards.dim() ? boards.size(0) : 0;
    if (boards.dim() != 2 || boards.size(1) != 32)
        throw py::value_error("boards must be [n, 32], got " + shape_text(boards));
    if (boards.scalar_type() != at::kShort) throw py::value_error("boards must be int16, got " + dtype_text(boards));
    if (!is_vector(control, n) || control.scalar_type() != at::kShort)
        throw py::value_error("control must be [" + std::to_string(n) + "] int16, got " + shape_text(control) + " " + dtype_text(control));
    if (!is_vector(rep, n) || rep.scalar_type() != at::kByte)
        throw py::value_error("rep must be [" + std::to_string(n) + "] uint8, got " + shape_text(rep) + " " + dtype_text(rep));
    return n;
}
void check_device(const Tensor& t, int device) {
    if (!t.is_cuda() || t.device().index() != device)
        throw py::value_error("inputs must live on cuda:" + std::to_string(device) + ", got " + device_text(t));
}
// The legality words, checked: contiguous or undefined.
Tensor check_legal(const std::optional<Tensor>& legal, int64_t n, int device) {
    if (!legal) return Tensor();
    check_device(*legal, device);
    if (legal->dim() != 2 || legal->size(0) != n || legal->size(1) != 32 || legal->scalar_type() != at::kLong)
        throw py::value_error("legal must be [" + std::to_string(n) + ", 32] int64, got " + shape_text(*legal) + " " + dtype_text(*legal));
    return legal->contiguous();
}
bf_handle* handle_of(int64_t h) { return reinterpret_cast<bf_handle*>(h); }

// Checks of the three calls' inputs before any buffer is made for them; returns n.
int64_t check_evaluation(int device, const Tensor& boards, const Tensor& control, const Tensor& rep,
                         const std::optional<Tensor>& legal) {
    const int64_t n = check_inputs(boards, control, rep);
    check_device(boards, device);
    check_device(control, device);
    check_device(rep, device);
    if (legal) (void)check_legal(legal, n, device);
    return n;
}

void forward(int64_t handle, const Tensor& boards, const Tensor& control, const Tensor& rep, const std::optional<Tensor>& legal,
             const Tensor& policy, const Tensor& promo, const Tensor& value) {
    const Tensor b = boards.contiguous(), c = control.contiguous(), r = rep.contiguous();
    const Tensor lg = legal ? legal->contiguous() : Tensor();
    call("bf_forward", [&] {
        return g_api.bf_forward(handle_of(handle), ptr<uint16_t>(b), ptr<int16_t>(c), ptr<uint8_t>(r), ptr<uint64_t>(lg),
                                static_cast<int>(b.size(0)), ptr(policy), ptr(promo), ptr<float>(value), stream_of(value.device()));
    });
}

void forward_priors(int64_t handle, const Tensor& boards, const Tensor& control, const Tensor& rep,
                    const std::optional<Tensor>& legal, int e_cap, const Tensor& prior, const Tensor& move, const Tensor& nedges,
                    const Tensor& value, const std::optional<Tensor>& policy, const std::optional<Tensor>& promo) {
    const Tensor b = boards.contiguous(), c = control.contiguous(), r = rep.contiguous();
    const Tensor lg = legal ? legal->contiguous() : Tensor();
    call("bf_forward_priors", [&] {
        return g_api.bf_forward_priors(handle_of(handle), ptr<uint16_t>(b), ptr<int16_t>(c), ptr<uint8_t>(r), ptr<uint64_t>(lg),
                                       static_cast<int>(b.size(0)), e_cap, ptr(prior), ptr<int16_t>(move), ptr<int>(nedges),
                                       ptr<float>(value), policy ? ptr(*policy) : nullptr, promo ? ptr(*promo) : nullptr,
                                       stream_of(value.device()));
    });
}

void forward_leaves(int64_t handle, const Tensor& boards, const Tensor& control, const Tensor& rep, const Tensor& leaf_index,
                    const Tensor& leaf_count, const std::optional<Tensor>& legal, const std::optional<Tensor>& policy,
                    const std::optional<Tensor>& promo, const Tensor& value, int e_cap, const std::optional<Tensor>& prior,
                    const std::optional<Tensor>& move, const std::optional<Tensor>& nedges) {
    const Tensor b = boards.contiguous(), c = control.contiguous(), r = rep.contiguous(), li = leaf_index.contiguous();
    const Tensor lg = legal ? legal->contiguous() : Tensor();
    call("bf_forward_leaves", [&] {
        return g_api.bf_forward_leaves(handle_of(handle), ptr<uint16_t>(b), ptr<int16_t>(c), ptr<uint8_t>(r), ptr<uint64_t>(lg),
                                       ptr<int>(li), ptr<int>(leaf_count), static_cast<int>(li.size(0)),
                                       policy ? ptr(*policy) : nullptr, promo ? ptr(*promo) : nullptr, ptr<float>(value), e_cap,
                                       prior ? ptr(*prior) : nullptr, move ? ptr<int16_t>(*move) : nullptr,
                                       nedges ? ptr<int>(*nedges) : nullptr, stream_of(value.device()));
    });
}

// ---- the host-buffer calls ----
void check_host(std::initializer_list<const Tensor*> tensors, const char* text) {
    for (const Tensor* t : tensors)
        if (t->is_cuda() || !t->is_contiguous()) throw py::value_error(text);
}
void forward_host(int64_t handle, const Tensor& boards, const Tensor& control, const Tensor& rep, const Tensor& policy,
                  const Tensor& promo, const Tensor& value, const std::optional<Tensor>& legal) {
    const int n = static_cast<int>(check_inputs(boards, control, rep));
    check_host({&boards, &control, &rep, &policy, &promo, &value}, "forward_host takes contiguous CPU tensors");
    call("bf_forward_host", [&] {
        return g_api.bf_forward_host(handle_of(handle), ptr<uint16_t>(boards), ptr<int16_t>(control), ptr<uint8_t>(rep),
                                     legal ? ptr<uint64_t>(*legal) : nullptr, n, ptr(policy), ptr(promo), ptr<float>(value));
    });
}
void forward_priors_host(int64_t handle, const Tensor& boards, const Tensor& control, const Tensor& rep, const Tensor& legal,
                         const Tensor& prior, const Tensor& move, const Tensor& nedges, const Tensor& value) {
    const int64_t n = check_inputs(boards, control, rep);
    check_host({&boards, &control, &rep, &legal, &prior, &move, &nedges, &value}, "forward_priors_host takes contiguous CPU tensors");
    const int64_t e_cap = prior.dim() > 1 ? prior.size(1) : -1;
    if (legal.dim() != 2 || legal.size(0) != n || legal.size(1) != 32 || legal.scalar_type() != at::kLong || move.dim() != 2 ||
        move.size(0) != n || move.size(1) != e_cap || move.scalar_type() != at::kShort || prior.scalar_type() != at::kHalf ||
        !is_vector(nedges, n) || nedges.scalar_type() != at::kInt || !is_vector(value, n) || value.scalar_type() != at::kFloat)
        throw py::value_error("forward_priors_host: legal [n,32] int64, prior [n,E] fp16, move [n,E] int16, "
                              "nedges [n] int32, value [n] fp32");
    call("bf_forward_priors_host", [&] {
        return g_api.bf_forward_priors_host(handle_of(handle), ptr<uint16_t>(boards), ptr<int16_t>(control), ptr<uint8_t>(rep),
                                            ptr<uint64_t>(legal), static_cast<int>(n), static_cast<int>(e_cap), ptr(prior),
                                            ptr<int16_t>(move), ptr<int>(nedges), ptr<float>(value));
    });
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("bind", &bind);
    m.def("movegen", &movegen);
    m.def("step", &step);
    m.def("hash_position", &hash_position);
    m.def("push_history", &push_history);
    m.def("repetition_count", &repetition_count);
    m.def("terminal", &terminal);
    m.def("check_evaluation", &check_evaluation);
    m.def("forward", &forward);
    m.def("forward_priors", &forward_priors);
    m.def("forward_leaves", &forward_leaves);
    m.def("forward_host", &forward_host);
    m.def("forward_priors_host", &forward_priors_host);
}
