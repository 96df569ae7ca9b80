// The host path of the Python operators (blockedattention_b200/apply.py): everything between a call and its kernel
// launches in native code -- argument checks, the lists' values, the plan, the result, autograd nodes.
//
// Why native: an operator on a small batch takes a few microseconds on the GPU, and the same steps in Python (tuple
// keys, ctypes conversions, device context managers, array copies of the lists) took 15 to 20 us a call, several times
// that in a backward pass.  Here a call whose lists were seen before does a handful of hash lookups.
//
// Lists are interned: equal values share one List object, so a plan's key holds pointers.  A list tensor on the GPU is
// read to the host once and remembered while it is alive (a bounded number of them; the memo holds the tensor, so its
// address cannot come back with other values, and an in-place write moves its version).  Lists on the host (numpy
// arrays, CPU tensors, sequences) are compared by value on every call.
//
// An operator holds the lock of Python while it looks at its arguments and lets go of it for everything after: reading a
// list from the GPU, creating and releasing plans and a full launch queue all wait for the device, and the process's other
// threads must not wait with them.
#include <Python.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>

#include <cstdlib>
#include <cstring>
#include <initializer_list>
#include <list>
#include <memory>
#include <mutex>
#include <string>
#include <unordered_map>
#include <utility>
#include <vector>

#include "blkattn.h"

namespace {

using at::Tensor;

// The lock of Python, let go of for a scope.
struct NoGil {
    PyThreadState* state;
    NoGil() : state(PyEval_SaveThread()) {}
    ~NoGil() { PyEval_RestoreThread(state); }
    NoGil(const NoGil&) = delete;
    NoGil& operator=(const NoGil&) = delete;
};

struct PyRef {
    PyObject* o;
    explicit PyRef(PyObject* x) : o(x) {}
    ~PyRef() { Py_XDECREF(o); }
    PyRef(const PyRef&) = delete;
    PyRef& operator=(const PyRef&) = delete;
};

PyObject* g_host_i64 = nullptr;  // plan._host_i64: any sequence -> contiguous int64 numpy array
PyObject* g_error = nullptr;     // _lib.BlkError
PyObject* g_traced = nullptr;    // apply._traced(operator, number of operands, arguments)

// A failed library call: blockedattention_b200._lib.BlkError, whatever thread it happens on -- the caller of an operator
// gets it from the entry below, the caller of a backward pass from torch's engine.
[[noreturn]] void fail(int code) {
    const std::string text = blk_last_error();
    const PyGILState_STATE held = PyGILState_Ensure();
    {
        PyRef err(PyObject_CallFunction(g_error, "is", code, text.c_str()));
        if (err.o) PyErr_SetObject(g_error, err.o);
    }
    python_error e;
    e.persist();
    PyGILState_Release(held);
    throw e;
}
inline void ok(int rc) {
    if (rc != BLK_OK) fail(rc);
}

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kHalf: return BLK_F16;
        case at::kBFloat16: return BLK_BF16;
        case at::kFloat: return BLK_F32;
        default: break;
    }
    TORCH_CHECK(false, "blockedattention_b200: dtype ", t, " is not supported (float16, bfloat16, float32)");
}

// ---- lists -------------------------------------------------------------------------------------------
struct List {
    std::vector<int64_t> v;
};
typedef std::shared_ptr<const List> ListP;

// Four independent multiply-add lanes: the lists of a batch of thousands of segments hash at memory speed.
uint64_t hash_values(const int64_t* p, size_t n) {
    const uint64_t m = 0x9E3779B97F4A7C15ull;
    uint64_t h[4] = {n, n ^ m, ~n, n + m};
    size_t i = 0;
    for (; i + 4 <= n; i += 4)
        for (int j = 0; j < 4; ++j) h[j] = (h[j] ^ (uint64_t)p[i + j]) * m + (h[j] >> 29);
    for (; i < n; ++i) h[0] = (h[0] ^ (uint64_t)p[i]) * m + (h[0] >> 29);
    uint64_t r = 0;
    for (int j = 0; j < 4; ++j) r = (r ^ h[j] ^ (h[j] >> 32)) * m;
    return r ^ (r >> 31);
}

std::mutex g_mu;  // guards the tables below; no plan or tensor is released and nothing of Python called while it is held

// Interned values.  Owners are plans and the memo of GPU list tensors; expired entries are swept as the table grows.
struct Interned {
    std::unordered_multimap<uint64_t, std::weak_ptr<const List>> table;
    size_t sweep_at = 64;
    ListP get(const int64_t* p, size_t n) {
        const uint64_t h = hash_values(p, n);
        auto range = table.equal_range(h);
        for (auto it = range.first; it != range.second; ++it)
            if (ListP l = it->second.lock())
                if (l->v.size() == n && (n == 0 || std::memcmp(l->v.data(), p, n * sizeof(int64_t)) == 0)) return l;
        if (table.size() >= sweep_at) {
            for (auto it = table.begin(); it != table.end();) it = it->second.expired() ? table.erase(it) : std::next(it);
            sweep_at = 64 + 2 * table.size();
        }
        auto l = std::make_shared<List>();
        l->v.assign(p, p + n);
        table.emplace(h, l);
        return l;
    }
};
Interned& interned() {
    static Interned* t = new Interned();
    return *t;
}

struct TensorKey {
    const void* ptr;
    int64_t version, numel, stride;
    int dtype, device;
    bool operator==(const TensorKey& o) const {
        return ptr == o.ptr && version == o.version && numel == o.numel && stride == o.stride && dtype == o.dtype && device == o.device;
    }
};
struct TensorKeyHash {
    size_t operator()(const TensorKey& k) const {
        return (size_t)(((uintptr_t)k.ptr >> 4) * 0x9E3779B97F4A7C15ull) ^ (size_t)(k.version * 1000003 + k.numel * 31 + k.stride * 7 + k.device);
    }
};

// Least recently used entries of a bounded map.
template <typename K, typename V, typename Hash>
struct Lru {
    typedef std::list<std::pair<K, V>> Order;
    Order order;
    std::unordered_map<K, typename Order::iterator, Hash> index;
    size_t most;
    explicit Lru(size_t n) : most(n) {}
    V* find(const K& k) {
        auto it = index.find(k);
        if (it == index.end()) return nullptr;
        if (it->second != order.begin()) order.splice(order.begin(), order, it->second);
        return &it->second->second;
    }
    // what falls out is handed back, to be released outside the lock
    void put(const K& k, V v, std::vector<V>* dropped) {
        order.emplace_front(k, std::move(v));
        index[k] = order.begin();
        while (order.size() > most) {
            dropped->push_back(std::move(order.back().second));
            index.erase(order.back().first);
            order.pop_back();
        }
    }
    void clear(std::vector<V>* dropped) {
        for (auto& e : order) dropped->push_back(std::move(e.second));
        index.clear();
        order.clear();
    }
};

struct Remembered {
    Tensor keep;
    ListP list;
};
Lru<TensorKey, Remembered, TensorKeyHash>& device_lists() {
    static auto* t = new Lru<TensorKey, Remembered, TensorKeyHash>(256);
    return *t;
}

ListP list_of_tensor(const Tensor& t) {
    const bool remember = t.is_cuda() && !t.is_inference();
    TensorKey key{};
    if (remember) {
        key = TensorKey{t.data_ptr(), (int64_t)t._version(), t.numel(), t.dim() ? t.stride(-1) : 1, (int)t.scalar_type(), (int)t.get_device()};
        std::lock_guard<std::mutex> g(g_mu);
        if (Remembered* r = device_lists().find(key))
            if (r->keep.strides() == t.strides() && r->keep.sizes() == t.sizes()) return r->list;
    }
    const Tensor h = t.detach().to(at::kCPU, at::kLong).contiguous();  // for a GPU list: the one copy of its values
    std::vector<Remembered> dropped;
    std::lock_guard<std::mutex> g(g_mu);
    ListP l = interned().get(h.data_ptr<int64_t>(), (size_t)h.numel());
    if (remember && !device_lists().find(key)) device_lists().put(key, Remembered{t, l}, &dropped);
    return l;
}

// A list argument: the values, or the tensor they are to be read from (both unset for None).
struct ListArg {
    ListP values;
    Tensor tensor;
    explicit operator bool() const { return values || tensor.defined(); }
    ListP read() const { return tensor.defined() ? list_of_tensor(tensor) : values; }
};
ListArg list_of(PyObject* o) {
    if (o == Py_None) return {};
    if (THPVariable_Check(o)) return {nullptr, THPVariable_Unpack(o)};
    auto from_buffer = [](PyObject* x, ListP* out) -> bool {
        Py_buffer b;
        if (PyObject_GetBuffer(x, &b, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT) != 0) {
            PyErr_Clear();
            return false;
        }
        const bool is64 = b.itemsize == 8 && b.format && (std::strcmp(b.format, "l") == 0 || std::strcmp(b.format, "q") == 0);
        if (is64) {
            std::lock_guard<std::mutex> g(g_mu);
            *out = interned().get(static_cast<const int64_t*>(b.buf), (size_t)(b.len / 8));
        }
        PyBuffer_Release(&b);
        return is64;
    };
    ListP l;
    if (PyObject_CheckBuffer(o) && from_buffer(o, &l)) return {l, {}};
    PyRef arr(PyObject_CallFunctionObjArgs(g_host_i64, o, nullptr));
    if (!arr.o) throw python_error();
    TORCH_CHECK(from_buffer(arr.o, &l), "a list or offset argument cannot be read as int64 values");
    return {l, {}};
}

// ---- plans -------------------------------------------------------------------------------------------
struct Plan {
    blk_plan_t* h = nullptr;
    ListP lists[6];              // M, N, K, mat1Accum, mat2Accum, outAccum as given: they keep the key's pointers valid
    std::vector<int64_t> M, N, K;
    int64_t S = 0, H = 0, Dm1 = 0, Dm2 = 0, Dout = 0, rows_q = 0, rows_kv = 0, d = 0;
    at::ScalarType dt = at::kHalf, odt = at::kHalf;
    bool ta = false, tb = false, softmax = false, compose = false;
    c10::Device device = c10::Device(c10::kCUDA, 0);
    // plans of the backward pass and of compositions, made when first needed; index: purpose, type
    std::shared_ptr<Plan> derived[5][3];
    ~Plan() {
        if (!h) return;
        // (the last owner may be an autograd node that Python releases; freeing device memory waits for the device)
        if (Py_IsInitialized() && PyGILState_Check()) {
            NoGil free;
            blk_plan_destroy(h);
        } else {
            blk_plan_destroy(h);
        }
    }
    void extents() { ok(blk_plan_extents(h, &Dm1, &Dm2, &Dout)); }
    void check(cudaStream_t st) const {
        if (h) ok(blk_plan_check(h, st));
    }
};
typedef std::shared_ptr<Plan> PlanP;

enum Purpose { FOR_GRAD1 = 0, FOR_GRAD2, FOR_SOFTMAX, FOR_SCORES, FOR_PRODUCT };

struct PlanKey {
    int op, dt, odt, flags, device, d;
    int64_t numel;
    const List* l[6];
    bool operator==(const PlanKey& o) const { return std::memcmp(this, &o, sizeof(PlanKey)) == 0; }
};
static_assert(sizeof(PlanKey) == 6 * sizeof(int) + 8 + 6 * sizeof(void*), "PlanKey is compared as bytes: no padding");
struct PlanKeyHash {
    size_t operator()(const PlanKey& k) const {
        uint64_t h = (uint64_t)(k.op * 7 + k.dt * 5 + k.odt * 3 + k.flags) * 0x9E3779B97F4A7C15ull + (uint64_t)k.numel + (uint64_t)k.d * 131;
        for (const List* l : k.l) h = (h ^ (uint64_t)(uintptr_t)l) * 0xC2B2AE3D27D4EB4Full + (h >> 31);
        return (size_t)(h ^ k.device);
    }
};
Lru<PlanKey, PlanP, PlanKeyHash>& plans() {
    static auto* t = new Lru<PlanKey, PlanP, PlanKeyHash>(32);
    return *t;
}

template <typename Make>
PlanP plan_for(const PlanKey& key, Make make) {
    {
        std::lock_guard<std::mutex> g(g_mu);
        if (PlanP* p = plans().find(key)) return *p;
    }
    PlanP p = make();  // outside the lock: creating a plan uploads its tables
    std::vector<PlanP> dropped;
    std::lock_guard<std::mutex> g(g_mu);
    if (PlanP* q = plans().find(key)) return *q;
    plans().put(key, p, &dropped);
    return p;
}

template <typename Make>
PlanP derived(const PlanP& p, Purpose what, at::ScalarType t, Make make) {
    const int i = dtype_code(t);
    {
        std::lock_guard<std::mutex> g(g_mu);
        if (p->derived[what][i]) return p->derived[what][i];
    }
    PlanP q = make();
    std::lock_guard<std::mutex> g(g_mu);
    if (!p->derived[what][i]) p->derived[what][i] = q;
    return p->derived[what][i];
}

PlanP make_gemm(const int64_t* M, const int64_t* N, const int64_t* K, int64_t S, const int64_t* a1, const int64_t* a2,
                const int64_t* ao, int64_t H, at::ScalarType dt, at::ScalarType odt, bool ta, bool tb, bool softmax,
                c10::Device dev) {
    auto p = std::make_shared<Plan>();
    p->M.assign(M, M + S);
    p->N.assign(N, N + S);
    p->K.assign(K, K + S);
    p->S = S;
    p->H = H;
    p->dt = dt;
    p->odt = odt;
    p->ta = ta;
    p->tb = tb;
    p->softmax = softmax;
    p->device = dev;
    ok(blk_gemm_plan_create(&p->h, M, N, K, a1, a2, ao, S, H, dtype_code(dt), dtype_code(odt), ta, tb,
                            softmax ? BLK_EPI_SOFTMAX : BLK_EPI_SCORES, dev.index()));
    p->extents();
    return p;
}

PlanP make_softmax(const std::vector<int64_t>& rows, const std::vector<int64_t>& cols, const int64_t* acc, int64_t H,
                   at::ScalarType dt, c10::Device dev) {
    auto p = std::make_shared<Plan>();
    p->M = rows;
    p->N = cols;
    p->S = (int64_t)rows.size();
    p->H = H;
    p->dt = p->odt = dt;
    p->device = dev;
    ok(blk_softmax_plan_create(&p->h, rows.data(), cols.data(), acc, p->S, H, dtype_code(dt), dev.index()));
    p->extents();
    return p;
}

// ---- running -----------------------------------------------------------------------------------------
void check_operand(const char* name, const Tensor& t) {
    // the two TORCH_CHECKs of upstream csrc/sparseBlockedAttention.h:6-8
    TORCH_CHECK(t.defined() && t.is_cuda(), name, " must be CUDA Tensor");
    TORCH_CHECK(t.is_contiguous(), name, " must be contiguous Tensor");
}

inline bool unaligned(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) != 0; }
inline Tensor aligned(const Tensor& t) { return unaligned(t) ? t.clone() : t; }
inline cudaStream_t stream_of(c10::Device d) { return c10::cuda::getCurrentCUDAStream(d.index()).stream(); }
inline Tensor empty2(int64_t a, int64_t b, at::ScalarType t, c10::Device d) {
    const int64_t s[2] = {a, b};
    return at::detail::empty_cuda(at::IntArrayRef(s, 2), t, d, std::nullopt);
}
// BLK_CHECK=1 reads the status word back after every run (a debugging switch, see plan.py)
inline void after_run(const Plan& p, cudaStream_t st) {
    const char* e = std::getenv("BLK_CHECK");
    if (e && e[0] && std::strcmp(e, "0") != 0) p.check(st);
}

// What a kernel is about to read through a raw pointer: looked at before every run, since an operand of a backward pass may
// come from a saved-tensor hook of the caller's.
void check_input(const char* name, const Tensor& t, at::ScalarType dt, int64_t H, int64_t D) {
    check_operand(name, t);
    TORCH_CHECK(t.scalar_type() == dt, name, " has dtype ", t.scalar_type(), ", the plan was built for ", dt);
    TORCH_CHECK(t.numel() == H * D, name, " has ", t.numel(), " elements, expected H*D = ", H, "*", D);
}

Tensor run_gemm(const Plan& p, const Tensor& m1, const Tensor& m2, double scale) {
    check_input("mat1", m1, p.dt, p.H, p.Dm1);
    check_input("mat2", m2, p.dt, p.H, p.Dm2);
    c10::cuda::CUDAGuard guard(p.device);
    const Tensor a = aligned(m1), b = aligned(m2);
    Tensor out = empty2(p.H, p.Dout, p.odt, p.device);
    cudaStream_t st = stream_of(p.device);
    ok(blk_gemm_run(p.h, a.data_ptr(), b.data_ptr(), out.data_ptr(), (float)scale, st));
    after_run(p, st);
    return out;
}

Tensor run_softmax(const Plan& p, const Tensor& src, const Tensor* into, double scale) {
    check_input("src", src, p.dt, p.H, p.Dm1);
    Tensor out;
    c10::cuda::CUDAGuard guard(p.device);
    if (into) {
        TORCH_CHECK(into->is_cuda() && into->is_contiguous() && into->scalar_type() == p.dt && into->numel() == src.numel(),
                    "out must be a contiguous CUDA tensor shaped like src");
        TORCH_CHECK(!unaligned(*into), "out must be 16-byte aligned");
        out = *into;
    } else {
        out = empty2(p.H, p.Dm1, p.dt, p.device);
    }
    const Tensor s = aligned(src);
    cudaStream_t st = stream_of(p.device);
    ok(blk_softmax_run(p.h, s.data_ptr(), out.data_ptr(), (float)scale, st));
    after_run(p, st);
    return out;
}

Tensor run_softmax_backward(const Plan& p, const Tensor& result, const Tensor& grad, double scale) {
    check_input("the softmax result", result, p.dt, p.H, p.Dm1);
    check_input("the gradient", grad, p.dt, p.H, p.Dm1);
    c10::cuda::CUDAGuard guard(p.device);
    const Tensor r = aligned(result), g = aligned(grad);
    Tensor out = empty2(p.H, p.Dm1, p.dt, p.device);
    cudaStream_t st = stream_of(p.device);
    ok(blk_softmax_backward_run(p.h, r.data_ptr(), g.data_ptr(), out.data_ptr(), (float)scale, st));
    after_run(p, st);
    return out;
}

Tensor run_attention(const Plan& p, const Tensor& q, const Tensor& k, const Tensor& v, double scale, bool tokens,
                     Tensor* lse = nullptr) {
    check_input("q", q, p.dt, p.H, p.rows_q * p.d);
    check_input("k", k, p.dt, p.H, p.rows_kv * p.d);
    check_input("v", v, p.dt, p.H, p.rows_kv * p.d);
    c10::cuda::CUDAGuard guard(p.device);
    const Tensor a = aligned(q), b = aligned(k), c = aligned(v);
    cudaStream_t st = stream_of(p.device);
    Tensor out;
    if (tokens) {
        const int64_t s[3] = {p.rows_q, p.H, p.d};
        out = at::detail::empty_cuda(at::IntArrayRef(s, 3), p.dt, p.device, std::nullopt);
        ok(blk_attention_run_strided(p.h, a.data_ptr(), b.data_ptr(), c.data_ptr(), out.data_ptr(), p.H * p.d, p.d, (float)scale, st));
    } else {
        out = empty2(p.H, p.rows_q * p.d, p.dt, p.device);
        if (lse) *lse = empty2(p.H, p.rows_q, at::kFloat, p.device);
        ok(blk_attention_run_lse(p.h, a.data_ptr(), b.data_ptr(), c.data_ptr(), out.data_ptr(),
                                 lse ? static_cast<float*>(lse->data_ptr()) : nullptr, (float)scale, st));
    }
    after_run(p, st);
    return out;
}

// ---- autograd ----------------------------------------------------------------------------------------
using torch::autograd::edge_list;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

template <typename N>
std::shared_ptr<N> new_node() {
    return std::shared_ptr<N>(new N(), torch::autograd::deleteNode);
}

// Whether a call records a node for its backward pass.  The nodes have no forward-mode derivative: a tangent is refused, as
// torch.autograd.Function refuses it, not dropped.
bool recorded(std::initializer_list<const Tensor*> operands) {
    bool any = false;
    if (at::GradMode::is_enabled())
        for (const Tensor* t : operands) any = any || t->requires_grad();
    if (any)
        for (const Tensor* t : operands)
            TORCH_CHECK_NOT_IMPLEMENTED(!t->_fw_grad(0).defined(), "the blocked operators have no forward-mode derivative");
    return any;
}

Tensor to_type(const Tensor& t, at::ScalarType s) { return t.scalar_type() == s ? t : t.to(s); }

// The two launches of upstream sparseBlockedGEMM::backward (csrc/sparseBlockedAttention.cpp:52-72):
//   mat1Grad = blockedGEMM(outGrad, mat2; offsets (out, mat2, mat1); lists (M, K, N); false, !transpose2)
//   mat2Grad = blockedGEMM(outGrad, mat1; offsets (out, mat1, mat2); lists (N, K, M); true, !transpose1)
struct Offsets {
    std::vector<int64_t> a1, a2, ao;
    explicit Offsets(const Plan& p) : a1(p.S + 1), a2(p.S + 1), ao(p.S + 1) {
        ok(blk_plan_offsets(p.h, a1.data(), a2.data(), ao.data()));
    }
};
Tensor gemm_grad1(const PlanP& p, const Tensor& g, const Tensor& mat2, double scale) {
    const auto t = g.scalar_type();
    PlanP q = derived(p, FOR_GRAD1, t, [&]() {
        const Offsets o(*p);
        return make_gemm(p->M.data(), p->K.data(), p->N.data(), p->S, o.ao.data(), o.a2.data(), o.a1.data(), p->H, t, t, false,
                         !p->tb, false, p->device);
    });
    return run_gemm(*q, g, to_type(mat2, t), scale);
}
Tensor gemm_grad2(const PlanP& p, const Tensor& g, const Tensor& mat1, double scale) {
    const auto t = g.scalar_type();
    PlanP q = derived(p, FOR_GRAD2, t, [&]() {
        const Offsets o(*p);
        return make_gemm(p->N.data(), p->K.data(), p->M.data(), p->S, o.ao.data(), o.a1.data(), o.a2.data(), p->H, t, t, true,
                         !p->ta, false, p->device);
    });
    return run_gemm(*q, g, to_type(mat1, t), scale);
}

struct BlockGEMMBackward : public Node {
    SavedVariable mat1_, mat2_, probs_;
    PlanP plan;
    double scale = 1.0;
    std::string name() const override { return "BlockGEMMBackward"; }
    void release_variables() override {
        mat1_.reset_data();
        mat2_.reset_data();
        probs_.reset_data();
    }
    variable_list apply(variable_list&& grads) override {
        variable_list res(2);
        if (!grads[0].defined()) return res;
        const Tensor mat1 = mat1_.unpack(), mat2 = mat2_.unpack();
        Tensor g = grads[0].contiguous();
        if (plan->softmax) {
            // d(scores * scale) from d(probabilities), then the products carry the scale
            const Tensor probs = to_type(probs_.unpack(shared_from_this()), g.scalar_type());
            PlanP sp = derived(plan, FOR_SOFTMAX, g.scalar_type(), [&]() {
                const Offsets o(*plan);
                return make_softmax(plan->M, plan->N, o.ao.data(), plan->H, g.scalar_type(), plan->device);
            });
            g = run_softmax_backward(*sp, probs, g, 1.0);
        }
        if (task_should_compute_output(0)) res[0] = to_type(gemm_grad1(plan, g, mat2, scale).reshape(mat1.sizes()), mat1.scalar_type());
        if (task_should_compute_output(1)) res[1] = to_type(gemm_grad2(plan, g, mat1, scale).reshape(mat2.sizes()), mat2.scalar_type());
        return res;
    }
};

struct BlockSoftmaxBackward : public Node {
    SavedVariable result_;
    PlanP plan;
    double scale = 1.0;
    std::vector<int64_t> shape;
    std::string name() const override { return "BlockSoftmaxBackward"; }
    void release_variables() override { result_.reset_data(); }
    variable_list apply(variable_list&& grads) override {
        variable_list res(1);
        if (!grads[0].defined() || !task_should_compute_output(0)) return res;
        const Tensor result = result_.unpack(shared_from_this());
        const Tensor g = grads[0].contiguous();
        PlanP p = plan;
        if (g.scalar_type() != p->dt)  // upstream converts the saved result to the gradient's type
            p = derived(plan, FOR_SOFTMAX, g.scalar_type(), [&]() {
                std::vector<int64_t> acc(plan->S + 1);
                ok(blk_plan_offsets(plan->h, acc.data(), nullptr, nullptr));
                return make_softmax(plan->M, plan->N, acc.data(), plan->H, g.scalar_type(), plan->device);
            });
        res[0] = run_softmax_backward(*p, to_type(result, g.scalar_type()), g, scale).reshape(shape);
        return res;
    }
};

Tensor gemm_op(const PlanP& p, const Tensor& mat1, const Tensor& mat2, double scale) {
    if (!recorded({&mat1, &mat2})) return run_gemm(*p, mat1, mat2, scale);
    auto node = new_node<BlockGEMMBackward>();
    node->set_next_edges(torch::autograd::collect_next_edges(mat1, mat2));
    node->plan = p;
    node->scale = scale;
    node->mat1_ = SavedVariable(mat1, false);
    node->mat2_ = SavedVariable(mat2, false);
    Tensor out = run_gemm(*p, mat1.detach(), mat2.detach(), scale);
    torch::autograd::set_history(out, node);
    if (p->softmax) node->probs_ = SavedVariable(out, true);
    return out;
}

// The backward kernels recompute the probabilities: segments beyond 64 x 64 from the saved row logarithms.  These want the
// result as well, which the caller may have written to since (a residual added in place): it is then computed again.
struct BlockAttentionBackward : public Node {
    SavedVariable q_, k_, v_, out_, lse_;
    c10::VariableVersion out_version;
    uint32_t out_saved = 0;
    PlanP plan;
    double scale = 1.0;
    std::string name() const override { return "BlockAttentionBackward"; }
    void release_variables() override {
        q_.reset_data();
        k_.reset_data();
        v_.reset_data();
        out_.reset_data();
        lse_.reset_data();
    }
    variable_list apply(variable_list&& grads) override {
        variable_list res(3);
        if (!grads[0].defined()) return res;
        const Plan& p = *plan;
        const Tensor q = to_type(q_.unpack(), p.dt), k = to_type(k_.unpack(), p.dt), v = to_type(v_.unpack(), p.dt);
        const Tensor out = out_version.current_version() == out_saved ? to_type(out_.unpack(shared_from_this()), p.dt)
                                                                      : run_attention(p, q, k, v, scale, false);
        const Tensor lse = lse_.unpack(), go = to_type(grads[0].contiguous(), p.dt);
        const int64_t nq = p.rows_q * p.d, nkv = p.rows_kv * p.d;
        check_input("q", q, p.dt, p.H, nq);
        check_input("k", k, p.dt, p.H, nkv);
        check_input("v", v, p.dt, p.H, nkv);
        check_input("the attention result", out, p.dt, p.H, nq);
        check_input("the row statistics", lse, at::kFloat, p.H, p.rows_q);
        check_input("the gradient", go, p.dt, p.H, nq);
        c10::cuda::CUDAGuard guard(p.device);
        const Tensor a = aligned(q), b = aligned(k), c = aligned(v), o = aligned(out), l = aligned(lse), g = aligned(go);
        Tensor work = empty2(p.H, p.rows_q, at::kFloat, p.device);
        Tensor dq = empty2(p.H, nq, p.dt, p.device), dk = empty2(p.H, nkv, p.dt, p.device), dv = empty2(p.H, nkv, p.dt, p.device);
        cudaStream_t st = stream_of(p.device);
        ok(blk_attention_backward_run(p.h, a.data_ptr(), b.data_ptr(), c.data_ptr(), o.data_ptr(),
                                      static_cast<const float*>(l.data_ptr()), g.data_ptr(), static_cast<float*>(work.data_ptr()),
                                      dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), (float)scale, st));
        after_run(p, st);
        res[0] = dq.reshape(q.sizes());
        res[1] = dk.reshape(k.sizes());
        res[2] = dv.reshape(v.sizes());
        return res;
    }
};

Tensor attention_op(const PlanP& p, const Tensor& q, const Tensor& k, const Tensor& v, double scale) {
    if (!recorded({&q, &k, &v})) return run_attention(*p, q, k, v, scale, false);
    auto node = new_node<BlockAttentionBackward>();
    node->set_next_edges(torch::autograd::collect_next_edges(q, k, v));
    node->plan = p;
    node->scale = scale;
    node->q_ = SavedVariable(q, false);
    node->k_ = SavedVariable(k, false);
    node->v_ = SavedVariable(v, false);
    ok(blk_attention_prepare_backward(p->h));
    Tensor lse;
    Tensor out = run_attention(*p, q.detach(), k.detach(), v.detach(), scale, false, &lse);
    torch::autograd::set_history(out, node);
    node->out_ = SavedVariable(out, true);
    node->out_version = torch::autograd::impl::version_counter(out);
    node->out_saved = node->out_version.current_version();
    node->lse_ = SavedVariable(lse, false);
    return out;
}

// ---- the operators -----------------------------------------------------------------------------------
// (the caller holds the argument, and with it the tensor, until the operator returns)
const Tensor& operand(const char* name, PyObject* o) {
    TORCH_CHECK(THPVariable_Check(o), name, " must be CUDA Tensor");
    const Tensor& t = THPVariable_Unpack(o);
    check_operand(name, t);
    return t;
}

int64_t dot(const std::vector<int64_t>& a, const std::vector<int64_t>& b) {
    int64_t s = 0;
    for (size_t i = 0; i < a.size(); ++i) s += a[i] * b[i];
    return s;
}
int64_t sum(const std::vector<int64_t>& a) {
    int64_t s = 0;
    for (int64_t x : a) s += x;
    return s;
}

double as_double(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return v;
}
bool as_bool(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw python_error();
    return v != 0;
}
at::ScalarType as_dtype(PyObject* o, at::ScalarType otherwise) {
    if (o == Py_None) return otherwise;
    TORCH_CHECK(THPDtype_Check(o), "out_dtype must be a torch.dtype");
    return reinterpret_cast<THPDtype*>(o)->scalar_type;
}

void same_lengths(const List& a, const List& b, const List& c) {
    TORCH_CHECK(a.v.size() == b.v.size() && a.v.size() == c.v.size(), "MList, NList and KList must have the same length");
}

// gemm(mat1, mat2, mat1Accum, mat2Accum, outAccum, MList, NList, KList, transpose1, transpose2, scale, out_dtype, softmax)
Tensor py_gemm(PyObject* const* a) {
    const Tensor &mat1 = operand("mat1", a[0]), &mat2 = operand("mat2", a[1]);
    const bool have_acc = a[2] != Py_None && a[3] != Py_None && a[4] != Py_None;
    const bool have_lists = a[5] != Py_None && a[6] != Py_None && a[7] != Py_None;
    TORCH_CHECK(have_acc || have_lists, "blockGEMM needs either mat1Accum/mat2Accum/outAccum or MList/NList/KList");
    TORCH_CHECK(mat1.scalar_type() == mat2.scalar_type(), "mat1 and mat2 must have the same dtype");
    const bool ta = as_bool(a[8]), tb = as_bool(a[9]), softmax = as_bool(a[12]);
    const double scale = as_double(a[10]);
    const auto dt = mat1.scalar_type(), odt = as_dtype(a[11], mat1.scalar_type());
    ListArg given[6];
    if (have_lists)
        for (int i = 0; i < 3; ++i) given[i] = list_of(a[5 + i]);
    if (have_acc)
        for (int i = 0; i < 3; ++i) given[3 + i] = list_of(a[2 + i]);
    const NoGil free;
    ListP l[6];
    for (int i = 0; i < 6; ++i) l[i] = given[i].read();
    PlanKey key{0, (int)dt, (int)odt, (int)ta | (int)tb << 1 | (int)softmax << 2, (int)mat1.get_device(), 0, mat1.numel(), {}};
    for (int i = 0; i < 6; ++i) key.l[i] = l[i].get();
    PlanP p = plan_for(key, [&]() {
        std::vector<int64_t> M, N, K;
        if (have_lists) {
            same_lengths(*l[0], *l[1], *l[2]);
            M = l[0]->v; N = l[1]->v; K = l[2]->v;
        } else {
            const auto &a1 = l[3]->v, &a2 = l[4]->v, &ao = l[5]->v;
            TORCH_CHECK(!a1.empty() && a1.size() == a2.size() && a1.size() == ao.size(),
                        "the offset tensors must have equal, non-zero lengths");
            const size_t S = a1.size() - 1;
            M.resize(S); N.resize(S); K.resize(S);
            ok(blk_lists_from_offsets(a1.data(), a2.data(), ao.data(), (int64_t)S, M.data(), N.data(), K.data()));
        }
        if (have_acc)
            for (int i = 3; i < 6; ++i)
                TORCH_CHECK(l[i]->v.size() == M.size() + 1, "offset arrays must have one more entry than the lists");
        const int64_t Dm1 = have_acc ? l[3]->v.back() : dot(M, K);
        TORCH_CHECK(Dm1 > 0 && mat1.numel() % Dm1 == 0, "mat1 has ", mat1.numel(), " elements, not a multiple of the packed extent ", Dm1);
        PlanP made = make_gemm(M.data(), N.data(), K.data(), (int64_t)M.size(), have_acc ? l[3]->v.data() : nullptr,
                               have_acc ? l[4]->v.data() : nullptr, have_acc ? l[5]->v.data() : nullptr, mat1.numel() / Dm1, dt,
                               odt, ta, tb, softmax, mat1.device());
        for (int i = 0; i < 6; ++i) made->lists[i] = l[i];
        return made;
    });
    return gemm_op(p, mat1, mat2, scale);
}

// softmax(src, rowList, colList, srcAccum, scale, out)
Tensor py_softmax(PyObject* const* a) {
    const Tensor& src = operand("src", a[0]);
    TORCH_CHECK(a[1] != Py_None && a[2] != Py_None, "blockSoftmax needs rowList and colList");
    const ListArg given[3] = {list_of(a[1]), list_of(a[2]), list_of(a[3])};
    const double scale = as_double(a[4]);
    Tensor out;
    if (a[5] != Py_None) {
        TORCH_CHECK(THPVariable_Check(a[5]), "out must be a contiguous CUDA tensor shaped like src");
        out = THPVariable_Unpack(a[5]);
    }
    const NoGil free;
    const ListP l[3] = {given[0].read(), given[1].read(), given[2].read()};
    const auto dt = src.scalar_type();
    PlanKey key{1, (int)dt, (int)dt, 0, (int)src.get_device(), 0, src.numel(), {l[0].get(), l[1].get(), l[2].get()}};
    PlanP p = plan_for(key, [&]() {
        TORCH_CHECK(l[0]->v.size() == l[1]->v.size(), "rowList and colList must have the same length");
        TORCH_CHECK(!l[2] || l[2]->v.size() == l[0]->v.size() + 1, "srcAccum must have one more entry than the lists");
        const int64_t D = l[2] ? l[2]->v.back() : dot(l[0]->v, l[1]->v);
        TORCH_CHECK(D > 0 && src.numel() % D == 0, "src has ", src.numel(), " elements, not a multiple of the packed extent ", D);
        PlanP made = make_softmax(l[0]->v, l[1]->v, l[2] ? l[2]->v.data() : nullptr, src.numel() / D, dt, src.device());
        for (int i = 0; i < 3; ++i) made->lists[i] = l[i];
        return made;
    });
    if (out.defined()) return run_softmax(*p, src.detach(), &out, scale);
    if (!recorded({&src})) return run_softmax(*p, src, nullptr, scale);
    auto node = new_node<BlockSoftmaxBackward>();
    node->set_next_edges(torch::autograd::collect_next_edges(src));
    node->plan = p;
    node->scale = scale;
    node->shape = src.sizes().vec();
    out = run_softmax(*p, src.detach(), nullptr, scale);
    torch::autograd::set_history(out, node);
    node->result_ = SavedVariable(out, true);
    return out;
}

PlanP attention_plan(const ListP& M, const ListP& N, int64_t H, int64_t d, at::ScalarType dt, c10::Device dev, bool may_compose) {
    PlanKey key{2, (int)dt, (int)dt, may_compose, (int)dev.index(), (int)d, H, {M.get(), N.get()}};
    return plan_for(key, [&]() {
        const auto &m = M->v, &n = N->v;
        TORCH_CHECK(m.size() == n.size(), "MList and NList must have the same length");
        auto p = std::make_shared<Plan>();
        p->M = m;
        p->N = n;
        p->K.assign(m.size(), d);
        p->S = (int64_t)m.size();
        p->rows_q = sum(m);
        p->rows_kv = sum(n);
        TORCH_CHECK(!may_compose || (p->rows_q > 0 && p->rows_kv > 0), "blockAttention needs at least one query row and one key row");
        p->d = d;
        p->H = H;
        p->dt = p->odt = dt;
        p->device = dev;
        p->lists[0] = M;
        p->lists[1] = N;
        bool fused = (d == 64 || d == 128) && (dt == at::kHalf || dt == at::kBFloat16);
        for (size_t s = 0; may_compose && fused && s < m.size(); ++s) fused = m[s] <= 0 || n[s] >= 1;
        if (fused || !may_compose) {
            const int rc = blk_attention_plan_create_dim(&p->h, m.data(), n.data(), p->S, p->H, d, dtype_code(dt), dev.index());
            if (rc == BLK_ERR_UNSUPPORTED && may_compose) p->h = nullptr;
            else ok(rc);
        }
        p->compose = p->h == nullptr;
        return p;
    });
}

// attention(q, k, v, MList, NList, scale, d)
Tensor py_attention(PyObject* const* a) {
    const Tensor &q = operand("q", a[0]), &k = operand("k", a[1]), &v = operand("v", a[2]);
    const ListArg m_list = list_of(a[3]), n_list = list_of(a[4]);
    TORCH_CHECK(m_list && n_list, "blockAttention needs MList and NList");
    const double scale = as_double(a[5]);
    const bool have_d = a[6] != Py_None;
    int64_t d = 0;
    if (have_d) {
        d = PyLong_AsLongLong(a[6]);
        if (d == -1 && PyErr_Occurred()) throw python_error();
    }
    const NoGil free;
    const ListP M = m_list.read(), N = n_list.read();
    const int64_t rows_q = sum(M->v), rows_kv = sum(N->v);
    TORCH_CHECK(rows_q > 0 && rows_kv > 0, "blockAttention needs at least one query row and one key row");
    if (!have_d) {
        // a (H, sum m_s * d) tensor tells d by its last extent; a flat one cannot (d and H only appear as a product)
        TORCH_CHECK(q.dim() >= 2 && q.size(-1) % rows_q == 0,
                    "give the head dimension d (a flat tensor cannot tell it apart from the number of heads)");
        d = q.size(-1) / rows_q;
    }
    TORCH_CHECK(d > 0 && q.numel() % (rows_q * d) == 0 && k.numel() == (q.numel() / (rows_q * d)) * rows_kv * d && v.numel() == k.numel(),
                "q / k / v do not match the packed extents of the lists");
    const auto dt = q.scalar_type();
    const bool one_type = k.scalar_type() == dt && v.scalar_type() == dt;
    const PlanP p = attention_plan(M, N, q.numel() / (rows_q * d), d, dt, q.device(), true);
    if (!p->compose && one_type) return attention_op(p, q, k, v, scale);
    // the composition of the two operators
    TORCH_CHECK(k.scalar_type() == dt && v.scalar_type() == dt, "mat1 and mat2 must have the same dtype");
    const auto& D = p->K;
    const PlanP ps = derived(p, FOR_SCORES, dt, [&]() {
        return make_gemm(p->M.data(), p->N.data(), D.data(), p->S, nullptr, nullptr, nullptr, p->H, dt, dt, false, false, true, p->device);
    });
    const PlanP pv = derived(p, FOR_PRODUCT, dt, [&]() {
        return make_gemm(p->M.data(), D.data(), p->N.data(), p->S, nullptr, nullptr, nullptr, p->H, dt, dt, false, true, false, p->device);
    });
    return gemm_op(pv, gemm_op(ps, q, k, scale), v, 1.0);
}

// attention_token_major(q, k, v, nList, scale)
Tensor py_attention_token_major(PyObject* const* a) {
    const Tensor &q = operand("q", a[0]), &k = operand("k", a[1]), &v = operand("v", a[2]);
    TORCH_CHECK(q.dim() == 3 && q.sizes() == k.sizes() && q.sizes() == v.sizes() && (q.size(2) == 64 || q.size(2) == 128),
                "q, k and v must all have shape (sum n, H, d), d 64 or 128");
    const ListArg n_list = list_of(a[3]);
    TORCH_CHECK(n_list, "blockAttentionTokenMajor needs nList");
    const double scale = as_double(a[4]);
    const NoGil free;
    const ListP n = n_list.read();
    const auto dt = q.scalar_type();
    const int64_t rows = sum(n->v);
    TORCH_CHECK(q.size(0) == rows && k.scalar_type() == dt && v.scalar_type() == dt && !unaligned(q) && !unaligned(k) && !unaligned(v),
                "q, k and v must be contiguous, 16-byte aligned CUDA tensors of one type and shape (", rows, ", ", q.size(1), ", ",
                q.size(2), ")");
    const PlanP p = attention_plan(n, n, q.size(1), q.size(2), dt, q.device(), false);
    return run_attention(*p, q.detach(), k.detach(), v.detach(), scale, true);
}

// scores_token_major(q, k, nList, scale, out_dtype, softmax)
Tensor py_scores_token_major(PyObject* const* a) {
    const Tensor &q = operand("q", a[0]), &k = operand("k", a[1]);
    TORCH_CHECK(q.dim() == 3 && q.sizes() == k.sizes(), "q and k must both have shape (sum n, H, d)");
    const ListArg n_list = list_of(a[2]);
    TORCH_CHECK(n_list, "blockAttnScoresTokenMajor needs nList");
    const double scale = as_double(a[3]);
    const auto dt = q.scalar_type(), odt = as_dtype(a[4], dt);
    const bool softmax = as_bool(a[5]);
    const NoGil free;
    const ListP n = n_list.read();
    TORCH_CHECK(!n->v.empty(), "blockAttnScoresTokenMajor needs at least one segment");
    const int64_t H = q.size(1), d = q.size(2);
    PlanKey key{3, (int)dt, (int)odt, (int)softmax, (int)q.get_device(), (int)d, H, {n.get()}};
    const PlanP p = plan_for(key, [&]() {
        const std::vector<int64_t> D(n->v.size(), d);
        PlanP made = make_gemm(n->v.data(), n->v.data(), D.data(), (int64_t)D.size(), nullptr, nullptr, nullptr, H, dt, odt, false,
                               false, softmax, q.device());
        made->lists[0] = n;
        made->rows_q = sum(n->v);
        return made;
    });
    for (const Tensor* t : {&q, &k})
        TORCH_CHECK(t->size(0) == p->rows_q && t->scalar_type() == dt && !unaligned(*t), "q and k must be 16-byte aligned, of one type and have shape (rows, H, d) = (",
                    p->rows_q, ", ", H, ", ", d, ")");
    c10::cuda::CUDAGuard guard(p->device);
    Tensor out = empty2(p->H, p->Dout, odt, p->device);
    cudaStream_t st = stream_of(p->device);
    ok(blk_gemm_run_strided(p->h, q.data_ptr(), H * d, d, k.data_ptr(), H * d, d, out.data_ptr(), (float)scale, st));
    after_run(*p, st);
    return out;
}

// ---- the module --------------------------------------------------------------------------------------
// F takes NARGS arguments, the first NTENSORS of them its operands.  torch.jit.trace sees nothing of what happens here: a
// call that it is to record goes to apply.py and comes back, with the tracer paused, from a torch.autograd.Function.
template <Tensor (*F)(PyObject* const*), const char* NAME, int NARGS, int NTENSORS>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(n == NARGS, "expected ", NARGS, " arguments");
    if (torch::jit::tracer::isTracing()) {
        PyRef rest(PyTuple_New(NARGS));
        for (int i = 0; rest.o && i < NARGS; ++i) {
            Py_INCREF(args[i]);
            PyTuple_SET_ITEM(rest.o, i, args[i]);
        }
        return rest.o ? PyObject_CallFunction(g_traced, "siO", NAME, NTENSORS, rest.o) : nullptr;
    }
    return THPVariable_Wrap(F(args));
    END_HANDLE_TH_ERRORS
}

PyObject* py_clear(PyObject*, PyObject*) {
    {
        const NoGil free;
        std::vector<PlanP> p;
        std::vector<Remembered> r;
        std::lock_guard<std::mutex> g(g_mu);
        plans().clear(&p);
        device_lists().clear(&r);
    }
    Py_RETURN_NONE;
}

// Synchronises the current stream of every cached plan's device; raises for a plan with a timed-out wait.
PyObject* py_check(PyObject*, PyObject*) {
    HANDLE_TH_ERRORS
    std::vector<PlanP> all;
    {
        std::lock_guard<std::mutex> g(g_mu);
        for (auto& e : plans().order) {
            all.push_back(e.second);
            for (auto& row : e.second->derived)
                for (auto& q : row)
                    if (q) all.push_back(q);
        }
    }
    {
        const NoGil free;
        for (const PlanP& p : all) {
            if (!p->h) continue;
            c10::cuda::CUDAGuard guard(p->device);
            p->check(stream_of(p->device));
        }
    }
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

// same_list(a, b): whether the plan cache takes two list arguments for the same list.  For tests and debugging.
PyObject* py_same_list(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(n == 2, "expected 2 arguments");
    const ListArg a = list_of(args[0]), b = list_of(args[1]);
    ListP la, lb;
    {
        const NoGil free;
        la = a.read();
        lb = b.read();
    }
    return PyBool_FromLong(la == lb);
    END_HANDLE_TH_ERRORS
}

// cached(): the numbers of plans and of GPU lists that are remembered.  For tests and debugging.
PyObject* py_cached(PyObject*, PyObject*) {
    std::lock_guard<std::mutex> g(g_mu);
    return Py_BuildValue("nn", (Py_ssize_t)plans().order.size(), (Py_ssize_t)device_lists().order.size());
}

// setup(_host_i64, BlkError, _traced)
PyObject* py_setup(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 3) {
        PyErr_SetString(PyExc_TypeError, "setup(host_i64, error_class, traced)");
        return nullptr;
    }
    for (Py_ssize_t i = 0; i < n; ++i) Py_INCREF(args[i]);
    g_host_i64 = args[0];
    g_error = args[1];
    g_traced = args[2];
    Py_RETURN_NONE;
}

#define BLK_ENTRY(name, nargs, ntensors) \
    {g_##name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<py_##name, g_##name, nargs, ntensors>)), METH_FASTCALL, nullptr}
constexpr char g_gemm[] = "gemm", g_softmax[] = "softmax", g_attention[] = "attention",
               g_attention_token_major[] = "attention_token_major", g_scores_token_major[] = "scores_token_major";
PyMethodDef g_methods[] = {
    BLK_ENTRY(gemm, 13, 2),
    BLK_ENTRY(softmax, 6, 1),
    BLK_ENTRY(attention, 7, 3),
    BLK_ENTRY(attention_token_major, 5, 3),
    BLK_ENTRY(scores_token_major, 6, 2),
    {"clear", py_clear, METH_NOARGS, nullptr},
    {"check", py_check, METH_NOARGS, nullptr},
    {"cached", py_cached, METH_NOARGS, nullptr},
    {"same_list", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&py_same_list)), METH_FASTCALL, nullptr},
    {"setup", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&py_setup)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_ops", "native host path of the operators", -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__ops(void) { return PyModule_Create(&g_module); }
