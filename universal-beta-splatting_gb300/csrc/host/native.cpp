// native.cpp -- the host path between Python and the C ABI (include/ubs.h):
// output and workspace allocation, camera tables, autograd nodes and the calls
// themselves, as one extension module (ubs_native) linked to the library.
//
// The Python modules keep the argument checks, shapes and result types of the
// public functions; what a small render spent its time on was below them.  At
// 10k primitives and 256 x 256 pixels the kernels of a training step take
// about 75 us and the step took 640: a Python autograd function costs about
// 25 us per direction, a ctypes call with 30 arguments 25 us besides its
// launches, a device guard for the current stream 15 us, and the intersection
// count was read only after the whole frame had run.  Here a direction is a
// few microseconds, and the count is copied as soon as the scan has produced
// it, so that the host prepares what follows while the frame still renders.
//
// The calls run without Python's lock, as ctypes and PyTorch's operators do: a
// full launch queue blocks the calling thread alone.
//
// Nothing is kept between calls: every call allocates its outputs and
// workspace from PyTorch's caching allocator on the current stream, and reads
// the current stream when it runs.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/CachingHostAllocator.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>
#include <cuda_runtime.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/utils/pybind.h>

#include <algorithm>
#include <functional>
#include <memory>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "../../../include/ubs.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

namespace {

// ------------------------------------------------------------------ calls
// CUDA events around entry-point calls while timing is on (ubs._lib).
struct Timing {
    std::mutex mu;
    bool on = false;
    std::vector<std::tuple<std::string, at::cuda::CUDAEvent, at::cuda::CUDAEvent>> rec;
} g_timing;

template <class F> void call(const char *name, F &&f) {
    bool timed;
    {
        std::lock_guard<std::mutex> lk(g_timing.mu);
        timed = g_timing.on;
    }
    int rc;
    if (timed) {
        at::cuda::CUDAEvent e0(cudaEventDefault), e1(cudaEventDefault);
        e0.record();
        rc = f();
        e1.record();
        std::lock_guard<std::mutex> lk(g_timing.mu);
        g_timing.rec.emplace_back(name, std::move(e0), std::move(e1));
    } else {
        rc = f();
    }
    TORCH_CHECK(rc == 0, name, " failed (", rc, "): ", ubs_last_error());
}
#define UBS_CALL(fn, ...) call(#fn, [&] { return fn(__VA_ARGS__); })

void *stream_of(const Tensor &t) {
    return c10::cuda::getCurrentCUDAStream(t.device().index()).stream();
}

// A float32 CUDA tensor in C order (a copy where the argument is not).
Tensor f32(const Tensor &t) {
    TORCH_CHECK_VALUE(t.is_cuda(), "expected a CUDA tensor, got device ", t.device());
    TORCH_CHECK_TYPE(t.scalar_type() == at::kFloat,
                     "the GB300 rasteriser computes in float32; got ", t.dtype());
    return t.contiguous();
}
const float *fp(const Tensor &t) { return t.defined() ? t.const_data_ptr<float>() : nullptr; }
float *fpm(Tensor &t) { return t.defined() ? t.mutable_data_ptr<float>() : nullptr; }
Tensor fempty(at::IntArrayRef s, const Tensor &like) {
    return at::empty(s, like.options().dtype(at::kFloat));
}
// Zeroes the first n bytes of t on its current stream.
void zero(Tensor &t, size_t n) {
    n = std::min<size_t>(n, t.nbytes());
    if (n)
        C10_CUDA_CHECK(cudaMemsetAsync(t.mutable_data_ptr(), 0, n,
                                       static_cast<cudaStream_t>(stream_of(t))));
}
Tensor fzeros(at::IntArrayRef s, const Tensor &like) {
    Tensor t = fempty(s, like);
    zero(t, t.nbytes());
    return t;
}
Tensor bytes(size_t n, const Tensor &like) {
    return at::empty({(int64_t)std::max<size_t>(n, 256)}, like.options().dtype(at::kByte));
}
// A gradient that reached the node, or zeros.
Tensor grad_or_zeros(const Tensor &g, at::IntArrayRef s, const Tensor &like) {
    return g.defined() ? f32(g) : fzeros(s, like);
}

// --------------------------------------------------------------- autograd
// A node whose backward is `bwd` over the saved tensors and the gradients of
// its outputs (undefined where none arrived).
struct OpNode : public torch::autograd::Node {
    using Backward = std::function<variable_list(OpNode &, const variable_list &, variable_list &)>;
    // what a kernel that reads a saved tensor relies on
    struct Kind {
        c10::SmallVector<int64_t, 4> sizes;
        at::ScalarType type;
        at::Device device;
    };
    std::string op;
    std::vector<SavedVariable> saved;
    std::vector<std::optional<Kind>> kinds;
    Backward bwd;

    // The saved tensors for a kernel.  Saved-tensor hooks may return anything:
    // other strides are copied to C order, another size, type or device raises.
    variable_list for_kernel(const variable_list &s) const {
        variable_list o;
        o.reserve(s.size());
        for (size_t i = 0; i < s.size(); ++i) {
            TORCH_CHECK_VALUE(s[i].defined() == kinds[i].has_value(), op, ": saved tensor ", i,
                              " is missing");
            if (s[i].defined()) {
                const Kind &k = *kinds[i];
                TORCH_CHECK_VALUE(s[i].device() == k.device, op, ": expected a saved tensor on ",
                                  k.device, ", got device ", s[i].device());
                TORCH_CHECK_TYPE(s[i].scalar_type() == k.type, op, ": expected a saved tensor of ",
                                 k.type, ", got ", s[i].scalar_type());
                TORCH_CHECK_VALUE(s[i].sizes() == at::IntArrayRef(k.sizes), op,
                                  ": expected a saved tensor of size ", at::IntArrayRef(k.sizes),
                                  ", got ", s[i].sizes());
                o.push_back(s[i].contiguous());
            } else {
                o.emplace_back();
            }
        }
        return o;
    }

    variable_list apply(variable_list &&grads) override {
        std::lock_guard<std::mutex> lk(mutex_);
        TORCH_CHECK(bwd, "Trying to backward through the graph a second time (", op, ")");
        variable_list s;
        s.reserve(saved.size());
        for (SavedVariable &v : saved) s.push_back(v.unpack(shared_from_this()));
        return bwd(*this, s, grads);
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lk(mutex_);
        for (SavedVariable &v : saved) v.reset_data();
        bwd = nullptr;
    }
    std::string name() const override { return op; }
};

// Forward-mode derivatives are not defined for these operators: raise instead
// of dropping the tangents.
void no_tangents(const char *op, at::ArrayRef<Tensor> inputs) {
    for (const Tensor &t : inputs)
        TORCH_CHECK_NOT_IMPLEMENTED(!t.defined() || !t._fw_grad(0).defined(), op,
                                    " has no forward-mode derivative");
}

bool wants_grad(at::ArrayRef<Tensor> inputs) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor &t : inputs)
        if (t.defined() && t.requires_grad()) return true;
    return false;
}

// Makes `outputs` (fresh tensors) the results of a node with these inputs;
// `saved_outputs` are saved as outputs of the node.
void attach(const char *op, at::ArrayRef<Tensor> inputs, at::ArrayRef<Tensor> outputs,
            at::ArrayRef<Tensor> saved, at::ArrayRef<Tensor> saved_outputs, OpNode::Backward bwd) {
    std::shared_ptr<OpNode> node(new OpNode(), torch::autograd::deleteNode);
    node->op = op;
    torch::autograd::edge_list edges;
    edges.reserve(inputs.size());
    for (const Tensor &t : inputs)
        edges.push_back(t.defined() && t.requires_grad()
                            ? torch::autograd::impl::gradient_edge(t)
                            : torch::autograd::Edge());
    node->set_next_edges(std::move(edges));
    for (const Tensor &t : outputs) torch::autograd::create_gradient_edge(const_cast<Tensor &>(t), node);
    node->saved.reserve(saved.size() + saved_outputs.size());
    node->kinds.reserve(saved.size() + saved_outputs.size());
    auto save = [&](const Tensor &t, bool is_output) {
        node->saved.emplace_back(t, is_output);
        node->kinds.emplace_back();
        if (t.defined())
            node->kinds.back() = OpNode::Kind{{t.sizes().begin(), t.sizes().end()},
                                              t.scalar_type(), t.device()};
    };
    for (const Tensor &t : saved) save(t, false);
    for (const Tensor &t : saved_outputs) save(t, true);
    node->bwd = std::move(bwd);
}

// ------------------------------------------------------------- fused render
// Device tables of a Views object and the launch geometry.
struct SceneCall {
    int32_t dim, C, n_buckets, tile;
    float eps2d, near_p, far_p, clip;
    bool exact;
    int64_t n_pixels, cap;
    Tensor viewmats, intr, centers, times, dims, tile_base, pix_base;
    Tensor ws; // released by the backward
};

// The intersection count and status of a frame, on their way to the host.
struct FrameStats {
    Tensor host; // pinned int64 [2]
    at::cuda::CUDAEvent ev;
    std::pair<int64_t, int64_t> wait() {
        ev.synchronize();
        const int64_t *p = host.const_data_ptr<int64_t>();
        return {p[0], p[1] & 0xffffffff};
    }
};

constexpr int kParams = 7; // xyz, mean, scale, l_triangle, opacity, beta, rgb

std::shared_ptr<SceneCall> scene_call(int32_t dim, const std::vector<Tensor> &tables,
                                      int32_t n_buckets, int64_t n_pixels, int32_t tile,
                                      double eps2d, double near_p, double far_p, double clip,
                                      bool exact, int64_t cap) {
    TORCH_CHECK_VALUE(tables.size() == 7, "seven view tables expected");
    auto c = std::make_shared<SceneCall>();
    c->dim = dim;
    c->n_buckets = n_buckets;
    c->n_pixels = n_pixels;
    c->tile = tile;
    c->eps2d = (float)eps2d;
    c->near_p = (float)near_p;
    c->far_p = (float)far_p;
    c->clip = (float)clip;
    c->exact = exact;
    c->cap = cap;
    c->viewmats = tables[0];
    c->intr = tables[1];
    c->centers = tables[2];
    c->times = tables[3];
    c->dims = tables[4];
    c->tile_base = tables[5];
    c->pix_base = tables[6];
    c->C = (int32_t)c->times.numel();
    for (const Tensor &t : tables)
        TORCH_CHECK_VALUE(t.is_cuda() && t.is_contiguous(),
                          "expected contiguous CUDA view tables, got device ", t.device());
    return c;
}

Tensor scene_param(const Tensor &t) {
    TORCH_CHECK_VALUE(t.is_cuda(), "expected a CUDA tensor, got device ", t.device());
    TORCH_CHECK_TYPE(t.scalar_type() == at::kFloat, "scene parameters must be float32");
    return t.contiguous();
}

// Renders.  stats: whether the count and status are copied to the host, which
// happens as soon as they are known (not capture safe).  With gradients, the
// outputs are attached to the parameters.  image: pinned host memory that takes
// the colours (and is returned as such), complete once the stream has been
// waited for; tiles of 16 pixels and more are stored there by the blend itself,
// smaller ones copied (their 96-byte rows use the link badly: a nearly empty
// 1080p frame 191 us against 46 + 135).
std::tuple<Tensor, Tensor, Tensor, Tensor, std::shared_ptr<FrameStats>>
scene_forward(const std::shared_ptr<SceneCall> &c, const std::vector<Tensor> &params,
              const Tensor &bg, const OptTensor &mask, int32_t color_mode, bool stats, bool grad,
              const OptTensor &image) {
    TORCH_CHECK_VALUE(params.size() == kParams, "seven scene parameters expected");
    std::vector<Tensor> in = params;
    in.push_back(bg); // a node's input, as in the operators; its gradient is undefined
    if (grad) no_tangents("scene render", in);
    const bool attached = grad && wants_grad(in);
    const at::NoGradGuard no_grad;
    std::vector<Tensor> p(kParams);
    for (int i = 0; i < kParams; ++i) p[i] = scene_param(params[i]);
    const c10::cuda::CUDAGuard guard(p[0].device());
    const Tensor b = f32(bg);
    const uint8_t *m = nullptr;
    if (mask) {
        TORCH_CHECK_VALUE(mask->is_cuda() && mask->is_contiguous(),
                          "expected a contiguous CUDA tensor, got device ", mask->device());
        TORCH_CHECK_TYPE(mask->scalar_type() == at::kByte, "expected a uint8 mask");
        m = mask->const_data_ptr<uint8_t>();
    }
    const int64_t N = p[0].size(0);
    c->ws = bytes(ubs_scene_workspace_bytes(c->C, N, c->n_buckets, c->cap), p[0]);
    float *host = nullptr; // the image's address on the device
    if (image) {
        TORCH_CHECK_VALUE(!attached && image->is_cpu() && image->is_pinned() &&
                              image->scalar_type() == at::kFloat && image->is_contiguous() &&
                              image->numel() == 3 * c->n_pixels,
                          "expected a pinned float32 image of the frame's size, without gradients");
        if (c->tile >= 16 && N > 0 &&
            cudaHostGetDevicePointer(reinterpret_cast<void **>(&host),
                                     image->mutable_data_ptr<float>(), 0) != cudaSuccess) {
            cudaGetLastError();
            host = nullptr;
        }
    }
    Tensor colors = host ? image->view({c->n_pixels, 3}) : fempty({c->n_pixels, 3}, p[0]);
    Tensor alphas = fempty({c->n_pixels}, p[0]);
    Tensor last = at::empty({c->n_pixels}, p[0].options().dtype(at::kInt));
    void *st = stream_of(p[0]);
    auto part = [&](int32_t parts, int64_t *counts) {
        UBS_CALL(ubs_scene_forward_parts, c->dim, N, fp(p[0]), fp(p[1]), fp(p[2]), fp(p[3]),
                 fp(p[4]), fp(p[5]), fp(p[6]), c->C, fp(c->viewmats), fp(c->intr), fp(c->centers),
                 fp(c->times), c->dims.const_data_ptr<int32_t>(),
                 c->tile_base.const_data_ptr<int32_t>(), c->pix_base.const_data_ptr<int64_t>(),
                 c->n_buckets, c->tile, c->eps2d, c->near_p, c->far_p, c->clip, fp(b),
                 host ? host : fpm(colors), fpm(alphas), last.mutable_data_ptr<int32_t>(), c->cap,
                 c->ws.mutable_data_ptr(), c->ws.nbytes(), m, color_mode,
                 host && (parts & UBS_SCENE_PART_BLEND) ? parts | UBS_SCENE_HOST_IMAGE : parts,
                 counts, st);
    };
    std::shared_ptr<FrameStats> fs; // none without stats
    if (!stats) {
        part(UBS_SCENE_PART_COUNT | UBS_SCENE_PART_BLEND, nullptr);
    } else {
        // the count kernel writes to the pinned slot itself: a copy would make
        // the frame wait for the copy engine
        fs = std::make_shared<FrameStats>();
        fs->host = at::empty({2}, at::TensorOptions().dtype(at::kLong).pinned_memory(true));
        part(UBS_SCENE_PART_COUNT, fs->host.mutable_data_ptr<int64_t>());
        const auto cs = c10::cuda::getCurrentCUDAStream(p[0].device().index());
        fs->ev.record(cs);
        // the slot outlives the kernel's write
        at::cuda::CachingHostAllocator_recordEvent(fs->host.mutable_data_ptr(),
                                                   fs->host.storage().data_ptr().get_context(), cs);
        part(UBS_SCENE_PART_BLEND, nullptr);
    }
    if (image) {
        if (!host) image->view({c->n_pixels, 3}).copy_(colors, /*non_blocking=*/true);
        // the memory outlives the kernel's stores (a copy records this itself)
        else
            at::cuda::CachingHostAllocator_recordEvent(
                image->mutable_data_ptr(), image->storage().data_ptr().get_context(),
                c10::cuda::getCurrentCUDAStream(p[0].device().index()));
        colors = image->view({c->n_pixels, 3});
    }
    Tensor ws = c->ws;
    if (attached) {
        const std::vector<int64_t> opacity_shape = params[4].sizes().vec();
        p.push_back(b);
        p.push_back(last);
        attach("SceneRenderBackward", in, {colors, alphas}, p, {alphas},
               [c, opacity_shape](OpNode &node, const variable_list &saved, variable_list &g) {
                   const at::NoGradGuard no_grad;
                   const variable_list s = node.for_kernel(saved);
                   TORCH_CHECK(c->ws.defined(), "scene_backward: the frame's workspace was "
                                                "released by an earlier backward");
                   const c10::cuda::CUDAGuard guard(s[0].device());
                   const Tensor vc = grad_or_zeros(g[0], {c->n_pixels, 3}, s[0]);
                   const Tensor va = grad_or_zeros(g[1], {c->n_pixels}, s[0]);
                   variable_list o(kParams + 1);
                   for (int i = 0; i < kParams; ++i) o[i] = at::empty_like(s[i]);
                   UBS_CALL(ubs_scene_backward, c->dim, s[0].size(0), fp(s[0]), fp(s[1]), fp(s[2]),
                            fp(s[3]), fp(s[4]), fp(s[5]), fp(s[6]), c->C, fp(c->viewmats),
                            fp(c->intr), fp(c->centers), fp(c->times),
                            c->dims.const_data_ptr<int32_t>(),
                            c->tile_base.const_data_ptr<int32_t>(),
                            c->pix_base.const_data_ptr<int64_t>(), c->n_buckets, c->tile,
                            c->eps2d, c->near_p, c->far_p, c->clip, fp(s[7]), fp(s[9]),
                            s[8].const_data_ptr<int32_t>(), fp(vc), fp(va), fpm(o[0]), fpm(o[1]),
                            fpm(o[2]), fpm(o[3]), fpm(o[4]), fpm(o[5]), fpm(o[6]),
                            (int32_t)c->exact, c->cap, c->ws.mutable_data_ptr(), c->ws.nbytes(),
                            stream_of(s[0]));
                   c->ws.reset();
                   o[4] = o[4].view(opacity_shape);
                   return o;
               });
    }
    return {colors, alphas, last, ws, fs};
}

// Camera tables of a Views object: one pinned staging buffer and one copy to
// the device, on `stream` (its id and device; default: the current one).  The
// cameras' own tensors are read on the current stream, which they were made on.
// Sections: pix_base int64 [C + 1], dims int32 [C, 4], tile_base
// int32 [C + 1], viewmats [C, 16], intrinsics [C, 4], centers [C, 3], times.
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, std::vector<int64_t>,
           std::vector<int64_t>>
pack_views(const std::vector<Tensor> &viewmats, const std::vector<Tensor> &Ks,
           const std::vector<OptTensor> &centers, const std::vector<double> &times,
           const std::vector<int64_t> &widths, const std::vector<int64_t> &heights, int64_t tile,
           const at::Device &device, const std::optional<std::pair<int64_t, int64_t>> &stream) {
    const at::NoGradGuard no_grad;
    const int64_t C = (int64_t)viewmats.size();
    const int64_t words = 2 * (C + 1) + 4 * C + (C + 1) + 24 * C;
    Tensor staging = at::empty({words}, at::TensorOptions().dtype(at::kInt).pinned_memory(
                                            at::globalContext().hasCUDA()));
    int32_t *w = staging.mutable_data_ptr<int32_t>();
    int64_t *pix = reinterpret_cast<int64_t *>(w);
    int32_t *dims = w + 2 * (C + 1), *tb = dims + 4 * C;
    float *vm = reinterpret_cast<float *>(tb + C + 1), *in = vm + 16 * C, *ce = in + 4 * C,
          *ti = ce + 3 * C;
    std::vector<int64_t> tile_base(C + 1, 0), pix_base(C + 1, 0);
    auto host = [](const Tensor &t) {
        return t.to(at::kCPU, at::kFloat).contiguous();
    };
    for (int64_t v = 0; v < C; ++v) {
        const Tensor m = host(viewmats[v]).reshape({16}), K = host(Ks[v]);
        const float *mp = m.const_data_ptr<float>();
        std::copy(mp, mp + 16, vm + 16 * v);
        const auto k = K.accessor<float, 2>();
        in[4 * v] = k[0][0];
        in[4 * v + 1] = k[1][1];
        in[4 * v + 2] = k[0][2];
        in[4 * v + 3] = k[1][2];
        const Tensor c = centers[v] ? host(*centers[v]).reshape({3})
                                    : -(m.view({4, 4}).narrow(0, 0, 3).narrow(1, 0, 3).t().mv(
                                          m.view({4, 4}).narrow(0, 0, 3).select(1, 3)));
        for (int i = 0; i < 3; ++i) ce[3 * v + i] = c[i].item<float>();
        ti[v] = (float)times[v];
        const int64_t tw = (widths[v] + tile - 1) / tile, th = (heights[v] + tile - 1) / tile;
        dims[4 * v] = (int32_t)widths[v];
        dims[4 * v + 1] = (int32_t)heights[v];
        dims[4 * v + 2] = (int32_t)tw;
        dims[4 * v + 3] = (int32_t)th;
        tile_base[v + 1] = tile_base[v] + tw * th;
        pix_base[v + 1] = pix_base[v] + widths[v] * heights[v];
    }
    TORCH_CHECK_VALUE(tile_base[C] < (1ll << 31), "too many tiles in one render call");
    for (int64_t v = 0; v <= C; ++v) {
        tb[v] = (int32_t)tile_base[v];
        pix[v] = pix_base[v];
    }
    Tensor dev;
    if (device.is_cuda()) {
        c10::cuda::OptionalCUDAStreamGuard on;
        if (stream)
            on.reset_stream(c10::Stream::unpack3(
                stream->first, (c10::DeviceIndex)stream->second, c10::DeviceType::CUDA));
        const c10::cuda::OptionalCUDAGuard guard(device);
        dev = staging.to(at::TensorOptions().device(device), /*non_blocking=*/true);
    } else {
        dev = staging.clone();
    }
    int64_t o = 0;
    auto take = [&](int64_t n) {
        Tensor t = dev.narrow(0, o, n);
        o += n;
        return t;
    };
    Tensor d_pix = take(2 * (C + 1)).view(at::kLong), d_dims = take(4 * C).view({C, 4});
    Tensor d_tb = take(C + 1);
    Tensor d_vm = take(16 * C).view(at::kFloat).view({C, 16});
    Tensor d_in = take(4 * C).view(at::kFloat).view({C, 4});
    Tensor d_ce = take(3 * C).view(at::kFloat).view({C, 3});
    Tensor d_ti = take(C).view(at::kFloat);
    return {staging, d_vm, d_in, d_ce, d_ti, d_dims, d_tb, d_pix, tile_base, pix_base};
}

// ------------------------------------------------------------------- losses
// The stored gradient of a loss times the incoming scalar.  One kernel over
// dense float32 tensors of one device; anything else (a gradient that is itself
// differentiated, what saved-tensor hooks may return) multiplies in general.
variable_list scaled(const variable_list &s, variable_list &g, size_t n) {
    variable_list o(n);
    if (!g[0].defined()) return o;
    const Tensor &x = s[0], &by = g[0];
    const auto plain = [](const Tensor &t) {
        const c10::DispatchKeySet k = t.key_set();
        return t.layout() == at::kStrided && t.is_cuda() && t.scalar_type() == at::kFloat &&
               !k.has(c10::DispatchKey::Python) && !k.has(c10::DispatchKey::FuncTorchBatched) &&
               !k.has(c10::DispatchKey::Batched) && !t.is_neg() && !t._fw_grad(0).defined();
    };
    if (at::GradMode::is_enabled() || !plain(x) || !plain(by) || by.dim() != 0 ||
        x.device() != by.device() || !x.is_non_overlapping_and_dense()) {
        o[0] = x * by;
        return o;
    }
    const c10::cuda::CUDAGuard guard(x.device());
    o[0] = at::empty_like(x);
    UBS_CALL(ubs_scale, fp(x), fp(by), fpm(o[0]), x.numel(), stream_of(x));
    return o;
}

// mean |x - y| and its gradient in one launch.
Tensor l1_loss(const Tensor &x, const Tensor &y) {
    no_tangents("l1_loss", {x, y});
    const bool grad = wants_grad({x});
    Tensor out, g;
    {
        const at::NoGradGuard no_grad;
        const c10::cuda::CUDAGuard guard(x.device());
        const int64_t n = x.numel();
        out = fempty({2}, x);
        Tensor ws = bytes(ubs_l1_loss_workspace_bytes(n), x);
        void *st = stream_of(x);
        zero(ws, 256);
        if (grad) g = at::empty_like(x);
        UBS_CALL(ubs_l1_loss, fp(x), fp(y), fpm(g), n, 1.0, fpm(out), ws.mutable_data_ptr(),
                 ws.nbytes(), st);
        out = out.select(0, 0);
    }
    if (!grad) return out;
    out = out.detach();
    attach("L1LossBackward", {x}, {out}, {g}, {},
           [](OpNode &, const variable_list &s, variable_list &gr) { return scaled(s, gr, 1); });
    return out;
}

// Result `index` of (mean map, mean |x - y|, loss) of ubs_ssim_loss.
Tensor ssim_loss(const Tensor &img, const Tensor &gt, bool channels_last, bool valid, double w0,
                 double w1, double w2, int64_t index) {
    no_tangents("ssim loss", {img, gt});
    const bool want = wants_grad({img});
    Tensor out, grad;
    {
        const at::NoGradGuard no_grad;
        const c10::cuda::CUDAGuard guard(img.device());
        const int64_t d = img.dim(), k = d - 3;
        auto strides = [&](const Tensor &t, int64_t (&s)[4]) {
            s[0] = d == 4 ? t.stride(0) : 0;
            s[1] = t.stride(channels_last ? k + 2 : k);
            s[2] = t.stride(channels_last ? k : k + 1);
            s[3] = t.stride(channels_last ? k + 1 : k + 2);
        };
        const int64_t n = d == 4 ? img.size(0) : 1, c = img.size(channels_last ? k + 2 : k),
                      h = img.size(channels_last ? k : k + 1),
                      w = img.size(channels_last ? k + 1 : k + 2);
        int64_t si[4], sg[4], sd[4];
        strides(img, si);
        strides(gt, sg);
        if (want) {
            grad = at::empty_like(img);
            strides(grad, sd);
        }
        out = fempty({3}, img);
        Tensor ws = at::empty({(int64_t)ubs_ssim_workspace_bytes((int32_t)n, (int32_t)c,
                                                                 (int32_t)h, (int32_t)w)},
                              img.options().dtype(at::kByte));
        void *st = stream_of(img);
        // the ticket counter (first bytes) starts at zero; the rest is written
        // before it is read
        zero(ws, 256);
        UBS_CALL(ubs_ssim_loss, img.const_data_ptr<float>(), si, gt.const_data_ptr<float>(), sg,
                 want ? grad.mutable_data_ptr<float>() : nullptr, want ? sd : nullptr, (int32_t)n,
                 (int32_t)c, (int32_t)h, (int32_t)w, (int32_t)valid, w0, w1, w2, fpm(out),
                 ws.mutable_data_ptr(), ws.nbytes(), st);
        out = out.select(0, index);
    }
    if (!want) return out;
    out = out.detach();
    attach("SsimLossBackward", {img}, {out}, {grad}, {},
           [](OpNode &, const variable_list &s, variable_list &gr) { return scaled(s, gr, 1); });
    return out;
}

// --------------------------------------------------------- drop-in operators
std::tuple<Tensor, Tensor, Tensor> cond(const Tensor &means_, const Tensor &covars_,
                                        const Tensor &opac_, const Tensor &betas_,
                                        const Tensor &query_, bool exact) {
    const std::vector<Tensor> in{means_, covars_, opac_, betas_, query_};
    no_tangents("cond_mean_convariance_opacity", in);
    Tensor om, oV, oo;
    variable_list s;
    {
        const at::NoGradGuard no_grad;
        for (const Tensor &t : in) s.push_back(f32(t));
        const c10::cuda::CUDAGuard guard(s[0].device());
        const int64_t N = s[0].size(0), D = s[0].size(1);
        om = fempty({N, 3}, s[0]);
        oV = fempty({N, 3, 3}, s[0]);
        oo = fempty({N, 1}, s[0]);
        UBS_CALL(ubs_cond_fwd, N, (int32_t)D, fp(s[0]), fp(s[1]), fp(s[2]), fp(s[3]), fp(s[4]),
                 fpm(om), fpm(oV), fpm(oo), stream_of(s[0]));
    }
    // no gradient through the query, as in the reference (but a node)
    if (wants_grad(in))
        attach("CondMeanConvarianceOpacityBackward", in, {om, oV, oo}, s, {},
               [exact](OpNode &node, const variable_list &saved, variable_list &g) {
                   const at::NoGradGuard no_grad;
                   const variable_list s = node.for_kernel(saved);
                   const c10::cuda::CUDAGuard guard(s[0].device());
                   const int64_t N = s[0].size(0), D = s[0].size(1);
                   const Tensor vm = grad_or_zeros(g[0], {N, 3}, s[0]);
                   const Tensor vV = grad_or_zeros(g[1], {N, 3, 3}, s[0]);
                   const Tensor vo = grad_or_zeros(g[2], {N, 1}, s[0]);
                   variable_list o{fempty({N, D}, s[0]), fempty({N, D, D}, s[0]),
                                   fempty(s[2].sizes(), s[0]), fempty({N, D - 3}, s[0]),
                                   Tensor()};
                   UBS_CALL(ubs_cond_bwd, N, (int32_t)D, fp(s[0]), fp(s[1]), fp(s[2]), fp(s[3]),
                            fp(s[4]), fp(vm), fp(vV), fp(vo), fpm(o[0]), fpm(o[1]), fpm(o[2]),
                            fpm(o[3]), (int32_t)exact, stream_of(s[0]));
                   return o;
               });
    return {om, oV, oo};
}

Tensor rotmat(const Tensor &l_triangle) {
    no_tangents("l_triangle_to_rotmat", {l_triangle});
    Tensor R;
    {
        const at::NoGradGuard no_grad;
        const Tensor l = f32(l_triangle);
        const c10::cuda::CUDAGuard guard(l.device());
        R = fempty({l.size(0), 3, 3}, l);
        UBS_CALL(ubs_l_triangle_to_rotmat_fwd, l.size(0), fp(l), l.size(1), fpm(R), stream_of(l));
    }
    if (wants_grad({l_triangle}))
        attach("LTriangleToRotmatBackward", {l_triangle}, {R}, {}, {},
               [](OpNode &, const variable_list &, variable_list &g) {
                   const at::NoGradGuard no_grad;
                   if (!g[0].defined()) return variable_list(1);
                   const Tensor v = f32(g[0]);
                   const c10::cuda::CUDAGuard guard(v.device());
                   Tensor o = fempty({v.size(0), 3}, v);
                   UBS_CALL(ubs_l_triangle_to_rotmat_bwd, v.size(0), fp(v), fpm(o), stream_of(v));
                   return variable_list{o};
               });
    return R;
}

Tensor covar(const Tensor &rot_, const Tensor &scale_, const Tensor &lt_, const Tensor &rest_i,
             const Tensor &rest_j, bool spatial_block) {
    no_tangents("rot_scale_l_triangle_to_covar", {rot_, scale_, lt_});
    Tensor out;
    variable_list s;
    {
        const at::NoGradGuard no_grad;
        s = {f32(rot_), f32(scale_), f32(lt_)};
        const c10::cuda::CUDAGuard guard(s[0].device());
        for (const Tensor &r : {rest_i, rest_j})
            s.push_back(r.to(s[0].device(), at::kInt).contiguous());
        const int64_t N = s[1].size(0), D = s[1].size(1), dim = spatial_block || D == 3 ? 3 : D;
        out = fempty({N, dim, dim}, s[0]);
        UBS_CALL(ubs_rot_scale_l_triangle_to_covar_fwd, N, (int32_t)D, fp(s[0]), fp(s[1]), fp(s[2]),
                 s[3].const_data_ptr<int32_t>(), s[4].const_data_ptr<int32_t>(),
                 (int32_t)s[3].numel(), (int32_t)spatial_block, fpm(out), stream_of(s[0]));
    }
    if (wants_grad({rot_, scale_, lt_}))
        attach("RotScaleLTriangleToCovarBackward", {rot_, scale_, lt_}, {out}, s, {},
               [spatial_block](OpNode &node, const variable_list &saved, variable_list &g) {
                   const at::NoGradGuard no_grad;
                   if (!g[0].defined()) return variable_list(3);
                   const variable_list s = node.for_kernel(saved);
                   const c10::cuda::CUDAGuard guard(s[0].device());
                   const int64_t N = s[1].size(0), D = s[1].size(1);
                   const Tensor v = f32(g[0]);
                   variable_list o{fempty({N, 3, 3}, s[0]), fempty({N, D}, s[0]),
                                   fempty({N, D * (D - 1) / 2}, s[0])};
                   UBS_CALL(ubs_rot_scale_l_triangle_to_covar_bwd, N, (int32_t)D, fp(s[0]),
                            fp(s[1]), fp(s[2]), s[3].const_data_ptr<int32_t>(),
                            s[4].const_data_ptr<int32_t>(), (int32_t)s[3].numel(),
                            (int32_t)spatial_block, fp(v), fpm(o[0]), fpm(o[1]), fpm(o[2]),
                            stream_of(s[0]));
                   return o;
               });
    return out;
}

std::tuple<Tensor, Tensor, Tensor, Tensor, OptTensor> projection(const Tensor &means_, const OptTensor &covars_, const OptTensor &quats_,
                     const OptTensor &scales_, const Tensor &viewmats_, const Tensor &Ks_,
                     int32_t W, int32_t H, double eps2d, double near_p, double far_p, double clip,
                     bool with_comps) {
    const std::vector<Tensor> in{means_, covars_.value_or(Tensor()), quats_.value_or(Tensor()),
                                 scales_.value_or(Tensor()), viewmats_, Ks_};
    no_tangents("fully_fused_projection", in);
    Tensor radii, m2, dep, con, comp;
    variable_list s(6);
    int32_t layout = 0;
    {
        const at::NoGradGuard no_grad;
        for (int i = 0; i < 6; ++i)
            if (in[i].defined() && (i == 0 || i > 3 || (i == 1) == in[1].defined())) s[i] = f32(in[i]);
        const c10::cuda::CUDAGuard guard(s[0].device());
        if (s[1].defined()) layout = s[1].dim() == 3 ? 9 : 6;
        const int64_t C = s[4].size(0), N = s[0].size(0);
        radii = at::empty({C, N}, s[0].options().dtype(at::kInt));
        m2 = fempty({C, N, 2}, s[0]);
        dep = fempty({C, N}, s[0]);
        con = fempty({C, N, 3}, s[0]);
        if (with_comps) comp = fempty({C, N}, s[0]);
        UBS_CALL(ubs_projection_fwd, (int32_t)C, N, fp(s[0]), fp(s[1]), layout, fp(s[2]), fp(s[3]),
                 fp(s[4]), fp(s[5]), W, H, (float)eps2d, (float)near_p, (float)far_p, (float)clip,
                 radii.mutable_data_ptr<int32_t>(), fpm(m2), fpm(dep), fpm(con), fpm(comp),
                 stream_of(s[0]));
    }
    if (wants_grad(in)) {
        std::vector<Tensor> outs{m2, dep, con}, so{con};
        if (with_comps) {
            outs.push_back(comp);
            so.push_back(comp);
        }
        s.push_back(radii);
        attach("FullyFusedProjectionBackward", in, outs, s, so,
               [=](OpNode &node, const variable_list &saved, variable_list &g) {
                   const at::NoGradGuard no_grad;
                   const variable_list s = node.for_kernel(saved);
                   const c10::cuda::CUDAGuard guard(s[0].device());
                   const int64_t C = s[4].size(0), N = s[0].size(0);
                   const Tensor vm = grad_or_zeros(g[0], {C, N, 2}, s[0]);
                   const Tensor vd = grad_or_zeros(g[1], {C, N}, s[0]);
                   const Tensor vc = grad_or_zeros(g[2], {C, N, 3}, s[0]);
                   const Tensor vk = with_comps ? grad_or_zeros(g[3], {C, N}, s[0]) : Tensor();
                   variable_list o(6); // none for the intrinsics
                   o[0] = fempty({N, 3}, s[0]);
                   if (s[1].defined()) {
                       o[1] = at::empty_like(s[1]);
                   } else {
                       o[2] = fempty({N, 4}, s[0]);
                       o[3] = fempty({N, 3}, s[0]);
                   }
                   if (node.task_should_compute_output(4)) o[4] = fempty({C, 4, 4}, s[0]);
                   UBS_CALL(ubs_projection_bwd, (int32_t)C, N, fp(s[0]), fp(s[1]), layout, fp(s[2]),
                            fp(s[3]), fp(s[4]), fp(s[5]), W, H, (float)eps2d,
                            s[6].const_data_ptr<int32_t>(), fp(s[7]),
                            with_comps ? fp(s[8]) : nullptr, fp(vm), fp(vd), fp(vc), fp(vk),
                            fpm(o[0]), fpm(o[1]), fpm(o[2]), fpm(o[3]), fpm(o[4]),
                            stream_of(s[0]));
                   return o;
               });
    }
    return {radii, m2, dep, con, with_comps ? OptTensor(comp) : std::nullopt};
}

// (tiles_per_gauss, isect_ids, flatten_ids, isect_offsets)
std::tuple<Tensor, Tensor, Tensor, Tensor> isect(const Tensor &means2d_, const Tensor &radii_,
                                                 const Tensor &depths_, int32_t ts, int32_t tw,
                                                 int32_t th, bool sort) {
    const at::NoGradGuard no_grad;
    const Tensor m2 = f32(means2d_), dep = f32(depths_);
    const c10::cuda::CUDAGuard guard(m2.device());
    TORCH_CHECK_VALUE(radii_.is_cuda(), "expected a CUDA tensor, got device ", radii_.device());
    const Tensor rad = radii_.to(at::kInt).contiguous();
    const int64_t C = m2.size(0), N = m2.size(1);
    const int32_t nt = tw * th;
    const auto ints = m2.options().dtype(at::kInt);
    void *st = stream_of(m2);
    Tensor tpg = at::empty({C, N}, ints), off = at::empty({C, th, tw}, ints);
    Tensor ws = bytes(ubs_isect_count_workspace_bytes((int32_t)C, N, nt), m2);
    int64_t T = 0;
    UBS_CALL(ubs_isect_count, (int32_t)C, N, fp(m2), rad.const_data_ptr<int32_t>(), fp(dep), ts, tw,
             th, tpg.mutable_data_ptr<int32_t>(), off.mutable_data_ptr<int32_t>(), &T,
             ws.mutable_data_ptr(), ws.nbytes(), st);
    Tensor ids = at::empty({T}, m2.options().dtype(at::kLong)), fl = at::empty({T}, ints);
    if (T > 0) {
        Tensor w2 = bytes(ubs_isect_sort_workspace_bytes((int32_t)C, N, nt, T), m2);
        UBS_CALL(ubs_isect_emit, (int32_t)C, N, fp(m2), rad.const_data_ptr<int32_t>(), fp(dep), ts,
                 tw, th, tpg.const_data_ptr<int32_t>(), off.const_data_ptr<int32_t>(), T,
                 (int32_t)sort, ids.mutable_data_ptr<int64_t>(), fl.mutable_data_ptr<int32_t>(),
                 w2.mutable_data_ptr(), w2.nbytes(), st);
    }
    return {tpg, ids, fl, off};
}

Tensor offset_encode(const Tensor &ids_, int32_t C, int32_t tw, int32_t th) {
    const at::NoGradGuard no_grad;
    TORCH_CHECK_VALUE(ids_.is_cuda(), "expected a CUDA tensor, got device ", ids_.device());
    const Tensor ids = ids_.to(at::kLong).contiguous();
    const c10::cuda::CUDAGuard guard(ids.device());
    Tensor off = at::empty({C, th, tw}, ids.options().dtype(at::kInt));
    UBS_CALL(ubs_isect_offset_encode, ids.numel(), ids.const_data_ptr<int64_t>(), C, tw, th,
             off.mutable_data_ptr<int32_t>(), stream_of(ids));
    return off;
}

std::tuple<Tensor, Tensor> raster(const Tensor &means2d_, const Tensor &conics_,
                                  const Tensor &colors_, const Tensor &opac_, const Tensor &betas_,
                                  const OptTensor &bg_, const OptTensor &masks_, int32_t W,
                                  int32_t H, int32_t ts, const Tensor &offsets_,
                                  const Tensor &flatten_) {
    const std::vector<Tensor> in{means2d_, conics_, colors_, opac_, betas_,
                                 bg_.value_or(Tensor())};
    no_tangents("rasterize_to_pixels", in);
    Tensor rc, ra, last, ws;
    variable_list s(6);
    {
        const at::NoGradGuard no_grad;
        for (int i = 0; i < 6; ++i)
            if (in[i].defined()) s[i] = f32(in[i]);
        const c10::cuda::CUDAGuard guard(s[0].device());
        for (const Tensor &t : {offsets_, flatten_})
            TORCH_CHECK_VALUE(t.is_cuda(), "expected a CUDA tensor, got device ", t.device());
        Tensor mask;
        if (masks_) {
            TORCH_CHECK_VALUE(masks_->is_cuda(), "expected a CUDA tensor, got device ",
                              masks_->device());
            mask = masks_->to(at::kByte).contiguous();
        }
        s.push_back(mask);
        s.push_back(offsets_.to(at::kInt).contiguous());
        s.push_back(flatten_.to(at::kInt).contiguous());
        const int64_t C = s[2].size(0), N = s[2].size(1), ch = s[2].size(2), T = s[8].numel();
        rc = fempty({C, H, W, ch}, s[0]);
        ra = fempty({C, H, W, 1}, s[0]);
        last = at::empty({C, H, W}, s[0].options().dtype(at::kInt));
        ws = bytes(ubs_raster_workspace_bytes(T, (int32_t)ch), s[0]);
        void *st = stream_of(s[0]);
        // one record per sorted intersection; the backward reuses the records
        UBS_CALL(ubs_raster_pack, (int32_t)C, N, (int32_t)ch, T, s[8].const_data_ptr<int32_t>(),
                 fp(s[0]), fp(s[1]), fp(s[3]), fp(s[4]), fp(s[2]), ws.mutable_data_ptr(),
                 ws.nbytes(), st);
        UBS_CALL(ubs_raster_fwd_packed, (int32_t)C, N, (int32_t)ch, T, fp(s[2]), fp(s[5]),
                 mask.defined() ? mask.const_data_ptr<uint8_t>() : nullptr, W, H, ts,
                 (int32_t)s[7].size(2), (int32_t)s[7].size(1), s[7].const_data_ptr<int32_t>(),
                 fpm(rc), fpm(ra), last.mutable_data_ptr<int32_t>(), 0, ws.mutable_data_ptr(),
                 ws.nbytes(), st);
    }
    if (wants_grad(in)) {
        s.push_back(last);
        auto held = std::make_shared<Tensor>(ws); // released by the backward
        attach("RasterizeToPixelsBackward", in, {rc, ra}, s, {ra},
               [=](OpNode &node, const variable_list &saved, variable_list &g) {
                   const at::NoGradGuard no_grad;
                   const variable_list s = node.for_kernel(saved);
                   TORCH_CHECK(held->defined(), "rasterize_to_pixels: the records were released "
                                                "by an earlier backward");
                   const c10::cuda::CUDAGuard guard(s[0].device());
                   const int64_t C = s[2].size(0), N = s[2].size(1), ch = s[2].size(2),
                                 T = s[8].numel();
                   const Tensor vc = grad_or_zeros(g[0], {C, H, W, ch}, s[0]);
                   const Tensor va = grad_or_zeros(g[1], {C, H, W, 1}, s[0]);
                   variable_list o(6);
                   for (int i = 0; i < 5; ++i) o[i] = fempty(s[i].sizes(), s[0]);
                   UBS_CALL(ubs_raster_bwd_packed, (int32_t)C, N, (int32_t)ch, T, fp(s[2]),
                            fp(s[5]), s[6].defined() ? s[6].const_data_ptr<uint8_t>() : nullptr, W,
                            H, ts, (int32_t)s[7].size(2), (int32_t)s[7].size(1),
                            s[7].const_data_ptr<int32_t>(), fp(s[10]),
                            s[9].const_data_ptr<int32_t>(), fp(vc), fp(va), fpm(o[0]), fpm(o[1]),
                            fpm(o[2]), fpm(o[3]), fpm(o[4]), 1, held->mutable_data_ptr(),
                            held->nbytes(), stream_of(s[0]));
                   held->reset();
                   if (s[5].defined() && node.task_should_compute_output(5))
                       o[5] = (vc * (1.0 - s[10])).sum(at::IntArrayRef{1, 2});
                   return o;
               });
    }
    return {rc, ra};
}

void timing_start() {
    std::lock_guard<std::mutex> lk(g_timing.mu);
    g_timing.rec.clear();
    g_timing.on = true;
}
// [(entry point, ms)] of the calls since timing_start; the device is idle.
std::vector<std::pair<std::string, double>> timing_stop() {
    std::lock_guard<std::mutex> lk(g_timing.mu);
    g_timing.on = false;
    std::vector<std::pair<std::string, double>> out;
    for (auto &[name, e0, e1] : g_timing.rec) out.emplace_back(name, (double)e0.elapsed_time(e1));
    g_timing.rec.clear();
    return out;
}

} // namespace

PYBIND11_MODULE(ubs_native, m) {
    py::class_<SceneCall, std::shared_ptr<SceneCall>>(m, "SceneCall")
        .def(py::init(&scene_call), py::arg("dim"), py::arg("tables"), py::arg("n_buckets"),
             py::arg("n_pixels"), py::arg("tile"), py::arg("eps2d"), py::arg("near"),
             py::arg("far"), py::arg("clip"), py::arg("exact"), py::arg("cap"));
    using NoGil = py::call_guard<py::gil_scoped_release>;
    py::class_<FrameStats, std::shared_ptr<FrameStats>>(m, "FrameStats")
        .def("wait", &FrameStats::wait, NoGil());
    m.def("scene_forward", &scene_forward, NoGil(), py::arg("call"), py::arg("params"),
          py::arg("bg"), py::arg("mask"), py::arg("color_mode"), py::arg("stats"), py::arg("grad"),
          py::arg("image") = py::none());
    m.def("pack_views", &pack_views, NoGil(), py::arg("viewmats"), py::arg("Ks"),
          py::arg("centers"), py::arg("times"), py::arg("widths"), py::arg("heights"),
          py::arg("tile"), py::arg("device"), py::arg("stream") = py::none());
    m.def("l1_loss", &l1_loss, NoGil());
    m.def("ssim_loss", &ssim_loss, NoGil());
    m.def("cond", &cond, NoGil());
    m.def("rotmat", &rotmat, NoGil());
    m.def("covar", &covar, NoGil());
    m.def("projection", &projection, NoGil());
    m.def("isect", &isect, NoGil());
    m.def("offset_encode", &offset_encode, NoGil());
    m.def("raster", &raster, NoGil());
    m.def("timing_start", &timing_start);
    m.def("timing_stop", &timing_stop);
}
