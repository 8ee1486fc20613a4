// Host side of the torch-level operators (lig_b200/ops.py): tensor checks,
// output and scratch allocation and the calls of the C ABI, for the paths a
// training loop or a decode takes on every iteration.
//
// At small images these paths are bound by the host: in Python each entry
// point cost 20-40 us of allocations, pointer conversions and stream lookups
// beside its launches.  Project + rasterize at 64x80 / 400 Gaussians: 164 us
// from Python in 14 launches, 83 from here; 60 now in 6 launches (25 us of device
// work).  A training iteration at 512^2 / 50k: 555 -> 347.  Every function runs without the GIL;
// nothing is kept between calls.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/extension.h>

#include <optional>
#include <stdexcept>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/lig_b200.h"

namespace {

using at::Tensor;
using Opt = std::optional<Tensor>;

namespace py = pybind11;

// Optional observer of the ABI calls (per-entry-point timing): called with
// (entry point, 0) before and (entry point, 1) after.
PyObject *g_observer = nullptr;

void observe(const char *name, int end) {
    if (!g_observer) return;
    py::gil_scoped_acquire gil;
    if (g_observer) py::reinterpret_borrow<py::object>(g_observer)(name, end);
}

// ValueError for invalid arguments, lig_b200._lib.LigError for the rest.
[[noreturn]] void raise_status(const char *name, int code) {
    if (code == LIG_ERR_INVALID) throw py::value_error(std::string(name) + ": invalid argument");
    py::gil_scoped_acquire gil;
    py::object cls = py::module_::import("lig_b200._lib").attr("LigError");
    PyErr_SetObject(cls.ptr(), cls(name, code).ptr());
    throw py::error_already_set();
}

template <typename F> void call(const char *name, F f) {
    observe(name, 0);
    const int rc = f();
    if (rc != LIG_OK) raise_status(name, rc);
    observe(name, 1);
}

void check_cuda(std::initializer_list<const Tensor *> ts) {
    for (const Tensor *t : ts)
        if (t->defined() && !t->is_cuda())
            throw std::runtime_error("lig_b200: tensors must be CUDA tensors (no CPU fallback)");
}

int dtype_code(const Tensor &t) {
    if (t.scalar_type() == at::kFloat) return LIG_F32;
    if (t.scalar_type() == at::kDouble) return LIG_F64;
    throw py::type_error(std::string("lig_b200 kernels take float32 or float64 tensors, got ") +
                               c10::toString(t.scalar_type()));
}

Tensor cont(const Tensor &t, at::ScalarType dt) {
    if (!t.defined()) return t;
    return (t.scalar_type() == dt ? t : t.to(dt)).contiguous();
}
Tensor value(const Opt &t) { return t.has_value() ? *t : Tensor(); }

void *ptr(const Tensor &t) { return t.defined() ? t.data_ptr() : nullptr; }

void *stream_of(const Tensor &t) {
    return (void *)c10::cuda::getCurrentCUDAStream(t.get_device()).stream();
}

Tensor empty(at::IntArrayRef sizes, const Tensor &like, at::ScalarType dt) {
    return at::empty(sizes, like.options().dtype(dt).requires_grad(false));
}

// row-strided view accepted by the kernels (unit inner stride)
Tensor rows(const Tensor &t, int64_t width) {
    if (t.dim() != 2 || t.size(1) != width || t.stride(1) != 1 || t.stride(0) < width)
        return t.contiguous();
    return t;
}

// ---------------------------------------------------------------- projection
std::vector<Tensor> project_fwd(const Tensor &in, const Tensor &means, const Opt &opac, int64_t h,
                                int64_t w, int64_t block, bool chol) {
    const Tensor op0 = value(opac);
    check_cuda({&in, &means, &op0});
    const Tensor in3 = in.contiguous();
    const at::ScalarType dt = in3.scalar_type();
    const Tensor mu = cont(means, dt), op = cont(op0, dt);
    const int code = dtype_code(in3);
    const int64_t n = in3.size(0);
    Tensor xys = empty({n, 2}, in3, dt), ext = empty({n, 2}, in3, dt), con = empty({n, 3}, in3, dt),
           cnt = empty({n}, in3, at::kInt);
    call("lig_project_fwd", [&] {
        return lig_project_fwd(code, (int)n, chol, ptr(in3), ptr(mu), ptr(op), (int)h, (int)w,
                               (int)block, ptr(xys), ptr(ext), ptr(con), (int32_t *)ptr(cnt),
                               stream_of(in3));
    });
    return {xys, ext, con, cnt};
}

std::vector<Tensor> project_bwd(const Tensor &in, const Tensor &means, const Opt &opac, int64_t h,
                                int64_t w, int64_t block, bool chol, const Tensor &v_xy0,
                                const Tensor &v_con0) {
    check_cuda({&in, &means, &v_xy0, &v_con0});
    const Tensor in3 = in.contiguous();
    const at::ScalarType dt = in3.scalar_type();
    const Tensor mu = cont(means, dt), op = cont(value(opac), dt);
    const Tensor v_xy = rows(v_xy0.to(dt), 2), v_con = rows(v_con0.to(dt), 3);
    const int code = dtype_code(in3);
    const int64_t n = in3.size(0);
    Tensor v_in3 = empty({n, 3}, in3, dt), v_mean = empty({n, 2}, in3, dt);
    call("lig_project_bwd", [&] {
        return lig_project_bwd(code, (int)n, chol, ptr(in3), ptr(mu), ptr(op), (int)h, (int)w,
                               (int)block, ptr(v_xy), v_xy.stride(0), ptr(v_con), v_con.stride(0),
                               ptr(v_in3), ptr(v_mean), stream_of(in3));
    });
    return {v_in3, v_mean};
}

// ------------------------------------------------------------------- binning
struct Binned {
    Tensor gids, bins, isect, ids, isect_sorted;
};

Tensor cumsum(const Tensor &counts, Tensor &total) {
    const Tensor cnt = cont(counts.reshape(-1), at::kInt);
    const int64_t n = cnt.size(0);
    Tensor cum = empty({n}, cnt, at::kInt);
    total = empty({1}, cnt, at::kInt);
    const size_t wsb = lig_cumsum_workspace_bytes((int)n);
    Tensor ws = empty({(int64_t)wsb}, cnt, at::kByte);
    call("lig_cumsum_tiles", [&] {
        return lig_cumsum_tiles((int)n, (const int32_t *)ptr(cnt), (int32_t *)ptr(cum),
                                (int32_t *)ptr(total), ptr(ws), wsb, stream_of(cnt));
    });
    return cum;
}

std::tuple<Tensor, Tensor> cumsum_tiles(const Tensor &counts) {
    check_cuda({&counts});
    Tensor total;
    Tensor cum = cumsum(counts, total);
    return {cum, total};
}

Binned run_bin(const Tensor &xys, const Tensor &ext, const Tensor &cum, const Tensor &total,
               int64_t h, int64_t w, int64_t block, int64_t capacity, bool want_keys) {
    const int64_t T = ((w + block - 1) / block) * ((h + block - 1) / block), n = xys.size(0);
    const int64_t cap = std::max<int64_t>(capacity, 0), len = std::max<int64_t>(cap, 1);
    const size_t wsb = lig_bin_workspace_bytes((int)n, (int)cap, (int)T);
    Tensor ws = empty({(int64_t)std::max<size_t>(wsb, 1)}, xys, at::kByte);
    Binned b;
    b.gids = empty({len}, xys, at::kInt);
    b.bins = empty({T, 2}, xys, at::kInt);
    Tensor status = empty({1}, xys, at::kInt);
    if (want_keys) {
        b.isect = empty({len}, xys, at::kLong);
        b.ids = empty({len}, xys, at::kInt);
        b.isect_sorted = empty({len}, xys, at::kLong);
    }
    const int code = dtype_code(xys);
    call("lig_bin", [&] {
        return lig_bin(code, (int)n, ptr(xys), ptr(ext), (const int32_t *)ptr(cum),
                       (const int32_t *)ptr(total), (int)h, (int)w, (int)block, (int)cap, ptr(ws),
                       wsb, (int32_t *)ptr(b.gids), (int32_t *)ptr(b.bins),
                       (int64_t *)ptr(b.isect), (int32_t *)ptr(b.ids),
                       (int64_t *)ptr(b.isect_sorted), (int32_t *)ptr(status), stream_of(xys));
    });
    return b;
}

std::vector<Opt> as_list(const Binned &b) {
    auto o = [](const Tensor &t) { return t.defined() ? Opt(t) : Opt(); };
    return {b.gids, b.bins, o(b.isect), o(b.ids), o(b.isect_sorted)};
}

std::vector<Opt> run_bin_py(const Tensor &xys, const Tensor &ext, const Tensor &cum,
                            const Tensor &total, int64_t h, int64_t w, int64_t block,
                            int64_t capacity, bool want_keys) {
    return as_list(run_bin(xys, ext, cum, total, h, w, block, capacity, want_keys));
}

// ----------------------------------------------------------------- rasterizer
std::vector<Opt> raster_fwd(int64_t h, int64_t w, int64_t block, const Tensor &gids,
                            const Tensor &bins, const Tensor &total, const Tensor &xys0,
                            const Tensor &con0, const Tensor &col0, const Opt &op0,
                            bool grad_aware) {
    const Tensor opv = value(op0);
    check_cuda({&xys0, &con0, &col0, &opv, &bins, &total});
    const Tensor xys = xys0.contiguous();
    const at::ScalarType dt = xys.scalar_type();
    const Tensor con = cont(con0, dt), col = cont(col0, dt), op = cont(opv, dt);
    const int64_t n = xys.size(0);
    const int code = dtype_code(xys);
    const size_t wsb = lig_raster_workspace_bytes(code, (int)n);
    Tensor ws = empty({(int64_t)wsb}, xys, at::kByte);
    Tensor img = empty({h, w, 3}, xys, dt), wsum = empty({h, w}, xys, dt),
           fin = empty({h, w}, xys, at::kInt), dx, dy, dxy;
    if (grad_aware) {
        dx = at::empty_like(img);
        dy = at::empty_like(img);
        dxy = at::empty_like(img);
    }
    call("lig_raster_fwd", [&] {
        return lig_raster_fwd(code, (int)h, (int)w, (int)block, (int)n, (const int32_t *)ptr(gids),
                              (const int32_t *)ptr(bins), (const int32_t *)ptr(total), ptr(xys),
                              ptr(con), ptr(col), ptr(op), ptr(ws), wsb, ptr(img), ptr(wsum),
                              ptr(dx), ptr(dy), ptr(dxy), (int32_t *)ptr(fin), stream_of(xys));
    });
    auto o = [](const Tensor &t) { return t.defined() ? Opt(t) : Opt(); };
    return {img, wsum, o(dx), o(dy), o(dxy), fin};
}

// Prefix sum, binning and forward rasterizer behind each other.  capacity < 0:
// wait for the intersection count before sizing the lists; else size them with
// that guess, check the count once everything is enqueued and redo binning and
// rasterizer when the guess was too small.  slot: pinned int32 [1] of the
// calling thread.  Returns (count, capacity, (cum, total), binning, images).
std::tuple<int64_t, int64_t, std::vector<Tensor>, std::vector<Opt>, std::vector<Opt>>
bin_raster_fwd(const Tensor &xys0, const Tensor &ext0, const Tensor &counts, const Tensor &con,
               const Tensor &col, const Opt &op, int64_t h, int64_t w, int64_t block,
               bool grad_aware, int64_t capacity, const Tensor &slot) {
    check_cuda({&xys0, &ext0, &counts});
    const Tensor xys = xys0.contiguous(), ext = cont(ext0, xys.scalar_type());
    Tensor total;
    const Tensor cum = cumsum(counts, total);
    const auto stream = c10::cuda::getCurrentCUDAStream(xys.get_device());
    C10_CUDA_CHECK(cudaMemcpyAsync(slot.data_ptr(), total.data_ptr(), sizeof(int32_t),
                                   cudaMemcpyDeviceToHost, stream));
    // (also when a later call throws: the slot is the thread's, and free again
    // once this function is left)
    struct Arrival {
        at::cuda::CUDAEvent event;
        bool waited = false;
        void wait() {
            waited = true;
            event.synchronize();
        }
        ~Arrival() {
            try {
                if (!waited) wait();
            } catch (...) {  // the CUDA error is the caller's next one
            }
        }
    } arrived;
    arrived.event.record(stream);
    auto wait = [&]() -> int64_t {
        arrived.wait();
        return *slot.data_ptr<int32_t>();
    };
    const bool guess = capacity >= 0;
    int64_t m = guess ? -1 : wait();
    int64_t cap = guess ? capacity : m;
    Binned b = run_bin(xys, ext, cum, total, h, w, block, cap, false);
    std::vector<Opt> img =
        raster_fwd(h, w, block, b.gids, b.bins, total, xys, con, col, op, grad_aware);
    if (guess) {
        m = wait();
        if (m > cap) {
            cap = m;
            b = run_bin(xys, ext, cum, total, h, w, block, cap, false);
            img = raster_fwd(h, w, block, b.gids, b.bins, total, xys, con, col, op, grad_aware);
        }
    }
    return {m, cap, {cum, total}, as_list(b), img};
}

std::vector<Opt> raster_bwd(int64_t h, int64_t w, int64_t block, const Tensor &gids,
                            const Tensor &bins, const Tensor &total, const Tensor &xys0,
                            const Tensor &con0, const Tensor &col0, const Opt &op0,
                            const Tensor &final_idx, const Tensor &v_img0, const Opt &v_wsum0,
                            const Opt &v_dx0, const Opt &v_dy0, const Opt &v_dxy0,
                            double alpha_clamp) {
    check_cuda({&xys0, &con0, &col0, &final_idx, &v_img0});
    const Tensor xys = xys0.contiguous();
    const at::ScalarType dt = xys.scalar_type();
    const Tensor con = cont(con0, dt), col = cont(col0, dt), op = cont(value(op0), dt);
    const Tensor v_img = cont(v_img0, dt), v_wsum = cont(value(v_wsum0), dt);
    const Tensor v_dx = cont(value(v_dx0), dt), v_dy = cont(value(v_dy0), dt),
                 v_dxy = cont(value(v_dxy0), dt);
    const Tensor fin = cont(final_idx, at::kInt);
    const int64_t n = xys.size(0);
    const int code = dtype_code(xys);
    const size_t wsb = lig_raster_workspace_bytes(code, (int)n);
    Tensor ws = empty({(int64_t)wsb}, xys, at::kByte);
    Tensor v_xy = empty({n, 2}, xys, dt), v_abs = empty({n, 2}, xys, dt),
           v_con = empty({n, 3}, xys, dt), v_rgb = empty({n, 3}, xys, dt), v_op;
    if (op.defined()) v_op = empty({n}, xys, dt);
    call("lig_raster_bwd", [&] {
        return lig_raster_bwd(code, (int)h, (int)w, (int)block, (int)n, (const int32_t *)ptr(gids),
                              (const int32_t *)ptr(bins), (const int32_t *)ptr(total), ptr(xys),
                              ptr(con), ptr(col), ptr(op), (const int32_t *)ptr(fin), ptr(v_img),
                              ptr(v_wsum), ptr(v_dx), ptr(v_dy), ptr(v_dxy), alpha_clamp, ptr(ws),
                              wsb, ptr(v_xy), ptr(v_abs), ptr(v_con), ptr(v_rgb), ptr(v_op),
                              stream_of(xys));
    });
    return {v_xy, v_abs, v_con, v_rgb, v_op.defined() ? Opt(v_op) : Opt()};
}

// -------------------------------------------------------------------- upscale
void upscale_channels(int64_t c) {
    if (c != 1 && c != 3)
        throw py::value_error("gradient-aware upscale expects [H, W, 3] (or [H, W, 1]) planes");
}

Tensor upscale_fwd(const Tensor &render0, const Tensor &dx0, const Tensor &dy0, const Tensor &dxy0,
                   int64_t dst_h, int64_t dst_w, std::optional<std::vector<double>> roi,
                   int64_t mode) {
    check_cuda({&render0, &dx0, &dy0, &dxy0});
    const Tensor f = render0.contiguous();
    const at::ScalarType dt = f.scalar_type();
    const Tensor dx = cont(dx0, dt), dy = cont(dy0, dt), dxy = cont(dxy0, dt);
    if (f.dim() != 3) throw py::value_error("not enough values to unpack (expected 3)");
    const int64_t h = f.size(0), w = f.size(1), c = f.size(2);
    upscale_channels(c);
    const std::vector<double> r = roi ? *roi : std::vector<double>{0., 0., (double)w, (double)h};
    Tensor out = empty({dst_h, dst_w, c}, f, dt);
    const int code = dtype_code(f);
    call("lig_upscale_fwd_nc", [&] {
        return lig_upscale_fwd_nc(code, (int)mode, (int)c, (int)h, (int)w, (int)dst_h, (int)dst_w,
                                  r.at(0), r.at(1), r.at(2), r.at(3), ptr(f), ptr(dx), ptr(dy),
                                  ptr(dxy), ptr(out), stream_of(f));
    });
    return out;
}

std::vector<Tensor> upscale_bwd(const Tensor &grad, int64_t h, int64_t w,
                                std::optional<std::vector<double>> roi, int64_t mode) {
    check_cuda({&grad});
    const Tensor g = grad.contiguous();
    const at::ScalarType dt = g.scalar_type();
    if (g.dim() != 3) throw py::value_error("not enough values to unpack (expected 3)");
    const int64_t dh = g.size(0), dw = g.size(1), c = g.size(2);
    upscale_channels(c);
    const std::vector<double> r = roi ? *roi : std::vector<double>{0., 0., (double)w, (double)h};
    std::vector<Tensor> o;
    for (int k = 0; k < 4; ++k) o.push_back(empty({h, w, c}, g, dt));
    const int code = dtype_code(g);
    call("lig_upscale_bwd_nc", [&] {
        return lig_upscale_bwd_nc(code, (int)mode, (int)c, (int)h, (int)w, (int)dh, (int)dw,
                                  r.at(0), r.at(1), r.at(2), r.at(3), ptr(g), ptr(o[0]), ptr(o[1]),
                                  ptr(o[2]), ptr(o[3]), stream_of(g));
    });
    return o;
}

}  // namespace

// Errors leave as torch's own Python exceptions (out of memory and the like).
#define LIG_DEF(f, name) m.def(name, torch::wrap_pybind_function_no_gil(f))

PYBIND11_MODULE(_host, m) {
    LIG_DEF(project_fwd, "project_fwd");
    LIG_DEF(project_bwd, "project_bwd");
    LIG_DEF(cumsum_tiles, "cumsum_tiles");
    LIG_DEF(run_bin_py, "run_bin");
    LIG_DEF(raster_fwd, "raster_fwd");
    LIG_DEF(bin_raster_fwd, "bin_raster_fwd");
    LIG_DEF(raster_bwd, "raster_bwd");
    LIG_DEF(upscale_fwd, "upscale_fwd");
    LIG_DEF(upscale_bwd, "upscale_bwd");
    m.def("set_observer", [](py::object f) {
        PyObject *old = g_observer;
        g_observer = f.is_none() ? nullptr : f.inc_ref().ptr();
        Py_XDECREF(old);
    });
}
