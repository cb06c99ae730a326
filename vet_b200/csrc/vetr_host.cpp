// Native host side of vet_b200/render.py: what a call of the rasterizer does on the host besides the launches - output tensors,
// addresses, parameter blocks - without an interpreter step per tensor.  A CPython extension over libtorch; the kernels
// are reached through include/vetr.h, by addresses that bind() is given, so that the library Python has loaded is the one
// that is called.  No state but those addresses.
//
// Why: a training batch of a small scene is bound by the host.  5 k points, two views 96x64, camera gradients: a pass takes
// 173 to 181 us with these steps in Python (64 us of it on the device), 84 to 89 us like this; 100 k points at 512x512 158 to
// 164 and 105 to 112 us (several GPUs; both times include a scan that became 3 us faster meanwhile).  The first again, 81 -> 73 us: parameters, addresses
// and sizes of a call in one step (scene), and output tensors without the dispatcher's way to at::empty (17 of them, 0.9 us each before).
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Device.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/torch.h>

#include <vector>

#include "../../include/vetr.h"

namespace
{
decltype(&vetr_forward) p_forward                       = nullptr;
decltype(&vetr_backward_phase) p_backward_phase         = nullptr;
decltype(&vetr_finalize_gradients) p_finalize_gradients = nullptr;
decltype(&vetr_l1_loss_grad) p_l1_loss_grad             = nullptr;
decltype(&vetr_zero_buffers) p_zero_buffers             = nullptr;
decltype(&vetr_pyramid_pixels) p_pyramid_pixels         = nullptr;
decltype(&vetr_list_capacity) p_list_capacity           = nullptr;

void require(bool ok, const char* what)
{
    TORCH_CHECK_VALUE(ok, what);
}
THPObjectPtr held(PyObject* o)  // a new reference, or the interpreter's error
{
    if (!o) throw python_error();
    return THPObjectPtr(o);
}
THPObjectPtr sequence(PyObject* o) { return held(PySequence_Fast(o, "expected a sequence")); }
long long integer(PyObject* o)
{
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
}
int32_t whole(PyObject* o)  // anything with __index__, cut to 32 bits as ctypes does
{
    THPObjectPtr i            = held(PyNumber_Index(o));
    const unsigned long long v = PyLong_AsUnsignedLongLongMask(i.get());
    if (v == ~0ull && PyErr_Occurred()) throw python_error();
    return (int32_t)v;
}
float real(PyObject* o)
{
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return (float)v;
}
template <typename T>
T* address(PyObject* o)
{
    return reinterpret_cast<T*>(integer(o));
}
// Tensors may be torch's own, or any object that answers to data_ptr() and the few others of a tensor's methods used here.
const at::Tensor* plain_tensor(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }
THPObjectPtr attribute(PyObject* o, const char* name)
{
    THPObjectPtr a(PyObject_GetAttrString(o, name));
    if (!a && PyErr_ExceptionMatches(PyExc_AttributeError))
    {
        PyErr_Clear();
        throw torch::TypeError("expected a tensor");
    }
    return held(a.release());
}
void* storage(PyObject* o)
{
    if (const at::Tensor* t = plain_tensor(o)) return t->data_ptr();
    return address<void>(held(PyObject_CallNoArgs(attribute(o, "data_ptr").get())).get());
}
// The same from the first dimension's index b0 on.
void* storage_from(PyObject* o, long long b0)
{
    if (b0 == 0) return storage(o);
    if (const at::Tensor* t = plain_tensor(o)) return static_cast<char*>(t->data_ptr()) + b0 * t->stride(0) * (long long)t->element_size();
    THPObjectPtr start = held(PyLong_FromLongLong(b0)), slice = held(PySlice_New(start.get(), nullptr, nullptr));
    return storage(held(PyObject_GetItem(o, slice.get())).get());
}
long long numel(PyObject* o)
{
    if (const at::Tensor* t = plain_tensor(o)) return t->numel();
    return integer(held(PyObject_CallNoArgs(attribute(o, "numel").get())).get());
}
int extent(PyObject* o, int dimension)  // of a tensor, or 0 for None
{
    if (o == Py_None) return 0;
    if (const at::Tensor* t = plain_tensor(o)) return (int)t->size(dimension);
    THPObjectPtr shape = attribute(o, "shape");
    return (int)integer(held(PySequence_GetItem(shape.get(), dimension)).get());
}
int rows(PyObject* o) { return extent(o, 0); }
template <typename T>
T* data(PyObject* o)  // a tensor, or None
{
    return o == Py_None ? nullptr : static_cast<T*>(storage(o));
}
at::TensorOptions on(PyObject* device, at::ScalarType type = at::kFloat)
{
    if (!THPDevice_Check(device)) throw torch::TypeError("expected a device");
    return at::TensorOptions().dtype(type).device(reinterpret_cast<THPDevice*>(device)->device);
}
// at::empty, without the dispatcher's way to it where the device is CUDA.
at::Tensor fresh(at::IntArrayRef size, const at::TensorOptions& opt)
{
    if (!opt.device().is_cuda()) return at::empty(size, opt);
    return at::Tensor(at::detail::empty_cuda(size, c10::typeMetaToScalarType(opt.dtype()), opt.device(), std::nullopt));
}
PyObject* wrap(at::Tensor t) { return held(THPVariable_Wrap(std::move(t))).release(); }

// Addresses, from view b0 on, of a sequence of per-level tensors [views, ...]; null for None.
struct Levels
{
    void* p[VETR_MAX_LAYERS] = {};
    bool given               = false;
    Levels(PyObject* list, long long b0, int levels)
    {
        if (list == Py_None) return;
        THPObjectPtr items = sequence(list);
        require(levels <= VETR_MAX_LAYERS && PySequence_Fast_GET_SIZE(items.get()) >= levels, "one tensor per level");
        for (int l = 0; l < levels; ++l) p[l] = storage_from(PySequence_Fast_GET_ITEM(items.get(), l), b0);
        given = true;
    }
    template <typename T>
    T* const* get() const
    {
        return given ? reinterpret_cast<T* const*>(p) : nullptr;
    }
};

struct Call
{
    PyObject* const* args;
    Py_ssize_t n;
    PyObject* operator[](Py_ssize_t i) const { return args[i]; }
    void expect(Py_ssize_t k) const { require(n == k, "wrong number of arguments"); }
};

PyObject* guarded(PyObject* (*f)(const Call&), PyObject* const* args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    return f(Call{args, n});
    END_HANDLE_TH_ERRORS
}

// bind(forward, backward_phase, finalize_gradients, l1_loss_grad, zero_buffers): addresses of the library's functions
PyObject* bind(const Call& c)
{
    c.expect(5);
    p_forward            = reinterpret_cast<decltype(p_forward)>(integer(c[0]));
    p_backward_phase     = reinterpret_cast<decltype(p_backward_phase)>(integer(c[1]));
    p_finalize_gradients = reinterpret_cast<decltype(p_finalize_gradients)>(integer(c[2]));
    p_l1_loss_grad       = reinterpret_cast<decltype(p_l1_loss_grad)>(integer(c[3]));
    p_zero_buffers       = reinterpret_cast<decltype(p_zero_buffers)>(integer(c[4]));
    Py_RETURN_NONE;
}

// bind_sizes(pyramid_pixels, list_capacity): the same
PyObject* bind_sizes(const Call& c)
{
    c.expect(2);
    p_pyramid_pixels = reinterpret_cast<decltype(p_pyramid_pixels)>(integer(c[0]));
    p_list_capacity  = reinterpret_cast<decltype(p_list_capacity)>(integer(c[1]));
    Py_RETURN_NONE;
}

// current_stream(device index) -> address of torch's current stream on that device
PyObject* current_stream(const Call& c)
{
    c.expect(1);
    return PyLong_FromVoidPtr(c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)integer(c[0])).stream());
}

// images(device, views, channels, w, h, levels, want_weight, want_mask, want_depth) -> (color, weight, mask, depth): lists of
// one tensor per level, or None
PyObject* images(const Call& c)
{
    c.expect(9);
    const auto opt  = on(c[0]);
    const int64_t B = integer(c[1]), C = integer(c[2]), w = integer(c[3]), h = integer(c[4]), levels = integer(c[5]);
    THPObjectPtr out = held(PyTuple_New(4));
    for (int kind = 0; kind < 4; ++kind)
    {
        const int wanted = kind == 0 ? 1 : PyObject_IsTrue(c[5 + kind]);
        if (wanted < 0) throw python_error();
        if (!wanted)
        {
            Py_INCREF(Py_None);
            PyTuple_SET_ITEM(out.get(), kind, Py_None);
            continue;
        }
        PyTuple_SET_ITEM(out.get(), kind, held(PyList_New(levels)).release());
        for (int64_t l = 0; l < levels; ++l)
            PyList_SET_ITEM(PyTuple_GET_ITEM(out.get(), kind), l, wrap(fresh({B, kind == 0 ? C : 1, h >> l, w >> l}, opt)));
    }
    return out.release();
}

// Every field from the dict's entry of that name, but the channel count.
void read_params(vetr_params& p, PyObject* dict, int32_t channels)
{
    const auto get = [&](const char* name)
    {
        THPObjectPtr key = held(PyUnicode_InternFromString(name));
        return held(PyObject_GetItem(dict, key.get()));
    };
    const auto i = [&](const char* name) { return whole(get(name).get()); };
    const auto f = [&](const char* name) { return real(get(name).get()); };
    p.render_mode = i("render_mode"), p.num_layers = i("num_layers"), i("num_channels"), p.num_channels = channels;
    p.drop_out_points_by_radius = i("drop_out_points_by_radius"), p.drop_out_radius_threshold = f("drop_out_radius_threshold");
    p.dist_cutoff = f("dist_cutoff"), p.use_environment_map = i("use_environment_map"), p.viewer_only = i("viewer_only");
    p.stability_cutoff_value = f("stability_cutoff_value"), p.debug_max_list_length = i("debug_max_list_length");
    p.need_point_gradient = i("need_point_gradient"), p.K_gradient_factor = f("K_gradient_factor");
    p.distortion_gradient_factor = f("distortion_gradient_factor"), p.output_background_mask_value = f("output_background_mask_value");
    p.background_alpha_to_point0 = i("background_alpha_to_point0"), p.keep_sorted_lists = i("keep_sorted_lists");
    p.depth_accept_blend = f("depth_accept_blend"), p.depth_accept = f("depth_accept"), p.ghost_gradients = i("ghost_gradients");
}

// params(address of vetr_params, dict, channels)
PyObject* params(const Call& c)
{
    c.expect(3);
    read_params(*address<vetr_params>(c[0]), c[1], (int32_t)integer(c[2]));
    Py_RETURN_NONE;
}

struct Scene  // _lib.Scene
{
    vetr_params params;
    vetr_cloud cloud;
    vetr_texture texture;
    vetr_cameras cameras;
};

// scene(address of Scene, dict of parameters, w, h, views, position, index, texture, confidence, background, poses, intrinsics) -> (points,
// levels, pixels of a view, capacity of the lists of that many views); the last two -1 where the library refuses the sizes
PyObject* scene(const Call& c)
{
    c.expect(12);
    Scene& s = *address<Scene>(c[0]);
    read_params(s.params, c[1], extent(c[7], 0));
    const int w = (int)integer(c[2]), h = (int)integer(c[3]), views = (int)integer(c[4]);
    s.cloud.position = static_cast<const float*>(storage(c[5])), s.cloud.index = static_cast<const int32_t*>(storage(c[6])), s.cloud.n = rows(c[5]);
    s.texture.texture = static_cast<const float*>(storage(c[7])), s.texture.confidence = static_cast<const float*>(storage(c[8]));
    s.texture.background = static_cast<const float*>(storage(c[9])), s.texture.n_tex = extent(c[7], 1);
    s.cameras.poses_se3 = static_cast<const double*>(storage(c[10])), s.cameras.intrinsics = static_cast<const float*>(storage(c[11]));
    s.cameras.n_img = rows(c[10]), s.cameras.n_cam = rows(c[11]);
    const long long pixels = p_pyramid_pixels(w, h, s.params.num_layers);
    const long long capacity = pixels > 0 ? p_list_capacity(s.cloud.n, views, w, h, &s.params) : -1;
    return held(Py_BuildValue("iiLL", s.cloud.n, s.params.num_layers, pixels, capacity)).release();
}

// views(address of an array of vetr_view, sequence of vet_b200.scenes.View)
PyObject* views(const Call& c)
{
    c.expect(2);
    vetr_view* out     = address<vetr_view>(c[0]);
    THPObjectPtr items = sequence(c[1]);
    for (Py_ssize_t k = 0; k < PySequence_Fast_GET_SIZE(items.get()); ++k)
    {
        PyObject* v    = PySequence_Fast_GET_ITEM(items.get(), k);
        const auto i   = [&](const char* name) { return whole(held(PyObject_GetAttrString(v, name)).get()); };
        const auto f   = [&](const char* name, float* to, Py_ssize_t n)
        {
            THPObjectPtr a = held(PyObject_GetAttrString(v, name)), s = sequence(a.get());
            const Py_ssize_t given = PySequence_Fast_GET_SIZE(s.get());
            require(given <= n, "crop has five entries and rot four");
            for (Py_ssize_t j = 0; j < n; ++j) to[j] = j < given ? real(PySequence_Fast_GET_ITEM(s.get(), j)) : 0.f;
        };
        vetr_view& o = out[k];
        o.w = i("w"), o.h = i("h"), o.image_index = i("image_index"), o.camera_index = i("camera_index"), o.camera_model = i("camera_model");
        f("crop", o.crop, 5), f("rot", o.rot, 4);
    }
    Py_RETURN_NONE;
}

// What forward and backward are given in common, in this order: ctx, params, cloud, texture, cameras, views, n_views, b0, dropout,
// lists, levels.  The structs are addresses; b0: first of the views in the images and in dropout ([views, n], or None).
struct Frame
{
    vetr_ctx* ctx;
    const vetr_params* params;
    const vetr_cloud* cloud;
    const vetr_texture* texture;
    const vetr_cameras* cameras;
    const vetr_view* views;
    int n_views;
    long long b0;
    const float* dropout;
    const vetr_lists* lists;
    int levels;
    explicit Frame(const Call& c)
        : ctx(address<vetr_ctx>(c[0])), params(address<const vetr_params>(c[1])), cloud(address<const vetr_cloud>(c[2])),
          texture(address<const vetr_texture>(c[3])), cameras(address<const vetr_cameras>(c[4])), views(address<const vetr_view>(c[5])),
          n_views((int)integer(c[6])), b0(integer(c[7])),
          dropout(c[8] == Py_None ? nullptr : static_cast<const float*>(storage_from(c[8], b0))), lists(address<const vetr_lists>(c[9])),
          levels((int)integer(c[10]))
    {
    }
};

// forward(<Frame>, color, weight, mask, depth) -> status
PyObject* forward(const Call& c)
{
    c.expect(15);
    const Frame f(c);
    const Levels color(c[11], f.b0, f.levels), weight(c[12], f.b0, f.levels), mask(c[13], f.b0, f.levels), depth(c[14], f.b0, f.levels);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = p_forward(f.ctx, f.params, f.cloud, f.texture, f.cameras, f.views, f.n_views, f.dropout, f.lists, color.get<float>(),
                   weight.get<float>(), mask.get<float>(), depth.get<float>());
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

// gradients(ctx, device, n, n_tex, channels, n_img, n_cam): zeroed buffers (desc, conf, background[, points][, pose, pose_count]
// [, intrinsics, intrinsics_count]), a part left out where its count is None, or the status of the call that zeroes them.  One
// launch zeroes them all: a fill of its own each costs more than the buffers of a small scene.
PyObject* gradients(const Call& c)
{
    c.expect(7);
    vetr_ctx* ctx    = address<vetr_ctx>(c[0]);
    const auto f32   = on(c[1]);
    const auto n_tex = integer(c[3]);
    std::vector<at::Tensor> t;
    t.reserve(8);
    t.push_back(fresh({n_tex, 4}, f32)), t.push_back(fresh({n_tex}, f32)), t.push_back(fresh({integer(c[4])}, f32));
    if (c[2] != Py_None) t.push_back(fresh({integer(c[2]), 4}, f32));
    if (c[5] != Py_None) t.push_back(fresh({integer(c[5]), 6}, on(c[1], at::kDouble))), t.push_back(fresh({integer(c[5])}, f32));
    if (c[6] != Py_None) t.push_back(fresh({integer(c[6]), 13}, f32)), t.push_back(fresh({integer(c[6])}, f32));
    void* p[8];
    int64_t bytes[8];
    for (size_t k = 0; k < t.size(); ++k) p[k] = t[k].data_ptr(), bytes[k] = (int64_t)t[k].nbytes();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = p_zero_buffers(ctx, p, bytes, (int)t.size());
    Py_END_ALLOW_THREADS
    if (rc != VETR_OK) return PyLong_FromLong(rc);
    THPObjectPtr out = held(PyTuple_New((Py_ssize_t)t.size()));
    for (size_t k = 0; k < t.size(); ++k) PyTuple_SET_ITEM(out.get(), (Py_ssize_t)k, wrap(std::move(t[k])));
    return out.release();
}

// backward(<Frame>, color, grad_color, desc, conf, points, background, pose, pose_count, intrinsics, intrinsics_count, phases) ->
// status; the images are contiguous
PyObject* backward(const Call& c)
{
    c.expect(22);
    const Frame f(c);
    const Levels color(c[11], f.b0, f.levels), grad(c[12], f.b0, f.levels);
    float *desc = data<float>(c[13]), *conf = data<float>(c[14]), *points = data<float>(c[15]), *background = data<float>(c[16]);
    double* pose      = data<double>(c[17]);
    float *pose_count = data<float>(c[18]), *intr = data<float>(c[19]), *intr_count = data<float>(c[20]);
    const int phases  = (int)integer(c[21]);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = p_backward_phase(f.ctx, f.params, f.cloud, f.texture, f.cameras, f.views, f.n_views, f.dropout, f.lists, color.get<const float>(),
                          grad.get<const float>(), desc, conf, points, background, pose, pose_count, intr, intr_count, phases);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

// finalize(ctx, device, channels, desc, points, pose, pose_count, intrinsics, intrinsics_count) -> texture gradient
// [channels, n_tex], or the status of a call that failed
PyObject* finalize(const Call& c)
{
    c.expect(9);
    vetr_ctx* ctx   = address<vetr_ctx>(c[0]);
    const int C     = (int)integer(c[2]), n_tex = rows(c[3]);
    at::Tensor out  = fresh({C, n_tex}, on(c[1]));
    const int n = rows(c[4]), n_img = rows(c[5]), n_cam = rows(c[7]);
    const float* desc       = data<const float>(c[3]);
    float *texture          = static_cast<float*>(out.data_ptr()), *points = data<float>(c[4]), *intr = data<float>(c[7]);
    double* pose            = data<double>(c[5]);
    const float *pose_count = data<const float>(c[6]), *intr_count = data<const float>(c[8]);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = p_finalize_gradients(ctx, C, n_tex, desc, texture, n, points, nullptr, n_img, pose, pose_count, n_cam, intr, intr_count);
    Py_END_ALLOW_THREADS
    if (rc != VETR_OK) return PyLong_FromLong(rc);
    return wrap(std::move(out));
}

// l1_loss_grad(ctx, images, targets, grads, loss) -> status
PyObject* l1_loss_grad(const Call& c)
{
    c.expect(5);
    vetr_ctx* ctx       = address<vetr_ctx>(c[0]);
    THPObjectPtr images = sequence(c[1]);
    if (PySequence_Fast_GET_SIZE(images.get()) > VETR_MAX_LAYERS) return PyLong_FromLong(VETR_E_INVALID_ARG);
    const int n = (int)PySequence_Fast_GET_SIZE(images.get());
    const Levels image(images.get(), 0, n), target(c[2], 0, n), grad(c[3], 0, n);
    int64_t numel[VETR_MAX_LAYERS] = {};
    for (int l = 0; l < n; ++l) numel[l] = ::numel(PySequence_Fast_GET_ITEM(images.get(), l));
    float* loss = data<float>(c[4]);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = p_l1_loss_grad(ctx, n, image.get<const float>(), target.get<const float>(), grad.get<float>(), numel, loss);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

#define VETR_METHOD(name) \
    {#name, (PyCFunction)(void*)(+[](PyObject*, PyObject* const* args, Py_ssize_t n) { return guarded(name, args, n); }), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {VETR_METHOD(bind),     VETR_METHOD(current_stream), VETR_METHOD(images),    VETR_METHOD(params),
                         VETR_METHOD(views),    VETR_METHOD(forward),        VETR_METHOD(gradients), VETR_METHOD(backward),
                         VETR_METHOD(finalize), VETR_METHOD(l1_loss_grad),   VETR_METHOD(bind_sizes), VETR_METHOD(scene), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};
}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
