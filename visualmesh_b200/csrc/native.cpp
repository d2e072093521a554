// Python's side of the engine's calls: marshalling of frames and results without an interpreter loop.
//
// visualmesh_b200/engine.py keeps the interface and the errors; this module does what it did per frame and per array through
// ctypes and numpy (5.4 us a frame to marshal, now 0.4; 6.3 ms to copy the results of the densest mesh into fresh pages, now none).
#define PY_SSIZE_T_CLEAN
#define NPY_NO_DEPRECATED_API NPY_2_0_API_VERSION
#include <Python.h>
#include <numpy/arrayobject.h>

#include <cstring>
#include <utility>

#include "../../include/vmcuda.h"

namespace {

PyObject *s_mesh, *s_Hoc, *s_lens, *s_image, *s_format, *s_ranges, *s_image_on_device, *s_value;
PyObject *s_dimensions, *s_projection, *s_focal_length, *s_centre, *s_k, *s_fov;

struct Ref {  // an owned reference
    PyObject* p;
    explicit Ref(PyObject* o = nullptr) : p(o) {}
    ~Ref() {
        Py_XDECREF(p);
    }
    Ref(const Ref&) = delete;
    Ref& operator=(const Ref&) = delete;
    explicit operator bool() const {
        return p != nullptr;
    }
};

PyArrayObject* array(const Ref& r) {
    return reinterpret_cast<PyArrayObject*>(r.p);
}
// o as a C-contiguous array of `kind` (the object itself when it is one already)
PyObject* to_array(PyObject* o, int kind) {
    return PyArray_FROM_OTF(o, kind, NPY_ARRAY_C_CONTIGUOUS | NPY_ARRAY_FORCECAST);
}

bool to_float(PyObject* o, float& out) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) return false;
    out = static_cast<float>(v);
    return true;
}
// int(o) for anything that has one (numpy integers included)
bool to_int(PyObject* o, long long& out) {
    Ref i(PyNumber_Long(o));
    if (!i) return false;
    out = PyLong_AsLongLong(i.p);
    if (out == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        const unsigned long long u = PyLong_AsUnsignedLongLong(i.p);
        if (u == static_cast<unsigned long long>(-1) && PyErr_Occurred()) return false;
        out = static_cast<long long>(u);
    }
    return true;
}
bool pair_of(PyObject* owner, PyObject* name, PyObject* (&out)[2]) {
    Ref seq(PyObject_GetAttr(owner, name));
    if (!seq) return false;
    out[0] = PySequence_GetItem(seq.p, 0);
    out[1] = out[0] != nullptr ? PySequence_GetItem(seq.p, 1) : nullptr;
    if (out[1] == nullptr) Py_CLEAR(out[0]);
    return out[1] != nullptr;
}
bool float_pair(PyObject* owner, PyObject* name, float* out) {
    PyObject* v[2] = {nullptr, nullptr};
    if (!pair_of(owner, name, v)) return false;
    const bool ok = to_float(v[0], out[0]) && to_float(v[1], out[1]);
    Py_DECREF(v[0]);
    Py_DECREF(v[1]);
    return ok;
}
bool float_attr(PyObject* owner, PyObject* name, float& out) {
    Ref v(PyObject_GetAttr(owner, name));
    return v && to_float(v.p, out);
}

bool to_lens(PyObject* lens, vm_lens& out) {
    PyObject* d[2] = {nullptr, nullptr};
    if (!pair_of(lens, s_dimensions, d)) return false;
    long long w = 0, h = 0, projection = 0;
    const bool ok = to_int(d[0], w) && to_int(d[1], h);
    Py_DECREF(d[0]);
    Py_DECREF(d[1]);
    Ref proj(ok ? PyObject_GetAttr(lens, s_projection) : nullptr);
    if (!proj || !to_int(proj.p, projection)) return false;
    std::memset(&out, 0, sizeof(out));
    out.dimensions[0] = static_cast<int32_t>(w);
    out.dimensions[1] = static_cast<int32_t>(h);
    out.projection    = static_cast<int32_t>(projection);
    return float_attr(lens, s_focal_length, out.focal_length) && float_pair(lens, s_centre, out.centre) && float_pair(lens, s_k, out.k)
           && float_attr(lens, s_fov, out.fov);
}

bool to_Hoc(PyObject* o, float* out) {
    Ref a(to_array(o, NPY_FLOAT32));
    if (!a) return false;
    if (PyArray_SIZE(array(a)) != 16) {
        PyErr_SetString(PyExc_ValueError, "Hoc must have 4 x 4 values");
        return false;
    }
    std::memcpy(out, PyArray_DATA(array(a)), 16 * sizeof(float));
    return true;
}

// the pairs of an array of ranges; a non-null pointer even for none of them: NULL means "look up on the device"
bool to_ranges(const Ref& a, const int32_t*& pairs, int32_t& n) {
    static const int32_t none[2] = {0, 0};
    const npy_intp size          = PyArray_SIZE(array(a));
    if (size % 2 != 0) {
        PyErr_SetString(PyExc_ValueError, "ranges must be pairs");
        return false;
    }
    pairs = size > 0 ? static_cast<const int32_t*>(PyArray_DATA(array(a))) : none;
    n     = static_cast<int32_t>(size / 2);
    return true;
}

// marshal(frames, out, device_mesh, plain_mesh, keep): fills the vm_frame array `out` (a writable buffer) from FrameInput objects.
// plain_mesh(mesh, Hoc), unless None, is asked for the Mesh of a frame, device_mesh(mesh) for its handle; arrays that have to stay
// alive are appended to keep.
PyObject* marshal(PyObject*, PyObject* args) {
    PyObject *frames, *out, *device_mesh, *plain_mesh, *keep;
    if (!PyArg_ParseTuple(args, "OOOOO!", &frames, &out, &device_mesh, &plain_mesh, &PyList_Type, &keep)) return nullptr;
    Py_buffer view;
    if (PyObject_GetBuffer(out, &view, PyBUF_WRITABLE | PyBUF_C_CONTIGUOUS) != 0) return nullptr;
    struct Release {
        Py_buffer* v;
        ~Release() {
            PyBuffer_Release(v);
        }
    } release{&view};
    Ref seq(PySequence_Fast(frames, "frames must be a sequence"));
    if (!seq) return nullptr;
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq.p);
    if (view.len < static_cast<Py_ssize_t>(sizeof(vm_frame)) * n) return PyErr_Format(PyExc_ValueError, "frame array too small");
    vm_frame* arr = static_cast<vm_frame*>(view.buf);
    Ref last_lens;  // frames of one camera share their lens object
    vm_lens lens;
    for (Py_ssize_t i = 0; i < n; ++i) {
        PyObject* fr = PySequence_Fast_GET_ITEM(seq.p, i);
        vm_frame& f  = arr[i];
        std::memset(&f, 0, sizeof(f));
        Ref H(PyObject_GetAttr(fr, s_Hoc));
        Ref mesh(H ? PyObject_GetAttr(fr, s_mesh) : nullptr);
        if (!mesh) return nullptr;
        if (plain_mesh != Py_None) {
            Ref plain(PyObject_CallFunctionObjArgs(plain_mesh, mesh.p, H.p, nullptr));
            if (!plain) return nullptr;
            std::swap(plain.p, mesh.p);
        }
        Ref handle(PyObject_CallOneArg(device_mesh, mesh.p));
        Ref value(handle ? PyObject_GetAttr(handle.p, s_value) : nullptr);
        if (!value) return nullptr;
        f.mesh = static_cast<const vm_mesh*>(PyLong_AsVoidPtr(value.p));
        if (PyErr_Occurred() || !to_Hoc(H.p, f.Hoc)) return nullptr;
        Ref ranges(PyObject_GetAttr(fr, s_ranges));
        if (!ranges) return nullptr;
        if (ranges.p != Py_None) {
            Ref r(to_array(ranges.p, NPY_INT32));
            if (!r || PyList_Append(keep, r.p) != 0 || !to_ranges(r, f.ranges, f.n_ranges)) return nullptr;
        }
        Ref l(PyObject_GetAttr(fr, s_lens));
        if (!l) return nullptr;
        if (l.p != last_lens.p) {
            if (!to_lens(l.p, lens)) return nullptr;
            std::swap(last_lens.p, l.p);
        }
        f.lens = lens;
        Ref image(PyObject_GetAttr(fr, s_image));
        if (!image) return nullptr;
        if (image.p == Py_None) continue;
        Ref on_device(PyObject_GetAttr(fr, s_image_on_device));
        Ref format(on_device ? PyObject_GetAttr(fr, s_format) : nullptr);
        long long code = 0;
        if (!format || !to_int(format.p, code)) return nullptr;
        f.format        = static_cast<uint32_t>(code);
        const int there = PyObject_IsTrue(on_device.p);
        if (there < 0) return nullptr;
        if (there) {
            long long at = 0;
            if (!to_int(image.p, at)) return nullptr;
            f.image           = reinterpret_cast<const void*>(at);
            f.image_on_device = 1;
        }
        else {
            Ref bytes(to_array(image.p, NPY_UINT8));
            if (!bytes || PyList_Append(keep, bytes.p) != 0) return nullptr;
            f.image = PyArray_DATA(array(bytes));
        }
    }
    Py_RETURN_NONE;
}

PyObject* view_of(const void* data, int kind, npy_intp rows, npy_intp columns) {
    npy_intp dims[2] = {rows, columns};
    return PyArray_SimpleNewFromData(columns > 0 ? 2 : 1, dims, kind, const_cast<void*>(data));
}

// views(address of a vm_batch_result): its offsets (a copy), then the four arrays as views of the engine's memory (None when the
// results were left on the device, and for missing classifications)
PyObject* views(PyObject*, PyObject* arg) {
    const auto* r = static_cast<const vm_batch_result*>(PyLong_AsVoidPtr(arg));
    if (r == nullptr) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_ValueError, "null result");
    npy_intp n = r->n_frames + 1;
    Ref offsets(PyArray_SimpleNew(1, &n, NPY_INT32));
    if (!offsets) return nullptr;
    void* to = PyArray_DATA(array(offsets));
    if (r->offsets != nullptr) { std::memcpy(to, r->offsets, sizeof(int32_t) * n); }
    else {
        std::memset(to, 0, sizeof(int32_t) * n);
    }
    if (r->on_device || r->offsets == nullptr) return PyTuple_Pack(5, offsets.p, Py_None, Py_None, Py_None, Py_None);
    const npy_intp points = r->offsets[r->n_frames], rows = points + r->n_frames;
    Ref px(view_of(r->pixel_coordinates, NPY_FLOAT32, points, 2));
    Ref gi(view_of(r->global_indices, NPY_INT32, points, 0));
    Ref nb(view_of(r->neighbourhood, NPY_INT32, rows, r->n_neighbours));
    Ref cls(r->n_classes > 0 ? view_of(r->classifications, NPY_FLOAT32, rows, r->n_classes) : Py_NewRef(Py_None));
    if (!px || !gi || !nb || !cls) return nullptr;
    return PyTuple_Pack(5, offsets.p, px.p, gi.p, nb.p, cls.p);
}

void give_back(PyObject* capsule) {
    vm_results_release(static_cast<vm_results*>(PyCapsule_GetPointer(capsule, "vm_results")));
}

// One array of a single frame's results: a view that keeps the results alive, or a copy when they could not be kept.
PyObject* own_array(const void* data, int kind, npy_intp rows, npy_intp columns, PyObject* keeper) {
    if (keeper != nullptr) {
        PyObject* a = view_of(data, kind, rows, columns);
        if (a == nullptr) return nullptr;
        if (PyArray_SetBaseObject(reinterpret_cast<PyArrayObject*>(a), Py_NewRef(keeper)) != 0) Py_CLEAR(a);
        return a;
    }
    npy_intp dims[2] = {rows, columns};
    PyObject* a      = PyArray_SimpleNew(columns > 0 ? 2 : 1, dims, kind);
    if (a != nullptr && rows > 0) std::memcpy(PyArray_DATA(reinterpret_cast<PyArrayObject*>(a)), data, PyArray_NBYTES(reinterpret_cast<PyArrayObject*>(a)));
    return a;
}

// call(engine, device mesh, host mesh or 0, ranges or None, Hoc, lens, image or None, format): one frame through vm_call (the lookup
// inside the call) or, without a host mesh, with the ranges given or looked up on the device. Returns the vm_status of a failed call, or
// (pixel coordinates, neighbourhood, global indices, classifications or None): the caller's own arrays, whose memory goes back to the
// engine when the last of them is gone.
PyObject* call(PyObject*, PyObject* args) {
    PyObject *engine_o, *mesh_o, *host_o, *ranges_o, *H_o, *lens_o, *image_o, *format_o;
    if (!PyArg_ParseTuple(args, "OOOOOOOO", &engine_o, &mesh_o, &host_o, &ranges_o, &H_o, &lens_o, &image_o, &format_o)) return nullptr;
    auto* engine     = static_cast<vm_engine*>(PyLong_AsVoidPtr(engine_o));
    const auto* mesh = static_cast<const vm_mesh*>(PyLong_AsVoidPtr(mesh_o));
    const auto* host = static_cast<const vm_hostmesh*>(PyLong_AsVoidPtr(host_o));
    float H[16];
    vm_lens lens;
    long long code = 0;
    if (PyErr_Occurred() || !to_Hoc(H_o, H) || !to_lens(lens_o, lens) || !to_int(format_o, code)) return nullptr;
    Ref image(image_o == Py_None ? nullptr : to_array(image_o, NPY_UINT8));
    if (image_o != Py_None && !image) return nullptr;
    const void* pixels = image ? PyArray_DATA(array(image)) : nullptr;
    Ref ranges(ranges_o == Py_None ? nullptr : to_array(ranges_o, NPY_INT32));
    if (ranges_o != Py_None && !ranges) return nullptr;
    const int32_t* pairs = nullptr;
    int32_t n_pairs      = 0;
    if (ranges && !to_ranges(ranges, pairs, n_pairs)) return nullptr;
    vm_batch_result r;
    vm_status status;
    Py_BEGIN_ALLOW_THREADS
    if (host != nullptr) { status = vm_call(engine, mesh, host, H, &lens, pixels, static_cast<uint32_t>(code), &r); }
    else if (pixels != nullptr) { status = vm_classify(engine, mesh, pairs, n_pairs, H, &lens, pixels, static_cast<uint32_t>(code), &r); }
    else {
        status = vm_project(engine, mesh, pairs, n_pairs, H, &lens, &r);
    }
    Py_END_ALLOW_THREADS
    if (status != VM_OK) return PyLong_FromLong(status);
    // an empty on-screen set gives a default-constructed result (cpp/visualmesh/engine/cpu/engine.hpp:193)
    const npy_intp points = r.offsets[1], rows = points > 0 ? points + 1 : 0;
    vm_results* kept = nullptr;
    if (points > 0) vm_results_keep(engine, &kept);
    Ref keeper(kept != nullptr ? PyCapsule_New(kept, "vm_results", give_back) : nullptr);
    if (kept != nullptr && !keeper) {
        vm_results_release(kept);
        return nullptr;
    }
    Ref px(own_array(r.pixel_coordinates, NPY_FLOAT32, points, 2, keeper.p));
    Ref gi(own_array(r.global_indices, NPY_INT32, points, 0, keeper.p));
    Ref nb(own_array(r.neighbourhood, NPY_INT32, rows, r.n_neighbours, keeper.p));
    Ref cls(r.n_classes > 0 ? own_array(r.classifications, NPY_FLOAT32, rows, r.n_classes, keeper.p) : Py_NewRef(Py_None));
    if (!px || !gi || !nb || !cls) return nullptr;
    return PyTuple_Pack(4, px.p, nb.p, gi.p, cls.p);
}

PyMethodDef methods[] = {
  {"marshal", marshal, METH_VARARGS, nullptr},
  {"views", views, METH_O, nullptr},
  {"call", call, METH_VARARGS, nullptr},
  {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Marshalling of frames and results for visualmesh_b200.engine.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
    import_array();
    struct {
        PyObject** to;
        const char* name;
    } names[] = {{&s_mesh, "mesh"}, {&s_Hoc, "Hoc"}, {&s_lens, "lens"}, {&s_image, "image"}, {&s_format, "format"}, {&s_ranges, "ranges"},
                 {&s_image_on_device, "image_on_device"}, {&s_value, "value"}, {&s_dimensions, "dimensions"}, {&s_projection, "projection"},
                 {&s_focal_length, "focal_length"}, {&s_centre, "centre"}, {&s_k, "k"}, {&s_fov, "fov"}};
    for (auto& n : names) {
        *n.to = PyUnicode_InternFromString(n.name);
        if (*n.to == nullptr) return nullptr;
    }
    return PyModule_Create(&module);
}
