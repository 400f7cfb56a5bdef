// graphtok_b200._host: what stands between a Python object and libgtok's calls in steps (gtok_x_measure and
// what follows it in gtok.h).
//
// The library takes text where Python keeps it (a str's own characters, a bytes object's bytes, those of a list
// one by one) and writes ids and bytes to the object that is returned, by way of its page-locked buffers: a call
// makes no intermediate Python object and one copy each way (a bytearray or a view is copied first).  Every
// function takes the handle as an integer and answers an error of the library with its (negative) code as an int.
// The module is not linked against the library: bind() takes the calls' addresses from whoever has loaded it, so
// that there is one copy of it in the process whatever else goes by the name libgtok.so on the library path.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#define NPY_NO_DEPRECATED_API NPY_1_7_API_VERSION
#define NPY_TARGET_VERSION NPY_1_22_API_VERSION
#include <numpy/arrayobject.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "../../include/gtok.h"
#include "result_memory.h"

namespace {

// Results from this size on are copied out with the interpreter lock let go.
constexpr uint64_t kLargeBytes = 256 << 10;

// The library's calls by address.
struct Lib {
    decltype(&gtok_x_set_max_bytes) set_max_bytes;
    decltype(&gtok_x_result_stream) result_stream;
    decltype(&gtok_x_measure) measure;
    decltype(&gtok_x_encode_measured) encode_measured;
    decltype(&gtok_x_take_ids) take_ids;
    decltype(&gtok_x_decode_room) decode_room;
    decltype(&gtok_x_decode_run) decode_run;
    decltype(&gtok_x_take_bytes) take_bytes;
} lib;
bool bound = false;
struct Need { const char* name; void* at; };
#define GTOK_NEED(f) {"gtok_x_" #f, &lib.f}
const Need kNeeds[] = {GTOK_NEED(set_max_bytes), GTOK_NEED(result_stream), GTOK_NEED(measure), GTOK_NEED(encode_measured), GTOK_NEED(take_ids), GTOK_NEED(decode_room),
                       GTOK_NEED(decode_run), GTOK_NEED(take_bytes)};

// bind(address): address(name) -> where that call of gtok.h is in the loaded library.
PyObject* py_bind(PyObject*, PyObject* address) {
    for (const Need& n : kNeeds) {
        PyObject* at = PyObject_CallFunction(address, "s", n.name);
        void* p = at ? PyLong_AsVoidPtr(at) : nullptr;
        Py_XDECREF(at);
        if (!p) {
            if (!PyErr_Occurred()) PyErr_Format(PyExc_ImportError, "no %s in the library", n.name);
            bound = false;
            return nullptr;
        }
        std::memcpy(n.at, &p, sizeof p);
    }
    bound = true;
    Py_RETURN_NONE;
}

// A handle of the bound library; none before there is one.
void* handle_of(PyObject* o) { return bound && PyLong_CheckExact(o) ? PyLong_AsVoidPtr(o) : nullptr; }

// The texts of one call: where each lies, and what keeps it there until the call is over.
struct Texts {
    std::vector<gtok_x_piece> pieces;
    std::vector<PyObject*> kept;
    gtok_x_piece one;
    ~Texts() {
        for (PyObject* o : kept) Py_XDECREF(o);
    }
    // False with an exception set: neither str nor bytes-like, or no memory to note it down.
    bool place(PyObject* o, gtok_x_piece* p) noexcept {
        try { return find(o, p); } catch (const std::bad_alloc&) { PyErr_NoMemory(); return false; }
    }
    // The same for the texts of a tuple, as `pieces`.
    bool place_all(PyObject* tuple) noexcept {
        const Py_ssize_t n = PyTuple_GET_SIZE(tuple);
        try {
            pieces.resize(static_cast<size_t>(n));
        } catch (const std::exception&) { PyErr_NoMemory(); return false; }
        for (Py_ssize_t i = 0; i < n; ++i)
            if (!place(PyTuple_GET_ITEM(tuple, i), &pieces[static_cast<size_t>(i)])) return false;
        return true;
    }

private:
    bool find(PyObject* o, gtok_x_piece* p) {
        if (PyUnicode_CheckExact(o)) {
            p->data = PyUnicode_DATA(o);
            p->units = static_cast<uint64_t>(PyUnicode_GET_LENGTH(o));
            const int width = PyUnicode_KIND(o);
            p->kind = PyUnicode_IS_COMPACT_ASCII(o) ? 1u : width == 1 ? 3u : static_cast<uint32_t>(width);
            return true;
        }
        if (PyBytes_CheckExact(o)) {
            p->data = PyBytes_AS_STRING(o);
            p->units = static_cast<uint64_t>(PyBytes_GET_SIZE(o));
            p->kind = 1;
            return true;
        }
        kept.push_back(nullptr);
        PyObject* made = nullptr;
        // (a bytearray or a view is taken as it is now: while the library works the interpreter lock is let go, and other threads
        // may write to it or resize it)
        if (PyUnicode_Check(o)) made = PyObject_CallMethod(o, "encode", "s", "utf-8");
        else if (PyBytes_Check(o) || PyByteArray_Check(o) || PyMemoryView_Check(o)) made = PyObject_Bytes(o);
        else { PyErr_SetString(PyExc_TypeError, "text must be str or bytes"); return false; }
        if (!made) return false;
        kept.back() = made;
        if (!PyBytes_Check(made)) { PyErr_SetString(PyExc_TypeError, "text must be str or bytes"); return false; }
        p->data = PyBytes_AS_STRING(made);
        p->units = static_cast<uint64_t>(PyBytes_GET_SIZE(made));
        p->kind = 1;
        return true;
    }
};

// The byte cap doubled until a text of `bytes` fits even if normalisation lengthens it (at most threefold).
void grow_cap(void* h, int64_t bytes) {
    uint64_t cap = lib.set_max_bytes(h, 0);
    const uint64_t need = static_cast<uint64_t>(bytes) * 3 + 64;
    if (!cap || cap >= need) return;
    while (cap < need) cap *= 2;
    lib.set_max_bytes(h, static_cast<uint32_t>(std::min<uint64_t>(cap, 0xFFFFFFFFull)));
}

// numpy's memory functions over result_memory.h; an array keeps the handler it was made with.
void* mem_get(void*, size_t size) { return result_memory::get(size); }
void* mem_zeroed(void*, size_t n, size_t each) { return std::calloc(n, each); }
void* mem_resize(void*, void* p, size_t size) { return std::realloc(p, size); }
void mem_put(void*, void* p, size_t) { result_memory::put(p); }
PyDataMem_Handler kMemory = {"graphtok_results", 1, {nullptr, mem_get, mem_zeroed, mem_resize, mem_put}};
PyObject* memory = nullptr;      // its capsule

// An array for `n` ids that owns its memory.
PyObject* new_ids(int64_t n) {
    npy_intp dim = static_cast<npy_intp>(n);
    if (static_cast<uint64_t>(n) * 4 < result_memory::kLeast) return PyArray_SimpleNew(1, &dim, NPY_UINT32);
    PyObject* usual = PyDataMem_GetHandler();
    if (!usual) return nullptr;
    if (usual != PyDataMem_DefaultHandler) { Py_DECREF(usual); return PyArray_SimpleNew(1, &dim, NPY_UINT32); }     // the program's own choice
    Py_DECREF(usual);
    usual = PyDataMem_SetHandler(memory);
    if (!usual) return nullptr;
    PyObject* ids = PyArray_SimpleNew(1, &dim, NPY_UINT32);
    PyObject* mine = PyDataMem_SetHandler(usual);
    Py_DECREF(usual);
    if (!mine) { Py_XDECREF(ids); return nullptr; }
    Py_DECREF(mine);
    return ids;
}
uint32_t* data_of(PyObject* a) { return static_cast<uint32_t*>(PyArray_DATA(reinterpret_cast<PyArrayObject*>(a))); }

// A character without UTF-8 form is among the texts: the interpreter's own error for it.
PyObject* raise_encode_error(PyObject* const* objs, Py_ssize_t n) {
    for (Py_ssize_t i = 0; i < n; ++i) {
        if (!PyUnicode_Check(objs[i])) continue;
        PyObject* b = PyUnicode_AsUTF8String(objs[i]);
        if (!b) return nullptr;
        Py_DECREF(b);
    }
    return PyLong_FromLong(-1);
}

// Measures and encodes `n` texts; the outcome is the id count, a negative code, or kSurrogate.
constexpr int64_t kSurrogate = -1000;
struct Outcome { int64_t bytes, ids; };
Outcome encode_texts(void* h, const gtok_x_piece* p, uint32_t n, bool batch, bool grow) {
    Outcome o;
    Py_BEGIN_ALLOW_THREADS
    o.bytes = lib.measure(h, p, n, batch ? 1 : 0);
    if (o.bytes < 0) o.ids = kSurrogate;
    else {
        if (grow) grow_cap(h, o.bytes);
        o.ids = lib.encode_measured(h, o.bytes, nullptr, 0, nullptr);
    }
    Py_END_ALLOW_THREADS
    return o;
}

// encode(handle, text, grow) -> uint32 array
PyObject* py_encode(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 3) { PyErr_SetString(PyExc_TypeError, "encode(handle, text, grow)"); return nullptr; }
    Texts t;
    if (!t.place(args[1], &t.one)) return nullptr;
    void* h = handle_of(args[0]);
    if (!h) return PyLong_FromLong(-1);
    const Outcome o = encode_texts(h, &t.one, 1, false, args[2] == Py_True);
    if (o.ids == kSurrogate) return raise_encode_error(args + 1, 1);
    if (o.ids < 0) return PyLong_FromLongLong(o.ids);
    PyObject* ids = new_ids(o.ids);
    if (!ids) return nullptr;
    int r;
    if (static_cast<uint64_t>(o.ids) * 4 < kLargeBytes) {
        r = lib.take_ids(h, data_of(ids), nullptr);
    } else {
        Py_BEGIN_ALLOW_THREADS
        r = lib.take_ids(h, data_of(ids), nullptr);
        Py_END_ALLOW_THREADS
    }
    if (r < 0) { Py_DECREF(ids); return PyLong_FromLong(r); }
    return ids;
}

// encode_batch(handle, texts (a tuple, at least one), grow) -> (uint32 ids, uint32 offsets)
PyObject* py_encode_batch(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 3 || !PyTuple_CheckExact(args[1])) { PyErr_SetString(PyExc_TypeError, "encode_batch(handle, tuple of texts, grow)"); return nullptr; }
    Texts t;
    if (!t.place_all(args[1])) return nullptr;
    void* h = handle_of(args[0]);
    if (!h) return PyLong_FromLong(-1);
    const Outcome o = encode_texts(h, t.pieces.data(), static_cast<uint32_t>(t.pieces.size()), true, args[2] == Py_True);
    if (o.ids == kSurrogate) return raise_encode_error(PySequence_Fast_ITEMS(args[1]), PyTuple_GET_SIZE(args[1]));
    if (o.ids < 0) return PyLong_FromLongLong(o.ids);
    PyObject* ids = new_ids(o.ids);
    if (!ids) return nullptr;
    npy_intp dim = static_cast<npy_intp>(t.pieces.size()) + 1;
    PyObject* off = PyArray_SimpleNew(1, &dim, NPY_UINT32);
    if (!off) { Py_DECREF(ids); return nullptr; }
    int r;
    Py_BEGIN_ALLOW_THREADS
    r = lib.take_ids(h, data_of(ids), data_of(off));
    Py_END_ALLOW_THREADS
    if (r < 0) { Py_DECREF(ids); Py_DECREF(off); return PyLong_FromLong(r); }
    return Py_BuildValue("(NN)", ids, off);
}

// encode_to_device(handle, text or tuple of texts, grow, make, queue) -> (what make(words) returned for the ids, id count,
// the same for the offsets or None).  make(words) returns a tensor of that many 32-bit words on the device, queue() the
// stream whose queued work may still use their memory.
PyObject* py_encode_to_device(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 5) { PyErr_SetString(PyExc_TypeError, "encode_to_device(handle, text or tuple, grow, make, queue)"); return nullptr; }
    const bool batch = PyTuple_CheckExact(args[1]);
    Texts t;
    if (batch ? !t.place_all(args[1]) : !t.place(args[1], &t.one)) return nullptr;
    void* h = handle_of(args[0]);
    if (!h) return PyLong_FromLong(-1);
    const gtok_x_piece* p = batch ? t.pieces.data() : &t.one;
    const uint32_t n = batch ? static_cast<uint32_t>(t.pieces.size()) : 1u;
    int64_t bytes;
    Py_BEGIN_ALLOW_THREADS
    bytes = lib.measure(h, p, n, batch ? 1 : 0);
    if (bytes >= 0 && args[2] == Py_True) grow_cap(h, bytes);
    Py_END_ALLOW_THREADS
    if (bytes < 0) return batch ? raise_encode_error(PySequence_Fast_ITEMS(args[1]), PyTuple_GET_SIZE(args[1])) : raise_encode_error(args + 1, 1);
    auto make = [&](uint64_t words, void** ptr) -> PyObject* {
        PyObject* w = PyLong_FromUnsignedLongLong(words);
        PyObject* tensor = w ? PyObject_CallOneArg(args[3], w) : nullptr;
        Py_XDECREF(w);
        PyObject* at = tensor ? PyObject_CallMethod(tensor, "data_ptr", nullptr) : nullptr;
        *ptr = at ? PyLong_AsVoidPtr(at) : nullptr;
        Py_XDECREF(at);
        if (PyErr_Occurred()) { Py_XDECREF(tensor); return nullptr; }
        return tensor;
    };
    void *ids_at = nullptr, *off_at = nullptr;
    PyObject* off = batch ? make(static_cast<uint64_t>(n) + 1, &off_at) : nullptr;
    if (batch && !off) return nullptr;
    // one id a byte is the most, but for text that normalisation lengthens (at most threefold)
    for (int attempt = 0; attempt < 2; ++attempt) {
        const uint64_t room = attempt ? 3 * static_cast<uint64_t>(bytes) + 64 : static_cast<uint64_t>(bytes) + 16;
        PyObject* ids = make(room, &ids_at);
        if (!ids) { Py_XDECREF(off); return nullptr; }
        PyObject* q = PyObject_CallNoArgs(args[4]);
        void* stream = q ? PyLong_AsVoidPtr(q) : nullptr;
        Py_XDECREF(q);
        if (PyErr_Occurred()) { Py_DECREF(ids); Py_XDECREF(off); return nullptr; }
        int64_t got;
        Py_BEGIN_ALLOW_THREADS
        got = lib.result_stream(h, stream) < 0 ? -1 : lib.encode_measured(h, bytes, ids_at, room, off_at);
        Py_END_ALLOW_THREADS
        if (got == -2 && attempt == 0) { Py_DECREF(ids); continue; }
        if (got < 0) { Py_DECREF(ids); Py_XDECREF(off); return PyLong_FromLongLong(got); }
        if (!off) { off = Py_None; Py_INCREF(off); }
        return Py_BuildValue("(NLN)", ids, static_cast<long long>(got), off);
    }
    return nullptr;
}

template <class T>
bool narrow(const T* s, uint32_t n, uint32_t* d) {
    uint64_t high = 0;
    for (uint32_t i = 0; i < n; ++i) {
        const uint64_t v = static_cast<uint64_t>(static_cast<int64_t>(s[i]));
        high |= v;
        d[i] = static_cast<uint32_t>(v);
    }
    return (high >> 32) == 0;
}

// (the first decoding call of a handle, and one that is larger than those before, make its buffers)
uint32_t* decode_room(void* h, uint32_t n) {
    uint32_t* room;
    Py_BEGIN_ALLOW_THREADS
    room = lib.decode_room(h, n);
    Py_END_ALLOW_THREADS
    return room;
}

// decode(handle, ids) -> bytes; None for an `ids` that this function does not take (the caller makes a uint32 array of it)
PyObject* py_decode(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 2) { PyErr_SetString(PyExc_TypeError, "decode(handle, ids)"); return nullptr; }
    void* h = handle_of(args[0]);
    PyObject* o = args[1];
    const uint32_t* ids = nullptr;
    uint32_t n = 0;
    bool fits = true;
    if (PyList_CheckExact(o)) {
        const Py_ssize_t len = PyList_GET_SIZE(o);
        if (!h || len == 0 || len > 0x3FFFFFFF) Py_RETURN_NONE;
        n = static_cast<uint32_t>(len);
        for (Py_ssize_t i = 0; i < len; ++i)
            if (!PyLong_CheckExact(PyList_GET_ITEM(o, i))) Py_RETURN_NONE;
        uint32_t* room = decode_room(h, n);
        if (!room) return PyLong_FromLong(-1);
        if (PyList_GET_SIZE(o) != len) Py_RETURN_NONE;              // (another thread has changed it meanwhile)
        for (Py_ssize_t i = 0; i < len; ++i) {
            int over = 0;
            if (!PyLong_CheckExact(PyList_GET_ITEM(o, i))) Py_RETURN_NONE;
            const long long v = PyLong_AsLongLongAndOverflow(PyList_GET_ITEM(o, i), &over);
            if (over || v < 0 || v > 0xFFFFFFFFll) { fits = false; break; }
            room[i] = static_cast<uint32_t>(v);
        }
        ids = room;
    } else if (PyArray_CheckExact(o)) {
        PyArrayObject* a = reinterpret_cast<PyArrayObject*>(o);
        const npy_intp len = PyArray_SIZE(a);
        const PyArray_Descr* d = PyArray_DESCR(a);
        const int width = static_cast<int>(PyArray_ITEMSIZE(a));
        if (!h || len == 0 || len > 0x3FFFFFFF || !PyArray_IS_C_CONTIGUOUS(a) || !PyArray_ISALIGNED(a) || !PyArray_ISNOTSWAPPED(a) ||
            (d->kind != 'u' && d->kind != 'i') || (width != 4 && width != 8))
            Py_RETURN_NONE;
        n = static_cast<uint32_t>(len);
        if (d->kind == 'u' && width == 4) ids = static_cast<const uint32_t*>(PyArray_DATA(a));
        else {
            uint32_t* room = decode_room(h, n);
            if (!room) return PyLong_FromLong(-1);
            const void* s = PyArray_DATA(a);
            Py_BEGIN_ALLOW_THREADS
            fits = width == 4 ? narrow(static_cast<const int32_t*>(s), n, room) : narrow(static_cast<const int64_t*>(s), n, room);
            Py_END_ALLOW_THREADS
            ids = room;
        }
    } else {
        Py_RETURN_NONE;
    }
    if (!fits) { PyErr_SetString(PyExc_ValueError, "token ids must fit 32 unsigned bits"); return nullptr; }
    int64_t total;
    Py_BEGIN_ALLOW_THREADS
    total = lib.decode_run(h, ids, n);
    Py_END_ALLOW_THREADS
    if (total < 0) return PyLong_FromLongLong(total);
    PyObject* bytes = PyBytes_FromStringAndSize(nullptr, static_cast<Py_ssize_t>(total));
    if (!bytes || total == 0) return bytes;
    int r;
    Py_BEGIN_ALLOW_THREADS
    r = lib.take_bytes(h, reinterpret_cast<uint8_t*>(PyBytes_AS_STRING(bytes)));
    Py_END_ALLOW_THREADS
    if (r < 0) { Py_DECREF(bytes); return PyLong_FromLong(r); }
    return bytes;
}

// users(change): +1 for a tokenizer that is opened, -1 when it is closed
PyObject* py_users(PyObject*, PyObject* change) {
    const long v = PyLong_AsLong(change);
    if (v == -1 && PyErr_Occurred()) return nullptr;
    result_memory::users(static_cast<int>(v));
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"users", py_users, METH_O, "users(change): tokenizers opened (+1) or closed (-1); memory of dropped results is kept while one is open"},
    {"bind", py_bind, METH_O, "bind(address): address(name) -> address of that call of gtok.h in the loaded library"},
    {"encode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_encode)), METH_FASTCALL, "encode(handle, text, grow) -> uint32 array, or an error code"},
    {"encode_batch", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_encode_batch)), METH_FASTCALL,
     "encode_batch(handle, texts, grow) -> (uint32 ids, uint32 offsets), or an error code"},
    {"encode_to_device", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_encode_to_device)), METH_FASTCALL,
     "encode_to_device(handle, text or tuple, grow, make, queue) -> (tensor, id count, offsets or None), or an error code"},
    {"decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_decode)), METH_FASTCALL, "decode(handle, ids) -> bytes, None, or an error code"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", "Python objects to and from libgtok's calls in steps.", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
    import_array();
    memory = PyCapsule_New(&kMemory, "mem_handler", nullptr);
    return memory ? PyModule_Create(&kModule) : nullptr;
}
