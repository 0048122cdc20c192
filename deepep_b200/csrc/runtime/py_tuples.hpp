// Tuples of a call's arguments and results, read and made through the C API: with pybind11's casters an item costs about
// 0.15 us, and a dispatch or combine passes some forty of them.
#pragma once

#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include <limits>
#include <optional>
#include <vector>

#include "runtime.hpp"

namespace ep {

class TupleReader {
public:
    TupleReader(PyObject* tuple, Py_ssize_t items) : tuple_(tuple) {
        if (!PyTuple_Check(tuple) || PyTuple_GET_SIZE(tuple) != items) throw pybind11::type_error("a call's arguments come as one tuple of fixed length");
    }
    PyObject* item(int i) const { return PyTuple_GET_ITEM(tuple_, i); }
    bool none(int i) const { return item(i) == Py_None; }
    at::Tensor tensor(int i) const {
        if (!THPVariable_Check(item(i))) throw pybind11::type_error("argument " + std::to_string(i) + " has to be a tensor");
        return THPVariable_Unpack(item(i));
    }
    std::optional<at::Tensor> maybe_tensor(int i) const { return none(i) ? std::nullopt : std::optional<at::Tensor>(tensor(i)); }
    int integer(int i) const {
        const long v = PyLong_AsLong(item(i));
        if (v == -1 && PyErr_Occurred() != nullptr) throw pybind11::error_already_set();
        if (v < std::numeric_limits<int>::min() || v > std::numeric_limits<int>::max()) throw pybind11::value_error("argument " + std::to_string(i) + " is out of range");
        return static_cast<int>(v);
    }
    bool flag(int i) const {
        const int v = PyObject_IsTrue(item(i));
        if (v < 0) throw pybind11::error_already_set();
        return v != 0;
    }
    std::optional<EventHandle> event(int i) const {
        if (none(i)) return std::nullopt;
        return pybind11::handle(item(i)).cast<EventHandle>();
    }

private:
    PyObject* tuple_;
};

class TupleWriter {
public:
    explicit TupleWriter(Py_ssize_t items) : tuple_(pybind11::reinterpret_steal<pybind11::tuple>(PyTuple_New(items))) {
        if (!tuple_) throw pybind11::error_already_set();
    }
    TupleWriter& put(const at::Tensor& t) { return set(THPVariable_Wrap(t)); }      // (an undefined tensor becomes None)
    TupleWriter& put(const std::optional<at::Tensor>& t) { return t.has_value() ? put(*t) : set(Py_NewRef(Py_None)); }
    TupleWriter& put(int v) { return set(PyLong_FromLong(v)); }
    TupleWriter& put(bool v) { return set(PyBool_FromLong(v ? 1 : 0)); }
    TupleWriter& put(const std::optional<EventHandle>& e) {
        return set(e.has_value() ? pybind11::cast(*e).release().ptr() : Py_NewRef(Py_None));
    }
    TupleWriter& put(const std::vector<int>& v) {
        PyObject* list = PyList_New(static_cast<Py_ssize_t>(v.size()));
        if (list == nullptr) throw pybind11::error_already_set();
        for (size_t i = 0; i < v.size(); ++i) PyList_SET_ITEM(list, static_cast<Py_ssize_t>(i), PyLong_FromLong(v[i]));
        return set(list);
    }
    pybind11::tuple take() { return std::move(tuple_); }

private:
    TupleWriter& set(PyObject* o) {
        if (o == nullptr) throw pybind11::error_already_set();
        PyTuple_SET_ITEM(tuple_.ptr(), next_++, o);
        return *this;
    }
    pybind11::tuple tuple_;
    Py_ssize_t next_ = 0;
};

}  // namespace ep
