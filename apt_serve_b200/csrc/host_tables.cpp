// Block tables of a decode batch from the engine's Python lists, padded into the int32 arrays that go to the GPU.
//
// The reference pads them in its model runner (additional_designs/worker/aptserve_model_runner.py:601-609).
// Nineteen thousand list elements (256 OPT-13B requests) cost numpy 30 ns each; read through the interpreter's own
// list and integer accessors they cost 3.  With one copy to the device and one allocation for the outputs a
// call of device_metadata.expand_decode_metadata went from 855 to 218 us.  A library of its own, because this one needs
// the Python process it is loaded into; called with the interpreter lock held (ctypes.PyDLL).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <stdint.h>
#include <string.h>

namespace {

// One row; false for anything but a list or tuple of plain integers of 32 bits that fits the width.
bool pack_row(PyObject* row, int64_t width, int32_t* out) {
  const bool list = PyList_CheckExact(row);
  if (!list && !PyTuple_CheckExact(row)) return false;
  const Py_ssize_t n = list ? PyList_GET_SIZE(row) : PyTuple_GET_SIZE(row);
  if (n > width) return false;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* x = list ? PyList_GET_ITEM(row, i) : PyTuple_GET_ITEM(row, i);
    if (!PyLong_CheckExact(x)) return false;
#if PY_VERSION_HEX >= 0x030C0000
    if (PyUnstable_Long_IsCompact((PyLongObject*)x)) {   // one digit: below 2^30, read without a call
      out[i] = (int32_t)PyUnstable_Long_CompactValue((PyLongObject*)x);
      continue;
    }
#endif
    int overflow = 0;
    const long v = PyLong_AsLongAndOverflow(x, &overflow);
    if (overflow != 0 || v < INT32_MIN || v > INT32_MAX) return false;
    out[i] = (int32_t)v;
  }
  memset(out + n, 0, (size_t)(width - n) * sizeof(int32_t));
  return true;
}

}  // namespace

// priv, shared, ref: [batch][width].  Row r of priv is tables[r], of shared shared_tables[r] for a hidden-cached request and
// zero otherwise, of ref (the reference's block_tables) the one of the two that the request's type selects.
// Returns 0, or 1 for arguments that are not lists of lists of plain integers (the arrays are then partly
// written and the caller takes its general path).
extern "C" int aps_pack_block_tables(PyObject* tables, PyObject* shared_tables, const uint8_t* use_hidden, int64_t batch,
                                     int64_t width, int32_t* priv, int32_t* shared, int32_t* ref) {
  if (!PyList_CheckExact(tables) || !PyList_CheckExact(shared_tables) || PyList_GET_SIZE(tables) != batch ||
      PyList_GET_SIZE(shared_tables) != batch)
    return 1;
  const size_t bytes = (size_t)width * sizeof(int32_t);
  for (int64_t r = 0; r < batch; ++r) {
    int32_t *p = priv + r * width, *s = shared + r * width;
    if (!pack_row(PyList_GET_ITEM(tables, r), width, p)) return 1;
    if (use_hidden[r]) {
      if (!pack_row(PyList_GET_ITEM(shared_tables, r), width, s)) return 1;
    } else {
      memset(s, 0, bytes);
    }
    memcpy(ref + r * width, use_hidden[r] ? s : p, bytes);
  }
  return 0;
}
