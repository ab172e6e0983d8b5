// Block tables of a decode batch from the engine's Python lists, padded into the int32 arrays that go to the GPU.
//
// The reference pads them in its model runner (additional_designs/worker/aptserve_model_runner.py:601-609).
// Eighteen thousand list elements (256 OPT-13B requests) cost numpy 30 ns each; read through the interpreter's own
// list and integer accessors they cost 3.  With one copy to the device and one allocation for the outputs a
// call of device_metadata.expand_decode_metadata went from 855 to 218 us, and with lengths, types and counts read here too and
// the tensors cut out of their buffers by one call from 222 to 160; read once and left unpadded it takes 120.  A library of its own, because this one needs
// the Python process it is loaded into; called with the interpreter lock held (ctypes.PyDLL).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <stdint.h>
#include <string.h>

namespace {

// A plain integer of 32 bits; false for anything else.
inline bool read_int(PyObject* x, int32_t* out) {
  if (!PyLong_CheckExact(x)) return false;
#if PY_VERSION_HEX >= 0x030C0000
  if (PyUnstable_Long_IsCompact((PyLongObject*)x)) {   // one digit: below 2^30, read without a call
    *out = (int32_t)PyUnstable_Long_CompactValue((PyLongObject*)x);
    return true;
  }
#endif
  int overflow = 0;
  const long v = PyLong_AsLongAndOverflow(x, &overflow);
  if (overflow != 0 || v < INT32_MIN || v > INT32_MAX) return false;
  *out = (int32_t)v;
  return true;
}

// One row; false for anything but a list or tuple of plain integers of 32 bits that fits the width.
bool pack_row(PyObject* row, int64_t width, int32_t* out) {
  const bool list = PyList_CheckExact(row);
  if (!list && !PyTuple_CheckExact(row)) return false;
  const Py_ssize_t n = list ? PyList_GET_SIZE(row) : PyTuple_GET_SIZE(row);
  if (n > width) return false;
  for (Py_ssize_t i = 0; i < n; ++i)
    if (!read_int(list ? PyList_GET_ITEM(row, i) : PyTuple_GET_ITEM(row, i), out + i)) return false;
  memset(out + n, 0, (size_t)(width - n) * sizeof(int32_t));
  return true;
}

// Entries of a list or tuple; -1 for anything else.
inline int64_t row_size(PyObject* row) {
  return PyList_CheckExact(row) || PyTuple_CheckExact(row) ? (int64_t)PySequence_Fast_GET_SIZE(row) : -1;
}

// The entries of a list or tuple.  The integers lie all over the heap: they are asked for ahead of their turn.
bool read_entries(PyObject* row, int32_t* out) {
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(row);
  PyObject** items = PySequence_Fast_ITEMS(row);
  for (Py_ssize_t i = 0; i < n; ++i) {
    if (i + 12 < n) __builtin_prefetch(items[i + 12]);
    if (!read_int(items[i], out + i)) return false;
  }
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

// What the tables' buffer is sized by, in one pass over the lists: counts = {hidden-cached requests, their tokens, the
// widest private table, the shortest and the longest length}; the lengths as they are in lens, the types (0 or 1) in types.
// Returns 0, or 1 for arguments that are not lists: lengths and tables of `batch`, plain integers and booleans.
extern "C" int aps_measure_decode_batch(PyObject* seq_lens, PyObject* use_hidden, PyObject* tables, int64_t batch,
                                        int32_t* lens, int32_t* types, int64_t* counts) {
  if (!PyList_CheckExact(seq_lens) || !PyList_CheckExact(use_hidden) || !PyList_CheckExact(tables) ||
      PyList_GET_SIZE(seq_lens) != batch || PyList_GET_SIZE(use_hidden) != batch || PyList_GET_SIZE(tables) != batch)
    return 1;
  int64_t n_hidden = 0, tokens = 0, width = 0, least = INT32_MAX, most = 0;
  for (int64_t r = 0; r < batch; ++r) {
    PyObject *h = PyList_GET_ITEM(use_hidden, r), *t = PyList_GET_ITEM(tables, r);
    if ((h != Py_True && h != Py_False) || !read_int(PyList_GET_ITEM(seq_lens, r), lens + r)) return 1;
    const bool list = PyList_CheckExact(t);
    if (!list && !PyTuple_CheckExact(t)) return 1;
    const int64_t n = list ? PyList_GET_SIZE(t) : PyTuple_GET_SIZE(t);
    types[r] = h == Py_True ? 1 : 0;
    n_hidden += types[r];
    tokens += types[r] ? lens[r] : 0;
    if (n > width) width = n;
    if (lens[r] < least) least = lens[r];
    if (lens[r] > most) most = lens[r];
  }
  counts[0] = n_hidden; counts[1] = tokens; counts[2] = width; counts[3] = least; counts[4] = most;
  return 0;
}

// The first request with more tokens than its private table, or its shared one if it is hidden-cached, has room for, -1 if
// none has, -2 if the tables are not lists of `batch` lists or tuples (shared ones of K/V-cached requests are not looked at).
// 256 requests: 4 us, one by one in Python 25.
extern "C" int64_t aps_first_too_long(PyObject* tables, PyObject* shared_tables, const int32_t* lens, const int32_t* types, int64_t batch,
                                      int64_t block_size) {
  if (!PyList_CheckExact(tables) || !PyList_CheckExact(shared_tables) || PyList_GET_SIZE(tables) != batch ||
      PyList_GET_SIZE(shared_tables) != batch)
    return -2;
  for (int64_t r = 0; r < batch; ++r) {
    const int64_t own = row_size(PyList_GET_ITEM(tables, r)), shared = types[r] != 0 ? row_size(PyList_GET_ITEM(shared_tables, r)) : own;
    if (own < 0 || shared < 0) return -2;
    if (lens[r] > (own < shared ? own : shared) * block_size) return r;
  }
  return -1;
}

// The buffer's sections, each a multiple of 32 words: the K/V-cached rows (int64), the private, shared and the reference's
// tables, lengths, types.  Returns as aps_pack_block_tables does.
extern "C" int aps_pack_decode_batch(PyObject* tables, PyObject* shared_tables, const int32_t* lens, const int32_t* types,
                                     int64_t batch, int64_t width, int64_t n_hidden, int32_t* out) {
  auto padded = [](int64_t n) { return (n + 31) / 32 * 32; };
  if (!PyList_CheckExact(tables) || !PyList_CheckExact(shared_tables) || PyList_GET_SIZE(tables) != batch ||
      PyList_GET_SIZE(shared_tables) != batch)
    return 1;
  int64_t* rows = (int64_t*)out;
  int32_t* priv = out + padded(2 * (batch - n_hidden));
  int32_t* shared = priv + padded(batch * width);
  int32_t* ref = shared + padded(batch * width);
  int32_t* d_lens = ref + padded(batch * width);
  const size_t bytes = (size_t)width * sizeof(int32_t);
  for (int64_t r = 0; r < batch; ++r) {
    int32_t *p = priv + r * width, *s = shared + r * width;
    if (!pack_row(PyList_GET_ITEM(tables, r), width, p)) return 1;
    if (types[r]) {
      if (!pack_row(PyList_GET_ITEM(shared_tables, r), width, s)) return 1;
    } else {
      *rows++ = r;
      memset(s, 0, bytes);
    }
    memcpy(ref + r * width, types[r] ? s : p, bytes);
  }
  memcpy(d_lens, lens, (size_t)batch * sizeof(int32_t));
  memcpy(d_lens + padded(batch), types, (size_t)batch * sizeof(int32_t));
  return 0;
}

// A decode batch without padding, which the GPU adds: one behind the other the K/V-cached rows (int64), lengths, types, where each
// request's table begins among the entries (batch + 1), the same of the shared tables, the entries, the hidden-cached requests'
// shared entries.  256 OPT-13B requests (18 000 entries in tables of 128): 76 KB instead of 396 KB written to the staging
// buffer and copied to the GPU.
//
// Sizes and entries are read in one call, during which the interpreter lock is not given away and no Python code runs: what comes
// back is the lists as they were at one moment, whatever other threads append to them (sized in one call and read in another, a table
// that had grown in between was written past the end of the buffer).
// counts = {hidden-cached requests, their tokens, the widest private table, the shortest and the longest length, entries,
// shared entries, the first request that has more tokens than its private table, or its shared one if it is hidden-cached, has
// room for, or -1}.  None for anything but lists of `batch` plain integers, booleans and lists or tuples of plain integers, and
// for shared tables wider than the widest private one.
extern "C" PyObject* aps_read_decode_lists(PyObject* seq_lens, PyObject* use_hidden, PyObject* tables, PyObject* shared_tables,
                                           int64_t batch, int64_t block_size, int64_t* counts) {
  PyObject* const given[4] = {seq_lens, use_hidden, tables, shared_tables};
  for (PyObject* list : given)
    if (!PyList_CheckExact(list) || PyList_GET_SIZE(list) != batch) Py_RETURN_NONE;
  int64_t n_hidden = 0, width = 0, widest_shared = 0, n_own = 0, n_shared = 0;
  for (int64_t r = 0; r < batch; ++r) {
    PyObject* h = PyList_GET_ITEM(use_hidden, r);
    const bool hidden = h == Py_True;
    if (!hidden && h != Py_False) Py_RETURN_NONE;
    const int64_t own = row_size(PyList_GET_ITEM(tables, r)), shared = hidden ? row_size(PyList_GET_ITEM(shared_tables, r)) : 0;
    if (own < 0 || shared < 0) Py_RETURN_NONE;
    n_hidden += hidden; n_own += own; n_shared += shared;
    if (own > width) width = own;
    if (shared > widest_shared) widest_shared = shared;
  }
  if (widest_shared > width || n_own > INT32_MAX || n_shared > INT32_MAX) Py_RETURN_NONE;
  const int64_t words = 2 * (batch - n_hidden) + 2 * batch + 2 * (batch + 1) + n_own + n_shared;
  PyObject* result = PyBytes_FromStringAndSize(nullptr, (Py_ssize_t)(words * sizeof(int32_t)));
  if (result == nullptr) return nullptr;
  // the bytes begin 32 behind an allocation's start: aligned for the rows
  int64_t* rows = (int64_t*)PyBytes_AS_STRING(result);
  int32_t* lens = (int32_t*)PyBytes_AS_STRING(result) + 2 * (batch - n_hidden);
  int32_t* types = lens + batch;
  int32_t* own_at = types + batch;
  int32_t* shared_at = own_at + batch + 1;
  int32_t* own = shared_at + batch + 1;
  int32_t* shared = own + n_own;
  int64_t tokens = 0, least = INT32_MAX, most = 0, o = 0, s = 0, too_long = -1;
  for (int64_t r = 0; r < batch; ++r) {
    PyObject *t = PyList_GET_ITEM(tables, r), *x = PyList_GET_ITEM(shared_tables, r);
    types[r] = PyList_GET_ITEM(use_hidden, r) == Py_True ? 1 : 0;
    own_at[r] = (int32_t)o; shared_at[r] = (int32_t)s;
    if (!read_int(PyList_GET_ITEM(seq_lens, r), lens + r) || !read_entries(t, own + o) || (types[r] != 0 && !read_entries(x, shared + s))) {
      Py_DECREF(result);
      Py_RETURN_NONE;
    }
    int64_t blocks = PySequence_Fast_GET_SIZE(t);
    o += blocks;
    if (types[r] != 0) {
      const int64_t n = PySequence_Fast_GET_SIZE(x);
      s += n;
      if (n < blocks) blocks = n;
      tokens += lens[r];
    } else {
      *rows++ = r;
    }
    if (too_long < 0 && lens[r] > blocks * block_size) too_long = r;
    if (lens[r] < least) least = lens[r];
    if (lens[r] > most) most = lens[r];
  }
  own_at[batch] = (int32_t)o; shared_at[batch] = (int32_t)s;
  const int64_t all[8] = {n_hidden, tokens, width, least, most, n_own, n_shared, too_long};
  memcpy(counts, all, sizeof(all));
  return result;
}
