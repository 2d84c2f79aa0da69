/* Adjacency masks from Python edge lists, for batches of graphs: the one part
 * of packing that touches every edge as a Python object (called through
 * ctypes.PyDLL, with the interpreter lock held). */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <stdint.h>

/* edges: list of count lists of (u, v) tuples; graph i has ns[i] <= 64 * words
 * vertices whose masks, `words` 64-bit words each, start at
 * out[words * offs[i]] (zeroed by the caller). Returns 0, or 1 for anything
 * but lists of pairs of integers in [0, ns[i]): the caller then takes its own
 * path, errors included. */
int gtd_pack_edges(PyObject* edges, const int64_t* ns, const int64_t* offs, int words, uint64_t* out) {
  if (!PyList_Check(edges))
    return 1;
  const Py_ssize_t count = PyList_GET_SIZE(edges);
  for (Py_ssize_t i = 0; i < count; ++i) {
    PyObject* list = PyList_GET_ITEM(edges, i);
    if (!PyList_Check(list))
      return 1;
    uint64_t* const adj = out + (int64_t)words * offs[i];
    const Py_ssize_t m = PyList_GET_SIZE(list);
    for (Py_ssize_t k = 0; k < m; ++k) {
      PyObject* e = PyList_GET_ITEM(list, k);
      if (!PyTuple_Check(e) || PyTuple_GET_SIZE(e) != 2)
        return 1;
      PyObject *pu = PyTuple_GET_ITEM(e, 0), *pv = PyTuple_GET_ITEM(e, 1);
      if (!PyLong_CheckExact(pu) || !PyLong_CheckExact(pv))
        return 1;
      int overflow = 0;
      const long u = PyLong_AsLongAndOverflow(pu, &overflow);
      if (overflow)
        return 1;
      const long v = PyLong_AsLongAndOverflow(pv, &overflow);
      if (overflow || u < 0 || v < 0 || u >= ns[i] || v >= ns[i])
        return 1;
      adj[words * u + (v >> 6)] |= (uint64_t)1 << (v & 63);
      adj[words * v + (u >> 6)] |= (uint64_t)1 << (u & 63);
    }
  }
  return 0;
}
