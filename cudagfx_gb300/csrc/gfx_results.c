/* gfx_results.c -- memory of large numpy results, kept for the next result of its size.
 *
 * A pool is a numpy data-memory handler (NEP 49).  Arrays made by empty() are ordinary arrays that
 * own their data; when the last reference to one goes, numpy hands its memory to the pool's free,
 * which keeps one block a size.  An array keeps its handler alive, so a pool outlives its owner
 * until the last of its arrays is gone.  All memory comes from and goes back to numpy's own
 * handler. */
#define PY_SSIZE_T_CLEAN
#define NPY_NO_DEPRECATED_API NPY_1_22_API_VERSION
#define NPY_TARGET_VERSION NPY_1_22_API_VERSION
#include <Python.h>
#include <numpy/arrayobject.h>
#include <pthread.h>
#include <stdlib.h>
#include <string.h>

#define KEPT_MOST 8 /* sizes */

typedef struct {
  PyDataMem_Handler handler;
  PyDataMemAllocator numpy;
  pthread_mutex_t mu;
  int open, n;
  size_t least, most;
  struct {
    size_t size;
    void* p;
  } kept[KEPT_MOST];
} Pool;

static void* pool_malloc(void* ctx, size_t size) {
  Pool* pool = (Pool*)ctx;
  void* p = NULL;
  pthread_mutex_lock(&pool->mu);
  for (int k = 0; k < pool->n; k++)
    if (pool->kept[k].size == size) {
      p = pool->kept[k].p;
      pool->kept[k] = pool->kept[--pool->n];
      break;
    }
  pthread_mutex_unlock(&pool->mu);
  return p ? p : pool->numpy.malloc(pool->numpy.ctx, size);
}
static void* pool_calloc(void* ctx, size_t n, size_t size) {
  Pool* pool = (Pool*)ctx;
  return pool->numpy.calloc(pool->numpy.ctx, n, size);
}
static void* pool_realloc(void* ctx, void* p, size_t size) {
  Pool* pool = (Pool*)ctx;
  return pool->numpy.realloc(pool->numpy.ctx, p, size);
}
static void pool_free(void* ctx, void* p, size_t size) {
  Pool* pool = (Pool*)ctx;
  if (p && size >= pool->least && size <= pool->most) {
    pthread_mutex_lock(&pool->mu);
    int keep = pool->open && pool->n < KEPT_MOST;
    for (int k = 0; k < pool->n; k++) keep = keep && pool->kept[k].size != size;
    if (keep) {
      pool->kept[pool->n].size = size;
      pool->kept[pool->n++].p = p;
    }
    pthread_mutex_unlock(&pool->mu);
    if (keep) return;
  }
  pool->numpy.free(pool->numpy.ctx, p, size);
}

static void pool_drop(Pool* pool) {
  pthread_mutex_lock(&pool->mu);
  pool->open = 0;
  for (int k = 0; k < pool->n; k++)
    pool->numpy.free(pool->numpy.ctx, pool->kept[k].p, pool->kept[k].size);
  pool->n = 0;
  pthread_mutex_unlock(&pool->mu);
}
static void pool_gone(PyObject* capsule) {
  Pool* pool = (Pool*)PyCapsule_GetPointer(capsule, "mem_handler");
  if (!pool) return;
  pool_drop(pool);
  pthread_mutex_destroy(&pool->mu);
  free(pool);
}

/* pool(least, most): blocks of least to most bytes are kept */
static PyObject* make_pool(PyObject* self, PyObject* args) {
  Py_ssize_t least, most;
  if (!PyArg_ParseTuple(args, "nn", &least, &most)) return NULL;
  const PyDataMem_Handler* def =
      (const PyDataMem_Handler*)PyCapsule_GetPointer(PyDataMem_DefaultHandler, "mem_handler");
  if (!def) return NULL;
  Pool* pool = (Pool*)calloc(1, sizeof(Pool));
  if (!pool) return PyErr_NoMemory();
  strcpy(pool->handler.name, "gfx_results");
  pool->handler.version = 1;
  pool->handler.allocator.ctx = pool;
  pool->handler.allocator.malloc = pool_malloc;
  pool->handler.allocator.calloc = pool_calloc;
  pool->handler.allocator.realloc = pool_realloc;
  pool->handler.allocator.free = pool_free;
  pool->numpy = def->allocator;
  pool->open = 1;
  pool->least = (size_t)least;
  pool->most = (size_t)most;
  pthread_mutex_init(&pool->mu, NULL);
  PyObject* capsule = PyCapsule_New(&pool->handler, "mem_handler", pool_gone);
  if (!capsule) {
    pthread_mutex_destroy(&pool->mu);
    free(pool);
  }
  return capsule;
}

/* empty(pool, shape): an array of doubles; only its data comes from the pool, the thread's numpy
 * handler is as before afterwards */
static PyObject* make_empty(PyObject* self, PyObject* args) {
  PyObject* capsule;
  PyArray_Dims shape = {NULL, 0};
  if (!PyArg_ParseTuple(args, "OO&", &capsule, PyArray_IntpConverter, &shape)) return NULL;
  PyObject* before = PyDataMem_SetHandler(capsule);
  PyObject* array = before ? PyArray_SimpleNew(shape.len, shape.ptr, NPY_DOUBLE) : NULL;
  PyDimMem_FREE(shape.ptr);
  if (!before) return NULL;
  PyObject* ours = PyDataMem_SetHandler(before);
  Py_DECREF(before);
  if (!ours) {
    Py_XDECREF(array);
    return NULL;
  }
  Py_DECREF(ours);
  return array;
}

static PyObject* close_pool(PyObject* self, PyObject* capsule) {
  Pool* pool = (Pool*)PyCapsule_GetPointer(capsule, "mem_handler");
  if (!pool) return NULL;
  pool_drop(pool);
  Py_RETURN_NONE;
}

/* kept(pool): [(address, bytes), ..] */
static PyObject* kept_blocks(PyObject* self, PyObject* capsule) {
  Pool* pool = (Pool*)PyCapsule_GetPointer(capsule, "mem_handler");
  if (!pool) return NULL;
  size_t at[KEPT_MOST], size[KEPT_MOST];
  pthread_mutex_lock(&pool->mu);
  const int n = pool->n;
  for (int k = 0; k < n; k++) {
    at[k] = (size_t)pool->kept[k].p;
    size[k] = pool->kept[k].size;
  }
  pthread_mutex_unlock(&pool->mu);
  PyObject* list = PyList_New(n);
  for (int k = 0; list && k < n; k++) {
    PyObject* x = Py_BuildValue("(Kn)", (unsigned long long)at[k], (Py_ssize_t)size[k]);
    if (x) PyList_SET_ITEM(list, k, x);
    else Py_CLEAR(list);
  }
  return list;
}

static PyMethodDef methods[] = {{"pool", make_pool, METH_VARARGS, NULL},
                                {"empty", make_empty, METH_VARARGS, NULL},
                                {"close", close_pool, METH_O, NULL},
                                {"kept", kept_blocks, METH_O, NULL},
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_results", NULL, -1, methods};

PyMODINIT_FUNC PyInit__results(void) {
  import_array();
  return PyModule_Create(&module);
}
