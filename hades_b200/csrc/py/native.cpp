// The host half of the calls that a training or serving loop makes per batch: argument checks, the
// tensors they return, the launches of libhades_b200, in one native call instead of some thirty
// Python and ctypes operations.  A small batch is bound by exactly that: 1,000 looked-up rows cost
// 6 us on the GPU and 19 us in Python.
//
// Nothing is kept between calls except, per thread, one pinned word through which a kernel hands the
// host a number (how many ids are distinct) while later kernels of the call still run.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>
#include <torch/csrc/autograd/python_variable.h>

#include <atomic>
#include <cstring>
#include <stdexcept>
#include <string>

#include "hades_b200.h"

namespace {

PyObject* g_error = nullptr;  // hades_b200._lib.HadesError

struct Status {};  // a library call failed; the Python error is set

void check(int rc) {
  if (rc == HB_OK) return;
  PyErr_Format(g_error ? g_error : PyExc_RuntimeError, "libhades_b200 status %d: %s", rc, hb_last_error());
  throw Status();
}

void require(bool ok, const char* what) {
  if (ok) return;
  PyErr_Format(PyExc_RuntimeError, "Check failed: %s", what);
  throw Status();
}

const at::Tensor& tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s: a tensor is expected", what);
    throw Status();
  }
  return THPVariable_Unpack(o);
}

bool none(PyObject* o) { return o == Py_None; }

long long integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw Status();
  return v;
}
void* pointer(PyObject* o) { return reinterpret_cast<void*>(static_cast<uintptr_t>(integer(o))); }

at::Tensor cuda_empty(at::IntArrayRef size, at::ScalarType type, const at::Device& dev) {
  return at::detail::empty_cuda(size, type, dev, std::nullopt);
}

void* stream_of(const at::Device& dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }

int64_t row_bytes(const at::Tensor& t) { return (t.dim() == 1 ? 1 : t.size(1)) * (int64_t)t.element_size(); }

void ids_ok(const at::Tensor& ids) {
  require(ids.is_cuda() && ids.scalar_type() == at::kLong, "ids is a CUDA int64 tensor");
}

template <typename F>
PyObject* guarded(F f) {
  try {
    return f();
  } catch (const Status&) {
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

void arity(Py_ssize_t n, Py_ssize_t want, const char* name) {
  if (n == want) return;
  PyErr_Format(PyExc_TypeError, "%s takes %zd arguments", name, want);
  throw Status();
}

PyObject* pack(std::initializer_list<PyObject*> items) {
  PyObject* t = PyTuple_New((Py_ssize_t)items.size());
  Py_ssize_t k = 0;
  for (PyObject* o : items) PyTuple_SET_ITEM(t, k++, o);
  return t;
}
PyObject* wrap_or_none(const at::Tensor& t) {
  if (t.defined()) return THPVariable_Wrap(t);
  Py_RETURN_NONE;
}

// A few words of pinned memory per thread that kernels of any device can write.
struct HostWord {
  volatile int64_t* word = nullptr;  // 8 of them
  ~HostWord() {
    if (word) cudaFreeHost(const_cast<int64_t*>(word));  // fails harmlessly when the runtime is gone
  }
  int64_t* arm() {
    if (!word) {
      void* p = nullptr;
      if (cudaHostAlloc(&p, 64, cudaHostAllocPortable) != cudaSuccess) {
        PyErr_SetString(PyExc_RuntimeError, "cudaHostAlloc of 64 bytes failed");
        throw Status();
      }
      word = static_cast<int64_t*>(p);
    }
    for (int k = 0; k < 8; ++k) word[k] = -1;
    return const_cast<int64_t*>(word);
  }
  // Waits until a kernel on `stream` has written the word.  The stream is asked now and then whether
  // it still runs, so that a launch that failed ends the wait with its error.
  int64_t wait(cudaStream_t stream, int which = 0) {
    volatile int64_t* word = this->word + which;
    int64_t v = -1;
    cudaError_t e = cudaSuccess;
    Py_BEGIN_ALLOW_THREADS;
    for (unsigned spins = 1; (v = *word) < 0; ++spins) {
      if ((spins & 0x3fff) == 0) {
        e = cudaStreamQuery(stream);
        if (e != cudaErrorNotReady) {
          v = *word;
          break;
        }
      }
#if defined(__x86_64__)
      __builtin_ia32_pause();
#endif
    }
    Py_END_ALLOW_THREADS;
    if (v < 0) {
      PyErr_Format(PyExc_RuntimeError, "no count arrived from the device: %s", cudaGetErrorString(e));
      throw Status();
    }
    return v;
  }
};
thread_local HostWord t_word;

// lookup_fetch(index, ids, cache_rows, cache_ptr, backing_ptr, out_rows | None, mode, mover, want_locs)
PyObject* lookup_fetch(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    arity(n_args, 9, "lookup_fetch");
    const at::Tensor& given = tensor(a[1], "ids");
    ids_ok(given);
    const at::Tensor ids = given.contiguous();
    const at::Tensor& rows = tensor(a[2], "cache_rows");
    const at::Device dev = ids.device();
    c10::cuda::CUDAGuard guard(dev);
    const int64_t n = ids.numel();
    at::Tensor out = none(a[5]) ? cuda_empty({n, rows.size(1)}, rows.scalar_type(), dev) : tensor(a[5], "out_rows");
    require(out.size(1) == rows.size(1), "out_rows.size(1) == cache_rows.size(1)");
    at::Tensor locs, found = cuda_empty({n}, at::kBool, dev);
    if (PyObject_IsTrue(a[8])) locs = cuda_empty({n}, at::kLong, dev);
    check(hb_lookup_fetch(static_cast<hb_index_t*>(pointer(a[0])), ids.data_ptr<int64_t>(), n, pointer(a[3]), pointer(a[4]),
                          row_bytes(rows), out.data_ptr(), locs.defined() ? locs.data_ptr<int64_t>() : nullptr,
                          static_cast<uint8_t*>(found.data_ptr()), (int)integer(a[6]), (int)integer(a[7]), stream_of(dev)));
    return pack({THPVariable_Wrap(out), wrap_or_none(locs), THPVariable_Wrap(found)});
  });
}

// unique_segsum(ids, grads, cnt | None, mean, id_bits) -> (unique ids, rows, counts), cut to the number
// of distinct ids, which is awaited while the rows are still being added up
PyObject* unique_segsum(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    arity(n_args, 5, "unique_segsum");
    const at::Tensor ids = tensor(a[0], "ids").contiguous();
    const at::Tensor grads = tensor(a[1], "grads").contiguous();
    const at::Device dev = ids.device();
    c10::cuda::CUDAGuard guard(dev);
    const int64_t n = ids.numel(), dim = grads.size(1);
    at::Tensor cnt;
    if (!none(a[2])) cnt = tensor(a[2], "cnt").contiguous();
    at::Tensor uniq = cuda_empty({n}, at::kLong, dev), counts = cuda_empty({n}, at::kLong, dev);
    at::Tensor sums = cuda_empty({n, dim}, at::kFloat, dev);
    const size_t need = hb_unique_segsum_workspace_bytes(n, dim);
    const at::Tensor ws = cuda_empty({(int64_t)need}, at::kByte, dev);
    void* st = stream_of(dev);
    int64_t* num = t_word.arm();
    check(hb_unique_segsum_f32(ids.data_ptr<int64_t>(), grads.data_ptr<float>(), cnt.defined() ? cnt.data_ptr<int64_t>() : nullptr,
                               n, nullptr, nullptr, 0, dim, (int)integer(a[4]), PyObject_IsTrue(a[3]),
                               uniq.data_ptr<int64_t>(), sums.data_ptr<float>(), counts.data_ptr<int64_t>(), num, nullptr,
                               nullptr, ws.data_ptr(), need, st));
    const int64_t u = t_word.wait(static_cast<cudaStream_t>(st));
    if (u == 0) throw std::runtime_error("the sort of the ids gave up waiting (hb_device_status)");
    return pack({THPVariable_Wrap(uniq.narrow(0, 0, u)), THPVariable_Wrap(sums.narrow(0, 0, u)),
                 THPVariable_Wrap(counts.narrow(0, 0, u))});
  });
}

// unique_update(ids, grads, cnt | None, n_dev | None, seg_counts | None, seg_cap, id_bits, optimiser, mean):
// optimiser: address of an hb_optim_t
PyObject* unique_update(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    arity(n_args, 9, "unique_update");
    const at::Tensor &ids = tensor(a[0], "idx"), &grads = tensor(a[1], "grad");
    const at::Device dev = ids.device();
    c10::cuda::CUDAGuard guard(dev);
    const int64_t n = ids.numel(), dim = grads.size(1);
    const hb_optim_t* opt = static_cast<const hb_optim_t*>(pointer(a[7]));
    auto i64 = [&](PyObject* o) -> const int64_t* { return none(o) ? nullptr : tensor(o, "count").data_ptr<int64_t>(); };
    const size_t need = hb_unique_update_workspace_bytes(n, dim, grads.data_ptr<float>(), opt);
    const at::Tensor ws = cuda_empty({(int64_t)need}, at::kByte, dev);
    check(hb_unique_update_f32(ids.data_ptr<int64_t>(), grads.data_ptr<float>(), i64(a[2]), n, i64(a[3]), i64(a[4]),
                               integer(a[5]), dim, (int)integer(a[6]), PyObject_IsTrue(a[8]),
                               opt, ws.data_ptr(), need, stream_of(dev)));
    Py_RETURN_NONE;
  });
}

// Kernels of a call read and write pinned buffers of that call: one that fails half way waits for them, and
// leaves no batch open.
struct InFlight {
  cudaStream_t stream;
  hb_index_t* index = nullptr;
  const int64_t* locs = nullptr;
  int64_t looked_up = 0;
  bool ended = false;
  ~InFlight() {
    if (ended) return;
    if (looked_up) hb_index_lookup_touch_end(index, locs, looked_up, stream);
    cudaStreamSynchronize(stream);
  }
};

// n ids as signed 32-bit numbers; false: some do not fit, found out within 512 ids of the first that does not, or at
// once from the last (sorted ids).  (Ids beyond 32 bits, 32,768 / 65,536: 48 / 79 us, 54 / 87 where all of a part was
// narrowed first, 47 / 78 without narrowing; one such id amid others near the end of a part still 54 / 71.)
__attribute__((optimize("O3"))) bool narrow(const int64_t* __restrict__ from, int32_t* __restrict__ to, int64_t n) {
  if (from[n - 1] != (int32_t)from[n - 1]) return false;
  for (int64_t at = 0; at < n; at += 512) {
    const int64_t end = n - at < 512 ? n : at + 512;
    uint64_t off = 0;  // (an id that fits lies in [0, 2^32) from -2^31 on)
    for (int64_t i = at; i < end; ++i) {
      off |= ((uint64_t)from[i] + 0x80000000ull) >> 32;
      to[i] = (int32_t)from[i];
    }
    if (off) return false;
  }
  return true;
}
__attribute__((optimize("O3"))) void widen(const int32_t* __restrict__ from, int64_t* __restrict__ to, int64_t n) {
  for (int64_t i = 0; i < n; ++i) to[i] = from[i];
}

at::Tensor pinned_empty(int64_t n) {
  return at::empty({n}, at::TensorOptions().dtype(at::kLong).pinned_memory(true));
}

// index_lookup(index, ids in host memory, device, mode, address of two words shared with other processes | 0) ->
// slots in host memory.  Ids and slots pass through two pinned buffers each, a part of the batch at a time: while
// the GPU looks one part up the host copies the next in and the one before out, and the ageing runs under the last
// copies and after.  Calls on the index from other streams wait for it; where another process has opened the index
// (words[0]), which can only be ordered by the host, the call does.  A process that opens it later finds in words[1]
// how many lookups to wait for: that is written before words[0] is read, so that one of the two waits.
// 500 ids: 25 us (two pageable copies: 70), 65,536: 65 (183; 85 with ids and slots in 64 bits on their way).
PyObject* index_lookup(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    arity(n_args, 5, "index_lookup");
    hb_index_t* h = static_cast<hb_index_t*>(pointer(a[0]));
    const at::Tensor ids = tensor(a[1], "ids").contiguous();
    const at::Device dev(at::kCUDA, (c10::DeviceIndex)integer(a[2]));
    const int mode = (int)integer(a[3]);
    c10::cuda::CUDAGuard guard(dev);
    cudaStream_t st = static_cast<cudaStream_t>(stream_of(dev));
    const int64_t n = ids.numel();
    at::Tensor out = at::empty_like(ids);
    // as few parts as 32,768 ids each allow, all of one size: a part costs the GPU some 10 us of trips over
    // PCIe whatever its size (65,536 ids in parts of 11,000: 109 us, 16,384: 87, 22,000: 74, 32,768: 65, 65,536: 70)
    constexpr int64_t kPart = 32768;
    const int64_t parts = (n + kPart - 1) / kPart, part = (n + parts - 1) / parts;
    const at::Tensor in = pinned_empty(2 * part), back = pinned_empty(2 * part);
    const at::Tensor locs = cuda_empty({n}, at::kLong, dev);
    const int64_t* src = ids.data_ptr<int64_t>();
    int64_t *to = out.data_ptr<int64_t>(), *pin = in.data_ptr<int64_t>(), *pback = back.data_ptr<int64_t>();
    volatile int64_t* words = t_word.arm();
    InFlight in_flight{st, h, locs.data_ptr<int64_t>()};
    auto length = [&](int64_t k) { return (k + 1) * part < n ? part : n - k * part; };
    bool narrowed[2] = {false, false};
    auto collect = [&](int64_t k) {
      t_word.wait(st, (int)(k & 1));
      words[k & 1] = -1;
      const int64_t* slots = pback + (k & 1) * part;
      if (narrowed[k & 1]) widen(reinterpret_cast<const int32_t*>(slots), to + k * part, length(k));
      else memcpy(to + k * part, slots, length(k) * sizeof(int64_t));
    };
    for (int64_t k = 0; k < parts; ++k) {
      if (k >= 2) collect(k - 2);
      int64_t *ids_in = pin + (k & 1) * part, *slots = pback + (k & 1) * part;
      int64_t* word = const_cast<int64_t*>(words + (k & 1));
      int32_t* ids32 = reinterpret_cast<int32_t*>(ids_in);
      narrowed[k & 1] = narrow(src + k * part, ids32, length(k));
      if (narrowed[k & 1]) {
        check(hb_index_lookup_touch_part32(h, ids32, length(k), locs.data_ptr<int64_t>(), k * part,
                                           reinterpret_cast<int32_t*>(slots), word, mode, st));
      } else {
        memcpy(ids_in, src + k * part, length(k) * sizeof(int64_t));
        check(hb_index_lookup_touch_part(h, ids_in, length(k), locs.data_ptr<int64_t>(), k * part, slots, word, mode, st));
      }
      in_flight.looked_up = k * part + length(k);
    }
    check(hb_index_lookup_touch_end(h, locs.data_ptr<int64_t>(), n, st));
    in_flight.looked_up = 0;
    for (int64_t k = parts < 2 ? 0 : parts - 2; k < parts; ++k) collect(k);
    volatile uint64_t* shared = static_cast<volatile uint64_t*>(pointer(a[4]));
    if (shared) {
      shared[1] = hb_index_lookups(h);
      std::atomic_thread_fence(std::memory_order_seq_cst);
    }
    if (shared && shared[0]) {
      cudaError_t e;
      Py_BEGIN_ALLOW_THREADS;
      e = cudaStreamSynchronize(st);
      Py_END_ALLOW_THREADS;
      if (e != cudaSuccess) throw std::runtime_error(cudaGetErrorString(e));
    }
    in_flight.ended = true;  // (what still runs uses device memory only)
    return THPVariable_Wrap(out);
  });
}

// index_add(index, ids in host memory, device) -> slots in host memory
PyObject* index_add(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    arity(n_args, 3, "index_add");
    hb_index_t* h = static_cast<hb_index_t*>(pointer(a[0]));
    const at::Tensor ids = tensor(a[1], "ids").contiguous();
    const at::Device dev(at::kCUDA, (c10::DeviceIndex)integer(a[2]));
    c10::cuda::CUDAGuard guard(dev);
    cudaStream_t st = static_cast<cudaStream_t>(stream_of(dev));
    const int64_t n = ids.numel();
    const size_t bytes = (size_t)n * sizeof(int64_t);
    at::Tensor out = at::empty_like(ids);
    const at::Tensor in = pinned_empty(n), back = pinned_empty(n);
    // up to here the walk writes its slots, one word at a time, to the pinned buffer (2,000 ids: 31 us, 41
    // with a copy); 50,000 ids: 125 us so, 93 with a copy
    const bool direct = n <= 16384;
    const at::Tensor dids = cuda_empty({n}, at::kLong, dev), locs = direct ? back : cuda_empty({n}, at::kLong, dev);
    const size_t need = hb_index_add_workspace_bytes(n);
    const at::Tensor ws = cuda_empty({(int64_t)need}, at::kByte, dev);
    memcpy(in.data_ptr(), ids.data_ptr(), bytes);
    InFlight in_flight{st};
    if (cudaMemcpyAsync(dids.data_ptr(), in.data_ptr(), bytes, cudaMemcpyHostToDevice, st) != cudaSuccess)
      throw std::runtime_error("copy of the ids to the device failed");
    check(hb_index_add(h, dids.data_ptr<int64_t>(), n, locs.data_ptr<int64_t>(), nullptr, ws.data_ptr(), need, st));
    cudaError_t e = cudaSuccess;
    Py_BEGIN_ALLOW_THREADS;
    if (!direct) e = cudaMemcpyAsync(back.data_ptr(), locs.data_ptr(), bytes, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    Py_END_ALLOW_THREADS;
    if (e != cudaSuccess) throw std::runtime_error(cudaGetErrorString(e));
    in_flight.ended = true;
    memcpy(out.data_ptr(), back.data_ptr(), bytes);
    return THPVariable_Wrap(out);
  });
}

// staging_flush(index | None, address of the hb_staging_t, cnt_threshold, rows the output holds, device) for
// one client -> (ids, rows, cnt, counts, number of stale rows); the number is read while the rows move
PyObject* staging_flush(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    arity(n_args, 5, "staging_flush");
    hb_index_t* h = none(a[0]) ? nullptr : static_cast<hb_index_t*>(pointer(a[0]));
    const hb_staging_t* s = static_cast<const hb_staging_t*>(pointer(a[1]));
    const int64_t cap = integer(a[3]);
    const at::Device dev(at::kCUDA, (c10::DeviceIndex)integer(a[4]));
    c10::cuda::CUDAGuard guard(dev);
    at::Tensor ids = cuda_empty({cap}, at::kLong, dev), rows = cuda_empty({cap, s->dim}, at::kFloat, dev);
    at::Tensor cnt = cuda_empty({cap}, at::kLong, dev), counts = cuda_empty({1}, at::kLong, dev);
    const size_t need = hb_staging_flush_workspace_bytes(s->slots, 1);
    const at::Tensor ws = cuda_empty({(int64_t)need}, at::kByte, dev);
    void* st = stream_of(dev);
    int64_t* num = t_word.arm();
    check(hb_staging_flush_counted(h, s, (int32_t)integer(a[2]), 1, cap, ids.data_ptr<int64_t>(), rows.data_ptr<float>(),
                                   cnt.data_ptr<int64_t>(), counts.data_ptr<int64_t>(), num, ws.data_ptr(), need, st));
    const int64_t stale = t_word.wait(static_cast<cudaStream_t>(st)), u = stale < cap ? stale : cap;
    return pack({THPVariable_Wrap(ids.narrow(0, 0, u)), THPVariable_Wrap(rows.narrow(0, 0, u)),
                 THPVariable_Wrap(cnt.narrow(0, 0, u)), THPVariable_Wrap(counts), PyLong_FromLongLong(stale)});
  });
}

// step_forward(step, desc, ids, dim, row dtype tensor, out_rows | None, want_locs, aside, ws | None)
// -> (rows, locs | None, found, counters, ws)
PyObject* step_forward(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    arity(n_args, 9, "step_forward");
    const at::Tensor& ids = tensor(a[2], "ids");
    ids_ok(ids);
    require(ids.is_contiguous(), "ids is contiguous");
    const at::Device dev = ids.device();
    c10::cuda::CUDAGuard guard(dev);
    const int64_t n = ids.numel(), dim = integer(a[3]);
    at::Tensor out = none(a[5]) ? cuda_empty({n, dim}, tensor(a[4], "rows").scalar_type(), dev) : tensor(a[5], "out_rows");
    require(out.size(1) == dim, "out_rows.size(1) == cache_rows.size(1)");
    require(out.is_contiguous(), "out_rows is contiguous");
    at::Tensor locs, found = cuda_empty({n}, at::kBool, dev), counters = cuda_empty({4}, at::kLong, dev);
    if (PyObject_IsTrue(a[6])) locs = cuda_empty({n}, at::kLong, dev);
    const size_t need = hb_step_workspace_bytes(n, dim);
    at::Tensor ws;
    if (!none(a[8])) ws = tensor(a[8], "ws");
    if (!ws.defined() || ws.numel() < (int64_t)need) ws = cuda_empty({(int64_t)(need + need / 4)}, at::kByte, dev);
    check(hb_step_forward(static_cast<hb_step_t*>(pointer(a[0])), static_cast<const hb_step_desc_t*>(pointer(a[1])),
                          ids.data_ptr<int64_t>(), n, out.data_ptr(), locs.defined() ? locs.data_ptr<int64_t>() : nullptr,
                          static_cast<uint8_t*>(found.data_ptr()), counters.data_ptr<int64_t>(), PyObject_IsTrue(a[7]),
                          ws.data_ptr(), (size_t)ws.numel(), stream_of(dev)));
    return pack({THPVariable_Wrap(out), wrap_or_none(locs), THPVariable_Wrap(found), THPVariable_Wrap(counters),
                 THPVariable_Wrap(ws)});
  });
}

// step_backward(step, desc, ids | None, n, grads, counters, ws)
PyObject* step_backward(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    arity(n_args, 7, "step_backward");
    const at::Tensor& grads = tensor(a[4], "grads");
    const at::Tensor& ws = tensor(a[6], "ws");
    const at::Device dev = grads.device();
    c10::cuda::CUDAGuard guard(dev);
    const int64_t n = integer(a[3]);
    const int64_t* ids = none(a[2]) ? nullptr : tensor(a[2], "ids").data_ptr<int64_t>();
    check(hb_step_backward(static_cast<hb_step_t*>(pointer(a[0])), static_cast<const hb_step_desc_t*>(pointer(a[1])), ids, n,
                           grads.data_ptr<float>(), tensor(a[5], "counters").data_ptr<int64_t>(), ws.data_ptr(),
                           (size_t)ws.numel(), stream_of(dev)));
    Py_RETURN_NONE;
  });
}

PyObject* set_error_class(PyObject*, PyObject* cls) {
  Py_XINCREF(cls);
  Py_XSETREF(g_error, cls);
  Py_RETURN_NONE;
}

#define HB_FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL
PyMethodDef g_methods[] = {
    {"lookup_fetch", HB_FAST(lookup_fetch), nullptr},
    {"unique_segsum", HB_FAST(unique_segsum), nullptr},
    {"unique_update", HB_FAST(unique_update), nullptr},
    {"index_lookup", HB_FAST(index_lookup), nullptr},
    {"index_add", HB_FAST(index_add), nullptr},
    {"staging_flush", HB_FAST(staging_flush), nullptr},
    {"step_forward", HB_FAST(step_forward), nullptr},
    {"step_backward", HB_FAST(step_backward), nullptr},
    {"set_error_class", set_error_class, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&g_module); }
