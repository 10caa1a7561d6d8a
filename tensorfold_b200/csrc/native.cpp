// The host path of the hot calls as a CPython extension: argument checks, output allocation and the C-ABI call in one
// place.  What bounds a small projection is not its kernel but the host around it: in Python (attribute walks, ctypes
// argument arrays, torch.empty, stream look-ups) one call took 21 us against 7 us on the GPU for 4096 x 4096 at four
// rows, and the seven calls of a dense layer 190 us against 90.
//
// Two kinds of functions: whole wrappers for the calls an engine issues per layer (matmul, matmul_set, prefill_matmul,
// matmul_act, add_rmsnorm, swiglu), and one thin thunk per C-ABI entry for the rest, which takes tensors where the entry
// takes pointers.  Refused arguments raise ValueError, failed launches RuntimeError.  The library itself stays free of
// Python and torch: its entry points are resolved with dlsym from the path the Python side loaded.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstdarg>
#include <map>
#include <tuple>
#include <utility>

#include "../../include/tensorfold_b200.h"

namespace {

// ---------------------------------------------------------------------------------------------------------------------
// the library's entry points
// ---------------------------------------------------------------------------------------------------------------------

#define TF_WRAPPED(X) X(tf_qmm) X(tf_qmm_set) X(tf_qmm_set_scratch_bytes) X(tf_qmm_window) X(tf_qmm_window_part_bytes) X(tf_qmm_prefill) X(tf_qmm_prefill_act) X(tf_qmm_act) \
  X(tf_add_rmsnorm) X(tf_swiglu)
#define TF_THUNKS(X) X(tf_pack) X(tf_pack_pair) X(tf_unpack) X(tf_group_sums) X(tf_affine_rows) X(tf_moe_plan) X(tf_moe_experts) \
  X(tf_moe_experts_prefill) X(tf_moe_gather) X(tf_moe_experts_sorted) X(tf_moe_router) X(tf_moe_router_tiles) X(tf_moe_topk) X(tf_moe_topk_local) X(tf_moe_combine)

#define TF_POINTER(name) decltype(&::name) p_##name = nullptr;
TF_WRAPPED(TF_POINTER)
TF_THUNKS(TF_POINTER)
decltype(&::tf_last_error) p_tf_last_error = nullptr;

PyObject* g_ensure_device = nullptr;      // Python: per-device set-up, called once a device
bool g_device_ready[64] = {};

struct Refused {};                        // a Python exception is set; unwinds to the wrapper

[[noreturn]] void refuse(const char* fmt, ...) {
  char text[256];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(text, sizeof text, fmt, ap);
  va_end(ap);
  PyErr_SetString(PyExc_ValueError, text);
  throw Refused{};
}

void check(int code, const char* what) {
  if (code == 0) return;
  const char* text = p_tf_last_error();
  if (code < 0) PyErr_Format(PyExc_ValueError, "%s: %s", what, text);
  else PyErr_Format(PyExc_RuntimeError, "%s: CUDA error %d: %s", what, code, text);
  throw Refused{};
}

// Runs a C-ABI call without the interpreter lock: a launch may wait for room in the stream's queue.
template <class Fn>
int unlocked(Fn&& fn) {
  PyThreadState* save = PyEval_SaveThread();
  const int rc = fn();
  PyEval_RestoreThread(save);
  return rc;
}

struct Owned {                            // a new reference
  PyObject* p;
  explicit Owned(PyObject* o) : p(o) {
    if (p == nullptr) throw Refused{};
  }
  Owned(const Owned&) = delete;
  ~Owned() { Py_XDECREF(p); }
};

const at::Tensor& tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) refuse("%s: a tensor is missing", what);
  return THPVariable_Unpack(o);
}

long long integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw Refused{};
  return v;
}

bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw Refused{};
  return v != 0;
}

double number(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw Refused{};
  return v;
}

// The current stream of the tensor's device, after the per-device set-up; the entry points take per-device state (error
// word, SM count, built-in scratch) from the CURRENT device, so the tensor must live there.
cudaStream_t stream_of(const at::Tensor& t) {
  if (!t.is_cuda()) refuse("operands must live on a CUDA device: this path has no CPU implementation");
  const int dev = t.get_device();
  if (dev < 0 || dev >= 64) refuse("device %d out of range", dev);
  if (!g_device_ready[dev]) {
    Owned done(PyObject_CallFunction(g_ensure_device, "i", dev));
    g_device_ready[dev] = true;
  }
  const int current = c10::cuda::current_device();
  if (dev != current)
    refuse("operands live on cuda:%d but cuda:%d is current: call under torch.cuda.device(tensor.device)", dev, current);
  return c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream();
}

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const at::Tensor& like) {
  return at::detail::empty_cuda(sizes, type, like.device(), std::nullopt);
}

bool aligned(const void* p, int bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; }

// ---------------------------------------------------------------------------------------------------------------------
// weights and rows
// ---------------------------------------------------------------------------------------------------------------------

PyObject *s_weight, *s_n, *s_k, *s_gs, *s_bits;      // interned attribute names of a packed weight

struct Weight {
  at::Tensor units;
  int n, k, gs, bits;

  Weight() = default;
  explicit Weight(PyObject* q) {
    Owned w(PyObject_GetAttr(q, s_weight));
    units = tensor(w.p, "weight");
    n = field(q, s_n), k = field(q, s_k), gs = field(q, s_gs), bits = field(q, s_bits);
    if (gs < 1) refuse("groups of %d", gs);
  }
  static int field(PyObject* q, PyObject* name) {
    Owned v(PyObject_GetAttr(q, name));
    return static_cast<int>(integer(v.p));
  }
  void check_units(const at::Tensor& x, const char* who) const {
    if (units.device() != x.device()) refuse("%s: x and the weight must share a CUDA device", who);
    if (units.dim() != 3 || units.stride(2) != 1 || units.stride(1) != units.size(2))
      refuse("%s: the tiled weight may be sliced by super-blocks of 128 columns only", who);
  }
};

// Rows of x the kernels can fetch: bulk copies read them in 16-byte pieces.
at::Tensor rows_of(const at::Tensor& x, int k, const char* who) {
  if (x.scalar_type() != at::kBFloat16 || x.dim() != 2 || x.size(1) != k) refuse("%s: x must be (M, %d) bf16", who, k);
  if (x.size(0) < 1) refuse("%s: x needs at least one row", who);
  if (x.stride(1) != 1 || (x.size(0) > 1 && x.stride(0) % 8) || !aligned(x.data_ptr(), 16)) return x.clone(at::MemoryFormat::Contiguous);
  return x;
}

// Kernels reach any CUDA memory and pinned host memory, nothing else.
void reachable(const at::Tensor& t, const char* what, const char* who) {
  if (t.is_cpu() && !t.is_pinned()) refuse("%s: %s lives in host memory that the device cannot reach", who, what);
}

const float* sums_of(PyObject* xs, const at::Tensor& x, int64_t kg, const char* who) {
  if (xs == Py_None) return nullptr;
  const at::Tensor& t = tensor(xs, who);
  const int64_t m = x.size(0);
  reachable(t, "xs", who);
  if (t.scalar_type() != at::kFloat || t.dim() != 2 || t.size(0) != m || t.size(1) != kg || !t.is_contiguous())
    refuse("%s: xs must be contiguous (%lld, %lld) fp32", who, static_cast<long long>(m), static_cast<long long>(kg));
  return t.data_ptr<float>();
}

// The caller's output, checked, or a new one.
at::Tensor out_of(PyObject* out, int64_t m, int64_t n, at::ScalarType type, const at::Tensor& x, const char* who) {
  if (out == Py_None) return empty({m, n}, type, x);
  const at::Tensor& t = tensor(out, who);
  if (t.dim() != 2 || t.size(0) != m || t.size(1) != n || t.scalar_type() != type || t.stride(1) != 1)
    refuse("%s: out must be (M, n) of the requested dtype with unit-stride rows", who);
  reachable(t, "out", who);
  return t;
}

PyObject* g_default_split = nullptr;      // Python: the load-time rule for K slices, a function of the shape only
std::map<std::tuple<int, int, int>, int> g_splits;

int split_of(PyObject* sk, const Weight& q) {
  if (sk != Py_None) {
    const int v = static_cast<int>(integer(sk));
    if (v != 0) return v;
  }
  const auto key = std::make_tuple(q.n, q.k, q.gs);
  const auto hit = g_splits.find(key);
  if (hit != g_splits.end()) return hit->second;
  Owned v(PyObject_CallFunction(g_default_split, "iii", q.n, q.k, q.gs));
  const int value = static_cast<int>(integer(v.p));
  if (g_splits.size() > 4096) g_splits.clear();
  g_splits[key] = value;
  return value;
}

// The area is handed out as a tensor: Python may replace it (a larger set) or drop it (reset_scratch) from another thread
// while a launch that uses it has given up the interpreter lock.
PyObject* g_scratch_for = nullptr;        // Python: (device, stream, bytes) -> the stream's scratch area
auto& g_scratch = *new std::map<std::pair<int, cudaStream_t>, at::Tensor>;       // (outlives the allocator's tear-down)

at::Tensor scratch_of(int dev, cudaStream_t stream, int64_t need) {
  const auto key = std::make_pair(dev, stream);
  const auto hit = g_scratch.find(key);
  if (hit != g_scratch.end() && hit->second.numel() >= need) return hit->second;
  Owned area(PyObject_CallFunction(g_scratch_for, "iKL", dev, static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream)),
                                   static_cast<long long>(need)));
  return g_scratch[key] = tensor(area.p, "scratch");
}

// ---------------------------------------------------------------------------------------------------------------------
// the matmuls
// ---------------------------------------------------------------------------------------------------------------------

constexpr int SET_MAX = 4, SET_ROWS = 16;
constexpr int CLUSTER_SLICES = 8;         // K slices tf_qmm adds on chip; more leave it through `part`

// Projections of the same 1 to 16 rows in one persistent launch; `outs` are filled in.  With `optional` it returns false where
// the sets' scratch has no room for the slices and cannot be given any (a new area during a capture): nothing is launched.
bool run_set(const at::Tensor& x, const Weight* q, const int* sk, int count, PyObject* xs, bool f32, at::Tensor* outs, bool pdl,
             const char* who, bool optional = false) {
  const cudaStream_t stream = stream_of(x);
  const int64_t m = x.size(0);
  const int k = q[0].k, kg = k / q[0].gs;
  const float* sums = sums_of(xs, x, kg, who);
  const void* tiled[SET_MAX];
  void* out[SET_MAX];
  int64_t stride[SET_MAX], ldo[SET_MAX];
  int n[SET_MAX];
  for (int i = 0; i < count; ++i) {
    q[i].check_units(x, who);
    if (sk[i] < 1 || sk[i] > kg) refuse("%s: 1 to K / gs slices (a slice holds one group at least)", who);
    tiled[i] = q[i].units.data_ptr(), stride[i] = q[i].units.stride(0), n[i] = q[i].n;
    out[i] = outs[i].data_ptr(), ldo[i] = outs[i].stride(0);
  }
  const int64_t need = p_tf_qmm_set_scratch_bytes(count, n, sk);
  if (need < 0 && optional) return false;
  if (need < 0) refuse("%s: bad shapes", who);
  at::Tensor scratch;
  try {
    scratch = scratch_of(x.get_device(), stream, need);
  } catch (const Refused&) {
    if (!optional) throw;
    PyErr_Clear();
    return false;
  }
  void* const area = scratch.data_ptr();
  const int64_t room = scratch.numel();
  const void* xp = x.data_ptr();
  const int64_t ldx = x.stride(0);
  check(unlocked([&] {
          return p_tf_qmm_set(xp, ldx, static_cast<int>(m), sums, k, q[0].bits, q[0].gs, count, tiled, stride, n, sk, out, ldo, f32,
                              area, room, pdl, stream);
        }),
        who);
  return true;
}

// Which of the two kernels for more than 16 rows (their bits are the same).  The tensor-memory kernel works on one block an
// SM and its roles start one after another, about 4 us that the tiled kernel does not pay, for each launch of up to 256 rows;
// that kernel in turn repeats its conversion and its mma.sync for every 64 rows, and makes the group sums again in every
// column block unless they are given.  And one warp adds all slices of 32 columns while its block waits, so a slice has to be
// worth it: the more slices there are, and the more affine steps (groups of 32) a weight costs.  Measured from graphs with
// weights past L2, over 256 to 17408 columns, 512 to 16384 inputs, 33 to 600 rows and six formats: of 1445 calls of 2^24
// products and more 4 are slower here than there, by 5% at most (242, by up to 2.2 times, without the slices' lines); with
// sums given 50, near the lines, by 17% at most (347).  Times in us (tensor memory / tiled), 4 bits in groups of 64: 17408 x
// 5120 in 4 slices 45 / 124 at 48 rows, 181 / 426 at 256; 1024 x 2048 15 / 13 at 48 and 53 / 50 at 600; 1536 x 4096 in 10
// slices 38 / 50 at 256; 1024 x 8192 in 21 of 399 thousand weights 44 / 41 at 128; 2048 x 16384 in 37 141 / 108 at 128; in
// groups of 32, 3072 x 5120 in 24 slices of 655 thousand 105 / 88 at 128, 4096 x 4096 in 18 of 932 thousand 37 / 44 at 33.
bool window_pays(int64_t m, const Weight& q, int sk, bool sums) {
  if (m <= 32 || sk > 32) return false;
  const int64_t weights = static_cast<int64_t>(q.n) * q.k, work = (m + 63) / 64 * weights, launches = (m + 255) / 256;
  const int64_t slice = (sk > 16 ? 720'000 : 600'000) * (q.gs == 32 ? 8 : 5) / 5;
  return work >= (int64_t{1} << 24) && weights >= sk * slice && (launches == 1 || work >= launches * (sums ? 20'000'000 : 12'000'000));
}

// The counters of the tensor-memory kernel's slices: zero, and left zero by every launch.  An eager call uses its stream's
// own 64 KB (made once a stream, returned by reset_scratch).  A captured call, whose graph may be replayed beside another
// graph captured on the same stream, uses counters that belong to the graph: the calls that one capture takes from a stream
// run one after another, so they share 64 KB, zeroed in the graph before the first of them (zeroed before every call,
// a 48-row dense layer with pdl replayed in 232 us against 225).  The tensor is held until the stream is
// seen outside that capture, so that nothing else in it gets the memory.
constexpr int64_t COUNTER_BYTES = 64 * 1024;
struct Counters {
  at::Tensor eager, captured;
  unsigned long long capture = 0;                  // the capture that `captured` belongs to
};
auto& g_counters = *new std::map<std::pair<int, cudaStream_t>, Counters>;

at::Tensor counters_of(const at::Tensor& x, cudaStream_t stream) {
  cudaStreamCaptureStatus status;
  unsigned long long capture = 0;
  C10_CUDA_CHECK(cudaStreamGetCaptureInfo(stream, &status, &capture));
  const bool capturing = status != cudaStreamCaptureStatusNone;
  const auto key = std::make_pair(static_cast<int>(x.get_device()), stream);
  auto known = g_counters.find(key);
  if (known != g_counters.end()) {
    Counters& c = known->second;
    if (c.captured.defined() && !(capturing && c.capture == capture)) c.captured = at::Tensor();
    const at::Tensor& zeroed = capturing ? c.captured : c.eager;
    if (zeroed.defined()) return zeroed;
  } else if (g_counters.size() < 256) {
    known = g_counters.emplace(key, Counters{}).first;
  }
  at::Tensor made = empty({COUNTER_BYTES}, at::kByte, x);
  made.zero_();
  if (known != g_counters.end()) {
    (capturing ? known->second.captured : known->second.eager) = made;
    if (capturing) known->second.capture = capture;
  }
  return made;
}

// matmul on the tensor-memory kernel.  False: the call is not one for it (8-bit codes, too many columns for its counters).
bool run_window(const at::Tensor& x, const Weight& q, int sk, const float* sums, bool f32, const at::Tensor& out, bool pdl,
                cudaStream_t stream, const char* who) {
  const int m = static_cast<int>(x.size(0));
  const int64_t need = p_tf_qmm_window_part_bytes(m, q.n, q.bits, sk);
  if (need < 0 || static_cast<int64_t>(sk) * (q.k / q.gs) > (1 << 30)) return false;
  at::Tensor part, counters;
  if (sk > 1) part = empty({need / 4}, at::kFloat, x), counters = counters_of(x, stream);
  check(unlocked([&] {
          return p_tf_qmm_window(x.data_ptr(), x.stride(0), m, sums, q.units.data_ptr(), q.units.stride(0), q.n, q.k, q.bits, q.gs, sk,
                                 out.data_ptr(), out.stride(0), f32, counters.defined() ? counters.data_ptr() : nullptr, COUNTER_BYTES,
                                 part.defined() ? part.data_ptr<float>() : nullptr, need, pdl, stream);
        }),
        who);
  return true;
}

// Whether a call of up to 16 rows takes the persistent kernel: always up to eight slices.  With more the tiled kernel and a
// second launch that adds the slices give the same bits and need no scratch.  A call alone is bound by its host path, so one
// launch wins (1024 x 3456 at 16 rows 10.3 us against 12.3); in a graph the second launch costs a microsecond, and a persistent
// kernel of few (column block, slice) units, whose blocks each start all of its roles, loses to it up to 16 slices: 4 bits in
// groups of 64 at 9 rows, 1024 x 3456 (72 units) 8.6 / 7.7 us, 1024 x 5120 (104) 9.2 / 8.4, 2048 x 5120 (208) 10.4 / 10.7,
// 1024 x 8192 in 21 slices 11.8 / 13.2.  With `pdl` both kernels start under the previous one's end, and the few units of very
// small projections as well in the one as in the other: 256 x 5120 (26) 8.3 / 8.4, 1024 x 5120 (104) 9.2 / 7.9, 1536 x 5120
// (156) 10.0 / 9.3, 2048 x 5120 (208) 10.1 / 10.1.  8-bit codes in groups of 128 over 8 rows, the most instructions a unit, are
// slower in it everywhere until the units fill the machine: 16 rows, 512 x 12288 18.3 / 15.1, 4096 x 8192 (320 units) 30.1 /
// 27.2 (alone 30.8 / 28.8), 3072 x 16384 (504) 38.9 / 44.4.
bool persistent_pays(int64_t m, const Weight& q, int sk, bool pdl, cudaStream_t stream) {
  if (sk <= CLUSTER_SLICES) return true;
  const int64_t units = (q.n + 127) / 128 * static_cast<int64_t>(sk);
  if (q.bits == 8 && q.gs == 128 && m > 8 && units < 448) return false;
  if (q.gs == 32 || sk > 16 || (pdl ? units < 48 || units >= 200 : units >= 112)) return true;
  cudaStreamCaptureStatus status;
  C10_CUDA_CHECK(cudaStreamIsCapturing(stream, &status));
  return status == cudaStreamCaptureStatusNone;
}

// matmul(x, q, xs, sk, f32, out, part, reduce, pdl, stream)
PyObject* matmul(PyObject* const* a) {
  const char* who = "matmul";
  const Weight q(a[1]);
  const at::Tensor x = rows_of(tensor(a[0], who), q.k, who);
  const cudaStream_t stream = stream_of(x);
  q.check_units(x, who);
  const int64_t m = x.size(0);
  const int kg = q.k / q.gs, sk = split_of(a[3], q);
  if (sk < 1 || sk > kg) refuse("matmul: 1 to K / gs slices (a slice holds one group at least)");
  const bool f32 = truth(a[4]), reduce = truth(a[7]), pdl = truth(a[8]);
  const bool slices = sk > 1 && !reduce;
  at::Tensor out;
  if (a[5] != Py_None || !slices) out = out_of(a[5], m, q.n, f32 ? at::kFloat : at::kBFloat16, x, who);
  if (truth(a[9]) && m <= SET_ROWS && a[6] == Py_None && !slices && persistent_pays(m, q, sk, pdl, stream) &&
      run_set(x, &q, &sk, 1, a[2], f32, &out, pdl, who, sk > CLUSTER_SLICES))
    return THPVariable_Wrap(out);
  const float* sums = sums_of(a[2], x, kg, who);
  if (truth(a[9]) && window_pays(m, q, sk, sums != nullptr) && a[6] == Py_None && !slices && run_window(x, q, sk, sums, f32, out, pdl, stream, who))
    return THPVariable_Wrap(out);
  at::Tensor part;
  if (sk > 1 && (!reduce || sk > CLUSTER_SLICES)) {
    if (a[6] == Py_None) {
      part = empty({sk, m, q.n}, at::kFloat, x);
    } else {
      part = tensor(a[6], who);
      if (part.scalar_type() != at::kFloat || !part.is_contiguous() || part.numel() < sk * m * q.n)
        refuse("matmul: part must hold (SK, M, n) fp32");
      reachable(part, "part", who);
    }
  }
  check(unlocked([&] {
          return p_tf_qmm(x.data_ptr(), x.stride(0), static_cast<int>(m), sums, q.units.data_ptr(), q.units.stride(0), q.n, q.k,
                          q.bits, q.gs, sk, out.defined() ? out.data_ptr() : nullptr, out.defined() ? out.stride(0) : 0, f32,
                          part.defined() ? part.data_ptr<float>() : nullptr, reduce, pdl, stream);
        }),
        who);
  if (!slices) return THPVariable_Wrap(out);
  return THPVariable_Wrap(part.reshape({-1}).narrow(0, 0, sk * m * q.n).view({sk, m, q.n}));
}

// matmul_set(x, qs, xs, sks, f32, outs, pdl)
PyObject* matmul_set(PyObject* const* a) {
  const char* who = "matmul_set";
  Owned qs(PySequence_Fast(a[1], "matmul_set: a sequence of weights"));
  const int count = static_cast<int>(PySequence_Fast_GET_SIZE(qs.p));
  if (count < 1 || count > SET_MAX) refuse("matmul_set: 1 to %d weights a set", SET_MAX);
  Weight q[SET_MAX];
  for (int i = 0; i < count; ++i) {
    q[i] = Weight(PySequence_Fast_GET_ITEM(qs.p, i));
    if (q[i].k != q[0].k || q[i].gs != q[0].gs || q[i].bits != q[0].bits)
      refuse("matmul_set: the weights of a set share K, group and bit width");
  }
  const at::Tensor x = rows_of(tensor(a[0], who), q[0].k, who);
  const int64_t m = x.size(0);
  if (m > SET_ROWS) refuse("matmul_set: at most %d rows (use matmul for larger windows)", SET_ROWS);
  stream_of(x);
  const bool f32 = truth(a[4]);
  int sk[SET_MAX];
  at::Tensor outs[SET_MAX];
  Owned sks(a[3] == Py_None ? PyTuple_New(0) : PySequence_Fast(a[3], "matmul_set: a sequence of slice counts"));
  Owned given(a[5] == Py_None ? PyTuple_New(0) : PySequence_Fast(a[5], "matmul_set: a sequence of outputs"));
  const bool own_sks = PySequence_Fast_GET_SIZE(sks.p) > 0, own_outs = a[5] != Py_None;
  if ((own_sks && PySequence_Fast_GET_SIZE(sks.p) < count) || (own_outs && PySequence_Fast_GET_SIZE(given.p) < count))
    refuse("matmul_set: one slice count and one output a weight");
  for (int i = 0; i < count; ++i) {
    sk[i] = split_of(own_sks ? PySequence_Fast_GET_ITEM(sks.p, i) : Py_None, q[i]);
    outs[i] = out_of(own_outs ? PySequence_Fast_GET_ITEM(given.p, i) : Py_None, m, q[i].n, f32 ? at::kFloat : at::kBFloat16, x, who);
  }
  run_set(x, q, sk, count, a[2], f32, outs, truth(a[6]), who);
  Owned list(PyList_New(count));
  for (int i = 0; i < count; ++i) PyList_SET_ITEM(list.p, i, THPVariable_Wrap(outs[i]));
  Py_INCREF(list.p);
  return list.p;
}

// prefill_matmul(x, q, f32, out): the formats the tcgen05 kernel takes
PyObject* prefill_matmul(PyObject* const* a) {
  const char* who = "prefill_matmul";
  const Weight q(a[1]);
  const at::Tensor x = rows_of(tensor(a[0], who), q.k, who);
  const cudaStream_t stream = stream_of(x);
  reachable(q.units, "the weight", who);
  const bool f32 = truth(a[2]);
  const at::Tensor out = out_of(a[3], x.size(0), q.n, f32 ? at::kFloat : at::kBFloat16, x, who);
  check(unlocked([&] {
          return p_tf_qmm_prefill(x.data_ptr(), x.stride(0), static_cast<int>(x.size(0)), q.units.data_ptr(), q.units.stride(0), q.n,
                                  q.k, q.gs, out.data_ptr(), out.stride(0), f32, stream);
        }),
        who);
  return THPVariable_Wrap(out);
}

// matmul_act(x, q, swiglu, limit, out, pdl, prefill)
PyObject* matmul_act(PyObject* const* a) {
  const char* who = "matmul_act";
  const Weight q(a[1]);
  const at::Tensor x = rows_of(tensor(a[0], who), q.k, who);
  const cudaStream_t stream = stream_of(x);
  reachable(q.units, "the weight", who);
  const bool swiglu = truth(a[2]), pdl = truth(a[5]), prefill = truth(a[6]) && q.bits == 4 && (q.gs == 32 || q.gs == 64);
  const float limit = static_cast<float>(number(a[3]));
  const int epi = swiglu ? 2 : 1, m = static_cast<int>(x.size(0));
  if (a[4] != Py_None) {
    const at::Tensor& t = tensor(a[4], who);
    if (t.dim() != 2 || t.size(0) != m || t.size(1) != (swiglu ? q.n / 2 : q.n) || t.scalar_type() != at::kBFloat16 || t.stride(1) != 1)
      refuse("matmul_act: out must be (M, columns) bf16 with unit-stride rows");
  }
  const at::Tensor out = out_of(a[4], m, swiglu ? q.n / 2 : q.n, at::kBFloat16, x, who);
  check(unlocked([&] {
          return prefill ? p_tf_qmm_prefill_act(x.data_ptr(), x.stride(0), m, q.units.data_ptr(), q.units.stride(0), q.n, q.k, q.gs,
                                                out.data_ptr(), out.stride(0), 0, epi, limit, stream)
                         : p_tf_qmm_act(x.data_ptr(), x.stride(0), m, q.units.data_ptr(), q.units.stride(0), q.n, q.k, q.bits, q.gs,
                                        out.data_ptr(), out.stride(0), epi, limit, pdl, stream);
        }),
        prefill ? "matmul_act (prefill)" : who);
  return THPVariable_Wrap(out);
}

// ---------------------------------------------------------------------------------------------------------------------
// glue
// ---------------------------------------------------------------------------------------------------------------------

at::Tensor glue_rows(PyObject* o, const char* who) {
  const at::Tensor& t = tensor(o, who);
  if (t.dim() != 2 || t.scalar_type() != at::kBFloat16 || !t.is_cuda()) refuse("%s: rows must be a 2-D bf16 CUDA tensor", who);
  return t.is_contiguous() ? t : t.contiguous();
}

// add_rmsnorm(x, r, w, eps, gs) -> (h, y, xs)
PyObject* add_rmsnorm(PyObject* const* a) {
  const char* who = "add_rmsnorm";
  const at::Tensor x = glue_rows(a[0], who);
  const int64_t rows = x.size(0), d = x.size(1), gs = integer(a[4]);
  at::Tensor r;
  if (a[1] != Py_None) {
    r = glue_rows(a[1], who);
    if (!r.sizes().equals(x.sizes())) refuse("add_rmsnorm: x and r must have the same shape");
  }
  const at::Tensor& wt = tensor(a[2], who);
  if (wt.scalar_type() != at::kBFloat16 || wt.dim() != 1 || wt.size(0) != d || !wt.is_cuda())
    refuse("add_rmsnorm: w must be a bf16 CUDA vector of the row length");
  if (gs < 1) refuse("add_rmsnorm: groups of 32, 64 or 128");
  const at::Tensor w = wt.contiguous();
  const cudaStream_t stream = stream_of(x);
  const at::Tensor h = r.defined() ? empty({rows, d}, at::kBFloat16, x) : x, y = empty({rows, d}, at::kBFloat16, x);
  const at::Tensor xs = empty({rows, d / gs}, at::kFloat, x);
  const float eps = static_cast<float>(number(a[3]));
  check(unlocked([&] {
          return p_tf_add_rmsnorm(x.data_ptr(), r.defined() ? r.data_ptr() : nullptr, w.data_ptr(), static_cast<int>(rows),
                                  static_cast<int>(d), eps, r.defined() ? h.data_ptr() : nullptr, y.data_ptr(), xs.data_ptr<float>(),
                                  static_cast<int>(gs), stream);
        }),
        who);
  if (r.defined() || x.is_same(tensor(a[0], who)))
    return Py_BuildValue("NNN", r.defined() ? THPVariable_Wrap(h) : Py_NewRef(a[0]), THPVariable_Wrap(y), THPVariable_Wrap(xs));
  return Py_BuildValue("NNN", THPVariable_Wrap(x), THPVariable_Wrap(y), THPVariable_Wrap(xs));
}

// swiglu(gate, up, gs) -> (out, xs)
PyObject* swiglu(PyObject* const* a) {
  const char* who = "swiglu";
  const at::Tensor gate = glue_rows(a[0], who), up = glue_rows(a[1], who);
  if (!gate.sizes().equals(up.sizes())) refuse("swiglu: gate and up must have the same shape");
  const int64_t rows = gate.size(0), n = gate.size(1), gs = integer(a[2]);
  if (gs < 1) refuse("swiglu: groups of 32, 64 or 128");
  const cudaStream_t stream = stream_of(gate);
  const at::Tensor out = empty({rows, n}, at::kBFloat16, gate), xs = empty({rows, n / gs}, at::kFloat, gate);
  check(unlocked([&] {
          return p_tf_swiglu(gate.data_ptr(), up.data_ptr(), static_cast<int>(rows), static_cast<int>(n), out.data_ptr(),
                             xs.data_ptr<float>(), static_cast<int>(gs), stream);
        }),
        who);
  return Py_BuildValue("NN", THPVariable_Wrap(out), THPVariable_Wrap(xs));
}

// ---------------------------------------------------------------------------------------------------------------------
// thunks: name(what, ...) calls the C-ABI entry `name` with tensors (or addresses, or None) for its pointers
// ---------------------------------------------------------------------------------------------------------------------

template <class T>
T convert(PyObject* o) {
  if constexpr (std::is_pointer_v<T>) {
    if (o == Py_None) return nullptr;
    if (THPVariable_Check(o)) return static_cast<T>(THPVariable_Unpack(o).data_ptr());
    void* p = PyLong_AsVoidPtr(o);
    if (p == nullptr && PyErr_Occurred()) throw Refused{};
    return static_cast<T>(p);
  } else if constexpr (std::is_floating_point_v<T>) {
    return static_cast<T>(number(o));
  } else {
    return static_cast<T>(integer(o));
  }
}

template <class... A, size_t... I>
PyObject* call_entry(int (*fn)(A...), PyObject* const* args, Py_ssize_t nargs, std::index_sequence<I...>) {
  if (nargs != static_cast<Py_ssize_t>(sizeof...(A)) + 1) {
    PyErr_Format(PyExc_TypeError, "%zu arguments wanted after the caller's name", sizeof...(A));
    throw Refused{};
  }
  const std::tuple<A...> values{convert<A>(args[1 + I])...};
  const int rc = unlocked([&] { return std::apply(fn, values); });
  if (rc != 0) {
    const char* what = PyUnicode_AsUTF8(args[0]);
    check(rc, what ? what : "call");
  }
  Py_RETURN_NONE;
}

template <class... A>
PyObject* thunk(int (*fn)(A...), PyObject* const* args, Py_ssize_t nargs) {
  return call_entry(fn, args, nargs, std::index_sequence_for<A...>{});
}

template <class Fn>
PyObject* guarded(Fn&& fn) {
  HANDLE_TH_ERRORS
  if (p_tf_last_error == nullptr) {
    PyErr_SetString(PyExc_RuntimeError, "bind() has not been called");
    return nullptr;
  }
  try {
    return fn();
  } catch (const Refused&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

#define TF_WHOLE(name, count)                                                                   \
  PyObject* py_##name(PyObject*, PyObject* const* args, Py_ssize_t nargs) {                     \
    if (nargs != count) return PyErr_Format(PyExc_TypeError, #name ": %d arguments", count);    \
    return guarded([&] { return name(args); });                                                 \
  }
TF_WHOLE(matmul, 10)
TF_WHOLE(matmul_set, 7)
TF_WHOLE(prefill_matmul, 4)
TF_WHOLE(matmul_act, 7)
TF_WHOLE(add_rmsnorm, 5)
TF_WHOLE(swiglu, 3)

#define TF_THUNK(name)                                                                          \
  PyObject* py_##name(PyObject*, PyObject* const* args, Py_ssize_t nargs) {                     \
    return guarded([&] { return thunk(p_##name, args, nargs); });                               \
  }
TF_THUNKS(TF_THUNK)

PyObject* py_stream_of(PyObject*, PyObject* t) {
  return guarded([&] { return PyLong_FromVoidPtr(stream_of(tensor(t, "stream_of"))); });
}

PyObject* py_forget_scratch(PyObject*, PyObject*) {
  g_scratch.clear();
  g_counters.clear();
  Py_RETURN_NONE;
}

// bind(library path, ensure_device)
PyObject* py_bind(PyObject*, PyObject* args) {
  const char* path;
  PyObject* ensure;
  if (!PyArg_ParseTuple(args, "sO", &path, &ensure)) return nullptr;
  void* handle = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (handle == nullptr) return PyErr_Format(PyExc_RuntimeError, "%s", dlerror());
#define TF_RESOLVE(name)                                                                        \
  p_##name = reinterpret_cast<decltype(p_##name)>(dlsym(handle, #name));                        \
  if (p_##name == nullptr) return PyErr_Format(PyExc_RuntimeError, "%s does not export " #name, path);
  TF_WRAPPED(TF_RESOLVE)
  TF_THUNKS(TF_RESOLVE)
  TF_RESOLVE(tf_last_error)
  Py_XSETREF(g_ensure_device, Py_NewRef(ensure));
  Py_RETURN_NONE;
}

// hooks(default_split, scratch_for): the Python rules the matmuls ask
PyObject* py_hooks(PyObject*, PyObject* args) {
  PyObject *split, *scratch;
  if (!PyArg_ParseTuple(args, "OO", &split, &scratch)) return nullptr;
  Py_XSETREF(g_default_split, Py_NewRef(split));
  Py_XSETREF(g_scratch_for, Py_NewRef(scratch));
  Py_RETURN_NONE;
}

#define TF_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr},
PyMethodDef g_methods[] = {
    {"bind", py_bind, METH_VARARGS, nullptr},
    {"hooks", py_hooks, METH_VARARGS, nullptr},
    {"stream_of", py_stream_of, METH_O, nullptr},
    {"forget_scratch", py_forget_scratch, METH_NOARGS, nullptr},
    TF_FAST(matmul) TF_FAST(matmul_set) TF_FAST(prefill_matmul) TF_FAST(matmul_act) TF_FAST(add_rmsnorm) TF_FAST(swiglu)
    TF_THUNKS(TF_FAST){nullptr, nullptr, 0, nullptr}};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
  s_weight = PyUnicode_InternFromString("weight"), s_n = PyUnicode_InternFromString("n"), s_k = PyUnicode_InternFromString("k");
  s_gs = PyUnicode_InternFromString("gs"), s_bits = PyUnicode_InternFromString("bits");
  return PyModule_Create(&g_module);
}
