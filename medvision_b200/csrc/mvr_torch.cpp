// Host path of the Python package: argument checks, result allocation, the autograd node of the roi modules, the upload of
// an augmentation call's rois and the launches, in one native call per operation.  Compiled against torch (the C ABI of
// libmvr.so stays free of it) into medvision_b200/_native*.so.
//
// Why native: a detection head's kernels run for 5-25 us and an augmentation of a small batch for 20-60 us, while the
// same steps in Python (ctypes marshalling, a Python autograd Function, a dozen small CPU tensor operations and views)
// took 18 us per forward, 98 us per forward + backward of a head and about 300 us per augmentation call.
#include <Python.h>

#include <atomic>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include <ATen/ATen.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/pybind.h>

#include "../../include/mvr.h"

namespace {

constexpr int kMaxDevices = 64;

// ---- small helpers ------------------------------------------------------------------------------

[[noreturn]] void raise(PyObject* kind, const std::string& what) {
  PyErr_SetString(kind, what.c_str());
  throw python_error();
}

std::string dtype_name(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return "float32";
    case at::kHalf: return "float16";
    case at::kDouble: return "float64";
    case at::kBFloat16: return "bfloat16";
    case at::kByte: return "uint8";
    case at::kChar: return "int8";
    case at::kShort: return "int16";
    case at::kInt: return "int32";
    case at::kLong: return "int64";
    case at::kBool: return "bool";
    default: return c10::toString(t);
  }
}

int dtype_code(at::ScalarType t) {
  return t == at::kFloat ? MVR_F32 : t == at::kHalf ? MVR_F16 : t == at::kDouble ? MVR_F64 : -1;
}

int label_code(at::ScalarType t) {
  return t == at::kByte ? MVR_LABEL_U8 : t == at::kShort ? MVR_LABEL_I16 : t == at::kInt ? MVR_LABEL_I32
         : t == at::kLong ? MVR_LABEL_I64 : -1;
}

void check_rc(int rc) { TORCH_CHECK(rc == MVR_OK, mvr_strerror(rc)); }

// Status word of a device: one int32 the kernels OR their status bits into.  Never freed (it may be written until the
// process ends).
std::mutex g_status_mutex;
at::Tensor* g_status[kMaxDevices] = {};

at::Tensor& status_word(int index) {
  TORCH_CHECK(index >= 0 && index < kMaxDevices, "device index out of range");
  std::lock_guard<std::mutex> lock(g_status_mutex);
  if (!g_status[index]) {
    at::NoGradGuard no_grad;
    g_status[index] = new at::Tensor(at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, index)));
  }
  return *g_status[index];
}

int* status_ptr(int index) { return (int*)status_word(index).data_ptr(); }

// ---- one roi operation --------------------------------------------------------------------------

struct RoiOp {
  int ndim, kind;      // kind: MVR_ROI_BOX / MVR_ROI_ROTATED
  int64_t out[3];      // od, oh, ow (od = 1 in 2D)
  float scale;
  int sampling, aligned, order;
  bool affine;         // the affine_* entry points: order 3 is allowed
  int width() const { return kind == MVR_ROI_BOX ? (ndim == 2 ? 5 : 7) : (ndim == 2 ? 6 : 10); }
  const char* what() const { return kind == MVR_ROI_BOX ? "RoIAlign" : "RoIAlignRotated"; }
};

std::string entry_name(const RoiOp& op, bool forward) {
  const std::string nd = op.ndim == 2 ? "2d" : "3d";
  if (op.affine) return "affine_" + nd;
  return std::string(op.kind == MVR_ROI_BOX ? "roi_align_" : "roi_align_rotated_") + nd + (forward ? "_forward" : "_backward");
}

void check_roi_tensors(const RoiOp& op, const at::Tensor& data, const at::Tensor& rois, const at::Tensor* other) {
  TORCH_CHECK(data.is_cuda(), op.what(), " is not implemented on CPU");
  TORCH_CHECK(rois.dim() == 2 && rois.size(1) == op.width(), "wrong roi size! size_rois should be ", op.width());
  TORCH_CHECK(rois.device() == data.device() && (!other || other->device() == data.device()),
              "expected all tensors to be on the same CUDA device");
  const auto t = data.scalar_type();
  TORCH_CHECK(rois.scalar_type() == t && (!other || other->scalar_type() == t), "expected scalar type torch.", dtype_name(t),
              " but found torch.", dtype_name(rois.scalar_type() != t ? rois.scalar_type() : other->scalar_type()));
}

// a: features (forward) or gradient of the output (backward); b: output or gradient of the features.  Both contiguous,
// rois contiguous, everything checked.
void launch_roi(const RoiOp& op, bool forward, const at::Tensor& a, const at::Tensor& rois, const at::Tensor& b) {
  const at::Tensor& feat = forward ? a : b;
  const bool d3 = op.ndim == 3;
  const int index = a.device().index();
  c10::cuda::CUDAGuard guard(a.device());
  void* stream = (void*)c10::cuda::getCurrentCUDAStream(index).stream();
  const int code = dtype_code(a.scalar_type());
  const int64_t N = feat.size(0), C = feat.size(1), D = d3 ? feat.size(2) : 1, H = feat.size(d3 ? 3 : 2), W = feat.size(d3 ? 4 : 3);
  int* status = status_ptr(index);
  int rc;
  if (op.affine) {
    rc = d3 ? mvr_affine_3d(a.data_ptr(), rois.data_ptr(), b.data_ptr(), code, N, C, D, H, W, rois.size(0), op.width(),
                            (int)op.out[0], (int)op.out[1], (int)op.out[2], op.scale, op.sampling, op.aligned, op.order, status, stream)
            : mvr_affine_2d(a.data_ptr(), rois.data_ptr(), b.data_ptr(), code, N, C, H, W, rois.size(0), op.width(),
                            (int)op.out[1], (int)op.out[2], op.scale, op.sampling, op.aligned, op.order, status, stream);
  } else {
    auto fn = forward ? mvr_roi_resample_fwd : mvr_roi_resample_bwd;
    rc = fn(a.data_ptr(), rois.data_ptr(), b.data_ptr(), code, op.ndim, op.kind, N, C, D, H, W, rois.size(0), op.width(),
            (int)op.out[0], (int)op.out[1], (int)op.out[2], op.scale, op.sampling, op.aligned, op.order, status, stream);
  }
  check_rc(rc);
}

void check_dtype_and_dims(const RoiOp& op, bool forward, const at::Tensor& a, const at::Tensor& feat) {
  TORCH_CHECK(dtype_code(a.scalar_type()) >= 0, "\"", entry_name(op, forward), "\" not implemented for '",
              dtype_name(a.scalar_type()), "'");
  TORCH_CHECK(feat.dim() == op.ndim + 2, entry_name(op, forward), ": expected a ", op.ndim + 2, "-D feature tensor");
}

std::vector<int64_t> result_shape(const RoiOp& op, int64_t R, int64_t C) {
  return op.ndim == 3 ? std::vector<int64_t>{R, C, op.out[0], op.out[1], op.out[2]}
                      : std::vector<int64_t>{R, C, op.out[1], op.out[2]};
}

// Forward into a new tensor; no autograd here.
at::Tensor roi_forward(const RoiOp& op, const at::Tensor& features, const at::Tensor& rois) {
  check_roi_tensors(op, features, rois, nullptr);
  check_dtype_and_dims(op, true, features, features);
  at::NoGradGuard no_grad;
  const at::Tensor f = features.contiguous(), r = rois.contiguous();
  at::Tensor out = at::empty(result_shape(op, r.size(0), f.size(1)), f.options().requires_grad(false));
  launch_roi(op, true, f, r, out);
  return out;
}

// at::zeros without its tensor iterator: one memset on the current stream.
at::Tensor zero_filled(at::IntArrayRef size, const at::TensorOptions& options) {
  at::Tensor t = at::empty(size, options);
  if (!t.is_cuda()) return t.zero_();
  if (t.numel() > 0) {
    c10::cuda::CUDAGuard guard(t.device());
    C10_CUDA_CHECK(cudaMemsetAsync(t.data_ptr(), 0, t.nbytes(), c10::cuda::getCurrentCUDAStream(t.device().index()).stream()));
  }
  return t;
}

// Gradient of the features.  The roi kernels add into a zero-filled tensor.
struct RoiBackward : public torch::autograd::Node {
  RoiOp op;
  torch::autograd::SavedVariable rois;
  std::vector<int64_t> feature_size;
  at::TensorOptions options;  // of the rois: the gradient takes their dtype, as rois.new_zeros does

  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    torch::autograd::variable_list result(2);
    const at::Tensor r = rois.unpack();
    if (!task_should_compute_output(0)) return result;
    at::NoGradGuard no_grad;
    at::Tensor gin = zero_filled(feature_size, options);
    if (grads[0].defined()) {
      const at::Tensor g = grads[0].contiguous();
      check_roi_tensors(op, g, r, &gin);
      check_dtype_and_dims(op, false, g, gin);
      launch_roi(op, false, g, r.contiguous(), gin);
    }
    result[0] = gin;
    return result;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    rois.reset_data();
  }
  std::string name() const override {
    return std::string(op.what()) + (op.ndim == 2 ? "2D" : "3D") + "FunctionBackward";
  }
};

bool has_tangent(const at::Tensor& t) { return torch::autograd::impl::get_autograd_meta(t) && t._fw_grad(/*level=*/0).defined(); }

at::Tensor roi_module_forward(const RoiOp& op, const at::Tensor& features, const at::Tensor& rois) {
  TORCH_CHECK_NOT_IMPLEMENTED(!has_tangent(features) && !has_tangent(rois), op.what(), " has no forward-mode derivative");
  at::Tensor out = roi_forward(op, features, rois);
  if (torch::autograd::compute_requires_grad(features, rois)) {
    auto node = std::shared_ptr<RoiBackward>(new RoiBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(features, rois));
    node->op = op;
    node->rois = torch::autograd::SavedVariable(rois, false);
    node->feature_size = features.sizes().vec();
    node->options = rois.options().requires_grad(false);
    torch::autograd::set_history(out, node);
  }
  return out;
}

// ---- affine_2d / affine_3d ------------------------------------------------------------------------

at::Tensor affine_forward(RoiOp op, const at::Tensor& features, const at::Tensor& rois) {
  at::NoGradGuard no_grad;
  if (op.order == 0) op.sampling = 1;  // averaging samples would blend labels
  // the rois take the dtype (and device) of the image, as rois.type(features.type()) does
  const at::Tensor r = rois.to(features.options().requires_grad(false), /*non_blocking=*/false, /*copy=*/false);
  return roi_forward(op, features, r);
}

// ---- label fields ---------------------------------------------------------------------------------

// Nearest resampling of integer labels into a given int32 tensor; false: no label kernel for the shape.
bool label_into(const at::Tensor& labels, const at::Tensor& rois, const at::Tensor& out, const RoiOp& op) {
  const bool d3 = op.ndim == 3;
  const int index = labels.device().index();
  c10::cuda::CUDAGuard guard(labels.device());
  void* stream = (void*)c10::cuda::getCurrentCUDAStream(index).stream();
  const int code = label_code(labels.scalar_type());
  const int64_t N = labels.size(0), C = labels.size(1), R = rois.size(0);
  int* status = status_ptr(index);
  const int rc = d3 ? mvr_affine_label_3d(labels.data_ptr(), code, (const float*)rois.data_ptr(), (int32_t*)out.data_ptr(), N, C,
                                          labels.size(2), labels.size(3), labels.size(4), R, op.width(), (int)op.out[0],
                                          (int)op.out[1], (int)op.out[2], op.scale, op.aligned, status, stream)
                    : mvr_affine_label_2d(labels.data_ptr(), code, (const float*)rois.data_ptr(), (int32_t*)out.data_ptr(), N, C,
                                          labels.size(2), labels.size(3), R, op.width(), (int)op.out[1], (int)op.out[2],
                                          op.scale, op.aligned, status, stream);
  if (rc == MVR_ERR_UNSUPPORTED) return false;
  check_rc(rc);
  return true;
}

void check_label_tensors(const RoiOp& op, const at::Tensor& labels, const at::Tensor& rois) {
  TORCH_CHECK(labels.is_cuda(), "RoIAlignRotated is not implemented on CPU");
  TORCH_CHECK(label_code(labels.scalar_type()) >= 0, "\"affine_label\" not implemented for '", dtype_name(labels.scalar_type()), "'");
  TORCH_CHECK(rois.dim() == 2 && rois.size(1) == op.width(), "wrong roi size! size_rois should be ", op.width());
}

at::Tensor label_forward(RoiOp op, const at::Tensor& labels, const at::Tensor& rois_any) {
  at::NoGradGuard no_grad;
  const at::Tensor rois = rois_any.to(at::TensorOptions().device(labels.device()).dtype(at::kFloat)).contiguous();
  if (label_code(labels.scalar_type()) >= 0) {
    check_label_tensors(op, labels, rois);
    const at::Tensor l = labels.contiguous();
    at::Tensor out = at::empty(result_shape(op, rois.size(0), l.size(1)), l.options().dtype(at::kInt));
    if (label_into(l, rois, out, op)) return out;
  }
  op.sampling = 1;
  op.order = 0;
  return affine_forward(op, labels.to(at::kFloat), rois).to(at::kInt);
}

// An image field and its label field in one go (one sample per voxel, orders 0 and 1); false: rois too small for the label
// kernels.
bool fields_into(const RoiOp& op, const at::Tensor& image, const at::Tensor& image_rois, const at::Tensor& image_out,
                 const at::Tensor& labels, const at::Tensor& label_rois, const at::Tensor& label_out) {
  const int index = image.device().index();
  c10::cuda::CUDAGuard guard(image.device());
  void* stream = (void*)c10::cuda::getCurrentCUDAStream(index).stream();
  int* status = status_ptr(index);
  const int code = dtype_code(image.scalar_type()), lcode = label_code(labels.scalar_type());
  const int rc = op.ndim == 3
      ? mvr_affine_fields_3d(image.data_ptr(), code, image_rois.data_ptr(), image_out.data_ptr(), image.size(1), labels.data_ptr(), lcode,
                             (const float*)label_rois.data_ptr(), (int32_t*)label_out.data_ptr(), labels.size(1), image.size(0),
                             image.size(2), image.size(3), image.size(4), image_rois.size(0), 10, (int)op.out[0], (int)op.out[1],
                             (int)op.out[2], op.scale, op.aligned, op.order, status, stream)
      : mvr_affine_fields_2d(image.data_ptr(), code, image_rois.data_ptr(), image_out.data_ptr(), image.size(1), labels.data_ptr(), lcode,
                             (const float*)label_rois.data_ptr(), (int32_t*)label_out.data_ptr(), labels.size(1), image.size(0),
                             image.size(2), image.size(3), image_rois.size(0), 6, (int)op.out[1], (int)op.out[2], op.scale,
                             op.aligned, op.order, status, stream);
  if (rc == MVR_ERR_UNSUPPORTED) return false;
  check_rc(rc);
  return true;
}

// ---- upload of a call's parameters ------------------------------------------------------------------
// The parameters of a transform are drawn on the host, so one small upload per call is inherent.  It is ONE asynchronous
// copy from pinned memory into a device buffer kept across calls.  A ring of kSlots such pairs per device: a slot is used
// again when the kernels that read it last are done (an event recorded behind them), so up to kSlots calls can be in
// flight; the ring is locked for the whole call, so any number of threads and streams may use it.  It holds kSlots times
// twice the largest call (some KB each) and goes away with release_staging().
//
// A call that is being captured into a CUDA graph takes no slot: a replay reads the host memory again, whatever eager calls
// have done to the ring since.  It gets pinned memory of its own, which the graph and everything instantiated from it hold
// as a user object, and device memory from the graph's own pool.
constexpr int kSlots = 8;

// Calls that allocate or wait must not break a capture that this or another thread has under way.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { C10_CUDA_CHECK(cudaThreadExchangeStreamCaptureMode(&mode)); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Pinned memory of graphs that are gone.  A user object's destructor may not call CUDA, so it only leaves the address here;
// the next eager upload and release_staging() free it.
struct Orphans {
  std::mutex mutex;
  std::vector<void*> memory;
  std::atomic<bool> any{false};
};
Orphans& orphans() {
  static Orphans* o = new Orphans();  // a graph may outlive every static
  return *o;
}
void CUDART_CB leave_orphan(void* memory) {
  Orphans& o = orphans();
  std::lock_guard<std::mutex> lock(o.mutex);
  o.memory.push_back(memory);
  o.any = true;
}
void free_orphans() {
  Orphans& o = orphans();
  if (!o.any) return;
  std::vector<void*> memory;
  {
    std::lock_guard<std::mutex> lock(o.mutex);
    memory.swap(o.memory);
    o.any = false;
  }
  RelaxedCapture relaxed;
  for (void* m : memory) cudaFreeHost(m);
}

struct Stage {
  std::mutex mutex;
  int64_t capacity = 0;  // bytes per slot
  void* host[kSlots] = {};
  at::Tensor dev[kSlots];
  cudaEvent_t event[kSlots] = {};
  bool recorded[kSlots] = {};
  int next = 0;

  void release() {
    RelaxedCapture relaxed;
    for (int k = 0; k < kSlots; ++k) {
      if (recorded[k]) C10_CUDA_CHECK(cudaEventSynchronize(event[k]));
      recorded[k] = false;
      if (host[k]) C10_CUDA_CHECK(cudaFreeHost(host[k]));
      host[k] = nullptr;
      dev[k] = at::Tensor();
    }
    capacity = 0;
  }
  void reserve(int64_t bytes, at::Device device) {
    if (bytes <= capacity) return;
    release();
    RelaxedCapture relaxed;
    const int64_t want = std::max<int64_t>(8192, 2 * bytes);
    for (int k = 0; k < kSlots; ++k) {
      C10_CUDA_CHECK(cudaHostAlloc(&host[k], (size_t)want, cudaHostAllocDefault));
      dev[k] = at::empty({want}, at::TensorOptions().dtype(at::kByte).device(device));
      if (!event[k]) C10_CUDA_CHECK(cudaEventCreateWithFlags(&event[k], cudaEventDisableTiming));
    }
    capacity = want;
  }
};
Stage* g_stage[kMaxDevices] = {};
std::mutex g_stage_mutex;

Stage& stage_of(int index) {
  TORCH_CHECK(index >= 0 && index < kMaxDevices, "device index out of range");
  std::lock_guard<std::mutex> lock(g_stage_mutex);
  if (!g_stage[index]) g_stage[index] = new Stage();  // lives until the process ends, like the CUDA context
  return *g_stage[index];
}

// The memory of one call: fill host(), send(), launch the kernels that read device(); the destructor marks the slot free
// behind them.
struct Upload {
  Stage& stage;
  std::unique_lock<std::mutex> lock;
  cudaStream_t stream;
  bool capturing;
  int slot = -1;
  void* own_host = nullptr;  // captured calls
  at::Tensor own_dev;

  Upload(int64_t bytes, at::Device device)
      : stage(stage_of(device.index())), stream(c10::cuda::getCurrentCUDAStream(device.index()).stream()) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    C10_CUDA_CHECK(cudaStreamIsCapturing(stream, &cs));
    capturing = cs != cudaStreamCaptureStatusNone;
    if (capturing) {
      own(std::max<int64_t>(bytes, 1), device);
      return;
    }
    free_orphans();
    lock = std::unique_lock<std::mutex>(stage.mutex);
    stage.reserve(bytes, device);
    slot = stage.next;
    stage.next = (slot + 1) % kSlots;
    if (stage.recorded[slot]) {
      RelaxedCapture relaxed;
      C10_CUDA_CHECK(cudaEventSynchronize(stage.event[slot]));
      stage.recorded[slot] = false;
    }
  }
  void own(int64_t bytes, at::Device device) {
    own_dev = at::empty({bytes}, at::TensorOptions().dtype(at::kByte).device(device));
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaGraph_t graph = nullptr;
    C10_CUDA_CHECK(cudaStreamGetCaptureInfo_v2(stream, &cs, nullptr, &graph, nullptr, nullptr));
    TORCH_CHECK(cs == cudaStreamCaptureStatusActive && graph, "the capture of the current stream is invalid");
    RelaxedCapture relaxed;
    C10_CUDA_CHECK(cudaHostAlloc(&own_host, (size_t)bytes, cudaHostAllocDefault));
    cudaUserObject_t object = nullptr;
    cudaError_t err = cudaUserObjectCreate(&object, own_host, leave_orphan, 1, cudaUserObjectNoDestructorSync);
    if (err != cudaSuccess) {
      cudaFreeHost(own_host);
    } else {
      err = cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove);
      if (err != cudaSuccess) cudaUserObjectRelease(object, 1);
    }
    C10_CUDA_CHECK(err);
  }
  void* host() { return capturing ? own_host : stage.host[slot]; }
  void* device() { return capturing ? own_dev.data_ptr() : stage.dev[slot].data_ptr(); }
  void send(int64_t bytes) { C10_CUDA_CHECK(cudaMemcpyAsync(device(), host(), (size_t)bytes, cudaMemcpyHostToDevice, stream)); }
  ~Upload() {
    if (capturing || slot < 0) return;
    if (cudaEventRecord(stage.event[slot], stream) == cudaSuccess) stage.recorded[slot] = true;
    else cudaStreamSynchronize(stream);
  }
};

// Rois of one call on the device, in float32 (label fields) and, rounded on the host exactly as the device cast rounds, in
// float16 (half images).
struct StagedRois {
  Upload up;
  at::Tensor f32, f16;

  StagedRois(const at::Tensor& rois, at::Device device) : up(rois.numel() * 6, device) {
    const int64_t n = rois.numel(), R = rois.size(0), K = rois.size(1);
    const float* src = (const float*)rois.data_ptr();
    float* h32 = (float*)up.host();
    at::Half* h16 = (at::Half*)(h32 + n);
    for (int64_t i = 0; i < n; ++i) {
      h32[i] = src[i];
      h16[i] = at::Half(src[i]);  // round to nearest even
    }
    up.send(n * 6);
    // views by pointer: the upload (its ring, or its graph) keeps the memory
    auto none = [](void*) {};
    f32 = at::from_blob(up.device(), {R, K}, none, at::TensorOptions().dtype(at::kFloat).device(device));
    f16 = at::from_blob((char*)up.device() + 4 * n, {R, K}, none, at::TensorOptions().dtype(at::kHalf).device(device));
  }
};

using Tensors = std::vector<at::Tensor>;

// Every image field (order `op.order`) and label field (nearest) of one augmentation call.
void resample_fields(RoiOp op, const Tensors& images, const Tensors& labels, const at::Tensor& rois_cpu, Tensors& images_out,
                     Tensors& labels_out) {
  at::NoGradGuard no_grad;
  const at::Device device = (images.empty() ? labels : images)[0].device();
  c10::cuda::CUDAGuard guard(device);
  const at::Tensor src = rois_cpu.to(at::kFloat).contiguous();
  StagedRois staged(src, device);
  auto rois_for = [&](const at::Tensor& t) {
    const at::Tensor& r = t.scalar_type() == at::kHalf ? staged.f16 : staged.f32;
    return t.device() == device ? r : r.to(t.device());
  };
  const int64_t R = src.size(0);
  size_t fused = 0;
  if (op.sampling == 1 && (op.order == 0 || op.order == 1)) {
    // pairs of (image field, label field): one call each
    for (; fused < images.size() && fused < labels.size(); ++fused) {
      const at::Tensor &im = images[fused], &lb = labels[fused];
      if (im.device() != device || lb.device() != device || im.size(0) != lb.size(0) || im.sizes().slice(2) != lb.sizes().slice(2) ||
          (im.scalar_type() != at::kHalf && im.scalar_type() != at::kFloat) || label_code(lb.scalar_type()) < 0)
        break;
      const at::Tensor i = im.contiguous(), l = lb.contiguous();
      at::Tensor io = at::empty(result_shape(op, R, i.size(1)), i.options().requires_grad(false));
      at::Tensor lo = at::empty(result_shape(op, R, l.size(1)), l.options().dtype(at::kInt));
      if (!fields_into(op, i, rois_for(i), io, l, staged.f32, lo)) lo = label_forward(op, l, staged.f32);
      images_out.push_back(io);
      labels_out.push_back(lo);
    }
  }
  for (size_t k = fused; k < images.size(); ++k) images_out.push_back(affine_forward(op, images[k], rois_for(images[k])));
  for (size_t k = fused; k < labels.size(); ++k)
    // = affine(label.float(), rois, out_size, 1.0, 1, True, 0).int() of the reference, on the integers themselves
    labels_out.push_back(label_forward(op, labels[k], labels[k].device() == device ? staged.f32 : staged.f32.to(labels[k].device())));
}

// ---- displacement-field warp ------------------------------------------------------------------------

at::Tensor apply_offset(const at::Tensor& input, const at::Tensor& offset_any, int order) {
  at::NoGradGuard no_grad;
  const int ndim = (int)input.dim() - 2;
  const std::string name = "deform_" + std::to_string(ndim) + "d";
  TORCH_CHECK(input.is_cuda(), "Not implemented on the CPU");
  TORCH_CHECK((ndim == 2 || ndim == 3) && offset_any.dim() == ndim + 2 && offset_any.size(1) == ndim &&
                  offset_any.sizes().slice(2) == input.sizes().slice(2) && offset_any.size(0) == input.size(0),
              name, ": offset must be (B, ", ndim, ", *spatial) for input (B, C, *spatial)");
  TORCH_CHECK(offset_any.device() == input.device(), "expected all tensors to be on the same CUDA device");
  const auto t = input.scalar_type(), ot = offset_any.scalar_type();
  TORCH_CHECK(t == at::kFloat || t == at::kHalf, "\"", name, "\" not implemented for '", dtype_name(t), "'");
  TORCH_CHECK(ot == t || (t == at::kHalf && ot == at::kFloat), "expected scalar type torch.", dtype_name(t), " but found torch.",
              dtype_name(ot));
  if (!input.is_contiguous()) raise(PyExc_AssertionError, "input tensor has to be contiguous");
  const at::Tensor offset = offset_any.contiguous();
  at::Tensor out = at::empty(input.sizes(), input.options().requires_grad(false));
  const int index = input.device().index();
  c10::cuda::CUDAGuard guard(input.device());
  void* stream = (void*)c10::cuda::getCurrentCUDAStream(index).stream();
  check_rc(ndim == 2 ? mvr_apply_offset_2d(input.data_ptr(), offset.data_ptr(), out.data_ptr(), dtype_code(t), dtype_code(ot),
                                           input.size(0), input.size(1), input.size(2), input.size(3), order, stream)
                     : mvr_apply_offset_3d(input.data_ptr(), offset.data_ptr(), out.data_ptr(), dtype_code(t), dtype_code(ot),
                                           input.size(0), input.size(1), input.size(2), input.size(3), input.size(4), order, stream));
  return out;
}

// ---- elastic deformation ------------------------------------------------------------------------------

// coarse (B, *grid, ndim) float32 on the host, halved as it goes up ("to smooth"); every image field and label field of one
// call, or the dense field.  False: no kernel for the grid.
bool elastic(const at::Tensor& coarse, int border, const std::vector<int64_t>& shape, at::ScalarType position_type,
             const Tensors& images, const Tensors& labels, at::Tensor* field, at::Device device, Tensors& images_out,
             Tensors& labels_out) {
  at::NoGradGuard no_grad;
  const int ndim = (int)shape.size();
  const int64_t B = coarse.size(0);
  const int gd = ndim == 3 ? (int)coarse.size(1) : 1, gh = (int)coarse.size(ndim - 1), gw = (int)coarse.size(ndim);
  const int64_t points = (int64_t)gd * gh * gw, D = ndim == 3 ? shape[0] : 1, H = shape[ndim - 2], W = shape[ndim - 1];
  c10::cuda::CUDAGuard guard(device);
  Upload up(coarse.numel() * 4, device);
  const float* src = (const float*)coarse.data_ptr();
  float* dst = (float*)up.host();
  for (int64_t b = 0; b < B; ++b)
    for (int64_t i = 0; i < points; ++i)
      for (int c = 0; c < ndim; ++c) dst[(b * ndim + c) * points + i] = src[(b * points + i) * ndim + c] / 2;
  up.send(coarse.numel() * 4);
  auto call = [&](const at::Tensor* im, const at::Tensor* lb, float* f) {
    at::Tensor i, l, io, lo;
    if (im) {
      i = im->contiguous();
      io = at::empty(i.sizes(), i.options().requires_grad(false));
    }
    if (lb) {
      l = lb->contiguous();
      lo = at::empty(l.sizes(), l.options().dtype(at::kInt));
    }
    const int rc = mvr_elastic((const float*)up.device(), ndim, gd, gh, gw, border, im ? i.data_ptr() : nullptr,
                               dtype_code(im ? i.scalar_type() : position_type), im ? io.data_ptr() : nullptr, im ? i.size(1) : 0,
                               lb ? l.data_ptr() : nullptr, lb ? label_code(l.scalar_type()) : 0,
                               lb ? (int32_t*)lo.data_ptr() : nullptr, lb ? l.size(1) : 0, f, B, D, H, W, (void*)up.stream);
    if (rc == MVR_ERR_UNSUPPORTED) return false;
    check_rc(rc);
    if (im) images_out.push_back(io);
    if (lb) labels_out.push_back(lo);
    return true;
  };
  if (field) {
    std::vector<int64_t> size{B, ndim};
    size.insert(size.end(), shape.begin(), shape.end());
    *field = at::empty(size, at::TensorOptions().dtype(at::kFloat).device(device));
    return call(nullptr, nullptr, (float*)field->data_ptr());
  }
  const size_t n = std::max(images.size(), labels.size());
  for (size_t k = 0; k < n; ++k) {
    const at::Tensor* im = k < images.size() ? &images[k] : nullptr;
    const at::Tensor* lb = k < labels.size() ? &labels[k] : nullptr;
    if (im && lb && im->scalar_type() == position_type) {
      if (!call(im, lb, nullptr)) return false;
    } else if ((im && !call(im, nullptr, nullptr)) || (lb && !call(nullptr, lb, nullptr))) {
      return false;
    }
  }
  return true;
}

// ---- parameter draws --------------------------------------------------------------------------------------
// numpy's global generator, drawn from natively through the C interface that numpy documents for extensions (the capsule of
// a BitGenerator).  The order and the arithmetic of the draws are numpy's: uniform(lo, hi) is lo + (hi - lo) * next_double,
// randint(0, n) masks 32-bit numbers and rejects those above n - 1 (and draws nothing for n = 1).

struct BitGen {
  void* state;
  uint64_t (*next_uint64)(void*);
  uint32_t (*next_uint32)(void*);
  double (*next_double)(void*);
  uint64_t (*next_raw)(void*);
};

// A C-contiguous numpy array of 8-byte (double / int64) or 4-byte (float) items.
struct Buffer {
  Py_buffer view;
  Buffer(PyObject* o, int itemsize, Py_ssize_t items, bool writable) {
    if (PyObject_GetBuffer(o, &view, PyBUF_C_CONTIGUOUS | (writable ? PyBUF_WRITABLE : 0)) != 0) throw python_error();
    if (view.itemsize != itemsize || view.len != items * itemsize) {
      PyBuffer_Release(&view);
      raise(PyExc_ValueError, "unexpected array size");
    }
  }
  ~Buffer() { PyBuffer_Release(&view); }
  Buffer(const Buffer&) = delete;
  template <typename T> T* as() { return (T*)view.buf; }
};

// ---- Python bindings ----------------------------------------------------------------------------------

const at::Tensor& tensor_arg(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) raise(PyExc_TypeError, std::string(name) + " must be a torch.Tensor");
  return THPVariable_Unpack(o);
}
long long int_arg(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);  // takes anything with __index__
  if (v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    PyObject* n = PyNumber_Long(o);  // int(o), as the ctypes wrappers did
    if (!n) throw python_error();
    const long long w = PyLong_AsLongLong(n);
    Py_DECREF(n);
    if (w == -1 && PyErr_Occurred()) throw python_error();
    return w;
  }
  return v;
}
double float_arg(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}
bool bool_arg(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw python_error();
  return v != 0;
}
int checked_size(long long v) {
  TORCH_CHECK(v >= INT32_MIN && v <= INT32_MAX, "output size out of range");
  return (int)v;
}
// int -> the same size on every axis; tuple of ndim ints -> as given; anything else is a TypeError
void out_size_arg(PyObject* o, int ndim, const char* name, RoiOp& op) {
  op.out[0] = 1;
  int64_t* dst = op.out + (3 - ndim);
  if (PyLong_Check(o)) {
    for (int i = 0; i < ndim; ++i) dst[i] = checked_size(int_arg(o));
    return;
  }
  if (!PyTuple_Check(o)) raise(PyExc_TypeError, "\"" + std::string(name) + "\" must be an integer or tuple of integers");
  if (PyTuple_GET_SIZE(o) != ndim) raise(PyExc_AssertionError, std::string(name) + " must have " + std::to_string(ndim) + " entries");
  for (int i = 0; i < ndim; ++i) {
    PyObject* v = PyTuple_GET_ITEM(o, i);
    if (!PyLong_Check(v)) raise(PyExc_AssertionError, std::string(name) + " must hold integers");
    dst[i] = checked_size(int_arg(v));
  }
}
void need(Py_ssize_t n, Py_ssize_t lo, Py_ssize_t hi) {
  if (n < lo || n > hi) raise(PyExc_TypeError, "expected " + std::to_string(lo) + " to " + std::to_string(hi) + " arguments, got " + std::to_string(n));
}

// roi_align_{2d,3d}(features, rois, output_size, spatial_scale, sampling_ratio=0, order=1)
// roi_align_rotated_{2d,3d}(features, rois, output_size, spatial_scale, sampling_ratio=0, aligned=True, order=1)
template <int NDIM, int KIND>
PyObject* py_roi(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need(n, 4, KIND == MVR_ROI_BOX ? 6 : 7);
  const at::Tensor &features = tensor_arg(a[0], "features"), &rois = tensor_arg(a[1], "rois");
  RoiOp op{};
  op.ndim = NDIM;
  op.kind = KIND;
  out_size_arg(a[2], NDIM, "output_size", op);
  op.scale = (float)float_arg(a[3]);
  op.sampling = n > 4 ? (int)int_arg(a[4]) : 0;
  if (KIND == MVR_ROI_BOX) {
    op.aligned = 0;
    op.order = n > 5 ? (int)int_arg(a[5]) : 1;
  } else {
    op.aligned = n > 5 ? bool_arg(a[5]) : 1;
    op.order = n > 6 ? (int)int_arg(a[6]) : 1;
  }
  if (features.dim() != NDIM + 2) raise(PyExc_AssertionError, "features must have " + std::to_string(NDIM + 2) + " dimensions");
  at::Tensor out;
  {
    pybind11::gil_scoped_release nogil;
    out = roi_module_forward(op, features, rois);
  }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// roi_call(kind, ndim, forward, affine, a, rois, b, out_sizes, spatial_scale, sampling_ratio, aligned, order): the extension
// surface, into a caller-allocated tensor
PyObject* py_roi_call(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need(n, 12, 12);
  RoiOp op{};
  op.kind = (int)int_arg(a[0]);
  op.ndim = (int)int_arg(a[1]);
  const bool forward = bool_arg(a[2]);
  op.affine = bool_arg(a[3]);
  const at::Tensor &x = tensor_arg(a[4], "tensor"), &rois = tensor_arg(a[5], "rois"), &b = tensor_arg(a[6], "tensor");
  op.out[0] = 1;
  for (int i = 0; i < op.ndim; ++i) op.out[3 - op.ndim + i] = checked_size(int_arg(PyTuple_GET_ITEM(a[7], i)));
  op.scale = (float)float_arg(a[8]);
  op.sampling = (int)int_arg(a[9]);
  op.aligned = bool_arg(a[10]);
  op.order = (int)int_arg(a[11]);
  {
    pybind11::gil_scoped_release nogil;
    at::NoGradGuard no_grad;
    check_roi_tensors(op, x, rois, &b);
    const at::Tensor& feat = forward ? x : b;
    check_dtype_and_dims(op, forward, x, feat);
    const at::Tensor xc = x.contiguous(), rc = rois.contiguous();
    const std::string name = entry_name(op, forward);
    TORCH_CHECK(b.is_contiguous(), name, ": the result tensor must be contiguous");
    const auto want = result_shape(op, rois.size(0), feat.size(1));
    const at::Tensor& other = forward ? b : x;
    TORCH_CHECK(other.sizes() == at::IntArrayRef(want), name, ": expected a tensor of shape ", at::IntArrayRef(want), ", got ", other.sizes());
    launch_roi(op, forward, xc, rc, b);
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

RoiOp affine_op(int ndim, PyObject* out_size, PyObject* scale, PyObject* sampling, PyObject* aligned, PyObject* order) {
  RoiOp op{};
  op.ndim = ndim;
  op.kind = MVR_ROI_ROTATED;
  op.affine = true;
  out_size_arg(out_size, ndim, "out_size", op);
  op.scale = (float)float_arg(scale);
  op.sampling = (int)int_arg(sampling);
  op.aligned = bool_arg(aligned);
  op.order = (int)int_arg(order);
  return op;
}

// affine(ndim, features, rois, out_size, spatial_scale, sampling_ratio, aligned, order)
PyObject* py_affine(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need(n, 8, 8);
  const int ndim = (int)int_arg(a[0]);
  const at::Tensor &features = tensor_arg(a[1], "features"), &rois = tensor_arg(a[2], "rois");
  const RoiOp op = affine_op(ndim, a[3], a[4], a[5], a[6], a[7]);
  if (features.scalar_type() != at::kFloat && features.scalar_type() != at::kHalf)
    raise(PyExc_AssertionError, "input must be float16 or float32 but got torch." + dtype_name(features.scalar_type()));
  if (op.order != 0 && op.order != 1 && op.order != 3)
    raise(PyExc_AssertionError, "order " + std::to_string(op.order) + " is not supported!");
  if (features.dim() != ndim + 2) raise(PyExc_AssertionError, "features must have " + std::to_string(ndim + 2) + " dimensions");
  at::Tensor out;
  {
    pybind11::gil_scoped_release nogil;
    out = affine_forward(op, features, rois);
  }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// affine_label(ndim, labels, rois, out_size, spatial_scale, aligned)
PyObject* py_affine_label(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need(n, 6, 6);
  const int ndim = (int)int_arg(a[0]);
  const at::Tensor &labels = tensor_arg(a[1], "labels"), &rois = tensor_arg(a[2], "rois");
  RoiOp op{};
  op.ndim = ndim;
  op.kind = MVR_ROI_ROTATED;
  op.affine = true;
  out_size_arg(a[3], ndim, "out_size", op);
  op.scale = (float)float_arg(a[4]);
  op.aligned = bool_arg(a[5]);
  if (labels.dim() != ndim + 2) raise(PyExc_AssertionError, "labels must have " + std::to_string(ndim + 2) + " dimensions");
  at::Tensor out;
  {
    pybind11::gil_scoped_release nogil;
    out = label_forward(op, labels, rois);
  }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// label_call(labels, rois, output, out_sizes, spatial_scale, aligned) -> bool: into a caller-allocated int32 tensor
PyObject* py_label_call(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need(n, 6, 6);
  const at::Tensor &labels = tensor_arg(a[0], "input"), &rois = tensor_arg(a[1], "rois"), &out = tensor_arg(a[2], "output");
  RoiOp op{};
  op.ndim = (int)labels.dim() - 2;
  op.kind = MVR_ROI_ROTATED;
  TORCH_CHECK(op.ndim == 2 || op.ndim == 3, "affine_label: expected a 4-D or 5-D label tensor");
  out_size_arg(a[3], op.ndim, "out_sizes", op);
  op.scale = (float)float_arg(a[4]);
  op.aligned = bool_arg(a[5]);
  bool done;
  {
    pybind11::gil_scoped_release nogil;
    at::NoGradGuard no_grad;
    check_label_tensors(op, labels, rois);
    TORCH_CHECK(rois.scalar_type() == at::kFloat && out.scalar_type() == at::kInt, "affine_label: rois must be float32 and the output int32");
    TORCH_CHECK(rois.device() == labels.device() && out.device() == labels.device(), "expected all tensors to be on the same CUDA device");
    const auto want = result_shape(op, rois.size(0), labels.size(1));
    TORCH_CHECK(out.is_contiguous() && out.sizes() == at::IntArrayRef(want), "affine_label: the output must be a contiguous (R, C, *out_size) tensor");
    done = label_into(labels.contiguous(), rois.contiguous(), out, op);
  }
  return PyBool_FromLong(done);
  END_HANDLE_TH_ERRORS
}

// fields_call(image, image_rois, image_out, labels, label_rois, label_out, out_sizes, spatial_scale, aligned, order)
PyObject* py_fields_call(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need(n, 10, 10);
  const at::Tensor &image = tensor_arg(a[0], "image"), &image_rois = tensor_arg(a[1], "image_rois"), &image_out = tensor_arg(a[2], "image_out"),
                   &labels = tensor_arg(a[3], "labels"), &label_rois = tensor_arg(a[4], "label_rois"), &label_out = tensor_arg(a[5], "label_out");
  RoiOp op{};
  op.ndim = 3;
  op.kind = MVR_ROI_ROTATED;
  out_size_arg(a[6], 3, "out_sizes", op);
  op.scale = (float)float_arg(a[7]);
  op.aligned = bool_arg(a[8]);
  op.order = (int)int_arg(a[9]);
  {
    pybind11::gil_scoped_release nogil;
    at::NoGradGuard no_grad;
    TORCH_CHECK(image.is_cuda() && labels.is_cuda(), "RoIAlignRotated is not implemented on CPU");
    TORCH_CHECK(image.dim() == 5 && labels.dim() == 5 && image.size(0) == labels.size(0) && image.sizes().slice(2) == labels.sizes().slice(2),
                "affine_fields_3d: image and labels must be (N, C, D, H, W) over the same volumes");
    const auto t = image.scalar_type();
    TORCH_CHECK(dtype_code(t) >= 0, "\"affine_3d\" not implemented for '", dtype_name(t), "'");
    TORCH_CHECK(label_code(labels.scalar_type()) >= 0 && t != at::kDouble,
                "affine_fields_3d: float16 / float32 image and uint8 / int16 / int32 / int64 labels");
    TORCH_CHECK(image_rois.dim() == 2 && image_rois.size(1) == 10 && label_rois.dim() == 2 && label_rois.size(1) == 10,
                "wrong roi size! size_rois should be 10");
    const int64_t R = image_rois.size(0);
    TORCH_CHECK(label_rois.size(0) == R && image_rois.scalar_type() == t && label_rois.scalar_type() == at::kFloat,
                "affine_fields_3d: rois in the image's dtype for the image and in float32 for the labels");
    for (const at::Tensor* x : {&image_rois, &image_out, &labels, &label_rois, &label_out})
      TORCH_CHECK(x->device() == image.device(), "expected all tensors to be on the same CUDA device");
    TORCH_CHECK(image_out.scalar_type() == t && label_out.scalar_type() == at::kInt, "affine_fields_3d: image_out in the image's dtype, label_out int32");
    TORCH_CHECK(image_out.sizes() == at::IntArrayRef(result_shape(op, R, image.size(1))) &&
                    label_out.sizes() == at::IntArrayRef(result_shape(op, R, labels.size(1))) && image_out.is_contiguous() && label_out.is_contiguous(),
                "affine_fields_3d: the results must be contiguous (R, C, *out_size) tensors");
    TORCH_CHECK(fields_into(op, image.contiguous(), image_rois.contiguous(), image_out, labels.contiguous(), label_rois.contiguous(), label_out),
                mvr_strerror(MVR_ERR_UNSUPPORTED));
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

Tensors tensor_list(PyObject* o, const char* name) {
  if (!PyList_Check(o)) raise(PyExc_TypeError, std::string(name) + " must be a list");
  Tensors v;
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(o); ++i) v.push_back(tensor_arg(PyList_GET_ITEM(o, i), name));
  return v;
}
PyObject* wrap_list(Tensors& v) {
  PyObject* list = PyList_New((Py_ssize_t)v.size());
  if (!list) throw python_error();
  for (size_t i = 0; i < v.size(); ++i) PyList_SET_ITEM(list, (Py_ssize_t)i, THPVariable_Wrap(std::move(v[i])));
  return list;
}

// resample_fields(ndim, images, labels, rois, out_size, sampling_ratio, order) -> (images, labels)
PyObject* py_resample_fields(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need(n, 7, 7);
  RoiOp op{};
  op.ndim = (int)int_arg(a[0]);
  op.kind = MVR_ROI_ROTATED;
  op.affine = true;
  Tensors images = tensor_list(a[1], "images"), labels = tensor_list(a[2], "labels");
  const at::Tensor& rois = tensor_arg(a[3], "rois");
  out_size_arg(a[4], op.ndim, "out_size", op);
  op.scale = 1.0f;
  op.aligned = 1;
  op.sampling = (int)int_arg(a[5]);
  op.order = (int)int_arg(a[6]);
  if (op.order != 0 && op.order != 1 && op.order != 3)
    raise(PyExc_AssertionError, "order " + std::to_string(op.order) + " is not supported!");
  for (const Tensors* v : {&images, &labels})
    for (const at::Tensor& t : *v) {
      if (!t.is_cuda()) raise(PyExc_AssertionError, "image should be cuda");
      if (t.dim() != op.ndim + 2) raise(PyExc_AssertionError, "image should be batch, channel, **dim");
    }
  for (const at::Tensor& t : images)
    if (t.scalar_type() != at::kFloat && t.scalar_type() != at::kHalf)
      raise(PyExc_AssertionError, "input must be float16 or float32 but got torch." + dtype_name(t.scalar_type()));
  TORCH_CHECK(rois.dim() == 2 && rois.size(1) == op.width() && !rois.is_cuda(), "rois: expected a CPU tensor of width ", op.width());
  Tensors images_out, labels_out;
  if (!images.empty() || !labels.empty()) {
    pybind11::gil_scoped_release nogil;
    resample_fields(op, images, labels, rois, images_out, labels_out);
  }
  PyObject* io = wrap_list(images_out);
  PyObject* lo = wrap_list(labels_out);
  PyObject* both = PyTuple_Pack(2, io, lo);
  Py_DECREF(io);
  Py_DECREF(lo);
  return both;
  END_HANDLE_TH_ERRORS
}

BitGen* bitgen_arg(PyObject* capsule) {
  BitGen* g = (BitGen*)PyCapsule_GetPointer(capsule, "BitGenerator");
  if (!g) throw python_error();
  return g;
}

// draw_affine(capsule, n, dim, (scale lo, hi), (shift lo, hi), (rotate lo, hi), scales, shifts, rotate): per sample scale, one
// shift per axis, rotation in degrees; fills float64 arrays (n, dim), (n, dim), (n, 1)
PyObject* py_draw_affine(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  need(n_args, 9, 9);
  BitGen* g = bitgen_arg(a[0]);
  const Py_ssize_t n = int_arg(a[1]), dim = int_arg(a[2]);
  double lo[3], span[3];
  for (int k = 0; k < 3; ++k) {
    lo[k] = float_arg(PyTuple_GET_ITEM(a[3 + k], 0));
    span[k] = float_arg(PyTuple_GET_ITEM(a[3 + k], 1)) - lo[k];
  }
  Buffer scales(a[6], 8, n * dim, true), shifts(a[7], 8, n * dim, true), rotate(a[8], 8, n, true);
  double *sc = scales.as<double>(), *sh = shifts.as<double>(), *ro = rotate.as<double>();
  for (Py_ssize_t i = 0; i < n; ++i) {
    const double s = 1 + (lo[0] + span[0] * g->next_double(g->state));
    for (Py_ssize_t d = 0; d < dim; ++d) sc[i * dim + d] = s;
    for (Py_ssize_t d = 0; d < dim; ++d) sh[i * dim + d] = 0 + (lo[1] + span[1] * g->next_double(g->state));
    ro[i] = 3.141592653589793 * (0 + (lo[2] + span[2] * g->next_double(g->state))) / 180;
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// draw_starts(capsule, n, image_shape, patch_size, start, end): randint(0, image - patch + 1) per patch and axis (d, h, w);
// fills int64 arrays (n, dim) in x, y, z order
PyObject* py_draw_starts(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  need(n_args, 6, 6);
  BitGen* g = bitgen_arg(a[0]);
  const Py_ssize_t n = int_arg(a[1]), dim = PyTuple_GET_SIZE(a[2]);
  if (dim > 3 || PyTuple_GET_SIZE(a[3]) != dim) raise(PyExc_ValueError, "unexpected shape");
  int64_t patch[3];
  uint32_t range[3], mask[3];
  for (Py_ssize_t d = 0; d < dim; ++d) {
    patch[d] = int_arg(PyTuple_GET_ITEM(a[3], d));
    const int64_t room = int_arg(PyTuple_GET_ITEM(a[2], d)) - patch[d];
    if (room < 0 || room >= 0xffffffffll) raise(PyExc_ValueError, "low >= high");
    range[d] = mask[d] = (uint32_t)room;
    for (int s = 1; s < 32; s <<= 1) mask[d] |= mask[d] >> s;
  }
  Buffer start(a[4], 8, n * dim, true), end(a[5], 8, n * dim, true);
  int64_t *st = start.as<int64_t>(), *en = end.as<int64_t>();
  for (Py_ssize_t i = 0; i < n; ++i)
    for (Py_ssize_t d = 0; d < dim; ++d) {
      uint32_t v = 0;
      if (range[d])
        while ((v = g->next_uint32(g->state) & mask[d]) > range[d]) {}
      st[i * dim + dim - 1 - d] = v;
      en[i * dim + dim - 1 - d] = v + patch[d];
    }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// draw_coarse(capsule, batch, grid, reach, border, out): 2 * float32(rand) - 1 times reach per component, the `border`
// outermost points of every axis zero; fills a float32 array (batch, *grid, dim).  reach: float32 array (dim).
PyObject* py_draw_coarse(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  need(n_args, 6, 6);
  BitGen* g = bitgen_arg(a[0]);
  const Py_ssize_t batch = int_arg(a[1]), dim = PyTuple_GET_SIZE(a[2]);
  const int border = (int)int_arg(a[4]);
  if (dim != 2 && dim != 3) raise(PyExc_ValueError, "unexpected shape");
  Py_ssize_t grid[3] = {1, 1, 1}, points = 1;
  for (Py_ssize_t d = 0; d < dim; ++d) points *= grid[3 - dim + d] = int_arg(PyTuple_GET_ITEM(a[2], d));
  Buffer reach(a[3], 4, dim, false), out(a[5], 4, batch * points * dim, true);
  const float* r = reach.as<float>();
  float* o = out.as<float>();
  auto locked = [&](Py_ssize_t i, int axis) { return i < border || i >= grid[axis] - border; };
  for (Py_ssize_t b = 0; b < batch; ++b)
    for (Py_ssize_t z = 0; z < grid[0]; ++z)
      for (Py_ssize_t y = 0; y < grid[1]; ++y) {
        const bool row_locked = (dim == 3 && locked(z, 0)) || locked(y, 1);
        for (Py_ssize_t x = 0; x < grid[2]; ++x) {
          const bool lock = row_locked || locked(x, 2);
          for (Py_ssize_t c = 0; c < dim; ++c) {
            const float u = (float)g->next_double(g->state);
            *o++ = lock ? 0.0f : (2 * u - 1) * r[c];
          }
        }
      }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// affine_rois(n, dim, images, scales, shifts, rotate, image_shape | None, start | None, end | None) -> CPU float32 (n, K):
// [i % images, center - shape * shifts / scales, shape / scales, angles], every step one float32 operation; centre and shape
// are the whole image's or the patch's (start + end) / 2 and end - start
PyObject* py_affine_rois(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  need(n_args, 9, 9);
  const Py_ssize_t n = int_arg(a[0]), dim = int_arg(a[1]), images = int_arg(a[2]);
  if (dim != 2 && dim != 3) raise(PyExc_ValueError, "unexpected shape");
  Buffer scales(a[3], 8, n * dim, false), shifts(a[4], 8, n * dim, false), rotate(a[5], 8, n, false);
  const double *sc = scales.as<double>(), *sh = shifts.as<double>(), *ro = rotate.as<double>();
  const bool whole = a[6] != Py_None;
  float image[3] = {0, 0, 0};
  if (whole)
    for (Py_ssize_t d = 0; d < dim; ++d) image[d] = (float)int_arg(PyTuple_GET_ITEM(a[6], dim - 1 - d));
  std::unique_ptr<Buffer> start, end;
  if (!whole) {
    start.reset(new Buffer(a[7], 8, n * dim, false));
    end.reset(new Buffer(a[8], 8, n * dim, false));
  }
  const Py_ssize_t K = dim == 2 ? 6 : 10;
  at::Tensor out = at::zeros({n, K}, at::kFloat);
  float* o = (float*)out.data_ptr();
  for (Py_ssize_t i = 0; i < n; ++i, o += K) {
    o[0] = (float)(i % images);
    for (Py_ssize_t d = 0; d < dim; ++d) {
      float centre, shape;
      if (whole) {
        shape = image[d];
        centre = shape / 2;
      } else {
        const float s = (float)start->as<int64_t>()[i * dim + d], e = (float)end->as<int64_t>()[i * dim + d];
        centre = (s + e) / 2;
        shape = e - s;
      }
      const float scale = (float)sc[i * dim + d], moved = shape * (float)sh[i * dim + d];
      o[1 + d] = centre - moved / scale;
      o[1 + dim + d] = shape / scale;
    }
    o[K - 1] = (float)ro[i];
  }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// apply_offset(input, offset, order)
PyObject* py_apply_offset(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need(n, 3, 3);
  const at::Tensor &input = tensor_arg(a[0], "input"), &offset = tensor_arg(a[1], "offset");
  const int order = (int)int_arg(a[2]);
  return THPVariable_Wrap(apply_offset(input, offset, order));
  END_HANDLE_TH_ERRORS
}

// elastic(coarse, border, shape, like, images, labels) -> (images, labels), or None where the two-step form is needed;
// elastic(coarse, border, shape, device, None, None) -> the dense field, or None.  `like`: a tensor of the type in which the
// sample positions are formed.
PyObject* py_elastic(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need(n, 6, 6);
  const at::Tensor& coarse = tensor_arg(a[0], "coarse");
  const int border = (int)int_arg(a[1]);
  std::vector<int64_t> shape;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(a[2]); ++i) shape.push_back(int_arg(PyTuple_GET_ITEM(a[2], i)));
  const int ndim = (int)shape.size();
  TORCH_CHECK((ndim == 2 || ndim == 3) && coarse.dim() == ndim + 2 && coarse.size(ndim + 1) == ndim && !coarse.is_cuda() &&
                  coarse.scalar_type() == at::kFloat && coarse.is_contiguous(),
              "coarse: expected a contiguous float32 CPU tensor (B, *grid, dim)");
  const at::Tensor& like = tensor_arg(a[3], "like");
  TORCH_CHECK(like.is_cuda(), "Not implemented on the CPU");
  if (a[4] == Py_None) {
    at::Tensor field;
    Tensors none;
    bool done;
    {
      pybind11::gil_scoped_release nogil;
      done = elastic(coarse, border, shape, at::kFloat, none, none, &field, like.device(), none, none);
    }
    if (!done) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(field));
  }
  Tensors images = tensor_list(a[4], "images"), labels = tensor_list(a[5], "labels");
  for (const Tensors* v : {&images, &labels})
    for (const at::Tensor& t : *v) {
      if (t.dim() != ndim + 2 || t.size(0) != coarse.size(0) || t.sizes().slice(2) != at::IntArrayRef(shape))
        raise(PyExc_AssertionError, "the fields of an elastic deformation must be (B, C, *image_shape)");
      if (t.device() != like.device() || (v == &images ? t.scalar_type() != at::kHalf && t.scalar_type() != at::kFloat : label_code(t.scalar_type()) < 0))
        Py_RETURN_NONE;
    }
  if (like.scalar_type() != at::kHalf && like.scalar_type() != at::kFloat) Py_RETURN_NONE;
  Tensors images_out, labels_out;
  bool done;
  {
    pybind11::gil_scoped_release nogil;
    done = elastic(coarse, border, shape, like.scalar_type(), images, labels, nullptr, like.device(), images_out, labels_out);
  }
  if (!done) Py_RETURN_NONE;
  PyObject* io = wrap_list(images_out);
  PyObject* lo = wrap_list(labels_out);
  PyObject* both = PyTuple_Pack(2, io, lo);
  Py_DECREF(io);
  Py_DECREF(lo);
  return both;
  END_HANDLE_TH_ERRORS
}

// status_word(index): the int32 tensor the kernels of that device OR their status bits into
PyObject* py_status_word(PyObject*, PyObject* index) {
  HANDLE_TH_ERRORS
  return THPVariable_Wrap(status_word((int)int_arg(index)));
  END_HANDLE_TH_ERRORS
}

// peak_allocated(): torch.cuda.max_memory_allocated() of the current device without building its table of statistics
PyObject* py_peak_allocated(PyObject*, PyObject*) {
  HANDLE_TH_ERRORS
  const auto stats = c10::cuda::CUDACachingAllocator::getDeviceStats(c10::cuda::current_device());
  return PyLong_FromLongLong(stats.allocated_bytes[(size_t)c10::CachingAllocator::StatType::AGGREGATE].peak);
  END_HANDLE_TH_ERRORS
}

// release_staging(index): give back the roi upload ring of a device
PyObject* py_release_staging(PyObject*, PyObject* index) {
  HANDLE_TH_ERRORS
  Stage& s = stage_of((int)int_arg(index));
  {
    pybind11::gil_scoped_release nogil;
    free_orphans();
    std::lock_guard<std::mutex> lock(s.mutex);
    s.release();
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

#define FAST(f) (PyCFunction)(void (*)(void)) f, METH_FASTCALL
PyMethodDef methods[] = {
    {"roi_align_2d", FAST((py_roi<2, MVR_ROI_BOX>)), nullptr},
    {"roi_align_3d", FAST((py_roi<3, MVR_ROI_BOX>)), nullptr},
    {"roi_align_rotated_2d", FAST((py_roi<2, MVR_ROI_ROTATED>)), nullptr},
    {"roi_align_rotated_3d", FAST((py_roi<3, MVR_ROI_ROTATED>)), nullptr},
    {"roi_call", FAST(py_roi_call), nullptr},
    {"affine", FAST(py_affine), nullptr},
    {"affine_label", FAST(py_affine_label), nullptr},
    {"label_call", FAST(py_label_call), nullptr},
    {"fields_call", FAST(py_fields_call), nullptr},
    {"resample_fields", FAST(py_resample_fields), nullptr},
    {"draw_affine", FAST(py_draw_affine), nullptr},
    {"draw_starts", FAST(py_draw_starts), nullptr},
    {"draw_coarse", FAST(py_draw_coarse), nullptr},
    {"affine_rois", FAST(py_affine_rois), nullptr},
    {"elastic", FAST(py_elastic), nullptr},
    {"apply_offset", FAST(py_apply_offset), nullptr},
    {"status_word", py_status_word, METH_O, nullptr},
    {"peak_allocated", py_peak_allocated, METH_NOARGS, nullptr},
    {"release_staging", py_release_staging, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
