#include "task_runtime.h"

#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <chrono>
#include <cmath>
#include <deque>
#include <thread>

#include "../common/host_utils.h"
#include "../ops/ops.h"

namespace hipress {
namespace runtime {

TaskRuntime& TaskRuntime::instance() {
  static TaskRuntime* rt = new TaskRuntime();  // leaked: must outlive worker threads at exit
  return *rt;
}

// Nobody waits for the lock with the interpreter lock in hand: whoever holds it may be waiting for workers,
// and they need the interpreter lock to let go of Python tensors.
std::unique_lock<std::mutex> TaskRuntime::life_lock() {
  std::unique_lock<std::mutex> lk(life_mu_, std::try_to_lock);
  if (!lk.owns_lock()) {
    if (PyGILState_Check()) {
      py::gil_scoped_release nogil;
      lk.lock();
    } else {
      lk.lock();
    }
  }
  return lk;
}

bool TaskRuntime::init(const std::string& alg_name, std::unordered_map<std::string, double> params,
                       int device_id, int rank_id, int size) {
  const auto life = life_lock();
  if (pool_) end_locked();
  CompAlg alg;
  alg.name = alg_name;
  int threads = kBackThreads;
  if (alg_name == "terngrad") {
    alg.enable_random = int(params["enable_random"]);
    alg.bitwidth = int(params["bitwidth"]);
  } else if (alg_name == "tbq") {
    alg.threshold = float(params["threshold"]);
    threads = 1;  // ref hp_cuda.cpp:843: tbq runs single-threaded
  } else if (alg_name == "graddrop") {
    alg.drop_ratio = params["drop_ratio"];
    alg.sample_rate = params["sample_rate"];
  } else if (alg_name == "powersgd") {
    alg.matrix_approximation_rank = int(params["matrix_approximation_rank"]);
  } else {
    return false;  // ref hp_cuda.cpp:851-854
  }
  if (params.count("seed")) alg.seed = uint64_t(params["seed"]);
  if (params.count("num_threads")) threads = std::max(1, int(params["num_threads"]));
  alg_ = alg;
  device_id_ = device_id;
  rank_ = rank_id;
  size_ = size;
  serial_ = 0;
  comp_.drain();
  decomp_.drain();
  root_.drain();
  {
    std::lock_guard<std::mutex> lk(err_mu_);
    errors_.clear();
  }
  pool_ = std::make_unique<WorkerPool>(threads, [](int) {}, [this](int, bool wait) { return settle(wait); });
  const double age_limit = params.count("task_age_limit") ? params["task_age_limit"] : 120.0;
  watchdog_ = std::make_unique<AgeWatchdog>(age_limit, [this](const std::string& label, double age) {
    add_error(label + ": still running after " + std::to_string(age) + " s (task age limit)");
  });
  return true;
}

bool TaskRuntime::end() {
  const auto life = life_lock();
  end_locked();
  return true;
}

void TaskRuntime::end_locked() {
  if (pool_) {
    pool_->drain();
    pool_->shutdown();
    pool_.reset();
  }
  watchdog_.reset();
  std::lock_guard<std::mutex> lk(map_mu_);
  gathered_.clear();
}

int TaskRuntime::num_threads() {
  const auto life = life_lock();
  return pool_ ? pool_->size() : 0;
}

int64_t TaskRuntime::graddrop_staging_bytes(int64_t n) const {
  return 4 + int64_t(int(2 * std::ceil(double(n) * (1 - alg_.drop_ratio)))) * 4;
}

FinishQueue& TaskRuntime::queue_for(int task_id) {
  switch (task_id) {
    case kCompTask:
    case kPowerSgdEncode1: return comp_;
    case kDecompTask:
    case kPowerSgdDecode: return decomp_;
    default: return root_;  // 30 and 50 (ref hp_cuda.cpp:1040-1060)
  }
}

std::vector<std::string> TaskRuntime::get_results(int task_id) {
  switch (task_id) {
    case kCompTask: case kPowerSgdEncode1:
    case kDecompTask: case kPowerSgdDecode:
    case kRootDecompCompTask: case kPowerSgdEncode2:
      return queue_for(task_id).drain();
    default:
      return {};
  }
}

std::vector<std::string> TaskRuntime::wait_results(int task_id, double timeout_s, unsigned long long seen) {
  switch (task_id) {
    case kCompTask: case kPowerSgdEncode1:
    case kDecompTask: case kPowerSgdDecode:
    case kRootDecompCompTask: case kPowerSgdEncode2:
      return queue_for(task_id).wait_drain(timeout_s, seen);
    default:   // no task has such an id: nothing will come
      std::this_thread::sleep_for(std::chrono::duration<double>(timeout_s));
      return {};
  }
}

unsigned long long TaskRuntime::error_marks(int task_id) { return queue_for(task_id).wakes(); }

void TaskRuntime::add_error(std::string text) {
  {
    std::lock_guard<std::mutex> lk(err_mu_);
    errors_.push_back(std::move(text));
  }
  comp_.wake();
  decomp_.wake();
  root_.wake();
}

std::vector<std::string> TaskRuntime::get_errors() {
  std::lock_guard<std::mutex> lk(err_mu_);
  std::vector<std::string> out;
  out.swap(errors_);
  return out;
}

namespace {
void check_input(const torch::Tensor& t, const char* name) {
  TORCH_CHECK(t.defined(), name, " is undefined");
  TORCH_CHECK(t.is_contiguous(), name, " must be contiguous");
}
}  // namespace

bool TaskRuntime::submit_without_residual(const std::string& name, torch::Tensor tensor,
                                          torch::Tensor B, torch::Tensor C, int is_root,
                                          int task_id) {
  check_input(tensor, "tensor");
  check_input(B, "B");
  check_input(C, "C");
  if (HP_UNLIKELY(is_root != 0 && is_root != 1)) return false;
  if (task_id != kCompTask && task_id != kDecompTask && task_id != kRootDecompCompTask) return false;
  Task t;
  t.tensor_name = name;
  t.tensor = tensor;
  t.B = B;
  t.C = C;
  t.is_root = is_root;
  t.task_id = task_id;
  return submit(std::move(t));
}

bool TaskRuntime::submit_with_residual(const std::string& name, torch::Tensor tensor,
                                       torch::Tensor residual, torch::Tensor B, torch::Tensor C,
                                       int is_root, int task_id) {
  check_input(tensor, "tensor");
  check_input(residual, "residual");
  check_input(B, "B");
  check_input(C, "C");
  if (HP_UNLIKELY(is_root != 0 && is_root != 1)) return false;
  if (task_id != kCompTask && task_id != kDecompTask && task_id != kRootDecompCompTask) return false;
  Task t;
  t.tensor_name = name;
  t.tensor = tensor;
  t.residual = residual;
  t.B = B;
  t.C = C;
  t.is_root = is_root;
  t.task_id = task_id;
  return submit(std::move(t));
}

bool TaskRuntime::submit_powersgd(const std::string& name, torch::Tensor tensor,
                                  torch::Tensor residual, torch::Tensor M, torch::Tensor P,
                                  torch::Tensor Q, int task_id) {
  check_input(tensor, "tensor");
  check_input(residual, "residual");
  check_input(M, "M");
  check_input(P, "P");
  check_input(Q, "Q");
  if (task_id != kPowerSgdEncode1 && task_id != kPowerSgdEncode2 && task_id != kPowerSgdDecode)
    return false;
  Task t;
  t.tensor_name = name;
  t.tensor = tensor;
  t.residual = residual;
  t.M = M;
  t.P = P;
  t.Q = Q;
  t.task_id = task_id;
  return submit(std::move(t));
}

namespace {
// Tasks of this worker whose kernels and copies are queued on its stream, oldest first.  The worker goes on
// to its next task instead of waiting for each: a copy of one overlaps the kernels of the next.
struct Queued {
  Task task;   // keeps the tensors
  std::unique_ptr<at::cuda::CUDAEvent> done;
};
std::deque<Queued>& queued() {
  thread_local std::deque<Queued> q;
  return q;
}
}  // namespace

// The last owner of a Python tensor needs the interpreter lock, which a worker would have to wait for with
// the next tasks behind it.  The tensors go back to the callers, who hold that lock, before the name is out.
void TaskRuntime::report(Task& t, const std::string& error) {
  const int task_id = t.task_id;
  const std::string name = t.tensor_name;
  watchdog_->done(t.serial);
  {
    std::lock_guard<std::mutex> lk(spent_mu_);
    spent_.push_back(std::move(t));
  }
  if (error.empty()) queue_for(task_id).push(name);
  else add_error(name + ": " + error);
}

void TaskRuntime::release_spent() {
  std::vector<Task> spent;
  std::lock_guard<std::mutex> lk(spent_mu_);
  spent.swap(spent_);
}

// Reports the tasks of this worker that are done: after every task those that the device has finished by
// then, and with `wait` all of them, one by one.  Returns how many are left.
int TaskRuntime::settle(bool wait) {
  std::deque<Queued>& q = queued();
  while (!q.empty()) {
    Queued& first = q.front();
    std::string error;
    try {
      c10::cuda::CUDAGuard dev(first.task.tensor.device());
      if (wait) first.done->synchronize();
      else if (!first.done->query()) break;
    } catch (const std::exception& e) {
      error = e.what();
    }
    report(first.task, error);
    q.pop_front();
  }
  return int(q.size());
}

bool TaskRuntime::submit(Task t) {
  release_spent();
  const auto life = life_lock();
  TORCH_CHECK(pool_ != nullptr && pool_->alive(), "hipress runtime is not initialised (call init first)");
  t.serial = serial_.fetch_add(1);
  // order the worker's stream after whatever the caller has queued so far
  std::shared_ptr<at::cuda::CUDAEvent> ready;
  if (t.tensor.is_cuda()) {
    ready = std::make_shared<at::cuda::CUDAEvent>();
    ready->record(at::cuda::getCurrentCUDAStream(t.tensor.get_device()));
  }
  watchdog_->track(t.serial, t.tensor_name + " (task " + std::to_string(t.task_id) + ")");
  pool_->submit([this, t, ready](int) mutable {
    std::string error;
    try {
      if (t.tensor.is_cuda()) {
        c10::cuda::CUDAGuard dev(t.tensor.device());
        // one high-priority stream per worker thread and device, taken from torch's pool
        thread_local std::unordered_map<int, c10::cuda::CUDAStream> streams;
        const int device = t.tensor.get_device();
        auto it = streams.find(device);
        if (it == streams.end())
          it = streams.emplace(device, c10::cuda::getStreamFromPool(/*isHighPriority=*/true, device)).first;
        c10::cuda::CUDAStream stream = it->second;
        c10::cuda::CUDAStreamGuard sg(stream);
        ready->block(stream);
        // a copy from or to pageable memory holds the worker up: the names before it go out first, and the
        // wait for its own costs nothing
        const bool blocking = t.C.defined() && !t.C.is_cuda() && !t.C.is_pinned();
        if (blocking) settle(true);
        run(t);
        if (blocking) {
          stream.synchronize();
        } else {
          auto done = std::make_unique<at::cuda::CUDAEvent>();
          done->record(stream);
          queued().push_back(Queued{std::move(t), std::move(done)});
          return;
        }
      } else {
        settle(true);   // the CPU codec takes its time: the names before it go out first
        run(t);
      }
    } catch (const std::exception& e) {
      error = e.what();
    }
    report(t, error);
  });
  return true;
}

void TaskRuntime::run(Task& t) {
  switch (t.task_id) {
    case kCompTask: run_compress(t); break;
    case kDecompTask: run_decompress(t); break;
    case kRootDecompCompTask: run_root(t); break;
    default: run_powersgd(t); break;
  }
}

namespace {
// Payloads up to this are stored into pinned host memory by the compressing kernel; larger ones would hold its SMs up
// for longer than the launch of a copy costs.  Four TBQ tasks and back: payloads of 64 KB 148 us, and 161 copied;
// of 1 MB 316 and 351.
constexpr int64_t kDirectBytes = 1 << 20;

uint64_t task_seed(const CompAlg& alg, const Task& t) {
  return alg.seed + 0x9E3779B97F4A7C15ull * (t.serial + 1);
}
// The first `bytes` bytes of `src` to `dst`, on the current stream.  The task keeps both tensors until its copies are
// done, so nothing has to be noted with the allocators, and slices and a dispatched copy, which cost the worker
// more than the copy itself, are only for what is not two plain byte buffers.
void copy_payload(const torch::Tensor& dst, const torch::Tensor& src, int64_t bytes) {
  auto plain = [&](const torch::Tensor& t) { return t.dim() == 1 && t.scalar_type() == torch::kUInt8 && t.is_contiguous(); };
  if (!plain(dst) || !plain(src) || dst.is_cuda() == src.is_cuda()) {
    dst.slice(0, 0, bytes).copy_(src.slice(0, 0, bytes), /*non_blocking=*/true);
    return;
  }
  const auto stream = at::cuda::getCurrentCUDAStream(dst.is_cuda() ? dst.get_device() : src.get_device());
  C10_CUDA_CHECK(cudaMemcpyAsync(dst.data_ptr(), src.data_ptr(), size_t(bytes),
                                 dst.is_cuda() ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, stream));
}

// Where the device sees C, when a payload of that size is stored there by the kernel itself beside its copy in B:
// pinned host memory, and few enough bytes that the SMs are not held up by the bus (see kDirectBytes).
uint8_t* direct_host(const Task& t, int64_t bytes) {
  if (bytes > kDirectBytes || !t.tensor.is_cuda() || t.C.is_cuda() || t.C.dim() != 1 || t.C.scalar_type() != torch::kUInt8 ||
      t.C.numel() < bytes || t.B.numel() < bytes || !t.C.is_pinned())
    return nullptr;
  void* at = nullptr;
  if (cudaHostGetDevicePointer(&at, t.C.data_ptr(), 0) != cudaSuccess) {
    cudaGetLastError();   // not mapped: copied instead
    return nullptr;
  }
  return static_cast<uint8_t*>(at);
}

// bytes of payload a task moves between B and C
int64_t staged_bytes(const TaskRuntime& rt, const Task& t) {
  if (rt.algorithm().name == "graddrop") return rt.graddrop_staging_bytes(t.tensor.numel());
  if (rt.algorithm().name == "tbq") return ops::tbq_payload_bytes(t.tensor.numel());
  return t.B.numel();  // terngrad: B is sized exactly
}
}  // namespace

void TaskRuntime::run_compress(Task& t) {
  const auto& a = alg_;
  auto g = t.tensor.view(-1);
  const int64_t bytes = std::min<int64_t>(staged_bytes(*this, t), std::min(t.B.numel(), t.C.numel()));
  uint8_t* const host = a.name == "graddrop" ? nullptr : direct_host(t, staged_bytes(*this, t));
  if (a.name == "terngrad") {
    ops::terngrad_compress_beside(g, t.B, a.bitwidth, a.enable_random != 0, int64_t(task_seed(a, t)), host);
  } else if (a.name == "tbq") {
    ops::tbq_compress_beside(g, t.residual.view(-1), t.B, a.threshold, host);
  } else if (a.name == "graddrop") {
    ops::sparse_compress(g, t.residual.view(-1), t.B, a.sample_rate, 1.0 - a.drop_ratio,
                         int64_t(task_seed(a, t)), true);
  } else {
    TORCH_CHECK(false, "task ", t.task_id, " is not valid for algorithm ", a.name);
  }
  if (host == nullptr) copy_payload(t.C, t.B, bytes);
}

void TaskRuntime::run_decompress(Task& t) {
  const auto& a = alg_;
  const int64_t bytes = std::min<int64_t>(staged_bytes(*this, t), std::min(t.B.numel(), t.C.numel()));
  copy_payload(t.B, t.C, bytes);
  auto out = t.tensor.view(-1);
  const bool add = t.is_root != 0;  // is_root doubles as "accumulate" (ref hp_cuda.cpp:236, 417, 567)
  if (a.name == "terngrad") {
    ops::terngrad_decompress({t.B}, out, add, 1.0, alg_.bitwidth);
  } else if (a.name == "tbq") {
    ops::tbq_decompress({t.B}, out, a.threshold, add, 1.0);
  } else if (a.name == "graddrop") {
    ops::sparse_decompress_beside(t.B.slice(0, 0, bytes), out, add);
  } else {
    TORCH_CHECK(false, "task ", t.task_id, " is not valid for algorithm ", a.name);
  }
}

void TaskRuntime::run_root(Task& t) {
  // C holds `size` payload slices of equal length, slice r from rank r.  All
  // slices but this rank's own are decoded into the dense tensor one after
  // another in ascending rank order -- the reference's order of accumulation,
  // own tensor first -- then the dense tensor is compressed into B and copied
  // to C[0:len]  (ref hp_cuda.cpp:241-271, 421-449, 571-601).
  const auto& a = alg_;
  const int64_t len = (a.name == "terngrad") ? t.B.numel() : staged_bytes(*this, t);
  TORCH_CHECK(t.C.numel() >= len * size_, "gathered buffer C holds fewer than size x payload bytes");
  torch::Tensor gathered;
  if (t.tensor.is_cuda() && !t.C.is_cuda()) {
    std::lock_guard<std::mutex> lk(map_mu_);
    auto it = gathered_.find(t.tensor_name);
    if (it == gathered_.end() || it->second.numel() != t.C.numel())
      it = gathered_.insert_or_assign(t.tensor_name, torch::empty_like(t.C, t.tensor.options().dtype(torch::kUInt8))).first;
    gathered = it->second;
    gathered.copy_(t.C, /*non_blocking=*/true);
  } else {
    gathered = t.C;
  }
  std::vector<torch::Tensor> peers;
  for (int r = 0; r < size_; ++r)
    if (r != rank_) peers.push_back(gathered.slice(0, int64_t(r) * len, int64_t(r + 1) * len));
  auto out = t.tensor.view(-1);
  const bool add = t.is_root != 0;
  for (size_t i = 0; i < peers.size(); ++i) {
    // the first peer overwrites unless the task accumulates; every later one adds
    const bool add_to = add || i > 0;
    if (a.name == "terngrad") ops::terngrad_decompress({peers[i]}, out, add_to, 1.0, alg_.bitwidth);
    else if (a.name == "tbq") ops::tbq_decompress({peers[i]}, out, a.threshold, add_to, 1.0);
    else if (a.name == "graddrop") ops::sparse_decompress_beside(peers[i], out, add_to);
    else TORCH_CHECK(false, "task 30 is not valid for algorithm ", a.name);
  }
  run_compress(t);
}

void TaskRuntime::run_powersgd(Task& t) {
  TORCH_CHECK(alg_.name == "powersgd", "task ", t.task_id, " needs algorithm powersgd");
  switch (t.task_id) {
    case kPowerSgdEncode1: ops::powersgd_encode1(t.tensor, t.residual, t.Q, t.M, t.P); break;
    case kPowerSgdEncode2: ops::powersgd_encode2(t.P, t.M, t.Q); break;
    default: ops::powersgd_decode(t.P, t.Q, t.M, t.residual, t.tensor); break;
  }
}

}  // namespace runtime
}  // namespace hipress
