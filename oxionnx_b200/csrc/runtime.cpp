// Context, weight residency, arena planning and the run loop of the oxb200 provider.
// The per-operator planning rules live in planner.cpp.
#include "runtime.hpp"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <condition_variable>
#include <cstring>
#include <thread>

namespace oxb {

std::vector<std::string> AttrMap::names() const {
  std::vector<std::string> out;
  for (auto& kv : ints) out.push_back(kv.first);
  for (auto& kv : floats) out.push_back(kv.first);
  for (auto& kv : strings) out.push_back(kv.first);
  for (auto& kv : int_lists) out.push_back(kv.first);
  for (auto& kv : float_lists) out.push_back(kv.first);
  return out;
}

// ---------------------------------------------------------------------------------------
// Context
// ---------------------------------------------------------------------------------------
Context::Context(int device, const oxb200_config& cfg) : device_(device), cfg_(cfg) {
  int count = 0;
  cudaError_t e = cudaGetDeviceCount(&count);
  if (e != cudaSuccess || count <= 0) {
    (void)cudaGetLastError();
    raise(OXB200_FAILED, "no CUDA device is available (%s); this provider has no CPU path", e == cudaSuccess ? "device count is 0" : cudaGetErrorString(e));
  }
  if (device < 0 || device >= count) raise(OXB200_FAILED, "device ordinal %d out of range (%d devices)", device, count);
  OXB_CUDA(cudaSetDevice(device));
  cudaDeviceProp prop;
  OXB_CUDA(cudaGetDeviceProperties(&prop, device));
  if (prop.major != 10) raise(OXB200_FAILED, "device %d is sm_%d%d; this library carries sm_100a code only", device, prop.major, prop.minor);
  OXB_CUDA(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
}

Context::~Context() {
  cudaSetDevice(device_);
  session.reset();
  release_caches();
  if (run_ev0) cudaEventDestroy(run_ev0);
  if (run_ev1) cudaEventDestroy(run_ev1);
  if (error_words_) cudaFreeHost(error_words_);
  if (stream_) cudaStreamDestroy(stream_);
}

void Context::make_current() { OXB_CUDA(cudaSetDevice(device_)); }

void Context::register_weight(const std::string& name, const float* lanes, uint64_t len, const uint64_t* shape, uint32_t rank, DT declared) {
  HostTensor t;
  t.declared = declared;
  t.shape.assign(shape, shape + rank);
  if ((uint64_t)prod(t.shape) != len) raise(OXB200_FAILED, "weight '%s': %llu lanes do not match its shape", name.c_str(), (unsigned long long)len);
  t.data.assign(lanes, lanes + len);
  weights_[name] = std::move(t);
  drop_dispatch_plans();
  // a re-registered weight invalidates its packed forms
  for (auto it = forms_.begin(); it != forms_.end();) {
    if (it->first.first == name) {
      cudaFree(it->second.ptr);
      counters.weight_bytes_resident -= it->second.bytes;
      it = forms_.erase(it);
    } else {
      ++it;
    }
  }
  resident_names_.erase(name);
}

const HostTensor* Context::weight(const std::string& name) const {
  auto it = weights_.find(name);
  return it == weights_.end() ? nullptr : &it->second;
}

bool Context::weight_resident(const std::string& name) const { return resident_names_.count(name) != 0; }

// Memory that this context only holds for reuse is given back before an allocation fails: first the free blocks, then the
// kept plans but the one in use.
void* Context::try_alloc_device(size_t bytes, cudaError_t* error) {
  void* p = nullptr;
  bytes = align_up(std::max<size_t>(bytes, 256), 256);
  cudaError_t e = cudaMalloc(&p, bytes);
  if (e == cudaErrorMemoryAllocation && drop_free_blocks()) {
    (void)cudaGetLastError();
    e = cudaMalloc(&p, bytes);
  }
  if (e == cudaErrorMemoryAllocation && drop_dispatch_plans()) {
    (void)cudaGetLastError();
    e = cudaMalloc(&p, bytes);
  }
  if (error) *error = e;
  if (e == cudaSuccess) return p;
  (void)cudaGetLastError();
  return nullptr;
}

void* Context::alloc_device(size_t bytes) {
  cudaError_t e = cudaSuccess;
  void* p = try_alloc_device(bytes, &e);
  OXB_CUDA(e);
  return p;
}

void Context::free_device(void* p) {
  if (p) cudaFree(p);
}

void* Context::resident_form(const std::string& name, const std::string& form, size_t bytes, const std::function<void(void*)>& fill_host,
                             bool cacheable) {
  auto key = std::make_pair(name, form);
  if (cacheable) {
    auto it = forms_.find(key);
    if (it != forms_.end() && it->second.bytes == bytes) return it->second.ptr;
  }
  std::vector<uint8_t> host(std::max<size_t>(bytes, 16), 0);
  fill_host(host.data());
  void* dev = alloc_device(bytes);
  OXB_CUDA(cudaMemcpyAsync(dev, host.data(), bytes, cudaMemcpyHostToDevice, stream_));
  OXB_CUDA(cudaStreamSynchronize(stream_));
  if (cacheable) {
    counters.weight_uploads += 1;
    forms_[key] = DeviceBuffer{dev, bytes};
    counters.weight_bytes_resident += bytes;
    resident_names_.insert(name);
  } else {
    // an operand of a one-node dispatch: activation traffic, not a resident weight
    counters.uploads += 1;
    counters.upload_bytes += bytes;
    temp_forms_.push_back(dev);
  }
  return dev;
}

void Context::free_temp_forms() {
  for (void* p : temp_forms_) cudaFree(p);
  temp_forms_.clear();
}

uint64_t Context::cached_bytes() const {
  uint64_t total = 0;
  for (const auto& kv : forms_) total += kv.second.bytes;
  return total;
}

constexpr size_t kDispatchPlans = 16, kDispatchPlanBytes = 256ull << 20;

Session* Context::find_dispatch_plan(const std::string& key) {
  for (DispatchEntry& e : dispatch_plans_)
    if (e.key == key) {
      e.used = ++dispatch_clock_;
      return e.plan.get();
    }
  return nullptr;
}

Session* Context::keep_dispatch_plan(const std::string& key, std::unique_ptr<Session>& plan) {
  const size_t bytes = plan->device_bytes();
  if (bytes > kDispatchPlanBytes / 4) return nullptr;
  while (!dispatch_plans_.empty()) {
    size_t total = bytes, oldest = 0;
    for (size_t i = 0; i < dispatch_plans_.size(); ++i) {
      total += dispatch_plans_[i].bytes;
      if (dispatch_plans_[i].used < dispatch_plans_[oldest].used) oldest = i;
    }
    if (total <= kDispatchPlanBytes && dispatch_plans_.size() < kDispatchPlans) break;
    dispatch_plans_.erase(dispatch_plans_.begin() + oldest);
  }
  DispatchEntry e;
  e.key = key, e.bytes = bytes, e.used = ++dispatch_clock_;
  e.plan = std::move(plan);
  dispatch_plans_.push_back(std::move(e));
  return dispatch_plans_.back().plan.get();
}

bool Context::drop_dispatch_plans() {
  const size_t before = dispatch_plans_.size();
  dispatch_plans_.erase(std::remove_if(dispatch_plans_.begin(), dispatch_plans_.end(), [&](const DispatchEntry& e) { return e.plan.get() != plan_in_use; }),
                        dispatch_plans_.end());
  return dispatch_plans_.size() != before;
}

constexpr size_t kFreeBlocks = 64, kFreeBlockBytes = 256ull << 20;

void* Context::take_block(size_t bytes, size_t* got) {
  bytes = align_up(std::max<size_t>(bytes, 256), 256);
  size_t best = free_blocks_.size();
  for (size_t i = 0; i < free_blocks_.size(); ++i)
    if (free_blocks_[i].bytes >= bytes && free_blocks_[i].bytes <= bytes + bytes / 4 && (best == free_blocks_.size() || free_blocks_[i].bytes < free_blocks_[best].bytes)) best = i;
  if (best < free_blocks_.size()) {
    const Block b = free_blocks_[best];
    free_blocks_.erase(free_blocks_.begin() + best);
    free_block_bytes_ -= b.bytes;
    *got = b.bytes;
    return b.ptr;
  }
  *got = bytes;
  return alloc_device(bytes);
}

void Context::give_block(void* ptr, size_t bytes) {
  if (free_blocks_.size() >= kFreeBlocks || free_block_bytes_ + bytes > kFreeBlockBytes) {
    cudaFree(ptr);  // waits for whatever still uses it
    return;
  }
  free_blocks_.push_back(Block{ptr, bytes});
  free_block_bytes_ += bytes;
}

bool Context::drop_free_blocks() {
  if (free_blocks_.empty()) return false;
  for (const Block& b : free_blocks_) cudaFree(b.ptr);
  free_blocks_.clear();
  free_block_bytes_ = 0;
  return true;
}

void Context::release_caches() {
  drop_dispatch_plans();
  drop_free_blocks();
  for (auto& kv : forms_) cudaFree(kv.second.ptr);
  forms_.clear();
  for (void* p : temp_forms_) cudaFree(p);
  temp_forms_.clear();
  resident_names_.clear();
  counters.weight_bytes_resident = 0;
  mover_.reset();
}

constexpr int kErrorWords = 64;

int* Context::take_error_word() {
  if (!error_words_) {
    OXB_CUDA(cudaMallocHost(&error_words_, kErrorWords * 64));
    for (int i = kErrorWords - 1; i >= 0; --i) free_error_words_.push_back(error_words_ + i * 16);
  }
  if (free_error_words_.empty()) raise(OXB200_FAILED, "more than %d plans are alive on one context", kErrorWords);
  int* w = free_error_words_.back();
  free_error_words_.pop_back();
  *w = 0;
  return w;
}

void Context::give_error_word(int* word) {
  if (word) free_error_words_.push_back(word);
}

bool host_pinned(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

// A cudaMemcpyAsync from pageable memory is staged by one thread of the driver (16 GB/s here; four lanes reach 35).
// The lanes' threads are kept: a fresh thread pays 100 us for its first CUDA call.  Pieces are handed out one by one,
// so the calling thread starts at once and a lane that wakes late costs nothing; 512 KB keeps a lane's two buffers
// inside a core's L2 and the pipeline's fill and drain short.
constexpr size_t kPiece = 512 << 10;
constexpr int kMoveLanes = 4;

struct MoveJob {
  uint8_t* dst;
  const uint8_t* src;
  size_t bytes;
  int64_t pieces;
  cudaStream_t stream;
  bool to_device;
  std::atomic<int64_t> next{0};
  std::atomic<int> failed{0};
};

struct MovePool {
  struct Lane {
    uint8_t* buf[2] = {nullptr, nullptr};
    cudaEvent_t done[2] = {nullptr, nullptr};
  };
  Lane lanes[kMoveLanes];
  std::vector<std::thread> threads;  // lanes 1 .. ; lane 0 is the calling thread's
  std::mutex mu;
  std::condition_variable wake, idle;
  MoveJob* job = nullptr;
  uint64_t generation = 0;
  int busy = 0;
  bool stop = false;
  const int device;

  explicit MovePool(int device_) : device(device_) {
    try {
      for (Lane& l : lanes)
        for (int b = 0; b < 2; ++b) {
          OXB_CUDA(cudaMallocHost(&l.buf[b], kPiece));
          OXB_CUDA(cudaEventCreateWithFlags(&l.done[b], cudaEventDisableTiming));
        }
      for (int t = 1; t < kMoveLanes; ++t) threads.emplace_back([this, t] { serve(t); });
    } catch (...) {
      close();
      throw;
    }
  }
  ~MovePool() { close(); }

  void close() {
    {
      std::lock_guard<std::mutex> lock(mu);
      stop = true;
    }
    wake.notify_all();
    for (auto& t : threads) t.join();
    threads.clear();
    for (Lane& l : lanes)
      for (int b = 0; b < 2; ++b) {
        if (l.done[b]) {
          cudaEventSynchronize(l.done[b]);
          cudaEventDestroy(l.done[b]);
        }
        if (l.buf[b]) cudaFreeHost(l.buf[b]);
        l.done[b] = nullptr, l.buf[b] = nullptr;
      }
  }

  static void work(Lane& l, MoveJob& j) {
    auto check = [&](cudaError_t e) {
      if (e != cudaSuccess) j.failed.store((int)e);
      return e == cudaSuccess;
    };
    auto at = [&](int64_t i) { return (size_t)i * kPiece; };
    auto len = [&](int64_t i) { return std::min(kPiece, j.bytes - at(i)); };
    int b = 0;
    int64_t behind = -1;  // the piece whose lanes are on their way into the other buffer (device to host)
    for (int64_t i; (i = j.next.fetch_add(1)) < j.pieces; b ^= 1) {
      if (j.to_device) {
        if (!check(cudaEventSynchronize(l.done[b]))) return;
        std::memcpy(l.buf[b], j.src + at(i), len(i));
        if (!check(cudaMemcpyAsync(j.dst + at(i), l.buf[b], len(i), cudaMemcpyHostToDevice, j.stream)) || !check(cudaEventRecord(l.done[b], j.stream))) return;
        continue;
      }
      if (!check(cudaMemcpyAsync(l.buf[b], j.src + at(i), len(i), cudaMemcpyDeviceToHost, j.stream)) || !check(cudaEventRecord(l.done[b], j.stream))) return;
      if (behind >= 0) {
        if (!check(cudaEventSynchronize(l.done[b ^ 1]))) return;
        std::memcpy(j.dst + at(behind), l.buf[b ^ 1], len(behind));
      }
      behind = i;
    }
    if (behind >= 0 && check(cudaEventSynchronize(l.done[b ^ 1]))) std::memcpy(j.dst + at(behind), l.buf[b ^ 1], len(behind));
  }

  void serve(int lane) {
    cudaSetDevice(device);
    uint64_t seen = 0;
    std::unique_lock<std::mutex> lock(mu);
    while (true) {
      wake.wait(lock, [&] { return stop || (job && generation != seen); });
      if (stop) return;
      seen = generation;
      MoveJob* j = job;
      ++busy;
      lock.unlock();
      work(lanes[lane], *j);
      lock.lock();
      if (--busy == 0) idle.notify_all();
    }
  }

  // One mover at a time: a context's calls hold its lock.
  void run(MoveJob& j) {
    {
      std::lock_guard<std::mutex> lock(mu);
      job = &j;
      ++generation;
    }
    if (j.pieces > 2) wake.notify_all();
    work(lanes[0], j);
    std::unique_lock<std::mutex> lock(mu);
    job = nullptr;  // a lane that has not woken by now finds nothing to do
    idle.wait(lock, [&] { return busy == 0; });
  }
};

void Context::move_pieces(void* dst, const void* src, size_t bytes, cudaStream_t s, bool to_device) {
  if (!mover_) mover_ = std::make_shared<MovePool>(device_);
  MoveJob j;
  j.dst = (uint8_t*)dst, j.src = (const uint8_t*)src, j.bytes = bytes;
  j.pieces = (int64_t)((bytes + kPiece - 1) / kPiece);
  j.stream = s, j.to_device = to_device;
  mover_->run(j);
  if (j.failed.load() != 0) raise(OXB200_FAILED, "CUDA error %s while moving host lanes", cudaGetErrorName((cudaError_t)j.failed.load()));
}

void Context::host_to_device(void* dst, const void* src, size_t bytes, cudaStream_t s) { move_pieces(dst, src, bytes, s, true); }
void Context::device_to_host(void* dst, const void* src, size_t bytes, cudaStream_t s) { move_pieces(dst, src, bytes, s, false); }

// ---------------------------------------------------------------------------------------
// Session: arena layout, upload, run, download
// ---------------------------------------------------------------------------------------
Session::~Session() {
  cudaSetDevice(ctx_->device());
  cudaStreamSynchronize(ctx_->stream());
  for (auto* p : umma_plans_) k::umma_plan_destroy(p);
  for (auto* g : umma_groups_) k::umma_group_destroy(g);
  for (auto* c : umma_chains_) k::umma_chain_destroy(c);
  for (auto* a : umma_attentions_) k::umma_attention_destroy(a);
  for (auto& s : steps_) {
    if (s.ev0) cudaEventDestroy(s.ev0);
    if (s.ev1) cudaEventDestroy(s.ev1);
  }
  if (arena_.ptr) cudaFree(arena_.ptr);
  for (auto& b : owned_) cudaFree(b.ptr);
  ctx_->give_error_word(err_flag_);
  if (small_stage_) cudaFreeHost(small_stage_);
  for (int f = 0; f < 2; ++f) {
    Flight& fl = flight_[f];
    if (fl.up) cudaEventDestroy(fl.up);
    if (fl.done) cudaEventDestroy(fl.done);
    if (fl.down) cudaEventDestroy(fl.down);
    if (f == 1 && pipe_double_)
      for (void* p : fl.in_dev) cudaFree(p);
    for (float* p : fl.out_host) cudaFreeHost(p);
    for (void* p : fl.out_dev) cudaFree(p);
  }
  if (copy_stream_) cudaStreamDestroy(copy_stream_);
  if (down_stream_) cudaStreamDestroy(down_stream_);
  for (auto& g : graphs_)
    if (g.exec) cudaGraphExecDestroy(g.exec);
}

Value* Session::find_value(const std::string& name) {
  auto it = index_.find(name);
  return it == index_.end() ? nullptr : &values_[it->second];
}

void Session::sync() {
  const cudaError_t e = cudaStreamSynchronize(ctx_->stream());
  small_stage_used_ = 0;
  std::vector<PendingCopy> out;
  out.swap(pending_out_);
  OXB_CUDA(e);
  for (const PendingCopy& c : out) std::memcpy(c.dst, c.src, c.bytes);
  out.clear();
  pending_out_.swap(out);  // keeps the allocation
  ctx_->counters.fences += 1;
}

// The error word lives in page-locked memory: a kernel that gives up writes it across PCIe, and after the run's fence
// the host reads it like any other word (a copy of it out of device memory was a second fence per run, 10 us).
int Session::check_error_flag() {
  const int flag = *(volatile int*)err_flag_;
  if (flag != 0) {
    *(volatile int*)err_flag_ = 0;
    for (auto* p : umma_plans_) k::umma_plan_reset_after_error(p);
    for (auto* c : umma_chains_) k::umma_chain_reset_after_error(c);
  }
  return flag;
}

// The host lanes of a feed for graph input `v`, checked against the plan: f32 lanes for an input declared f32, typed
// lanes of the declared type otherwise.
static const void* feed_lanes(const oxb200_operand& f, const Value& v, const char* name) {
  if ((int64_t)f.len != v.numel()) raise(OXB200_FAILED, "run: feed '%s' has %llu lanes, the plan expects %lld", name, (unsigned long long)f.len, (long long)v.numel());
  if (f.rank != v.shape.size()) raise(OXB200_FAILED, "run: feed '%s' rank differs from the planned shape", name);
  for (uint32_t d = 0; d < f.rank; ++d)
    if ((int64_t)f.shape[d] != v.shape[d]) raise(OXB200_FAILED, "run: feed '%s' shape differs from the planned shape", name);
  if (v.dt == DT::F32) {
    if (f.lanes) return f.lanes;
    if (f.typed && f.dtype == OXB200_DT_F32) return f.typed;
    raise(OXB200_FAILED, "run: feed '%s' has no f32 host lanes", name);
  }
  if (!f.typed || f.dtype != (int32_t)v.dt)
    raise(OXB200_FAILED, "run: graph input '%s' was declared %s; its feed must carry typed lanes of that type", name, dt_name(v.dt));
  return f.typed;
}

// A run that failed half way leaves copies in the staging memory that nobody will collect.
void Session::begin_copies() {
  if (small_stage_used_ == 0 && pending_out_.empty()) return;
  pending_out_.clear();
  OXB_CUDA(cudaStreamSynchronize(ctx_->stream()));
  small_stage_used_ = 0;
}

void Session::upload(const oxb200_operand* feeds, uint32_t n) {
  begin_copies();
  for (auto& in : input_staging_) {
    const oxb200_operand* f = nullptr;
    for (uint32_t i = 0; i < n; ++i)
      if (feeds[i].name && in.first == feeds[i].name) f = &feeds[i];
    if (!f) raise(OXB200_FAILED, "run: no feed for graph input '%s'", in.first.c_str());
    Value& v = values_[in.second];
    if (external_bind_.count(in.first)) continue;  // bound to a value that already lives on the device
    const void* src = feed_lanes(*f, v, in.first.c_str());
    stage_in(v.ptr, src, (size_t)v.numel() * dt_size(v.dt));
    ctx_->counters.uploads += 1;
    ctx_->counters.upload_bytes += (uint64_t)v.numel() * dt_size(v.dt);
  }
}

// Feeds and fetches up to this size go through the session's own staging memory with one host copy, and between that and
// the device by a kernel of the stream (copy_bytes); above it a
// pageable buffer is moved in pieces by several threads (Context::move_pieces).
constexpr size_t kSmallCopy = 256 * 1024;
// Between the two the driver's own staging of an upload is the faster one (3 MB: 0.16 ms less than the lanes, 10 MB:
// 0.17 ms less; 20 MB: 0.3 ms more, 38 MB: 1.6 ms more).  A download is always better off in pieces (8 MB: 0.9 ms less).
constexpr size_t kLanesUpload = 16 << 20;

// The next `bytes` of the staging memory of the run being assembled, or nullptr when they do not fit.
void* Session::small_stage(size_t bytes) {
  if (!small_stage_) {
    size_t total = 0;
    for (const auto* list : {&input_staging_, &output_staging_})
      for (const auto& io : *list) {
        const size_t n = (size_t)values_[io.second].numel() * 4;
        if (n <= kSmallCopy) total += align_up(n, 64);
      }
    if (total == 0) return nullptr;
    OXB_CUDA(cudaMallocHost(&small_stage_, total));
    small_stage_bytes_ = total;
  }
  bytes = align_up(bytes, 64);
  if (small_stage_used_ + bytes > small_stage_bytes_) return nullptr;
  void* p = small_stage_ + small_stage_used_;
  small_stage_used_ += bytes;
  return p;
}

void Session::stage_in(void* dst, const void* src, size_t bytes) {
  if (bytes == 0) return;
  if (bytes <= kSmallCopy) {
    if (void* st = small_stage(bytes)) {
      std::memcpy(st, src, bytes);
      k::copy_bytes(dst, st, bytes, ctx_->stream());
      return;
    }
  } else if (bytes >= kLanesUpload && !host_pinned(src)) {
    ctx_->host_to_device(dst, src, bytes, ctx_->stream());
    return;
  }
  OXB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx_->stream()));
}

// Enqueues (or, for a large pageable destination, performs) the copy of an output; sync() hands the staged ones over.
void Session::stage_out(void* dst, const void* src, size_t bytes) {
  if (bytes == 0) return;
  if (bytes <= kSmallCopy) {
    if (void* st = small_stage(bytes)) {
      pending_out_.push_back(PendingCopy{dst, st, bytes});
      k::copy_bytes(st, src, bytes, ctx_->stream());
      return;
    }
  } else if (!host_pinned(dst)) {
    ctx_->device_to_host(dst, src, bytes, ctx_->stream());
    return;
  }
  OXB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, ctx_->stream()));
}

bool Session::capture_graph(GraphSlot& g) {
  cudaStream_t s = ctx_->stream();
  const oxb200_counters before = ctx_->counters;
  if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  bool ok = true;
  try {
    for (auto& st : steps_) st.launch(s);
  } catch (...) {
    ok = false;
  }
  cudaGraph_t graph = nullptr;
  if (cudaStreamEndCapture(s, &graph) != cudaSuccess || !graph) ok = false;
  if (ok && cudaGraphInstantiate(&g.exec, graph, 0) != cudaSuccess) ok = false;
  if (graph) cudaGraphDestroy(graph);
  (void)cudaGetLastError();
  // a recording executes nothing: the counters go back, and each replay adds what it stands for
  g.d_kernel = ctx_->counters.kernel_launches - before.kernel_launches;
  g.d_umma = ctx_->counters.umma_launches - before.umma_launches;
  g.d_simt = ctx_->counters.simt_launches - before.simt_launches;
  g.d_glue = ctx_->counters.glue_launches - before.glue_launches;
  ctx_->counters = before;
  if (!ok) {
    if (g.exec) cudaGraphExecDestroy(g.exec);
    g.exec = nullptr;
  }
  return ok;
}

bool Session::replay_graph() {
  std::vector<void*> key;
  for (auto& in : input_staging_) key.push_back(values_[in.second].ptr);
  GraphSlot* g = nullptr;
  for (auto& c : graphs_)
    if (c.key == key) g = &c;
  if (!g) {
    if (graphs_.size() >= 4) return false;  // more input buffers than the pipeline ever rotates through
    graphs_.push_back(GraphSlot{});
    g = &graphs_.back();
    g->key = key;
  }
  if (g->poisoned) return false;
  if (!g->exec) {
    // the first run on these addresses goes the ordinary way: it sets the kernels' one-time attributes
    if (!g->warmed) {
      g->warmed = true;
      return false;
    }
    if (!capture_graph(*g)) {
      g->poisoned = true;
      ctx_->counters.graph_poisoned += 1;
      return false;
    }
    ctx_->counters.graph_captures += 1;
  }
  OXB_CUDA(cudaGraphLaunch(g->exec, ctx_->stream()));
  ctx_->counters.graph_replays += 1;
  ctx_->counters.kernel_launches += g->d_kernel;
  ctx_->counters.umma_launches += g->d_umma;
  ctx_->counters.simt_launches += g->d_simt;
  ctx_->counters.glue_launches += g->d_glue;
  for (auto& st : steps_) st.launches += 1;
  return true;
}

void Session::run_steps(bool profile) {
  cudaStream_t s = ctx_->stream();
  if (graph_allowed_ && !profile && ctx_->cfg().cuda_graph && !ctx_->cfg().verify && replay_graph()) return;
  for (auto& st : steps_) {
    if (profile) {
      if (!st.ev0) {
        OXB_CUDA(cudaEventCreate(&st.ev0));
        OXB_CUDA(cudaEventCreate(&st.ev1));
      }
      OXB_CUDA(cudaEventRecord(st.ev0, s));
    }
    st.launch(s);
    st.launches += 1;
    if (profile) OXB_CUDA(cudaEventRecord(st.ev1, s));
  }
  OXB_CUDA(cudaGetLastError());
}

static void write_result_shape(const Value& v, oxb200_result* r) {
  r->rank = (uint32_t)v.shape.size();
  for (size_t d = 0; d < v.shape.size() && d < OXB200_MAX_RANK; ++d) r->shape[d] = (uint64_t)v.shape[d];
  r->len = (uint64_t)v.numel();
}

void Session::download(oxb200_result* fetches, uint32_t n) {
  begin_copies();
  download_async(fetches, n);
  finish_download();
}

void Session::finish_download() {
  sync();
  int flag = check_error_flag();
  if (flag)
    raise(OXB200_FAILED, flag == 20 ? "Gather: an index is out of range (device code %d); results are not valid" : "a tensor-core kernel gave up on a bounded wait (code %d); results are not valid", flag);
}

void Session::download_async(oxb200_result* fetches, uint32_t n) {
  if (n != outputs_.size()) raise(OXB200_FAILED, "run: %u fetch slots for %zu graph outputs", n, outputs_.size());
  // validate everything first, then copy: a rejected write leaves the caller's buffers untouched
  // (write_node_outputs, root crate src/session/run/dispatch.rs:335-455)
  for (uint32_t i = 0; i < n; ++i) {
    const Value& v = values_[output_staging_[i].second];
    if (fetches[i].lanes && fetches[i].cap < (uint64_t)v.numel())
      raise(OXB200_FAILED, "run: fetch buffer for '%s' holds %llu lanes, %lld needed", outputs_[i].c_str(), (unsigned long long)fetches[i].cap, (long long)v.numel());
  }
  for (uint32_t i = 0; i < n; ++i) {
    const Value& v = values_[output_staging_[i].second];
    write_result_shape(v, &fetches[i]);
    if (fetches[i].lanes && v.numel() > 0) {
      stage_out(fetches[i].lanes, v.ptr, (size_t)v.numel() * 4);
      ctx_->counters.downloads += 1;
      ctx_->counters.download_bytes += (uint64_t)v.numel() * 4;
    }
  }
}

void Session::fetch_value(const std::string& name, oxb200_result* out) {
  Value* v = find_value(name);
  if (!v) raise(OXB200_FAILED, "fetch_value: '%s' is not a value of the planned graph", name.c_str());
  if (!v->ptr) raise(OXB200_FAILED, "fetch_value: '%s' has no device storage (fused away)", name.c_str());
  write_result_shape(*v, out);
  if (!out->lanes) return;
  if (out->cap < (uint64_t)v->numel()) raise(OXB200_FAILED, "fetch_value: buffer too small for '%s'", name.c_str());
  int64_t n = v->numel();
  if (n == 0) return;
  // convert to f32 lanes in the logical order through a temporary
  void* tmp = ctx_->alloc_device((size_t)n * 4);
  k::Dims4 d{1, 1, 1, 1};
  if (v->shape.size() == 4) d = k::Dims4{v->shape[0], v->shape[1], v->shape[2], v->shape[3]};
  else d = k::Dims4{n, 1, 1, 1};
  k::TensorRef src{v->ptr, v->dt, v->shape.size() == 4 ? v->layout : Layout::PLAIN, d};
  k::TensorRef dst{tmp, DT::F32, Layout::PLAIN, d};
  const Value* root = v;
  while (root->alias_of >= 0) root = &values_[root->alias_of];
  if (root->out_seq > 0) {  // f32 rows that their linear left transposed within sequences: [sequence][channel][row]
    const int64_t seq = root->out_seq, ch = root->shape.back();
    k::transpose_perm(v->ptr, tmp, k::Dims4{1, n / (seq * ch), seq, ch}, k::Dims4{0, seq * ch, 1, seq}, ctx_->stream());
  } else {
    k::convert(src, dst, ctx_->stream());
  }
  OXB_CUDA(cudaMemcpyAsync(out->lanes, tmp, (size_t)n * 4, cudaMemcpyDeviceToHost, ctx_->stream()));
  sync();
  ctx_->free_device(tmp);
  ctx_->counters.downloads += 1;
  ctx_->counters.download_bytes += (uint64_t)n * 4;
}

// ---- pipelined runs ---------------------------------------------------------------------------
void Session::rebind_input(int value_index, void* ptr) {
  if (values_[value_index].ptr == ptr) return;  // and so are its aliases: they are only ever re-pointed here
  values_[value_index].ptr = ptr;
  for (Value& v : values_) {  // values that share the input's storage (Reshape, Flatten, Identity)
    int root = v.alias_of;
    while (root >= 0 && values_[root].alias_of >= 0) root = values_[root].alias_of;
    if (root == value_index) v.ptr = ptr;
  }
}

void Session::prepare_pipeline() {
  if (pipe_ready_) return;
  // uploads and downloads have a stream each: a download waits for its run, and an upload queued behind it
  // in the same stream would wait for that run too instead of overlapping it
  OXB_CUDA(cudaStreamCreateWithFlags(&copy_stream_, cudaStreamNonBlocking));
  OXB_CUDA(cudaStreamCreateWithFlags(&down_stream_, cudaStreamNonBlocking));
  // A second input buffer is only safe when no step has the input's address built into a tensor map:
  // the tensor-core steps are the ones that do, so none of them may read an input (or an alias of one).
  pipe_double_ = external_bind_.empty();
  for (const Step& st : steps_) {
    if (st.family != 0) continue;
    for (int r : st.reads) {
      int root = r;
      while (values_[root].alias_of >= 0) root = values_[root].alias_of;
      for (auto& in : input_staging_)
        if (in.second == root) pipe_double_ = false;
    }
  }
  for (int f = 0; f < 2; ++f) {
    Flight& fl = flight_[f];
    OXB_CUDA(cudaEventCreateWithFlags(&fl.up, cudaEventDisableTiming));
    OXB_CUDA(cudaEventCreateWithFlags(&fl.done, cudaEventDisableTiming));
    OXB_CUDA(cudaEventCreateWithFlags(&fl.down, cudaEventDisableTiming));
    for (auto& in : input_staging_) {
      void* p = values_[in.second].ptr;
      if (f == 1 && pipe_double_) p = ctx_->alloc_device((size_t)values_[in.second].numel() * dt_size(values_[in.second].dt));
      fl.in_dev.push_back(p);
    }
    for (auto& out : output_staging_) {
      float* p = nullptr;
      OXB_CUDA(cudaMallocHost(&p, std::max<size_t>((size_t)values_[out.second].numel() * 4, 4)));
      fl.out_host.push_back(p);
      fl.out_dev.push_back(ctx_->alloc_device((size_t)values_[out.second].numel() * 4));
    }
  }
  pipe_ready_ = true;
}

void Session::submit(const oxb200_operand* feeds, uint32_t n, bool profile) {
  prepare_pipeline();
  Flight& fl = flight_[submit_idx_];
  Flight& prev = flight_[submit_idx_ ^ 1];
  if (fl.busy) raise(OXB200_FAILED, "submit: two runs are already in flight; collect one first");
  cudaStream_t main = ctx_->stream();
  // without a second input buffer the upload must wait until the previous run has read the inputs
  // validate every feed before the first input is re-pointed: a rejected submission leaves the plan as it was
  std::vector<const void*> srcs(input_staging_.size(), nullptr);
  for (size_t i = 0; i < input_staging_.size(); ++i) {
    const auto& in = input_staging_[i];
    const oxb200_operand* f = nullptr;
    for (uint32_t k2 = 0; k2 < n; ++k2)
      if (feeds[k2].name && in.first == feeds[k2].name) f = &feeds[k2];
    if (!f) raise(OXB200_FAILED, "submit: no feed for graph input '%s'", in.first.c_str());
    srcs[i] = feed_lanes(*f, values_[in.second], in.first.c_str());
  }
  if (!pipe_double_ && prev.busy) OXB_CUDA(cudaStreamWaitEvent(copy_stream_, prev.done, 0));
  for (size_t i = 0; i < input_staging_.size(); ++i) {
    const auto& in = input_staging_[i];
    Value& v = values_[in.second];
    const size_t bytes = (size_t)v.numel() * dt_size(v.dt);
    if (bytes >= kLanesUpload && !host_pinned(srcs[i])) ctx_->host_to_device(fl.in_dev[i], srcs[i], bytes, copy_stream_);
    else OXB_CUDA(cudaMemcpyAsync(fl.in_dev[i], srcs[i], bytes, cudaMemcpyHostToDevice, copy_stream_));
    ctx_->counters.uploads += 1;
    ctx_->counters.upload_bytes += (uint64_t)v.numel() * dt_size(v.dt);
    rebind_input(in.second, fl.in_dev[i]);
  }
  OXB_CUDA(cudaEventRecord(fl.up, copy_stream_));
  OXB_CUDA(cudaStreamWaitEvent(main, fl.up, 0));
  run_steps(profile);
  // the outputs move to this slot's own device buffers (a device-to-device copy, microseconds), so that the next
  // run may overwrite the arena while the download is still crossing PCIe
  for (size_t i = 0; i < output_staging_.size(); ++i) {
    const Value& v = values_[output_staging_[i].second];
    if (v.numel() > 0) OXB_CUDA(cudaMemcpyAsync(fl.out_dev[i], v.ptr, (size_t)v.numel() * 4, cudaMemcpyDeviceToDevice, main));
  }
  OXB_CUDA(cudaEventRecord(fl.done, main));
  OXB_CUDA(cudaStreamWaitEvent(down_stream_, fl.done, 0));
  for (size_t i = 0; i < output_staging_.size(); ++i) {
    const Value& v = values_[output_staging_[i].second];
    if (v.numel() > 0) OXB_CUDA(cudaMemcpyAsync(fl.out_host[i], fl.out_dev[i], (size_t)v.numel() * 4, cudaMemcpyDeviceToHost, down_stream_));
    ctx_->counters.downloads += 1;
    ctx_->counters.download_bytes += (uint64_t)v.numel() * 4;
  }
  OXB_CUDA(cudaEventRecord(fl.down, down_stream_));
  fl.busy = true;
  submit_idx_ ^= 1;
}

void Session::collect(oxb200_result* fetches, uint32_t n) {
  Flight& fl = flight_[collect_idx_];
  if (!fl.busy) raise(OXB200_FAILED, "collect: no run is in flight");
  if (n != outputs_.size()) raise(OXB200_FAILED, "collect: %u fetch slots for %zu graph outputs", n, outputs_.size());
  for (uint32_t i = 0; i < n; ++i) {
    const Value& v = values_[output_staging_[i].second];
    if (fetches[i].lanes && fetches[i].cap < (uint64_t)v.numel())
      raise(OXB200_FAILED, "collect: fetch buffer for '%s' holds %llu lanes, %lld needed", outputs_[i].c_str(), (unsigned long long)fetches[i].cap, (long long)v.numel());
  }
  OXB_CUDA(cudaEventSynchronize(fl.down));
  ctx_->counters.fences += 1;
  fl.busy = false;
  collect_idx_ ^= 1;
  const int flag = *(volatile int*)err_flag_;
  if (flag != 0 || fl.poisoned) {
    // The error word is shared by the runs in flight: let the other run finish before the word is cleared (its
    // kernels may still write it), and fail it as well.
    fl.poisoned = false;
    Flight& other = flight_[collect_idx_];
    OXB_CUDA(cudaStreamSynchronize(ctx_->stream()));
    OXB_CUDA(cudaStreamSynchronize(down_stream_));
    if (other.busy) other.poisoned = true;
    *(volatile int*)err_flag_ = 0;
    for (auto* p : umma_plans_) k::umma_plan_reset_after_error(p);
    for (auto* c : umma_chains_) k::umma_chain_reset_after_error(c);
    raise(OXB200_FAILED, "a kernel reported code %d during a pipelined run (or the run before it failed while this one was in flight); results are not valid", flag);
  }
  for (uint32_t i = 0; i < n; ++i) {
    const Value& v = values_[output_staging_[i].second];
    write_result_shape(v, &fetches[i]);
    if (fetches[i].lanes && v.numel() > 0) std::memcpy(fetches[i].lanes, fl.out_host[i], (size_t)v.numel() * 4);
  }
}

void Session::bind_external(const std::string& name, void* ptr, DT dt, Layout layout) { external_bind_[name] = {ptr, {dt, layout}}; }

void Session::use_resident(const std::string& name, const void* ptr) {
  if (in_tensor_map_.empty())
    for (auto& in : input_staging_) in_tensor_map_.push_back(input_in_tensor_map(in.second) ? 1 : 0);
  for (size_t i = 0; i < input_staging_.size(); ++i) {
    if (input_staging_[i].first != name) continue;
    Value& v = values_[input_staging_[i].second];
    if (in_tensor_map_[i]) OXB_CUDA(cudaMemcpyAsync(v.ptr, ptr, v.bytes, cudaMemcpyDeviceToDevice, ctx_->stream()));
    else rebind_input(input_staging_[i].second, const_cast<void*>(ptr));
  }
}

void Session::use_host(const std::string& name, const void* lanes) {
  for (auto& in : input_staging_) {
    if (in.first != name) continue;
    const size_t bytes = (size_t)values_[in.second].numel() * 4;
    stage_in(values_[in.second].ptr, lanes, bytes);
    ctx_->counters.uploads += 1;
    ctx_->counters.upload_bytes += bytes;
  }
}

size_t Session::device_bytes() const {
  size_t n = arena_.bytes;
  for (const DeviceBuffer& b : owned_) n += b.bytes;
  return n;
}

// ---- device I/O binding -------------------------------------------------------------------------
bool Session::input_in_tensor_map(int value_index) const {
  // the tensor-core steps build their operands' addresses into tensor maps at plan time
  for (const Step& st : steps_) {
    if (st.family != 0) continue;
    for (int r : st.reads) {
      int root = r;
      while (values_[root].alias_of >= 0) root = values_[root].alias_of;
      if (root == value_index) return true;
    }
  }
  return false;
}

void Session::bind_input_device(const std::string& name, const void* ptr, DT dt, uint64_t len) {
  if (in_flight() > 0) raise(OXB200_FAILED, "bind_input_device: pipelined runs are in flight; collect them first");
  for (size_t i = 0; i < input_staging_.size(); ++i) {
    if (input_staging_[i].first != name) continue;
    const Value& v = values_[input_staging_[i].second];
    if (external_bind_.count(name)) raise(OXB200_FAILED, "bind_input_device: '%s' is a resident dispatch operand", name.c_str());
    if (dt != v.dt) raise(OXB200_FAILED, "bind_input_device: '%s' was planned as %s, the buffer is %s", name.c_str(), dt_name(v.dt), dt_name(dt));
    if ((int64_t)len != v.numel()) raise(OXB200_FAILED, "bind_input_device: '%s' has %lld elements, the buffer %llu", name.c_str(), (long long)v.numel(), (unsigned long long)len);
    if (!ptr || ((uintptr_t)ptr & 15) != 0) raise(OXB200_FAILED, "bind_input_device: the buffer of '%s' must be a 16-byte aligned device address", name.c_str());
    if (own_in_ptr_.empty())
      for (auto& in : input_staging_) own_in_ptr_.push_back(values_[in.second].ptr);
    bound_in_[(int)i] = ptr;
    return;
  }
  raise(OXB200_FAILED, "bind_input_device: '%s' is not an input of the planned graph", name.c_str());
}

void Session::bind_output_device(const std::string& name, void* ptr, uint64_t cap) {
  for (size_t i = 0; i < output_staging_.size(); ++i) {
    if (output_staging_[i].first != name) continue;
    const Value& v = values_[output_staging_[i].second];
    if (cap < (uint64_t)v.numel()) raise(OXB200_FAILED, "bind_output_device: '%s' has %lld lanes, the buffer holds %llu", name.c_str(), (long long)v.numel(), (unsigned long long)cap);
    if (!ptr || ((uintptr_t)ptr & 3) != 0) raise(OXB200_FAILED, "bind_output_device: the buffer of '%s' must be a 4-byte aligned device address", name.c_str());
    bound_out_[(int)i] = {ptr, cap};
    return;
  }
  raise(OXB200_FAILED, "bind_output_device: '%s' is not an output of the planned graph", name.c_str());
}

void Session::output_device_ptr(const std::string& name, void** ptr, uint64_t* len) {
  for (size_t i = 0; i < output_staging_.size(); ++i) {
    if (output_staging_[i].first != name) continue;
    const Value& v = values_[output_staging_[i].second];
    if (ptr) *ptr = v.ptr;
    if (len) *len = (uint64_t)v.numel();
    return;
  }
  raise(OXB200_FAILED, "output_device_ptr: '%s' is not an output of the planned graph", name.c_str());
}

void Session::clear_bindings() {
  if (!own_in_ptr_.empty())
    for (size_t i = 0; i < input_staging_.size(); ++i) rebind_input(input_staging_[i].second, own_in_ptr_[i]);
  bound_in_.clear();
  bound_out_.clear();
}

// Between a bound buffer and the session's own: up to 1 MB by a kernel that takes part in the dependent launches, above it
// at the rate of the driver's copy.  A call that binds an output of 64 KB / 256 KB / 512 KB / 1 MB, kernel against driver:
// 28.7 / 29.4 / 22.9 / 23.9 against 30.8 / 32.5 / 25.6 / 26.2 us.  To an address that is not 16-byte aligned the kernel
// moves bytes: 28.9 / 31.1 / 26.4 / 29.9 against 30.8 / 32.1 / 25.6 / 29.8 us, so there the line is 256 KB.
static void copy_on_device(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  const bool aligned = (((uintptr_t)dst | (uintptr_t)src) & 15) == 0;
  if (bytes <= (aligned ? 1u << 20 : 256u << 10)) k::copy_bytes(dst, src, bytes, s);
  else OXB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, s));
}

// A bound input is read in place when no tensor map holds its buffer's address; otherwise its lanes are copied
// device-to-device into the buffer the maps were built for (no host traffic either way).
void Session::apply_input_bindings() {
  if (in_tensor_map_.empty())
    for (auto& in : input_staging_) in_tensor_map_.push_back(input_in_tensor_map(in.second) ? 1 : 0);
  for (auto& kv : bound_in_) {
    const int vi = input_staging_[kv.first].second;
    Value& v = values_[vi];
    if (in_tensor_map_[kv.first]) {
      if (v.ptr != own_in_ptr_[kv.first]) rebind_input(vi, own_in_ptr_[kv.first]);
      copy_on_device(v.ptr, kv.second, (size_t)v.numel() * dt_size(v.dt), ctx_->stream());
    } else {
      rebind_input(vi, const_cast<void*>(kv.second));
    }
  }
}

void Session::run_bound(const oxb200_operand* feeds, uint32_t n, oxb200_result* fetches, uint32_t nf, bool profile) {
  if (in_flight() > 0) raise(OXB200_FAILED, "run_bound: pipelined runs are in flight; collect them first");
  if (fetches && nf != outputs_.size()) raise(OXB200_FAILED, "run_bound: %u fetch slots for %zu graph outputs", nf, outputs_.size());
  begin_copies();
  // unbound inputs come from the host as in run()
  for (size_t i = 0; i < input_staging_.size(); ++i) {
    if (bound_in_.count((int)i)) continue;
    const auto& in = input_staging_[i];
    if (external_bind_.count(in.first)) continue;
    const oxb200_operand* f = nullptr;
    for (uint32_t k2 = 0; k2 < n; ++k2)
      if (feeds && feeds[k2].name && in.first == feeds[k2].name) f = &feeds[k2];
    if (!f) raise(OXB200_FAILED, "run_bound: graph input '%s' is neither bound nor fed", in.first.c_str());
    Value& v = values_[in.second];
    const void* src = feed_lanes(*f, v, in.first.c_str());
    stage_in(v.ptr, src, (size_t)v.numel() * dt_size(v.dt));
    ctx_->counters.uploads += 1;
    ctx_->counters.upload_bytes += (uint64_t)v.numel() * dt_size(v.dt);
  }
  apply_input_bindings();
  run_steps(profile);
  for (auto& kv : bound_out_) {
    const Value& v = values_[output_staging_[kv.first].second];
    if (v.numel() > 0 && kv.second.first != v.ptr)
      copy_on_device(kv.second.first, v.ptr, (size_t)v.numel() * 4, ctx_->stream());
  }
  if (fetches) {
    for (uint32_t i = 0; i < nf; ++i) {
      const Value& v = values_[output_staging_[i].second];
      if (fetches[i].lanes && fetches[i].cap < (uint64_t)v.numel())
        raise(OXB200_FAILED, "run_bound: fetch buffer for '%s' holds %llu lanes, %lld needed", outputs_[i].c_str(), (unsigned long long)fetches[i].cap, (long long)v.numel());
    }
    for (uint32_t i = 0; i < nf; ++i) {
      const Value& v = values_[output_staging_[i].second];
      write_result_shape(v, &fetches[i]);
      if (fetches[i].lanes && v.numel() > 0) {
        stage_out(fetches[i].lanes, v.ptr, (size_t)v.numel() * 4);
        ctx_->counters.downloads += 1;
        ctx_->counters.download_bytes += (uint64_t)v.numel() * 4;
      }
    }
  }
  finish_download();
}

}  // namespace oxb
