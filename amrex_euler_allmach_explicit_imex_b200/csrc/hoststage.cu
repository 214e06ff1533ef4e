// Copies between a caller's pageable host box and the device through the
// context's own page-locked staging buffers.
//
// A copy from pageable memory makes the CUDA driver stage it through a small
// pinned buffer of its own, one chunk at a time, behind the calling thread:
// at 2560x640 a state (52 MB) crosses at about 13 GB/s.  Here the rows of a
// band are first copied by a few host threads into a pinned staging copy of
// the state (compact: 4 planes of nx x ny), and the band then crosses by DMA
// while the threads copy the next band, so the host copies and the transfer
// overlap.  The staging buffers (one per direction) are allocated on the
// first pageable call and kept by the context.
//
// Batches of solves cross through one small ring of pinned bands that the
// batches of the process share (band_transfer, below).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstring>
#include <functional>
#include <memory>
#include <mutex>
#include <string>
#include <thread>

#include "copypool.h"
#include "ctx.h"

struct HostStage {
  double* in = nullptr;   // pinned: what crosses to the device
  double* out = nullptr;  // pinned: what comes back
  size_t doubles = 0;
  CopyPool* pool = nullptr;
  ~HostStage()
  {
    delete pool;
    if (in) cudaFreeHost(in);
    if (out) cudaFreeHost(out);
  }
};

bool host_pageable(const void* p)
{
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();  // an unknown pointer is plain host memory
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

// three quarters of the host threads, with the caller (measured on a 16-thread
// host at 2560x640: 3, 7, 11, 15 workers gave 0.40, 0.51, 0.62, 0.57 G
// cell-updates/s through the host step)
static CopyPool* new_pool()
{
  const unsigned hw = std::thread::hardware_concurrency();
  return new CopyPool(std::max(1, std::min(15, static_cast<int>(hw * 3 / 4) - 1)));
}

HostStage* host_stage(ecg_ctx* c)
{
  const size_t need = 4 * static_cast<size_t>(c->grid.nx) * static_cast<size_t>(c->grid.ny);
  if (c->stage && c->stage->doubles >= need) return c->stage;
  delete c->stage;
  c->stage = nullptr;
  HostStage* s = new HostStage();
  s->doubles = need;
  if (cudaMallocHost(&s->in, sizeof(double) * need) != cudaSuccess ||
      cudaMallocHost(&s->out, sizeof(double) * need) != cudaSuccess) {
    c->err = "pinned staging buffers: allocation failed";
    cudaGetLastError();
    delete s;
    return nullptr;
  }
  s->pool = new_pool();
  c->stage = s;
  return s;
}

void host_stage_destroy(HostStage* s) { delete s; }
double* host_stage_in(HostStage* s) { return s->in; }
double* host_stage_out(HostStage* s) { return s->out; }

// Rows [r0, r1) of the 4 planes: the caller's box (rows jstride apart, planes
// nstride apart, from its Array4 base already offset to cell (0, 0)) to the
// compact stage (to_stage), or back.  One task per plane and slice of rows.
void host_stage_copy(HostStage* s, double* stage, double* host, int64_t jstride, int64_t nstride, int nx, int ny,
                     int r0, int r1, bool to_stage)
{
  constexpr int kRowsPerTask = 16;
  const int rows = r1 - r0;
  if (rows <= 0) return;
  const int slices = (rows + kRowsPerTask - 1) / kRowsPerTask;
  const size_t plane = static_cast<size_t>(nx) * static_cast<size_t>(ny);
  const std::function<void(int)> job = [&](int k) {
    const int n = k / slices, sl = k % slices;
    const int a = r0 + sl * kRowsPerTask, b = std::min(r1, a + kRowsPerTask);
    for (int r = a; r < b; ++r) {
      double* st = stage + n * plane + static_cast<size_t>(r) * nx;
      double* h = host + n * nstride + static_cast<int64_t>(r) * jstride;
      if (to_stage) std::memcpy(st, h, sizeof(double) * nx);
      else std::memcpy(h, st, sizeof(double) * nx);
    }
  };
  s->pool->run(4 * slices, job);
}

// ---- batches: a shared ring of pinned bands ---------------------------------------
//
// The ring and its threads are made by the first batch that needs them, shared
// by every batch alive and freed with the last, so what is pinned does not grow
// with the number or the size of the batches.  One transfer holds the ring at a
// time; a transfer that finds it taken goes without.

// 4 bands of 2 MB (page-locking takes 2 to 5 ms from 1 MB to 8; with 512 KB bands
// the calling thread's 60 us a band held large boxes up).
namespace {
constexpr int kBandBytes = 1 << 21;
constexpr size_t kBandDoubles = kBandBytes / sizeof(double);

// Waits for a short while (a band crosses in 40 us) without going to sleep, then
// politely.
template <class Ready>
void await(Ready ready)
{
  for (int i = 0; !ready(); ++i) {
    if (i < 2000) std::this_thread::yield();
    else std::this_thread::sleep_for(std::chrono::microseconds(50));
  }
}
}  // namespace

struct BandRing {
  double* slots = nullptr;  // pinned, kBands bands of kBandDoubles
  std::unique_ptr<CopyPool> pool;
  std::mutex mu;
  ~BandRing()
  {
    if (slots) cudaFreeHost(slots);
  }
};

std::shared_ptr<BandRing> band_ring()
{
  static std::mutex mu;
  static std::weak_ptr<BandRing> shared;
  try {
    std::lock_guard<std::mutex> lock(mu);
    std::shared_ptr<BandRing> r = shared.lock();
    if (r) return r;
    r = std::make_shared<BandRing>();
    if (cudaHostAlloc(&r->slots, static_cast<size_t>(kBandBytes) * kBands, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      r->slots = nullptr;
      return nullptr;
    }
    r->pool.reset(new_pool());
    if (r->pool->workers() < 1) return nullptr;
    shared = r;
    return r;
  } catch (...) {
    return nullptr;
  }
}

// The pieces are rows of one plane that fit a band, in order; piece k goes
// through band k % kBands.  A box whose pieces all have a band of their own is
// copied a piece at a time by the threads together (64 solves of 256x256: 0.16 ms
// each up and down; 0.2 to 0.4 the other way, the calling thread waiting for
// threads that had yet to wake).  In a larger one the threads run through the
// pieces on their own, a task at a time (joined after every band they took twice
// as long into fresh pages), held back by `open`, the pieces whose band is theirs:
// to the device, empty again; to the host, filled.  The calling thread makes
// every CUDA call.
BandResult band_transfer(BandRing& ring, double* host, int64_t jstride, int64_t nstride, double* dev, long long pitch,
                         long long plane, int nx, int ny, bool upload, cudaStream_t stream, cudaEvent_t* event,
                         cudaError_t& err)
{
  if (static_cast<size_t>(nx) > kBandDoubles) return BandResult::kNotTaken;
  std::unique_lock<std::mutex> lock(ring.mu, std::try_to_lock);
  if (!lock.owns_lock()) return BandResult::kNotTaken;
  const int rows = std::min(ny, static_cast<int>(kBandDoubles / nx)), per = (ny + rows - 1) / rows, pieces = 4 * per;
  const size_t row = sizeof(double) * nx, dpitch = sizeof(double) * pitch;
  const int per_task = std::max(1, static_cast<int>(65536 / row)), tasks = (rows + per_task - 1) / per_task;
  std::atomic<int> open{0}, copied[kBands] = {};
  std::atomic<bool> stop{false};
  auto slot = [&](int k) { return ring.slots + (k % kBands) * kBandDoubles; };
  auto first = [&](int k) { return k % per * rows; };
  auto count = [&](int k) { return std::min(ny, first(k) + rows) - first(k); };
  auto task = [&](int n) {
    const int k = n / tasks, t = n % tasks;
    await([&] { return open > k || stop; });
    if (stop) return;
    double* st = slot(k);
    double* h = host + (k / per) * nstride + first(k) * jstride;
    for (int r = t * per_task, e = std::min(count(k), r + per_task); r < e; ++r) {
      if (upload) std::memcpy(st + static_cast<size_t>(r) * nx, h + r * jstride, row);
      else std::memcpy(h + r * jstride, st + static_cast<size_t>(r) * nx, row);
    }
    ++copied[k % kBands];
  };
  // the caller's side
  auto cross = [&](int k) {
    double* d = dev + (k / per) * plane + first(k) * pitch;
    err = upload ? cudaMemcpy2DAsync(d, dpitch, slot(k), row, row, count(k), cudaMemcpyHostToDevice, stream)
                 : cudaMemcpy2DAsync(slot(k), row, d, dpitch, row, count(k), cudaMemcpyDeviceToHost, stream);
    if (err == cudaSuccess) err = cudaEventRecord(event[k % kBands], stream);
    return err == cudaSuccess;
  };
  auto crossed = [&](int k) {
    err = cudaEventSynchronize(event[k % kBands]);
    return err == cudaSuccess;
  };
  const std::function<void(int)> f = std::ref(task);  // (std::ref: nothing to allocate)
  CopyPool::Job job;
  job.f = &f;
  job.n = pieces * tasks;
  // (the caller copies too while it waits: the threads take 0.1 ms to wake)
  auto copied_out = [&](int k) {
    await([&] {
      while (copied[k % kBands] != (k / kBands + 1) * tasks)
        if (!ring.pool->help(job, open * tasks)) return false;
      return true;
    });
  };
  bool ok = true, begun = false;
  if (pieces <= kBands) {
    open = pieces;
    auto copy = [&](int k) {
      const auto one = [&, k](int t) { task(k * tasks + t); };
      ring.pool->run(tasks, std::ref(one));
    };
    for (int k = 0; ok && k < pieces; ++k) {
      if (upload) copy(k);
      ok = cross(k);
    }
    for (int k = 0; ok && !upload && k < pieces; ++k) {
      ok = crossed(k);
      if (ok) copy(k);
    }
  } else if (upload) {
    constexpr int kLag = kBands / 2;  // copies in flight behind the piece being handed over
    open = kBands;
    begun = true;
    ring.pool->begin(job);
    for (int k = 0; ok && k < pieces; ++k) {
      copied_out(k);
      ok = cross(k) && (k < kLag || crossed(k - kLag));
      if (ok && k >= kLag) open = k - kLag + kBands + 1;
    }
  } else {
    for (int k = 0; ok && k < kBands; ++k) ok = cross(k);
    ok = ok && crossed(0);  // (behind whatever the stream still runs: the threads start after it)
    if (ok) {
      open = 1;
      begun = true;
      ring.pool->begin(job);
      for (int k = 1; ok && k < pieces; ++k) {
        // the band of piece k - 1 + kBands is free once piece k - 1 is copied
        ok = crossed(k);
        if (ok) open = k + 1;
        if (ok && k - 1 + kBands < pieces) {
          copied_out(k - 1);
          ok = cross(k - 1 + kBands);
        }
      }
    }
  }
  if (!ok) stop = true;
  if (begun) ring.pool->finish(job);
  // no copy of this transfer outlives the hold on the bands
  const cudaError_t e = cudaStreamSynchronize(stream);
  if (ok) err = e;
  return err == cudaSuccess ? BandResult::kDone : BandResult::kFailed;
}
