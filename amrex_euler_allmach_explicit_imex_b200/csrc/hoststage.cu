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
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <functional>
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

// A stage of its own with room for `doubles`, for one direction at a time
// (host_stage_in: to the device, else host_stage_out); null when the pinned
// buffer cannot be allocated.
HostStage* host_stage_sized(HostStage* s, size_t doubles, bool to_device)
{
  if (!s) {
    s = new HostStage();
    s->doubles = doubles;
    s->pool = new_pool();
  }
  double*& buf = to_device ? s->in : s->out;
  if (!buf && cudaMallocHost(&buf, sizeof(double) * s->doubles) != cudaSuccess) {
    cudaGetLastError();
    buf = nullptr;
  }
  return s;
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
