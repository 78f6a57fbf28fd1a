// colony_internal.h -- the colony object behind the opaque aco_colony
// handle, shared by the translation units of the library (not installed).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <sys/mman.h>
#include <unistd.h>

#include <string>
#include <vector>

#include "acogpu.h"
#include "aco_kernels.h"

struct aco_colony {
  aco_params p;
  int n = 0, m = 0, K = 0, ld = 0, ldk = 0, ldm = 0;
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  int32_t *dist = nullptr;
  float *eta = nullptr, *tau = nullptr, *choice = nullptr;
  int32_t *nn = nullptr;
  float *eta_nn = nullptr, *tau_nn = nullptr, *choice_nn = nullptr;
  int32_t *tours = nullptr;
  int64_t *newlen = nullptr, *len = nullptr;
  int32_t *succT = nullptr, *predT = nullptr, *gbtour = nullptr;
  int32_t *age = nullptr, *perf = nullptr;
  uint8_t *valid = nullptr;
  float *mean = nullptr;
  int32_t *dep_col = nullptr;
  float *dep_delta = nullptr;
  int32_t *plan = nullptr;  // aging colonies: the ants' roles of an iteration
  aco::ColonyState *st = nullptr;
  int16_t *nn16 = nullptr;  // candidate ids as int16, pitch ldk (k <= 32 kernels)
  float *xy = nullptr;      // coordinates (x then y) when created from coordinates
  bool staged = false;      // construction by the staged kernel
  bool direct = false;      // construction by the direct (L2-row) kernel
  int cluster = 0;          // construction by the cluster kernel: CTAs per cluster
  bool rows = false;        // construction by the long-row kernel (k > 32)
  bool rows_staged = false; // ... with the rows in shared memory
  bool neg_dist = false;    // a distance is negative: deposits may be
  bool is_signed = false;   // weights may be negative: the general kernel only
  int32_t *nn2 = nullptr;   // fallback second tier (see ColonyDev)
  float *t2v = nullptr;
  float *mout = nullptr;
  int t2 = 0;
  int staged_grid = 0, staged_warps = 0;
  int tune_warps = 0;  // ants per CTA forced by the autotuner (0: the plan's choice)
  int num_sms = 0, max_smem_optin = 0;
  std::vector<void *> allocations;
  bool initialized = false;
  int64_t optimum = -1;
  int apb = 4;
  int64_t launches = 0;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t graph_exec = nullptr;
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
  // Host copy of the device state block, valid until the next call that
  // enqueues work on the colony: the getters of one iteration share one
  // device-to-host read.  A colony read on its own stages it through a
  // pinned word allocated at its first read; a batch reads all its
  // instances through one pinned array of its own.
  aco::ColonyState h_cache{};
  aco::ColonyState *h_state = nullptr;
  bool state_fresh = false;
  std::string err;
};

// Maps the pages of a host buffer that a device-to-host copy is about to
// fill.  A caller's fresh buffer has no pages yet, and on this machine the
// copy then takes a fault from the GPU's side for each of them, about 70 us a
// 64 KB page: 64 MB (the pheromone at n = 4096) took 58.6 ms to read, and 2.3
// ms with the pages populated first; 2.4 MB 2.7 and 0.11 ms.  Buffers below
// 128 KB mostly come from a heap that is mapped already (malloc maps larger
// ones afresh).  On pages that are there already (a kept or pinned buffer) the
// call walks them for nothing: 0.7 us of a 15 us read of 160 KB, 2 of 36 us for
// 4 MB, 30 of 392 us for 64 MB.  So from 2 MB on, a buffer whose middle and last
// pages are there counts as mapped; asking takes 1.1 us.  The buffer's contents
// do not change; where the kernel cannot populate (EINVAL, or memory that is not
// the process's) the copy runs as before.
inline void prefault(void *p, size_t bytes) {
#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif
  static const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
  if (!p || bytes < (128u << 10)) return;
  const uintptr_t a = (uintptr_t)p / page * page;
  const uintptr_t e = ((uintptr_t)p + bytes + page - 1) / page * page;
  auto there = [](uintptr_t at) {
    unsigned char in = 0;
    return mincore(reinterpret_cast<void *>(at), 1, &in) == 0 && (in & 1);
  };
  const uintptr_t mid = ((uintptr_t)p + bytes / 2) / page * page;
  if (bytes >= (2u << 20) && there(e - page) && there(mid)) return;
  madvise(reinterpret_cast<void *>(a), e - a, MADV_POPULATE_WRITE);
}

// Every call that enqueues work on a colony (or rewrites its state) marks the
// cached state block stale.
inline void state_changed(aco_colony *c) { c->state_fresh = false; }

namespace aco {
// Device view of a colony (pointers and parameters passed to the kernels).
ColonyDev colony_dev(const aco_colony *c);
// Records `msg` as the colony's last error and returns `status`.
int colony_fail(aco_colony *c, int status, const std::string &msg);
// After a row pass over weights that a caller brought (initialise, written
// pheromone, a checkpoint, a prior): reads whether any is negative and, if the
// answer changed, chooses the construction kernel again.  The fast kernels
// settle picks by bounds on sums of weights that are not negative; the general
// kernel adds entry by entry and takes any.  errors: also reports the device's
// error words.
int colony_check_signs(aco_colony *c, bool errors);
}  // namespace aco
