// Plan and launcher of the resident time loop (resident.cuh).
#pragma once
#include <cstddef>
#include <vector>
#include <cuda_runtime.h>

namespace swfwi {

struct ResidentArgs;

// How a sweep over n slots is cut: `rounds` launches of up to `slots` slots,
// `cps` CTAs a slot.
struct ResidentPlan {
  bool ok = false;
  bool thin = false;   // slabs of fewer than 6 rows
  int rows = 0;        // rows a slot is cut into
  bool wide = false;   // the two-pass form
  int rounds = 0, slots = 0, cps = 0, rmax = 0, zp = 0, ngroups = 0, ogroups = 0, chunks = 0, helpers = 0;
  int cap_src = 0, cap_rec = 0, cap_stage = 0;
  size_t smem = 0, halo = 0;   // bytes a CTA, uint4 elements of the exchange buffer
};

// src_hist / rec_hist: per padded row, the most source / receiver points any
// slot has there.
ResidentPlan plan_resident(int arith, bool back, int n, int nx, int nz, int bx0, bool strips, const std::vector<int> &src_hist,
                           const std::vector<int> &rec_hist);
// Estimated time a step of the plan, and of the streaming kernels on a batch
// of `points` field points (own_velocity: a velocity model per slot).
double resident_us(const ResidentPlan &p, int arith, bool back);
double streamed_us(int arith, bool back, double points, bool own_velocity);
// One launch over nslots <= p.slots slots; the plan's fields of `a` are set here.
void launch_resident(int arith, bool back, const ResidentPlan &p, ResidentArgs a, int nslots, cudaStream_t st);

}  // namespace swfwi
