// traverse_form.h -- how a CWBVH traversal of n rays launches, for the host
// code and a host test.
#pragma once

#include <cstdint>

// The traversal launch forms a context can choose (obvhs_ctx_set_traversal_config):
// block size and stack placement.  Form 0 is the default.
struct TravForm {
  int block;
  bool smem_stack;
};
constexpr TravForm TRAV_FORMS[] = {{128, false}, {64, false}, {256, false}, {64, true}, {128, true}};
constexpr int N_TRAV_FORMS = 5;

// Maps (block, smem_stack) to a launch form, (0, 0) to the default; -1 when
// there is none.
inline int trav_form_index(uint32_t block, int smem_stack) {
  if (block == 0 && !smem_stack) return 0;
  for (int f = 0; f < N_TRAV_FORMS; f++)
    if ((uint32_t)TRAV_FORMS[f].block == block && TRAV_FORMS[f].smem_stack == (smem_stack != 0)) return f;
  return -1;
}

// Rays a warp takes at a time.  A call of few rays is a chain of dependent
// loads per ray, and a warp takes the time of all its rays' different steps
// together, so they are spread: one ray a warp while that gives each of the
// SMs' four schedulers at most two warps, then two, four, ... (1,000 host rays
// on 10k triangles 88.6 -> 78.9 us the call, 3,000 on 100k 111.6 -> 105.2,
// 14,400 149 -> 144; from 30,000 rays even.  Four warps a scheduler: 30,000
// rays 159 -> 167 us; one: 3,000 rays 108 us).  The kernels that take 32 are
// compiled apart: with the count in a register they ran 1-1.6 % slower.
// Only the default form is compiled for fewer than 32: a context that has
// chosen another gets it for every call.
inline uint32_t trav_rays_per_warp(uint32_t n, int num_sms, int form) {
  uint32_t lanes = form == 0 ? 1 : 32;
  while (lanes < 32 && (uint64_t)lanes * (uint64_t)num_sms * 8 < n) lanes *= 2;
  return lanes;
}
