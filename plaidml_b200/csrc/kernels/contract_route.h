// Which contractions leave the general kernel for the strided form of the lean kernels.  Host side only; the rule looks
// at the descriptor alone.
#pragma once

#include <stdint.h>

#include <cstring>

#include "generic.h"

namespace pmlb {

// The lean kernel's form: see generic.cu.  Output dims are single variables without offset, everything is integral,
// offsets fit 32 bits, at most four of the variables that are not in the output have a range above 1, and at most four
// bounds tests remain after those that the ranges imply are dropped.
inline bool lean_form(const GenericParams& p, LeanParams* out) {
  std::memset(out, 0, sizeof(*out));
  if (!p.direct || p.out_elems <= 0 || p.out_elems >= (1ll << 31)) return false;
  if (p.combo != PMLB_COMBO_NONE && p.combo != PMLB_COMBO_MUL && p.combo != PMLB_COMBO_ADD) return false;
  for (int i = 0; i < p.n_idx; ++i) {
    if (p.range[i] <= 0 || p.range[i] >= (1ll << 31)) return false;
  }
  auto fits = [](long long v) { return v > -(1ll << 31) && v < (1ll << 31); };
  // output dims, extent-1 dims dropped
  int var_of[PMLB_MAX_RANK];
  int rank = 0;
  bool in_out[PMLB_MAX_IDX] = {false};
  for (int d = 0; d < p.out.rank; ++d) {
    const int v = p.out_var[d];
    in_out[v] = true;
    if (p.out.off[d] != 0 || p.range[v] < p.out.sizes[d]) return false;
    if (p.out.sizes[d] == 1) continue;
    out->size[rank] = static_cast<int>(p.out.sizes[d]);
    out->out_stride[rank] = p.out.strides[d];
    out->init_stride[rank] = p.has_init ? p.init.strides[d] : 0;
    var_of[rank++] = v;
  }
  out->rank = rank;
  // loops over the other variables, in their order
  int loops[4];
  int n_loop = 0;
  for (int i = 0; i < p.n_idx; ++i) {
    if (in_out[i] || p.range[i] == 1) continue;
    if (n_loop == 4) return false;
    loops[n_loop++] = i;
  }
  for (int j = 0; j < 4; ++j) {
    const int from = j - (4 - n_loop);   // (the innermost loop is number 3)
    out->loop[j] = from >= 0 ? static_cast<int>(p.range[loops[from]]) : 1;
  }
  auto add_check = [&](const int* coef, long long off, long long size) {
    // the range of the expression over the whole index box
    long long lo = off, hi = off;
    for (int i = 0; i < p.n_idx; ++i) {
      long long r = p.range[i] - 1;
      for (int d = 0; d < p.out.rank; ++d) {
        if (p.out_var[d] == i) r = p.out.sizes[d] - 1;
      }
      (coef[i] < 0 ? lo : hi) += coef[i] * r;
    }
    if (lo >= 0 && hi < size) return true;
    // (with room for a kernel to look a few elements past an end)
    if (out->n_check == 4 || lo < -(1ll << 30) || hi > (1ll << 30) || size < 0 || size > (1ll << 30)) return false;
    LeanParams::Check& c = out->check[out->n_check++];
    c.base = static_cast<int>(off);
    c.size = static_cast<int>(size);
    for (int d = 0; d < rank; ++d) c.out[d] = coef[var_of[d]];
    for (int j = 0; j < 4; ++j) c.loop[j] = j >= 4 - n_loop ? coef[loops[j - (4 - n_loop)]] : 0;
    return true;
  };
  for (int s = 0; s < p.n_src; ++s) {
    const GAccess& a = p.src[s];
    long long coef[PMLB_MAX_IDX] = {0}, base = 0, lo = 0, hi = 0;
    for (int d = 0; d < a.rank; ++d) {
      if (a.den[d] != 1) return false;
      base += a.off[d] * a.strides[d];
      for (int i = 0; i < p.n_idx; ++i) coef[i] += static_cast<long long>(a.coef[d][i]) * a.strides[d];
      if (!add_check(a.coef[d], a.off[d], a.sizes[d])) return false;
    }
    lo = hi = base;
    for (int i = 0; i < p.n_idx; ++i) (coef[i] < 0 ? lo : hi) += coef[i] * (p.range[i] - 1);
    if (!fits(base) || !fits(lo) || !fits(hi)) return false;
    out->src[s].base = static_cast<int>(base);
    for (int d = 0; d < rank; ++d) out->src[s].out[d] = static_cast<int>(coef[var_of[d]]);
    for (int j = 0; j < 4; ++j) out->src[s].loop[j] = j >= 4 - n_loop ? static_cast<int>(coef[loops[j - (4 - n_loop)]]) : 0;
  }
  for (int c = 0; c < p.n_cons; ++c) {
    if (!add_check(p.cons_coef[c], p.cons_off[c], p.cons_range[c])) return false;
  }
  for (int d = 0; d < rank; ++d) out->fd_size[d] = make_fastdiv(static_cast<uint32_t>(out->size[d]));
  out->elems = p.out_elems;
  out->agg = p.agg;
  out->combo = p.combo;
  out->has_init = p.has_init;
  out->out_dtype = p.out.dtype;
  out->init_dtype = p.init.dtype;
  for (int s = 0; s < p.n_src; ++s) out->src[s].dtype = p.src[s].dtype;
  out->n_src = p.n_src;
  return true;
}

}  // namespace pmlb
