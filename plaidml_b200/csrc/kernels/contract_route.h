// Which contractions leave the general kernel: matrix products for the tensor cores, and the strided form of the lean
// kernel.  Host side only; both rules look at the descriptor alone.
#pragma once

#include <stdint.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <vector>

#include "generic.h"

namespace pmlb {

// A contraction as batch x (m x k times k x n) with the strides of every role in elements.
struct ProductForm {
  long long batch = 1, m = 1, n = 1, k = 1;
  int a = 0, b = 1;              // sources in the roles of A and B
  long long am = 0, ak = 0, bk = 0, bn = 0, cm = 0;   // A(i, k), B(k, j), C(i, j): C's columns are contiguous
  long long ab = 0, bb = 0, cb = 0;                   // between batch entries
};

// Sum of products of two f32 tensors into f32 whose index expressions are single variables: every variable is a row
// (output and one source), a column (output and the other), a term (both sources) or a batch index (all three).  The
// variables of a role must merge into one dimension; A and B each need a contiguous dimension, the output contiguous
// columns (exchanging the sources transposes the product).  Every output element must be reached and every read in
// range, since the tensor-core kernel tests neither.  More than 32768 multiply-adds: up to there the lean kernel adds the
// terms one by one in f32, which small exact expectations rely on (the planner draws the same line for its GEMMs).
// Whether the product is also faster there: product_pays.
inline bool product_form(const GenericParams& p, ProductForm* out) {
  if (p.agg != PMLB_AGG_SUM || p.combo != PMLB_COMBO_MUL || p.n_src != 2 || p.n_cons != 0 || p.has_init) return false;
  if (p.out.dtype != PMLB_F32 || p.src[0].dtype != PMLB_F32 || p.src[1].dtype != PMLB_F32) return false;
  const GAccess* t[3] = {&p.out, &p.src[0], &p.src[1]};
  long long stride[3][PMLB_MAX_IDX];
  bool has[3][PMLB_MAX_IDX];
  double macs = 1;
  for (int i = 0; i < p.n_idx; ++i) {
    if (p.range[i] <= 0) return false;
    macs *= static_cast<double>(p.range[i]);
    for (int s = 0; s < 3; ++s) has[s][i] = false, stride[s][i] = 0;
  }
  if (macs <= 32768.0) return false;
  for (int s = 0; s < 3; ++s) {
    for (int d = 0; d < t[s]->rank; ++d) {
      if (t[s]->off[d] != 0 || t[s]->den[d] != 1 || t[s]->strides[d] < 0) return false;
      int var = -1;
      for (int i = 0; i < p.n_idx; ++i) {
        if (t[s]->coef[d][i] == 0 || p.range[i] == 1) continue;   // (a single-valued variable is 0)
        if (var >= 0 || t[s]->coef[d][i] != 1) return false;
        var = i;
      }
      if (var < 0) {
        if (t[s]->sizes[d] < 1 || (s == 0 && t[s]->sizes[d] != 1)) return false;
        continue;
      }
      if (has[s][var]) return false;   // a diagonal
      if (s == 0 ? p.range[var] != t[s]->sizes[d] : p.range[var] > t[s]->sizes[d]) return false;
      has[s][var] = true;
      stride[s][var] = t[s]->strides[d];
    }
  }
  for (int order = 0; order < 2; ++order) {
    const int sa = 1 + order, sb = 2 - order;
    struct Role {
      std::vector<int> vars;
      long long extent = 1, so = 0, sa = 0, sb = 0;
    } m, n, k, b;
    bool ok = true;
    for (int i = 0; i < p.n_idx && ok; ++i) {
      if (p.range[i] == 1) continue;
      const bool o = has[0][i], x = has[sa][i], y = has[sb][i];
      if (o && x && y) b.vars.push_back(i);
      else if (o && x) m.vars.push_back(i);
      else if (o && y) n.vars.push_back(i);
      else if (x && y) k.vars.push_back(i);
      else ok = false;
    }
    auto merge = [&](Role* r, int key) {
      std::sort(r->vars.begin(), r->vars.end(), [&](int x, int y) { return stride[key][x] > stride[key][y]; });
      for (size_t j = 0; j < r->vars.size(); ++j) {
        const int v = r->vars[j];
        r->extent *= p.range[v];
        if (j + 1 == r->vars.size()) {
          r->so = stride[0][v], r->sa = stride[sa][v], r->sb = stride[sb][v];
        } else {
          const int w = r->vars[j + 1];
          for (int s = 0; s < 3; ++s) {
            if (has[s][v] && stride[s][v] != stride[s][w] * p.range[w]) return false;
          }
        }
      }
      return true;
    };
    ok = ok && merge(&m, 0) && merge(&n, 0) && merge(&b, 0) && merge(&k, sa);
    if (!ok || m.extent > INT_MAX || n.extent > INT_MAX || k.extent > INT_MAX || b.extent > INT_MAX) continue;
    if (n.extent > 1 && n.so != 1) continue;
    if (m.extent > 1 && n.extent > 1 && m.so < n.extent) continue;
    if (m.extent > 1 && m.sa != 1 && k.extent > 1 && k.sa != 1) continue;
    if (n.extent > 1 && n.sb != 1 && k.extent > 1 && k.sb != 1) continue;
    out->batch = b.extent, out->m = m.extent, out->n = n.extent, out->k = k.extent;
    out->a = sa - 1, out->b = sb - 1;
    out->am = m.sa, out->ak = k.sa, out->bk = k.sb, out->bn = n.sb, out->cm = m.so;
    out->ab = b.sa, out->bb = b.sb, out->cb = b.so;
    return true;
  }
  return false;
}

// Whether a contraction of product form goes to the tensor cores, `product_us` being the estimate for the tiles that would
// be launched.  Fewer than 16 terms stay with the lean (else the general) kernel: there a plain f32 sum is as exact, one
// k-block of the tensor-core kernel is 64 terms, and it was the slower one at every shape measured (4096 x 4096 outer
// product 13 against 55 us, 512 x 512 x 8 terms 4.8 against 5.5).  From 16 on the estimates decide: batch entries and
// single rows or columns cost a 128 x 64 tile each, whatever part of it exists.  The lean kernel takes 0.22 us per term
// (its threads add term by term) or 6 multiply-adds per picosecond, the general one 2.3 us or 0.06 (B200, graph replays
// of 137 shapes).  Lean against tensor cores: 65536 dot products of 64 terms 37 against 2209 us, 256 products of 32 x 32
// x 32 10.7 against 11.3, 64 x 64 x 16 6.2 against 5.1, 4096 products of 64 x 64 x 64 236 against 168, 4096 x 512 x 512
// with A transposed 23 ms (general), 945 (lean) against 23 us.
inline bool product_pays(const ProductForm& f, bool lean, double product_us) {
  if (f.k < 16) return false;
  const double terms = static_cast<double>(f.k), macs = terms * f.m * f.n * f.batch;
  const double other_us = 2.5 + (lean ? std::max(0.22 * terms, macs / 6e6) : std::max(2.3 * terms, macs / 6e4));
  return product_us <= 0.95 * other_us;
}

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
