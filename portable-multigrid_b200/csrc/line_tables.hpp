// Host tables of the line kernels, built once per degree and type.
#pragma once

#include "fields.hpp"
#include "line_kernels.cuh"

namespace pmg {

template <int N, typename T> const kern::LineTab<N, T> &line_tables() {
  static const kern::LineTab<N, T> tab = [] {
    const Tables1D &t = cached_tables(N - 1);
    kern::LineTab<N, T> k;
    kern::fill_even_odd<N>(k, t.S.data(), t.SD.data());
    for (int q = 0; q < N; ++q) k.W[q] = (T)t.W[q];
    return k;
  }();
  return tab;
}

template <int N, typename T> const kern::BoxTab<N, T> &box_tables() {
  static const kern::BoxTab<N, T> tab = [] {
    const Tables1D &t = cached_tables(N - 1);
    auto product = [&](const std::vector<double> &a, int i, int j) { // sum_q a_i(q) w_q a_j(q)
      double v = 0.0;
      for (int q = 0; q < N; ++q) v += a[i * N + q] * t.W[q] * a[j * N + q];
      return v;
    };
    kern::BoxTab<N, T> k;
    kern::fill_even_odd(k.eM, [&](int i, int j) { return product(t.S, i, j); });
    kern::fill_even_odd(k.eK, [&](int i, int j) { return product(t.SD, i, j); });
    return k;
  }();
  return tab;
}

} // namespace pmg
