// Plan object of the KNN pooling, shared by the pooling kernels and the training-step kernels.
#pragma once
#include "common.cuh"

struct fovi_knnpool_plan {
  int n_in = 0, n_out = 0, K = 0;
  int* idx = nullptr;     // [n_out, K] neighbour indices, pad = n_in
  float* wgt = nullptr;   // [n_out, K] neighbour weights of the 'gaussian' mode (null until set)
  // The same table from the inputs' side: the places (n << 8 | k) that read input m are t_entry[t_start[m] .. t_start[m + 1]), in ascending order.
  int* t_start = nullptr; // [n_in + 1]; null: more than 255 neighbours or 2^23 outputs
  int* t_entry = nullptr;
};
