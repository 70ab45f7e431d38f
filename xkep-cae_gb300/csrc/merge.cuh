// The pair-table merge between its two files: broadphase.cu orders the merged rows, pair.cu moves their state.
#pragma once

#include "xk_common.cuh"

// Sources of merged rows that do not continue an old row: a new pair, or MERGE_OLD - o: the old-only row o.
constexpr int32_t MERGE_NEW = -1, MERGE_OLD = -2;

// The old state's float table, which holds it, and the screened detection narrowphase taken on the way.
struct MergeScreen {
  const xk_pairs32* old32;
  const double* u;
  const float* node32;
  const xk_contact_params* cp;
  int32_t* n_exact;
};

// State of the *n merged rows (at most `most`) of out, whose ea and eb are written.  list: with screen, scratch of
// most + 1 words.
xk_status xk_merge_rows(const xk_mesh* m, const xk_pairs* old, const int32_t* src, const int64_t* n, long long most,
                        xk_pairs* out, const MergeScreen* screen, int32_t* list, cudaStream_t st);
