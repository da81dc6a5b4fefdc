// Flat forest layout for batched prediction on the device.
#pragma once
#include "device_common.cuh"

namespace lgbm_b200 {

// A node of the compact layout, 8 bytes: a step of a tree walk is one 8-byte
// load and one comparison. The two children lie side by side; a walk goes to
// the first one when x <= threshold, else, and with NaN, to the second one,
// where x is the feature's value or (kPNodeNegate) its negative:
//   - NaN to the right: the children are (left, right), x = v and threshold
//     the largest f32 not above the f64 threshold. The feature values are
//     f32, so the comparison is the f64 one.
//   - NaN to the left: the children are (right, left), x = -v and threshold the
//     largest f32 below -t, so that x <= threshold is v > t.
// A leaf at place i has the first child i - 1 and a NaN threshold, so that a
// walk that goes on past its leaf stays there.
struct PNode {
  float threshold;  // categorical: the index of the bitset (into cat_bnd), as bits
  uint32_t meta;    // first child (16 bits) | feature (13) | zero inverts | categorical | negate
};
constexpr int kPNodeFeatureBits = 13;
constexpr uint32_t kPNodeZeroFlip = 1u << 29, kPNodeCat = 1u << 30, kPNodeNegate = 1u << 31;
constexpr int32_t kPNodeMaxLeaves = 32767;  // node indices of a tree fit 16 bits

// The layout of forests the compact one cannot hold (a tree of more leaves,
// a larger feature index). Categorical nodes keep the index of their category
// bitset (into cat_bnd) in the threshold's bits.
struct __align__(8) DNodeWide {
  double threshold;
  int32_t feat_dt;  // real feature column (low 24 bits) | decision_type << 24
  int32_t pad;
  int32_t left, right;  // child node, or ~leaf
};

constexpr int32_t kNodeFeatureBits = 24;

struct DForest {
  int32_t num_trees, ntpi;
  bool compact;           // nodes are PNode, else DNodeWide
  int32_t max_nodes;      // compact: the most nodes of a tree, padding included
  bool special;           // compact: some node is categorical or inverts at zero
  int32_t max_feature;    // the largest feature index
  const int4* tree;       // [num_trees] (first node, first leaf value, num_leaves, compact: nodes with padding)
  const void* nodes;      // trees concatenated
  const int32_t* cat_bnd; // bitset word ranges
  const uint32_t* cat_words;  // category bitsets
  const double* leaf_value;   // compact: by node
};

// Raw scores out[r * ntpi + k] of rows X[r * ncol ...] (device pointers).
// Allocates nothing.
cudaError_t launch_predict(const DForest& f, const float* X, int64_t nrow, int32_t ncol, double* out, cudaStream_t s);

// Device, stream, flat layout and trees per iteration of a forest made by
// lgbm_b200_forest_create.
void forest_parts(const LgbmB200Forest* F, int* device, cudaStream_t* stream, const DForest** f, int32_t* ntpi);

}  // namespace lgbm_b200
