// 3D rotation-based Laplace FMM on the device (plain FP64 form).
#pragma once
#include "m2l_gemm.cuh"

namespace lfmm {

struct SolveStats {
	int N = 0, depth = 0;
	size_t n_particles = 0, n_cells = 0, n_leaves = 0, targets_num = 0;
	size_t n_far_pairs = 0, n_close_pairs = 0, n_p2p_pairs = 0;
	size_t n_m2p = 0, n_w = 0, n_x = 0;
	float ms_tree = 0, ms_upward = 0, ms_m2l = 0, ms_l2l = 0, ms_leaves = 0, ms_total = 0;
	float ms_m2l_kernel = 0;     // inside the M2L GEMMs (3D: tensor-core launches; 2D: every level's)
	int n_m2l_kernel = 0;        // those launches
};

// Solve on device-resident inputs; pot (n_out) and field (n_out x 3) are
// device pointers, n_out = nt if nt > 0 else ns.  N = number of degrees
// (order p + 1), depth = uniform tree depth (levels), both already resolved.
int fmm3d_solve_device(Context& ctx, const ParticleInput& in, int N, int depth, double* pot, double* field,
                       SolveStats* stats, DevTree* tree_out = nullptr);

// Scaled-expansion solver on the adaptive-form tree (max_leaf = 0: uniform
// depth `depth`; > 0: adaptive, at most `depth` levels): precision 0 = FP64,
// 1 = mixed (FP32 expansions / near field, FP64 M2L on levels 2-3, FP64 tile
// sums and self term).  N <= 18.
// Vector charges (in.srcq: 3 doubles per source): field = sum q x d / r^3.
int fmm3d_solve_vector(Context& ctx, const ParticleInput& in, int N, int depth, int max_leaf, int precision,
                       double* field, SolveStats* stats);
// level_N (optional, depth entries): the M2L order of each level, the
// degrees of the source multipoles its M2L uses (0 or >= N: N); honoured on
// the tensor-core (mixed-form FP32) levels, whose expansions keep N degrees.
int fmm3d_solve_scaled(Context& ctx, const ParticleInput& in, int N, int depth, int max_leaf, int precision,
                       double* pot, double* field, SolveStats* stats, DevTree* tree_out = nullptr,
                       const int* level_N = nullptr);
// The same on a tree built by tree_build_adaptive (phase events 0 and 1, the
// tree build, are the caller's when timing).
int fmm3d_scaled_on_tree(Context& ctx, const DevTree& t, int N, int precision, double* pot, double* field,
                         SolveStats* stats, const int* level_N = nullptr);

// The plain form's leaves (uniform tree, unscaled expansions [cell][Nx2]): P2M
// of every leaf, and the near field with (inner != nullptr) the local
// expansions, written to pot and field in input order.
int plain_p2m(Context& ctx, const DevTree& t, int N, double2* outer);
int plain_leaves(Context& ctx, const DevTree& t, int N, const double2* inner, double* pot, double* field);

// One leaf's P2M or one cell's P2L alone (lfmm_debug_leaf_sums).
template <typename real>
int debug_leaf_sums(Context& ctx, bool irregular, int N, size_t n_lists, const size_t* off, const double* xyz,
                    const double* q, double* out);

// Dense FP64 M2L operators [343][MT][MT] for cell size h (h = 1: the
// level-independent scaled operators): built into out (m2l_ops_bytes), which the
// FP32 and tensor-core sets are converted from, or cached in the context (the
// FP64 form's low orders, m2l_dense64).
inline size_t m2l_ops_bytes(int N) { return sizeof(double) * 343 * (size_t)m2l_padded(N) * m2l_padded(N); }
int m2l_ops_build(Context& ctx, int N, double h, double* out);
double* m2l_ops_fp64(Context& ctx, int N, double h);
float* m2l_ops_fp32(Context& ctx, int N);

} // namespace lfmm
