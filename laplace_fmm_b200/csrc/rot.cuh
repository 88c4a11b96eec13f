// FP64 translations (M2M, M2L, L2L) in factored form on the FP64 tensor
// cores: rotate the expansion so that the offset lies on the z axis, translate
// along it, rotate back (reference cpu/multipole3d.cpp:115-226), for tiles of
// targets that share one offset per slot.  After the rotation about z the map
// splits into one real block per degree (rotation about y, real and imaginary
// parts apart) and one per order (axial translation, the same for both parts):
// about 6 N^3 multiply-adds per pair against the dense operator's N^4, and no
// operator of the size of an expansion squared to build, keep or stream.
#pragma once
#include "m2l_gemm.cuh"

namespace lfmm {

enum RotMode { ROT_M2L = 0, ROT_M2M = 1, ROT_L2L = 2 };

// Blocks are stored as 8 x 4 fragments of mma.m8n8k4 (32 lanes, row lane / 4,
// column lane % 4): block n (size n + 1) has ceil((n+1)/8) x ceil((n+1)/4) of
// them, starting at fragment rot_frag0(n).
__host__ __device__ constexpr int rot_ksteps(int n) { return (n + 4) / 4; }
__host__ __device__ constexpr int rot_mtiles(int n) { return (n + 8) / 8; }
__host__ __device__ constexpr int rot_frag0(int n)
{
	return n < 4 ? n : n < 8 ? 4 + 2 * (n - 4) : n < 12 ? 12 + 6 * (n - 8) : n < 16 ? 36 + 8 * (n - 12) : 68 + 15 * (n - 16);
}
// Axial blocks of one cell size: |d|^2 = 4 .. 27 (M2L), M2M, L2L.
constexpr int ROT_AX_M2M = 24, ROT_AX_L2L = 25, ROT_AX = 26;

// Axial tables [nh][ROT_AX][rot_frag0(N)][32] for nh cell sizes, in the arena
// (nullptr when it cannot grow).  scaled: the scaled expansions' operators
// (h[0] = 1); otherwise entry i serves level i: M2L between cells of size h[i],
// M2M onto them from their children, L2L onto them from their parents.
const double* rot_axial_tables(Context& ctx, int N, const double* h, int nh, bool scaled);
inline const double* rot_axial_level(const double* tab, int N, int i) { return tab + (size_t)i * ROT_AX * rot_frag0(N) * 32; }

// One level's translations.  src: the source cells' expansions [cell][Nx2]
// (complex); dst: the targets', overwritten (M2L, M2M; cells outside
// plan.order keep theirs) or added to (L2L).  plan.vtab: [cell][189], [cell][8]
// or [cell][1] source cells (-1: none).  N <= 18.
template <typename real>
int rot_translate(Context& ctx, RotMode mode, const M2LPlan& plan, const real* src, real* dst, int N,
                  const double* axial);

// M2M plan of level L (slot = child octant): the cells with children, in
// order, and their children's level-local indices.
int m2m_plan_build(Context& ctx, const DevTree& t, int L, M2LPlan& plan);

} // namespace lfmm
