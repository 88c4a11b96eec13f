// 3D rotation-based Laplace FMM, plain FP64 form.
//
// Operators follow the reference's CPU solver (cpu/multipole3d.cpp): P2M
// 20-49, rotate-z / rotate-y 51-113, M2M / M2L / L2L as rotate, z-translate,
// rotate back 115-226, passes 228-412, P2P + L2P 855-1294.  The translations
// run on the factored engine (rot.cu), the leaves on far_kernels.cuh; the
// per-pair rotation kernels here (warp per box, lanes own coefficients) are the
// LFMM_M2L=rotation engine and build the dense operators.
#include "fmm3d.cuh"
#include "m2l_gemm.cuh"
#include "rot.cuh"
#include <algorithm>

namespace lfmm {

namespace {

constexpr int CMAX = (MAXN3 * (MAXN3 + 1) / 2 + 31) / 32;   // coefficients per lane (6)
constexpr int NX2MAX = MAXN3 * (MAXN3 + 1) / 2;             // 171
constexpr int WPB = 4;                                      // warps per block, box kernels


enum { OP_M2M = 0, OP_M2L = 1, OP_L2L = 2 };

struct Exp {
	int N, Nx2;
	double2* outer;
	double2* inner;
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{ return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }

__device__ __forceinline__ int dir_id(int dx, int dy, int dz) { return (dx + 3) * 49 + (dy + 3) * 7 + (dz + 3); }

__device__ __forceinline__ void coords3(uint64_t code, int* c)
{ c[0] = (int)compact3(code >> 2); c[1] = (int)compact3(code >> 1); c[2] = (int)compact3(code); }

// res[n,m] = d(n,m,0) a[n,0] + sum_k (Re a[n,k](d_{m,k}+d_{m,-k}), Im a[n,k](d_{m,k}-d_{m,-k}))
__device__ __forceinline__ void rotate_y_warp(const double2* __restrict__ in, double2* __restrict__ out,
                                              const double* __restrict__ D, int Nx2)
{
	const int lane = threadIdx.x & 31;
#pragma unroll
	for (int t = 0; t < CMAX; ++t) {
		int c = lane + 32 * t;
		if (c < Nx2) {
			const int n = tri_row(c), m = c - tix(n, 0);
			const double* Dr = D + dix(n, m, 0);
			double vr = 0.0, vi = 0.0;
			const double2* row = in + tix(n, 0);
			for (int k = 1; k <= n; ++k) {
				double z1 = Dr[k], z2 = Dr[-k];
				double2 w = row[k];
				vr = fma(w.x, z1 + z2, vr);
				vi = fma(w.y, z1 - z2, vi);
			}
			double d0 = Dr[0];
			vr = fma(d0, row[0].x, vr);
			vi = fma(d0, row[0].y, vi);
			out[c] = make_double2(vr, vi);
		}
	}
}

struct Smem {
	double2 a[NX2MAX];
	double2 b[NX2MAX];
	double rn[2 * MAXN3 + 2];
};

// acc += R_z(-phi) R_y(-theta) T_z(rho) R_y(theta) R_z(phi) src, warp-cooperative.
template <int OP>
__device__ void translate_warp(const double2* __restrict__ src, double px, double py, double pz, int dirid,
                               double2 (&acc)[CMAX], int N, int Nx2, Smem& sm, const DevTables& T, unsigned* flags)
{
	const int lane = threadIdx.x & 31;
	int4 di = T.dirinfo[dirid];
	if (di.x < 0 || di.y < 0 || di.z < 0 || di.w < 0) {
		if (lane == 0) atomicOr(flags, DEV_ERR_DIRECTION);
		return;
	}
	const double* D1 = T.dmat + (size_t)di.x * dsize(MAXN3);
	const double* D2 = T.dmat + (size_t)di.y * dsize(MAXN3);
	const double2* E1 = T.emat + di.z * MAXN3;
	const double2* E2 = T.emat + di.w * MAXN3;
	double rho = sqrt(px * px + py * py + pz * pz) + 1e-12;
	if (OP == OP_M2L) {
		double inv = 1.0 / rho;
		for (int i = lane; i < 2 * N + 1; i += 32) {
			double p = 1.0;
			for (int j = 0; j < i; ++j) p *= inv;
			sm.rn[i] = p;
		}
	} else {
		for (int i = lane; i < N; i += 32) {
			double p = 1.0;
			for (int j = 0; j < i; ++j) p *= rho;
			sm.rn[i] = p;
		}
	}
#pragma unroll
	for (int t = 0; t < CMAX; ++t) {
		int c = lane + 32 * t;
		if (c < Nx2) sm.a[c] = cmul(src[c], E1[c - tix(tri_row(c), 0)]);
	}
	__syncwarp();
	rotate_y_warp(sm.a, sm.b, D1, Nx2);
	__syncwarp();
	const double* cube = OP == OP_M2L ? T.m2l : (OP == OP_M2M ? T.m2m : T.l2l);
#pragma unroll
	for (int t = 0; t < CMAX; ++t) {
		int c = lane + 32 * t;
		if (c < Nx2) {
			const int j = tri_row(c), k = c - tix(j, 0);
			const double* cf = cube + (j * MAXN3 + k) * MAXN3;
			double sr = 0.0, si = 0.0;
			if (OP == OP_M2L) {
				for (int n = k; n < N; ++n) {
					double f = cf[n] * sm.rn[j + n + 1];
					double2 w = sm.b[tix(n, k)];
					sr = fma(f, w.x, sr); si = fma(f, w.y, si);
				}
			} else if (OP == OP_M2M) {
				for (int n = 0; j - n >= k; ++n) {
					double f = cf[n] * sm.rn[n];
					double2 w = sm.b[tix(j - n, k)];
					sr = fma(f, w.x, sr); si = fma(f, w.y, si);
				}
			} else {
				for (int n = j; n < N; ++n) {
					double f = cf[n] * sm.rn[n - j];
					double2 w = sm.b[tix(n, k)];
					sr = fma(f, w.x, sr); si = fma(f, w.y, si);
				}
			}
			sm.a[c] = make_double2(sr, si);
		}
	}
	__syncwarp();
	rotate_y_warp(sm.a, sm.b, D2, Nx2);
	__syncwarp();
#pragma unroll
	for (int t = 0; t < CMAX; ++t) {
		int c = lane + 32 * t;
		if (c < Nx2) {
			double2 v = cmul(sm.b[c], E2[c - tix(tri_row(c), 0)]);
			acc[t].x += v.x; acc[t].y += v.y;
		}
	}
	__syncwarp();
}

// ---------------------------------------------------------------- M2M
__global__ void __launch_bounds__(WPB * 32) m2m_kernel(DevTree t, Exp E, int L, DevTables T, unsigned* flags)
{
	__shared__ Smem sm[WPB];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	size_t c = (size_t)blockIdx.x * WPB + w;
	if (c >= t.lsize[L]) return;
	size_t g = t.loff[L] + c, cb = t.loff[L + 1];
	double2 acc[CMAX];
#pragma unroll
	for (int k = 0; k < CMAX; ++k) acc[k] = make_double2(0.0, 0.0);
	for (uint32_t k = t.beg[g]; k < t.end[g]; ++k) {
		size_t gk = cb + k;
		uint64_t oct = t.code[gk] & 7ull;
		int d = dir_id(2 * (int)((oct >> 2) & 1) - 1, 2 * (int)((oct >> 1) & 1) - 1, 2 * (int)(oct & 1) - 1);
		translate_warp<OP_M2M>(E.outer + gk * E.Nx2, t.cx[gk] - t.cx[g], t.cy[gk] - t.cy[g], t.cz[gk] - t.cz[g], d,
		                       acc, E.N, E.Nx2, sm[w], T, flags);
	}
	double2* out = E.outer + g * E.Nx2;
#pragma unroll
	for (int k = 0; k < CMAX; ++k) {
		int cc = lane + 32 * k;
		if (cc < E.Nx2) out[cc] = acc[k];
	}
}

// ---------------------------------------------------------------- M2L
// Far list of c: children of the parent's close cells and of the parent that
// are not adjacent to c (reference cpu/morton_tree.cpp:147-208), in that order.
__global__ void __launch_bounds__(WPB * 32) m2l_kernel(DevTree t, Exp E, int L, DevTables T, unsigned* flags)
{
	__shared__ Smem sm[WPB];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	size_t c = (size_t)blockIdx.x * WPB + w;
	if (c >= t.lsize[L]) return;
	size_t off = t.loff[L], poff = t.loff[L - 1];
	size_t g = off + c;
	int me[3];
	coords3(t.code[g], me);
	double2 acc[CMAX];
#pragma unroll
	for (int k = 0; k < CMAX; ++k) acc[k] = make_double2(0.0, 0.0);
	int32_t p = t.parent[g];
	int npc = t.close_cnt[poff + p];
	const int32_t* pl = t.close_idx + (poff + p) * t.close_stride;
	const double cx = t.cx[g], cy = t.cy[g], cz = t.cz[g];
	for (int e = 0; e <= npc; ++e) {
		int32_t pn = e < npc ? pl[e] : p;
		for (uint32_t k = t.beg[poff + pn]; k < t.end[poff + pn]; ++k) {
			if (k == c) continue;
			size_t gk = off + k;
			int o[3];
			coords3(t.code[gk], o);
			int dx = o[0] - me[0], dy = o[1] - me[1], dz = o[2] - me[2];
			if (max(max(abs(dx), abs(dy)), abs(dz)) <= 1) continue;
			translate_warp<OP_M2L>(E.outer + gk * E.Nx2, t.cx[gk] - cx, t.cy[gk] - cy, t.cz[gk] - cz,
			                       dir_id(dx, dy, dz), acc, E.N, E.Nx2, sm[w], T, flags);
		}
	}
	double2* out = E.inner + g * E.Nx2;
#pragma unroll
	for (int k = 0; k < CMAX; ++k) {
		int cc = lane + 32 * k;
		if (cc < E.Nx2) out[cc] = acc[k];
	}
}

// ---------------------------------------------------------------- L2L
__global__ void __launch_bounds__(WPB * 32) l2l_kernel(DevTree t, Exp E, int L, DevTables T, unsigned* flags)
{
	__shared__ Smem sm[WPB];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	size_t c = (size_t)blockIdx.x * WPB + w;
	if (c >= t.lsize[L]) return;
	size_t g = t.loff[L] + c;
	size_t gp = t.loff[L - 1] + t.parent[g];
	double2* out = E.inner + g * E.Nx2;
	double2 acc[CMAX];
#pragma unroll
	for (int k = 0; k < CMAX; ++k) {
		int cc = lane + 32 * k;
		acc[k] = cc < E.Nx2 ? out[cc] : make_double2(0.0, 0.0);
	}
	uint64_t oct = t.code[g] & 7ull;
	int d = dir_id(1 - 2 * (int)((oct >> 2) & 1), 1 - 2 * (int)((oct >> 1) & 1), 1 - 2 * (int)(oct & 1));
	translate_warp<OP_L2L>(E.inner + gp * E.Nx2, t.cx[gp] - t.cx[g], t.cy[gp] - t.cy[g], t.cz[gp] - t.cz[g], d, acc,
	                       E.N, E.Nx2, sm[w], T, flags);
#pragma unroll
	for (int k = 0; k < CMAX; ++k) {
		int cc = lane + 32 * k;
		if (cc < E.Nx2) out[cc] = acc[k];
	}
}

// Dense M2L operators of one level: column r of T_d is the rotation-based
// M2L (the same translate_warp as the per-pair path) applied to the r-th
// unit vector, for the far offset d * h.  out: [343][MT][MT], pre-zeroed.
__global__ void __launch_bounds__(WPB * 32) m2l_ops_kernel(int N, int MT, double h, DevTables T, double* out,
                                                           unsigned* flags)
{
	__shared__ Smem sm[WPB];
	__shared__ double2 unit[WPB][NX2MAX];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const int Nx2 = N * (N + 1) / 2, R = 2 * Nx2;
	size_t task = (size_t)blockIdx.x * WPB + w;
	int dirid = (int)(task / R), r = (int)(task % R);
	if (dirid >= 343) return;
	int dx = dirid / 49 - 3, dy = (dirid / 7) % 7 - 3, dz = dirid % 7 - 3;
	if (max(max(abs(dx), abs(dy)), abs(dz)) <= 1) return;
	for (int c = lane; c < Nx2; c += 32)
		unit[w][c] = make_double2(c == r / 2 && !(r & 1) ? 1.0 : 0.0, c == r / 2 && (r & 1) ? 1.0 : 0.0);
	__syncwarp();
	double2 acc[CMAX];
#pragma unroll
	for (int k = 0; k < CMAX; ++k) acc[k] = make_double2(0.0, 0.0);
	translate_warp<OP_M2L>(unit[w], dx * h, dy * h, dz * h, dirid, acc, N, Nx2, sm[w], T, flags);
	double* op = out + (size_t)dirid * MT * MT;
#pragma unroll
	for (int k = 0; k < CMAX; ++k) {
		int c = lane + 32 * k;
		if (c < Nx2) {
			op[(size_t)(2 * c) * MT + r] = acc[k].x;
			op[(size_t)(2 * c + 1) * MT + r] = acc[k].y;
		}
	}
}

} // namespace

int m2l_ops_build(Context& ctx, int N, double h, double* out)
{
	const int MT = m2l_padded(N), R = N * (N + 1);
	LFMM_CUDA(ctx, cudaMemsetAsync(out, 0, m2l_ops_bytes(N), ctx.stream));
	m2l_ops_kernel<<<div_up((size_t)343 * R, WPB), WPB * 32, 0, ctx.stream>>>(N, MT, h, ctx.tables.d, out,
	                                                                          ctx.dev_flags);
	LFMM_CUDA(ctx, cudaGetLastError());
	return OK;
}

double* m2l_ops_fp64(Context& ctx, int N, double h)
{
	for (auto& e : ctx.opcache)
		if (e.N == N && e.prec == 0 && e.h == h) { e.stamp = ++ctx.opcache_clock; return static_cast<double*>(e.ptr); }
	opcache_make_room(ctx);
	OpCacheEntry e;
	e.N = N; e.prec = 0; e.h = h; e.bytes = m2l_ops_bytes(N); e.stamp = ++ctx.opcache_clock;
	if (cudaMalloc(&e.ptr, e.bytes) != cudaSuccess) { cudaGetLastError(); ctx.last_error = "m2l operators: out of memory"; return nullptr; }
	if (m2l_ops_build(ctx, N, h, static_cast<double*>(e.ptr))) { cudaFree(e.ptr); return nullptr; }
	ctx.opcache.push_back(e);
	return static_cast<double*>(e.ptr);
}

int fmm3d_solve_device(Context& ctx, const ParticleInput& in, int N, int depth, double* pot, double* field,
                       SolveStats* stats, DevTree* tree_out)
{
	if (N < 1 || N > MAXN3) { ctx.last_error = "order out of range (1 <= N <= 18)"; return ERR_ARG; }
	int st;
	cudaStream_t s = ctx.stream;
	const bool timing = ctx.timing != 0;
	if (timing) LFMM_CUDA(ctx, cudaEventRecord(ctx.ev[0], s));
	DevTree t;
	st = tree_build(ctx, in, depth, t);
	if (st) return st;
	if (timing) LFMM_CUDA(ctx, cudaEventRecord(ctx.ev[1], s));
	Exp E;
	E.N = N; E.Nx2 = N * (N + 1) / 2;
	E.outer = static_cast<double2*>(ctx.arena.take(sizeof(double2) * t.ncells * E.Nx2));
	E.inner = static_cast<double2*>(ctx.arena.take(sizeof(double2) * t.ncells * E.Nx2));
	unsigned long long* counters = static_cast<unsigned long long*>(ctx.arena.take(32));
	if (!E.outer || !E.inner || !counters) { ctx.last_error = "fmm3d: device allocation failed"; return ERR_OOM; }
	const int LL = depth - 1;
	const size_t n_out = in.nt ? in.nt : in.ns;
	LFMM_CUDA(ctx, cudaMemsetAsync(pot, 0, sizeof(double) * n_out, s));
	LFMM_CUDA(ctx, cudaMemsetAsync(field, 0, sizeof(double) * 3 * n_out, s));
	size_t lo = depth > 2 ? t.loff[2] : t.ncells;
	LFMM_CUDA(ctx, cudaMemsetAsync(E.inner, 0, sizeof(double2) * lo * E.Nx2, s));
	// upward
	if (depth > 2)                         // no far pairs on levels 0 and 1
		if ((st = plain_p2m(ctx, t, N, E.outer))) return st;
	// factored translations unless the per-pair rotations are asked for; the
	// upward pass ends at level 2, the coarsest with far pairs
	const bool rot = ctx.m2l_engine != 1;
	const double* ax = nullptr;
	if (rot && depth > 2) {
		double h[MAX_LEVELS];
		for (int L = 0; L < depth; ++L) h[L] = t.geo_host[3] / (double)(1ull << L);
		if (!(ax = rot_axial_tables(ctx, N, h, depth, false))) return ERR_OOM;
	}
	auto flat = [&](double2* e, int L) { return reinterpret_cast<double*>(e + t.loff[L] * E.Nx2); };
	for (int L = depth - 2; L >= 2; --L) {
		if (rot) {
			M2LPlan mp;
			if ((st = m2m_plan_build(ctx, t, L, mp))) return st;
			if ((st = rot_translate<double>(ctx, ROT_M2M, mp, flat(E.outer, L + 1), flat(E.outer, L), N,
			                                rot_axial_level(ax, N, L))))
				return st;
		} else {
			m2m_kernel<<<div_up(t.lsize[L], WPB), WPB * 32, 0, s>>>(t, E, L, ctx.tables.d, ctx.dev_flags);
		}
	}
	if (timing) LFMM_CUDA(ctx, cudaEventRecord(ctx.ev[2], s));
	// downward
	std::vector<M2LPlan> plans(depth);
	for (int L = 2; L < depth; ++L) {
		if (rot) {
			if ((st = m2l_plan_build(ctx, t, L, plans[L]))) return st;
			if (m2l_dense64(N, t.lsize[L])) {
				const double* ops = m2l_ops_fp64(ctx, N, t.geo_host[3] / (double)(1ull << L));
				if (!ops) return ERR_OOM;
				st = m2l_gemm64(ctx, plans[L], ops, flat(E.outer, L), flat(E.inner, L), N);
			} else {
				st = rot_translate<double>(ctx, ROT_M2L, plans[L], flat(E.outer, L), flat(E.inner, L), N,
				                           rot_axial_level(ax, N, L));
			}
			if (st) return st;
		} else {
			m2l_kernel<<<div_up(t.lsize[L], WPB), WPB * 32, 0, s>>>(t, E, L, ctx.tables.d, ctx.dev_flags);
		}
	}
	if (timing) LFMM_CUDA(ctx, cudaEventRecord(ctx.ev[3], s));
	for (int L = 3; L < depth; ++L) {
		if (rot) {
			// the level's cells grouped by octant (its M2L plan), one slot: the parent
			M2LPlan lp = plans[L];
			lp.vtab = t.parent + t.loff[L];
			if ((st = rot_translate<double>(ctx, ROT_L2L, lp, flat(E.inner, L - 1), flat(E.inner, L), N,
			                                rot_axial_level(ax, N, L))))
				return st;
		} else {
			l2l_kernel<<<div_up(t.lsize[L], WPB), WPB * 32, 0, s>>>(t, E, L, ctx.tables.d, ctx.dev_flags);
		}
	}
	if (timing) LFMM_CUDA(ctx, cudaEventRecord(ctx.ev[4], s));
	if ((st = plain_leaves(ctx, t, N, depth > 2 ? E.inner : nullptr, pot, field))) return st;
	if (timing) LFMM_CUDA(ctx, cudaEventRecord(ctx.ev[5], s));
	LFMM_CUDA(ctx, cudaGetLastError());
	if (stats) {
		unsigned long long h[3];
		if ((st = tree_count_pairs(ctx, t, counters, h))) return st;
		stats->N = N; stats->depth = depth;
		stats->n_particles = t.n; stats->n_cells = t.ncells; stats->n_leaves = t.lsize[LL];
		stats->targets_num = t.targets_num;
		stats->n_far_pairs = h[0]; stats->n_close_pairs = h[1]; stats->n_p2p_pairs = h[2];
		if (timing) {
			cudaEventElapsedTime(&stats->ms_tree, ctx.ev[0], ctx.ev[1]);
			cudaEventElapsedTime(&stats->ms_upward, ctx.ev[1], ctx.ev[2]);
			cudaEventElapsedTime(&stats->ms_m2l, ctx.ev[2], ctx.ev[3]);
			cudaEventElapsedTime(&stats->ms_l2l, ctx.ev[3], ctx.ev[4]);
			cudaEventElapsedTime(&stats->ms_leaves, ctx.ev[4], ctx.ev[5]);
			cudaEventElapsedTime(&stats->ms_total, ctx.ev[0], ctx.ev[5]);
		}
	}
	if (tree_out) *tree_out = t;
	return OK;
}

} // namespace lfmm
