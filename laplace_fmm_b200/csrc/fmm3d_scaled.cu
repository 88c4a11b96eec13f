// 3D FMM in scaled expansions on the adaptive-form tree (uniform when
// max_leaf = 0): plain FP64 or mixed (FP32 expansions and near field, FP64
// M2L accumulation on levels 2-3, FP64 tile sums and self term).
// Passes: P2M (every leaf, any level) -> M2M -> M2L (V) ->
// P2L (X) -> L2L -> leaves: P2P (self + U), M2P (W), L2P.
#include <cmath>
#include "far_kernels.cuh"
#include "m2l_tc.cuh"
#include "rot.cuh"
#include <algorithm>
#include <mutex>
#include <type_traits>

namespace lfmm {

using namespace scaled;

namespace {

std::mutex g_const_mu;
bool g_scaled_const_ready[64] = {};

int upload_scaled_constants(Context& ctx)
{
	std::lock_guard<std::mutex> lock(g_const_mu);
	if (ctx.device < 0 || ctx.device >= 64) { ctx.last_error = "device index above 63"; return ERR_ARG; }
	if (g_scaled_const_ready[ctx.device]) return OK;
	float2 rec_f[NXD];
	double2 rec_d[NXD];
	GradF grad_f[2][NXD];
	GradD grad_d[2][NXD];
	for (int n = 0; n <= MAXN3; ++n)
		for (int m = 0; m <= n; ++m) {
			const int i = tix(n, m);
			const double d1 = (double)(n + 1) * (n + 1) - (double)m * m;
			rec_d[i] = make_double2((2.0 * n + 1.0) / std::sqrt(d1), std::sqrt(((double)n * n - (double)m * m) / d1));
			rec_f[i] = make_float2((float)rec_d[i].x, (float)rec_d[i].y);
			const double z[2] = {(n + 1.0 - m) * (n + 1 + m), std::max((n - m) * (n + m), 0) * 1.0};
			const double p[2] = {(n + 2.0 - m) * (n + 1 - m), std::max((n + m - 1) * (n + m), 0) * 1.0};
			const double q[2] = {(n + 2.0 + m) * (n + 1 + m), std::max((n - m - 1) * (n - m), 0) * 1.0};
			for (int k = 0; k < 2; ++k) {
				grad_d[k][i] = GradD{std::sqrt(z[k]), std::sqrt(p[k]), std::sqrt(q[k]), n | m << 8};
				grad_f[k][i] = GradF{(float)grad_d[k][i].z, (float)grad_d[k][i].p, (float)grad_d[k][i].m, n | m << 8};
			}
		}
	double S_d[MAXN3 + 1];
	float S_f[MAXN3 + 1];
	S_d[0] = 1.0;
	for (int m = 1; m <= MAXN3; ++m) S_d[m] = -S_d[m - 1] * std::sqrt((2.0 * m - 1.0) / (2.0 * m));
	for (int m = 0; m <= MAXN3; ++m) S_f[m] = (float)S_d[m];
	LFMM_CUDA(ctx, cudaMemcpyToSymbol(g_rec_f, rec_f, sizeof(rec_f)));
	LFMM_CUDA(ctx, cudaMemcpyToSymbol(g_rec_d, rec_d, sizeof(rec_d)));
	LFMM_CUDA(ctx, cudaMemcpyToSymbol(g_grad_f, grad_f, sizeof(grad_f)));
	LFMM_CUDA(ctx, cudaMemcpyToSymbol(g_grad_d, grad_d, sizeof(grad_d)));
	LFMM_CUDA(ctx, cudaMemcpyToSymbol(g_S_f, S_f, sizeof(S_f)));
	LFMM_CUDA(ctx, cudaMemcpyToSymbol(g_S_d, S_d, sizeof(S_d)));
	LFMM_CUDA(ctx, constants_ready());
	g_scaled_const_ready[ctx.device] = true;
	return OK;
}

// Dense FP64 scaled M2M operators, one per child octant o (the octant bits
// of the child's code): column r is translate_scaled applied to the r-th unit
// vector.  out: [8][MT][MT], pre-zeroed.
__global__ void __launch_bounds__(WPB * 32) m2m_ops_kernel(int N, int MT, DevTables T, double* __restrict__ out,
                                                           unsigned* flags)
{
	__shared__ ShiftSmem sm[WPB];
	__shared__ double2 unit[WPB][NX2MAX];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const int Nx2 = N * (N + 1) / 2, R = 2 * Nx2;
	const size_t task = (size_t)blockIdx.x * WPB + w;
	const int o = (int)(task / R), r = (int)(task % R);
	if (o >= 8) return;
	const int bx = (o >> 2) & 1, by = (o >> 1) & 1, bz = o & 1;
	const int d = dir_id(2 * bx - 1, 2 * by - 1, 2 * bz - 1);
	for (int c = lane; c < Nx2; c += 32)
		unit[w][c] = make_double2(c == r / 2 && !(r & 1) ? 1.0 : 0.0, c == r / 2 && (r & 1) ? 1.0 : 0.0);
	__syncwarp();
	double2 acc[CMAX];
#pragma unroll
	for (int k = 0; k < CMAX; ++k) acc[k] = make_double2(0.0, 0.0);
	translate_scaled(unit[w], d, acc, N, Nx2, sm[w], T, flags);
	double* op = out + (size_t)o * MT * MT;
#pragma unroll
	for (int k = 0; k < CMAX; ++k) {
		const int c = lane + 32 * k;
		if (c < Nx2) {
			op[(size_t)(2 * c) * MT + r] = acc[k].x;
			op[(size_t)(2 * c + 1) * MT + r] = acc[k].y;
		}
	}
}

// The tensor-core M2M operators of order N, cached in the context (built
// once; the plan's warm solves build them before capture).  nullptr on
// failure, with st = ERR_OOM or ERR_CUDA.
const uint4* m2m_ops_tc(Context& ctx, int N, int& st)
{
	st = OK;
	constexpr int tag = 30;
	for (auto& e : ctx.opcache)
		if (e.N == N && e.prec == tag) { e.stamp = ++ctx.opcache_clock; return static_cast<const uint4*>(e.ptr); }
	const int MT = m2l_padded(N), R = N * (N + 1);
	const size_t bytes64 = sizeof(double) * 8 * (size_t)MT * MT;
	const size_t bytes_tc = tc_ops_bytes(8, N);
	opcache_make_room(ctx);
	double* d = nullptr;
	void* tc = nullptr;
	if (cudaMalloc(&d, bytes64) != cudaSuccess || cudaMalloc(&tc, bytes_tc) != cudaSuccess) {
		cudaGetLastError();
		if (d) cudaFree(d);
		ctx.last_error = "M2M operators: out of memory";
		st = ERR_OOM;
		return nullptr;
	}
	cudaMemsetAsync(d, 0, bytes64, ctx.stream);
	m2m_ops_kernel<<<div_up((size_t)8 * R, WPB), WPB * 32, 0, ctx.stream>>>(N, MT, ctx.tables.d, d,
	                                                                        ctx.dev_flags);
	st = cudaGetLastError() == cudaSuccess ? tc_ops_convert(ctx, d, 8, N, tc) : ERR_CUDA;
	if (cudaStreamSynchronize(ctx.stream) != cudaSuccess) st = ERR_CUDA;
	cudaFree(d);
	if (st != OK) {
		cudaFree(tc);
		ctx.last_error = "M2M operators: build failed";
		return nullptr;
	}
	OpCacheEntry e;
	e.N = N; e.prec = tag; e.h = 1.0; e.bytes = bytes_tc;
	e.stamp = ++ctx.opcache_clock; e.ptr = tc;
	ctx.opcache.push_back(e);
	return static_cast<const uint4*>(tc);
}

// Levels of the mixed form's FP32 expansions that take the factored FP64
// translations instead of the tensor-core engine (B200, rot_kernel against
// m2l_tc_kernel, us).  M2L: a tensor-core launch costs 105-240 (N = 8-18) on
// the smallest levels, where its 128-target tiles are mostly empty; the
// factored one 20-105 up to 150 cells, 46 / 94 / 187 / 256 (N = 8 / 12 / 16 /
// 18) at 300-512 cells, 136 / 298 / 615 / 837 at 1341, against 142 / 172 / 240
// / 306 for the tensor cores: the line lies at 512.  M2M at N = 16: 51 / 61 /
// 87 / 90 at 55 / 1341 / 4169 / 4096 cells against 82-136, but 625 against
// 281 at 32,768.
constexpr size_t ROT_M2L_CELLS = 512, ROT_M2M_CELLS = 6144;

// Instances of the chain kernels by the steps of their busiest lane.
template <typename F>
void by_steps(int N, F go)
{
	if (N <= 8) go(std::integral_constant<int, 8>());
	else if (N <= 12) go(std::integral_constant<int, 12>());
	else if (N <= 16) go(std::integral_constant<int, 17>());
	else if (N <= 17) go(std::integral_constant<int, 20>());
	else go(std::integral_constant<int, 23>());
}

// P2M of every leaf.
template <typename real>
void launch_p2m(Context& ctx, const DevTree& t, int N, typename V2<real>::t* outer)
{
	by_steps(N, [&](auto st_) {
		p2m_scaled_kernel<real, decltype(st_)::value>
			<<<std::min(div_up(t.nleaves, FWPB), 8u * (unsigned)ctx.num_sms), FWPB * 32, 0, ctx.stream>>>(t, N, outer);
	});
}

// P2L of every X list.
template <typename real>
int launch_p2l(Context& ctx, const DevTree& t, int N, typename V2<real>::t* inner)
{
	cudaStream_t s = ctx.stream;
	// counter, list of longs, list of shorts (at most one cell per entry)
	const size_t nlong = t.n_x / FAR_SHORT + 1;
	uint32_t* next = static_cast<uint32_t*>(ctx.arena.take(sizeof(uint32_t) * (nlong + t.n_x + 3)));
	if (!next) { ctx.last_error = "scaled solve: allocation failed"; return ERR_OOM; }
	uint32_t *longs = next + 1, *shorts = longs + 1 + nlong;
	LFMM_CUDA(ctx, cudaMemsetAsync(next, 0, 2 * sizeof(uint32_t), s));
	LFMM_CUDA(ctx, cudaMemsetAsync(shorts, 0, sizeof(uint32_t), s));
	x_select_kernel<<<div_up(t.ncells, 256), 256, 0, s>>>(t, shorts, longs);
	by_steps(N, [&](auto st_) {
		p2l_kernel<real, decltype(st_)::value><<<8 * ctx.num_sms, FWPB * 32, 0, s>>>(t, N, inner, next, shorts);
		p2l_long_kernel<real, decltype(st_)::value><<<2 * ctx.num_sms, FWL * 32, 0, s>>>(t, N, inner, longs);
	});
	LFMM_CUDA(ctx, cudaGetLastError());
	return OK;
}

// The dense FP64 M2L of a level (m2l_dense64); FP32 expansions are widened
// into scratch and rounded back.
template <typename real>
int dense64(Context& ctx, const M2LPlan& plan, const real* mult, real* loc, int N)
{
	const double* ops = m2l_ops_fp64(ctx, N, 1.0);
	if (!ops) return ERR_OOM;
	if constexpr (sizeof(real) == sizeof(double)) {
		return m2l_gemm64(ctx, plan, ops, mult, loc, N);
	} else {
		const size_t n = plan.cells * (size_t)N * (N + 1);
		double* m = static_cast<double*>(ctx.arena.take(sizeof(double) * n));
		double* l = static_cast<double*>(ctx.arena.take(sizeof(double) * n));
		if (!m || !l) { ctx.last_error = "scaled solve: allocation failed"; return ERR_OOM; }
		convert_kernel<<<div_up(n, 256), 256, 0, ctx.stream>>>(mult, m, n);
		if (int st = m2l_gemm64(ctx, plan, ops, m, l, N)) return st;
		convert_kernel<<<div_up(n, 256), 256, 0, ctx.stream>>>(l, loc, n);
		LFMM_CUDA(ctx, cudaGetLastError());
		return OK;
	}
}

template <typename real>
int solve_t(Context& ctx, const DevTree& t, int N, double* pot, double* field, SolveStats* stats,
            const int* level_N)
{
	using v2 = typename V2<real>::t;
	cudaStream_t s = ctx.stream;
	const bool timing = ctx.timing != 0;
	const int Nx2 = N * (N + 1) / 2;
	const size_t C = t.ncells;
	v2* outer = static_cast<v2*>(ctx.arena.take(sizeof(v2) * C * Nx2));
	v2* inner = static_cast<v2*>(ctx.arena.take(sizeof(v2) * C * Nx2));
	const bool coarse64 = sizeof(real) == sizeof(float);
	if (!outer || !inner) {
		ctx.last_error = "scaled solve: allocation failed";
		return ERR_OOM;
	}
	const size_t n_out = t.nt ? t.nt : t.n - t.nt;
	LFMM_CUDA(ctx, cudaMemsetAsync(pot, 0, sizeof(double) * n_out, s));
	LFMM_CUDA(ctx, cudaMemsetAsync(field, 0, sizeof(double) * 3 * n_out, s));
	LFMM_CUDA(ctx, cudaMemsetAsync(outer, 0, sizeof(v2) * C * Nx2, s));
	LFMM_CUDA(ctx, cudaMemsetAsync(inner, 0, sizeof(v2) * C * Nx2, s));
	const unsigned resident = 8u * (unsigned)ctx.num_sms;
	if (t.depth > 2) launch_p2m<real>(ctx, t, N, outer);   // multipoles below level 2 reach nothing
	int st;
	// the tensor-core engine on the FP32 expansions' larger levels (M2L; M2M
	// through dense scaled operators, one per child octant)
	const bool tc = sizeof(real) == sizeof(float) && ctx.m2l_engine == 3 && m2l_tc_supported(N);
	// every other translation (the FP64 form's, the mixed form's L2L, the M2L of
	// its levels 2 and 3, its small levels) goes through the factored FP64
	// engine; the upward pass ends at level 2, the coarsest whose multipoles
	// anything reads
	const double unit_h = 1.0;
	const double* ax = t.depth > 2 ? rot_axial_tables(ctx, N, &unit_h, 1, true) : nullptr;
	if (t.depth > 2 && !ax) return ERR_OOM;
	auto flat = [&](v2* e, int L) { return reinterpret_cast<real*>(e + t.loff[L] * Nx2); };
	for (int L = t.depth - 2; L >= 2; --L) {
		if (t.lsize[L] == 0) continue;
		M2LPlan mp;
		if ((st = m2m_plan_build(ctx, t, L, mp))) return st;
		if (tc && t.lsize[L] > ROT_M2M_CELLS) {
			const uint4* mops = m2m_ops_tc(ctx, N, st);
			if (!mops) return st;
			st = m2m_gemm_tc(ctx, mp, mops, reinterpret_cast<const float*>(outer + t.loff[L + 1] * Nx2),
			                 reinterpret_cast<float*>(outer + t.loff[L] * Nx2), N, t.lsize[L + 1]);
		} else {
			st = rot_translate<real>(ctx, ROT_M2M, mp, flat(outer, L + 1), flat(outer, L), N, ax);
		}
		if (st) return st;
	}
	if (timing) LFMM_CUDA(ctx, cudaEventRecord(ctx.ev[2], s));
	std::vector<M2LPlan> plans(t.depth);
	if (t.depth > 2) {
		for (int L = 2; L < t.depth; ++L) {
			if (t.lsize[L] == 0) continue;
			M2LPlan& plan = plans[L];
			if ((st = m2l_plan_build(ctx, t, L, plan))) return st;
			const real* mL = reinterpret_cast<const real*>(outer + t.loff[L] * Nx2);
			real* lL = reinterpret_cast<real*>(inner + t.loff[L] * Nx2);
			// a level's own source order (level_N) is the tensor-core engine's
			const bool own_n = level_N && level_N[L] > 0 && level_N[L] < N;
			if (!coarse64 || L <= 3 || (tc && t.lsize[L] <= ROT_M2L_CELLS && !own_n)) {
				if (m2l_dense64(N, t.lsize[L])) {
					if ((st = dense64<real>(ctx, plan, mL, lL, N))) return st;
				} else if ((st = rot_translate<real>(ctx, ROT_M2L, plan, mL, lL, N, ax))) {
					return st;
				}
			} else if (tc) {
				// tcgen05 hi/lo GEMM on the FP32 levels (FP16 or TF32 operands)
				float t_inv = 1.f;
				const uint4* tc = m2l_ops_tc(ctx, N, &t_inv);
				if (!tc) return ERR_OOM;
				if ((st = m2l_gemm_tc(ctx, plan, tc, reinterpret_cast<const float*>(mL), reinterpret_cast<float*>(lL), N,
				                      level_N ? level_N[L] : 0, t_inv)))
					return st;
			} else {
				const float* ops = m2l_ops_fp32(ctx, N);
				if (!ops) return ERR_OOM;
				if ((st = m2l_gemm(ctx, plan, ops, reinterpret_cast<const float*>(mL), reinterpret_cast<float*>(lL), N)))
					return st;
			}
		}
	}
	if (t.adaptive && t.n_x > 0 && (st = launch_p2l<real>(ctx, t, N, inner))) return st;
	if (timing) LFMM_CUDA(ctx, cudaEventRecord(ctx.ev[3], s));
	for (int L = 3; L < t.depth; ++L) {
		if (t.lsize[L] == 0) continue;
		// the level's cells grouped by octant (its M2L plan), one slot: the parent
		M2LPlan lp = plans[L];
		lp.vtab = t.parent + t.loff[L];
		st = rot_translate<real>(ctx, ROT_L2L, lp, flat(inner, L - 1), flat(inner, L), N, ax);
		if (st) return st;
	}
	if (timing) LFMM_CUDA(ctx, cudaEventRecord(ctx.ev[4], s));
	// the near field, then the expansions added onto it: resident grids taking
	// leaves from a counter
	uint32_t* next = static_cast<uint32_t*>(ctx.arena.take(sizeof(uint32_t) * (5 + t.n_w / FAR_SHORT)));
	if (!next) { ctx.last_error = "scaled solve: allocation failed"; return ERR_OOM; }
	uint32_t* longs = next + 3;
	LFMM_CUDA(ctx, cudaMemsetAsync(next, 0, 4 * sizeof(uint32_t), s));
	constexpr int LWP = 4;
	if constexpr (sizeof(real) == sizeof(float))
		p2p_f32_kernel<LWP><<<6 * ctx.num_sms, LWP * 32, 0, s>>>(t, pot, field, next);
	else
		p2p_f64_kernel<LWP><<<resident, LWP * 32, 0, s>>>(t, pot, field, next);
	const size_t sm_e = eval_smem<real>(FWPB, N), sm_l = eval_smem<real>(FWL, N);
	LFMM_CUDA(ctx, smem_limit(ctx.device, reinterpret_cast<const void*>(eval_scaled_kernel<real>), eval_smem<real>(FWPB, MAXN3)));
	LFMM_CUDA(ctx, smem_limit(ctx.device, reinterpret_cast<const void*>(eval_long_kernel<real>), eval_smem<real>(FWL, MAXN3)));
	eval_scaled_kernel<real><<<resident, FWPB * 32, sm_e, s>>>(t, outer, inner, N, pot, field, next + 1, longs);
	if (t.n_w > FAR_SHORT)
		eval_long_kernel<real><<<2 * ctx.num_sms, FWL * 32, sm_l, s>>>(t, outer, inner, N, pot, field, next + 2, longs);
	if (timing) LFMM_CUDA(ctx, cudaEventRecord(ctx.ev[5], s));
	LFMM_CUDA(ctx, cudaGetLastError());
	(void)stats;
	return OK;
}

} // namespace

// P2M of one leaf, or P2L of one cell, from the sources of n_lists lists (P2M:
// one list), given in the scaled frame of the leaf or cell; out: the N (N + 1) / 2
// coefficients (re, im), widened to FP64.
template <typename real>
int debug_leaf_sums(Context& ctx, bool irregular, int N, size_t n_lists, const size_t* off, const double* xyz,
                    const double* q, double* out)
{
	using v2 = typename V2<real>::t;
	if (int st = upload_scaled_constants(ctx)) return st;
	cudaStream_t s = ctx.stream;
	const size_t n = off[n_lists], C = n_lists + 1, Nx2 = (size_t)N * (N + 1) / 2;
	// cell 0: the leaf or cell, of size 1 about the origin; cells 1 ..: the lists
	std::vector<double> xs(4 * n);
	for (size_t i = 0; i < n; ++i) { for (int d = 0; d < 3; ++d) xs[d * n + i] = xyz[3 * i + d]; xs[3 * n + i] = q[i]; }
	std::vector<uint32_t> u(2 * C + C + 1);
	std::vector<int32_t> idx(C);
	u[0] = 0; u[C] = (uint32_t)n;
	for (size_t k = 1; k < C; ++k) { u[k] = (uint32_t)off[k - 1]; u[C + k] = (uint32_t)off[k]; idx[k - 1] = (int32_t)k; }
	for (size_t k = 0; k <= C; ++k) u[2 * C + k] = k ? (uint32_t)n_lists : 0u;
	ctx.arena.reset();
	double* x = static_cast<double*>(ctx.arena.take(sizeof(double) * (4 * n + 3)));
	uint32_t* du = static_cast<uint32_t*>(ctx.arena.take(sizeof(uint32_t) * u.size()));
	int32_t* di = static_cast<int32_t*>(ctx.arena.take(sizeof(int32_t) * (C + 1)));
	uint8_t* lev = static_cast<uint8_t*>(ctx.arena.take(C));
	v2* e = static_cast<v2*>(ctx.arena.take(sizeof(v2) * Nx2));
	if (!x || !du || !di || !lev || !e) { ctx.last_error = "leaf sums: allocation failed"; return ERR_OOM; }
	LFMM_CUDA(ctx, cudaMemcpyAsync(x, xs.data(), sizeof(double) * xs.size(), cudaMemcpyHostToDevice, s));
	LFMM_CUDA(ctx, cudaMemsetAsync(x + 4 * n, 0, 3 * sizeof(double), s));
	LFMM_CUDA(ctx, cudaMemcpyAsync(du, u.data(), sizeof(uint32_t) * u.size(), cudaMemcpyHostToDevice, s));
	LFMM_CUDA(ctx, cudaMemcpyAsync(di, idx.data(), sizeof(int32_t) * C, cudaMemcpyHostToDevice, s));
	LFMM_CUDA(ctx, cudaMemsetAsync(di + C, 0, sizeof(int32_t), s));
	LFMM_CUDA(ctx, cudaMemsetAsync(lev, 0, C, s));
	LFMM_CUDA(ctx, cudaMemsetAsync(e, 0, sizeof(v2) * Nx2, s));
	DevTree t;
	t.n = n; t.ncells = 1; t.nleaves = 1; t.adaptive = true; t.n_x = n_lists; t.geo_host[3] = 1.0;
	t.x = x; t.y = x + n; t.z = x + 2 * n; t.q = x + 3 * n;
	t.cx = x + 4 * n; t.cy = x + 4 * n + 1; t.cz = x + 4 * n + 2;
	t.pbeg = du; t.send = du + C; t.x_off = du + 2 * C; t.x_idx = di; t.leaves = di + C; t.lev = lev;
	if (irregular) {
		if (int st = launch_p2l<real>(ctx, t, N, e)) return st;
	} else {
		launch_p2m<real>(ctx, t, N, e);
	}
	std::vector<v2> h(Nx2);
	LFMM_CUDA(ctx, cudaMemcpyAsync(h.data(), e, sizeof(v2) * Nx2, cudaMemcpyDeviceToHost, s));
	LFMM_CUDA(ctx, cudaStreamSynchronize(s));
	for (size_t c = 0; c < Nx2; ++c) { out[2 * c] = h[c].x; out[2 * c + 1] = h[c].y; }
	ctx.arena.settle();
	return OK;
}

int plain_p2m(Context& ctx, const DevTree& t, int N, double2* outer)
{
	if (int st = upload_scaled_constants(ctx)) return st;
	by_steps(N, [&](auto st_) {
		p2m_plain_kernel<decltype(st_)::value>
			<<<div_up(t.lsize[t.depth - 1], FWPB), FWPB * 32, 0, ctx.stream>>>(t, N, outer);
	});
	LFMM_CUDA(ctx, cudaGetLastError());
	return OK;
}

int plain_leaves(Context& ctx, const DevTree& t, int N, const double2* inner, double* pot, double* field)
{
	if (int st = upload_scaled_constants(ctx)) return st;
	const unsigned nl = (unsigned)t.lsize[t.depth - 1];
	const dim3 grid(nl, std::min(64u, std::max(1u, 4u * (unsigned)ctx.num_sms / nl)));
	const size_t smem = eval_smem<double>(1, N);
	if (inner)
		leaves_plain_kernel<true><<<grid, FWL * 32, smem, ctx.stream>>>(t, inner, N, pot, field);
	else
		leaves_plain_kernel<false><<<grid, FWL * 32, 0, ctx.stream>>>(t, inner, N, pot, field);
	LFMM_CUDA(ctx, cudaGetLastError());
	return OK;
}

template int debug_leaf_sums<float>(Context&, bool, int, size_t, const size_t*, const double*, const double*, double*);
template int debug_leaf_sums<double>(Context&, bool, int, size_t, const size_t*, const double*, const double*, double*);

float* m2l_ops_fp32(Context& ctx, int N)
{
	for (auto& e : ctx.opcache)
		if (e.N == N && e.prec == 1) { e.stamp = ++ctx.opcache_clock; return static_cast<float*>(e.ptr); }
	const size_t bytes = m2l_ops_bytes(N), cnt = bytes / sizeof(double);
	opcache_make_room(ctx);
	OpCacheEntry e;
	e.N = N; e.prec = 1; e.h = 1.0; e.bytes = cnt * sizeof(float); e.stamp = ++ctx.opcache_clock;
	double* d = nullptr;
	if (cudaMalloc(&d, bytes) != cudaSuccess || cudaMalloc(&e.ptr, e.bytes) != cudaSuccess) {
		cudaGetLastError();
		cudaFree(d);
		ctx.last_error = "m2l operators: out of memory";
		return nullptr;
	}
	bool ok = m2l_ops_build(ctx, N, 1.0, d) == OK;
	if (ok) {
		convert_kernel<<<div_up(cnt, 256), 256, 0, ctx.stream>>>(d, static_cast<float*>(e.ptr), cnt);
		ok = cudaStreamSynchronize(ctx.stream) == cudaSuccess;
	}
	cudaFree(d);
	if (!ok) {
		cudaFree(e.ptr);
		ctx.last_error = "m2l operators: build failed";
		return nullptr;
	}
	ctx.opcache.push_back(e);
	return static_cast<float*>(e.ptr);
}

int fmm3d_solve_scaled(Context& ctx, const ParticleInput& in, int N, int depth, int max_leaf, int precision,
                       double* pot, double* field, SolveStats* stats, DevTree* tree_out, const int* level_N)
{
	if (N < 1 || N > MAXN3) { ctx.last_error = "order out of range (1 <= N <= 18)"; return ERR_ARG; }
	if (!m2l_gemm_supported(N)) { ctx.last_error = "scaled / mixed / adaptive forms support N <= 18"; return ERR_UNSUPPORTED; }
	if (max_leaf < 0) { ctx.last_error = "max_leaf must be >= 0"; return ERR_ARG; }
	int st = upload_scaled_constants(ctx);
	if (st) return st;
	cudaStream_t s = ctx.stream;
	const bool timing = ctx.timing != 0;
	ctx.kev_used = 0;
	if (timing) LFMM_CUDA(ctx, cudaEventRecord(ctx.ev[0], s));
	DevTree t;
	if ((st = tree_build_adaptive(ctx, in, depth, max_leaf, t))) return st;
	if (timing) LFMM_CUDA(ctx, cudaEventRecord(ctx.ev[1], s));
	if ((st = fmm3d_scaled_on_tree(ctx, t, N, precision, pot, field, stats, level_N))) return st;
	if (tree_out) *tree_out = t;
	return OK;
}

int fmm3d_scaled_on_tree(Context& ctx, const DevTree& t, int N, int precision, double* pot, double* field,
                         SolveStats* stats, const int* level_N)
{
	if (N < 1 || N > MAXN3 || !m2l_gemm_supported(N)) {
		ctx.last_error = "scaled / mixed / adaptive forms support N <= 18";
		return ERR_UNSUPPORTED;
	}
	int st = upload_scaled_constants(ctx);
	if (st) return st;
	const bool timing = ctx.timing != 0;
	st = precision == 1 ? solve_t<float>(ctx, t, N, pot, field, stats, level_N)
	                    : solve_t<double>(ctx, t, N, pot, field, stats, level_N);
	if (st) return st;
	if (stats) {
		unsigned long long h[4];
		if ((st = tree_adaptive_counts(ctx, t, h))) return st;
		stats->N = N; stats->depth = t.depth;
		stats->n_particles = t.n; stats->n_cells = t.ncells; stats->n_leaves = t.nleaves;
		stats->targets_num = t.targets_num;
		stats->n_far_pairs = h[0]; stats->n_close_pairs = h[1]; stats->n_p2p_pairs = h[2];
		stats->n_m2p = h[3]; stats->n_w = t.n_w; stats->n_x = t.n_x;
		if (timing) {
			cudaEventElapsedTime(&stats->ms_tree, ctx.ev[0], ctx.ev[1]);
			cudaEventElapsedTime(&stats->ms_upward, ctx.ev[1], ctx.ev[2]);
			cudaEventElapsedTime(&stats->ms_m2l, ctx.ev[2], ctx.ev[3]);
			cudaEventElapsedTime(&stats->ms_l2l, ctx.ev[3], ctx.ev[4]);
			cudaEventElapsedTime(&stats->ms_leaves, ctx.ev[4], ctx.ev[5]);
			cudaEventElapsedTime(&stats->ms_total, ctx.ev[0], ctx.ev[5]);
			for (int k = 0; k + 1 < ctx.kev_used; k += 2) {
				float ms = 0.f;
				cudaEventElapsedTime(&ms, ctx.kev[k], ctx.kev[k + 1]);
				stats->ms_m2l_kernel += ms;
				++stats->n_m2l_kernel;
			}
		}
	}
	return OK;
}

} // namespace lfmm
