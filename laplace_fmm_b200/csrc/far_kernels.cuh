// Particles to expansions (P2M, P2L) and expansions to particles (M2P, L2P)
// of the scaled-expansion solver, FP32 or FP64, through Cartesian solid
// harmonics; included only by fmm3d_scaled.cu.
//
// Orthonormal basis B_nm = r^n Y_nm (regular) and r^-(n+1) Y_nm (irregular),
// Y_nm = sqrt((n-m)!/(n+m)!) P_n^m(cos t) e^{i m phi} with the Condon-Shortley
// phase:
//   B_mm = S_m w^m B_00, w = x + iy (or w / r^2), B_00 = 1 (or 1/r),
//   S_m = prod_{k<=m} -sqrt((2k - 1) / (2k)),
//   B_{n+1,m} = a_nm z B_nm - b_nm r^2 B_{n-1,m}   (or (a z B_nm - b B_{n-1,m}) / r^2)
// with (a_nm, b_nm) = ((2n + 1) / sqrt((n+1)^2 - m^2), sqrt((n^2 - m^2) / ((n+1)^2 - m^2)));
// b_mm = 0 starts each order's chain.
#pragma once
#include "scaled_kernels.cuh"
#include <type_traits>

namespace lfmm {
namespace scaled {

// a, b at tix(n, m), n <= MAXN3; S_m; the gradient's factors at tix(n, k)
// (regular and irregular: d/dz, and the two neighbours of d/dx -+ i d/dy)
__device__ float2 g_rec_f[NXD];
__device__ double2 g_rec_d[NXD];
__device__ float g_S_f[MAXN3 + 1];
__device__ double g_S_d[MAXN3 + 1];
struct GradF { float z, p, m; int nk; };
struct GradD { double z, p, m; int nk; };
__device__ GradF g_grad_f[2][NXD];
__device__ GradD g_grad_d[2][NXD];
template <typename real> struct FarTab;
template <> struct FarTab<float> {
	using grad = GradF;
	static __device__ __forceinline__ float2 rec(int i) { return g_rec_f[i]; }
	static __device__ __forceinline__ float S(int m) { return g_S_f[m]; }
	static __device__ __forceinline__ GradF g(int irr, int i) { return g_grad_f[irr][i]; }
};
template <> struct FarTab<double> {
	using grad = GradD;
	static __device__ __forceinline__ double2 rec(int i) { return g_rec_d[i]; }
	static __device__ __forceinline__ double S(int m) { return g_S_d[m]; }
	static __device__ __forceinline__ GradD g(int irr, int i) { return g_grad_d[irr][i]; }
};

// FP64: the reference's spherical coordinates take r + 1e-12 as the radius and
// cos t = z / (r + 1e-12) (common/simple_math.h:101-117), which moves a point
// away from the z axis by rho'^2 = rho^2 + (2 r + 1e-12) 1e-12; the parity of
// the plain form's outputs at 1e-12 needs the same point here.  The scaled form
// moves its targets too (the vector form is held to the reference at 1e-12), by
// 1e-12 of the cell's size: a target exactly on the axis of its leaf or of a W
// cell is evaluated up to 1e-6 cells beside it (at N = 18 up to 8e-7 of the field
// at such a target of a clustered set, 6e-13 at the others).
__device__ __forceinline__ void reference_point(double& x, double& y, double z)
{
	constexpr double e = 1e-12;
	const double rho2 = x * x + y * y, d = (2.0 * sqrt(rho2 + z * z) + e) * e;
	if (fabs(x) + fabs(y) < e) { x = sqrt(rho2 + d); y = 0.0; return; }
	const double f = sqrt(1.0 + d / rho2);
	x *= f; y *= f;
}

// ---- P2M, P2L ------------------------------------------------------------
// Eight lanes per particle, four particles per warp.  Lane l runs the chains
// of the orders l, 15 - l and 16 + l one after another, so the coefficients
// spread over the lanes (N = 16: 17 steps each) and every sum stays in a
// register until the cell's last particle.  FP32 sums are compensated (Kahan):
// the leaves' rounding errors would add up over the whole far field, and the
// form before summed 32 particles in FP64 (orders 0 and 1) or in a tree.
// Against it, single coefficients of leaves of 8 to 96 and of X lists of 60 to
// 1,920 sources are off FP64 by 0.95 to 1.005 times as much (geometric means by
// order and degree).  FP32 takes two particles per lane group at once for the
// latencies of the compensation.
// Issue slots 60 % busy at 16 warps per SM, the rest the chains' own latencies.
// A lane-per-particle form that summed the lanes' values through shared memory
// took 840 M instructions and 1150 us for the P2L of 1,048,576 clustered
// particles at N = 16 (95.7k X entries), and 279 M for their P2M (this form: 416
// and 129 M).  Compensating every step, not only the first six, takes the P2M of
// 16.8M particles at N = 17 from 2.54 to 2.66 ms and their P2L from 5.2 to 5.9
// (P2M 3.14 with the totals of every step formed in every lane).
constexpr int CHL = 8;
// steps of the busiest lane (N = 17: 20, N = 18: 23)
__host__ __device__ constexpr int chain_steps(int N) { return N <= 15 ? N : N == 16 ? 17 : N == 17 ? 20 : 23; }

template <typename real> struct ChainTab {
	typename V2<real>::t ab[23 * CHL];
	int16_t out[23 * CHL];             // tix(n, m), or -1: past the lane's last chain
	real S[MAXN3 + 1];
};

// Filled by the whole block (nt threads); the caller synchronises.
template <typename real>
__device__ __forceinline__ void chain_tab_fill(ChainTab<real>& tb, int N, int tid, int nt)
{
	for (int e = tid; e < chain_steps(N) * CHL; e += nt) {
		const int s = e / CHL, l = e % CHL;
		const int l1 = max(N - l, 0), l2 = max(N - (15 - l), 0), l3 = max(N - (16 + l), 0);
		int m = -1, n = 0;
		if (s < l1) { m = l; n = l + s; }
		else if (s < l1 + l2) { m = 15 - l; n = m + s - l1; }
		else if (s < l1 + l2 + l3) { m = 16 + l; n = m + s - l1 - l2; }
		tb.ab[e] = m < 0 ? V2<real>::make(0, 0) : FarTab<real>::rec(tix(n, m));
		tb.out[e] = m < 0 ? (int16_t)-1 : (int16_t)tix(n, m);
	}
	for (int m = tid; m < N; m += nt) tb.S[m] = FarTab<real>::S(m);
}

// Sums of a cell over the particles of a lane group: a (FP32: plus c, what the
// additions to a have rounded off).
template <typename real, int STEPS> struct ChainAcc {
	typename V2<real>::t a[STEPS];
	typename V2<real>::t c[STEPS];     // FP32 compensation
	__device__ __forceinline__ void clear()
	{
#pragma unroll
		for (int s = 0; s < STEPS; ++s) {
			a[s] = V2<real>::make(0, 0);
			if constexpr (sizeof(real) == sizeof(float)) c[s] = make_float2(0.f, 0.f);
		}
	}
};

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
// a + c gains y - c (Kahan): y holds what is to be added and c
__device__ __forceinline__ void kahan(float2& a, float2& c, float2 y)
{
	const float2 t = add2(a, y);
	c = sub2(y, sub2(t, a));
	a = t;
}

template <typename real>
__device__ __forceinline__ typename V2<real>::t cm(typename V2<real>::t a, typename V2<real>::t b)
{ return V2<real>::make(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }

// One particle's chains on a lane: c = B_nm(x, y, z) at the lane's current step
// (the sums are conjugated when stored).
template <bool IRR, typename real, int STEPS> struct Chain {
	using v2 = typename V2<real>::t;
	real z, r2;                        // IRR: 1 / r^2
	v2 c, p, c2, c3;                   // this degree, the one below; the starts of chains 2 and 3
	__device__ __forceinline__ void start(const ChainTab<real>& tb, real x, real y, real z_, int l, int N)
	{
		z = z_;
		const real rr = x * x + y * y + z * z;
		r2 = IRR ? real(1) / rr : rr;
		const real b0 = IRR ? rsq<real>(rr) : real(1);
		const v2 w = V2<real>::make(IRR ? x * r2 : x, IRR ? y * r2 : y);
		const v2 w2 = cm<real>(w, w), w4 = cm<real>(w2, w2), one = V2<real>::make(1, 0);
		// w^l and w^(7 - l)
		v2 up = (l & 1) ? w : one, dn = (l & 1) ? one : w;
		if (l & 2) up = cm<real>(up, w2); else dn = cm<real>(dn, w2);
		if (l & 4) up = cm<real>(up, w4); else dn = cm<real>(dn, w4);
		p = c2 = c3 = V2<real>::make(0, 0);
		const real s1 = l < N ? b0 * tb.S[l] : real(0);
		c = V2<real>::make(up.x * s1, up.y * s1);
		if (STEPS > 8) {
			const v2 w8 = cm<real>(w4, w4);
			if (15 - l < N) {
				const real s2 = b0 * tb.S[15 - l];
				c2 = cm<real>(dn, w8);
				c2 = V2<real>::make(c2.x * s2, c2.y * s2);
			}
			if (STEPS > 17 && 16 + l < N) {
				const real s3 = b0 * tb.S[16 + l];
				c3 = cm<real>(up, cm<real>(w8, w8));
				c3 = V2<real>::make(c3.x * s3, c3.y * s3);
			}
		}
	}
	// the start of chain 2 or 3 at step s (l1, l12: the steps where they begin);
	// chain 2 starts at step N - l >= N - 7, chain 3 at 2 N - 15 (N = 17, 18)
	__device__ __forceinline__ void enter(int s, int l1, int l12)
	{
		if (STEPS > 8 && s >= (STEPS > 17 ? 10 : STEPS > 12 ? 6 : 2) && s == l1) c = c2;
		if (STEPS > 17 && (s == 19 || s == 21) && s == l12) c = c3;
	}
	__device__ __forceinline__ void next(v2 ab)
	{
		const real az = ab.x * z, bb = IRR ? ab.y : ab.y * r2;
		real nx = fma(az, c.x, -bb * p.x), ny = fma(az, c.y, -bb * p.y);
		if (IRR) { nx *= r2; ny *= r2; }
		p = c; c = V2<real>::make(nx, ny);
	}
};

// K particles per lane group added, q c in the fused multiply-adds that also
// take up the compensation; with K = 2 the table is read once for both.
template <bool IRR, typename real, int STEPS, int K>
__device__ __forceinline__ void chain_add(ChainAcc<real, STEPS>& A, const ChainTab<real>& tb, const real (&q)[K],
                                          const real (&x)[K], const real (&y)[K], const real (&z)[K], int N)
{
	const int l = threadIdx.x & (CHL - 1), l1 = N - l, l12 = l1 + N - 15 + l, T = chain_steps(N);
	Chain<IRR, real, STEPS> h[K];
#pragma unroll
	for (int j = 0; j < K; ++j) h[j].start(tb, x[j], y[j], z[j], l, N);
#pragma unroll
	for (int s = 0; s < STEPS; ++s) {
		if (s >= T) break;
		const typename V2<real>::t ab = tb.ab[s * CHL + l];
#pragma unroll
		for (int j = 0; j < K; ++j) h[j].enter(s, l1, l12);
		if constexpr (sizeof(real) == sizeof(float)) {
#pragma unroll
			for (int j = 0; j < K; ++j)
				kahan(A.a[s], A.c[s], __ffma2_rn(make_float2(q[j], q[j]), h[j].c, A.c[s]));
		} else {
#pragma unroll
			for (int j = 0; j < K; ++j) { A.a[s].x = fma(q[j], h[j].c.x, A.a[s].x); A.a[s].y = fma(q[j], h[j].c.y, A.a[s].y); }
		}
#pragma unroll
		for (int j = 0; j < K; ++j) h[j].next(ab);
	}
}

// K particles of every lane group from the lanes r + group, r + 4 + group.
template <bool IRR, typename real, int STEPS, int K>
__device__ __forceinline__ void chain_take(ChainAcc<real, STEPS>& A, const ChainTab<real>& tb, real q, real x, real y,
                                           real z, int r, int N)
{
	real qk[K], xk[K], yk[K], zk[K];
#pragma unroll
	for (int j = 0; j < K; ++j) {
		const int f = r + 4 * j + (threadIdx.x & 31) / CHL;
		qk[j] = __shfl_sync(0xffffffffu, q, f); xk[j] = __shfl_sync(0xffffffffu, x, f);
		yk[j] = __shfl_sync(0xffffffffu, y, f); zk[j] = __shfl_sync(0xffffffffu, z, f);
	}
	chain_add<IRR, real, STEPS, K>(A, tb, qk, xk, yk, zk, N);
}

// The first cnt lanes' particles (the others: q = 0), eight at a time in FP32
// and a rest of up to four, or four at a time.
template <bool IRR, typename real, int STEPS>
__device__ __forceinline__ void chain_add32(ChainAcc<real, STEPS>& A, const ChainTab<real>& tb, real q, real x, real y,
                                            real z, int cnt, int N)
{
	int r = 0;
	if constexpr (sizeof(real) == sizeof(float))
		for (; r + 4 < cnt; r += 8) chain_take<IRR, real, STEPS, 2>(A, tb, q, x, y, z, r, N);
	for (; r < cnt; r += 4) chain_take<IRR, real, STEPS, 1>(A, tb, q, x, y, z, r, N);
}

// The four lane groups' sums added up: lane group u ends with the totals of the
// steps 4 k + chain_sub() (a quarter of the exchanges of totals in every lane).
// FP32: exact sums of two (Knuth), their errors carried in c, added in last.
template <typename real> struct ChainVal {
	typename V2<real>::t a, c;             // c: FP32 only
};
__device__ __forceinline__ int chain_sub() { return (threadIdx.x >> 3 & 1) | (threadIdx.x >> 3 & 2); }

// keep the second (odd) or the first, plus the partner's (lane ^ o) of the same
template <typename real>
__device__ __forceinline__ ChainVal<real> chain_pair(const ChainVal<real>& x, const ChainVal<real>& y, bool odd, int o)
{
	ChainVal<real> k = odd ? y : x;
	const ChainVal<real> g = odd ? x : y;
	typename V2<real>::t b;
	b.x = __shfl_xor_sync(0xffffffffu, g.a.x, o);
	b.y = __shfl_xor_sync(0xffffffffu, g.a.y, o);
	if constexpr (sizeof(real) == sizeof(float)) {
		const float2 d = make_float2(__shfl_xor_sync(0xffffffffu, g.c.x, o), __shfl_xor_sync(0xffffffffu, g.c.y, o));
		const float2 a = k.a, u = add2(a, b), bv = sub2(u, a), err = add2(sub2(a, sub2(u, bv)), sub2(b, bv));
		k.a = u;
		k.c = add2(add2(k.c, d), err);
	} else {
		k.a.x += b.x; k.a.y += b.y;
	}
	return k;
}

template <typename real, int STEPS>
__device__ __forceinline__ void chain_reduce(const ChainAcc<real, STEPS>& A, int N,
                                             typename V2<real>::t (&tot)[(STEPS + 3) / 4])
{
	const int T = chain_steps(N), sub = chain_sub();
	auto val = [&](int s) {
		ChainVal<real> v;
		v.a = s < STEPS ? A.a[s < STEPS ? s : 0] : V2<real>::make(0, 0);
		if constexpr (sizeof(real) == sizeof(float)) v.c = s < STEPS ? A.c[s < STEPS ? s : 0] : make_float2(0.f, 0.f);
		return v;
	};
#pragma unroll
	for (int k = 0; k < (STEPS + 3) / 4; ++k) {
		if (4 * k >= T) break;
		const ChainVal<real> lo = chain_pair<real>(val(4 * k), val(4 * k + 1), sub & 1, CHL);
		const ChainVal<real> hi = chain_pair<real>(val(4 * k + 2), val(4 * k + 3), sub & 1, CHL);
		const ChainVal<real> v = chain_pair<real>(lo, hi, sub & 2, 2 * CHL);
		if constexpr (sizeof(real) == sizeof(float)) tot[k] = add2(v.a, v.c);
		else tot[k] = v.a;
	}
}

// out(index, total) for the coefficients whose totals this lane holds.
template <typename real, int STEPS, typename F>
__device__ __forceinline__ void chain_out(const ChainTab<real>& tb, int N, const typename V2<real>::t (&tot)[(STEPS + 3) / 4],
                                          F out)
{
	const int T = chain_steps(N), l = threadIdx.x & (CHL - 1), sub = chain_sub();
#pragma unroll
	for (int k = 0; k < (STEPS + 3) / 4; ++k) {
		const int s = 4 * k + sub;
		if (s >= T) break;
		const int o = tb.out[s * CHL + l];
		if (o >= 0) out(o, tot[k]);
	}
}

constexpr int FWPB = 4;                // warps per block (one leaf or cell each)
constexpr int FWL = 8;                 // warps per block on long lists
constexpr uint32_t FAR_SHORT = 8;      // lists up to this length are one warp's

// P2M: one warp per leaf at a time, in the leaf's scaled frame.
template <typename real, int STEPS>
__global__ void __launch_bounds__(FWPB * 32) p2m_scaled_kernel(DevTree t, int N, typename V2<real>::t* __restrict__ outer)
{
	__shared__ ChainTab<real> tb;
	chain_tab_fill(tb, N, threadIdx.x, FWPB * 32);
	__syncthreads();
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, Nx2 = N * (N + 1) / 2;
	for (size_t li = (size_t)blockIdx.x * FWPB + w; li < t.nleaves; li += (size_t)gridDim.x * FWPB) {
		const size_t g = t.leaves[li];
		const double ih = 1.0 / cell_size(t, g), cx = t.cx[g], cy = t.cy[g], cz = t.cz[g];
		const uint32_t b = t.pbeg[g], e = t.send[g];
		ChainAcc<real, STEPS> A;
		A.clear();
		for (uint32_t base = b; base < e; base += 32) {
			const uint32_t i = base + lane;
			real q = 0, x = 0, y = 0, z = 0;
			if (i < e) {
				q = (real)t.q[i];
				x = (real)((t.x[i] - cx) * ih); y = (real)((t.y[i] - cy) * ih); z = (real)((t.z[i] - cz) * ih);
			}
			chain_add32<false, real, STEPS>(A, tb, q, x, y, z, (int)min(32u, e - base), N);
		}
		typename V2<real>::t tot[(STEPS + 3) / 4];
		chain_reduce<real, STEPS>(A, N, tot);
		typename V2<real>::t* out = outer + g * Nx2;
		chain_out<real, STEPS>(tb, N, tot, [&](int o, typename V2<real>::t v) { out[o] = V2<real>::make(v.x, -v.y); });
	}
}

// The sources of cell g's X list as one sequence, 32 at a time (lane =
// source): batches w, w + nw, ... of every 32 list entries.
template <typename real, int STEPS>
__device__ __forceinline__ void p2l_sum(const DevTree& t, size_t g, uint32_t xb, uint32_t xe, int w, int nw, int N,
                                        const ChainTab<real>& tb, ChainAcc<real, STEPS>& A)
{
	const int lane = threadIdx.x & 31;
	const double ih = 1.0 / cell_size(t, g), cx = t.cx[g], cy = t.cy[g], cz = t.cz[g];
	for (uint32_t e0 = xb; e0 < xe; e0 += 32) {
		uint32_t b = 0, n = 0;
		if (e0 + lane < xe) {
			const int32_t C = t.x_idx[e0 + lane];
			b = t.pbeg[C]; n = t.send[C] - b;
		}
		const SourceRun run(b, n);
		for (uint32_t f0 = 32u * w; f0 < run.total; f0 += 32u * nw) {
			const uint32_t f = f0 + lane, i = run.at(f);
			real q = 0, x = 0, y = 0, z = 1;   // past the end: q = 0 at a finite point
			if (f < run.total) {
				q = (real)t.q[i];
				x = (real)((t.x[i] - cx) * ih); y = (real)((t.y[i] - cy) * ih); z = (real)((t.z[i] - cz) * ih);
			}
			chain_add32<true, real, STEPS>(A, tb, q, x, y, z, (int)min(32u, run.total - f0), N);
		}
	}
}

// The cells with an X list: up to FAR_SHORT entries into shorts, longer ones
// into longs (entry 0 of each: the count, zeroed).  Both kernels below take
// cells from these lists, since the cells beside a refinement hold most of the
// entries and lie together.
__global__ void x_select_kernel(DevTree t, uint32_t* __restrict__ shorts, uint32_t* __restrict__ longs)
{
	const size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (g >= t.ncells) return;
	const uint32_t n = t.x_off[g + 1] - t.x_off[g];
	if (n == 0) return;
	uint32_t* l = n > FAR_SHORT ? longs : shorts;
	l[1 + atomicAdd(l, 1u)] = (uint32_t)g;
}

// P2L over the X lists: inner[g] += irregular harmonics of every X leaf's
// sources about g's centre (scaled by g's size); a warp per cell, from a
// counter.
template <typename real, int STEPS>
__global__ void __launch_bounds__(FWPB * 32) p2l_kernel(DevTree t, int N, typename V2<real>::t* __restrict__ inner,
                                                       uint32_t* __restrict__ next, const uint32_t* __restrict__ shorts)
{
	__shared__ ChainTab<real> tb;
	chain_tab_fill(tb, N, threadIdx.x, FWPB * 32);
	__syncthreads();
	const int lane = threadIdx.x & 31, Nx2 = N * (N + 1) / 2;
	const uint32_t cnt = shorts[0];
	for (;;) {
		uint32_t it = 0;
		if (lane == 0) it = atomicAdd(next, 1u);
		it = __shfl_sync(0xffffffffu, it, 0);
		if (it >= cnt) return;
		const size_t g = shorts[1 + it];
		ChainAcc<real, STEPS> A;
		A.clear();
		p2l_sum<real, STEPS>(t, g, t.x_off[g], t.x_off[g + 1], 0, 1, N, tb, A);
		typename V2<real>::t tot[(STEPS + 3) / 4];
		chain_reduce<real, STEPS>(A, N, tot);
		typename V2<real>::t* out = inner + g * Nx2;
		chain_out<real, STEPS>(tb, N, tot, [&](int o, typename V2<real>::t v) {
			const typename V2<real>::t a = out[o];
			out[o] = V2<real>::make(a.x + v.x, a.y - v.y);
		});
	}
}

// The long lists: one block per cell, its warps take the batches of sources in
// turn and their sums are added in warp order (FP64).
template <typename real, int STEPS>
__global__ void __launch_bounds__(FWL * 32, sizeof(real) == sizeof(float) ? 2 : 1) p2l_long_kernel(DevTree t, int N, typename V2<real>::t* __restrict__ inner,
                                                           const uint32_t* __restrict__ longs)
{
	__shared__ ChainTab<real> tb;
	__shared__ typename V2<real>::t part[FWL][NX2MAX];
	chain_tab_fill(tb, N, threadIdx.x, FWL * 32);
	__syncthreads();
	const int w = threadIdx.x >> 5, Nx2 = N * (N + 1) / 2;
	const uint32_t cnt = longs[0];
	for (uint32_t it = blockIdx.x; it < cnt; it += gridDim.x) {
		const size_t g = longs[1 + it];
		ChainAcc<real, STEPS> A;
		A.clear();
		p2l_sum<real, STEPS>(t, g, t.x_off[g], t.x_off[g + 1], w, FWL, N, tb, A);
		typename V2<real>::t tot[(STEPS + 3) / 4];
		chain_reduce<real, STEPS>(A, N, tot);
		chain_out<real, STEPS>(tb, N, tot, [&](int o, typename V2<real>::t v) { part[w][o] = v; });
		__syncthreads();
		for (int c = threadIdx.x; c < Nx2; c += FWL * 32) {
			double re = 0.0, im = 0.0;
			for (int k = 0; k < FWL; ++k) { re += (double)part[k][c].x; im += (double)part[k][c].y; }
			typename V2<real>::t a = inner[g * Nx2 + c];
			inner[g * Nx2 + c] = V2<real>::make((real)((double)a.x + re), (real)((double)a.y - im));
		}
		__syncthreads();
	}
}

// ---- M2P, L2P --------------------------------------------------------------
// A real field phi = sum_{n, m >= 0} (2 - d_m0) Re(E_nm B_nm) (E stored for
// m >= 0; the m < 0 coefficients are (-1)^m conj(E_n|m|)) has, with the
// derivative rules
//   regular:   d_z B_nm = sqrt((n-m)(n+m)) B_{n-1,m},
//              (d_x + i d_y) B_nm = sqrt((n-m)(n-m-1)) B_{n-1,m+1},
//              (d_x - i d_y) B_nm = -sqrt((n+m)(n+m-1)) B_{n-1,m-1},
//   irregular: d_z B_nm = -sqrt((n+1-m)(n+1+m)) B_{n+1,m},
//              (d_x + i d_y) B_nm = sqrt((n+m+1)(n+m+2)) B_{n+1,m+1},
//              (d_x - i d_y) B_nm = -sqrt((n-m+1)(n-m+2)) B_{n+1,m-1},
// a gradient that is again a real field in the same basis, of degree one
// less (local) or one more (multipole).  derive_coefs turns E into the
// potential's and the three gradient components' coefficients (the weight
// (2 - d_m0) folded in), order after order: row k (N+1) - k (k-1) / 2 + n - k
// holds degree n of order k; eval_chains streams one target's harmonics
// through them.
template <typename real> struct __align__(16) CoefRow {
	// the real parts of the four sets, then their negated imaginary parts
	real re[4], im[4];
};

__device__ __forceinline__ int coef_row(int N, int n, int k) { return k * (N + 1) - k * (k - 1) / 2 + n - k; }

template <bool IRR, typename real>
__device__ __forceinline__ void derive_coefs(const typename V2<real>::t* __restrict__ E, int N, CoefRow<real>* C, int tid,
                                             int nt)
{
	using v2 = typename V2<real>::t;
	const int NB = IRR ? N + 1 : N, NG = IRR ? N + 1 : N - 1;
	for (int e = tid; e < NB * (NB + 1) / 2; e += nt) {
		const auto f = FarTab<real>::g(IRR, e);
		const int n = f.nk & 255, k = f.nk >> 8;
		CoefRow<real> o;
		v2 c = V2<real>::make(0, 0);
		if (n < N) c = E[e];
		o.re[0] = k ? 2 * c.x : c.x; o.im[0] = k ? -2 * c.y : real(0);
		o.re[1] = o.re[2] = o.re[3] = o.im[1] = o.im[2] = o.im[3] = 0;
		if (n < NG) {
			const int d = IRR ? n - 1 : n + 1;             // degree of the source coefficients
			v2 c0 = V2<real>::make(0, 0), cl = c0, cr = c0;
			if (d >= k) c0 = E[tix(d, k)];
			if (k == 0) {
				c0.y = 0;
				if (d >= 1) { const v2 u = E[tix(d, 1)]; cl = V2<real>::make(-u.x, u.y); }
			} else if (d >= k - 1) {
				cl = E[tix(d, k - 1)];
				if (k == 1) cl.y = 0;
			}
			if (d >= k + 1) cr = E[tix(d, k + 1)];
			const real sg = IRR ? real(-1) : real(1);
			const v2 Z = V2<real>::make(sg * c0.x * f.z, sg * c0.y * f.z);
			const v2 P = V2<real>::make(cl.x * f.p, cl.y * f.p), M = V2<real>::make(-cr.x * f.m, -cr.y * f.m);
			// d_x = (P + M) / 2, d_y = (P - M) / 2i; weight 2 for k > 0
			const real w = k ? real(1) : real(0.5);
			o.re[1] = w * (P.x + M.x); o.im[1] = -(w * (P.y + M.y));
			o.re[2] = w * (P.y - M.y); o.im[2] = w * (P.x - M.x);
			o.re[3] = 2 * w * Z.x; o.im[3] = -(2 * w * Z.y);
		}
		C[coef_row(N, n, k)] = o;
	}
}

// phi and grad phi at K points (the expansion's scaled frame), the orders
// g, g + G, ... (G a power of two up to 8).  K targets share the rows' reads:
// a 16-byte broadcast read returns 512 bytes to the warp, four cycles of the
// SM's shared-memory path, so with one target per lane the reads (10 cycles a
// row) outweigh the arithmetic (5).
template <bool IRR, typename real, int K>
__device__ __forceinline__ void eval_chains(const CoefRow<real>* __restrict__ C, const typename V2<real>::t* __restrict__ ab,
                                            const real* __restrict__ S, const real (&x)[K], const real (&y)[K],
                                            const real (&z)[K], int N, int g, int G, real (&sum)[K][4])
{
	using v2 = typename V2<real>::t;
	const int NB = IRR ? N + 1 : N;
	real q2[K];                                // r^2 or 1 / r^2
	v2 wG[K], pw[K];
#pragma unroll
	for (int j = 0; j < K; ++j) {
		const real r2 = x[j] * x[j] + y[j] * y[j] + z[j] * z[j];
		q2[j] = IRR ? real(1) / r2 : r2;
		wG[j] = V2<real>::make(IRR ? x[j] * q2[j] : x[j], IRR ? y[j] * q2[j] : y[j]);
		pw[j] = V2<real>::make(IRR ? rsq<real>(r2) : real(1), 0);
		for (int b = 1; b < G; b <<= 1) {      // pw = w^g B_00, wG = w^G
			if (g & b) pw[j] = cm<real>(pw[j], wG[j]);
			wG[j] = cm<real>(wG[j], wG[j]);
		}
		sum[j][0] = sum[j][1] = sum[j][2] = sum[j][3] = 0;
	}
	for (int m = g; m < NB; m += G) {
		const real s = S[m];
		real px[K], py[K], cx[K], cy[K];
#pragma unroll
		for (int j = 0; j < K; ++j) { px[j] = py[j] = 0; cx[j] = pw[j].x * s; cy[j] = pw[j].y * s; }
		const int r0 = coef_row(N, m, m);
		const CoefRow<real>* row = C + r0;
		const v2* rec = ab + r0;
#pragma unroll 2
		for (int n = m; n < NB; ++n, ++row, ++rec) {
			const CoefRow<real> c = *row;
			const v2 r = *rec;
#pragma unroll
			for (int j = 0; j < K; ++j) {
#pragma unroll
				for (int k = 0; k < 4; ++k) sum[j][k] = fma(c.re[k], cx[j], fma(c.im[k], cy[j], sum[j][k]));
				const real az = r.x * z[j], bb = IRR ? r.y : r.y * q2[j];
				real nx = fma(az, cx[j], -bb * px[j]), ny = fma(az, cy[j], -bb * py[j]);
				if (IRR) { nx *= q2[j]; ny *= q2[j]; }
				px[j] = cx[j]; py[j] = cy[j]; cx[j] = nx; cy[j] = ny;
			}
		}
#pragma unroll
		for (int j = 0; j < K; ++j) pw[j] = cm<real>(pw[j], wG[j]);
	}
}

// Recurrence constants of a block, in the rows' order.
template <typename real>
__device__ __forceinline__ void eval_tab_fill(typename V2<real>::t* ab, real* S, int N, int tid, int nt)
{
	for (int e = tid; e < (N + 1) * (N + 2) / 2; e += nt) {
		const int n = tri_row(e), k = e - tix(n, 0);
		ab[coef_row(N, n, k)] = FarTab<real>::rec(e);
	}
	for (int m = tid; m <= N; m += nt) S[m] = FarTab<real>::S(m);
}

template <typename real> __host__ __device__ constexpr size_t eval_smem(int warps, int N)
{
	return ((size_t)warps * sizeof(CoefRow<real>) + 2 * sizeof(real)) * ((N + 1) * (N + 2) / 2) + sizeof(real) * (MAXN3 + 2);
}

// Targets t0 .. t0 + np - 1 of a leaf on one warp, K per lane: TP lanes (the
// smallest power of two from 4 on that holds them) per group of orders,
// 32 / TP groups; lane ti of a group has targets ti, ti + TP, ...
template <int K> struct EvalPass {
	int lt, ti, g, G, np;
	uint32_t t0;
	__device__ __forceinline__ EvalPass(uint32_t t0_, int np_) : np(np_), t0(t0_)
	{
		const int lane = threadIdx.x & 31;
		lt = 2;
		while ((K << lt) < np) ++lt;
		ti = lane & ((1 << lt) - 1); g = lane >> lt; G = 32 >> lt;
	}
	__device__ __forceinline__ int idx(int j) const { return ti + (j << lt); }
	__device__ __forceinline__ uint32_t at(int j) const { return t0 + min(idx(j), np - 1); }
};
// Most targets of a pass, and the passes of n targets (about equal).
template <typename real> __host__ __device__ constexpr int eval_cap() { return sizeof(real) == sizeof(float) ? 48 : 32; }
// Targets per lane of a pass of np: at N = 16 a row costs about
// max(3 + 16 K, 40) issue slots (40: its shared-memory reads) and 32 / TP = 8,
// 4, 2 groups have 27, 45, 81 rows, so three per lane are cheaper for 9-12,
// 17-24 and 33-48 targets.
__device__ __forceinline__ bool eval_three(int np) { return (np > 8 && np <= 12) || (np > 16 && np <= 24) || np > 32; }

template <bool IRR, typename real, int K>
__device__ __forceinline__ void eval_add(const EvalPass<K>& p, const DevTree& t, size_t D, const CoefRow<real>* C,
                                         const typename V2<real>::t* ab, const real* S, int N, double (&out)[K][4])
{
	const double ih = 1.0 / cell_size(t, D), cx = t.cx[D], cy = t.cy[D], cz = t.cz[D];
	real s[K][4], xr[K], yr[K], zr[K];
#pragma unroll
	for (int j = 0; j < K; ++j) {
		const uint32_t i = p.at(j);
		double x = (t.x[i] - cx) * ih, y = (t.y[i] - cy) * ih;
		const double z = (t.z[i] - cz) * ih;
		if constexpr (sizeof(real) == sizeof(double)) reference_point(x, y, z);
		xr[j] = (real)x; yr[j] = (real)y; zr[j] = (real)z;
	}
	eval_chains<IRR, real, K>(C, ab, S, xr, yr, zr, N, p.g, p.G, s);
#pragma unroll
	for (int j = 0; j < K; ++j) {
		out[j][0] += (double)s[j][0] * ih;
#pragma unroll
		for (int k = 1; k < 4; ++k) out[j][k] -= (double)s[j][k] * ih * ih;
	}
}

// One pass of a leaf on one warp: its W entries e0, e0 + step, ... below we,
// and its local expansion where that sequence reaches we; the sums over the
// groups of orders end in every lane.
template <typename real, int K>
__device__ __forceinline__ void eval_pass(const EvalPass<K>& p, const DevTree& t, size_t g, uint32_t e0, uint32_t step,
                                          uint32_t we, const typename V2<real>::t* __restrict__ outer,
                                          const typename V2<real>::t* __restrict__ inner, int N, CoefRow<real>* C,
                                          const typename V2<real>::t* ab, const real* S, double (&o)[K][4])
{
	const int lane = threadIdx.x & 31, Nx2 = N * (N + 1) / 2;
#pragma unroll
	for (int j = 0; j < K; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.0;
	for (uint32_t e = e0; e <= we; e += step) {
		__syncwarp();
		if (e < we) {
			const size_t D = t.w_idx[e];
			derive_coefs<true, real>(outer + D * Nx2, N, C, lane, 32);
			__syncwarp();
			eval_add<true, real, K>(p, t, D, C, ab, S, N, o);
		} else {
			derive_coefs<false, real>(inner + g * Nx2, N, C, lane, 32);
			__syncwarp();
			eval_add<false, real, K>(p, t, g, C, ab, S, N, o);
		}
	}
	for (int s = 1 << p.lt; s < 32; s <<= 1)
#pragma unroll
		for (int j = 0; j < K; ++j)
#pragma unroll
			for (int k = 0; k < 4; ++k) o[j][k] += __shfl_xor_sync(0xffffffffu, o[j][k], s);
}

// M2P over the W list and L2P of the leaf's local expansion, added onto the
// near field already in the outputs: one warp per leaf at a time (from a
// counter), each expansion's coefficients derived once per pass of at most
// eval_cap targets.  Leaves with more than FAR_SHORT W entries go to `longs`.
// FP32: about 16 instructions per coefficient and target on rows read as 16-byte
// broadcasts; 1,000,000 clustered particles at N = 16: 392 us, issue slots 52 %
// busy, the largest stall the expansions' and targets' loads.  Before (a target
// per lane, rows in degree order, square roots in the derivation, one warp for a
// list of any length) 300,007 clustered particles at N = 16 took 2640 us.
template <typename real>
__global__ void __launch_bounds__(FWPB * 32, sizeof(real) == sizeof(float) ? 5 : 4) eval_scaled_kernel(DevTree t, const typename V2<real>::t* __restrict__ outer,
                                                               const typename V2<real>::t* __restrict__ inner, int N,
                                                               double* __restrict__ pot_out,
                                                               double* __restrict__ fld_out,
                                                               unsigned* __restrict__ next_leaf,
                                                               uint32_t* __restrict__ longs)
{
	using v2 = typename V2<real>::t;
	extern __shared__ __align__(16) unsigned char sm_eval[];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, R = (N + 1) * (N + 2) / 2;
	CoefRow<real>* C = reinterpret_cast<CoefRow<real>*>(sm_eval) + w * R;
	v2* ab = reinterpret_cast<v2*>(reinterpret_cast<CoefRow<real>*>(sm_eval) + FWPB * R);
	real* S = reinterpret_cast<real*>(ab + R);
	eval_tab_fill<real>(ab, S, N, threadIdx.x, FWPB * 32);
	__syncthreads();
	for (;;) {
		unsigned lid = 0;
		if (lane == 0) lid = atomicAdd(next_leaf, 1u);
		const size_t li = __shfl_sync(0xffffffffu, lid, 0);
		if (li >= t.nleaves) return;
		const size_t g = t.leaves[li];
		const uint32_t tb = t.tbeg[g], nt = t.tend[g] - tb;
		if (t.tend[g] <= tb) continue;
		const uint32_t wb = t.w_off[li], we = t.w_off[li + 1];
		if (we - wb > FAR_SHORT) {
			if (lane == 0) longs[1 + atomicAdd(longs, 1u)] = (uint32_t)li;
			continue;
		}
		const uint32_t passes = (nt + eval_cap<real>() - 1) / eval_cap<real>(), per = (nt + passes - 1) / passes;
		auto go = [&](auto kc, uint32_t t0, int np) {
			constexpr int K = decltype(kc)::value;
			const EvalPass<K> p(t0, np);
			double o[K][4];
			eval_pass<real, K>(p, t, g, wb, 1, we, outer, inner, N, C, ab, S, o);
#pragma unroll
			for (int j = 0; j < K; ++j)
				if (p.g == 0 && p.idx(j) < np) {
					const size_t r = t.orig[p.at(j)];
					if (r >= t.n_out()) continue;
					pot_out[r] += o[j][0];
					fld_out[3 * r] += o[j][1]; fld_out[3 * r + 1] += o[j][2]; fld_out[3 * r + 2] += o[j][3];
				}
		};
		for (uint32_t k0 = 0; k0 < nt; k0 += per) {
			const int np = (int)min(per, nt - k0);
			if (sizeof(real) == sizeof(float) && eval_three(np)) {
				if constexpr (sizeof(real) == sizeof(float)) go(std::integral_constant<int, 3>(), tb + k0, np);
			} else {
				go(std::integral_constant<int, 2>(), tb + k0, np);
			}
		}
	}
}

// The long W lists: a block takes a leaf's even or odd passes from a counter,
// its warps the W entries (and, as one more entry, the leaf's local expansion)
// in turn; their sums are added in warp order.
template <typename real>
__global__ void __launch_bounds__(FWL * 32, 2) eval_long_kernel(DevTree t, const typename V2<real>::t* __restrict__ outer,
                                                            const typename V2<real>::t* __restrict__ inner, int N,
                                                            double* __restrict__ pot_out, double* __restrict__ fld_out,
                                                            uint32_t* __restrict__ next,
                                                            const uint32_t* __restrict__ longs)
{
	using v2 = typename V2<real>::t;
	extern __shared__ __align__(16) unsigned char sm_eval[];
	__shared__ double part[FWL][eval_cap<real>()][4];
	__shared__ uint32_t s_item;
	const int w = threadIdx.x >> 5, R = (N + 1) * (N + 2) / 2;
	CoefRow<real>* C = reinterpret_cast<CoefRow<real>*>(sm_eval) + w * R;
	v2* ab = reinterpret_cast<v2*>(reinterpret_cast<CoefRow<real>*>(sm_eval) + FWL * R);
	real* S = reinterpret_cast<real*>(ab + R);
	eval_tab_fill<real>(ab, S, N, threadIdx.x, FWL * 32);
	__syncthreads();
	const uint32_t cnt = longs[0];
	for (;;) {
		if (threadIdx.x == 0) s_item = atomicAdd(next, 1u);
		__syncthreads();
		const uint32_t item = s_item;
		if (item >= 2 * cnt) return;
		const size_t li = longs[1 + item / 2], g = t.leaves[li];
		const uint32_t tb = t.tbeg[g], nt = t.tend[g] - tb, wb = t.w_off[li], we = t.w_off[li + 1];
		const uint32_t passes = (nt + eval_cap<real>() - 1) / eval_cap<real>(), per = (nt + passes - 1) / passes;
		auto go = [&](auto kc, uint32_t t0, int np) {
			constexpr int K = decltype(kc)::value;
			const EvalPass<K> p(t0, np);
			double o[K][4];
			eval_pass<real, K>(p, t, g, wb + w, FWL, we, outer, inner, N, C, ab, S, o);
#pragma unroll
			for (int j = 0; j < K; ++j)
				if (p.g == 0 && p.idx(j) < np) {
#pragma unroll
					for (int k = 0; k < 4; ++k) part[w][p.idx(j)][k] = o[j][k];
				}
		};
		__syncthreads();                       // the item is read before the next is taken
		for (uint32_t k0 = (item & 1) * per; k0 < nt; k0 += 2 * per) {
			const int np = (int)min(per, nt - k0);
			__syncthreads();                   // the last pass's sums are read
			if (sizeof(real) == sizeof(float) && eval_three(np)) {
				if constexpr (sizeof(real) == sizeof(float)) go(std::integral_constant<int, 3>(), tb + k0, np);
			} else {
				go(std::integral_constant<int, 2>(), tb + k0, np);
			}
			__syncthreads();
			const int tt = threadIdx.x >> 2, k = threadIdx.x & 3;
			if (tt < np) {
				double v = 0.0;
				for (int q = 0; q < FWL; ++q) v += part[q][tt][k];
				const size_t r = t.orig[tb + k0 + tt];
				if (r < t.n_out()) {
					if (k == 0) pot_out[r] += v; else fld_out[3 * r + k - 1] += v;
				}
			}
		}
	}
}

// ---- near field of the FP64 form -------------------------------------------
// One warp per leaf at a time (from a counter); targets in passes of up to 32,
// fewer share the sources out between groups of lanes; sources of the leaf and
// its U list staged 32 at a time, four of them per step of a lane, so that their
// reciprocal square roots overlap (one at a time: 300,007 clustered particles 748
// us, now 606; 8,475 in eight leaves, one warp each, 38 ms, now 15).  Writes pot
// (with the reference's self term) and field in input order; eval_scaled_kernel
// adds the expansions.
template <int LW>
__global__ void __launch_bounds__(LW * 32) p2p_f64_kernel(DevTree t, double* __restrict__ pot_out,
                                                         double* __restrict__ fld_out, unsigned* __restrict__ next_leaf)
{
	__shared__ double4 ss[LW][32];
	const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const bool tmode = t.targets_num > 0;
	for (;;) {
		unsigned lid = 0;
		if (lane == 0) lid = atomicAdd(next_leaf, 1u);
		const size_t li = __shfl_sync(0xffffffffu, lid, 0);
		if (li >= t.nleaves) return;
		const size_t g = t.leaves[li];
		const uint32_t tb = t.tbeg[g], te = t.tend[g];
		if (tb >= te) continue;
		const uint32_t ub = t.u_off[li], ue = t.u_off[li + 1];
		const double cx = t.cx[g], cy = t.cy[g], cz = t.cz[g];
		for (uint32_t t0 = tb; t0 < te; t0 += 32) {
			const int np = (int)min(32u, te - t0);
			int lt = 0;
			while ((1 << lt) < np) ++lt;
			const int ti = lane & ((1 << lt) - 1), ph = lane >> lt, G = 32 >> lt;
			const uint32_t i = t0 + min(ti, np - 1);
			const double xi = t.x[i] - cx, yi = t.y[i] - cy, zi = t.z[i] - cz;
			double pot = 0.0, fx = 0.0, fy = 0.0, fz = 0.0;
			for (int64_t e = (int64_t)ub - 1; e < (int64_t)ue; ++e) {
				const size_t sc_ = e < (int64_t)ub ? g : (size_t)t.u_idx[e];
				const uint32_t sb = t.pbeg[sc_], se = t.send[sc_];
				for (uint32_t s0 = sb; s0 < se; s0 += 32) {
					const int cnt = (int)min(32u, se - s0);
					__syncwarp();
					if (lane < cnt) {
						const uint32_t j = s0 + lane;
						ss[w][lane] = make_double4(t.x[j] - cx, t.y[j] - cy, t.z[j] - cz, t.q[j]);
					}
					__syncwarp();
					const int self = sc_ == g ? (int)i - (int)s0 : -1;
					auto pairs = [&](auto mc, int j) {
						constexpr int M = decltype(mc)::value;
						double dx[M], dy[M], dz[M], q[M], r2[M];
						bool far = false;
#pragma unroll
						for (int m = 0; m < M; ++m) {
							const double4 s = ss[w][j + m * G];
							dx[m] = xi - s.x; dy[m] = yi - s.y; dz[m] = zi - s.z;
							q[m] = j + m * G == self ? 0.0 : s.w;
							r2[m] = fmax(fma(dx[m], dx[m], fma(dy[m], dy[m], dz[m] * dz[m])), FORCE_EPS2);
							far |= beyond_1e300(r2[m]);
						}
						auto add = [&](int m, double inv) {
							const double qi = q[m] * inv, qi3 = qi * inv * inv;
							pot += qi;
							fx = fma(dx[m], qi3, fx); fy = fma(dy[m], qi3, fy); fz = fma(dz[m], qi3, fz);
						};
						if (far) {
							for (int m = 0; m < M; ++m) add(m, rsqrt_refined(r2[m]));
						} else {
							double inv[M];
#pragma unroll
							for (int m = 0; m < M; ++m) inv[m] = rsqrt_below_1e300(r2[m]);
#pragma unroll
							for (int m = 0; m < M; ++m) add(m, inv[m]);
						}
					};
					int j = ph;
					for (; j + 3 * G < cnt; j += 4 * G) pairs(std::integral_constant<int, 4>(), j);
					for (; j < cnt; j += G) pairs(std::integral_constant<int, 1>(), j);
				}
			}
			for (int o = 1 << lt; o < 32; o <<= 1) {
				pot += __shfl_xor_sync(0xffffffffu, pot, o);
				fx += __shfl_xor_sync(0xffffffffu, fx, o);
				fy += __shfl_xor_sync(0xffffffffu, fy, o);
				fz += __shfl_xor_sync(0xffffffffu, fz, o);
			}
			if (ti < np && ph == 0) {
				if (!tmode) pot += t.q[i] * (1.0 / FORCE_EPS);
				const size_t o = t.orig[i];
				if (o < t.n_out()) {
					pot_out[o] = pot;
					fld_out[3 * o] = fx; fld_out[3 * o + 1] = fy; fld_out[3 * o + 2] = fz;
				}
			}
		}
	}
}

// ---- leaves of the plain form ----------------------------------------------
// (uniform tree, unscaled expansions; the same harmonics at the reference's
// points)

// P2M: one warp per leaf.
template <int STEPS>
__global__ void __launch_bounds__(FWPB * 32) p2m_plain_kernel(DevTree t, int N, double2* __restrict__ outer)
{
	__shared__ ChainTab<double> tb;
	chain_tab_fill(tb, N, threadIdx.x, FWPB * 32);
	__syncthreads();
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, LL = t.depth - 1, Nx2 = N * (N + 1) / 2;
	const size_t leaf = (size_t)blockIdx.x * FWPB + w;
	if (leaf >= t.lsize[LL]) return;
	const size_t g = t.loff[LL] + leaf;
	const double cx = t.cx[g], cy = t.cy[g], cz = t.cz[g];
	const uint32_t e = t.end[g];
	ChainAcc<double, STEPS> A;
	A.clear();
	for (uint32_t base = t.beg[g]; base < e; base += 32) {
		const uint32_t i = base + lane;
		double q = 0, x = 0, y = 0, z = 0;
		if (i < e) {
			q = t.q[i]; x = t.x[i] - cx; y = t.y[i] - cy; z = t.z[i] - cz;
			reference_point(x, y, z);
		}
		chain_add32<false, double, STEPS>(A, tb, q, x, y, z, (int)min(32u, e - base), N);
	}
	double2 tot[(STEPS + 3) / 4];
	chain_reduce<double, STEPS>(A, N, tot);
	chain_out<double, STEPS>(tb, N, tot, [&](int o, double2 v) { outer[g * Nx2 + o] = make_double2(v.x, -v.y); });
}

// Near field and (FAR) local expansion of 32 targets of a leaf on a block of
// eight warps: the warps take the staged 32-source tiles of the leaf and its
// close cells in turn and every eighth order of the expansion; fewer than 17
// targets share a tile's sources out between groups of lanes.  Chunks of 32
// targets are spread over gridDim.y where the leaves alone would not fill the
// GPU.  FP64 pipe bound (about 22 operations per pair).  Before (a block of 128
// threads per leaf, thread = target, the reference's spherical form per
// target): 8 leaves of 256 particles 565 us, 4,096 of 32 at N = 9 617 us, 512
// of 157 (39 targets) at N = 18 368 us.
template <bool FAR>
__global__ void __launch_bounds__(FWL * 32, 2) leaves_plain_kernel(DevTree t, const double2* __restrict__ inner, int N,
                                                                  double* __restrict__ pot_out,
                                                                  double* __restrict__ fld_out)
{
	extern __shared__ __align__(16) unsigned char sm_eval[];
	__shared__ double4 ss[FWL][32];
	__shared__ double part[FWL][32][4];
	const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, LL = t.depth - 1, R = (N + 1) * (N + 2) / 2;
	CoefRow<double>* C = reinterpret_cast<CoefRow<double>*>(sm_eval);
	double2* ab = reinterpret_cast<double2*>(C + R);
	double* S = reinterpret_cast<double*>(ab + R);
	const size_t off = t.loff[LL], g = off + blockIdx.x;
	const bool tmode = t.targets_num > 0;
	const uint32_t tb = tmode ? t.tbeg[g] : t.beg[g], te = tmode ? t.tend[g] : t.end[g];
	if (tb + 32 * blockIdx.y >= te) return;
	if (FAR) {
		eval_tab_fill<double>(ab, S, N, tid, FWL * 32);
		derive_coefs<false, double>(inner + g * (size_t)(N * (N + 1) / 2), N, C, tid, FWL * 32);
	}
	const int ncl = t.close_cnt[g];
	const int32_t* cl = t.close_idx + g * t.close_stride;
	const double cx = t.cx[g], cy = t.cy[g], cz = t.cz[g];
	for (uint32_t t0 = tb + 32 * blockIdx.y; t0 < te; t0 += 32 * gridDim.y) {
		const int np = (int)min(32u, te - t0);
		int lt = 0;
		while ((1 << lt) < np) ++lt;
		const int ti = lane & ((1 << lt) - 1), ph = lane >> lt, G = 32 >> lt;
		const uint32_t i = t0 + min(ti, np - 1);
		const double xi = t.x[i], yi = t.y[i], zi = t.z[i];
		double o[4] = {0.0, 0.0, 0.0, 0.0};
		int turn = 0;
		for (int e = -1; e < ncl; ++e) {
			const size_t sc = e < 0 ? g : off + cl[e];
			const uint32_t sb = t.beg[sc], se = t.end[sc];
			for (uint32_t s0 = sb; s0 < se; s0 += 32) {
				if ((turn++ & (FWL - 1)) != w) continue;
				const int cnt = (int)min(32u, se - s0);
				__syncwarp();
				if (lane < cnt) {
					const uint32_t j = s0 + lane;
					ss[w][lane] = make_double4(t.x[j], t.y[j], t.z[j], t.q[j]);
				}
				__syncwarp();
				for (int j = ph; j < cnt; j += G) {
					const double4 s = ss[w][j];
					const double dx = xi - s.x, dy = yi - s.y, dz = zi - s.z;
					const double inv = rsqrt_refined(fmax(dx * dx + dy * dy + dz * dz, FORCE_EPS2));
					const double qi = s.w * inv, qi3 = qi * inv * inv;
					o[0] += qi;
					o[1] = fma(dx, qi3, o[1]); o[2] = fma(dy, qi3, o[2]); o[3] = fma(dz, qi3, o[3]);
				}
			}
		}
		for (int s = 1 << lt; s < 32; s <<= 1)
#pragma unroll
			for (int k = 0; k < 4; ++k) o[k] += __shfl_xor_sync(0xffffffffu, o[k], s);
		__syncthreads();                       // the rows are derived; the last chunk's sums are read
		if (FAR) {
			double x[1] = {xi - cx}, y[1] = {yi - cy}, z[1] = {zi - cz}, s[1][4];
			reference_point(x[0], y[0], z[0]);
			eval_chains<false, double, 1>(C, ab, S, x, y, z, N, w, FWL, s);
			o[0] += s[0][0];
#pragma unroll
			for (int k = 1; k < 4; ++k) o[k] -= s[0][k];
		}
		if (ph == 0 && ti < np) {
#pragma unroll
			for (int k = 0; k < 4; ++k) part[w][ti][k] = o[k];
		}
		__syncthreads();
		const int tt = tid >> 2, k = tid & 3;
		if (tt < np) {
			double v = 0.0;
			for (int q = 0; q < FWL; ++q) v += part[q][tt][k];
			const size_t r = t.orig[t0 + tt];
			if (r < t.n_out()) {
				if (k == 0) pot_out[r] = v; else fld_out[3 * r + k - 1] = v;
			}
		}
	}
}

} // namespace scaled
} // namespace lfmm
