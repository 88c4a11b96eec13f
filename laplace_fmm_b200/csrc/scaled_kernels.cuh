// Device kernels of the scaled-expansion 3D solver (plain FP64 or mixed
// FP32), included only by fmm3d_scaled.cu.  Scaled expansions: multipole
// a_nm / h^n and local L_nm h^(n+1) for a cell of size h; every operator is
// then level-independent and every coefficient O(total charge):
//   M2L   rho / h = |d|                      (one operator per far offset d)
//   M2M   (rho / h_child)^n, row j times 2^-j
//   L2L   (rho / h_parent)^(n-j), row j times 2^-(j+1)
//   P2M / L2P / P2L / M2P with r / h; potential times 1/h, field times 1/h^2.
#pragma once
#include "fmm3d.cuh"
#include "m2l_gemm.cuh"

namespace lfmm {
namespace scaled {

constexpr int CMAX = (MAXN3 * (MAXN3 + 1) / 2 + 31) / 32;
constexpr int NX2MAX = MAXN3 * (MAXN3 + 1) / 2;
constexpr int WPB = 4;

template <typename real> struct V2;
template <> struct V2<double> { using t = double2; static __device__ __forceinline__ double2 make(double a, double b) { return make_double2(a, b); } };
template <> struct V2<float> { using t = float2; static __device__ __forceinline__ float2 make(float a, float b) { return make_float2(a, b); } };

constexpr int NXD = (MAXN3 + 1) * (MAXN3 + 2) / 2;   // coefficients of degree <= MAXN3
__device__ __forceinline__ double2 cmulv(double2 a, double2 b)
{ return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }

__device__ __forceinline__ int dir_id(int dx, int dy, int dz) { return (dx + 3) * 49 + (dy + 3) * 7 + (dz + 3); }

struct ShiftSmem {
	double2 a[NX2MAX];
	double2 b[NX2MAX];
	double rn[2 * MAXN3 + 2];
};

__device__ __forceinline__ void rotate_y_t(const double2* __restrict__ in, double2* __restrict__ out,
                                           const double* __restrict__ D, int Nx2)
{
	const int lane = threadIdx.x & 31;
#pragma unroll
	for (int t = 0; t < CMAX; ++t) {
		int c = lane + 32 * t;
		if (c < Nx2) {
			const int n = tri_row(c), m = c - tix(n, 0);
			const double* Dr = D + dix(n, m, 0);
			double vr = 0, vi = 0;
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

// Scaled M2M from one of the 8 children (warp-cooperative), FP64: builds the
// dense operators.
__device__ inline void translate_scaled(const double2* __restrict__ src, int dirid, double2 (&acc)[CMAX], int N,
                                        int Nx2, ShiftSmem& sm, const DevTables& T, unsigned* flags)
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
	const double rho = 0.86602540378443864676;     // rho / h_child = sqrt(3) / 2
	for (int i = lane; i < N; i += 32) {
		double p = 1.0;
		for (int j = 0; j < i; ++j) p *= rho;
		sm.rn[i] = p;
	}
#pragma unroll
	for (int t = 0; t < CMAX; ++t) {
		int c = lane + 32 * t;
		if (c < Nx2) sm.a[c] = cmulv(src[c], E1[c - tix(tri_row(c), 0)]);
	}
	__syncwarp();
	rotate_y_t(sm.a, sm.b, D1, Nx2);
	__syncwarp();
#pragma unroll
	for (int t = 0; t < CMAX; ++t) {
		int c = lane + 32 * t;
		if (c < Nx2) {
			const int j = tri_row(c), k = c - tix(j, 0);
			const double* cf = T.m2m + (j * MAXN3 + k) * MAXN3;
			double sr = 0, si = 0;
			for (int n = 0; j - n >= k; ++n) {
				double f = cf[n] * sm.rn[n];
				double2 w = sm.b[tix(j - n, k)];
				sr = fma(f, w.x, sr); si = fma(f, w.y, si);
			}
			const double s = ldexp(1.0, -j);
			sm.a[c] = make_double2(sr * s, si * s);
		}
	}
	__syncwarp();
	rotate_y_t(sm.a, sm.b, D2, Nx2);
	__syncwarp();
#pragma unroll
	for (int t = 0; t < CMAX; ++t) {
		int c = lane + 32 * t;
		if (c < Nx2) {
			const double2 v = cmulv(sm.b[c], E2[c - tix(tri_row(c), 0)]);
			acc[t].x += v.x; acc[t].y += v.y;
		}
	}
	__syncwarp();
}

template <typename real> __device__ __forceinline__ real rsq(real x);
template <> __device__ __forceinline__ float rsq<float>(float x) { return rsqrtf(x); }
template <> __device__ __forceinline__ double rsq<double>(double x) { return rsqrt(x); }
template <typename from, typename to>
__global__ void convert_kernel(const from* __restrict__ in, to* __restrict__ out, size_t n)
{
	size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) out[i] = (to)in[i];
}

// FP32 near field on its own (few registers, high occupancy): one warp per
// leaf, targets in passes of up to 32; a pass of np <= 16 targets runs
// TP = np rounded up to a power of two targets at once and splits the
// sources into 32 / TP phases (groups of 4), summed by shuffles.  Sources of
// the leaf and its U list are staged 32 at a time as negated hi + lo offsets in the
// target leaf's frame, padded with zero charges to a multiple of 4 and read
// as float4; the self pair is only tested for in the leaf's own chunks.
// Partial sums over 16 sources in FP32, carried in FP64; 1/r from the
// hardware approximation (relative error below 2^-22.9; r^2 >= 1e-8 is never
// subnormal).  Writes pot (with the reference's self term) and field in
// input order; the expansions are added by eval_scaled_kernel.  One target per
// lane: two or three, which share the sources' reads, took 20.5 and 21.7 ms
// instead of 19.4 on the 16.8M workload (fewer resident warps).
__device__ __forceinline__ float rsqrt_approx(float x)
{
	float y;
	asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
	return y;
}

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// Sources are staged NEGATED (leaf centre minus source, hi and lo), so each
// offset is a packed add: dx = (xi + sx) + (xl + lx), the same value as the
// difference.  Two sources per packed FP32 instruction (add / mul / fma
// .f32x2, sm_100); the clamp and 1/r stay scalar.
template <bool SELF>
__device__ __forceinline__ void p2p_f32_chunk(const float* __restrict__ sx, const float* __restrict__ sy,
                                              const float* __restrict__ sz, const float* __restrict__ lx,
                                              const float* __restrict__ ly, const float* __restrict__ lz,
                                              const float* __restrict__ sq, int cnt4, int jb, int js, int self,
                                              float xi, float yi, float zi, float xl, float yl, float zl,
                                              double& pot, double& fx, double& fy, double& fz)
{
	const float2 xi2 = f2(xi, xi), yi2 = f2(yi, yi), zi2 = f2(zi, zi);
	const float2 xl2 = f2(xl, xl), yl2 = f2(yl, yl), zl2 = f2(zl, zl);
	const float eps2 = (float)FORCE_EPS2;
	for (int j0 = jb; j0 < cnt4; j0 += 4 * js) {
		float2 p = f2(0.f, 0.f), ax = p, ay = p, az = p;
#pragma unroll
		for (int h = 0; h < 4; ++h) {
			const int j = j0 + js * h;
			if (j < cnt4) {
				const float4 X = *reinterpret_cast<const float4*>(sx + j), Y = *reinterpret_cast<const float4*>(sy + j);
				const float4 Z = *reinterpret_cast<const float4*>(sz + j), XL = *reinterpret_cast<const float4*>(lx + j);
				const float4 YL = *reinterpret_cast<const float4*>(ly + j), ZL = *reinterpret_cast<const float4*>(lz + j);
				const float4 Q = *reinterpret_cast<const float4*>(sq + j);
				const float2 xs[2] = {f2(X.x, X.y), f2(X.z, X.w)}, ys[2] = {f2(Y.x, Y.y), f2(Y.z, Y.w)};
				const float2 zs[2] = {f2(Z.x, Z.y), f2(Z.z, Z.w)}, xls[2] = {f2(XL.x, XL.y), f2(XL.z, XL.w)};
				const float2 yls[2] = {f2(YL.x, YL.y), f2(YL.z, YL.w)}, zls[2] = {f2(ZL.x, ZL.y), f2(ZL.z, ZL.w)};
				const float2 qs[2] = {f2(Q.x, Q.y), f2(Q.z, Q.w)};
#pragma unroll
				for (int k = 0; k < 2; ++k) {
					const float2 dx = __fadd2_rn(__fadd2_rn(xi2, xs[k]), __fadd2_rn(xl2, xls[k]));
					const float2 dy = __fadd2_rn(__fadd2_rn(yi2, ys[k]), __fadd2_rn(yl2, yls[k]));
					const float2 dz = __fadd2_rn(__fadd2_rn(zi2, zs[k]), __fadd2_rn(zl2, zls[k]));
					const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
					const float2 inv = f2(rsqrt_approx(fmaxf(r2.x, eps2)), rsqrt_approx(fmaxf(r2.y, eps2)));
					float2 qi = __fmul2_rn(qs[k], inv);
					if (SELF) {
						if (j + 2 * k == self) qi.x = 0.f;
						if (j + 2 * k + 1 == self) qi.y = 0.f;
					}
					const float2 qi3 = __fmul2_rn(qi, __fmul2_rn(inv, inv));
					p = __fadd2_rn(p, qi);
					ax = __ffma2_rn(dx, qi3, ax); ay = __ffma2_rn(dy, qi3, ay); az = __ffma2_rn(dz, qi3, az);
				}
			}
		}
		pot += (double)p.x + (double)p.y; fx += (double)ax.x + (double)ax.y;
		fy += (double)ay.x + (double)ay.y; fz += (double)az.x + (double)az.y;
	}
}

template <int LW>
__global__ void __launch_bounds__(LW * 32, 768 / (LW * 32)) p2p_f32_kernel(DevTree t, double* __restrict__ pot_out,
                                                         double* __restrict__ fld_out, unsigned* __restrict__ next_leaf)
{
	__shared__ __align__(16) float sx[LW][32], sy[LW][32], sz[LW][32], sq[LW][32];
	__shared__ __align__(16) float lx[LW][32], ly[LW][32], lz[LW][32];
	const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const bool tmode = t.targets_num > 0;
	// a resident grid: each warp takes the next leaf from a counter
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
			int lt = 0;                            // log2 of the targets run at once
			while ((1 << lt) < np) ++lt;
			const int ti = lane & ((1 << lt) - 1), ph = lane >> lt, G = 32 >> lt;
			const uint32_t i = t0 + ti;
			const bool valid = ti < np;
			float xi = 0.f, yi = 0.f, zi = 0.f, xl = 0.f, yl = 0.f, zl = 0.f;
			if (valid) {
				const double ax_ = t.x[i] - cx, ay_ = t.y[i] - cy, az_ = t.z[i] - cz;
				xi = (float)ax_; yi = (float)ay_; zi = (float)az_;
				xl = (float)(ax_ - (double)xi); yl = (float)(ay_ - (double)yi); zl = (float)(az_ - (double)zi);
			}
			double pot = 0.0, fx = 0.0, fy = 0.0, fz = 0.0;
			for (int64_t e = (int64_t)ub - 1; e < (int64_t)ue; ++e) {
				const bool own = e < (int64_t)ub;
				const size_t sc_ = own ? g : (size_t)t.u_idx[e];
				const uint32_t sb = t.pbeg[sc_], se = t.send[sc_];
				for (uint32_t s0 = sb; s0 < se; s0 += 32) {
					const int cnt = min(32u, se - s0), cnt4 = (cnt + 3) & ~3;
					__syncwarp();
					if (lane < cnt) {
						const uint32_t j = s0 + lane;
						const double dx_ = cx - t.x[j], dy_ = cy - t.y[j], dz_ = cz - t.z[j];   // negated
						const float hx = (float)dx_, hy = (float)dy_, hz = (float)dz_;
						sx[w][lane] = hx; sy[w][lane] = hy; sz[w][lane] = hz;
						lx[w][lane] = (float)(dx_ - (double)hx); ly[w][lane] = (float)(dy_ - (double)hy);
						lz[w][lane] = (float)(dz_ - (double)hz);
						sq[w][lane] = (float)t.q[j];
					} else if (lane < cnt4) {
						sx[w][lane] = sy[w][lane] = sz[w][lane] = 0.f;
						lx[w][lane] = ly[w][lane] = lz[w][lane] = 0.f;
						sq[w][lane] = 0.f;
					}
					__syncwarp();
					if (valid) {
						if (own)
							p2p_f32_chunk<true>(sx[w], sy[w], sz[w], lx[w], ly[w], lz[w], sq[w], cnt4, 4 * ph, 4 * G,
							                    (int)(i - s0), xi, yi, zi, xl, yl, zl, pot, fx, fy, fz);
						else
							p2p_f32_chunk<false>(sx[w], sy[w], sz[w], lx[w], ly[w], lz[w], sq[w], cnt4, 4 * ph, 4 * G, -1, xi,
							                     yi, zi, xl, yl, zl, pot, fx, fy, fz);
					}
				}
			}
			for (int o = 1 << lt; o < 32; o <<= 1) {
				pot += __shfl_xor_sync(0xffffffffu, pot, o);
				fx += __shfl_xor_sync(0xffffffffu, fx, o);
				fy += __shfl_xor_sync(0xffffffffu, fy, o);
				fz += __shfl_xor_sync(0xffffffffu, fz, o);
			}
			if (valid && ph == 0) {
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

} // namespace scaled
} // namespace lfmm
