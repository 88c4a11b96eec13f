// Shared device/host helpers for the B200 Laplace FMM (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstddef>

namespace lfmm {

constexpr int WARP = 32;
constexpr double FORCE_EPS = 1.0e-4;            // distance clamp (reference common/defs.h:24)
constexpr double FORCE_EPS2 = FORCE_EPS * FORCE_EPS;
constexpr int MAXN3 = 18;                       // max degrees in 3D (reference common/defs.h:33)
constexpr int MAXN2 = 30;                       // max degrees in 2D (reference common/defs.h:32)
constexpr int AUTO = 0x7fffffff;                // FMM_AUTO (reference common/defs.h:22)
constexpr double PI = 3.14159265358979323846;

// Triangular (n,m) index, 0 <= m <= n (reference common/utils.h:130-147).
__host__ __device__ constexpr inline int tix(int n, int m) { return n * (n + 1) / 2 + m; }
// The degree n of triangular index c = tix(n, m) (m = c - tix(n, 0)), computed
// rather than looked up: lanes of a warp ask for different c, which a
// constant-memory table would serialise.
__device__ __forceinline__ int tri_row(int c)
{
	// n = (sqrt(8c + 1) - 1) / 2 from the hardware reciprocal square root
	// (r >= 1); the estimate is within one of n, which the two steps correct
	const float r = 8.f * (float)c + 1.f;
	int n = (int)((r * rsqrtf(r) - 1.f) * 0.5f);
	if (tix(n + 1, 0) <= c) ++n;
	if (tix(n, 0) > c) --n;
	return n;
}
// Wigner-d (n,m,k) index, |k| <= n (reference common/special_functions.cpp:216-221).
__host__ __device__ constexpr inline int dix(int n, int m, int k)
{ return n * (n + 1) * (4 * n - 1) / 6 + m * (2 * n + 1) + (k + n); }
__host__ __device__ constexpr inline int dsize(int N) { return N * (N + 1) * (4 * N - 1) / 6; }
__host__ __device__ constexpr inline double sgn_n(int n) { return (n & 1) ? -1.0 : 1.0; }

// Status codes returned across the C ABI.
enum Status : int {
	OK = 0,
	ERR_ARG = -1,
	ERR_CUDA = -2,
	ERR_OOM = -3,
	ERR_DEVICE = -4,     // a device-side check failed (error flag set by a kernel)
	ERR_UNSUPPORTED = -5,
};

// Device-side error flags, OR-ed by kernels that detect a broken invariant;
// the host reads them after a solve and turns them into ERR_DEVICE.
enum DeviceError : unsigned {
	DEV_ERR_LIST_OVERFLOW = 1u,
	DEV_ERR_DIRECTION = 2u,
	DEV_ERR_RANGE = 4u,
};

template <typename T>
__device__ __forceinline__ T warp_sum(T v)
{
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	return v;
}

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

// (-1)^n as a double
__device__ __forceinline__ double dsgn(int n) { return (n & 1) ? -1.0 : 1.0; }

// x >= 1e300, infinite, NaN or negative, from the high word: an integer
// comparison, since the kernels that ask are bound by the FP64 pipe.
__device__ __forceinline__ bool beyond_1e300(double x) { return (unsigned)__double2hiint(x) >= 0x7E37E43Cu; }

// 1 / sqrt(x), x > 0: the hardware's FP64 reciprocal square root approximation
// (rsqrt.approx.ftz.f64, no FP32 round trip; measured seed error 2^-20.1)
// refined by one third-order step of the binomial series (1 - r)^(-1/2) =
// 1 + r/2 + 3r^2/8 + ..., r = 1 - x y^2: a seed error e leaves ~(5/16)(2e)^3, below
// FP64 rounding for e < 2^-18, beside the roundings of x y (half of 2^-53) and of
// the last sum (2^-53; measured 1.4e-16 in all).  The FP64 square root and divide
// above 1e300.
__device__ __forceinline__ double rsqrt_below_1e300(double x)
{
	double y;
	asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
	const double r = fma(-x * y, y, 1.0);
	return fma(y * r, fma(r, 0.375, 0.5), y);
}
__device__ __forceinline__ double rsqrt_refined(double x)
{
	return beyond_1e300(x) ? 1.0 / sqrt(x) : rsqrt_below_1e300(x);
}

// q / x, x > 0; plain: |q| is below 1e300.  The hardware's FP64 reciprocal
// approximation y (1 - x y = e) refined once, y (1 + e), off by e^2 < 2^-36 for a
// seed error below 2^-18; then the quotient q y corrected by its remainder, which
// leaves the rounding of the last sum (2^-72 before it).  The FP64 divide where q
// or x is not below 1e300.
__device__ __forceinline__ double quotient_refined(double q, double x, bool plain)
{
	if (beyond_1e300(x) || !plain) return q / x;
	double y;
	asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
	y = fma(y, fma(-x, y, 1.0), y);
	const double p = q * y;
	return fma(fma(-p, x, q), y, p);
}

// FP64 tensor-core MMA (mma.sync m8n8k4): D = A B + D, A 8x4 (lane: row lane/4,
// column lane%4), B 4x8 (lane: row lane%4, column lane/4), D 8x8 (lane: row
// lane/4, columns 2 (lane%4) + 0, 1).
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b)
{
	asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
	             : "+d"(d[0]), "+d"(d[1])
	             : "d"(a), "d"(b));
}

// Asynchronous copies to shared memory: bytes < 16 fills the rest with zeros.
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes = 16)
{
	const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src)
{
	const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
	asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(PENDING) : "memory"); }

// Morton helpers: spread / gather every dim-th bit.
__host__ __device__ inline uint64_t spread3(uint64_t v)
{
	v &= 0x1fffffull;
	v = (v | (v << 32)) & 0x001f00000000ffffull;
	v = (v | (v << 16)) & 0x001f0000ff0000ffull;
	v = (v | (v << 8)) & 0x100f00f00f00f00full;
	v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
	v = (v | (v << 2)) & 0x1249249249249249ull;
	return v;
}
__host__ __device__ inline uint32_t compact3(uint64_t v)
{
	v &= 0x1249249249249249ull;
	v = (v ^ (v >> 2)) & 0x10c30c30c30c30c3ull;
	v = (v ^ (v >> 4)) & 0x100f00f00f00f00full;
	v = (v ^ (v >> 8)) & 0x001f0000ff0000ffull;
	v = (v ^ (v >> 16)) & 0x001f00000000ffffull;
	v = (v ^ (v >> 32)) & 0x1fffffull;
	return (uint32_t)v;
}
__host__ __device__ inline uint64_t spread2(uint64_t v)
{
	v &= 0xffffffffull;
	v = (v | (v << 16)) & 0x0000ffff0000ffffull;
	v = (v | (v << 8)) & 0x00ff00ff00ff00ffull;
	v = (v | (v << 4)) & 0x0f0f0f0f0f0f0f0full;
	v = (v | (v << 2)) & 0x3333333333333333ull;
	v = (v | (v << 1)) & 0x5555555555555555ull;
	return v;
}
__host__ __device__ inline uint32_t compact2(uint64_t v)
{
	v &= 0x5555555555555555ull;
	v = (v ^ (v >> 1)) & 0x3333333333333333ull;
	v = (v ^ (v >> 2)) & 0x0f0f0f0f0f0f0f0full;
	v = (v ^ (v >> 4)) & 0x00ff00ff00ff00ffull;
	v = (v ^ (v >> 8)) & 0x0000ffff0000ffffull;
	v = (v ^ (v >> 16)) & 0x00000000ffffffffull;
	return (uint32_t)v;
}

inline unsigned div_up(size_t a, size_t b) { return (unsigned)((a + b - 1) / b); }

} // namespace lfmm
