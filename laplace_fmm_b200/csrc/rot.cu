// Factored FP64 translations on the FP64 tensor cores (see rot.cuh).
#include "rot.cuh"
#include <algorithm>
#include <cmath>

namespace lfmm {

namespace {

constexpr int RT = 32;             // targets per tile: four 8-column MMA tiles
constexpr int RLD = 36;            // row stride (doubles) of a staged plane: the fragment reads are conflict-free
constexpr int RWMAX = 16;          // most warps per block
constexpr int RJOBS = 2;           // most jobs per warp
constexpr int RPAD = 4;            // zero rows behind the last block (the k padding reads past it)

// The (degree block, row tile) jobs of one warp; the same list serves all
// three products: a block of degree n has the size of the axial block of
// order N - 1 - n.
struct RotJobs {
	uint8_t n[RWMAX][RJOBS];
	uint8_t mt[RWMAX][RJOBS];
	uint8_t cnt[RWMAX];
};

struct RotSizes {
	double h[MAX_LEVELS];
};

// Axial blocks in fragment order: block n of table e is order m = N - 1 - n,
// rows and columns the degrees m .. N - 1.
__global__ void rot_axial_kernel(int N, RotSizes sz, bool scaled, DevTables T, double* __restrict__ out)
{
	const int F = rot_frag0(N);
	const int e = blockIdx.y, lv = blockIdx.z;
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= F * 32) return;
	const int f = i >> 5, lane = i & 31;
	int n = 0;
	while (rot_frag0(n + 1) <= f) ++n;
	const int kt = (f - rot_frag0(n)) % rot_ksteps(n), mt = (f - rot_frag0(n)) / rot_ksteps(n);
	const int r = 8 * mt + (lane >> 2), c = 4 * kt + (lane & 3);
	const int m = N - 1 - n, j = m + r, k = m + c;      // target and source degree
	double v = 0.0;
	if (r <= n && c <= n) {
		const double h = sz.h[lv];
		int p;
		double base;
		const double* cube;
		if (e < ROT_AX_M2M) {
			base = 1.0 / (h * sqrt((double)(e + 4)) + 1e-12);
			p = j + k + 1;
			cube = T.m2l + (j * MAXN3 + m) * MAXN3 + k;
		} else if (e == ROT_AX_M2M) {
			base = scaled ? 0.86602540378443864676 : 0.43301270189221932338 * h + 1e-12;
			p = j - k;
			cube = T.m2m + (j * MAXN3 + m) * MAXN3 + p;
		} else {
			base = scaled ? 0.43301270189221932338 : 0.86602540378443864676 * h + 1e-12;
			p = k - j;
			cube = T.l2l + (j * MAXN3 + m) * MAXN3 + k;
		}
		if (p >= 0) {
			double w = 1.0;
			for (int q = 0; q < p; ++q) w *= base;
			v = *cube * w;
			if (scaled && e >= ROT_AX_M2M) v = ldexp(v, e == ROT_AX_M2M ? -j : -(j + 1));
		}
	}
	out[((size_t)lv * ROT_AX + e) * F * 32 + i] = v;
}

template <typename real> struct C2;
template <> struct C2<double> { using t = double2; };
template <> struct C2<float> { using t = float2; };

inline int rot_rows(int N) { return N * (N + 1) / 2 + RPAD; }
inline int rot_raw_ld(int N) { return (N * (N + 1) / 2 + 3) / 8 * 8 + 4; }   // 4 mod 8, >= Nx2
inline size_t rot_planes(int N) { return sizeof(double) * 2 * (size_t)rot_rows(N) * RLD; }
inline size_t rot_raw(int N, size_t elem) { return elem * (size_t)RT * rot_raw_ld(N); }

// Dynamic shared memory of order N; apart: the raw gather has a place of its
// own beside X and Y where that leaves room for the blocks an SM holds (two up
// to N = 12), else it lies in Y: apart, the next slot's sources arrive during
// all three products instead of the last one.
size_t rot_smem(int N, size_t elem, bool& apart)
{
	const size_t room = N <= 12 ? (size_t)101 << 10 : (size_t)206 << 10;
	const size_t planes = rot_planes(N), raw = rot_raw(N, elem);
	apart = 2 * planes + raw <= room;
	return apart ? 2 * planes + raw : planes + std::max(planes, raw);
}

// Orders that share a kernel instance: the largest of N's.
constexpr int rot_last(int N) { return N <= 8 ? 8 : N <= 12 ? 12 : N <= 16 ? 16 : MAXN3; }

// The most shared memory that a launch of N's instance asks for.
size_t rot_smem_limit(int N, size_t elem)
{
	size_t most = 0;
	bool apart;
	for (int n = rot_last(N); n > 0 && rot_last(n) == rot_last(N); --n) most = std::max(most, rot_smem(n, elem, apart));
	return most;
}

// Block of 8 or 16 warps per (class, tile of at most 32 targets) and slot
// range.  Per
// non-empty slot, the sources present are gathered into consecutive columns
// (cp.async, ahead of their use), multiplied by e^{i m phi} into two planes
// (real, imaginary) of buffer X, and go through
//   Y = D(theta) X per degree,  X = Z Y per order,  acc += e^{-i m phi} D(-theta) X
// with the FP64 MMAs of a warp's jobs; the last product reads each target's
// column through the slot's map (absent: the zero column RT), so the
// accumulators (registers) stay with the targets while the first two run on
// the columns present only.  The matrices' fragments come from L2 (25 KB per
// slot at N = 9, 110 KB at N = 18), loaded for the next product before the
// barrier that precedes it.
// What bounds it: the FP64 MMAs are about a third of the time (N = 9: 31 % of
// the tensor pipe's active cycles), the rest is the four barriers and latencies of a
// slot, which is why a warp holds at most two jobs and an SM 16 warps (with 8
// warps of up to four jobs at N = 18 the M2L of 56k pairs took 491 us instead
// of 279).  Against dense operators on the same pipe (m8n8k4 MMAs over the
// N (N+1) square): M2L of 131,072 uniform particles, N = 9, 1222 -> 760 us; of
// 60,013 + 20,011 at N = 18, 4180 -> 371; of 300,007 clustered at N = 11 7674
// -> 2790; of 256 problems in one forest (13.8M particles, N = 15-18) levels
// 2 and 3 133.7 -> 32.6 ms.
template <typename real, int MODE, int RW, int JOBS, int KT>
__global__ void __launch_bounds__(RW * 32, RW == 8 ? 2 : 1) rot_kernel(const typename C2<real>::t* __restrict__ src,
                                                         typename C2<real>::t* __restrict__ dst,
                                                         const int32_t* __restrict__ vtab,
                                                         const int32_t* __restrict__ order,
                                                         const uint32_t* __restrict__ cls_count, int N,
                                                         const double2* __restrict__ rotf,
                                                         const double2* __restrict__ emat,
                                                         const int4* __restrict__ dirinfo,
                                                         const double* __restrict__ axial,
                                                         const __grid_constant__ RotJobs jobs, bool raw_apart, int tile,
                                                         double2* __restrict__ part, size_t cells, unsigned* flags)
{
	using v2 = typename C2<real>::t;
	constexpr int SLOTS = MODE == ROT_M2L ? M2L_SLOTS : MODE == ROT_M2M ? 8 : 1;
	extern __shared__ __align__(16) double sm_rot[];
	__shared__ uint32_t s_mask[SLOTS];
	__shared__ short4 s_dir[SLOTS];            // rotation slots (theta, -theta) and phase slots (phi, -phi)
	__shared__ int8_t s_ax[SLOTS];
	__shared__ int16_t s_list[SLOTS];
	__shared__ int32_t s_tgt[RT];
	__shared__ uint8_t s_m[MAXN3 * (MAXN3 + 1) / 2 + 1];
	// per job and lane: {X read offset, Y store offset, Y read offset, X store
	// offset}; a store offset of -1: the lane's row lies past the block
	__shared__ int4 s_off[RW * JOBS][32];
	__shared__ int s_cls, s_cnt, s_nt;
	__shared__ uint32_t s_start;
	const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
	const int Nx2 = N * (N + 1) / 2, rows = Nx2 + RPAD, F = rot_frag0(N);
	const int S = gridDim.y, sidx = blockIdx.y;
	const int slot0 = sidx * SLOTS / S, slot1 = (sidx + 1) * SLOTS / S;
	const int P = rows * RLD;
	double* X = sm_rot;                        // [2][rows][RLD], row tix(n, m)
	double* Y = sm_rot + 2 * P;                // [2][rows][RLD], orders one after another; or the raw gather
	if (tid == 0) {
		uint32_t b = blockIdx.x, start = 0;
		int cls = -1, nn = 0;
		for (int o = 0; o < (MODE == ROT_M2M ? 1 : 8); ++o) {
			const uint32_t cnt = cls_count[o], tiles = (cnt + tile - 1) / tile;
			if (b < tiles) { cls = o; start += b * tile; nn = (int)min((uint32_t)tile, cnt - b * tile); break; }
			b -= tiles; start += cnt;
		}
		s_cls = cls; s_nt = nn; s_start = start; s_cnt = 0;
	}
	__syncthreads();
	const int cls = s_cls;
	if (cls < 0) return;
	// X's zero column and padding rows (Y's are cleared in every slot); what the
	// columns of absent sources hold reaches no target
	for (int i = tid; i < 2 * rows; i += RW * 32) X[i * RLD + RT] = 0.0;
	if (tid < RPAD * RLD) X[Nx2 * RLD + tid] = X[P + Nx2 * RLD + tid] = 0.0;
	for (int c = tid; c < Nx2; c += RW * 32) s_m[c] = (uint8_t)(c - tix(tri_row(c), 0));
	const int32_t my_tgt = lane < s_nt ? order[s_start + lane] : -1;     // lane = target, every warp alike
	if (tid < RT) s_tgt[tid] = my_tgt;
	auto put_dir = [&](int sl, int dx, int dy, int dz, int e) {
		int4 di = dirinfo[(dx + 3) * 49 + (dy + 3) * 7 + (dz + 3)];
		if (di.x < 0 || di.y < 0 || di.z < 0 || di.w < 0) {
			atomicOr(flags, DEV_ERR_DIRECTION);
			di = make_int4(0, 0, 0, 0);
		}
		s_dir[sl] = make_short4((short)di.x, (short)di.y, (short)di.z, (short)di.w);
		s_ax[sl] = (int8_t)e;
	};
	if (MODE == ROT_M2L) {
		if (tid < 216) {
			// the class's far offsets in lexicographic order: slot = rank among
			// the 6^3 candidates without the 27 near ones
			const int ox = (cls >> 2) & 1, oy = (cls >> 1) & 1, oz = cls & 1;
			const int a = tid / 36, b = tid / 6 % 6, c = tid % 6;
			const int dx = a - 2 - ox, dy = b - 2 - oy, dz = c - 2 - oz;
			if (max(max(abs(dx), abs(dy)), abs(dz)) > 1) {
				const int na = min(max(a - ox - 1, 0), 3), nb = min(max(b - oy - 1, 0), 3), nc = min(max(c - oz - 1, 0), 3);
				const int near = 9 * na + (abs(dx) <= 1 ? 3 * nb + (abs(dy) <= 1 ? nc : 0) : 0);
				put_dir(tid - near, dx, dy, dz, dx * dx + dy * dy + dz * dz - 4);
			}
		}
	} else if (tid < SLOTS) {
		const int o = MODE == ROT_M2M ? tid : cls, sg = MODE == ROT_M2M ? 1 : -1;
		put_dir(tid, sg * (2 * ((o >> 2) & 1) - 1), sg * (2 * ((o >> 1) & 1) - 1), sg * (2 * (o & 1) - 1),
		        MODE == ROT_M2M ? ROT_AX_M2M : ROT_AX_L2L);
	}
	for (int sl = slot0 + w; sl < slot1; sl += RW) {
		const int32_t v = my_tgt >= 0 ? vtab[(size_t)my_tgt * SLOTS + sl] : -1;
		const uint32_t mk = __ballot_sync(0xffffffffu, v >= 0);
		if (lane == 0) s_mask[sl] = mk;
	}
	const int njobs = jobs.cnt[w];
	int jn[JOBS], jk[JOBS], jf[JOBS];          // degree (block) and row tile << 8, k steps, first fragment
#pragma unroll
	for (int q = 0; q < JOBS; ++q) {
		const int n = q < njobs ? jobs.n[w][q] : 0, mt = q < njobs ? jobs.mt[w][q] : 0;
		jn[q] = n | mt << 8; jk[q] = rot_ksteps(n); jf[q] = rot_frag0(n) + mt * rot_ksteps(n);
		const int r = 8 * mt + g, m = N - 1 - n;           // row in the block; the axial block's order
		int4 o;
		o.x = (tix(n, 0) + t4) * RLD;
		o.y = r <= n ? (r * N - r * (r - 1) / 2 + n - r) * RLD + 2 * t4 : -1;
		o.z = (m * N - m * (m - 1) / 2 + t4) * RLD;
		o.w = r <= n ? tix(m + r, m) * RLD + 2 * t4 : -1;
		s_off[w * JOBS + q][lane] = o;
	}
	__syncthreads();
	if (tid < 32) {                            // the non-empty slots, in order
		int n = 0;
		for (int b = slot0; b < slot1; b += 32) {
			const bool on = b + lane < slot1 && s_mask[b + lane] != 0;
			const uint32_t mk = __ballot_sync(0xffffffffu, on);
			if (on) s_list[n + __popc(mk & ((1u << lane) - 1))] = (int16_t)(b + lane);
			n += __popc(mk);
		}
		if (lane == 0) s_cnt = n;
	}
	__syncthreads();
	const int nl = s_cnt;
	const int raw_ld = (Nx2 + 3) / 8 * 8 + 4, Q4 = (Nx2 + 3) >> 2;
	v2* raw = reinterpret_cast<v2*>(raw_apart ? Y + 2 * P : Y);
	// this lane's source in slot list entry j
	auto source_of = [&](int j) -> int32_t {
		if (j >= nl) return -1;
		const int sl = s_list[j];
		return (s_mask[sl] >> lane) & 1u ? vtab[(size_t)my_tgt * SLOTS + sl] : -1;
	};
	// gather of a slot with sources v (mask mk): column = rank of the target
	// among those present; warp w brings in targets w, w + 8, ...
	auto gather = [&](uint32_t mk, int32_t v) {
#pragma unroll
		for (int i = 0; i < RT / RW; ++i) {
			const int t = w + RW * i;
			const int32_t s = __shfl_sync(0xffffffffu, v, t);
			if ((mk >> t) & 1u) {
				const v2* from = src + (size_t)s * Nx2;
				v2* to = raw + __popc(mk & ((1u << t) - 1)) * raw_ld;
				for (int c = lane; c < Nx2; c += 32) {
					if constexpr (sizeof(real) == sizeof(double)) cp_async16(to + c, from + c);
					else cp_async8(to + c, from + c);
				}
			}
		}
		cp_async_commit();
	};
	auto load_rot = [&](double2 (&a)[KT], int slot_d, int q) {
		const double2* f = rotf + ((size_t)slot_d * rot_frag0(MAXN3) + jf[q]) * 32 + lane;
#pragma unroll
		for (int k = 0; k < KT; ++k)
			if (k < jk[q]) a[k] = f[k * 32];
	};
	auto load_ax = [&](double2 (&a)[KT], const double* tab, int q) {
		const double* f = tab + (size_t)jf[q] * 32 + lane;
#pragma unroll
		for (int k = 0; k < KT; ++k)
			if (k < jk[q]) a[k].x = f[k * 32];
	};
	// one plane's product of a job on nct column tiles: to = A from
	auto product = [&](const double2 (&a)[KT], bool im, int K, int nct, const double* from, double* to, int st) {
		double c[4][2];
#pragma unroll
		for (int ct = 0; ct < 4; ++ct) c[ct][0] = c[ct][1] = 0.0;
		if (nct == 4) {
#pragma unroll
			for (int k = 0; k < KT; ++k)
				if (k < K) {
					double b[4];
#pragma unroll
					for (int ct = 0; ct < 4; ++ct) b[ct] = from[4 * k * RLD + 8 * ct];
#pragma unroll
					for (int ct = 0; ct < 4; ++ct) dmma(c[ct], im ? a[k].y : a[k].x, b[ct]);
				}
		} else {
#pragma unroll
			for (int k = 0; k < KT; ++k)
				if (k < K) {
#pragma unroll
					for (int ct = 0; ct < 3; ++ct)
						if (ct < nct) dmma(c[ct], im ? a[k].y : a[k].x, from[4 * k * RLD + 8 * ct]);
				}
		}
		if (st >= 0) {
#pragma unroll
			for (int ct = 0; ct < 4; ++ct)
				if (ct < nct) *reinterpret_cast<double2*>(to + st + 8 * ct) = make_double2(c[ct][0], c[ct][1]);
		}
	};
	double acc[JOBS][4][2][2];                 // [job][column tile][re, im][column 2 t4 + 0, 1]
#pragma unroll
	for (int q = 0; q < JOBS; ++q)
#pragma unroll
		for (int ct = 0; ct < 4; ++ct) acc[q][ct][0][0] = acc[q][ct][0][1] = acc[q][ct][1][0] = acc[q][ct][1][1] = 0.0;
	double2 an[KT];
#pragma unroll
	for (int k = 0; k < KT; ++k) an[k] = make_double2(0.0, 0.0);
	short4 di = make_short4(0, 0, 0, 0);
	int32_t vn = source_of(0);                 // one slot ahead of its gather
	if (nl > 0) {
		gather(s_mask[s_list[0]], vn);
		vn = source_of(1);
		di = s_dir[s_list[0]];
		if (njobs) load_rot(an, di.x, 0);
	}
	for (int j = 0; j < nl; ++j) {
		const int sl = s_list[j], sln = s_list[min(j + 1, nl - 1)];
		const uint32_t mk = s_mask[sl];
		const int p = __popc(mk), nct = (p + 7) >> 3;
		const bool more = j + 1 < nl;
		const double* ax = axial + (size_t)s_ax[sl] * F * 32;
		cp_async_wait<0>();
		__syncthreads();
		{
			// raw columns times e^{i m phi} -> planes; warp: 8 columns x 4 coefficients at a time
			const double2* E1 = emat + di.z * MAXN3;
			int c4 = w, cg = 0;
			for (;;) {
				while (c4 >= Q4) { c4 -= Q4; ++cg; }
				if (cg >= nct) break;
				const int col = 8 * cg + g, c = 4 * c4 + t4;
				if (col < p && c < Nx2) {
					const v2 a = raw[col * raw_ld + c];
					const double2 e = E1[s_m[c]];
					double* x = X + c * RLD + col;
					x[0] = (double)a.x * e.x - (double)a.y * e.y;
					x[P] = (double)a.x * e.y + (double)a.y * e.x;
				}
				c4 += RW;
			}
		}
		__syncthreads();
		if (raw_apart && more) { gather(s_mask[sln], vn); vn = source_of(j + 2); }
		if (tid < RPAD * RLD) { Y[Nx2 * RLD + tid] = 0.0; Y[P + Nx2 * RLD + tid] = 0.0; }
		// Y = D(theta) X, per degree n
#pragma unroll
		for (int q = 0; q < JOBS; ++q) {
			if (q < njobs) {
				const int q1 = q + 1 < JOBS ? q + 1 : q;
				const bool last = q + 1 >= JOBS || q + 1 >= njobs;
				const int4 o = s_off[w * JOBS + q][lane];
				product(an, false, jk[q], nct, X + o.x + g, Y, o.y);
				product(an, true, jk[q], nct, X + P + o.x + g, Y + P, o.y);
				if (last) load_ax(an, ax, 0); else load_rot(an, di.x, q1);
			}
		}
		__syncthreads();
		// X = Z Y, per order m = N - 1 - n
#pragma unroll
		for (int q = 0; q < JOBS; ++q) {
			if (q < njobs) {
				const int q1 = q + 1 < JOBS ? q + 1 : q;
				const bool last = q + 1 >= JOBS || q + 1 >= njobs;
				const int4 o = s_off[w * JOBS + q][lane];
				product(an, false, jk[q], nct, Y + o.z + g, X, o.w);
				product(an, false, jk[q], nct, Y + P + o.z + g, X + P, o.w);
				if (last) load_rot(an, di.y, 0); else load_ax(an, ax, q1);
			}
		}
		__syncthreads();
		const short4 dc = di;
		di = s_dir[sln];
		if (!raw_apart && more) { gather(s_mask[sln], vn); vn = source_of(j + 2); }
		// acc += e^{-i m phi} D(-theta) X, target columns through the map
		int pos[4];
#pragma unroll
		for (int ct = 0; ct < 4; ++ct) {
			const int c = 8 * ct + g;
			pos[ct] = (mk >> c) & 1u ? __popc(mk & ((1u << c) - 1)) : RT;
		}
#pragma unroll
		for (int q = 0; q < JOBS; ++q) {
			if (q < njobs) {
				const int q1 = q + 1 < JOBS ? q + 1 : q;
				const bool last = q + 1 >= JOBS || q + 1 >= njobs;
				const int4 o = s_off[w * JOBS + q][lane];
				const int m = min(8 * (jn[q] >> 8) + g, N - 1);
				const double2 e = emat[dc.w * MAXN3 + m];
				const double* xb = X + o.x;
#pragma unroll
				for (int ct = 0; ct < 4; ++ct)
					if ((mk >> (8 * ct)) & 0xffu) {
						double cr[2] = {0.0, 0.0}, ci[2] = {0.0, 0.0};
						const double* xc = xb + pos[ct];
#pragma unroll
						for (int k = 0; k < KT; ++k)
							if (k < jk[q]) {
								const double br = xc[4 * k * RLD], bi = xc[P + 4 * k * RLD];
								dmma(cr, an[k].x, br);
								dmma(ci, an[k].y, bi);
							}
#pragma unroll
						for (int h = 0; h < 2; ++h) {
							acc[q][ct][0][h] = fma(cr[h], e.x, fma(-ci[h], e.y, acc[q][ct][0][h]));
							acc[q][ct][1][h] = fma(cr[h], e.y, fma(ci[h], e.x, acc[q][ct][1][h]));
						}
					}
				if (!last) load_rot(an, dc.y, q1); else if (more) load_rot(an, di.x, 0);
			}
		}
	}
	if (S > 1) part += (size_t)sidx * cells * Nx2;
#pragma unroll
	for (int q = 0; q < JOBS; ++q) {
		const int n = jn[q] & 255, m = 8 * (jn[q] >> 8) + g;
		if (q < njobs && m <= n) {
#pragma unroll
			for (int ct = 0; ct < 4; ++ct)
#pragma unroll
				for (int h = 0; h < 2; ++h) {
					const int32_t tg = s_tgt[8 * ct + 2 * t4 + h];
					if (tg < 0) continue;
					const size_t o = (size_t)tg * Nx2 + tix(n, m);
					double2 v = make_double2(acc[q][ct][0][h], acc[q][ct][1][h]);
					if (S > 1) { part[o] = v; continue; }
					v2 out;
					if (MODE == ROT_L2L) { const v2 a = dst[o]; v.x += (double)a.x; v.y += (double)a.y; }
					out.x = (real)v.x; out.y = (real)v.y;
					dst[o] = out;
				}
		}
	}
}

// The S partial sums of every coefficient added in order.
template <typename real>
__global__ void rot_reduce_kernel(const double* __restrict__ part, real* __restrict__ dst, size_t n, int S)
{
	const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	double s = part[i];
	for (int k = 1; k < S; ++k) s += part[(size_t)k * n + i];
	dst[i] = (real)s;
}

// Longest-first assignment of the (block, row tile) jobs of order N to nw
// warps, at most RJOBS each; returns the longest list.
int rot_jobs(int N, int nw, RotJobs& J)
{
	J = RotJobs{};
	int load[RWMAX] = {}, most = 0;
	for (int n = N - 1; n >= 0; --n)
		for (int mt = 0; mt < rot_mtiles(n); ++mt) {
			int best = -1;
			for (int w = 0; w < nw; ++w)
				if (J.cnt[w] < RJOBS && (best < 0 || load[w] < load[best])) best = w;
			J.n[best][J.cnt[best]] = (uint8_t)n;
			J.mt[best][J.cnt[best]] = (uint8_t)mt;
			load[best] += rot_ksteps(n);
			most = std::max(most, (int)++J.cnt[best]);
		}
	return most;
}

// M2M plan of level L: the non-leaf cells (order, one class; a leaf keeps its
// P2M expansion) and their children by octant (vtab[cell][8]: level-local
// index at L + 1, or -1).
__global__ void m2m_plan_kernel(DevTree t, int L, int32_t* __restrict__ vtab, int32_t* __restrict__ order,
                                uint32_t* __restrict__ count)
{
	const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (c >= t.lsize[L]) return;
	const size_t g = t.loff[L] + c, cb = t.loff[L + 1];
	if (t.beg[g] >= t.end[g]) return;
	for (uint32_t k = t.beg[g]; k < t.end[g]; ++k) vtab[c * 8 + (size_t)(t.code[cb + k] & 7ull)] = (int32_t)k;
	order[atomicAdd(count, 1u)] = (int32_t)c;
}

} // namespace

int m2m_plan_build(Context& ctx, const DevTree& t, int L, M2LPlan& plan)
{
	const size_t m = t.lsize[L];
	plan.cells = m;
	plan.vtab = static_cast<int32_t*>(ctx.arena.take(sizeof(int32_t) * 8 * m));
	plan.order = static_cast<int32_t*>(ctx.arena.take(sizeof(int32_t) * m));
	plan.oct_count = static_cast<uint32_t*>(ctx.arena.take(sizeof(uint32_t) * 8));
	if (!plan.vtab || !plan.order || !plan.oct_count) { ctx.last_error = "m2m plan: allocation failed"; return ERR_OOM; }
	LFMM_CUDA(ctx, cudaMemsetAsync(plan.vtab, 0xff, sizeof(int32_t) * 8 * m, ctx.stream));
	LFMM_CUDA(ctx, cudaMemsetAsync(plan.oct_count, 0, sizeof(uint32_t) * 8, ctx.stream));
	m2m_plan_kernel<<<div_up(m, 256), 256, 0, ctx.stream>>>(t, L, plan.vtab, plan.order, plan.oct_count);
	LFMM_CUDA(ctx, cudaGetLastError());
	return OK;
}

const double* rot_axial_tables(Context& ctx, int N, const double* h, int nh, bool scaled)
{
	const int F = rot_frag0(N);
	double* out = static_cast<double*>(ctx.arena.take(sizeof(double) * (size_t)nh * ROT_AX * F * 32));
	if (!out) { ctx.last_error = "axial tables: allocation failed"; return nullptr; }
	RotSizes sz{};
	for (int i = 0; i < nh; ++i) sz.h[i] = h[i];
	rot_axial_kernel<<<dim3(div_up(F * 32, 256), ROT_AX, nh), 256, 0, ctx.stream>>>(N, sz, scaled, ctx.tables.d, out);
	if (cudaGetLastError() != cudaSuccess) { ctx.last_error = "axial tables: launch failed"; return nullptr; }
	return out;
}

template <typename real>
int rot_translate(Context& ctx, RotMode mode, const M2LPlan& plan, const real* src, real* dst, int N,
                  const double* axial)
{
	using v2 = typename C2<real>::t;
	if (N < 1 || N > MAXN3) { ctx.last_error = "translations: order out of range"; return ERR_UNSUPPORTED; }
	if (plan.cells == 0) return OK;
	// targets per tile: fewer than 32 where that still leaves at most one block
	// per SM (a slot's three products are shorter, its latencies stay)
	int tile = RT;
	if (mode != ROT_M2L)
		while (tile > 8 && plan.cells / (tile / 2) + 8 <= (size_t)ctx.num_sms) tile /= 2;
	const unsigned tiles = (unsigned)(plan.cells / tile + (mode == ROT_M2M ? 1 : 8));
	// slots per block: the split S that needs the fewest rounds of blocks (the
	// octant classes are about equal), a block costing its share of the 189
	// slots and about 3 slots' time beside them (filling the buffers, the slot
	// list, the partial sums)
	int S = 1;
	double* part = nullptr;
	if (mode == ROT_M2L) {
		const double full = 8.0 * (double)((plan.cells + 8 * RT - 1) / (8 * RT));
		const double per_round = (N <= 12 ? 2.0 : 1.0) * ctx.num_sms;
		double best = 1e300;
		for (int k = 1; k <= 32; ++k) {
			const double t = std::ceil(full * k / per_round) * ((double)M2L_SLOTS / k + 3.0);
			if (t < 0.98 * best) { best = t; S = k; }
		}
		if (S > 1) {
			part = static_cast<double*>(ctx.arena.take(sizeof(double) * (size_t)S * plan.cells * N * (N + 1)));
			if (!part) S = 1;
		}
	}
	// 8 warps in blocks of which an SM holds two up to N = 12 (16 jobs); above,
	// the buffers leave room for one block, of 16 warps (N = 18: 30 jobs)
	const int nw = N <= 12 ? 8 : 16;
	RotJobs J;
	rot_jobs(N, nw, J);
	bool apart;
	const size_t smem = rot_smem(N, sizeof(v2), apart), limit = rot_smem_limit(N, sizeof(v2));
	cudaStream_t s = ctx.stream;
	const DevTables& T = ctx.tables.d;
	auto go = [&](auto kern) -> cudaError_t {
		const cudaError_t e = smem_limit(ctx.device, reinterpret_cast<const void*>(kern), limit, true);
		if (e != cudaSuccess) return e;
		kern<<<dim3(tiles, S), nw * 32, smem, s>>>(reinterpret_cast<const v2*>(src), reinterpret_cast<v2*>(dst), plan.vtab,
		                                           plan.order, plan.oct_count, N, T.rotf, T.emat, T.dirinfo, axial, J, apart, tile,
		                                           reinterpret_cast<double2*>(part), plan.cells, ctx.dev_flags);
		return cudaGetLastError();
	};
	cudaError_t e = cudaErrorInvalidValue;
	// <warps, jobs per warp, k steps of the largest block>
#define LFMM_ROT_GO(MODE)                                                                                             \
	if (N <= 8) e = go(rot_kernel<real, MODE, 8, 1, 2>);                                                              \
	else if (N <= 12) e = go(rot_kernel<real, MODE, 8, 2, 3>);                                                        \
	else if (N <= 16) e = go(rot_kernel<real, MODE, 16, 2, 4>);                                                       \
	else e = go(rot_kernel<real, MODE, 16, 2, 5>);
	if (mode == ROT_M2L) { LFMM_ROT_GO(ROT_M2L) }
	else if (mode == ROT_M2M) { LFMM_ROT_GO(ROT_M2M) }
	else { LFMM_ROT_GO(ROT_L2L) }
#undef LFMM_ROT_GO
	if (e != cudaSuccess) return cuda_fail(ctx, e, "rot_kernel");
	if (S > 1) {
		const size_t nel = plan.cells * (size_t)N * (N + 1);
		rot_reduce_kernel<real><<<div_up(nel, 256), 256, 0, s>>>(part, dst, nel, S);
		LFMM_CUDA(ctx, cudaGetLastError());
	}
	return OK;
}

template int rot_translate<double>(Context&, RotMode, const M2LPlan&, const double*, double*, int, const double*);
template int rot_translate<float>(Context&, RotMode, const M2LPlan&, const float*, float*, int, const double*);

} // namespace lfmm
