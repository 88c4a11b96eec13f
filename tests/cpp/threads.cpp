// Two host threads, a context each, solving at different orders at the same
// time: threads <dim> <precision> <N0> <N1> <depth> <max_leaf> <rounds>.
// precision: 0 FP64, 1 mixed; 2: thread 0 executes a mixed plan instead.
// Prints the failed and the changed calls of each thread and the last error.
// Every change of a kernel's attributes is followed by a pause in which the
// other thread runs, so a limit set for one launch meets the other's.
#include "lfmm.h"
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>
#include <thread>
#include <vector>

#include <chrono>
#include <cuda_runtime.h>
#include <dlfcn.h>

// takes the runtime's place for the library
extern "C" cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v)
{
	using fn = cudaError_t (*)(const void*, cudaFuncAttribute, int);
	static fn real = reinterpret_cast<fn>(dlsym(RTLD_NEXT, "cudaFuncSetAttribute"));
	const cudaError_t e = real ? real(f, a, v) : cudaErrorUnknown;
	std::this_thread::sleep_for(std::chrono::microseconds(200));
	return e;
}

int main(int argc, char** argv)
{
	if (argc != 8) return 2;
	const int dim = std::atoi(argv[1]), form = std::atoi(argv[2]), N[2] = {std::atoi(argv[3]), std::atoi(argv[4])};
	const int depth = std::atoi(argv[5]), max_leaf = std::atoi(argv[6]), rounds = std::atoi(argv[7]);
	const size_t n = 3000;
	std::mt19937_64 rng(5);
	std::uniform_real_distribution<double> u(0.0, 1.0);
	std::vector<double> x(dim * n), q(n);
	for (auto& v : x) v = u(rng);
	for (auto& v : q) v = u(rng) - 0.5;
	std::atomic<int> ready{0};
	int failed[2] = {0, 0}, changed[2] = {0, 0};
	std::string msg[2];
	auto work = [&](int k) {
		lfmm_ctx* ctx = nullptr;
		lfmm_options o{};
		if (lfmm_create(&ctx, &o) != LFMM_OK) { failed[k] = -1; ++ready; return; }
		lfmm_solve_opts s{N[k], depth, max_leaf, form ? LFMM_PRECISION_MIXED : LFMM_PRECISION_FP64, 1e-8};
		std::vector<double> pot(n), fld(dim * n), pot0, fld0;
		const bool plan = form == 2 && k == 0;
		double *dx = nullptr, *dq = nullptr, *dp = nullptr, *df = nullptr;
		lfmm_plan* P = nullptr;
		if (plan) {
			cudaMalloc(&dx, sizeof(double) * 3 * n); cudaMalloc(&dq, sizeof(double) * n);
			cudaMalloc(&dp, sizeof(double) * n); cudaMalloc(&df, sizeof(double) * 3 * n);
			cudaMemcpy(dx, x.data(), sizeof(double) * 3 * n, cudaMemcpyHostToDevice);
			cudaMemcpy(dq, q.data(), sizeof(double) * n, cudaMemcpyHostToDevice);
			if (lfmm3d_plan_create(ctx, n, dx, dq, &s, &P) != LFMM_OK) failed[k] = -2;
		}
		auto once = [&]() -> int {
			if (plan) {
				const int st = P ? lfmm3d_plan_execute(P, dq, dp, df) : LFMM_ERR_ARG;
				if (st) return st;
				if (cudaStreamSynchronize((cudaStream_t)lfmm_stream(ctx)) != cudaSuccess) return LFMM_ERR_CUDA;
				cudaMemcpy(pot.data(), dp, sizeof(double) * n, cudaMemcpyDeviceToHost);
				cudaMemcpy(fld.data(), df, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost);
				return LFMM_OK;
			}
			return dim == 2 ? lfmm2d_solve_ex(ctx, n, x.data(), q.data(), 0, nullptr, &s, pot.data(), fld.data(), nullptr)
			                : lfmm3d_solve_ex(ctx, n, x.data(), q.data(), 0, nullptr, &s, pot.data(), fld.data(), nullptr);
		};
		// the other thread's first solves race with these, so a failure here counts too
		for (int r = 0; r < 3; ++r)
			if (once() != LFMM_OK) { ++failed[k]; msg[k] = lfmm_last_error(ctx); }
		++ready;
		while (ready.load() < 2) std::this_thread::yield();
		for (int r = 0; r < rounds; ++r) {
			if (once() != LFMM_OK) { ++failed[k]; msg[k] = lfmm_last_error(ctx); continue; }
			if (pot0.empty()) { pot0 = pot; fld0 = fld; }
			if (std::memcmp(pot.data(), pot0.data(), sizeof(double) * n) ||
			    std::memcmp(fld.data(), fld0.data(), sizeof(double) * dim * n))
				++changed[k];
		}
		lfmm3d_plan_destroy(P);
		cudaFree(dx); cudaFree(dq); cudaFree(dp); cudaFree(df);
		lfmm_destroy(ctx);
	};
	std::thread a(work, 0), b(work, 1);
	a.join();
	b.join();
	std::printf("failed %d %d changed %d %d %s|%s\n", failed[0], failed[1], changed[0], changed[1], msg[0].c_str(),
	            msg[1].c_str());
	return failed[0] || failed[1] || changed[0] || changed[1];
}
