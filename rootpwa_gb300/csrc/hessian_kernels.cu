// hessian_kernels.cu -- per-event operands of the analytic Hessian.
//
// The event term of pwaLikelihood::Hessian (partialWaveFit/pwaLikelihood.cc:
// 676-735) is a sum over events of products of
//   d_s = S_{r(s),e(s)} conj(A_{w(s)})      (slot s = (rank, wave))
// weighted by f^2 (f = 2/L) plus a same-(rank, reflectivity) block of
// f A_i conj(A_j).  This kernel writes, for one slab of events, the complex
// columns [d; conj(d); 1] and [A; 1] with weights f^2 and f, so that two
// weighted complex Gram products (the tensor-core Gram of gram_tc.cu, TF32x3,
// in pairs of 48-row groups for the wide first set) yield
//   sum f^2 d_i conj(d_j), sum f^2 d_i d_j, sum f^2 d_i, sum f^2,
//   sum f A_i conj(A_j), sum f
// from which the host assembles the three real blocks the reference keeps
// per slot pair.  Coherent sums are FP32; the Gram sums FP32 in tensor
// memory per few tiles and FP64 across CTAs and slabs.

#include "pwa_internal.h"

#include <algorithm>

namespace pwa {
namespace {

constexpr int kMaxRW = 1024;  // rank x waves held in shared memory

// One event per thread, two passes over its amplitudes: the coherent sums of
// all ranks together (at most kPrepRanks, the ranks that the FdF kernels take),
// then the columns.  Bound by the columns' stores
// (16 bytes per slot and event plus 8 per wave); a pass per rank and purpose,
// one load in flight each, took 413 us for 87 waves, rank 2 and 250,001 events
// (0.88 GB), 214 now.
constexpr int kPrepRanks = 4;

// element of the tiled store (storeIndex; B is a power of two), the event's
// part of it computed once
struct EventRow {
	const float2* base;  // wave 0 of the event's block
	uint32_t p, B;
	__device__ __forceinline__ float2 operator[](int w) const
	{
		const uint32_t rot = (B / 32) * ((uint32_t)w & (512 / B - 1));
		return __ldg(base + (size_t)w * B + ((p + rot) & (B - 1)));
	}
};

__device__ __forceinline__ void coherentSums(const EventRow& amps, const float2* Vs, int W0, int W, int R, float2 (&S0)[kPrepRanks], float2 (&S1)[kPrepRanks])
{
#pragma unroll
	for (int r = 0; r < kPrepRanks; ++r)
		S0[r] = S1[r] = make_float2(0.f, 0.f);
	auto add = [&](int from, int to, float2(&S)[kPrepRanks]) {
#pragma unroll 8
		for (int w = from; w < to; ++w) {
			const float2 a = amps[w];
#pragma unroll
			for (int r = 0; r < kPrepRanks; ++r)
				if (r < R) {
					const float2 v = Vs[r * W + w];
					S[r].x = fmaf(v.x, a.x, fmaf(-v.y, a.y, S[r].x));
					S[r].y = fmaf(v.x, a.y, fmaf(v.y, a.x, S[r].y));
				}
		}
	};
	add(0, W0, S0);
	add(W0, W, S1);
}

__global__ void __launch_bounds__(256) hessPrepKernel(const float2* __restrict__ amps, uint64_t nEvents, uint32_t B,
                                                      uint64_t e0, uint64_t slab, int W0, int W, int R, int P,
                                                      const double* __restrict__ par, const int* __restrict__ slotRe,
                                                      const int* __restrict__ slotIm, float2* __restrict__ Y1,
                                                      float2* __restrict__ Y2, double* __restrict__ w1,
                                                      double* __restrict__ w2)
{
	__shared__ float2 Vs[kMaxRW];
	const int nS = R * W;
	for (int k = threadIdx.x; k < nS; k += blockDim.x) {
		const int ir = slotRe[k], ii = slotIm[k];
		Vs[k] = make_float2(ir >= 0 ? (float)par[ir] : 0.f, ii >= 0 ? (float)par[ii] : 0.f);
	}
	__syncthreads();
	const double flat = par[P - 1];
	const float flat2 = (float)(flat * flat);
	for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < slab; t += (uint64_t)gridDim.x * blockDim.x) {
		const uint64_t ev = e0 + t;
		const bool valid = ev < nEvents;
		const uint64_t col = valid ? ev : 0;
		const EventRow row{amps + (col & ~(uint64_t)(B - 1)) * W, (uint32_t)(col & (B - 1)), B};
		float2 S0[kPrepRanks], S1[kPrepRanks];
		// L and f
		float L = flat2;
		coherentSums(row, Vs, W0, W, R, S0, S1);
#pragma unroll
		for (int r = 0; r < kPrepRanks; ++r)
			if (r < R) {
				L = fmaf(S0[r].x, S0[r].x, fmaf(S0[r].y, S0[r].y, L));
				L = fmaf(S1[r].x, S1[r].x, fmaf(S1[r].y, S1[r].y, L));
			}
		const float f = valid ? 2.f / L : 0.f;
		w1[t] = valid ? (double)f * (double)f : 0.;
		w2[t] = valid ? (double)f : 0.;
		// d_s, conj(d_s) and the amplitudes
		auto columns = [&](int from, int to, const float2(&S)[kPrepRanks]) {
#pragma unroll 4
			for (int w = from; w < to; ++w) {
				const float2 a = row[w];
#pragma unroll
				for (int r = 0; r < kPrepRanks; ++r)
					if (r < R) {
						// S conj(a)
						const float2 d = make_float2(S[r].x * a.x + S[r].y * a.y, S[r].y * a.x - S[r].x * a.y);
						const size_t k = (size_t)(r * W + w);
						Y1[k * slab + t] = d;
						Y1[(nS + k) * slab + t] = make_float2(d.x, -d.y);
					}
				Y2[(size_t)w * slab + t] = a;
			}
		};
		columns(0, W0, S0);
		columns(W0, W, S1);
		Y1[(size_t)(2 * nS) * slab + t] = make_float2(1.f, 0.f);
		Y2[(size_t)W * slab + t] = make_float2(1.f, 0.f);
	}
}

}  // namespace

int launchHessPrep(const float2* amps, uint64_t nEvents, uint32_t B, uint64_t e0, uint64_t slab, int W0, int W,
                   int R, int P, const double* par, const int* slotRe, const int* slotIm, float2* Y1, float2* Y2,
                   double* w1, double* w2, cudaStream_t s)
{
	if (R < 1 || R > kPrepRanks || R * W > kMaxRW)
		return setError(kErrUnsupported, "Hessian kernel supports rank 1..4 and rank x waves <= 1024");
	const int threads = 256;
	const int blocks = (int)std::max<uint64_t>(1, std::min<uint64_t>((slab + threads - 1) / threads, 8192));
	hessPrepKernel<<<blocks, threads, 0, s>>>(amps, nEvents, B, e0, slab, W0, W, R, P, par, slotRe, slotIm, Y1, Y2,
	                                          w1, w2);
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "hessian prep launch");
}

}  // namespace pwa
