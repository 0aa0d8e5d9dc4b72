// isobar.cu -- GPU evaluation of the three-body isobar decay amplitudes
// (isobarHelicityAmplitude::amplitude, decayAmplitude/isobarAmplitude.cc:98-262,
// isobarHelicityAmplitude.cc:64-195): one amplitude per wave and event,
// row-major [wave][event], complex128 with FP64 arithmetic throughout, or
// complex64 with the frames and kinematics in FP64 and the per-wave
// arithmetic in FP32 (GB300 runs FP32 at 64 times its FP64 rate; the
// likelihood's amplitude store is complex64).
//
// A thread takes one symmetrisation term (instance) of one event: the
// lanes of an event sit side by side, 2^n of them, and add their terms by
// shuffles.  The Gottfried-Jackson frame is built once per event by the first
// threads of the block.  Each thread then fills its column of a table in
// shared memory -- the factors that the waves share -- and runs the plan's
// program over it (isobar_math.cuh); the plan is the same for all threads and
// is read through the read-only cache.
//
// What bounds it: in complex128 the FP64 pipe (2 lanes per clock and SM; 76 %
// busy at 40,001 events x 88 waves), in complex64 the latency of 16 warps per
// SM, which the tables' shared memory allows, with the FP64 pipe 43 % busy
// for the frames and the pi pi S-wave.  One thread per event that evaluated
// every wave's D functions took 4.42 ms (complex128, 40,001 events) and
// 2.05 ms (complex64, 300,000 events) where this takes 1.15 and 1.47 ms.
#include "isobar_math.cuh"
#include "pwa_internal.h"

#include <algorithm>

namespace pwa {

namespace {

// Threads per SM that the registers are limited for: FP32 tables of a 3pi
// wave set are 0.3 KB per thread, FP64 ones twice that.  The tables decide how
// many fit, so that the limit matters little: complex64, 300,000 events x 88
// waves 1.54 ms at 512, 1.56 at 640 and 768, 1.59 at 1,024; complex128, 40,001
// events 1.26 at 256 and 512, 1.25 at 384 and 640.
constexpr int kThreadsPerSM32 = 640, kThreadsPerSM64 = 384;

template <typename T, int B>
__global__ void __launch_bounds__(B, (sizeof(T) == 4 ? kThreadsPerSM32 : kThreadsPerSM64) / B)
    isobarAmplitudeKernel(const iso::PlanView P, const double* __restrict__ beam, const double* __restrict__ fs,
                          uint64_t n, T* __restrict__ amps, int log2Inst)
{
	extern __shared__ __align__(16) unsigned char smem[];
	const int tid = threadIdx.x, perTile = B >> log2Inst;
	double* const frames = reinterpret_cast<double*>(smem);  // [12][perTile]
	T* const table = reinterpret_cast<T*>(frames + 12 * perTile);
	const int inst = tid & ((1 << log2Inst) - 1), ev = tid >> log2Inst;
	const iso::Table<T> tab{table + 2 * tid, B};
	// the frame of event e with its particles permuted
	auto frame = [&](uint64_t e, const int32_t* perm, iso::LV (&g)[3]) {
		double bp[3], fp[3][3];
		for (int k = 0; k < 3; ++k)
			bp[k] = __ldg(beam + k * n + e);
		for (int i = 0; i < 3; ++i)
			for (int k = 0; k < 3; ++k)
				fp[i][k] = __ldg(fs + (uint64_t)(3 * perm[i] + k) * n + e);
		iso::gjFrame(P, bp, fp, g);
	};
	for (uint64_t e0 = (uint64_t)blockIdx.x * perTile; e0 < n; e0 += (uint64_t)gridDim.x * perTile) {
		__syncthreads();
		if (tid < perTile) {
			iso::LV g[3];
			frame(min(e0 + tid, n - 1), P.perms, g);
			for (int i = 0; i < 3; ++i) {
				frames[(4 * i) * perTile + tid] = g[i].p.x;
				frames[(4 * i + 1) * perTile + tid] = g[i].p.y;
				frames[(4 * i + 2) * perTile + tid] = g[i].p.z;
				frames[(4 * i + 3) * perTile + tid] = g[i].e;
			}
		}
		__syncthreads();
		const uint64_t e = e0 + ev;
		const bool inside = e < n;
		for (uint32_t b = 0; b < P.nBatches; ++b) {
			const iso::Batch& Bt = P.batches[b];
			const bool used = inst < Bt.nInst;
			const int32_t* perm = P.perms + (used ? 3 * P.insts[Bt.inst0 + inst] : 0);
			const int slots[3] = {Bt.a, Bt.b, Bt.c};
			iso::LV v[3];  // isobar daughters and bachelor
			if (iso::permutesEqualMasses(P, perm)) {
				for (int i = 0; i < 3; ++i) {
					const double* f = frames + 4 * perm[slots[i]] * perTile + ev;
					v[i] = iso::LV{iso::V3{f[0], f[perTile], f[2 * perTile]}, f[3 * perTile]};
				}
			} else {
				iso::LV g[3];
				frame(min(e, n - 1), perm, g);
				for (int i = 0; i < 3; ++i)
					v[i] = slots[i] == 0 ? g[0] : slots[i] == 1 ? g[1] : g[2];
			}
			T c2, s2;
			{
				const iso::Kin<T> k = iso::kinematics<T>(v[0], v[1], v[2], Bt.bachelorFirst != 0, P.canonical != 0);
				iso::fillTable<T>(P, Bt, k, tab);
				c2 = k.c2X;
				s2 = k.s2X;
			}
			T f = T(0);
			int row = -1;
			iso::batchWaves<T>(P, Bt, tab, c2, s2, [&](const iso::WaveOp& W, iso::C2T<T> v) {
				if (W.factor0 != row) {
					row = W.factor0;
					f = used ? iso::pick<T>(P.factors[row + inst], P.factorsF[row + inst]) : T(0);
				}
				T re = f == T(0) ? T(0) : f * v.re, im = f == T(0) ? T(0) : f * v.im;
				T* out = amps + 2 * ((uint64_t)W.wave * n + e);
				if (log2Inst == 0) {
					if (inside) {
						out[0] = re;
						out[1] = im;
					}
					return;
				}
				// the first two lanes of an event store a component each:
				// 128 consecutive bytes per warp with two lanes per event
				const T give = (inst & 1) ? re : im;
				T sum = ((inst & 1) ? im : re) + __shfl_xor_sync(0xffffffffu, give, 1);
				for (int o = 2; o < (1 << log2Inst); o <<= 1)
					sum += __shfl_xor_sync(0xffffffffu, sum, o);
				if (inside && inst < 2)
					out[inst] = sum;
			});
		}
	}
}

template <typename T, int B>
int launchIsobarT(const iso::PlanView& v, const double* beam, const double* fs, uint64_t n, T* amps, int log2Inst,
                  int sms, size_t smem, cudaStream_t s)
{
	auto kern = isobarAmplitudeKernel<T, B>;
	if (smem > 48 * 1024)
		PWA_CHECK(cudaCheck(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
		                    "cudaFuncSetAttribute(isobar)"));
	int perSM = 1;
	PWA_CHECK(cudaCheck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, kern, B, smem), "isobar occupancy"));
	const uint64_t perTile = B >> log2Inst;
	const unsigned blocks = (unsigned)std::min<uint64_t>((n + perTile - 1) / perTile, (uint64_t)sms * std::max(1, perSM));
	kern<<<blocks, B, smem, s>>>(v, beam, fs, n, amps, log2Inst);
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "isobar amplitude kernel");
}

template <typename T>
int launchIsobar(const iso::PlanView& v, const double* beam, const double* fs, uint64_t n, T* amps, int sms,
                 cudaStream_t s)
{
	int log2Inst = 0;
	while ((1 << log2Inst) < v.maxInst)
		++log2Inst;
	auto bytes = [&](int B) { return (size_t)12 * (B >> log2Inst) * sizeof(double) + (size_t)((v.tableSize + 1) & ~1) * B * sizeof(T); };
	// 128 threads where at least two blocks' tables fit on an SM; fewer for
	// plans with many factors, and for inputs that would leave SMs idle
	constexpr size_t kTwo = 112 * 1024;
	if (bytes(128) <= kTwo && (n << log2Inst) >= (uint64_t)sms * 128)
		return launchIsobarT<T, 128>(v, beam, fs, n, amps, log2Inst, sms, bytes(128), s);
	if (bytes(64) <= kTwo && (n << log2Inst) >= (uint64_t)sms * 64)
		return launchIsobarT<T, 64>(v, beam, fs, n, amps, log2Inst, sms, bytes(64), s);
	return launchIsobarT<T, 32>(v, beam, fs, n, amps, log2Inst, sms, bytes(32), s);
}

}  // namespace

int launchIsobarAmplitudes(const iso::PlanView& v, const double* beam, const double* fs, uint64_t n, void* amps,
                           bool fp32, cudaStream_t s)
{
	if (n == 0 || v.nWaves == 0)
		return kOk;
	int dev = 0, sms = 0;
	PWA_CHECK(cudaCheck(cudaGetDevice(&dev), "cudaGetDevice"));
	PWA_CHECK(cudaCheck(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count"));
	if (fp32)
		return launchIsobar<float>(v, beam, fs, n, static_cast<float*>(amps), sms, s);
	return launchIsobar<double>(v, beam, fs, n, static_cast<double*>(amps), sms, s);
}

}  // namespace pwa
