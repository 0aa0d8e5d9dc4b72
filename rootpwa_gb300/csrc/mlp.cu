// mlp.cu -- the warm-start network: a 3-layer perceptron
//   h1 = relu(W1 x + b1), h2 = relu(W2 h1 + b2), y = W3 h2 + b3
// with BF16 weights and activations, FP32 accumulation, FP32 master weights,
// its backward pass and an Adam update, all as hand-written kernels.
//
// One tensor-core GEMM kernel serves every product: C[M][N] = sum_k A(m, k)
// B(k, n) with A and B read through strides (so that X W^T, dY W and dY^T X
// are the same kernel).  Every BF16 matrix is stored with its rows padded
// with zeros to a multiple of eight elements, so that all operand loads are
// 16-byte vectors (the 5203-wide input rows would otherwise start at odd
// two-byte offsets).  128 x 128 output tiles; per K step of 64 the
// four loader warps read both operand tiles and write them in the canonical
// K-major 128-byte-swizzled layout (8 x 8 blocks transposed in registers where
// the other dimension is contiguous), one thread issues four tcgen05.mma
// kind::f16 (BF16 operands, M = N = 128, K = 16) into an FP32 accumulator in
// tensor memory (128 columns), two operand stages alternate.  The product is
// split into K slices, one block per (tile, slice), so that the grid covers
// the GPU (the batch has 256 rows, the layers 102 to 512 columns); the loader
// warps then move the accumulator to the slice's FP32 partials, and a second
// kernel sums the slices in slice order (deterministic) and applies the
// epilogue: bias, relu or a relu mask, FP32 and/or BF16 stores.
//
// What bounds it: latency (a block has one to three K steps) and, for the two
// products over the 5203 inputs, the slices' partials in L2.  256 rows of
// 5203-512-512-102, caches cold: the products took 22 us on average with
// single-element operand loads and one row per lane in the drain; vector
// loads alone left 12 to 15 us and, for the first layer and its weight
// gradient, 32 and 44; with rows stored whole, 7 and 13 and 16.  A training
// step takes 172 us against 352 before (Adam's 83 MB among them: 21 us).

#include "pwa_internal.h"
#include "tcgen05.cuh"

#include <cuda_bf16.h>

#include <algorithm>

namespace pwa {
namespace {

constexpr int kTcTile = 128;                       // output tile 128 x 128
constexpr int kTcK = 64;                           // K per stage: one 128-byte row of BF16
constexpr int kTcLoadWarps = 4;                    // loaders, then the drain (warp = lane quarter)
constexpr int kTcMmaWarp = kTcLoadWarps;           // warp 4
constexpr int kTcThreads = (kTcLoadWarps + 1) * 32;
constexpr int kTcStages = 2;
constexpr uint32_t kTcOpBytes = kTcTile * 128u;    // one operand tile: 128 rows x 64 BF16
constexpr uint32_t kTcCols = 128;                  // tensor-memory columns of the accumulator
constexpr size_t kTcSmem = 1024 + 2u * kTcStages * kTcOpBytes + 128;

// bias, relu, relu mask and the FP32 / BF16 stores of one output element
__device__ __forceinline__ void mlpEpilogue(const MlpGemm& g, int m, int n, float v)
{
	const size_t o = (size_t)m * g.N + n, o16 = (size_t)m * g.ld16 + n;
	if (g.bias)
		v += g.bias[n];
	if (g.relu)
		v = fmaxf(v, 0.f);
	const __nv_bfloat16* mask = reinterpret_cast<const __nv_bfloat16*>(g.mask);
	if (mask && !(__bfloat162float(mask[o16]) > 0.f))
		v = 0.f;
	if (g.C32)
		g.C32[o] = v;
	if (g.C16)
		reinterpret_cast<__nv_bfloat16*>(g.C16)[o16] = __float2bfloat16_rn(v);
}

// one 128 x 64 operand tile in the K-major swizzled layout: row r, k of
// element (r, k) = X[r * ldr + k * ldk] of rows r0.., k0.. (zero beyond nR
// rows or kEnd); one of ldr, ldk is 1, the other a multiple of 8, and X is
// 16-byte aligned with zeros after the last element of a padded row.  128
// loader threads, eight 16-byte loads each.
__device__ __forceinline__ void loadTile(unsigned char* dst, const uint16_t* X, size_t ldr, size_t ldk, int contigK,
                                         int r0, int nR, int k0, int kEnd, int t)
{
	const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
	if (contigK) {
		// thread t: chunks t, t + 128, ...: row c / 8, k-chunk c % 8.  kEnd is a
		// multiple of 8 or the end of the padded rows
		uint4 v[8];
#pragma unroll
		for (int j = 0; j < 8; ++j) {
			const int c = t + 128 * j, r = c >> 3, kc = (c & 7) * 8;
			v[j] = (r0 + r < nR && k0 + kc < kEnd)
			           ? __ldg(reinterpret_cast<const uint4*>(X + (size_t)(r0 + r) * ldr + k0 + kc))
			           : zero;
		}
#pragma unroll
		for (int j = 0; j < 8; ++j) {
			const int c = t + 128 * j, r = c >> 3, kc = (c & 7) * 8;
			*reinterpret_cast<uint4*>(dst + swzOffset16(r, kc)) = v[j];
		}
	} else {
		// thread t: the 8 x 8 block of rows 8 (t / 8) .. and k 8 (t % 8) ..:
		// one load per k, then each row's eight k together
		const int rb = (t >> 3) * 8, kb = (t & 7) * 8;
		uint32_t v[8][4];
#pragma unroll
		for (int i = 0; i < 8; ++i) {
			const uint4 q = (r0 + rb < nR && k0 + kb + i < kEnd)
			                    ? __ldg(reinterpret_cast<const uint4*>(X + (size_t)(k0 + kb + i) * ldk + r0 + rb))
			                    : zero;
			v[i][0] = q.x;
			v[i][1] = q.y;
			v[i][2] = q.z;
			v[i][3] = q.w;
		}
#pragma unroll
		for (int r = 0; r < 8; ++r) {
			uint32_t w[4];
#pragma unroll
			for (int i = 0; i < 4; ++i)
				w[i] = __byte_perm(v[2 * i][r >> 1], v[2 * i + 1][r >> 1], (r & 1) ? 0x7632 : 0x5410);
			*reinterpret_cast<uint4*>(dst + swzOffset16(rb + r, kb)) = make_uint4(w[0], w[1], w[2], w[3]);
		}
	}
}

// C tile (blockIdx.y, blockIdx.x) over K slice blockIdx.z -> g.work[z][M][N]
__global__ void __launch_bounds__(kTcThreads) mlpGemmTcKernel(const MlpGemm g, int kPerSlice)
{
	extern __shared__ __align__(1024) unsigned char smemRaw[];
	unsigned char* smem =
	    reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
	unsigned char* opA = smem;                                 // [stages][128 x 128 B]
	unsigned char* opB = smem + kTcStages * kTcOpBytes;        // [stages][128 x 128 B]
	uint64_t* full = reinterpret_cast<uint64_t*>(opB + kTcStages * kTcOpBytes);
	uint64_t* empty = full + kTcStages;
	uint64_t* done = empty + kTcStages;
	uint32_t* tmemHolder = reinterpret_cast<uint32_t*>(done + 1);
	__shared__ unsigned sFail;

	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int m0 = blockIdx.y * kTcTile, n0 = blockIdx.x * kTcTile;
	const int kBeg = (int)blockIdx.z * kPerSlice, kEnd = min(g.K, kBeg + kPerSlice);
	const int nSteps = kEnd > kBeg ? (kEnd - kBeg + kTcK - 1) / kTcK : 0;
	const uint16_t* A = g.A;
	const uint16_t* B = g.B;

	if (tid == 0) {
		for (int s = 0; s < kTcStages; ++s) {
			barInit(&full[s], kTcLoadWarps);
			barInit(&empty[s], 1);
		}
		barInit(done, 1);
		sFail = 0u;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == kTcMmaWarp) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sAddr(tmemHolder)),
		             "r"(kTcCols)
		             : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	const uint32_t tmem = *tmemHolder;

	if (warp < kTcLoadWarps) {
		// ---- loaders: both operand tiles of every K step ----
		bool ok = true;
		for (int t = 0; t < nSteps; ++t) {
			const int s = t % kTcStages;
			if (t >= kTcStages && !barWait(&empty[s], (uint32_t)(((t / kTcStages) - 1) & 1))) {
				atomicOr(g.devErr, (unsigned)kDevErrTimeout);
				sFail = 1u;
				ok = false;
				break;
			}
			const int k0 = kBeg + t * kTcK;
			// A(m, k) = A[m lda_m + k lda_k]; B(k, n) = B[k ldb_k + n ldb_n] as rows n
			loadTile(opA + s * kTcOpBytes, A, g.lda_m, g.lda_k, g.aContigK, m0, g.M, k0, kEnd, tid);
			loadTile(opB + s * kTcOpBytes, B, g.ldb_n, g.ldb_k, g.bContigK, n0, g.N, k0, kEnd, tid);
			asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
			__syncwarp();
			if (lane == 0)
				barArrive(&full[s]);
		}
		// ---- drain: the accumulator rows of this warp's lane quarter ----
		if (ok && nSteps > 0 && !barWait(done, 0u)) {
			atomicOr(g.devErr, (unsigned)kDevErrTimeout);
			ok = false;
		}
		if (ok) {
			asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
			// through shared memory (the operand stages are done with), so that
			// a row's 128 columns are stored together: one lane per row would
			// write every 32-byte sector eight times.  16-byte piece q of row r
			// at q ^ r: conflict-free both ways.
			float4* const rows = reinterpret_cast<float4*>(opA) + warp * 32 * 32;
#pragma unroll 2
			for (int c = 0; c < kTcTile; c += 16) {
				uint32_t r[16];
				if (nSteps > 0) {
					tmemLd16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, r);
					asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
				} else {
#pragma unroll
					for (int i = 0; i < 16; ++i)
						r[i] = 0u;
				}
#pragma unroll
				for (int i = 0; i < 4; ++i)
					rows[lane * 32 + ((c / 4 + i) ^ lane)] =
					    make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]),
					                __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
			}
			__syncwarp();
			const int ldw = mlpWorkLd(g.N), n = n0 + 4 * lane, mw = m0 + warp * 32;
			float* out = g.work + ((size_t)blockIdx.z * g.M + mw) * ldw + n;
			if (n < ldw)
#pragma unroll 8
				for (int r = 0; r < 32; ++r)
					if (mw + r < g.M)
						*reinterpret_cast<float4*>(out + (size_t)r * ldw) = rows[r * 32 + (lane ^ r)];
		}
	} else if (lane == 0) {
		// ---- MMA issuer ----
		const uint32_t idesc = idescBf16(kTcTile, kTcTile);
		int t = 0;
		for (; t < nSteps; ++t) {
			const int s = t % kTcStages;
			if (!barWait(&full[s], (uint32_t)((t / kTcStages) & 1))) {
				atomicOr(g.devErr, (unsigned)kDevErrTimeout);
				sFail = 1u;
				break;
			}
			asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
			const uint64_t aD = smemDesc(sAddr(opA + s * kTcOpBytes)), bD = smemDesc(sAddr(opB + s * kTcOpBytes));
#pragma unroll
			for (uint32_t kk = 0; kk < 4; ++kk)
				mmaBf16(tmem, aD + 2 * kk, bD + 2 * kk, idesc, (t > 0 || kk > 0) ? 1u : 0u);
			mmaCommit(&empty[s]);
		}
		// all MMAs of this block complete before the drain reads tensor memory
		mmaCommit(done);
		if (t < nSteps || nSteps == 0)
			barWait(done, 0u);
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	if (warp == kTcMmaWarp) {
		asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcCols) : "memory");
	}
}

// sum of the K slices' partials in slice order, then the epilogue: four
// columns per thread
__global__ void __launch_bounds__(128) mlpSplitReduceKernel(const MlpGemm g)
{
	const int ldw = mlpWorkLd(g.N), n = 4 * (blockIdx.x * 128 + threadIdx.x);
	if (n >= g.N)
		return;
	const size_t slice = (size_t)g.M * ldw;
	for (int m = blockIdx.y; m < g.M; m += gridDim.y) {
		const float4* p = reinterpret_cast<const float4*>(g.work + (size_t)m * ldw + n);
		float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
		for (int z = 0; z < g.splitK; ++z) {
			const float4 q = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p) + z * slice));
			v[0] += q.x;
			v[1] += q.y;
			v[2] += q.z;
			v[3] += q.w;
		}
#pragma unroll
		for (int i = 0; i < 4; ++i)
			if (n + i < g.N)
				mlpEpilogue(g, m, n + i, v[i]);
	}
}

// column sums of an FP32 [M][N] matrix (bias gradients), rows in order: the
// block brings 256 rows of 32 columns to shared memory at a time, one warp adds
// them (with that warp's own loads, 64 rows in flight, 256 rows took 8 us).
constexpr int kColRows = 256;
__global__ void __launch_bounds__(256) colSumKernel(const float* __restrict__ X, int M, int N, float* out)
{
	__shared__ float tile[kColRows][32];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = blockIdx.x * 32 + lane;
	float s = 0.f;
	for (int m0 = 0; m0 < M; m0 += kColRows) {
		const int rows = min(kColRows, M - m0);
		float v[kColRows / 8];
#pragma unroll
		for (int i = 0; i < kColRows / 8; ++i)
			v[i] = n < N && warp + 8 * i < rows ? __ldg(X + (size_t)(m0 + warp + 8 * i) * N + n) : 0.f;
#pragma unroll
		for (int i = 0; i < kColRows / 8; ++i)
			tile[warp + 8 * i][lane] = v[i];
		__syncthreads();
		if (warp == 0) {
#pragma unroll 32
			for (int i = 0; i < rows; ++i)
				s += tile[i][lane];
		}
		__syncthreads();
	}
	if (warp == 0 && n < N)
		out[n] = s;
}

// squared error sum over n values (FP64 total, times `scale`) and
// dY = 2 (Y - T) scale (BF16 copy in rows of ld16)
__global__ void mseKernel(const float* Y, const float* T, int n, int N, int ld16, float scale, float* dY32, uint16_t* dY16,
                          double* loss)
{
	double part = 0.;
	__nv_bfloat16* d16 = reinterpret_cast<__nv_bfloat16*>(dY16);
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
		const float d = Y[i] - T[i];
		part += (double)d * d;
		const float gval = 2.f * d * scale;
		dY32[i] = gval;
		d16[(size_t)(i / N) * ld16 + i % N] = __float2bfloat16_rn(gval);
	}
	for (int o = 16; o > 0; o >>= 1)
		part += __shfl_xor_sync(0xffffffffu, part, o);
	if ((threadIdx.x & 31) == 0)
		atomicAdd(loss, part * (double)scale);
}

// element i of the parameter vector in the padded BF16 weights, or -1 (bias)
__device__ __forceinline__ long long w16Index(const MlpWeights& w, size_t i)
{
	long long o = -1;
#pragma unroll
	for (int l = 0; l < 3; ++l) {
		const size_t q = i - w.from[l];  // wraps below the matrix
		if (q < (size_t)w.rows[l] * w.cols[l]) {
			const size_t r = q <= 0xffffffffull ? (size_t)((uint32_t)q / (uint32_t)w.cols[l]) : q / w.cols[l];
			o = (long long)(w.to[l] + r * w.ld[l] + (q - r * w.cols[l]));
		}
	}
	return o;
}

// Adam on FP32 master weights; refreshes the BF16 copy.  Four parameters per
// thread (the arrays come from the allocator, 16-byte aligned; every index into
// the thread's own copies is known at compile time, so that they and the
// weights' map stay in registers: 21 us for 3 M parameters, 24 with the map
// indexed in local memory).  The moments'
// fused multiply-adds are written out: a run's weights do not depend on which
// product the compiler fuses.
__global__ void __launch_bounds__(256) adamKernel(float* w, const float* __restrict__ g, float* m, float* v,
                                                  uint16_t* w16, size_t n, float lr, float b1, float b2, float eps,
                                                  float c1, float c2, const MlpWeights map)
{
	__nv_bfloat16* o16 = reinterpret_cast<__nv_bfloat16*>(w16);
	const size_t i0 = 4 * (blockIdx.x * (size_t)256 + threadIdx.x);
	if (i0 >= n)
		return;
	const int k = (int)min((size_t)4, n - i0);
	alignas(16) float gi[4], mi[4], vi[4], wi[4];
	if (k == 4) {
		*reinterpret_cast<float4*>(gi) = *reinterpret_cast<const float4*>(g + i0);
		*reinterpret_cast<float4*>(mi) = *reinterpret_cast<const float4*>(m + i0);
		*reinterpret_cast<float4*>(vi) = *reinterpret_cast<const float4*>(v + i0);
		*reinterpret_cast<float4*>(wi) = *reinterpret_cast<const float4*>(w + i0);
	} else {
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			const size_t i = j < k ? i0 + j : i0;
			gi[j] = g[i];
			mi[j] = m[i];
			vi[j] = v[i];
			wi[j] = w[i];
		}
	}
#pragma unroll
	for (int j = 0; j < 4; ++j) {
		mi[j] = __fmaf_rn(1.f - b1, gi[j], __fmul_rn(b1, mi[j]));
		vi[j] = __fmaf_rn(__fmul_rn(1.f - b2, gi[j]), gi[j], __fmul_rn(b2, vi[j]));
		wi[j] = wi[j] - lr * (mi[j] / c1) / (sqrtf(vi[j] / c2) + eps);
	}
	if (k == 4) {
		*reinterpret_cast<float4*>(m + i0) = *reinterpret_cast<float4*>(mi);
		*reinterpret_cast<float4*>(v + i0) = *reinterpret_cast<float4*>(vi);
		*reinterpret_cast<float4*>(w + i0) = *reinterpret_cast<float4*>(wi);
	} else {
#pragma unroll
		for (int j = 0; j < 4; ++j)
			if (j < k) {
				m[i0 + j] = mi[j];
				v[i0 + j] = vi[j];
				w[i0 + j] = wi[j];
			}
	}
#pragma unroll
	for (int j = 0; j < 4; ++j) {
		const long long o = j < k ? w16Index(map, i0 + j) : -1;
		if (o >= 0)
			o16[o] = __float2bfloat16_rn(wi[j]);
	}
}

__global__ void weights16Kernel(const float* w, uint16_t* w16, size_t n, const MlpWeights map)
{
	__nv_bfloat16* o16 = reinterpret_cast<__nv_bfloat16*>(w16);
	for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
		const long long o = w16Index(map, i);
		if (o >= 0)
			o16[o] = __float2bfloat16_rn(w[i]);
	}
}

// rows of `cols` FP32 values into BF16 rows of ld >= cols (zeros after them)
__global__ void toBf16Kernel(const float* x, uint16_t* y, size_t rows, int cols, int ld)
{
	__nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(y);
	for (size_t r = blockIdx.y; r < rows; r += gridDim.y)
		for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ld; c += gridDim.x * blockDim.x)
			o[r * ld + c] = __float2bfloat16_rn(c < cols ? x[r * cols + c] : 0.f);
}

// rows idx[r] of src -> dst [r] in units of U (16 or 4 bytes)
template <typename U>
__global__ void gatherRowsKernel(const U* __restrict__ src, const uint32_t* idx, int rows, int units, U* dst)
{
	for (int r = blockIdx.x; r < rows; r += gridDim.x) {
		const U* s = src + (size_t)idx[r] * units;
		for (int i = threadIdx.x; i < units; i += blockDim.x)
			dst[(size_t)r * units + i] = s[i];
	}
}

}  // namespace

int mlpGemmSplit(const MlpGemm& g, int numSMs)
{
	// K slices of whole K steps, so that the blocks cover the SMs about twice
	const int tiles = ((g.N + kTcTile - 1) / kTcTile) * ((g.M + kTcTile - 1) / kTcTile);
	const int steps = (g.K + kTcK - 1) / kTcK;
	return std::max(1, std::min(steps, (2 * numSMs + tiles - 1) / tiles));
}

int launchMlpGemm(const MlpGemm& g, cudaStream_t s)
{
	if (g.M <= 0 || g.N <= 0 || g.K <= 0)
		return setError(kErrArg, "MLP GEMM: empty shape");
	if (!g.work || g.splitK < 1 || !g.devErr)
		return setError(kErrArg, "MLP GEMM: workspace, K slices and error flag required");
	const int steps = (g.K + kTcK - 1) / kTcK;
	const int kPerSlice = ((steps + g.splitK - 1) / g.splitK) * kTcK;
	const int slices = (g.K + kPerSlice - 1) / kPerSlice;
	static bool configured = false;
	if (!configured) {
		PWA_CHECK(cudaCheck(cudaFuncSetAttribute(mlpGemmTcKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                                         (int)kTcSmem),
		                    "MLP GEMM smem attribute"));
		configured = true;
	}
	dim3 grid((g.N + kTcTile - 1) / kTcTile, (g.M + kTcTile - 1) / kTcTile, slices);
	mlpGemmTcKernel<<<grid, kTcThreads, kTcSmem, s>>>(g, kPerSlice);
	countLaunches(1);
	PWA_CHECK(cudaCheck(cudaGetLastError(), "MLP GEMM launch"));
	MlpGemm r = g;
	r.splitK = slices;
	const dim3 rgrid((g.N + 511) / 512, std::min(g.M, 65535));
	mlpSplitReduceKernel<<<rgrid, 128, 0, s>>>(r);
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "MLP split-K reduce launch");
}

int launchColSum(const float* X, int M, int N, float* out, cudaStream_t s)
{
	colSumKernel<<<(N + 31) / 32, 256, 0, s>>>(X, M, N, out);
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "column sum launch");
}

int launchMse(const float* Y, const float* T, int n, int N, int ld16, float scale, float* dY32, uint16_t* dY16,
              double* loss, cudaStream_t s)
{
	const int blocks = std::min(1024, std::max(1, (n + 255) / 256));
	mseKernel<<<blocks, 256, 0, s>>>(Y, T, n, N, ld16, scale, dY32, dY16, loss);
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "MSE launch");
}

int launchAdam(float* w, const float* g, float* m, float* v, uint16_t* w16, size_t n, float lr, float b1, float b2,
               float eps, float c1, float c2, const MlpWeights& map, cudaStream_t s)
{
	const unsigned blocks = (unsigned)std::max<size_t>(1, (n + 1023) / 1024);
	adamKernel<<<blocks, 256, 0, s>>>(w, g, m, v, w16, n, lr, b1, b2, eps, c1, c2, map);
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "Adam launch");
}

int launchWeights16(const float* w, uint16_t* w16, size_t n, const MlpWeights& map, cudaStream_t s)
{
	const int blocks = (int)std::min<size_t>(4096, std::max<size_t>(1, (n + 255) / 256));
	weights16Kernel<<<blocks, 256, 0, s>>>(w, w16, n, map);
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "bf16 weights launch");
}

int launchToBf16(const float* x, uint16_t* y, size_t rows, int cols, int ld, cudaStream_t s)
{
	const dim3 grid((unsigned)((ld + 255) / 256), (unsigned)std::min<size_t>(rows, 4096));
	toBf16Kernel<<<grid, 256, 0, s>>>(x, y, rows, cols, ld);
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "bf16 conversion launch");
}

int launchGatherRows(const void* src, const uint32_t* idx, int rows, size_t rowBytes, void* dst, cudaStream_t s)
{
	// rows of whole 16-byte units, or of FP32 values
	const int blocks = std::min(4096, std::max(1, rows));
	if (rowBytes % 16 == 0)
		gatherRowsKernel<<<blocks, 256, 0, s>>>(static_cast<const uint4*>(src), idx, rows, (int)(rowBytes / 16),
		                                        static_cast<uint4*>(dst));
	else
		gatherRowsKernel<<<blocks, 256, 0, s>>>(static_cast<const uint32_t*>(src), idx, rows, (int)(rowBytes / 4),
		                                        static_cast<uint32_t*>(dst));
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "row gather launch");
}

}  // namespace pwa
