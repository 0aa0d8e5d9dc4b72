// integral_kernels.cu -- SIMT Gram kernels for the MC integral matrices.
//
// Computes the raw sums of ampIntegralMatrix::integrate
// (decayAmplitude/ampIntegralMatrix.cc:408-469)
//   I_ij = sum_k w_k A_{i,k} conj(A_{j,k})
// over K = events x sub-amplitudes.  gramTriKernel forms the upper triangle
// in 4 x 4 thread tiles (FP32 or FP64 products and sums) for one contiguous
// chunk of K per thread group; chunk partials are summed in FP64 by a second
// kernel, which also mirrors the upper triangle into the lower one (the
// reference's matrix is exactly Hermitian, since a conj(b) and b conj(a) round
// identically).  Wave sets too wide for its shared memory take gramSimtKernel
// (64 x 64 output tiles).
// The tensor-core variant lives in gram_tc.cu.

#include "pwa_internal.h"
#include "device_common.cuh"

#include <algorithm>

namespace pwa {
namespace {

constexpr int kTile = 64;
constexpr int kKT = 16;

template <typename In>
struct InTraits;
template <>
struct InTraits<float2> {
	__device__ static double2 load(const float2* p, uint64_t i)
	{
		const float2 v = p[i];
		return make_double2(v.x, v.y);
	}
};
template <>
struct InTraits<double2> {
	__device__ static double2 load(const double2* p, uint64_t i) { return p[i]; }
};

template <typename T>
struct Cplx {
	T x, y;
};

template <typename In, typename Acc>
__global__ void __launch_bounds__(256) gramSimtKernel(const In* __restrict__ amps, uint64_t K, uint64_t ldK, int W,
                                                      const double* __restrict__ weightK, double* partials,
                                                      int tilesPerSide, uint64_t chunkLen)
{
	__shared__ Cplx<Acc> sa[kKT][kTile + 1];
	__shared__ Cplx<Acc> sb[kKT][kTile + 1];
	// decode upper-triangle tile index (ti <= tj)
	int t = blockIdx.x, ti = 0;
	while (t >= tilesPerSide - ti) {
		t -= tilesPerSide - ti;
		++ti;
	}
	const int tj = ti + t;
	const int chunk = blockIdx.y;
	const uint64_t k0 = (uint64_t)chunk * chunkLen;
	const uint64_t k1 = min(K, k0 + chunkLen);
	const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
	const int i0 = ti * kTile, j0 = tj * kTile;

	Cplx<Acc> acc[4][4];
#pragma unroll
	for (int a = 0; a < 4; ++a)
#pragma unroll
		for (int b = 0; b < 4; ++b)
			acc[a][b] = Cplx<Acc>{Acc(0), Acc(0)};

	for (uint64_t kb = k0; kb < k1; kb += kKT) {
		// load 64 rows x 16 K of both operands; thread -> (row, k) pairs
		for (int idx = threadIdx.x; idx < kTile * kKT; idx += 256) {
			const int row = idx / kKT, kk = idx - row * kKT;
			const uint64_t k = kb + kk;
			Cplx<Acc> va{Acc(0), Acc(0)}, vb{Acc(0), Acc(0)};
			if (k < k1) {
				const int gi = i0 + row, gj = j0 + row;
				const Acc w = weightK ? (Acc)weightK[k] : Acc(1);
				if (gi < W) {
					const double2 v = InTraits<In>::load(amps, (uint64_t)gi * ldK + k);
					va = Cplx<Acc>{(Acc)v.x * w, (Acc)v.y * w};
				}
				if (gj < W) {
					const double2 v = InTraits<In>::load(amps, (uint64_t)gj * ldK + k);
					vb = Cplx<Acc>{(Acc)v.x, (Acc)v.y};
				}
			}
			sa[kk][row] = va;
			sb[kk][row] = vb;
		}
		__syncthreads();
#pragma unroll
		for (int kk = 0; kk < kKT; ++kk) {
			Cplx<Acc> a[4], b[4];
#pragma unroll
			for (int q = 0; q < 4; ++q) {
				a[q] = sa[kk][ty + 16 * q];
				b[q] = sb[kk][tx + 16 * q];
			}
#pragma unroll
			for (int p = 0; p < 4; ++p)
#pragma unroll
				for (int q = 0; q < 4; ++q) {
					// a conj(b)
					acc[p][q].x = fma(a[p].x, b[q].x, fma(a[p].y, b[q].y, acc[p][q].x));
					acc[p][q].y = fma(a[p].y, b[q].x, fma(-a[p].x, b[q].y, acc[p][q].y));
				}
		}
		__syncthreads();
	}
	double* out = partials + (size_t)chunk * W * W * 2;
#pragma unroll
	for (int p = 0; p < 4; ++p)
#pragma unroll
		for (int q = 0; q < 4; ++q) {
			const int gi = i0 + ty + 16 * p, gj = j0 + tx + 16 * q;
			if (gi < W && gj < W && gi <= gj) {
				out[((size_t)gi * W + gj) * 2] = (double)acc[p][q].x;
				out[((size_t)gi * W + gj) * 2 + 1] = (double)acc[p][q].y;
			}
		}
}

// ---------------------------------------------------------------------------
// Triangle kernel
// ---------------------------------------------------------------------------
// The W rows form g = ceil(W / 4) groups of four, and the pairs of groups
// (I, J >= I) are the thread tiles: 253 at 87 waves, 4048 complex products
// for the 3828 of the triangle, where 64 x 64 tiles form 12288 (a block of
// 256 threads then holds the whole matrix and reads each amplitude once).
// Small wave sets put several chunks of K side by side in one block.
//
// What bounds it: the arithmetic pipes.  GB300 issues 2 FP64 FMAs per clock
// and SM against 128 FP32 ones: in FP64 the triangle of 87 waves needs 3.7 ms
// per 150,000 events, whatever the loads do.
constexpr int kTriThreads = 256;

// Staged operands of one step, and the loads of a thread tile (rows of group
// I, columns of group J).  AccF32 keeps rows 2h, 2h + 1 of a group side by side
// (one 16-byte load brings both) and the groups' halves apart, AccF64 the four
// rows apart: the lanes of a warp, whose J are consecutive, read consecutive
// 16-byte pieces.
__device__ __forceinline__ float4 ldOp(const float2* p) { return *reinterpret_cast<const float4*>(p); }

// 8 bytes from global to shared memory in the background, or zeros
__device__ __forceinline__ void copyAsync8(void* dst, const void* src, bool valid)
{
	asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smemAddr(dst)), "l"(src), "r"(valid ? 8 : 0) : "memory");
}

// one staged row of a slice: element offset of its first amplitude, steps of
// K it has, position of its first operand (24 bits) and slice
struct __align__(16) TriSlot {
	uint64_t off;
	uint32_t lim, base;
};

// Accumulators of a thread tile.  AccF32 keeps gramSimtKernel's order of the
// four FMAs of a complex product (the imaginary parts' products first), so
// FP32 sums over the same chunks are the same bits.
struct AccF32 {
	typedef float2 Op;
	typedef float Weight;
	static constexpr int kUnroll = 2, kFold = 0;
	static constexpr bool kAsync = true;
	float2 s[4][4];
	__device__ void init()
	{
		for (int p = 0; p < 4; ++p)
			for (int q = 0; q < 4; ++q)
				s[p][q] = make_float2(0.f, 0.f);
	}
	static __device__ __forceinline__ int pos(int G, int row) { return ((((row >> 1) & 1) * G + (row >> 2)) << 1) | (row & 1); }
	template <bool WT>
	__device__ void step(const float2* A, const float2* B, int G, int I, int J, float w)
	{
		float2 a[4], b[4];
#pragma unroll
		for (int h = 0; h < 2; ++h) {
			const float4 x = ldOp(A + 2 * (h * G + I)), y = ldOp(B + 2 * (h * G + J));
			a[2 * h] = make_float2(x.x, x.y);
			a[2 * h + 1] = make_float2(x.z, x.w);
			b[2 * h] = make_float2(y.x, y.y);
			b[2 * h + 1] = make_float2(y.z, y.w);
		}
#pragma unroll
		for (int p = 0; p < 4; ++p) {
			if (WT)
				a[p] = make_float2(a[p].x * w, a[p].y * w);
			const float2 ar = make_float2(a[p].y, -a[p].x);
#pragma unroll
			for (int q = 0; q < 4; ++q) {
				s[p][q] = ffma2(ar, make_float2(b[q].y, b[q].y), s[p][q]);
				s[p][q] = ffma2(a[p], make_float2(b[q].x, b[q].x), s[p][q]);
			}
		}
	}
	__device__ double2 result(int p, int q) const { return make_double2(s[p][q].x, s[p][q].y); }
};

// Its sums are added to the chunk's partials every kFold steps: the rounding of
// a diagonal element's squares does not average out (squares of FP32 numbers
// have few low bits), so that its error grows with the run.  87 waves x 150,000
// events against quad precision, mean of four draws: runs of 496 events 1.4e-15,
// of 128 8.4e-16, of 64 3.8e-16, and of 752 (64 x 64 tiles) 5.4e-16.  The folds
// cost 0.7 % of 4.23 ms.
struct AccF64 {
	typedef double2 Op;
	typedef double Weight;
	static constexpr int kUnroll = 2, kFold = 64;
	static constexpr bool kAsync = false;
	double2 s[4][4];
	__device__ void init()
	{
		for (int p = 0; p < 4; ++p)
			for (int q = 0; q < 4; ++q)
				s[p][q] = make_double2(0., 0.);
	}
	static __device__ __forceinline__ int pos(int G, int row) { return (row & 3) * G + (row >> 2); }
	template <bool WT>
	__device__ void step(const double2* A, const double2* B, int G, int I, int J, double)
	{
		double2 a[4], b[4];
#pragma unroll
		for (int q = 0; q < 4; ++q) {
			a[q] = A[q * G + I];
			b[q] = B[q * G + J];
		}
#pragma unroll
		for (int p = 0; p < 4; ++p)
#pragma unroll
			for (int q = 0; q < 4; ++q) {
				s[p][q].x = fma(a[p].x, b[q].x, fma(a[p].y, b[q].y, s[p][q].x));
				s[p][q].y = fma(a[p].y, b[q].x, fma(-a[p].x, b[q].y, s[p][q].y));
			}
	}
	__device__ double2 result(int p, int q) const { return s[p][q]; }
};

struct TriArgs {
	uint64_t K, ldK, chunkLen;
	int W, g;              // rows, groups of four
	int nTiles;            // thread tiles: g (g + 1) / 2
	int tilesPerSlice;     // thread tiles of a slice in one block
	int slices, chunks;    // chunks of K side by side in a block; chunks in all
	const double* weightK;
	double* partials;
};

// One block: `slices` chunks of K, one thread tile per thread.  KT steps of
// K are staged per round in two buffers: the FP32 operands by asynchronous
// copies that run while the previous round is used (held in registers for
// that time, they spilled: 355 against 247 us per weighted call of 50 waves,
// 300,001 events), the FP64 ones
// converted and weighted on the way, beside which the FP64 pipe hides their
// loads.
template <typename Acc, typename In, int KT, bool WT>
__global__ void __launch_bounds__(kTriThreads, 2) gramTriKernel(const In* __restrict__ amps, const TriArgs a)
{
	typedef typename Acc::Op Op;
	extern __shared__ __align__(16) unsigned char smemRaw[];
	const int tid = threadIdx.x, nThreads = blockDim.x;
	// thread tile (I, J) of this thread, first group I0 of the block
	const int sl = tid / a.tilesPerSlice;
	const int t = blockIdx.x * kTriThreads + (tid - sl * a.tilesPerSlice);
	int I = 0, J = blockIdx.x * kTriThreads;
	while (J >= a.g - I)
		J -= a.g - I++;
	const int I0 = I;
	J += t - blockIdx.x * kTriThreads;
	while (I < a.g && J >= a.g - I)
		J -= a.g - I++;
	J += I;
	const int G = a.g - I0, rows = 4 * G;        // staged groups and rows
	// a step's operands are an odd number of 16-byte pieces, so that the KT
	// threads which stage a row store to different banks
	constexpr int kPad = 16 / sizeof(Op);
	const int ld = rows + kPad, stepOps = KT * ld;
	constexpr bool kTwo = WT && !Acc::kAsync;  // weighted copies beside the operands
	const int bufOps = a.slices * stepOps * (kTwo ? 2 : 1);
	Op* const buf0 = reinterpret_cast<Op*>(smemRaw);
	const uint64_t chunk0 = (uint64_t)blockIdx.y * (unsigned)a.slices;
	const bool inside = chunk0 + sl < (uint64_t)a.chunks;
	const bool mine = sl < a.slices && t < a.nTiles && (Acc::kFold == 0 || inside);
	Acc acc;
	acc.init();

	// staged rows (slice, row); their weights as the accumulators take them,
	// for two rounds
	const int total = a.slices * rows;
	TriSlot* const slots = reinterpret_cast<TriSlot*>(buf0 + 2 * bufOps);
	typename Acc::Weight* const wbuf = reinterpret_cast<typename Acc::Weight*>(slots + total);
	for (int n = tid; n < total; n += nThreads) {
		const int s = n / rows, row = n - s * rows;
		const uint64_t k0 = (chunk0 + s) * a.chunkLen;
		TriSlot z;
		z.off = (uint64_t)(4 * I0 + row) * a.ldK + k0;
		z.lim = (4 * I0 + row < a.W && k0 < a.K) ? (uint32_t)min(a.chunkLen, a.K - k0) : 0u;
		z.base = (uint32_t)(s * stepOps + Acc::pos(G, row)) | (uint32_t)s << 24;
		slots[n] = z;
	}
	// the weight of step kb + tid % KT of slice tid / KT
	const bool wMine = WT && tid < a.slices * KT;
	const uint64_t wk0 = (chunk0 + tid / KT) * a.chunkLen + (tid & (KT - 1));
	auto weight = [&](uint32_t kb) {
		const uint64_t k = wk0 + kb;
		return (wMine && kb + (tid & (KT - 1)) < a.chunkLen && k < a.K) ? a.weightK[k] : 0.;
	};
	if (wMine) {
		wbuf[tid] = (typename Acc::Weight)weight(0);
		wbuf[a.slices * KT + tid] = (typename Acc::Weight)weight(KT);
	}
	__syncthreads();
	// thread: step kk of rows tid / KT, + rowStep, ...
	const int kk = tid & (KT - 1), rowStep = nThreads / KT;
	auto stage = [&](Op* buf, uint32_t kb, int round) {
		for (int n = tid / KT; n < total; n += rowStep) {
			const TriSlot z = slots[n];
			Op* d = buf + (z.base & 0xffffffu) + kk * ld;
			const bool valid = kb + kk < z.lim;
			const In* src = amps + (valid ? z.off + kb + kk : 0);
			if constexpr (Acc::kAsync) {
				copyAsync8(d, src, valid);
			} else {
				In v{0, 0};
				if (valid)
					v = *src;
				*d = Op{(double)v.x, (double)v.y};
				if (kTwo) {
					const double w = wbuf[((round & 1) * a.slices + (z.base >> 24)) * KT + kk];
					d[a.slices * stepOps] = Op{(double)v.x * w, (double)v.y * w};
				}
			}
		}
		if constexpr (Acc::kAsync)
			asm volatile("cp.async.commit_group;" ::: "memory");
	};
	auto arrived = [&]() {
		if constexpr (Acc::kAsync)
			asm volatile("cp.async.wait_group 0;" ::: "memory");
		__syncthreads();
	};

	// the thread's sums into the chunk's partials, or added to what is there
	// (no other thread touches these elements: the atomic add is one that
	// does not wait for what it adds to)
	auto store = [&](bool add) {
		double2* out = reinterpret_cast<double2*>(a.partials) + (size_t)(chunk0 + sl) * a.W * a.W;
#pragma unroll
		for (int p = 0; p < 4; ++p)
#pragma unroll
			for (int q = 0; q < 4; ++q) {
				const int gi = 4 * I + p, gj = 4 * J + q;
				if (gi <= gj && gj < a.W) {
					const double2 v = acc.result(p, q);
					double2* o = out + (size_t)gi * a.W + gj;
					if (add) {
						atomicAdd(&o->x, v.x);
						atomicAdd(&o->y, v.y);
					} else {
						*o = v;
					}
				}
			}
	};

	stage(buf0, 0, 0);
	arrived();
	const uint32_t len = (uint32_t)a.chunkLen;
	int cur = 0;
	for (uint32_t kb = 0, round = 0; kb < len; kb += KT, ++round) {
		const bool more = kb + KT < len;
		Op* const next = buf0 + (cur ^ 1) * bufOps;
		if (Acc::kAsync && more)
			stage(next, kb + KT, round + 1);
		const double wNext = weight(kb + 2 * KT);
		if (mine) {
			const Op* b0 = buf0 + cur * bufOps + sl * stepOps;
			const Op* a0 = kTwo ? b0 + a.slices * stepOps : b0;
			const typename Acc::Weight* w0 = wbuf + ((round & 1) * a.slices + sl) * KT;
#pragma unroll Acc::kUnroll
			for (int q = 0; q < KT; ++q)
				acc.template step<WT>(a0 + q * ld, b0 + q * ld, G, I - I0, J - I0, WT ? w0[q] : 0);
			if constexpr (Acc::kFold > 0) {
				if (!more || (kb + KT) % Acc::kFold == 0) {
					store(kb >= (uint32_t)Acc::kFold);
					acc.init();
				}
			}
		}
		if (!Acc::kAsync && more)
			stage(next, kb + KT, round + 1);
		// round + 2's weights replace this round's, which have been read: by
		// the staging in the last round, or else when all threads arrive
		if (!Acc::kAsync && wMine)
			wbuf[(round & 1) * a.slices * KT + tid] = (typename Acc::Weight)wNext;
		arrived();
		if (Acc::kAsync && wMine)
			wbuf[(round & 1) * a.slices * KT + tid] = (typename Acc::Weight)wNext;
		cur ^= 1;
	}
	if (Acc::kFold == 0 && mine && inside)
		store(false);
}

// Sums chunk partials (upper triangle) in FP64 and writes the full Hermitian
// matrix; the diagonal's imaginary part is exactly zero as in the reference.
// A block holds 8 neighbouring elements x 16 slices of the chunks: the 128
// bytes of a chunk's 8 elements are read together and the loads of a thread are
// independent.  Order of the sum, the same on every run: slice y adds chunks
// y, y + 16, ... in order, then the slices are added in order.  What bounds it
// is the FP64 pipe of the SMs that have a block: 8 elements each rather than 32
// take 24.6 us instead of 51.3 for 5 to 24 waves and 2,432 chunks, 10.3 instead
// of 16.4 for 5 to 32 waves and 608, 14.4 instead of 16.4 for 87 waves and 304
// (one thread per element, chunk after chunk: 252 to 382, 66 to 98 and 51 us).
constexpr int kRedElems = 8, kRedSlices = 16;
__global__ void __launch_bounds__(kRedElems * kRedSlices) gramReduceKernel(const double* partials, int chunks, int W,
                                                                          double* out, int accumulate)
{
	__shared__ double2 part[kRedSlices][kRedElems + 1];
	const int n = W * W, x = threadIdx.x & (kRedElems - 1), y = threadIdx.x / kRedElems;
	const int e = blockIdx.x * kRedElems + x;
	const int i = e / W, j = e - i * W;
	const bool mine = e < n && i <= j;
	double re = 0., im = 0.;
	if (mine) {
		const double2* p = reinterpret_cast<const double2*>(partials) + e;
#pragma unroll 8
		for (int c = y; c < chunks; c += kRedSlices) {
			const double2 v = p[(size_t)c * n];
			re += v.x;
			im += v.y;
		}
	}
	part[y][x] = make_double2(re, im);
	__syncthreads();
	if (y != 0 || !mine)
		return;
	for (int s = 1; s < kRedSlices; ++s) {
		re += part[s][x].x;
		im += part[s][x].y;
	}
	if (i == j)
		im = 0.;
	if (accumulate) {
		re += out[(size_t)e * 2];
		im += out[(size_t)e * 2 + 1];
	}
	out[(size_t)e * 2] = re;
	out[(size_t)e * 2 + 1] = im;
	out[((size_t)j * W + i) * 2] = re;
	out[((size_t)j * W + i) * 2 + 1] = -im;
}

constexpr size_t kTriSmemMax = 112 * 1024;  // two blocks per SM

// shared memory of one chunk: two rounds of operands, the row table, weights
size_t triSliceBytes(int g, int KT, size_t opBytes, bool weighted)
{
	return (size_t)2 * KT * (4 * g * opBytes + 16) * (weighted && opBytes == sizeof(double2) ? 2 : 1) + (size_t)4 * g * sizeof(TriSlot) +
	       2 * KT * sizeof(double);
}

// most chunks that a block of gramTriKernel holds side by side with KT steps
// per round; 0 when one does not fit
int triSlices(int W, int KT, size_t opBytes, bool weighted)
{
	const int g = (W + 3) / 4, nt = g * (g + 1) / 2;
	const size_t one = triSliceBytes(g, KT, opBytes, weighted);
	if (one > kTriSmemMax)
		return 0;
	return (int)std::min<size_t>(kTriSmemMax / one, std::min(8, std::max(1, kTriThreads / nt)));
}

template <typename Acc, typename In, int KT, bool WT>
int launchTriT(const In* amps, TriArgs t, int numSMs, cudaStream_t s)
{
	t.nTiles = t.g * (t.g + 1) / 2;
	const int blocksX = (t.nTiles + kTriThreads - 1) / kTriThreads;
	// chunks side by side only where the grid keeps two blocks for each SM
	t.slices = std::max(1, std::min(triSlices(t.W, KT, sizeof(typename Acc::Op), WT),
	                                t.chunks * blocksX / (2 * numSMs)));
	t.tilesPerSlice = std::min(t.nTiles, kTriThreads);
	const size_t smem = t.slices * triSliceBytes(t.g, KT, sizeof(typename Acc::Op), WT);
	auto kern = gramTriKernel<Acc, In, KT, WT>;
	if (smem > 48 * 1024)
		PWA_CHECK(cudaCheck(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
		                    "cudaFuncSetAttribute(gram)"));
	const dim3 grid(blocksX, (t.chunks + t.slices - 1) / t.slices);
	// a thread per tile, and with weights one for each of a round's
	const int threads = (std::max(t.slices * t.tilesPerSlice, WT ? t.slices * KT : 0) + 31) / 32 * 32;
	kern<<<grid, threads, smem, s>>>(amps, t);
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "gram triangle launch");
}

template <typename Acc, typename In>
int launchTri(const In* amps, const TriArgs& t, int numSMs, cudaStream_t s)
{
	static_assert(sizeof(TriSlot) == 16, "row table entry");
	const bool wide = triSlices(t.W, 16, sizeof(typename Acc::Op), t.weightK != nullptr) == 0;
	if (t.weightK)
		return wide ? launchTriT<Acc, In, 8, true>(amps, t, numSMs, s)
		            : launchTriT<Acc, In, 16, true>(amps, t, numSMs, s);
	return wide ? launchTriT<Acc, In, 8, false>(amps, t, numSMs, s) : launchTriT<Acc, In, 16, false>(amps, t, numSMs, s);
}

bool triFits(int W, int precision, bool weighted)
{
	return triSlices(W, 8, precision == 0 ? sizeof(double2) : sizeof(float2), weighted) > 0;
}

}  // namespace

// Chunks of K: the FP32 sums depend on them in their last bits, so they stay
// the division that 64 x 64 tiles needed to fill the GPU; FP64 sums take two
// blocks of the triangle kernel per SM.
int gramSimtChunks(const GramArgs& a, int precision, int numSMs)
{
	const uint64_t most = std::max<uint64_t>(1, a.K / 64);
	if (precision == 0 && triFits(a.W, 0, a.weightK != nullptr)) {
		const int g = (a.W + 3) / 4, nt = g * (g + 1) / 2, blocks = (nt + kTriThreads - 1) / kTriThreads;
		const int slices = std::min(8, std::max(1, kTriThreads / nt));
		return (int)std::min<uint64_t>(most, (uint64_t)std::max(1, 2 * numSMs / blocks * slices));
	}
	const int tps = (a.W + kTile - 1) / kTile, nTiles = tps * (tps + 1) / 2;
	return (int)std::min<uint64_t>(most, (uint64_t)std::max(1, (4 * numSMs + nTiles - 1) / nTiles));
}

int launchGramSimt(const GramArgs& a, int precision, int numSMs, cudaStream_t s)
{
	const uint64_t chunkLen = ((a.K + a.chunks - 1) / a.chunks + kKT - 1) / kKT * kKT;
	if (triFits(a.W, precision, a.weightK != nullptr)) {
		TriArgs t{};
		t.K = a.K;
		t.ldK = a.ldK;
		t.chunkLen = chunkLen;
		t.W = a.W;
		t.g = (a.W + 3) / 4;
		t.chunks = a.chunks;
		t.weightK = a.weightK;
		t.partials = a.partials;
		if (precision != 0)
			return launchTri<AccF32, float2>(a.amps, t, numSMs, s);
		if (a.amps64)
			return launchTri<AccF64, double2>(a.amps64, t, numSMs, s);
		return launchTri<AccF64, float2>(a.amps, t, numSMs, s);
	}
	const int tps = (a.W + kTile - 1) / kTile;
	const int nTiles = tps * (tps + 1) / 2;
	dim3 grid(nTiles, a.chunks);
	if (precision == 0) {
		if (a.amps64)
			gramSimtKernel<double2, double><<<grid, 256, 0, s>>>(a.amps64, a.K, a.ldK, a.W, a.weightK, a.partials, tps,
			                                                     chunkLen);
		else
			gramSimtKernel<float2, double><<<grid, 256, 0, s>>>(a.amps, a.K, a.ldK, a.W, a.weightK, a.partials, tps,
			                                                    chunkLen);
	} else {
		gramSimtKernel<float2, float><<<grid, 256, 0, s>>>(a.amps, a.K, a.ldK, a.W, a.weightK, a.partials, tps,
		                                                   chunkLen);
	}
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "gram SIMT launch");
}

// weights of importance-sampled events (ampIntegralMatrix.cc:408-429): a
// block takes a contiguous run of events, its threads strided compensated
// sums combined in a fixed order
__global__ void __launch_bounds__(256) inverseWeightsKernel(const double* __restrict__ w, uint64_t n, uint32_t nSub,
                                                            double* out, double* sums)
{
	__shared__ double part[256];
	const uint64_t run = (n + gridDim.x - 1) / gridDim.x, k0 = blockIdx.x * run, k1 = min(n, k0 + run);
	double sum = 0., comp = 0.;
	for (uint64_t k = k0 + threadIdx.x; k < k1; k += 256) {
		const double v = 1. / w[k];
		for (uint32_t s = 0; s < nSub; ++s)
			out[k * nSub + s] = v;
		const double y = v - comp, t = sum + y;
		comp = (t - sum) - y;
		sum = t;
	}
	part[threadIdx.x] = sum - comp;
	__syncthreads();
	for (int o = 128; o > 0; o >>= 1) {
		if ((int)threadIdx.x < o)
			part[threadIdx.x] += part[threadIdx.x + o];
		__syncthreads();
	}
	if (threadIdx.x == 0)
		sums[blockIdx.x] = part[0];
}

int launchInverseWeights(const double* w, uint64_t n, uint32_t nSub, double* out, double* sums, cudaStream_t s)
{
	inverseWeightsKernel<<<kWeightBlocks, 256, 0, s>>>(w, n, nSub, out, sums);
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "weights launch");
}

// out += the blocks of a Gram of two row groups: rows and columns i < G of
// blk belong to group a (global index a G + i), the others to group b
// (b G + i - G); the cross blocks are always added, the diagonal blocks of
// group a / b only when addAA / addBB (another pair may supply them);
// indices >= nOut are padding and skipped.  One group (G = n2) adds all.
__global__ void gramBlockAddKernel(const double* blk, int n2, int G, int a, int b, int nOut, int addAA, int addBB,
                                   double* out)
{
	const int n = n2 * n2;
	for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
		const int i = e / n2, j = e - i * n2;
		const bool ia = i < G, ja = j < G;
		if ((ia && ja && !addAA) || (!ia && !ja && !addBB))
			continue;
		const int gi = ia ? a * G + i : b * G + (i - G), gj = ja ? a * G + j : b * G + (j - G);
		if (gi >= nOut || gj >= nOut)
			continue;
		out[((size_t)gi * nOut + gj) * 2] += blk[(size_t)e * 2];
		out[((size_t)gi * nOut + gj) * 2 + 1] += blk[(size_t)e * 2 + 1];
	}
}

int launchGramBlockAdd(const double* blk, int n2, int G, int a, int b, int nOut, int addAA, int addBB, double* out,
                       cudaStream_t s)
{
	const int n = n2 * n2;
	const int blocks = std::max(1, std::min(1024, (n + 255) / 256));
	gramBlockAddKernel<<<blocks, 256, 0, s>>>(blk, n2, G, a, b, nOut, addAA, addBB, out);
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "gram block add launch");
}

int launchGramReduce(const double* partials, int chunks, int W, double* out, int accumulate, cudaStream_t s)
{
	gramReduceKernel<<<(W * W + kRedElems - 1) / kRedElems, kRedElems * kRedSlices, 0, s>>>(partials, chunks, W, out,
	                                                                                      accumulate);
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "gram reduce launch");
}

namespace {

// out[w] = sum_k a[w][k] (complex64 rows of stride ld): one block per row,
// compensated FP32 sums per thread (GB300's FP64 pipe is a small fraction
// of its FP32 rate, and one FP64 add per element made this kernel slower
// than the Gram itself), FP64 across the block's threads, a fixed reduction
// order (thread-strided partial sums, then a shared-memory tree), so the
// result does not depend on the run.
__global__ void __launch_bounds__(256) rowSumsKernel(const float2* __restrict__ a, uint64_t n, uint64_t ld,
                                                     double* out)
{
	__shared__ double sre[256], sim[256];
	const float2* row = a + (uint64_t)blockIdx.x * ld;
	float re = 0.f, im = 0.f, cre = 0.f, cim = 0.f;
	for (uint64_t k = threadIdx.x; k < n; k += 256) {
		const float2 v = row[k];
		const float yr = v.x - cre, tr = re + yr;
		cre = (tr - re) - yr;
		re = tr;
		const float yi = v.y - cim, ti = im + yi;
		cim = (ti - im) - yi;
		im = ti;
	}
	sre[threadIdx.x] = (double)re - (double)cre;
	sim[threadIdx.x] = (double)im - (double)cim;
	__syncthreads();
	for (int o = 128; o > 0; o >>= 1) {
		if ((int)threadIdx.x < o) {
			sre[threadIdx.x] += sre[threadIdx.x + o];
			sim[threadIdx.x] += sim[threadIdx.x + o];
		}
		__syncthreads();
	}
	if (threadIdx.x == 0) {
		out[2 * blockIdx.x] = sre[0];
		out[2 * blockIdx.x + 1] = sim[0];
	}
}

}  // namespace

int launchRowSums(const float2* a, uint64_t n, uint64_t ld, int W, double* out, cudaStream_t s)
{
	rowSumsKernel<<<W, 256, 0, s>>>(a, n, ld, out);
	countLaunches(1);
	return cudaCheck(cudaGetLastError(), "row sums launch");
}

}  // namespace pwa
