/*
 * BC7 decode and result-reduction kernels (used by the C ABI layer only).
 */
#pragma once

#include "bc7_encode.cuh"

namespace nebc7 {

/* Decodes blocks to BGRA pixels (src/Bc7Core.cpp:1904 DecompressKernel):
   one thread per pixel. */
__global__ void KDecode(const uint8_t* blocks, uint8_t* bgra, long long stride, int blocksW, int nblocks)
{
	const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= (long long)nblocks * 16)
		return;
	const int k = int(t >> 4), i = int(t & 15);
	const uint4 b = *reinterpret_cast<const uint4*>(blocks + (long long)k * 16);
	const uint64_t lo = uint64_t(b.x) | (uint64_t(b.y) << 32);
	const uint64_t hi = uint64_t(b.z) | (uint64_t(b.w) << 32);
	uint8_t px[4];
	Ep best[3];
	int param, mode;
	DecodeBlock(lo, hi, i, px, best, param, mode);
	const int bx = k % blocksW, by = k / blocksW;
	uint8_t* p = bgra + ((long long)by * 4 + (i >> 2)) * stride + (long long)bx * 16 + (i & 3) * 4;
	*reinterpret_cast<uchar4*>(p) = make_uchar4(px[3], px[1], px[2], px[0]);
}

/* Deterministic sums of n per-block results: a fixed-shape tree of 256
   threads, so repeated runs give identical double sums; thread 0 returns them.
   A thread's results are read eight at a time and added in order: the reads
   are in flight together (one at a time the sums of a 1118x1105 image took
   93 us, four times what its additions do). */
__device__ __forceinline__ void SumResults(const BlockResult* r, int n, long long& errAlpha, long long& errColor, double& ssimAlpha,
	double& ssimColor)
{
	__shared__ long long sa[256], sc[256];
	__shared__ double qa[256], qc[256];
	const int t = threadIdx.x;
	long long a = 0, c = 0;
	double x = 0, y = 0;
	for (int i = t; i < n; i += 256 * 8)
	{
		BlockResult v[8];
#pragma unroll
		for (int j = 0; j < 8; j++)
			if (i + 256 * j < n)
				v[j] = r[i + 256 * j];
#pragma unroll
		for (int j = 0; j < 8; j++)
			if (i + 256 * j < n)
			{
				a += v[j].errAlpha;
				c += v[j].errColor;
				x = __dadd_rn(x, v[j].ssimAlpha);
				y = __dadd_rn(y, v[j].ssimColor);
			}
	}
	sa[t] = a;
	sc[t] = c;
	qa[t] = x;
	qc[t] = y;
	__syncthreads();
	for (int s = 128; s > 0; s >>= 1)
	{
		if (t < s)
		{
			sa[t] += sa[t + s];
			sc[t] += sc[t + s];
			qa[t] = __dadd_rn(qa[t], qa[t + s]);
			qc[t] = __dadd_rn(qc[t], qc[t + s]);
		}
		__syncthreads();
	}
	errAlpha = sa[0];
	errColor = sc[0];
	ssimAlpha = qa[0];
	ssimColor = qc[0];
}

/* Sums of one texture's results. */
__global__ void KReduceResults(const BlockResult* r, int n, long long* errs, double* ssims)
{
	long long a, c;
	double x, y;
	SumResults(r, n, a, c, x, y);
	if (threadIdx.x == 0)
	{
		errs[0] = a;
		errs[1] = c;
		ssims[0] = x;
		ssims[1] = y;
	}
}

/* Per-texture sums of a batch: CTA t reduces the per-block results of
   table entry t (its own array, or its queue positions of r) with the tree of
   KReduceResults (so a texture's sums do not depend on the batch), into
   sums[tex[t].id] = { errAlpha, errColor } and ssims[...] = { alpha, color }. */
__global__ void KReduceTextures(const BlockResult* r, const TexDesc* tex, long long* errs, double* ssims)
{
	const TexDesc& d = tex[blockIdx.x];
	long long a, c;
	double x, y;
	SumResults(d.results ? d.results : r + d.first, d.nblocks, a, c, x, y);
	if (threadIdx.x == 0)
	{
		errs[2 * d.id] = a;
		errs[2 * d.id + 1] = c;
		ssims[2 * d.id] = x;
		ssims[2 * d.id + 1] = y;
	}
}

} // namespace nebc7
