/*
 * BC7 decode and result-reduction kernels (used by the C ABI layer only).
 */
#pragma once

#include "bc7_encode.cuh"

namespace nebc7 {

/* A 128-bit block read from its low end. */
struct BlockBits
{
	uint32_t w[4];

	__device__ __forceinline__ unsigned Take(int n)
	{
		const unsigned v = w[0] & ((1u << n) - 1);
		w[0] = __funnelshift_r(w[0], w[1], n);
		w[1] = __funnelshift_r(w[1], w[2], n);
		w[2] = __funnelshift_r(w[2], w[3], n);
		w[3] >>= n;
		return v;
	}
};

/* Endpoint bytes e0 and e1 (four channels) interpolated by w / 64, two
   channels to a multiplication (at most 255 * 64 + 32 each). */
__device__ __forceinline__ uint32_t LerpBytes(uint32_t e0, uint32_t e1, int w)
{
	const uint32_t even = ((e0 & 0x00FF00FFu) * (64 - w) + (e1 & 0x00FF00FFu) * w + 0x00200020u) >> 6;
	const uint32_t odd = ((e0 >> 8) & 0x00FF00FFu) * (64 - w) + ((e1 >> 8) & 0x00FF00FFu) * w + 0x00200020u;
	return (even & 0x00FF00FFu) | ((odd << 2) & 0xFF00FF00u);
}

/* The index bits of a block, every index `bits` wide: the anchors' missing
   top bits put back as 0 (anchors ascending; -1 for none). */
__device__ __forceinline__ uint64_t WidenIndices(uint64_t v, int bits, int a1, int a2)
{
	v = InsertZeroBit(v, bits - 1);
	if (a1 >= 0)
		v = InsertZeroBit(v, a1 * bits + bits - 1);
	if (a2 >= 0)
		v = InsertZeroBit(v, a2 * bits + bits - 1);
	return v;
}

/* Decodes blocks to BGRA pixels (src/Bc7Core.cpp:1904 DecompressKernel): one
   thread per block, so that its header is read once and a warp writes 512
   contiguous bytes of a pixel row.  Memory bound: 16 bytes in and 64 out per
   block.  One thread per pixel decoded every header 16 times and kept it in
   local memory.  `wide`: the rows are 16-byte aligned. */
__global__ void __launch_bounds__(128) KDecode(const uint8_t* blocks, uint8_t* bgra, long long stride, int blocksW, int nblocks, bool wide)
{
	/* interpolation weights by index width and index */
	__shared__ uint8_t weights[5][16];
	if (threadIdx.x < 16)
	{
		const int i = threadIdx.x;
		weights[2][i] = uint8_t(c_interp2[i & 3]);
		weights[3][i] = uint8_t(c_interp3[i & 7]);
		weights[4][i] = uint8_t(c_interp4[i]);
	}
	__syncthreads();
	const int k = blockIdx.x * blockDim.x + threadIdx.x;
	if (k >= nblocks)
		return;
	const uint4 raw = reinterpret_cast<const uint4*>(blocks)[k];
	BlockBits b{ { raw.x, raw.y, raw.z, raw.w } };
	const int mode = (raw.x & 0xFF) ? __ffs(int(raw.x & 0xFF)) - 1 : 8;
	/* per mode: subsets, colour, alpha and index bits (a nibble per mode) */
	auto field = [&](uint32_t packed) { return int((packed >> (4 * (mode & 7))) & 0xF); };
	const int ns = field(0x21112323u), cbits = field(0x57757564u), abits = field(0x57860000u);
	const int ib = field(0x24222233u);
	const bool split = mode == 4 || mode == 5;   /* separate colour and alpha-slot indices */
	b.Take(mode + 1 < 8 ? mode + 1 : 8);
	const int part = int(b.Take(ns > 1 ? (mode == 0 ? 4 : 6) : 0));
	const int rotation = int(b.Take(split ? 2 : 0));
	const bool idx32 = b.Take(mode == 4 ? 1 : 0) != 0;

	/* endpoints as BGRA bytes, subset s: e[s][0], e[s][1] */
	uint32_t e[3][2] = { { 0, 0 }, { 0, 0 }, { 0, 0 } };
	/* a p-bit per endpoint except in modes 2, 4, 5 (mode 1: per subset); the
	   values are left at the top of their byte, above the p-bit's place */
	const bool pbit = mode != 2 && !split;
	const int cw = cbits + int(pbit), aw = abits + int(pbit);
#pragma unroll
	for (int c = 0; c < 4; c++)
	{
		/* stored order R, G, B, A; BGRA byte of each */
		const int at = c == 0 ? 16 : (c == 1 ? 8 : (c == 2 ? 0 : 24));
		const int n = c < 3 ? cbits : abits, width = c < 3 ? cw : aw;
#pragma unroll
		for (int s = 0; s < 3; s++)
#pragma unroll
			for (int h = 0; h < 2; h++)
				if (s < ns)
					e[s][h] |= (n ? b.Take(n) << (8 - width + int(pbit)) : 0u) << at;
	}
	if (pbit)
	{
		const uint32_t ones = (0x00010101u << (8 - cw)) | (abits ? 0x01000000u << (8 - aw) : 0u);
#pragma unroll
		for (int s = 0; s < 3; s++)
			if (s < ns)
			{
				const unsigned p0 = b.Take(1), p1 = mode == 1 ? p0 : b.Take(1);
				e[s][0] |= p0 ? ones : 0u;
				e[s][1] |= p1 ? ones : 0u;
			}
	}
	/* the top bits repeated below (Expand, every channel at once) */
#pragma unroll
	for (int s = 0; s < 3; s++)
#pragma unroll
		for (int h = 0; h < 2; h++)
		{
			const uint32_t v = e[s][h];
			const uint32_t col = v & 0x00FFFFFFu, low = (0xFFu >> cw) * 0x00010101u;
			const uint32_t alpha = v >> 24;
			e[s][h] = col | ((col >> cw) & low) | (abits ? (alpha | (alpha >> aw)) << 24 : 0xFF000000u);
		}

	const uint64_t lo = uint64_t(b.w[0]) | (uint64_t(b.w[1]) << 32), hi = b.w[2];
	uint64_t idxC, idxA = 0;
	int ibA = 2, ibC = ib;
	if (split)
	{
		const uint64_t first = lo & 0x7FFFFFFFull;
		const uint64_t second = (lo >> 31) | (hi << 33);
		const int second_bits = mode == 4 ? 3 : 2;
		const uint64_t i0 = WidenIndices(first, 2, -1, -1);
		const uint64_t i1 = WidenIndices(second & ((1ull << (16 * second_bits - 1)) - 1), second_bits, -1, -1);
		idxC = idx32 ? i1 : i0;
		idxA = idx32 ? i0 : i1;
		ibC = idx32 ? second_bits : 2;
		ibA = idx32 ? 2 : second_bits;
	}
	else
	{
		int a1 = -1, a2 = -1;
		if (ns == 2)
			a1 = c_anchor22[part];
		else if (ns == 3)
		{
			const int x = c_anchor23[part], y = c_anchor33[part];
			a1 = x < y ? x : y;
			a2 = x < y ? y : x;
		}
		idxC = WidenIndices(lo, ib, a1, a2);
	}
	uint32_t subsets = ns == 3 ? c_part3[part] : (ns == 2 ? c_part2[part] : 0u);
	/* the channel that a rotation swaps with alpha: R, G, B */
	const int swap = rotation == 0 ? 24 : (rotation == 1 ? 16 : (rotation == 2 ? 8 : 0));

	const unsigned maskC = (1u << ibC) - 1;
	const int bx = k % blocksW, by = k / blocksW;
	uint8_t* out = bgra + (long long)by * 4 * stride + (long long)bx * 16;
#pragma unroll
	for (int r = 0; r < 4; r++, out += stride)
	{
		uint32_t px[4];
		unsigned rowC = unsigned(idxC), rowA = unsigned(idxA);
		idxC >>= 4 * ibC;
		idxA >>= 4 * ibA;
#pragma unroll
		for (int x = 0; x < 4; x++)
		{
			const unsigned s = subsets & 3;
			subsets >>= 2;
			const uint32_t e0 = s == 0 ? e[0][0] : (s == 1 ? e[1][0] : e[2][0]);
			const uint32_t e1 = s == 0 ? e[0][1] : (s == 1 ? e[1][1] : e[2][1]);
			uint32_t v = LerpBytes(e0, e1, weights[ibC][rowC & maskC]);
			rowC >>= ibC;
			if (split)
			{
				const uint32_t slot = LerpBytes(e0, e1, weights[ibA][rowA & ((1u << ibA) - 1)]) >> 24;
				rowA >>= ibA;
				/* the slot's value is the rotated channel's, whose own is alpha's */
				const uint32_t own = (v >> swap) & 0xFF;
				v = (v & 0x00FFFFFFu & ~(0xFFu << swap)) | (slot << swap);
				if (swap != 24)
					v |= own << 24;
			}
			px[x] = mode == 8 ? 0u : v;
		}
		if (wide)
			*reinterpret_cast<uint4*>(out) = make_uint4(px[0], px[1], px[2], px[3]);
		else
		{
			uint32_t* o = reinterpret_cast<uint32_t*>(out);
#pragma unroll
			for (int x = 0; x < 4; x++)
				o[x] = px[x];
		}
	}
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
