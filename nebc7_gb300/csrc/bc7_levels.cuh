/*
 * BC7 block encoder for sm_103a -- per-channel candidate endpoint lists and
 * lower-bound estimates, warp-cooperative.
 *
 * ChannelLevels reproduces the reference's LevelsBuffer::
 * ComputeChannelLevelsReduced (src/SnippetLevelsBuffer.h:43-270), the nibble
 * variant of src/SnippetLevelsBufferHalf.h:43-223 and the single-best
 * variant (:148-188).  For one channel of one pixel subset it enumerates a
 * window of quantised endpoint pairs c, scores each by
 *   e(c) = sum_i D(x_i, c)^2   (D from the level tables),
 * keeps those with e < top, and returns the maxSize smallest keys
 * (e << 16 | c) in ascending order.  The reference collects all survivors
 * and radix-sorts them stably on e; since survivors are produced in
 * ascending c, that is the same as the smallest keys of the 32-bit key, which
 * is what the warp keeps here: lanes score 32 candidates at a time and a
 * bitonic merge folds them into a lane-resident sorted top-N.  Candidates are
 * visited in ascending c, so once the list is full a later candidate can only
 * enter with a strictly smaller error.
 *
 * The window arithmetic keeps the reference's 32-bit wrap-around behaviour
 * (its water can be negative for a later channel of a subset), and the
 * candidate set follows the chunking of its 16-wide AVX2 scan.
 */
#pragma once

#include "bc7_block.cuh"

namespace nebc7 {

struct ChanList
{
	int minErr;
	int count;
};

__device__ __forceinline__ int Wadd(int a, int b) { return int(unsigned(a) + unsigned(b)); }
__device__ __forceinline__ int Wsub(int a, int b) { return int(unsigned(a) - unsigned(b)); }
__device__ __forceinline__ unsigned Shr32(unsigned v, unsigned s) { return v >> (s & 31); }

/* A reduced table's s-bit endpoint expanded to 8 bits by bit replication. */
__device__ __forceinline__ int ExpandTo8(int v, int s)
{
	return s >= 8 ? v : ((v << (8 - s)) | (v >> (2 * s - 8)));
}

/* The reduced tables of s-bit endpoints hold, for every x, the 8-bit
   table's entry at the expanded endpoints; the 8-bit byte tables of 2- and
   3-bit indices are stored by endpoint differences (DiffAt).  For
   candidate cc (endpoints cc >> s, cc & (2^s - 1)) the difference-table
   entry of channel value x is table[DiffBase(cc, s) - 513 x]: one lookup
   per term, as in the per-x layout, but in a region near the table's
   diagonal that every block shares, where the per-x rows of the distinct
   values of a channel lie far apart. */
__device__ __forceinline__ int DiffBase(int cc, int s)
{
	const int eH = ExpandTo8(cc >> s, s), eL = ExpandTo8(cc & ((1 << s) - 1), s);
	return (eH << 9) + eL + 255 * 513;
}

/* d with d*d < top (src/SnippetLevelsBuffer.h:78-88): truncated single
   precision square root, NaN (negative top) giving INT_MIN. */
template<int kD>
__device__ __forceinline__ int WindowRadius(int top)
{
	int d;
	if (top < 0)
		d = int(0x80000000u);
	else
		d = __float2int_rz(__fsqrt_rn(__int2float_rn(top)));
	const int sq = int(unsigned(d) * unsigned(d));   /* x86 imul wraps */
	d = Wsub(d, sq >= top ? 1 : 0);
	if (kD)
	{
		d = int(unsigned(d) << kD);
		d = Wadd(d, (1 << kD) - 1);
	}
	return d;
}

struct Window
{
	int LH, HL, HH;
};

/* src/SnippetLevelsBuffer.h:122-132 */
__device__ __forceinline__ Window MakeWindow(int L, int H, int d, int bits, int shift)
{
	const int tailmask = (1 << (8 - bits)) - 1;
	int LH = min(Wadd(L, d), 255);
	int HL = max(Wsub(H, d), 0);
	LH = min(Wadd(Wsub(H, H >> shift), tailmask), Wsub(LH, LH >> shift)) & ~tailmask;
	HL = max(Wsub(L, L >> shift), Wadd(Wsub(HL, HL >> shift), tailmask)) & ~tailmask;
	Window w;
	w.LH = LH >> (8 - shift);
	w.HL = HL >> (8 - shift);
	w.HH = 0x100 >> (8 - shift);
	return w;
}

/* Packed candidate index -> endpoint pair color (e0 | e1 << 8), honouring a
   channel whose oriented bounds run high to low (src/SnippetLevelsBuffer.h:230-268). */
__device__ __forceinline__ int DecodeColor(int c, int shift, bool reverse)
{
	if (reverse)
	{
		const int cL = (c >> shift) << (8 - shift);
		const int cH = (c & ((1 << shift) - 1)) << (8 - shift);
		return ((cH + (cH >> shift)) << 8) + cL + (cL >> shift);
	}
	if (shift != 8)
	{
		const int cH = (c >> shift) << (8 - shift);
		const int cL = (c & ((1 << shift) - 1)) << (8 - shift);
		return ((cH + (cH >> shift)) << 8) + cL + (cL >> shift);
	}
	return c;
}

/* Lane-resident sorted list of the N smallest keys (lane j holds the j-th). */
__device__ __forceinline__ unsigned BitonicSort32(unsigned v, int lane)
{
#pragma unroll
	for (int k = 2; k <= 32; k <<= 1)
	{
#pragma unroll
		for (int j = k >> 1; j > 0; j >>= 1)
		{
			const unsigned o = __shfl_xor_sync(kFull, v, j);
			const bool keepMin = ((lane & j) == 0) == ((lane & k) == 0);
			v = keepMin ? min(v, o) : max(v, o);
		}
	}
	return v;
}

/* Folds the lanes' keys (`want`: the lanes with one below the list's last)
   into the list of the N smallest.  A few keys are inserted one by one (about
   12 instructions each), more by a bitonic sort and merge (about 90). */
__device__ __forceinline__ unsigned MergeTop(unsigned list, unsigned key, unsigned want, int lane, int N)
{
	if (__popc(want) <= 6)
	{
		do
		{
			const unsigned k = __shfl_sync(kFull, key, __ffs(want) - 1);
			want &= want - 1;
			const int at = __popc(__ballot_sync(kFull, list < k));
			const unsigned up = __shfl_up_sync(kFull, list, 1);
			list = lane < at ? list : (lane == at ? k : up);
		} while (want);
		return lane < N ? list : 0xFFFFFFFFu;
	}
	const unsigned s = BitonicSort32((want >> lane) & 1 ? key : 0xFFFFFFFFu, lane);
	const unsigned r = __shfl_sync(kFull, s, 31 - lane);
	unsigned m = min(list, r);
#pragma unroll
	for (int j = 16; j > 0; j >>= 1)
	{
		const unsigned o = __shfl_xor_sync(kFull, m, j);
		m = ((lane & j) == 0) ? min(m, o) : max(m, o);
	}
	return lane < N ? m : 0xFFFFFFFFu;
}

/* The distinct values of channel `c` among the first `count` pixels of an
   area: the table offset x * stride, and the multiplicity with the value
   above it (count | x << 8).  The scans sum a candidate's error once per
   distinct value (the integer sums, and so the saturated ones, are the
   same).  The smallest and the largest value (L, H) come first: they reject
   most candidates, which the scans test after every fourth value.  Entries
   of count 0 fill up to a multiple of 4.  Returns how many values. */
__device__ __forceinline__ int DistinctValues(const Area& ar, int count, int c, int L, int H, int stride, int2* values, int lane)
{
	const int x = lane < count ? int(ar.px[lane & 15][c]) : -1 - lane;
	const unsigned peers = __match_any_sync(kFull, x);
	const bool leader = lane < count && (__ffs(peers) - 1) == lane;
	const unsigned all = __ballot_sync(kFull, leader);
	const unsigned low = __ballot_sync(kFull, leader && x == L);
	const unsigned high = __ballot_sync(kFull, leader && x == H) & ~low;
	const unsigned rest = all & ~(low | high);
	const int n = __popc(all), first = __popc(low | high);
	if (leader)
	{
		const int slot = x == L ? 0 : (x == H ? __popc(low) : first + __popc(rest & ((1u << lane) - 1)));
		values[slot] = make_int2(x * stride, __popc(peers) | (x << 8));
	}
	if (lane >= n && lane < ((n + 3) & ~3))
		values[lane] = make_int2(0, 0);
	__syncwarp();
	return n;
}

/* Four distinct values in registers: the first four, which every batch of a
   scan reads. */
struct ValueGroup
{
	int off[4];
	unsigned mult[4];

	__device__ __forceinline__ void Load(const int2* values)
	{
		const int4 a = reinterpret_cast<const int4*>(values)[0], b = reinterpret_cast<const int4*>(values)[1];
		off[0] = a.x, off[1] = a.z, off[2] = b.x, off[3] = b.z;
		mult[0] = a.y & 0xFF, mult[1] = a.w & 0xFF, mult[2] = b.y & 0xFF, mult[3] = b.w & 0xFF;
	}

	/* sum of mult * D^2; SQUARED: the table holds the squares */
	template<bool SQUARED>
	__device__ __forceinline__ unsigned Sum(const uint8_t* row) const
	{
		const unsigned v0 = row[off[0]], v1 = row[off[1]], v2 = row[off[2]], v3 = row[off[3]];
		if (SQUARED)
			return (mult[0] * v0 + mult[1] * v1) + (mult[2] * v2 + mult[3] * v3);
		return (mult[0] * v0 * v0 + mult[1] * v1 * v1) + (mult[2] * v2 * v2 + mult[3] * v3 * v3);
	}
};

/* The rest of a lane's error sum after its first group of four values (`s`),
   given up after a group once no lane's sum is at most `limit`.  Returns
   whether some lane's is.  Warp-collective. */
template<bool SQUARED>
__device__ __forceinline__ bool CandidateRest(const uint8_t* row, const int2* values, int n, bool on, int limit, int& s)
{
	for (int u = 4;; u += 4)
	{
		if (!__any_sync(kFull, on && s <= limit))
			return false;
		if (u >= n)
			return true;
		ValueGroup g;
		g.Load(values + u);
		s += int(g.Sum<SQUARED>(row));
	}
}

/* Error sum of a lane's candidate (`row`: its place in the table, the values'
   offsets go from there), given up as CandidateRest. */
template<bool SQUARED>
__device__ __forceinline__ bool CandidateSum(const uint8_t* row, const ValueGroup& first, const int2* values, int n, bool on, int limit,
	int& sum)
{
	sum = int(first.Sum<SQUARED>(row));
	return CandidateRest<SQUARED>(row, values, n, on, limit, sum);
}

/* Sets node 0 (a zero-error candidate) of a list. */
__device__ __forceinline__ ChanList ZeroList(int2* nodes, int color, int lane)
{
	if (lane == 0)
		nodes[0] = make_int2(0, color);
	__syncwarp();
	return ChanList{ 0, 1 };
}

/* The warps that search a block together: the CTA's four, or one alone
   (size 1).  They exchange candidate lists through shared memory. */
struct TeamExchange
{
	unsigned list[2][4][32];   /* two buffers, taken in turn: one barrier a scan */
};

struct Team
{
	int size, rank;
	TeamExchange* exchange;
	int turn;                  /* buffer of the next scan */

	__device__ __forceinline__ void Sync() const
	{
		if (size > 1)
			__syncthreads();
		else
			__syncwarp();
	}
};

__device__ __forceinline__ Team SingleWarp() { return Team{ 1, 0, nullptr, 0 }; }

/* The N smallest keys of the team's lists (each sorted over the lanes), in
   every warp. */
__device__ __forceinline__ unsigned TeamMerge(unsigned list, Team& team, int lane, int N)
{
	TeamExchange& x = *team.exchange;
	x.list[team.turn][team.rank][lane] = list;
	__syncthreads();
#pragma unroll 1
	for (int w = 1; w < 4; w++)
	{
		/* the smaller half of two sorted lists is bitonic */
		unsigned m = min(list, x.list[team.turn][(team.rank + w) & 3][31 - lane]);
#pragma unroll
		for (int j = 16; j > 0; j >>= 1)
		{
			const unsigned o = __shfl_xor_sync(kFull, m, j);
			m = ((lane & j) == 0) ? min(m, o) : max(m, o);
		}
		list = m;
	}
	team.turn ^= 1;
	return lane < N ? list : 0xFFFFFFFFu;
}

/* Place of candidate cc in a table: by differences (DiffBase), or the
   per-x layout of mode 1's shared-p-bit table. */
__device__ __forceinline__ int CandidateBase(int cc, int shift, bool byDiff)
{
	return byDiff ? DiffBase(cc, shift) : cc;
}

/* Table offset of a value x from a candidate's place: x times this. */
__device__ __forceinline__ int ValueStride(int shift, bool byDiff)
{
	return byDiff ? -513 : 1 << (2 * shift);
}

/* LevelsBuffer and LevelsBufferHalf: writes up to maxSize nodes (err, color).
 *
 * What bounds it: the latency of the table reads (256 KB, mostly in L2) and the
 * chains behind them, about 1200 candidates a scan in the default preset and
 * 4000 in an alpha block's mode 6; so two batches are in flight at a time
 * (64x64 icon 0.76 -> 0.73 ms, refinement of a 1024x1024 photo, precise, 8.6 ->
 * 8.2).  Every row of the window has the same candidates (low endpoints up to
 * the window's, rounded up as the reference's 16-wide chunks do), so rows and
 * columns are taken as one sequence of candidates in ascending order, 32 a
 * batch with every lane in use, and a batch ends after the four values that
 * reject most unless a lane can still enter the list. */
template<int kD, bool HALF>
__device__ __forceinline__ ChanList ChannelLevelsScan(int2* nodes, const Area& ar, int offset, int weight, int water, int bits, int pbits,
	bool transparent, const uint8_t* table, bool byDiff, int maxSize, int2* values, Team& team, int lane)
{
	ChanList res{ MaxColorError<kD>() * 2, 0 };
	const AreaInfo& ai = ar.info;
	const int shift = bits + int(pbits >= 0 || HALF);
	const int count = transparent ? ai.active : ai.count;
	if (transparent && !count)
		return ZeroList(nodes, (pbits < 0) ? 0 : (pbits << (7 - bits)), lane);

	int top = (water + weight - 1) / weight;
	if (!top)
		return res;
	const int d = WindowRadius<kD>(top);

	const int L = int(int16_t(ai.minmax[2 * offset]));
	const int H = int(int16_t(ai.minmax[2 * offset + 1]));
	const bool reverse = (L != int(int16_t(ai.bounds[2 * offset])));

	if ((pbits < 0) || ((pbits >> 8) == (pbits & 1)))
	{
		if (L == H && ((((L >> shift) ^ L) & ((1 << (8 - shift)) - 1)) == 0))
		{
			if ((pbits < 0) || (((L >> (8 - shift)) & 1) == (pbits & 1)))
				return ZeroList(nodes, (H << 8) + L, lane);
		}
	}

	const Window win = MakeWindow(L, H, d, bits, shift);
	/* errors up to `limit` are below the top: the half tables compare signed
	   (a negative top rejects everything), the byte tables the low 16 bits */
	int limit = HALF ? min(top, 15 * 15 * 16 + 1) - 1 : (min(top, 0xFFFF) & 0xFFFF) - 1;

	const bool pvar = HALF || pbits >= 0;
	const int pH = reverse ? (pbits & 1) : (pbits >> 8);
	const int pL = reverse ? (pbits >> 8) : (pbits & 1);
	const int step = pvar ? 2 : 1;
	/* low endpoints of a row: 0 .. LH | 7; a window of a negative top that
	   wrapped below zero leaves the part of the first chunk that the
	   reference's shift count (modulo 32) does */
	const int span = win.LH >= 0 ? (win.LH | 7) : ((win.LH | 7) & (pvar ? 31 : 15));
	const int rowLen = pvar ? (span >> 1) + 1 : span + 1;
	/* a team's warps take every fourth batch */
	const int stride = 32 * team.size, start = 32 * team.rank + lane;
	const int stepRows = stride / rowLen, stepCols = stride - stepRows * rowLen;

	const int n = DistinctValues(ar, count, offset, L, H, ValueStride(shift, byDiff), values, lane);
	ValueGroup first;
	first.Load(values);

	/* list: the maxSize smallest keys so far, lane j the j-th; thr: its last
	   key (all ones until the list is full), which changes only on a merge */
	unsigned list = 0xFFFFFFFFu;
	unsigned thr = 0xFFFFFFFFu;
	int row = start / rowLen, col = start - row * rowLen;
	int iH = win.HL + (pvar ? pH : 0);   /* the batch's first row */
	/* the next candidates; row stays relative to the batch's first */
	auto advance = [&]() {
		row += stepRows;
		col += stepCols;
		if (col >= rowLen)
		{
			col -= rowLen;
			row++;
		}
	};
	while (iH < win.HH)
	{
		/* two batches at a time */
		int cc[2];
		bool on[2];
#pragma unroll
		for (int h = 0; h < 2; h++)
		{
			const int myH = iH + row * step;
			on[h] = myH < win.HH;
			cc[h] = on[h] ? (myH << shift) + col * step + (pvar ? pL : 0) : 0;
			advance();
		}
		const uint8_t* const place[2] = { table + CandidateBase(cc[0], shift, byDiff), table + CandidateBase(cc[1], shift, byDiff) };
		const unsigned s0 = first.Sum<HALF>(place[0]), s1 = first.Sum<HALF>(place[1]);
		if (__any_sync(kFull, (on[0] && int(s0) <= limit) || (on[1] && int(s1) <= limit)))
		{
#pragma unroll 1
			for (int h = 0; h < 2; h++)
			{
				const bool mine = h ? on[1] : on[0];
				int s = int(h ? s1 : s0);
				if (CandidateRest<HALF>(h ? place[1] : place[0], values, n, mine, limit, s))
				{
					const unsigned key = (unsigned(s) << 16) | unsigned(h ? cc[1] : cc[0]);
					const unsigned want = __ballot_sync(kFull, mine && s <= limit && key < thr);
					if (want)
					{
						list = MergeTop(list, key, want, lane, maxSize);
						thr = __shfl_sync(kFull, list, maxSize - 1);
						limit = min(limit, int(thr >> 16));
					}
				}
			}
			/* maxSize zero-error candidates found: later ones (larger c)
			   cannot enter */
			if (thr < 0x10000u)
				break;
		}
		const int ahead = __shfl_sync(kFull, row, 0);
		iH += ahead * step;
		row -= ahead;
	}
	if (team.size > 1)
		list = TeamMerge(list, team, lane, maxSize);
	const int stored = __popc(__ballot_sync(kFull, list != 0xFFFFFFFFu));
	if (stored)
	{
		res.count = stored;
		const unsigned k0 = __shfl_sync(kFull, list, 0);
		res.minErr = int(k0 >> 16) * weight;
		if (lane < res.count)
			nodes[lane] = make_int2(int(list >> 16) * weight, DecodeColor(int(list & 0xFFFF), shift, reverse));
	}
	__syncwarp();
	return res;
}

/* The scan as its call sites take it (NEBC7_SHARED: out of line in the single
   kernels). */
template<int kD, bool HALF>
__device__ NEBC7_SHARED ChanList ChannelLevels(int2* nodes, const Area& ar, int offset, int weight, int water, int bits, int pbits,
	bool transparent, const uint8_t* table, bool byDiff, int maxSize, int2* values, Team& team, int lane)
{
	return ChannelLevelsScan<kD, HALF>(nodes, ar, offset, weight, water, bits, pbits, transparent, table, byDiff, maxSize, values, team, lane);
}

/* Single best candidate over the narrower window of the alpha slot of modes
   4 and 5 (src/SnippetLevelsBuffer.h:148-188, 433-490): a row's low endpoints
   go up to its high one. */
template<int kD>
__device__ NEBC7_SHARED ChanList ChannelLevelsSingle(int2* nodes, const Area& ar, int offset, int weight, int water, int bits,
	bool transparent, const uint8_t* table, int2* values, int lane)
{
	ChanList res{ MaxColorError<kD>() * 2, 0 };
	const AreaInfo& ai = ar.info;
	const int shift = bits;
	const int count = transparent ? ai.active : ai.count;
	if (transparent && !count)
		return ZeroList(nodes, 0, lane);
	int top = (water + weight - 1) / weight;
	if (!top)
		return res;
	const int d = WindowRadius<kD>(top);
	const int L = int(int16_t(ai.minmax[2 * offset]));
	const int H = int(int16_t(ai.minmax[2 * offset + 1]));
	const bool reverse = (L != int(int16_t(ai.bounds[2 * offset])));
	if (L == H && ((((L >> shift) ^ L) & ((1 << (8 - shift)) - 1)) == 0))
		return ZeroList(nodes, (H << 8) + L, lane);
	const Window win = MakeWindow(L, H, d, bits, shift);
	int limit = (min(top, 0xFFFF) & 0xFFFF) - 1;
	const int n = DistinctValues(ar, count, offset, L, H, ValueStride(shift, true), values, lane);
	ValueGroup first;
	first.Load(values);

	unsigned best = 0xFFFFFFFFu;
	/* two rows per batch when only a row's first chunk can be on */
	const bool twoRows = win.LH < 16;
	for (int iH0 = win.HL; iH0 < win.HH; iH0 += twoRows ? 2 : 1)
	{
		for (int b = 0;; b++)
		{
			const int half = lane >> 4, j = lane & 15;
			const int iH = twoRows ? iH0 + half : iH0;
			const int cH = iH << shift;
			const int hL = min(win.LH, iH) + cH;
			const int c = cH + 16 * (twoRows ? b : 2 * b + half);
			const unsigned mask = Shr32(~0u, unsigned(max(0, Wsub(c | 15, hL | 7))) << 1);
			const bool chunkOn = (iH < win.HH) && ((c == cH) || (c <= hL));
			if (!__any_sync(kFull, chunkOn))
				break;
			const bool on = chunkOn && ((mask >> (2 * j)) & 1);
			const int cc = on ? c + j : 0;
			int s;
			if (CandidateSum<false>(table + DiffBase(cc, shift), first, values, n, on, limit, s))
			{
				if (on && s <= limit)
					best = min(best, (unsigned(s) << 16) | unsigned(cc));
				/* equal errors keep the earlier candidate */
				limit = min(limit, int(__reduce_min_sync(kFull, best) >> 16) - 1);
			}
		}
	}
	best = __reduce_min_sync(kFull, best);
	if (best != 0xFFFFFFFFu)
	{
		const int e = int(best >> 16) * weight;
		res.minErr = e;
		res.count = 1;
		if (lane == 0)
			nodes[0] = make_int2(e, DecodeColor(int(best & 0xFFFF), shift, reverse));
	}
	__syncwarp();
	return res;
}

/* LevelsMinimum::EstimateChannelLevelsReduced (src/SnippetLevelsMinimum.h:117-311):
   the smallest e(c) over the window (or top), rows pruned by their cut-table
   lower bound.  The minimum does not depend on the visiting order; a batch
   ends after the first four values unless a lane is below the running best
   (of the batches of a precise encode one in six gets further). */
template<int kD>
__device__ NEBC7_SHARED int EstimateChannelLevels(const Area& ar, int offset, int weight, int water, int bits, bool transparent,
	const uint8_t* table, bool byDiff, const uint16_t* tower, int2* values, int lane)
{
	const AreaInfo& ai = ar.info;
	const int count = transparent ? ai.active : ai.count;
	if (transparent && !count)
		return 0;
	int top = (water + weight - 1) / weight;
	if (!top)
		return 0;
	const int L = int(int16_t(ai.minmax[2 * offset]));
	const int H = int(int16_t(ai.minmax[2 * offset + 1]));
	if (L == H)
		return 0;
	if (bits == 7 && H - L <= 5)
		return 0;
	if (bits == 8 && H - L <= 3)
		return 0;
	const Window win = MakeWindow(L, H, WindowRadius<kD>(top), bits, bits);
	if (top > 0xFFFF)
		top = 0xFFFF;
	const int n = DistinctValues(ar, count, offset, L, H, ValueStride(bits, byDiff), values, lane);
	ValueGroup first;
	first.Load(values);

	int best = top;
	for (int base = win.HL; base < win.HH; base += 32)
	{
		/* lane k holds the cut bound of row base + k */
		const int iHl = base + lane;
		unsigned bound = 0x7FFFFFFF;
		if (iHl < win.HH)
		{
			auto cut = [&](int e) { return unsigned(e & 0xFF) * tower[((e >> 8) << bits) + iHl]; };
			bound = 0;
			for (int u = 0; u < n; u += 4)
			{
				const int4 a = *reinterpret_cast<const int4*>(values + u), b = *reinterpret_cast<const int4*>(values + u + 2);
				bound += (cut(a.y) + cut(a.w)) + (cut(b.y) + cut(b.w));
			}
			bound = min(bound, 0xFFFFu);
		}
		/* the rows whose bound is below the best, in order */
		int next = 0;
		for (;;)
		{
			const unsigned open = __ballot_sync(kFull, lane >= next && int(bound) < best);
			if (!open)
				break;
			const int r = __ffs(open) - 1;
			next = r + 1;
			const int iH = base + r;
			const int cH = iH << bits;
			for (int iL = cH, hL = min(win.LH, iH) + cH; iL <= hL; iL += 32)
			{
				/* iL + lane stays in row iH (iL <= hL, iL - cH a multiple of 32) */
				int s;
				if (CandidateSum<false>(table + CandidateBase(iL + lane, bits, byDiff), first, values, n, true, best - 1, s))
					best = __reduce_min_sync(kFull, min(s, best));
			}
		}
	}
	return best * weight;
}

} // namespace nebc7
