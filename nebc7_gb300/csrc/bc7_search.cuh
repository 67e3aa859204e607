/*
 * BC7 block encoder for sm_103a -- refinement and full searches (the
 * reference's "normal" and "slow" passes, ModeN::CompressBlock and
 * ModeN::CompressBlockFull).
 *
 * The exhaustive search over per-channel candidate lists (the reference's
 * TryVariants) visits combinations in a fixed nested order and keeps each
 * one whose error is strictly below the running best ("water"), skipping
 * combinations by comparing bounds (a sorted channel error plus the other
 * channels' minima, or a memoised error over a subset of channels) with the
 * water.  Where those bounds are lower bounds of the error, the search ends
 * with the first combination, in its order, of the smallest error below the
 * water; SearchThree, SearchFour2 and SearchFour4 compute that, one warp or a
 * CTA's four.  Where masked pixels can make a bound exceed the error (modes 4
 * and 5), TryVariantsRot keeps the reference's order of tests: the outer loops
 * uniform and in order, the memoised errors of a loop level at once (lane =
 * list entry), the innermost channel's candidates in parallel and their
 * acceptances replayed in order.
 */
#pragma once

#include "bc7_fast.cuh"
#include "bc7_levels.cuh"
#include "bc7_pca.cuh"

namespace nebc7 {

constexpr bool kHasNormalPasses = true;


constexpr int kBig = 0x7FFFFFFF;

/* Above every error (16 pixels of weight 2000 at distance 127: 5.2e8), and
   still an int after another error is added. */
constexpr int kFar = 0x3FFFFFFF;

/* int4 entries per pixel of the candidate table: 20 candidates and one of
   padding, so that the pixels of a column lie in different banks. */
constexpr int kTableRow = 21;

/* The partitions of a three-subset search that its estimates leave. */
struct __align__(16) ThreeEstimates
{
	int2 order[64];      /* (estimate, partition) */
	int lines[64][2];    /* per partition, estimates of subsets 2 and 3 */
	int est[64][3][3];   /* per partition, subset, channel (G, R, B) estimates */
	int count;
};

/* Per-warp search state.  The staged kernels reserve only the bytes up to the
   last member their pass uses (SearchBytes), so that more of the SM's memory
   is L1. */
struct __align__(16) SearchState
{
	int2 values[16];         /* distinct channel values of the subset being scanned (DistinctValues) */
	ChanList chan[4][4];     /* [p-bit variant][channel]: the lists' minima and lengths */
	int bound[2][4];         /* [subset][channel]: lower-bound estimates of a two-subset search */
	int4 plane[4 * 16];      /* error planes of the combination search, [pixel][level]: three of
	                            4 levels or two of 8 */
	int2 lists[4][4][32];    /* [p-bit variant][channel][entry] = (error, color) */
	union
	{
		ThreeEstimates three;         /* the three-subset searches */
		int4 table[16 * kTableRow];   /* four channels, 2-bit indices: R's terms, [pixel][candidate] */
		int plane16[3][256];          /* four channels, 4-bit indices: planes of 16 levels */
	};
	struct
	{
		int2 order[64];
		int lines[64][2];
	} pca;                   /* OPTION_PCA: (estimate, partition), the subsets' bounds */
};

/* ---------------------------------------------------------------------- */
/* Partial error planes                                                   */
/*                                                                        */
/* For endpoints fixed on some channels, plane[i][k] holds the weighted   */
/* squared distances of pixel i to level k summed over those channels.    */
/* A candidate for one more channel then costs one channel per pixel and  */
/* level instead of all four; the sums are the same integers.             */
/* ---------------------------------------------------------------------- */

/* dst[i][k] = src[i][k] (0 without src) + w * q(x_i,c - v_k(col))^2 for the
   first np pixels of the area, L = 1 << IB levels. */
template<int kD, int IB>
__device__ __forceinline__ void PlaneAdd(int* dst, const int* src, const Area& ar, int np, int c, int col, int w, int lane)
{
	constexpr int L = 1 << IB;
	const int e0 = col & 0xFF, e1 = (col >> 8) & 0xFF;
	/* entry e = lane + 32 m has level e & (L - 1) = lane & (L - 1) */
	const int v = Interp(e0, e1, InterpWeights(IB)[lane & (L - 1)]);
	for (int e = lane; e < np * L; e += 32)
	{
		const int q = Q<kD>(int(ar.px[e >> IB][c]) - v);
		dst[e] = (src ? src[e] : 0) + w * q * q;
	}
	__syncwarp();
}

/* sum_i min_k (plane[i][k] + w * q(x_i,c - v_k(col))^2), stopping once the
   sum reaches `limit` (the same partial sums as the four-channel error). */
template<int kD, int IB>
__device__ __forceinline__ int PlaneError(const int* plane, const Area& ar, int np, int c, int col, int w, int limit)
{
	constexpr int L = 1 << IB;
	const int* wk = InterpWeights(IB);
	const int e0 = col & 0xFF, e1 = (col >> 8) & 0xFF;
	int v[L];
#pragma unroll
	for (int k = 0; k < L; k++)
		v[k] = Interp(e0, e1, wk[k]);
	int sum = 0;
	for (int i = 0; i < np; i++)
	{
		const int x = ar.px[i][c];
		const int4* row = reinterpret_cast<const int4*>(plane + i * L);
		int best = kBig;
#pragma unroll
		for (int k4 = 0; k4 < L / 4; k4++)
		{
			const int4 pv = row[k4];
			const int q0 = Q<kD>(x - v[4 * k4]), q1 = Q<kD>(x - v[4 * k4 + 1]);
			const int q2 = Q<kD>(x - v[4 * k4 + 2]), q3 = Q<kD>(x - v[4 * k4 + 3]);
			best = min(best, min(min(pv.x + w * q0 * q0, pv.y + w * q1 * q1), min(pv.z + w * q2 * q2, pv.w + w * q3 * q3)));
		}
		sum += best;
		if (!(limit > sum))
			break;
	}
	return sum;
}

/* ---------------------------------------------------------------------- */
/* Errors over an area, with early exit at `water` (only used to reject)   */
/* ---------------------------------------------------------------------- */

template<int kD, int BITS>
__device__ NEBC7_PASS int AreaError(const Area& ar, int active, Ep ep, const int w[4], int water)
{
	LevelSet<BITS> Lv;
	Lv.Init(ep);
	int sum = 0;
	for (int i = 0; i < active; i++)
	{
		const int p0 = ar.px[i][0], p1 = ar.px[i][1], p2 = ar.px[i][2], p3 = ar.px[i][3];
		int best = kBig;
#pragma unroll
		for (int k = 0; k < (1 << BITS); k++)
		{
			const int q0 = Q<kD>(p0 - Lv.v[k][0]), q1 = Q<kD>(p1 - Lv.v[k][1]);
			const int q2 = Q<kD>(p2 - Lv.v[k][2]), q3 = Q<kD>(p3 - Lv.v[k][3]);
			best = min(best, w[0] * q0 * q0 + w[1] * q1 * q1 + w[2] * q2 * q2 + w[3] * q3 * q3);
		}
		sum += best;
		if (!(water > sum))
			break;
	}
	return sum;
}

/* Mode 4/5 error on Area1 (see RotErrorExact) with early exit. */
template<int kD, int CB, int AB, bool MODE4>
__device__ __noinline__ int RotErrorW(const Area& ar, const AreaInfo& ai, Ep epImg, int rotation, const int w[4], int water)
{
	const int a = RotChannel(rotation);
	LevelSet<CB> LC;
	LevelSet<AB> LA;
	LC.Init(epImg);
	LA.Init(epImg);
	int sum = 0;
	const int n = MODE4 ? ai.active : 16;
	for (int i = 0; i < n; i++)
	{
		int px[4], mk[4];
#pragma unroll
		for (int c = 0; c < 4; c++)
		{
			px[c] = ar.px[i][c];
			mk[c] = ar.mk[i][c];
		}
		int bestc = kBig;
#pragma unroll
		for (int k = 0; k < (1 << CB); k++)
		{
			int e = 0;
#pragma unroll
			for (int c = 0; c < 4; c++)
			{
				const int q = Q<kD>(px[c] - LC.v[k][c]);
				e += (c == a) ? 0 : w[c] * ((q * q) & mk[c]);
			}
			bestc = min(bestc, e);
		}
		int besta = kBig;
#pragma unroll
		for (int k = 0; k < (1 << AB); k++)
		{
			int e = 0;
#pragma unroll
			for (int c = 0; c < 4; c++)
			{
				const int q = Q<kD>(px[c] - LA.v[k][c]);
				e += (c == a) ? w[c] * ((q * q) & mk[c]) : 0;
			}
			besta = min(besta, e);
		}
		sum += besta;
		sum += bestc;
		if (!(water > sum))
			return sum;
	}
	if (MODE4 && ai.active < 16)
	{
		const int m = min(EpGet(epImg, 0), EpGet(epImg, 1));
		const int q = Q<kD>(m);
		sum += q * q * (w[0] * (16 - ai.active));
	}
	return sum;
}

__device__ __forceinline__ Ep Ep2(int c0, int col0, int c1, int col1)
{
	return EpSetCh(EpSetCh(0, c0, col0), c1, col1);
}

/* The innermost loop of a combination search, replayed in the reference's
   order.  Lane j holds candidate j of the innermost (sorted) list: `brk` is
   its sorted bound (the loop ends at the first lane with brk >= water),
   `skip` its memoised bound (the lane is passed over when skip >= water) and
   `err` its error, computed with an early exit at the water in force when
   the loop started (exact whenever below it).  A lane is accepted when, at
   the running water, it is the first later lane with all three below the
   water; the water then drops to its error.  With arbitrary pixel masks the
   bounds are not always lower bounds of the error, so the order matters.
   Returns the last accepted lane or -1. */
__device__ __forceinline__ int ReplayInner(bool valid, int brk, int skip, int err, int& water, int lane)
{
	int taken = -1;
	for (;;)
	{
		const unsigned m = __ballot_sync(kFull, valid && lane > taken && brk < water && skip < water && err < water);
		if (!m)
			break;
		taken = __ffs(m) - 1;
		water = __shfl_sync(kFull, err, taken);
	}
	return taken;
}

/* The channel weights by value: an argument of the out-of-line searches
   that stays in registers. */
struct Weights
{
	int a, g, r, b;
};

__device__ __forceinline__ Weights WeightsOf(const Params& P)
{
	return Weights{ P.wA, P.wG, P.wR, P.wB };
}

/* A search's outcome: the water it leaves and the endpoints that reached it. */
struct Found
{
	int water;
	Ep best;
};

/* min over four levels of a plane row plus a candidate's terms; each step is
   one fused add-and-minimum. */
__device__ __forceinline__ int RowMin(int4 p, int4 t)
{
	return __viaddmin_s32(p.x, t.x, __viaddmin_s32(p.y, t.y, __viaddmin_s32(p.z, t.z, p.w + t.w)));
}

/* w * q(x - level)^2 at the four levels of the endpoint pair `col`. */
template<int kD>
__device__ __forceinline__ int4 LevelTerms(int x, int col, int w)
{
	const int e0 = col & 0xFF, e1 = (col >> 8) & 0xFF;
	const int q0 = Q<kD>(x - e0), q1 = Q<kD>(x - Interp(e0, e1, 21)), q2 = Q<kD>(x - Interp(e0, e1, 43)), q3 = Q<kD>(x - e1);
	return make_int4(w * q0 * q0, w * q1 * q1, w * q2 * q2, w * q3 * q3);
}

/* A lane's candidate terms per pixel and level, kept in registers: the
   weighted squares with four levels, the plain squares two to a register
   with eight (at most 127^2 each). */
template<int kD, int IB>
struct LaneTerms
{
	int4 t[16];

	/* x: the pixel values of the searched channel; rows from np on are zero */
	__device__ __forceinline__ void Init(const Area& ar, int np, int c, int col, int w)
	{
		const int e0 = col & 0xFF, e1 = (col >> 8) & 0xFF;
		int v[8];
		if (IB == 3)
		{
#pragma unroll
			for (int k = 0; k < 8; k++)
				v[k] = Interp(e0, e1, c_interp3[k]);
		}
#pragma unroll
		for (int i = 0; i < 16; i++)
		{
			t[i] = make_int4(0, 0, 0, 0);
			if (i < np)
			{
				const int x = ar.px[i][c];
				if (IB == 2)
					t[i] = LevelTerms<kD>(x, col, w);
				else
				{
					int q[8];
#pragma unroll
					for (int k = 0; k < 8; k++)
						q[k] = Q<kD>(x - v[k]);
					t[i] = make_int4(q[0] * q[0] + ((q[1] * q[1]) << 16), q[2] * q[2] + ((q[3] * q[3]) << 16),
						q[4] * q[4] + ((q[5] * q[5]) << 16), q[6] * q[6] + ((q[7] * q[7]) << 16));
				}
			}
		}
	}

	/* Error of the lane's candidate over a plane of np pixels (rows up to the
	   next multiple of four are zero).  Ends once no lane is below its limit,
	   so a lane's value is exact whenever it is below it.  Warp-collective:
	   every lane calls it. */
	__device__ __forceinline__ int Error(const int4* plane, int np, int w, int limit) const
	{
		int sum = 0;
#pragma unroll
		for (int i = 0; i < 16; i += 4)
		{
			if (i >= np)
				break;
#pragma unroll
			for (int j = i; j < i + 4; j++)
			{
				if (IB == 2)
					sum += RowMin(plane[j], t[j]);
				else
				{
					const int4 a = plane[2 * j], b = plane[2 * j + 1];
					auto two = [&](int p0, int p1, int q) { return min(p0 + w * (q & 0xFFFF), p1 + w * int(unsigned(q) >> 16)); };
					sum += min(min(two(a.x, a.y, t[j].x), two(a.z, a.w, t[j].y)), min(two(b.x, b.y, t[j].z), two(b.z, b.w, t[j].w)));
				}
			}
			if (!__any_sync(kFull, sum < limit))
				break;
		}
		return sum;
	}
};

constexpr int kNoLimit = int(0x80000000u);   /* the limit of a lane without a candidate */

/* The entries of a [pixel][level] plane that a lane holds: pixel
   lane / L + (32 / L) m, level lane % L. */
template<int kD, int IB>
struct PlaneLanes
{
	static constexpr int L = 1 << IB, N = L / 2;
	int wk, row, np;

	__device__ __forceinline__ PlaneLanes(int np_, int lane) : wk(InterpWeights(IB)[lane & (L - 1)]), row(lane >> IB), np(np_) {}

	__device__ __forceinline__ void Pixels(const Area& ar, int c, int (&x)[N]) const
	{
#pragma unroll
		for (int m = 0; m < N; m++)
			x[m] = row + (32 / L) * m < np ? int(ar.px[row + (32 / L) * m][c]) : 0;
	}

	/* dst = src + the terms of the endpoint pair `col` */
	__device__ __forceinline__ void Add(int (&dst)[N], const int (&src)[N], const int (&x)[N], int col, int w) const
	{
		const int v = Interp(col & 0xFF, (col >> 8) & 0xFF, wk);
#pragma unroll
		for (int m = 0; m < N; m++)
		{
			const int q = Q<kD>(x[m] - v);
			dst[m] = row + (32 / L) * m < np ? src[m] + w * q * q : 0;
		}
	}

	__device__ __forceinline__ void Load(int (&e)[N], const int4* plane, int lane) const
	{
		const int* p = reinterpret_cast<const int*>(plane);
#pragma unroll
		for (int m = 0; m < N; m++)
			e[m] = (32 / L) * m < np ? p[lane + 32 * m] : 0;
	}

	__device__ __forceinline__ void Store2(int4* plane, const int (&e)[N], int4* plane2, const int (&f)[N], int lane) const
	{
		int* p = reinterpret_cast<int*>(plane);
		int* q = reinterpret_cast<int*>(plane2);
#pragma unroll
		for (int m = 0; m < N; m++)
			if ((32 / L) * m < np)
			{
				p[lane + 32 * m] = e[m];
				q[lane + 32 * m] = f[m];
			}
		__syncwarp();
	}

	__device__ __forceinline__ void Store(int4* plane, const int (&e)[N], int lane) const
	{
		int* p = reinterpret_cast<int*>(plane);
#pragma unroll
		for (int m = 0; m < N; m++)
			if ((32 / L) * m < np)
				p[lane + 32 * m] = e[m];
		__syncwarp();
	}
};

/* ---------------------------------------------------------------------- */
/* Three channels with one index (src/Bc7CoreMode0.cpp:242-415; modes 4, 5) */
/* ---------------------------------------------------------------------- */

/* What the warps of a team share of one combination search: the smallest
   error found so far with its place in the search's order (error << 32 |
   variant, four list indices; three channels use the last three), and the next unit of each variant. */
struct TeamSearch
{
	unsigned long long key;
	int next[4];
};

/* Place of a combination in the search's order. */
__device__ __forceinline__ unsigned SearchPlace(int v, int i0, int i1, int i2, int i3)
{
	return unsigned(((((v << 5 | i0) << 5 | i1) << 5 | i2) << 5) | i3);
}

/* What a team shares of a block's search. */
struct TeamState
{
	TeamSearch search;
	TeamExchange exchange;
	int bound[2][4];       /* [subset][channel] estimates */
	int valid;             /* variants whose lists leave room */
	int task[4];           /* the CTA's tasks: queue position, first candidate, first improvement, how many */
	int open[4];           /* which of them are open */
};

/* Starts a team's search from `water`; the last one's outcome is read. */
__device__ __forceinline__ void StartTeamSearch(TeamState& ts, int water)
{
	__syncthreads();
	if (threadIdx.x == 0)
	{
		ts.search.key = (unsigned long long)(unsigned(water)) << 32;
		ts.search.next[0] = ts.search.next[1] = ts.search.next[2] = ts.search.next[3] = 0;
		ts.valid = 0;
	}
	__syncthreads();
}

/* One channel's sorted candidate list in a search: its pixels' channel, its
   weight, and the list. */
struct SearchChannel
{
	int c, w;
	const int2* list;
	int n, minErr;
};

/* A three-channel search's outcome; taken: an improving combination's
   endpoint colours are in x, y, z. */
struct Found3
{
	int water;
	int taken, x, y, z;
};

/* The combination search over three channels that share an index.  As in
   SearchFour2, every bound is a lower bound, so the sequential search ends
   with the first combination, in its order, of the smallest error below the
   water.  z's candidates are the lanes, their terms in registers; y's errors
   are summed once per x candidate.  hidden: the pixels that count only with
   their alpha of 0 (x is then the alpha channel). */
template<int kD, int IB>
__device__ NEBC7_SHARED Found3 SearchThree(const Area& ar, int np, SearchChannel X, SearchChannel Y, SearchChannel Z, int hidden,
	int water, int4* planes, const Team& team, TeamState* ts, int lane)
{
	Found3 f{ water, 0, 0, 0, 0 };
	const bool shared = team.size > 1;
	if (shared)
		StartTeamSearch(*ts, water);
	if (X.minErr + Y.minErr + Z.minErr >= water)
		return f;
	const int2 ly = lane < Y.n ? Y.list[lane] : make_int2(kFar, 0);
	const int2 lz = lane < Z.n ? Z.list[lane] : make_int2(kFar, 0);
	int4* const pX = planes;
	int4* const pXY = planes + 4 * (1 << IB);
	LaneTerms<kD, IB> terms;
	int sums = 0;   /* error sums of z's candidates so far */
	using Lanes = PlaneLanes<kD, IB>;
	const Lanes pl(np, lane);
	int xx[Lanes::N], xy[Lanes::N], gx[Lanes::N], gy[Lanes::N];
	pl.Pixels(ar, X.c, xx);
	pl.Pixels(ar, Y.c, xy);
	const int none[Lanes::N] = {};
	/* the error that a combination at (ix, iy) has to be below (SearchFour2) */
	auto refresh = [&](int ix, int iy) {
		if (shared)
		{
			const unsigned long long k = *reinterpret_cast<volatile unsigned long long*>(&ts->search.key);
			water = int(k >> 32) + int(unsigned(k) > SearchPlace(0, 0, ix, iy, 31));
		}
	};
	for (int ix = 0;; ix++)
	{
		if (shared)
		{
			int u = 0;
			if (lane == 0)
				u = atomicAdd(&ts->search.next[0], 1);
			ix = __shfl_sync(kFull, u, 0);
		}
		if (ix >= X.n)
			break;
		refresh(ix, 0);
		const int2 lx = X.list[ix];
		if (lx.x + Y.minErr + Z.minErr >= water)
			break;
		int ea = 0;
		if (hidden)
		{
			const int q = Q<kD>(min(lx.y & 0xFF, (lx.y >> 8) & 0xFF));
			ea = q * q * (X.w * hidden);
		}
		pl.Add(gx, none, xx, lx.y, X.w);
		__syncwarp();
		pl.Store(pX, gx, lane);
		/* joint errors of this x candidate with every y one */
		int errXY = kFar;
		if (lane < Y.n)
			errXY = PlaneError<kD, IB>(reinterpret_cast<const int*>(pX), ar, np, Y.c, ly.y, Y.w, water - ea - Z.minErr) + ea;
		/* the first pass sums x's plane with every z candidate (errXZ), the
		   others take the y candidates still open */
		int errXZ = 0, iy = -1;
		for (;;)
		{
			const unsigned open = __ballot_sync(kFull, lane > iy && ly.x + lx.x + Z.minErr < water && errXY + Z.minErr < water);
			if (!open)
				break;
			const bool first = iy < 0 && errXZ == 0;
			int2 y = make_int2(0, 0);
			bool eval = lane < Z.n;
			const int4* plane = pX;
			int limit = water - ea - Y.minErr;
			if (!first)
			{
				iy = __ffs(open) - 1;
				refresh(ix, iy);
				const int eXY = __shfl_sync(kFull, errXY, iy);
				y = make_int2(__shfl_sync(kFull, ly.x, iy), __shfl_sync(kFull, ly.y, iy));
				eval = lz.x + eXY < water && errXZ - 1 + y.x < water;
				if (!__any_sync(kFull, eval))
					continue;
				pl.Add(gy, gx, xy, y.y, Y.w);
				pl.Store(pXY, gy, lane);
				plane = pXY;
				limit = water - ea;
			}
			/* the terms in registers pay from the third sum on */
			if (sums == 2)
				terms.Init(ar, np, Z.c, lz.y, Z.w);
			int sum = 0;
			if (sums >= 2)
				sum = terms.Error(plane, np, Z.w, eval ? limit : kNoLimit);
			else if (eval)
				sum = PlaneError<kD, IB>(reinterpret_cast<const int*>(plane), ar, np, Z.c, lz.y, Z.w, limit);
			sums++;
			const int err = eval ? sum + ea : kFar;
			if (first)
			{
				/* 1 + the error: never 0, so that the first pass runs once */
				errXZ = err + 1;
				continue;
			}
			/* the first lane of the smallest error below the water */
			const int low = __reduce_min_sync(kFull, err);
			if (low < water)
			{
				const int j = __ffs(__ballot_sync(kFull, err == low)) - 1;
				water = low;
				if (!shared)
				{
					f.taken = 1;
					f.x = lx.y;
					f.y = y.y;
					f.z = __shfl_sync(kFull, lz.y, j);
				}
				else if (lane == 0)
					atomicMin(&ts->search.key, (unsigned long long)(unsigned(low)) << 32 | SearchPlace(0, 0, ix, iy, j));
			}
		}
	}
	if (shared)
	{
		__syncthreads();
		const unsigned long long k = ts->search.key;
		const unsigned place = unsigned(k);
		water = int(k >> 32);
		f.taken = water < f.water;
		f.x = X.list[(place >> 10) & 31].y;
		f.y = Y.list[(place >> 5) & 31].y;
		f.z = Z.list[place & 31].y;
	}
	f.water = water;
	return f;
}

/* Candidate lists and estimates of the opaque modes: table by differences
   (DiffBase), except mode 1's shared-p-bit table, which marks endpoint pairs
   of different parity (0xFF; its estimates read them) and stays in the per-x
   layout. */
struct Spec3
{
	int bits;               /* candidate list bits */
	const uint8_t* table;
	bool byDiff;
	int estBits;
	const uint16_t* estTower;
	int variants;           /* p-bit variants */
};

__device__ __forceinline__ Spec3 GetSpec3(int mode, const LevelTables& T)
{
	if (mode == 0)
		return Spec3{ 4, T.d3v8, true, 5, T.c3v5, 4 };
	if (mode == 1)
		return Spec3{ 6, T.d3v7s, false, 7, T.c3v7s, 2 };
	if (mode == 2)
		return Spec3{ 5, T.d2v8, true, 5, T.c2v5, 1 };
	return Spec3{ 7, T.d2v8, true, 8, T.c2v8, 4 };
}

/* p-bit variant v in the reference's order 0x0101, 0, 1, 1 << 8 (low byte:
   the low endpoint's). */
__device__ __forceinline__ int VariantPbits(int v)
{
	return v == 0 ? 0x0101 : (v == 1 ? 0 : (v == 2 ? 1 : 1 << 8));
}

__device__ __forceinline__ int ChannelWeight(const Params& P, int c)
{
	return c == 0 ? P.wA : (c == 1 ? P.wG : (c == 2 ? P.wR : P.wB));
}

/* The passes below keep one call site of each scan, estimate and combination
   search, in loops over the subsets, variants and channels: inlined, a
   kernel holds one copy of each and no call saves registers on the thread's
   stack (a precise mode-2 search spent more loads on its stack than on the
   tables, with 14 % of them hits). */

/* Subset::InitLevels (src/Bc7CoreMode0.cpp:249-268) for variant v; estR,
   estB: lower bounds of the later channels' errors. */
template<int kD>
__device__ NEBC7_PASS bool InitLevels3(SearchState& ss, int v, const Area& ar, const Params& P, const Spec3& sp, bool pbit, int water,
	int estR, int estB, Team& team, int lane)
{
	int used = 0;
#pragma unroll 1
	for (int c = 1; c < 4; c++)
	{
		const int rest = c == 1 ? estR + estB : (c == 2 ? estB : 0);
		const ChanList cl = ChannelLevels<kD, false>(ss.lists[v][c - 1], ar, c, ChannelWeight(P, c), water - used - rest, sp.bits,
			pbit ? VariantPbits(v) : -1, false, sp.table, sp.byDiff, 32, ss.values, team, lane);
		if (lane == 0)
			ss.chan[v][c - 1] = cl;
		used += cl.minErr;
		if (used >= water)
			return false;
	}
	__syncwarp();
	return true;
}

/* Subsets (src/Bc7CoreMode0.cpp:366-415): all variants' lists start from
   the same water, then the variants are searched in order. */
template<int kD, int MODE>
__device__ NEBC7_PASS int SearchSubset3(SearchState& ss, const Area& ar, const Params& P, const Spec3& sp, int water, int estR, int estB,
	Ep& best, bool& any, Team& team, TeamState* ts, int lane)
{
	constexpr int IB = (MODE == 0 || MODE == 1) ? 3 : 2;
	int valid = 0;
#pragma unroll 1
	for (int v = 0; v < sp.variants; v++)
		valid |= int(InitLevels3<kD>(ss, v, ar, P, sp, MODE != 2, water, estR, estB, team, lane)) << v;
	any = valid != 0;
#pragma unroll 1
	for (int v = 0; v < sp.variants; v++)
	{
		if (!((valid >> v) & 1))
			continue;
		auto channel = [&](int c, int w) { return SearchChannel{ c, w, ss.lists[v][c - 1], ss.chan[v][c - 1].count, ss.chan[v][c - 1].minErr }; };
		const Found3 f = SearchThree<kD, IB>(ar, ar.info.active, channel(1, P.wG), channel(2, P.wR), channel(3, P.wB), 0, water,
			ss.plane, team, ts, lane);
		water = f.water;
		if (f.taken)
			best = EpSetCh(Ep2(1, f.x, 2, f.y), 3, f.z);
	}
	return water;
}

/* Subset s of partition p into `ar` (its pixels and ar.info); `orient` as
   for SubsetStats. */
template<int kD>
__device__ NEBC7_PASS void BuildSubset(WarpState& st, const CellRegs& R, const Params& P, Area& ar, int ns, int p, int s, bool orient,
	int lane)
{
	const uint32_t part = ns == 3 ? c_part3[p] : c_part2[p];
	const uint32_t member = Member(part, s);
	const int anchor = Anchor(ns, p, s);
	SubsetStats(ar.info, st, R, P, member, anchor, orient, lane);
	BuildAreaList(ar, st, R, member, anchor, lane);
}

/* ModeN::CompressBlock for modes 0-3 (src/Bc7CoreMode0.cpp:417-498). */
template<int kD, int MODE>
__device__ NEBC7_PASS void RefineOpaque(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const LevelTables& T, Team& team,
	TeamState* ts, int lane)
{
	constexpr int NS = (MODE == 0 || MODE == 2) ? 3 : 2;
	constexpr int IB = (MODE == 0 || MODE == 1) ? 3 : 2;
	const Spec3 sp = GetSpec3(MODE, T);
	const int wGRB[4] = { 0, P.wG, P.wR, P.wB };
	Ep mc0 = R.best[0], mc1 = R.best[1], mc2 = R.best[2];
	int error = R.opaqueAlphaError;
	if (error < R.errTotal)
	{
#pragma unroll 1
		for (int s = 0; s < NS; s++)
		{
			BuildSubset<kD>(st, R, P, st.sub[0], NS, R.bestParam, s, true, lane);
			Ep b = s == 0 ? mc0 : (s == 1 ? mc1 : mc2);
			int water = AreaError<kD, IB>(st.sub[0], st.sub[0].info.active, b, wGRB, MaxColorError<kD>());
			if (water)
			{
				bool any;
				const int w2 = SearchSubset3<kD, MODE>(ss, st.sub[0], P, sp, water, 0, 0, b, any, team, ts, lane);
				if (any)
				{
					water = w2;
					if (s == 0)
						mc0 = b;
					else if (s == 1)
						mc1 = b;
					else
						mc2 = b;
				}
				error += water;
			}
		}
		if (R.errTotal > error)
		{
			R.errTotal = error;
			R.best[0] = mc0;
			R.best[1] = mc1;
			if (NS == 3)
				R.best[2] = mc2;
		}
	}
}

/* EstimateLevels of modes 0-3 (src/Bc7CoreMode0.cpp:500-530): est[0..2] get
   the estimates of G, R, B. */
template<int kD>
__device__ NEBC7_PASS int EstimateLevels3(SearchState& ss, const Area& ar, const Params& P, const Spec3& sp, int water, int* est, int lane)
{
	int error = 0;
#pragma unroll 1
	for (int c = 1; c < 4; c++)
	{
		if (!(error < water))
			return water;
		const int l = EstimateChannelLevels<kD>(ar, c, ChannelWeight(P, c), water - error, sp.estBits, false, sp.table, sp.byDiff,
			sp.estTower, ss.values, lane);
		if (lane == 0)
			est[c - 1] = l;
		error += l;
	}
	__syncwarp();
	return error < water ? error : water;
}

__device__ __forceinline__ void StableSortOrder(int2* order, int n, int lane)
{
	/* stable sort by unsigned error (src/Bc7Core.cpp:564 radix_sort_partitions)
	   of entries that the reference lists in ascending partition order:
	   rank = number of entries that must precede */
	int2 mine[2];
	int rank[2];
#pragma unroll
	for (int h = 0; h < 2; h++)
	{
		const int i = lane + 32 * h;
		rank[h] = -1;
		mine[h] = make_int2(0, 0);
		if (i < n)
		{
			mine[h] = order[i];
			int r = 0;
			for (int k = 0; k < n; k++)
			{
				const int2 o = order[k];
				r += (unsigned(o.x) < unsigned(mine[h].x)) || (o.x == mine[h].x && o.y < mine[h].y);
			}
			rank[h] = r;
		}
	}
	__syncwarp();
#pragma unroll
	for (int h = 0; h < 2; h++)
		if (rank[h] >= 0)
			order[rank[h]] = mine[h];
	__syncwarp();
}

/* ---------------------------------------------------------------------- */
/* A bound of every endpoint pair at once                                  */
/* ---------------------------------------------------------------------- */

/* The channels of a bound: their weights' roots (zero outside), the sum and
   the least of the weights. */
struct LineWeights
{
	float root[4], sum;
	int least;
};

__device__ __forceinline__ LineWeights LineWeightsOf(const Params& P, unsigned channels)
{
	LineWeights lw;
	lw.sum = 0.0f;
	lw.least = 0x7FFFFFFF;
#pragma unroll
	for (int c = 0; c < 4; c++)
	{
		const int w = (channels >> c) & 1 ? ChannelWeight(P, c) : 0;
		lw.root[c] = sqrtf(float(w));
		lw.sum += float(w);
		if ((channels >> c) & 1)
			lw.least = min(lw.least, w);
	}
	return lw;
}

/* Sums of pixels' values and products (the upper triangle) over the channels
   FIRST..3. */
template<int FIRST>
struct Moments
{
	int n, sum[4], xy[4][4];
};

/* A lower bound of the error of the pixels of `mo` in one subset, whatever its
   endpoints and indices: the levels of a subset lie on a line of color space
   but for their rounding, and no line comes closer to the pixels than their
   principal axis.
 *
 * With weighted channels (x_c sqrt(w_c)) the squared distances to the best line
 * sum to trace - l, l the largest eigenvalue of the scatter matrix M, and
 * l^4 <= |M^4| (Frobenius).  An interpolated level is at most 1/2 from the
 * line in each channel, and 2 |d >> 1| at most 1 from |d| (kD 1), so the root
 * of the error falls short of the root of that sum by at most
 * (1/2 or 3/2) sqrt(n sum(w)); with kD 0 a difference past 127 counts as 127,
 * and such a candidate's error is at least 127^2 of the least weight.  The
 * moments are exact (n sum(x y) < 2^24); the factors next to 1 cover the float
 * arithmetic on them, about 1e-6.
 *
 * It ends most partitions of mode 7 before their scans (1118x1105 alpha texture,
 * default: 45.1 -> 13.4 ms of the pass; 1700x940: 1013 -> 173 ms of the call),
 * a quarter of the time of mode 1's.  The three-subset and rotation searches go
 * without: their blocks' errors are near the rounding slack, and the bound cost
 * more than it saved (precise 1024x1024 photo 40.1 -> 47.6 ms). */
template<int kD, int FIRST>
__device__ __forceinline__ int LineBoundOf(const Moments<FIRST>& mo, const LineWeights& lw)
{
	const float n = float(mo.n);
	float m[4][4], trace = 0.0f;
#pragma unroll
	for (int c = FIRST; c < 4; c++)
#pragma unroll
		for (int d = c; d < 4; d++)
		{
			m[c][d] = m[d][c] = float(mo.n * mo.xy[c][d] - mo.sum[c] * mo.sum[d]) * (lw.root[c] * lw.root[d]);
			if (c == d)
				trace += m[c][c];
		}
	if (mo.n < 3 || !(trace > 0.0f))
		return 0;   /* two pixels lie on a line */
	const float scale = 1.0f / trace;
#pragma unroll
	for (int c = FIRST; c < 4; c++)
#pragma unroll
		for (int d = FIRST; d < 4; d++)
			m[c][d] *= scale;
	float norm = 0.0f;
#pragma unroll
	for (int step = 0; step < 2; step++)
	{
		float q[4][4];
		norm = 0.0f;
#pragma unroll
		for (int c = FIRST; c < 4; c++)
#pragma unroll
			for (int d = c; d < 4; d++)
			{
				float t = 0.0f;
#pragma unroll
				for (int k = FIRST; k < 4; k++)
					t += m[c][k] * m[k][d];
				q[c][d] = q[d][c] = t;
				norm += c == d ? t * t : 2.0f * t * t;
			}
#pragma unroll
		for (int c = FIRST; c < 4; c++)
#pragma unroll
			for (int d = FIRST; d < 4; d++)
				m[c][d] = q[c][d];
	}
	/* |M^4| = sqrt(norm); its fourth root, of a trace of 1 */
	const float top = sqrtf(sqrtf(sqrtf(norm))) * 1.00001f + 0.00001f;
	const float off = trace / n * fmaxf(1.0f - top, 0.0f) * 0.99999f;
	const float root = fmaxf(sqrtf(off) - (kD ? 1.5f : 0.5f) * 1.00001f * sqrtf(n * lw.sum), 0.0f);
	const int b = int(fminf(root * root * (kD ? 0.25f : 1.0f) * 0.9999f, 1.0e9f));
	return kD ? b : min(b, lw.least * 127 * 127);
}

/* LineBoundOf for the first np pixels of an area.  Warp-collective. */
template<int kD, int FIRST>
__device__ __forceinline__ int LineBound(const Area& ar, int np, const LineWeights& lw, int lane)
{
	Moments<FIRST> mo;
	mo.n = np;
	int x[4];
#pragma unroll
	for (int c = FIRST; c < 4; c++)
	{
		x[c] = lane < np ? int(ar.px[lane][c]) : 0;
		mo.sum[c] = int(__reduce_add_sync(kFull, unsigned(x[c])));
	}
#pragma unroll
	for (int c = FIRST; c < 4; c++)
#pragma unroll
		for (int d = c; d < 4; d++)
			mo.xy[c][d] = int(__reduce_add_sync(kFull, unsigned(x[c] * x[d])));
	return LineBoundOf<kD, FIRST>(mo, lw);
}

/* The estimates of partition p of a full search of modes 0 and 2 (the first
   loop of src/Bc7CoreMode0.cpp:532-642): its subsets' estimates to out.three,
   and whether they leave room below the error. */
template<int kD, int MODE>
__device__ __forceinline__ bool ThreeSubsetsEstimate(WarpState& st, SearchState& ss, SearchState& out, const CellRegs& R, const Params& P,
	const Spec3& sp, int p, int& total, int lane)
{
	int water = R.errTotal - R.denoiseStep - R.opaqueAlphaError;
	total = R.opaqueAlphaError + R.denoiseStep;
#pragma unroll 1
	for (int s = 0; s < 3; s++)
	{
		BuildSubset<kD>(st, R, P, st.sub[0], 3, p, s, false, lane);
		const int line = EstimateLevels3<kD>(ss, st.sub[0], P, sp, water, out.three.est[p][s], lane);
		if (!(line < water))
			return false;
		if (lane == 0 && s)
			out.three.lines[p][s - 1] = line;
		water -= line;
		total += line;
	}
	return true;
}

/* The search of partition p from its estimates (the second loop); returns
   whether it ends the full search. */
template<int kD, int MODE>
__device__ __forceinline__ bool ThreeSubsetsPartition(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const Spec3& sp, int p,
	int lane)
{
	Ep mc0 = 0, mc1 = 0, mc2 = 0;
	int error = R.opaqueAlphaError;
	Team one = SingleWarp();
#pragma unroll 1
	for (int s = 0; s < 3; s++)
	{
		const int rest = s == 0 ? ss.three.lines[p][0] + ss.three.lines[p][1] : (s == 1 ? ss.three.lines[p][1] : 0);
		const int water = R.errTotal - R.denoiseStep - error - rest;
		BuildSubset<kD>(st, R, P, st.sub[0], 3, p, s, true, lane);
		bool any;
		Ep b = 0;
		const int r = SearchSubset3<kD, MODE>(ss, st.sub[0], P, sp, water, ss.three.est[p][s][1], ss.three.est[p][s][2], b, any, one, nullptr, lane);
		if (!any || !(r < water))
			return false;
		error += r;
		if (s == 0)
			mc0 = b;
		else if (s == 1)
			mc1 = b;
		else
			mc2 = b;
	}
	R.errTotal = error;
	R.best[0] = mc0;
	R.best[1] = mc1;
	R.best[2] = mc2;
	R.bestParam = p;
	R.bestMode = MODE;
	return error <= R.opaqueAlphaError;
}

/* The estimates of a full search of modes 0 and 2 (the first loop of
   src/Bc7CoreMode0.cpp:532-642, src/Bc7CoreMode2.cpp:456-566), sorted, in
   ss.three of the team's first warp.  A team's warps take every size-th
   partition (all estimates are from the block's error, whatever the order);
   their states are `stateStride` bytes apart. */
template<int kD, int MODE>
__device__ __forceinline__ void ThreeSubsetsEstimates(WarpState& st, SearchState& ss, const CellRegs& R, const Params& P, const Spec3& sp,
	const Team& team, size_t stateStride, int lane)
{
	constexpr int NP = MODE == 0 ? 16 : 64;
	SearchState& s0 = *reinterpret_cast<SearchState*>(reinterpret_cast<unsigned char*>(&ss) - team.rank * stateStride);
	if (team.rank == 0 && lane == 0)
		s0.three.count = 0;
	team.Sync();
#pragma unroll 1
	for (int p = team.rank; p < NP; p += team.size)
	{
		if (R.personalMode == MODE && R.personalParam == p)
			continue;
		int total;
		if (ThreeSubsetsEstimate<kD, MODE>(st, ss, s0, R, P, sp, p, total, lane) && lane == 0)
			s0.three.order[atomicAdd(&s0.three.count, 1)] = make_int2(total, p);
	}
	team.Sync();
	if (team.rank == 0)
		StableSortOrder(ss.three.order, ss.three.count, lane);
}

/* Full searches of modes 0 and 2. */
template<int kD, int MODE>
__device__ NEBC7_PASS void FullThreeSubsets(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const LevelTables& T, int lane)
{
	const Spec3 sp = GetSpec3(MODE, T);
	ThreeSubsetsEstimates<kD, MODE>(st, ss, R, P, sp, SingleWarp(), 0, lane);
	const int count = ss.three.count;
#pragma unroll 1
	for (int i = 0; i < count; i++)
	{
		const int2 o = ss.three.order[i];
		if (o.x < R.errTotal && ThreeSubsetsPartition<kD, MODE>(st, ss, R, P, sp, o.y, lane))
			return;
	}
}

/* The partition search of modes 1 and 3 from its estimates (the second
   loop of src/Bc7CoreMode1.cpp:473-571, src/Bc7CoreMode3.cpp:471-569):
   partition p with the principal-axis bounds line0, line1 (0 without
   OPTION_PCA).  Returns true when the search ends the full pass. */
template<int kD, int MODE>
__device__ __forceinline__ bool TwoSubsetsPartition(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const Spec3& sp, int p,
	int line0, int line1, int lane)
{
	const int room = R.errTotal - R.denoiseStep - R.opaqueAlphaError;
	const LineWeights lw = LineWeightsOf(P, 14);
	int low[2] = { 0, 0 };
#pragma unroll 1
	for (int s = 0; s < 2; s++)
	{
		BuildSubset<kD>(st, R, P, st.sub[s], 2, p, s, true, lane);
		low[0] = low[1];
		low[1] = LineBound<kD, 1>(st.sub[s], st.sub[s].info.active, lw, lane);
	}
	if (low[0] + low[1] >= room)
		return false;
#pragma unroll 1
	for (int s = 0; s < 2; s++)
	{
		const int water = room - line1 - (s == 0 ? 0 : line0);
		const int line = EstimateLevels3<kD>(ss, st.sub[s], P, sp, water, ss.bound[s], lane);
		if (s == 0)
			line0 = max(line0, line);
		else
			line1 = max(line1, line);
		if (!((s == 0 ? line0 : line1) < water))
			return false;
	}
	/* OPTION_PCA's bounds may exceed the errors: then only the reference's
	   own tests use them */
	if (!P.pca && max(line0, low[0]) + max(line1, low[1]) >= room)
		return false;
	Team one = SingleWarp();
	Ep mc0 = 0, mc1 = 0;
	int error = 0;
#pragma unroll 1
	for (int s = 0; s < 2; s++)
	{
		const int water = room - (s == 0 ? line1 : error);
		bool any;
		Ep b = 0;
		const int r = SearchSubset3<kD, MODE>(ss, st.sub[s], P, sp, water, ss.bound[s][1], ss.bound[s][2], b, any, one, nullptr, lane);
		if (!any || !(r < water))
			return false;
		error += r;
		if (s == 0 && error + low[1] >= room)
			return false;
		if (s == 0)
			mc0 = b;
		else
			mc1 = b;
	}
	R.errTotal = error + R.opaqueAlphaError;
	R.best[0] = mc0;
	R.best[1] = mc1;
	R.bestParam = p;
	R.bestMode = MODE;
	return error <= 0;
}

/* The partitions' principal-axis bounds and their order (AreaGetBestPca3,
   src/Bc7Core.cpp:494; EstimateBest, src/Bc7CoreMode7.cpp:559-572): ss.pca
   lists the partitions whose bounds leave room.  OPTION_PCA only. */
template<int kD, int MODE>
__device__ __noinline__ int PcaPartitions(WarpState& st, SearchState& ss, const CellRegs& R, const Params& P, int base, int lane)
{
	int count = 0;
#pragma unroll 1
	for (int p = 0; p < 64; p++)
	{
		if (R.personalMode == MODE && R.personalParam == p)
			continue;
		int water = R.errTotal - R.denoiseStep - base, total = base + R.denoiseStep;
		bool room = true;
#pragma unroll 1
		for (int s = 0; s < 2 && room; s++)
		{
			BuildSubset<kD>(st, R, P, st.sub[s], 2, p, s, true, lane);
			const int line = PcaBound<kD>(st.sub[s], st.sub[s].info, P, MODE == 7 && !st.sub[s].info.opaque ? 4 : 3, lane);
			room = line < water;
			water -= line;
			total += line;
			if (lane == 0)
				ss.pca.lines[p][s] = line;
		}
		if (room)
		{
			if (lane == 0)
				ss.pca.order[count] = make_int2(total, p);
			count++;
		}
	}
	__syncwarp();
	StableSortOrder(ss.pca.order, count, lane);
	return count;
}

/* Full searches of modes 1 and 3 (src/Bc7CoreMode1.cpp:473-571,
   src/Bc7CoreMode3.cpp:471-569).  Without OPTION_PCA every partition's
   bound is zero, so every partition enters with estimate OA + step and the
   stable sort keeps index order; with it, the partitions are estimated and
   sorted first.  Without OPTION_PCA the search may resume at partition
   `from` (the partitions before it searched already, R as they left it). */
template<int kD, int MODE>
__device__ NEBC7_PASS void FullTwoSubsets(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const LevelTables& T, int lane,
	int from = 0)
{
	const Spec3 sp = GetSpec3(MODE, T);
	const int count = P.pca ? PcaPartitions<kD, MODE>(st, ss, R, P, R.opaqueAlphaError, lane) : 64;
#pragma unroll 1
	for (int i = P.pca ? 0 : from; i < count; i++)
	{
		int p = i, line0 = 0, line1 = 0, estimate = R.opaqueAlphaError + R.denoiseStep;
		if (P.pca)
		{
			estimate = ss.pca.order[i].x;
			p = ss.pca.order[i].y;
			line0 = ss.pca.lines[p][0];
			line1 = ss.pca.lines[p][1];
		}
		else if (R.personalMode == MODE && R.personalParam == p)
			continue;
		if (estimate < R.errTotal && TwoSubsetsPartition<kD, MODE>(st, ss, R, P, sp, p, line0, line1, lane))
			return;
	}
}

/* ---------------------------------------------------------------------- */
/* Modes 6, 6Index2, 7: four channels with the transparent-alpha term       */
/* ---------------------------------------------------------------------- */

/* The four-channel combination search with 2-bit indices (modes 7 and
   6Index2; src/Bc7CoreMode6.cpp:1163-1331) over the lists of variant v.
 *
 * Every bound that the reference compares here is a lower bound of the error
 * it stands for: a channel's list error takes each pixel's nearest level on
 * its own, over the same pixels and with the same transparent-alpha term as
 * the joint error, and a joint error over fewer channels drops non-negative
 * terms.  So the sequential search ends with the first combination, in its
 * order, of the smallest error below the water, and any lower bound may
 * skip: besides the reference's, the sums below take the entry's own list
 * error where the reference takes the list's minimum, and a level's errors
 * are computed only when some combination under it is still open.  For the
 * same reason the warps of a team may take the alpha candidates (an opaque
 * area's single one: every fourth G candidate) in any order: the smallest
 * (error, place) wins, and a warp keeps a combination of the team's error
 * that lies before the team's.
 *
 * What bounds it: instruction issue in the error sums.  A candidate's terms
 * w q^2 per pixel and level do not depend on the outer loops, so B's are kept
 * in the lane's registers (lane = candidate) and R's in a shared-memory
 * table, and a pixel costs one broadcast read of the plane and four fused
 * add-minimum steps instead of four differences, squares and products.  Two
 * G candidates at a time share a pass over R's table, and an alpha
 * candidate's R and G sums one over its plane: the sums are chains of shared
 * loads, and two in flight hide each other's latency (mode 7 pass of a
 * 1118x1105 alpha texture: 47.2 -> 45.1 ms). */
template<int kD>
__device__ __forceinline__ Found SearchFour2(SearchState& ss, const ChanList (&chan)[4], const int2 (*lists)[32], int v, const Area& ar, int count,
	int np, bool opq, Weights w, const uint8_t* alphaTable, Ep best, int water, TeamSearch* team, int lane)
{
	const int4 m01 = *reinterpret_cast<const int4*>(&chan[0]), m23 = *reinterpret_cast<const int4*>(&chan[2]);
	const int min0 = m01.x, n0 = m01.y, min1 = m01.z, n1 = m01.w;
	const int min2 = m23.x, n2 = m23.y, min3 = m23.z, n3 = m23.w;
	if (min0 + min1 + min2 + min3 >= water)
		return Found{ water, best };
	const int2 l1 = lane < n1 ? lists[1][lane] : make_int2(kFar, 0);
	const int2 l2 = lane < n2 ? lists[2][lane] : make_int2(kFar, 0);
	const int2 l3 = lane < n3 ? lists[3][lane] : make_int2(kFar, 0);
	int4* const pA = ss.plane;
	int4* const pAG = (ss.plane + 16);
	int4* const pAGR = (ss.plane + 32);
	const int at = lane < kTableRow - 1 ? lane : kTableRow - 1;

	/* R's table, B's registers */
	LaneTerms<kD, 2> termsB;
	termsB.Init(ar, np, 3, l3.y, w.b);
	if (lane < kTableRow)
		for (int i = 0; i < ((np + 3) & ~3); i++)
			ss.table[i * kTableRow + lane] = i < np ? LevelTerms<kD>(int(ar.px[i][2]), l2.y, w.r) : make_int4(0, 0, 0, 0);
	const PlaneLanes<kD, 2> pl(np, lane);
	int xa[2], xg[2], ga[2], gg[2], gr[2];
	pl.Pixels(ar, 0, xa);
	pl.Pixels(ar, 1, xg);
	const int zero[2] = { 0, 0 };
	/* a team's units: the alpha candidates, or the four stripes of an opaque
	   area's G candidates */
	const int stripes = team && opq ? 4 : 1;

	/* the error that a combination at (i0, i1) has to be below: one above the
	   team's where the team's combination lies behind it */
	auto refresh = [&](int i0, int i1) {
		if (team)
		{
			const unsigned long long k = *reinterpret_cast<volatile unsigned long long*>(&team->key);
			water = int(k >> 32) + int(unsigned(k) > SearchPlace(v, i0, i1, 31, 31));
		}
	};

	for (int unit = 0;; unit++)
	{
		if (team)
		{
			int u = 0;
			if (lane == 0)
				u = atomicAdd(&team->next[v], 1);
			unit = __shfl_sync(kFull, u, 0);
		}
		if (unit >= n0 * stripes)
			break;
		const int i0 = team && opq ? 0 : unit;
		refresh(i0, 0);
		const int2 a = lists[0][i0];
		const int e0 = a.x;
		if (e0 + min1 + min2 + min3 >= water)
			break;
		int ea = (count - np) * w.a;
		if (count > np)
		{
			const int d = DiffAt(alphaTable, 0, a.y & 0xFF, (a.y >> 8) & 0xFF);
			ea *= d * d;
		}
		pl.Add(ga, zero, xa, a.y, w.a);
		__syncwarp();
		pl.Store(pA, ga, lane);
		/* joint errors of this alpha candidate with every R and every G one
		   (an opaque area's alpha term is zero: the list errors are they) */
		int errAR = l2.x + e0, errAG = l1.x + e0;
		if (!opq)
		{
			/* both in one pass over the plane */
			const int limitR = lane < n2 ? water - ea - min1 - min3 : kNoLimit, limitG = lane < n1 ? water - ea - min2 - min3 : kNoLimit;
			int sumR = 0, sumG = 0;
			for (int i = 0; i < np; i += 2)
			{
#pragma unroll
				for (int j = i; j < i + 2; j++)
				{
					const int4 row = pA[j];
					sumR += RowMin(row, ss.table[j * kTableRow + at]);
					sumG += j < np ? RowMin(row, LevelTerms<kD>(int(ar.px[j][1]), l1.y, w.g)) : 0;
				}
				if (!__any_sync(kFull, sumR < limitR || sumG < limitG))
					break;
			}
			errAR = lane < n2 ? sumR + ea : kFar;
			errAG = lane < n1 ? sumG + ea : kFar;
		}
		const bool mine = stripes == 1 || (lane & 3) == unit;
		int i1 = 0;
		for (;;)
		{
			/* the next G candidate still open */
			const unsigned open1 = __ballot_sync(kFull, lane >= i1 && mine && l1.x + e0 + min2 + min3 < water && errAG + min2 + min3 < water);
			if (!open1)
				break;
			/* two of them at a time: a pass over R's table serves both */
			const int first = __ffs(open1) - 1, more = int(open1 & (open1 - 1));
			const int second = more ? __ffs(more) - 1 : first;
			i1 = second + 1;
			refresh(i0, first);
			const int colG[2] = { __shfl_sync(kFull, l1.y, first), __shfl_sync(kFull, l1.y, second) };
			int errAGR[2];
			{
				const int eAG0 = __shfl_sync(kFull, errAG, first), eAG1 = __shfl_sync(kFull, errAG, second);
				const int eG0 = __shfl_sync(kFull, l1.x, first), eG1 = __shfl_sync(kFull, l1.x, second);
				const bool openR0 = l2.x + eAG0 + min3 < water && errAR + eG0 + min3 < water;
				const bool openR1 = more && l2.x + eAG1 + min3 < water && errAR + eG1 + min3 < water;
				if (!__any_sync(kFull, openR0 || openR1))
					continue;
				pl.Add(gg, ga, xg, colG[0], w.g);
				pl.Add(gr, ga, xg, colG[1], w.g);
				pl.Store2(pAG, gg, pAG + 32, gr, lane);
				const int limit0 = openR0 ? water - ea - min3 : kNoLimit, limit1 = openR1 ? water - ea - min3 : kNoLimit;
				int sum0 = 0, sum1 = 0;
				for (int i = 0; i < np; i += 2)
				{
#pragma unroll
					for (int j = i; j < i + 2; j++)
					{
						const int4 t = ss.table[j * kTableRow + at];
						sum0 += RowMin(pAG[j], t);
						sum1 += RowMin(pAG[j + 32], t);
					}
					if (!__any_sync(kFull, sum0 < limit0 || sum1 < limit1))
						break;
				}
				errAGR[0] = openR0 ? sum0 + ea : kFar;
				errAGR[1] = openR1 ? sum1 + ea : kFar;
			}
#pragma unroll 1
			for (int h = 0; h < 2; h++)
			{
				const int place1 = h ? second : first;
				const int errR = h ? errAGR[1] : errAGR[0];
				if (h)
					refresh(i0, place1);
				unsigned open2 = __ballot_sync(kFull, errR + min3 < water);
				if (!open2)
					continue;
				const int4* const plane = pAG + 32 * h;
				const int eAG = __shfl_sync(kFull, errAG, place1);
				const bool openB = l3.x + eAG + min2 < water;
				const int sumB = termsB.Error(plane, np, w.b, openB ? water - ea - min2 : kNoLimit);
				const int errAGB = openB ? sumB + ea : kFar;
				pl.Load(gg, plane, lane);
				while (open2)
				{
					const int i2 = __ffs(open2) - 1;
					open2 &= open2 - 1;
					const int e2 = __shfl_sync(kFull, errR, i2);
					const int2 r = make_int2(__shfl_sync(kFull, l2.x, i2), __shfl_sync(kFull, l2.y, i2));
					const bool eval = l3.x + e2 < water && errAGB + r.x < water;
					if (!__any_sync(kFull, eval))
						continue;
					const int* t = reinterpret_cast<const int*>(ss.table) + (pl.row * kTableRow + i2) * 4 + (lane & 3);
					gr[0] = pl.row < np ? gg[0] + t[0] : 0;
					gr[1] = pl.row + 8 < np ? gg[1] + t[8 * kTableRow * 4] : 0;
					pl.Store(pAGR, gr, lane);
					const int sum = termsB.Error(pAGR, np, w.b, eval ? water - ea : kNoLimit);
					const int err = eval ? sum + ea : kFar;
					/* the first lane of the smallest error below the water */
					const int low = __reduce_min_sync(kFull, err);
					if (low < water)
					{
						const int j = __ffs(__ballot_sync(kFull, err == low)) - 1;
						water = low;
						if (!team)
							best = EpSetCh(EpSetCh(Ep2(0, a.y, 1, h ? colG[1] : colG[0]), 2, r.y), 3, __shfl_sync(kFull, l3.y, j));
						else if (lane == 0)
							atomicMin(&team->key, (unsigned long long)(unsigned(low)) << 32 | SearchPlace(v, i0, place1, i2, j));
					}
				}
			}
		}
	}
	return Found{ water, best };
}

/* The same search with 4-bit indices (mode 6): sixteen levels a pixel do not
   fit registers or a table, so a candidate's terms are computed per plane. */
template<int kD>
__device__ __forceinline__ Found SearchFour4(SearchState& ss, int v, const Area& ar, int count, int np, bool opq, Weights w,
	const uint8_t* alphaTable, Ep best, int water, TeamSearch* team, int lane)
{
	const int4 m01 = *reinterpret_cast<const int4*>(&ss.chan[v][0]), m23 = *reinterpret_cast<const int4*>(&ss.chan[v][2]);
	const int min0 = m01.x, n0 = m01.y, min1 = m01.z, n1 = m01.w;
	const int min2 = m23.x, n2 = m23.y, min3 = m23.z, n3 = m23.w;
	if (min0 + min1 + min2 + min3 >= water)
		return Found{ water, best };
	const int2 l1 = lane < n1 ? ss.lists[v][1][lane] : make_int2(kFar, 0);
	const int2 l2 = lane < n2 ? ss.lists[v][2][lane] : make_int2(kFar, 0);
	const int2 l3 = lane < n3 ? ss.lists[v][3][lane] : make_int2(kFar, 0);
	int* const pA = ss.plane16[0];
	int* const pAG = ss.plane16[1];
	int* const pAGR = ss.plane16[2];
	const int stripes = team && opq ? 4 : 1;
	auto refresh = [&](int i0, int i1) {
		if (team)
		{
			const unsigned long long k = *reinterpret_cast<volatile unsigned long long*>(&team->key);
			water = int(k >> 32) + int(unsigned(k) > SearchPlace(0, i0, i1, 31, 31));
		}
	};
	for (int unit = 0;; unit++)
	{
		if (team)
		{
			int u = 0;
			if (lane == 0)
				u = atomicAdd(&team->next[0], 1);
			unit = __shfl_sync(kFull, u, 0);
		}
		if (unit >= n0 * stripes)
			break;
		const int i0 = team && opq ? 0 : unit;
		refresh(i0, 0);
		const int2 a = ss.lists[v][0][i0];
		const int e0 = a.x;
		if (e0 + min1 + min2 + min3 >= water)
			break;
		int ea = (count - np) * w.a;
		if (count > np)
		{
			const int d = HalfAt(alphaTable, 0, a.y & 0xFF, (a.y >> 8) & 0xFF);
			ea *= d * d;
		}
		PlaneAdd<kD, 4>(pA, nullptr, ar, np, 0, a.y, w.a, lane);
		int errAR = l2.x + e0, errAG = l1.x + e0;
		if (!opq)
		{
			if (lane < n2)
				errAR = PlaneError<kD, 4>(pA, ar, np, 2, l2.y, w.r, water - ea - min1 - min3) + ea;
			if (lane < n1)
				errAG = PlaneError<kD, 4>(pA, ar, np, 1, l1.y, w.g, water - ea - min2 - min3) + ea;
		}
		const bool mine = stripes == 1 || (lane & 3) == unit;
		int i1 = 0;
		for (;;)
		{
			const unsigned open1 = __ballot_sync(kFull, lane >= i1 && mine && l1.x + e0 + min2 + min3 < water && errAG + min2 + min3 < water);
			if (!open1)
				break;
			i1 = __ffs(open1) - 1;
			refresh(i0, i1);
			const int place1 = i1;
			const int eAG = __shfl_sync(kFull, errAG, i1);
			const int2 g = make_int2(__shfl_sync(kFull, l1.x, i1), __shfl_sync(kFull, l1.y, i1));
			i1++;
			const bool openR = l2.x + eAG + min3 < water && errAR + g.x + min3 < water;
			if (!__any_sync(kFull, openR))
				continue;
			PlaneAdd<kD, 4>(pAG, pA, ar, np, 1, g.y, w.g, lane);
			int errAGR = kFar, errAGB = kFar;
			if (openR)
				errAGR = PlaneError<kD, 4>(pAG, ar, np, 2, l2.y, w.r, water - ea - min3) + ea;
			unsigned open2 = __ballot_sync(kFull, errAGR + min3 < water);
			if (!open2)
				continue;
			if (l3.x + eAG + min2 < water)
				errAGB = PlaneError<kD, 4>(pAG, ar, np, 3, l3.y, w.b, water - ea - min2) + ea;
			while (open2)
			{
				const int i2 = __ffs(open2) - 1;
				open2 &= open2 - 1;
				const int e2 = __shfl_sync(kFull, errAGR, i2);
				const int2 r = make_int2(__shfl_sync(kFull, l2.x, i2), __shfl_sync(kFull, l2.y, i2));
				const bool eval = l3.x + e2 < water && errAGB + r.x < water;
				if (!__any_sync(kFull, eval))
					continue;
				PlaneAdd<kD, 4>(pAGR, pAG, ar, np, 2, r.y, w.r, lane);
				int err = kFar;
				if (eval)
					err = PlaneError<kD, 4>(pAGR, ar, np, 3, l3.y, w.b, water - ea) + ea;
				const int low = __reduce_min_sync(kFull, err);
				if (low < water)
				{
					const int j = __ffs(__ballot_sync(kFull, err == low)) - 1;
					water = low;
					if (!team)
						best = EpSetCh(EpSetCh(Ep2(0, a.y, 1, g.y), 2, r.y), 3, __shfl_sync(kFull, l3.y, j));
					else if (lane == 0)
						atomicMin(&team->key, (unsigned long long)(unsigned(low)) << 32 | SearchPlace(0, i0, place1, i2, j));
				}
			}
		}
	}
	return Found{ water, best };
}

/* The search of index width IB over the lists of slot `slot`: with 4-bit indices
   those of `ss`, with 2-bit ones those of `from` (a team's other warp's). */
template<int kD, int IB>
__device__ NEBC7_SHARED Found SearchFour(SearchState& ss, const SearchState& from, int slot, int v, const Area& ar, Weights w, const uint8_t* alphaTable,
	Ep best, int water, TeamSearch* team, int lane)
{
	const AreaInfo& ai = ar.info;
	if constexpr (IB == 4)
		return SearchFour4<kD>(ss, slot, ar, ai.count, ai.active, ai.opaque, w, alphaTable, best, water, team, lane);
	else
		return SearchFour2<kD>(ss, from.chan[slot], from.lists[slot], v, ar, ai.count, ai.active, ai.opaque, w, alphaTable, best, water, team,
			lane);
}

/* The endpoints of a team's outcome in the lists it was found in. */
__device__ __forceinline__ Ep PlaceEndpoints(const int2 (*lists)[32], unsigned place)
{
	return EpSetCh(EpSetCh(Ep2(0, lists[0][(place >> 15) & 31].y, 1, lists[1][(place >> 10) & 31].y), 2, lists[2][(place >> 5) & 31].y), 3,
		lists[3][place & 31].y);
}

/* Subset::InitLevels of modes 6 / 6Index2 (9) / 7 (src/Bc7CoreMode6.cpp:
   1130-1161, src/Bc7CoreMode7.cpp:237-268) for the p-bits of variant pv into
   the lists of slot v; est: lower bounds of the channels' errors, or null.
   Every warp of a team gets the whole lists. */
template<int kD, int MODE>
__device__ NEBC7_PASS bool InitLevels4(SearchState& ss, int v, int pv, const Area& ar, const Params& P, const LevelTables& T, int water,
	const int* est, Team& team, int lane)
{
	int used = 0;
	int rest = est ? est[1] + est[2] + est[3] : 0;
#pragma unroll 1
	for (int c = 0; c < 4; c++)
	{
		ChanList cl;
		if (c == 0 && ar.info.opaque)
			cl = ZeroList(ss.lists[v][0], 0xFFFF, lane);
		else
			cl = ChannelLevels<kD, MODE != 7>(ss.lists[v][c], ar, c, ChannelWeight(P, c), water - used - rest, MODE == 7 ? 5 : 7,
				VariantPbits(pv), c != 0, MODE == 6 ? T.h4s : (MODE == 9 ? T.h2s : T.d2v8), true, 20, ss.values, team, lane);
		if (lane == 0)
			ss.chan[v][c] = cl;
		used += cl.minErr;
		if (used >= water)
			return false;
		if (est && c < 3)
			rest -= est[c + 1];
	}
	__syncwarp();
	return true;
}

/* Mode 6 / 6Index2 CompressSubset (src/Bc7CoreMode6.cpp:1334-1364): each
   later p-bit variant starts from the water left by the earlier ones. */
template<int kD, int MODE>
__device__ NEBC7_PASS int CompressSubsetSingle(SearchState& ss, const Area& ar, const Params& P, const LevelTables& T, Ep& mc, int water,
	Team& team, TeamState* ts, int lane)
{
#pragma unroll 1
	for (int v = 0; v < (ar.info.opaque ? 1 : 4); v++)
	{
		if (!InitLevels4<kD, MODE>(ss, 0, v, ar, P, T, water, nullptr, team, lane))
			continue;
		if (team.size > 1)
			StartTeamSearch(*ts, water);
		const Found f = SearchFour<kD, MODE == 6 ? 4 : 2>(ss, ss, 0, 0, ar, WeightsOf(P), MODE == 6 ? T.d4h : T.d2v8, mc,
			team.size > 1 ? water + 1 : water, team.size > 1 ? &ts->search : nullptr, lane);
		if (team.size > 1)
		{
			__syncthreads();
			const unsigned long long k = ts->search.key;
			if (int(k >> 32) < water)
			{
				water = int(k >> 32);
				mc = PlaceEndpoints(ss.lists[0], unsigned(k));
			}
		}
		else
		{
			water = f.water;
			mc = f.best;
		}
	}
	return water;
}

/* Mode 7 Subsets (src/Bc7CoreMode7.cpp:441-494): all variants' lists start
   from the same water.  A team's warps make a variant's lists each, in slot 0
   of their own state (`stateStride` bytes apart), then take each other's alpha
   candidates. */
template<int kD>
__device__ NEBC7_PASS int SearchSubset7(SearchState& ss, const Area& ar, const Params& P, const LevelTables& T, int water, const int* est,
	Ep& best, bool& any, Team& team, TeamState* ts, size_t stateStride, int lane)
{
	const int nv = ar.info.opaque ? 1 : 4;
	const bool shared = team.size > 1;
	if (shared)
		StartTeamSearch(*ts, water);
	Team one = SingleWarp();
	int valid = 0;
#pragma unroll 1
	for (int v = team.rank; v < nv; v += team.size)
		valid |= int(InitLevels4<kD, 7>(ss, shared ? 0 : v, v, ar, P, T, water, est, one, lane)) << v;
	if (shared)
	{
		if (lane == 0 && valid)
			atomicOr(&ts->valid, valid);
		__syncthreads();
		valid = ts->valid;
	}
	any = valid != 0;
	if (!any)
		return water;
	const unsigned char* const first = reinterpret_cast<const unsigned char*>(&ss) - team.rank * stateStride;
#pragma unroll 1
	for (int dv = 0; dv < nv; dv++)
	{
		/* a team's warp takes its own variant first, then the others' units */
		const int v = (team.rank + dv) & (nv - 1);
		if (!((valid >> v) & 1))
			continue;
		const SearchState& sv = shared ? *reinterpret_cast<const SearchState*>(first + v * stateStride) : ss;
		const int slot = shared ? 0 : v;
		int limit = water;
		if (shared)
		{
			if (*reinterpret_cast<volatile int*>(&ts->search.next[v]) >= sv.chan[0][0].count * (ar.info.opaque ? 4 : 1))
				continue;
			limit = int(*reinterpret_cast<volatile unsigned long long*>(&ts->search.key) >> 32) + 1;
		}
		const Found f = SearchFour<kD, 2>(ss, sv, slot, v, ar, WeightsOf(P), T.d2v8, best, limit, shared ? &ts->search : nullptr, lane);
		if (!shared)
		{
			water = f.water;
			best = f.best;
		}
	}
	if (shared)
	{
		__syncthreads();
		const unsigned long long k = ts->search.key;
		if (int(k >> 32) < water)
		{
			water = int(k >> 32);
			best = PlaceEndpoints(reinterpret_cast<const SearchState*>(first + (unsigned(k) >> 20) * stateStride)->lists[0], unsigned(k));
		}
	}
	return water;
}

template<int kD, int MODE>
__device__ NEBC7_PASS void RefineMode6(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const LevelTables& T, Team& team,
	TeamState* ts, int lane)
{
	/* src/Bc7CoreMode6.cpp:1366-1381 */
	Ep mc = R.best[0];
	const int error = CompressSubsetSingle<kD, MODE>(ss, st.area1, P, T, mc, R.errTotal, team, ts, lane);
	if (R.errTotal > error)
	{
		R.errTotal = error;
		R.best[0] = mc;
	}
}

template<int kD>
__device__ NEBC7_PASS void FullMode6(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const LevelTables& T, Team& team,
	TeamState* ts, int lane)
{
	/* src/Bc7CoreMode6.cpp:1398-1422 */
	if (R.personalMode == 6)
		return;
	const int step = R.denoiseStep;
	/* EstimateBest (src/Bc7CoreMode6.cpp:1383-1396): 0 without OPTION_PCA */
	const int line = P.pca ? PcaBound<kD>(st.area1, R.a1, P, R.a1.opaque ? 3 : 4, lane) : 0;
	if (line < R.errTotal - step && LineBound<kD, 0>(st.area1, st.area1.info.active, LineWeightsOf(P, 15), lane) < R.errTotal - step)
	{
		Ep mc = 0;
		const int error = CompressSubsetSingle<kD, 6>(ss, st.area1, P, T, mc, R.errTotal - step, team, ts, lane);
		if (R.errTotal > error + step)
		{
			R.errTotal = error;
			R.best[0] = mc;
			R.bestMode = 6;
		}
	}
}

template<int kD>
__device__ NEBC7_PASS void RefineMode7(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const LevelTables& T, Team& team,
	TeamState* ts, size_t stateStride, int lane)
{
	/* src/Bc7CoreMode7.cpp:496-557 */
	Ep mc0 = R.best[0], mc1 = R.best[1];
	const int w[4] = { P.wA, P.wG, P.wR, P.wB };
	int error = 0;
#pragma unroll 1
	for (int s = 0; s < 2; s++)
	{
		Area& ar = st.sub[0];
		BuildSubset<kD>(st, R, P, ar, 2, R.bestParam, s, true, lane);
		Ep b = s == 0 ? mc0 : mc1;
		int water = AreaError<kD, 2>(ar, ar.info.active, b, w, 2 * MaxColorError<kD>());
		water += TransparentError2(T, P, ar.info.count, ar.info.active, int(b & 0xFFFF));
		if (water)
		{
			bool any;
			const int r = SearchSubset7<kD>(ss, ar, P, T, water, nullptr, b, any, team, ts, stateStride, lane);
			if (any)
			{
				water = r;
				if (s == 0)
					mc0 = b;
				else
					mc1 = b;
			}
			error += water;
		}
	}
	if (R.errTotal > error)
	{
		R.errTotal = error;
		R.best[0] = mc0;
		R.best[1] = mc1;
	}
}

/* EstimateLevels of mode 7 (src/Bc7CoreMode7.cpp:574-627): est[0..3] get the
   estimates of A, G, R, B. */
template<int kD>
__device__ NEBC7_PASS int EstimateLevels7(SearchState& ss, const Area& ar, const Params& P, const LevelTables& T, int water, int* est,
	int lane)
{
	if (!(0 < water))
		return water;
	if (!ar.info.active)
	{
		__syncwarp();
		if (lane < 4)
			est[lane] = 0;
		__syncwarp();
		return 0;
	}
	int error = 0;
#pragma unroll 1
	for (int c = 0; c < 4; c++)
	{
		if (!(error < water))
			return water;
		int l = 0;
		if (c || !ar.info.opaque)
			l = EstimateChannelLevels<kD>(ar, c, ChannelWeight(P, c), water - error, 6, c != 0, T.d2v8, true, T.c2v6, ss.values, lane);
		if (lane == 0)
			est[c] = l;
		error += l;
	}
	__syncwarp();
	return error < water ? error : water;
}

/* The partition search of mode 7 from its estimates (the second loop of
   src/Bc7CoreMode7.cpp:629-725): partition p with the principal-axis bounds
   line0, line1 (0 without OPTION_PCA).  Returns true when the search ends
   the full pass. */
template<int kD>
__device__ __forceinline__ bool Mode7Partition(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const LevelTables& T,
	int p, int line0, int line1, int lane)
{
	const int room = R.errTotal - R.denoiseStep;
	const LineWeights lw = LineWeightsOf(P, 15);
	int low[2] = { 0, 0 };
#pragma unroll 1
	for (int s = 0; s < 2; s++)
	{
		BuildSubset<kD>(st, R, P, st.sub[s], 2, p, s, true, lane);
		low[0] = low[1];
		low[1] = LineBound<kD, 0>(st.sub[s], st.sub[s].info.active, lw, lane);
	}
	if (low[0] + low[1] >= room)
		return false;
#pragma unroll 1
	for (int s = 0; s < 2; s++)
	{
		const int water = room - line1 - (s == 0 ? 0 : line0);
		const int line = EstimateLevels7<kD>(ss, st.sub[s], P, T, water, ss.bound[s], lane);
		if (s == 0)
			line0 = max(line0, line);
		else
			line1 = max(line1, line);
		if (!((s == 0 ? line0 : line1) < water))
			return false;
	}
	Ep mc0 = 0, mc1 = 0;
	int error = 0;
	Team one = SingleWarp();
#pragma unroll 1
	for (int s = 0; s < 2; s++)
	{
		const int water = room - (s == 0 ? line1 : error);
		bool any;
		Ep b = 0;
		const int r = SearchSubset7<kD>(ss, st.sub[s], P, T, water, ss.bound[s], b, any, one, nullptr, 0, lane);
		if (!any || !(r < water))
			return false;
		error += r;
		if (s == 0)
			mc0 = b;
		else
			mc1 = b;
	}
	R.errTotal = error;
	R.best[0] = mc0;
	R.best[1] = mc1;
	R.bestParam = p;
	R.bestMode = 7;
	return error <= 0;
}

/* Whether the line bounds of partition p's subsets leave room for mode 7. */
template<int kD>
__device__ __forceinline__ bool Mode7Open(WarpState& st, const CellRegs& R, const Params& P, int p, int lane)
{
	const LineWeights lw = LineWeightsOf(P, 15);
	int low = 0;
#pragma unroll 1
	for (int s = 0; s < 2; s++)
	{
		BuildSubset<kD>(st, R, P, st.sub[s], 2, p, s, true, lane);
		low += LineBound<kD, 0>(st.sub[s], st.sub[s].info.active, lw, lane);
	}
	return low < R.errTotal - R.denoiseStep;
}

/* Mode7Partition by the CTA's four warps: the four channels' estimates, the
   four p-bit variants' lists and the alpha candidates of the searches are
   theirs; each warp keeps the block and its subsets in its own state.
   The estimates take the subset's whole water where the reference takes what
   the earlier channels leave: an estimate below that rest is the same (a
   candidate below it lies in both windows), and one that is not ends the
   subset either way.  A hard partition of an alpha block takes a team 2 to
   4 ms, a warp alone three to four times as long. */
template<int kD>
__device__ __forceinline__ bool Mode7PartitionTeam(WarpState& st, SearchState& ss, TeamState& ts, size_t stateStride, CellRegs& R, const Params& P,
	const LevelTables& T, int p, int rank, int lane)
{
	Team team{ 4, rank, &ts.exchange, 0 };
	const int room = R.errTotal - R.denoiseStep;
	const LineWeights lw = LineWeightsOf(P, 15);
	int line1 = 0, used = 0, low[2];
#pragma unroll 1
	for (int s = 0; s < 2; s++)
	{
		BuildSubset<kD>(st, R, P, st.sub[s], 2, p, s, true, lane);
		const int b = LineBound<kD, 0>(st.sub[s], st.sub[s].info.active, lw, lane);
		low[1] = b;
		if (s == 0)
			low[0] = b;
	}
	if (low[0] + low[1] >= room)
		return false;
#pragma unroll 1
	for (int s = 0; s < 2; s++)
	{
		const Area& ar = st.sub[s];
		const int water = room - used;
		int l = 0;
		if (ar.info.active && (rank || !ar.info.opaque) && water > 0)
			l = EstimateChannelLevels<kD>(ar, rank, ChannelWeight(P, rank), water, 6, rank != 0, T.d2v8, true, T.c2v6, ss.values, lane);
		if (lane == 0)
			ts.bound[s][rank] = l;
		team.Sync();
		int error = 0;
#pragma unroll
		for (int c = 0; c < 4; c++)
			error = error < water ? error + ts.bound[s][c] : error;
		if (!(error < water))
			return false;
		used += error;
		line1 = error;
		if (s == 0 ? max(error, low[0]) + low[1] >= room : max(used - error, low[0]) + max(error, low[1]) >= room)
			return false;
	}
	Ep mc0 = 0, mc1 = 0;
	int error = 0;
#pragma unroll 1
	for (int s = 0; s < 2; s++)
	{
		const int water = room - (s == 0 ? line1 : error);
		bool any;
		Ep b = 0;
		const int r = SearchSubset7<kD>(ss, st.sub[s], P, T, water, ts.bound[s], b, any, team, &ts, stateStride, lane);
		if (!any || !(r < water))
			return false;
		error += r;
		if (s == 0 && error + low[1] >= room)
			return false;
		if (s == 0)
			mc0 = b;
		else
			mc1 = b;
	}
	R.errTotal = error;
	R.best[0] = mc0;
	R.best[1] = mc1;
	R.bestParam = p;
	R.bestMode = 7;
	return error <= 0;
}

template<int kD>
__device__ NEBC7_PASS void FullMode7(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const LevelTables& T, int lane,
	int from = 0)
{
	/* src/Bc7CoreMode7.cpp:629-725; without OPTION_PCA every partition enters
	   with estimate step (ties keep index order), and the search may resume
	   at partition `from` */
	const int count = P.pca ? PcaPartitions<kD, 7>(st, ss, R, P, 0, lane) : 64;
#pragma unroll 1
	for (int i = P.pca ? 0 : from; i < count; i++)
	{
		int p = i, line0 = 0, line1 = 0, estimate = R.denoiseStep;
		if (P.pca)
		{
			estimate = ss.pca.order[i].x;
			p = ss.pca.order[i].y;
			line0 = ss.pca.lines[p][0];
			line1 = ss.pca.lines[p][1];
		}
		else if (R.personalMode == 7 && R.personalParam == p)
			continue;
		if (estimate < R.errTotal && Mode7Partition<kD>(st, ss, R, P, T, p, line0, line1, lane))
			return;
	}
}

/* ---------------------------------------------------------------------- */
/* Modes 4 and 5: rotation, separate color / alpha-slot indices            */
/* ---------------------------------------------------------------------- */

template<int kD, int MODE, int CB, int AB>
__device__ __noinline__ int TryVariantsRot(const Area& ar, const AreaInfo& ai, const Params& P, const SearchState& ss, Ep& bestStorage,
	int water, int rot, int lane)
{
	const ChanList (&cl)[4] = ss.chan[0];
	const int minA = cl[0].minErr, minG = cl[1].minErr, minR = cl[2].minErr, minB = cl[3].minErr;
	if (minA + minG + minR + minB >= water)
		return water;
	const int nA = (rot == 0) ? 1 : cl[0].count;
	const int nG = (rot == 2) ? 1 : cl[1].count;
	const int nR = (rot == 1) ? 1 : cl[2].count;
	const int nB = (rot == 3) ? 1 : cl[3].count;
	const int wAG[4] = { P.wA, P.wG, 0, 0 };
	const int wAR[4] = { P.wA, 0, P.wR, 0 };
	const int wAGR[4] = { P.wA, P.wG, P.wR, 0 };
	const int wAGB[4] = { P.wA, P.wG, 0, P.wB };
	const int wAGRB[4] = { P.wA, P.wG, P.wR, P.wB };
	const int2* LA = ss.lists[0][0];
	const int2* LG = ss.lists[0][1];
	const int2* LR = ss.lists[0][2];
	const int2* LB = ss.lists[0][3];
	const int colB = lane < nB ? LB[lane].y : 0;
	const int eBbase = lane < nB ? LB[lane].x : kBig;
	for (int iA = 0; iA < nA; iA++)
	{
		const int eA = LA[iA].x;
		if (eA + minG + minR + minB >= water)
			break;
		const int cA = LA[iA].y;
		int memAR = kBig, pairAG = kBig;
		if ((rot == 2 || rot == 3) && lane < nR)
			memAR = RotErrorW<kD, CB, AB, MODE == 4>(ar, ai, Ep2(0, cA, 2, LR[lane].y), rot, wAR, water - minG - minB);
		if ((rot == 1 || rot == 3) && lane < nG)
			pairAG = RotErrorW<kD, CB, AB, MODE == 4>(ar, ai, Ep2(0, cA, 1, LG[lane].y), rot, wAG, water - minR - minB);
		for (int iG = 0; iG < nG; iG++)
		{
			int eG = LG[iG].x + eA;
			if (eG + minR + minB >= water)
				break;
			const int cG = LG[iG].y;
			if (rot == 1 || rot == 3)
			{
				eG = __shfl_sync(kFull, pairAG, iG);
				if (eG + minR + minB >= water)
					continue;
			}
			const Ep baseAG = Ep2(0, cA, 1, cG);
			int memAGB = kBig, pairAGR = kBig;
			if (rot != 3 && lane < nB)
				memAGB = RotErrorW<kD, CB, AB, MODE == 4>(ar, ai, EpSetCh(baseAG, 3, LB[lane].y), rot, wAGB, water - minR);
			if ((rot == 0 || rot == 3) && lane < nR)
				pairAGR = RotErrorW<kD, CB, AB, MODE == 4>(ar, ai, EpSetCh(baseAG, 2, LR[lane].y), rot, wAGR, water - minB);
			for (int iR = 0; iR < nR; iR++)
			{
				int eR = LR[iR].x + eG;
				if (eR + minB >= water)
					break;
				const int cR = LR[iR].y;
				if (rot == 2 || rot == 3)
				{
					const int ear = __shfl_sync(kFull, memAR, iR);
					if (ear + minG + minB >= water)
						continue;
					if (rot == 2)
						eR = ear + LG[iG].x;
				}
				if (rot == 0 || rot == 3)
				{
					eR = __shfl_sync(kFull, pairAGR, iR);
					if (eR + minB >= water)
						continue;
				}
				const Ep baseAGR = EpSetCh(baseAG, 2, cR);
				const bool valid = lane < nB;
				const int brk = valid ? eBbase + eR : kBig;
				const int skip = (valid && rot != 3) ? memAGB + minR : brk;
				int err = kBig;
				if (valid && brk < water && skip < water)
				{
					if (rot == 1)
						err = memAGB + LR[iR].x;
					else if (rot == 3)
						err = brk;
					else
						err = RotErrorW<kD, CB, AB, MODE == 4>(ar, ai, EpSetCh(baseAGR, 3, colB), rot, wAGRB, water);
				}
				const int jl = ReplayInner(valid, brk, skip, err, water, lane);
				if (jl >= 0)
					bestStorage = EpSwapRot(EpSetCh(baseAGR, 3, __shfl_sync(kFull, colB, jl)), rot);
			}
		}
	}
	return water;
}

/* Subset InitLevels of modes 4 / 5 (src/Bc7CoreMode4.cpp:1264-1322, :1505-1563,
   src/Bc7CoreMode5.cpp:628-686) + TryVariants. */
template<int kD, int MODE>
__device__ NEBC7_PASS int CompressRotSubset(WarpState& st, SearchState& ss, const CellRegs& R, const Params& P, const LevelTables& T,
	Ep& mcStorage, int water, int rotation, Team& team, TeamState* ts, int lane)
{
	const Area& ar = st.area1;
	const AreaInfo& ai = ar.info;
	const bool idx32 = MODE == 4 && (rotation & 4);
	const int a = RotChannel(rotation);
	int cbits, abits;
	const uint8_t *ctab, *atab;
	if (MODE == 4)
	{
		cbits = 5;
		abits = 6;
		ctab = idx32 ? T.d3v8 : T.d2v8;
		atab = idx32 ? T.d2v8 : T.d3v8;
	}
	else
	{
		cbits = 7;
		abits = 8;
		ctab = T.d2v8;
		atab = T.d2v8;
	}
	/* With every visible pixel's masks full the bounds are lower bounds (the
	   slot channel's list error is its exact error, and a hidden pixel counts
	   with its alpha of 0 alone): the three channels that share the colour
	   index are searched by SearchThree, the slot channel's one candidate a
	   constant.  Other masks can make a bound exceed the error, and the
	   reference's order of tests decides: TryVariantsRot. */
	bool full = true;
	if (lane < ai.active)
		full = (ar.mk[lane][0] & ar.mk[lane][1] & ar.mk[lane][2] & ar.mk[lane][3]) == 0xFFFF;
	full = __all_sync(kFull, full);
	int used = 0;
#pragma unroll 1
	for (int c = 0; c < 4; c++)
	{
		const int w = ChannelWeight(P, c);
		ChanList cl;
		if (c == 0 && ai.opaque)
			cl = ZeroList(ss.lists[0][0], 0xFFFF, lane);
		else if (c == a)
			cl = ChannelLevelsSingle<kD>(ss.lists[0][c], ar, c, w, water - used, abits, c != 0, atab, ss.values, lane);
		else
			cl = ChannelLevels<kD, false>(ss.lists[0][c], ar, c, w, water - used, cbits, -1, c != 0, ctab, true, 32, ss.values, team, lane);
		if (lane == 0)
			ss.chan[0][c] = cl;
		used += cl.minErr;
		if (used >= water)
			return water;
	}
	__syncwarp();
	const int rot = rotation & 3;
	if (full)
	{
		const int x = a == 0 ? 1 : 0, y = a <= 1 ? 2 : 1, z = a == 3 ? 2 : 3;
		auto channel = [&](int c) {
			return SearchChannel{ c, ChannelWeight(P, c), ss.lists[0][c], ss.chan[0][c].count, ss.chan[0][c].minErr };
		};
		const int slot = ss.chan[0][a].minErr;   /* its only candidate's error */
		const int hidden = a != 0 ? 16 - ai.active : 0;
		Found3 f;
		if (idx32)
			f = SearchThree<kD, 3>(ar, ai.active, channel(x), channel(y), channel(z), hidden, water - slot, ss.plane, team, ts, lane);
		else
			f = SearchThree<kD, 2>(ar, ai.active, channel(x), channel(y), channel(z), hidden, water - slot, ss.plane, team, ts, lane);
		if (f.taken)
			mcStorage = EpSwapRot(EpSetCh(EpSetCh(Ep2(x, f.x, y, f.y), z, f.z), a, ss.lists[0][a][0].y), rot);
		return f.water + slot;
	}
	if (MODE == 5)
		return TryVariantsRot<kD, 5, 2, 2>(ar, ai, P, ss, mcStorage, water, rot, lane);
	if (idx32)
		return TryVariantsRot<kD, 4, 3, 2>(ar, ai, P, ss, mcStorage, water, rot, lane);
	return TryVariantsRot<kD, 4, 2, 3>(ar, ai, P, ss, mcStorage, water, rot, lane);
}

template<int kD>
__device__ NEBC7_PASS void RefineMode4(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const LevelTables& T, Team& team, TeamState* ts,
	int lane)
{
	/* src/Bc7CoreMode4.cpp:1795-1822 */
	int rotation = R.bestParam;
#pragma unroll 1
	for (int i = 0; i < 2; i++, rotation ^= 4)
	{
		Ep mc = 0;
		const int error = CompressRotSubset<kD, 4>(st, ss, R, P, T, mc, R.errTotal, rotation, team, ts, lane);
		if (R.errTotal > error)
		{
			R.errTotal = error;
			R.best[0] = mc;
			R.bestParam = rotation;
			if (error <= 0)
				break;
		}
	}
}

template<int kD>
__device__ NEBC7_PASS void RefineMode5(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const LevelTables& T, Team& team, TeamState* ts,
	int lane)
{
	/* src/Bc7CoreMode5.cpp:890-911 */
	Ep mc = 0;
	const int error = CompressRotSubset<kD, 5>(st, ss, R, P, T, mc, R.errTotal, R.bestParam, team, ts, lane);
	if (R.errTotal > error)
	{
		R.errTotal = error;
		R.best[0] = mc;
	}
}

template<int kD, int MODE>
__device__ NEBC7_PASS void FullRot(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const LevelTables& T, int lane,
	int from = 0)
{
	/* src/Bc7CoreMode4.cpp:1824-1857, src/Bc7CoreMode5.cpp:913-946; the
	   search may resume at choice `from` */
	const int step = R.denoiseStep;
	constexpr int NR = MODE == 4 ? 8 : 4;
	Team one = SingleWarp();
#pragma unroll 1
	for (int ri = from; ri < NR; ri++)
	{
		const int rotation = MODE == 4 ? c_rot4[ri] : c_rot5[ri];
		if (MODE == 4 && R.personalMode == 4 && !((R.personalParam ^ rotation) & 3))
			continue;
		if (MODE == 5 && R.personalMode == 5 && R.personalParam == rotation)
			continue;
		Ep mc = 0;
		int error = step;
		if (error < R.errTotal)
			error += CompressRotSubset<kD, MODE>(st, ss, R, P, T, mc, R.errTotal - error, rotation, one, nullptr, lane);
		if (R.errTotal > error)
		{
			R.errTotal = error - step;
			R.best[0] = mc;
			R.bestParam = rotation;
			R.bestMode = MODE;
			if (error <= step)
				break;
		}
	}
}

/* ---------------------------------------------------------------------- */
/* The normal / slow pass chain (src/Bc7Core.cpp:1604-1745)                */
/* ---------------------------------------------------------------------- */

template<int kD>
__device__ void NormalPasses(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const LevelTables& T, int lane)
{
	Team one = SingleWarp();
	const int OA = R.opaqueAlphaError;
	const int step = R.denoiseStep;

	switch (R.bestMode)
	{
	case 0: if (R.errTotal > OA) RefineOpaque<kD, 0>(st, ss, R, P, T, one, nullptr, lane); break;
	case 1: if (R.errTotal > OA) RefineOpaque<kD, 1>(st, ss, R, P, T, one, nullptr, lane); break;
	case 2: if (R.errTotal > OA) RefineOpaque<kD, 2>(st, ss, R, P, T, one, nullptr, lane); break;
	case 3: if (R.errTotal > OA) RefineOpaque<kD, 3>(st, ss, R, P, T, one, nullptr, lane); break;
	case 4: if (R.errTotal > 0) RefineMode4<kD>(st, ss, R, P, T, one, nullptr, lane); break;
	case 5: if (R.errTotal > 0) RefineMode5<kD>(st, ss, R, P, T, one, nullptr, lane); break;
	case 6: if (R.errTotal > 0) RefineMode6<kD, 6>(st, ss, R, P, T, one, nullptr, lane); break;
	case 7: if (R.errTotal > 0) RefineMode7<kD>(st, ss, R, P, T, one, nullptr, 0, lane); break;
	case 9: if (R.errTotal > 0) RefineMode6<kD, 9>(st, ss, R, P, T, one, nullptr, lane); break;
	}

	R.personalParam = R.bestParam;
	R.personalMode = R.bestMode;

	if (R.a1.opaque)
	{
		if (R.errTotal > OA + step)
		{
			FullThreeSubsets<kD, 2>(st, ss, R, P, T, lane);
			if (R.errTotal > OA + step)
			{
				FullThreeSubsets<kD, 0>(st, ss, R, P, T, lane);
				if (P.doSlow && R.errTotal > OA + step)
				{
					FullTwoSubsets<kD, 1>(st, ss, R, P, T, lane);
					if (R.errTotal > OA + step)
					{
						FullTwoSubsets<kD, 3>(st, ss, R, P, T, lane);
						if (R.errTotal > step)
						{
							FullRot<kD, 5>(st, ss, R, P, T, lane);
							if (R.errTotal > step)
							{
								FullRot<kD, 4>(st, ss, R, P, T, lane);
								if (R.errTotal > step)
								{
									FullMode7<kD>(st, ss, R, P, T, lane);
									if (R.errTotal > step)
										FullMode6<kD>(st, ss, R, P, T, one, nullptr, lane);
								}
							}
						}
					}
				}
			}
		}
	}
	else
	{
		if (R.errTotal > step)
		{
			FullRot<kD, 5>(st, ss, R, P, T, lane);
			if (R.errTotal > step)
			{
				FullRot<kD, 4>(st, ss, R, P, T, lane);
				if (R.errTotal > step)
				{
					FullMode7<kD>(st, ss, R, P, T, lane);
					if (P.doSlow && R.errTotal > step)
						FullMode6<kD>(st, ss, R, P, T, one, nullptr, lane);
				}
			}
		}
	}
}

} // namespace nebc7
