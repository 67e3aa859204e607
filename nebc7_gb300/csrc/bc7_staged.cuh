/*
 * BC7 block encoder for sm_103a -- the staged encode of every refining preset
 * (default, precise, /slow, /data, mixed batches).
 *
 * The per-block pipeline of src/Bc7Core.cpp:1516-1823 runs as a sequence of
 * persistent kernels instead of one: the start of the draft chain (the
 * starting block, the Mode6Index2 and mode 6 fast passes), the rest of the
 * draft chain, the refinement, one or two kernels per full-search pass of the
 * normal and slow chains (src/Bc7Core.cpp:1604-1745), then the final pack,
 * self-check and quality sums.  The warps of an SM so run the same few
 * kilobytes of instructions; in a single kernel whose warps sit in different
 * passes the instruction working set outgrows the instruction cache and most
 * issue slots are lost to instruction fetch.  And a pass can hand its hard
 * blocks to several warps: a 1000x516 alpha texture of the default preset took
 * 424 ms in one kernel, a single block most of them, and takes 32 ms so.
 *
 * Between kernels a block's state (the reference's Cell scalars: best
 * endpoints, mode, partition, errors, stepping values, the starting block)
 * is kept in a BlockRecord per queue position; the pixel data and the
 * whole-block area are rebuilt from the texture when a pass starts.  A block
 * that ends a pass counts itself into a bucket of its next one (Publish,
 * StageBucket), and KStageList gathers each pass's blocks bucket by bucket.
 * The passes, their order and their entry conditions are those of
 * NormalPasses, so the blocks are the same bits as the single-kernel
 * encode's.
 *
 * The searches of a few hard blocks take most of a pass, and one warp per
 * block would leave the GPU waiting for them.  So
 * - the refinement, the three-subset searches and the full mode 6 search run
 *   their few or first blocks with a CTA's four warps each (TeamBlocks);
 * - the full searches of modes 1, 3 and 7 (64 two-subset partitions each) and of
 *   modes 4 and 5 (8 and 4 rotation / index-size choices) are split passes, and
 *   so are the partitions that the estimates of modes 2 and 0 leave of a block
 *   (ThreeSubsetsStage).
 * A split pass runs in rounds.  In a round every candidate (partition or
 * rotation) of a block is a task of its own, searched from the block's error at
 * the start of the round.  The candidates before the block's first improving
 * candidate f searched from that error, as the reference's loop does, so their
 * verdicts stand; f's result is the reference's too.  The block's last task
 * commits the round: it applies f and ends the pass, or appends the block's
 * next round, from candidate f + 1 with the new error, to the queue that the
 * running warps take tasks from.  Improvements are rare, so most blocks finish
 * in the first round.  Blocks whose result was not kept, or that must run whole
 * (OPTION_PCA), finish the pass in one warp each.
 */
#pragma once

#include "bc7_encode.cuh"

namespace nebc7 {

/* The passes after the first kernel, in chain order: the rest of the draft
   chain, then the normal and slow chains; kStepFinish packs. */
enum StageStep
{
	kStepDraftRest = 0,    /* fast passes of modes 4, 5, 7 and the opaque modes 3, 1, 2, 0 */
	kStepRefine,
	kStepFull3Mode2,
	kStepFull3Mode0,
	kStepFull2Mode1,
	kStepFull2Mode3,
	kStepRot5,
	kStepRot4,
	kStepMode7,
	kStepMode6,
	kStepFinish,
	kNumStages
};

constexpr int kStageDraft = -1;
constexpr int kStepNone = -1;   /* finished in the first kernel (an exact starting block) */

/* The kinds of refinement, in the order of their list: few blocks with long
   searches first. */
enum RefineKind
{
	kRefine6 = 0,    /* mode 6 of blocks with alpha */
	kRefine7,
	kRefine6Index2,  /* of blocks with alpha */
	kRefineOpaque,   /* modes 0-3 */
	kRefineRot,      /* modes 4 and 5 */
	kRefineEasy,     /* modes 6 and 6Index2 of opaque blocks: one p-bit variant, one alpha candidate */
	kRefineKinds
};

__device__ __forceinline__ int RefineKindOf(int mode, bool opaque)
{
	if (mode < 6)
		return mode < 4 ? kRefineOpaque : kRefineRot;
	return mode == 7 ? kRefine7 : (opaque ? kRefineEasy : (mode == 6 ? kRefine6 : kRefine6Index2));
}

/* Buckets of the refinement's list per kind; the first ones, modes 6, 6Index2
   and 7 of blocks with alpha, can search long. */
constexpr int kRefineBuckets = 256 / kRefineKinds;
constexpr int kRefineHeavy = kRefineOpaque * kRefineBuckets;

/* A block's Cell scalars between pass kernels. */
struct __align__(16) BlockRecord
{
	Ep best[3];
	uint64_t startLo, startHi;   /* the starting block (self-check fallback) */
	int bestParam, bestMode, opaqueAlphaError, errAlpha;
	int errTotal, personalParam, personalMode, denoiseStep;
	int water;                   /* the error at the start of the draft chain */
	int opaque;                  /* the whole-block area's opaque flag */
	int handed;                  /* 1 + its slot of handed estimates, or 0 */
	int denoise;                 /* which of the two code paths (kD) it takes */
};

/* An improving candidate of a split pass: its endpoints, error and
   parameter (partition or rotation), and whether it ends the full search
   (src/Bc7CoreMode1.cpp:563-564, src/Bc7CoreMode7.cpp:719-720,
   src/Bc7CoreMode4.cpp:1852-1853). */
struct __align__(16) SplitResult
{
	Ep best0, best1, best2;
	int error, end, param;
	int pad[3];
};

/* The split passes. */
constexpr int kSplitMaxBlocks = 1 << 24;    /* blocks of a pass split into tasks (the task count stays an int) */
constexpr int kSplitSerial = -1;            /* firstImp: the block's pass runs whole (OPTION_PCA) */
constexpr int kSplitNone = 0x7FFFFFFF;      /* firstImp: no improvement yet */
/* firstImp otherwise: the candidate above the slot of its kept result, or above
   kSplitNoSlot if there was no room for it.  Every slot is below that mark
   (SplitResultCap). */
constexpr int kSplitSlotBits = 24;
constexpr int kSplitNoSlot = (1 << kSplitSlotBits) - 1;
/* Polls of a warp that waits for a later round's tasks (2 us and more each)
   before it leaves them to the others: about ten seconds. */
constexpr int kSplitPolls = 1 << 22;

__host__ __device__ constexpr int SplitIndex(int S)
{
	return S == kStepFull2Mode1 ? 0 : (S == kStepFull2Mode3 ? 1 : (S == kStepRot5 ? 2 : (S == kStepRot4 ? 3 : (S == kStepMode7 ? 4 :
		(S == kStepFull3Mode2 ? 5 : (S == kStepFull3Mode0 ? 6 : -1))))));
}

constexpr int kSplitPasses = 7;
constexpr int kSplitMaxTasks = 64;   /* candidates of a block at most */

/* The three-subset passes estimate first, a warp or a team per block, and hand
   a block to the tasks when more than kInlineCandidates partitions are left:
   a photo's hardest blocks searched 30 and more one after another, 7 ms in
   one warp with the rest of the GPU idle, where most blocks have one to
   four. */
__host__ __device__ constexpr bool ThreeSubsetStep(int S)
{
	return S == kStepFull3Mode2 || S == kStepFull3Mode0;
}

constexpr int kInlineCandidates = 6;
/* A longer list fills the GPU as it is.  Precise photos handed over and inline:
   64x64 1.98 and 3.82 ms, 256x256 9.73 and 10.25, 320x320 12.0 and 11.5, 512x512
   23.3 and 19.7, 1024x1024 44.8 and 39.6; /data normal maps 256x256 (short lists)
   2.15 and 5.28, 512x512 4.21 and 8.00: from 5000 blocks to this line the
   precise preset loses 5 %, beyond it handing over would lose more. */
constexpr int kHandOverBlocks = 8192;
constexpr int kHandedBlocks = 2048;   /* blocks whose estimates a pass can hand over; the others finish inline */

/* Candidates (tasks) per block of split pass S, and its mode. */
__host__ __device__ constexpr int SplitTasks(int S)
{
	return S == kStepRot4 ? 8 : (S == kStepRot5 ? 4 : (S == kStepFull3Mode0 ? 16 : 64));
}

__host__ __device__ constexpr int SplitMode(int S)
{
	return S == kStepFull2Mode1 ? 1 : (S == kStepFull2Mode3 ? 3 : (S == kStepRot5 ? 5 : (S == kStepRot4 ? 4 : (S == kStepMode7 ? 7 :
		(S == kStepFull3Mode2 ? 2 : 0)))));
}

/* Kernel launches of a staged encode: the draft kernel, then per pass its
   list and its kernel, a split pass's remainder; without /slow the passes that
   only it reaches are left out. */
__host__ __device__ constexpr bool StageLaunched(int S, bool slow)
{
	return slow || (S != kStepFull2Mode1 && S != kStepFull2Mode3 && S != kStepMode6);
}

__host__ __device__ constexpr int StagedLaunches(bool slow)
{
	int n = 1;
	for (int S = 0; S < kNumStages; S++)
		if (StageLaunched(S, slow))
			n += ThreeSubsetStep(S) ? 4 : (SplitIndex(S) >= 0 ? 3 : 2);
	return n;
}

/* The task queue of a split pass (zero before the draft kernel).  The first
   round's tasks are those of the pass's list, the later rounds' entries are
   appended to Stages::later; polled together in one 16-byte read. */
struct __align__(16) SplitQueue
{
	int laterHead, laterTail;   /* later tasks taken, later entries published */
	int finished;               /* blocks that have left the pass */
	int laterReserve;           /* later entries reserved */
	int pad0[28];
	int head;                   /* first-round tasks taken */
	int kept;                   /* results kept */
	int restCount, restHead;    /* the one-warp remainder */
	int handedCount;            /* blocks handed over (three-subset passes) */
	int pad1[27];
};

/* Waits for the kernels before this one in its stream.  Every kernel of the
   staged form starts with this and can be launched as the programmatic dependent
   of the one before it, so that its launch overlaps that one's end; a pass without
   blocks then returns at once.  Of the chain's 24 to 32 kernels most find nothing
   to do in an easy texture: 64x64 of one colour 371 -> 310 us a call, a 64x64
   photo 724 -> 650, loose cells 287 -> 216. */
__device__ __forceinline__ void WaitForLaunch()
{
	asm volatile("griddepcontrol.wait;" ::: "memory");
}

/* Per-launch state of a staged encode (one entry per queue position). */
struct Stages
{
	BlockRecord* rec;
	int* next;        /* the pass a position waits for, kStepFinish, or kStepNone */
	int* list;        /* positions of the pass being run, in queue order */
	int* count;       /* [kNumStages] list lengths, then the number of blocks of the refinement's heavy buckets */
	int* counters;    /* [kNumStages + 1] work-queue heads, zero before the draft kernel */
	int* hist;        /* [kNumStages][256] blocks per bucket of the passes' lists, zero before the draft kernel */
	int* cursor;      /* [kNumStages][256] positions taken, zero before the draft kernel */
	int total;        /* positions */
	int mixed;        /* whether blocks of both denoise forms are in the launch */
	/* split passes */
	int* start;       /* per position: the first candidate of the block's round */
	int* firstImp;    /* per position: (candidate << kSplitSlotBits) | result slot of the round's first improvement */
	int* pending;     /* per position: the round's candidates not done */
	int* later;       /* the blocks of the later rounds, in the order they were appended */
	int laterCap;
	int* rest;        /* the blocks of the one-warp remainder */
	SplitQueue* split;   /* [kSplitPasses] */
	int* handed;      /* the blocks handed over by a three-subset pass, */
	ThreeEstimates* estimates;   /* and their estimates, by slot */
	int handedCap;
	SplitResult* imp;
	int impCap;
};

/* Bucket of position k in the list of pass `stage`: 8 per octave of the
   error, largest first, for the searches (their cost grows with it: the
   longest start first and no SM waits behind a late hard block), 4 per octave
   and denoised blocks first in a mixed launch (the two forms are different
   code), for the refinement by kind and 1.3 per octave within it (so that the
   warps of an SM run the same code), else by position. */
__device__ __forceinline__ int StageBucket(const Stages& sg, int stage, int k, int error, int mode, bool opaque, int denoise)
{
	if (stage < kStepRefine || stage == kStepFinish)
		return int((long long)k * 256 / sg.total);
	const unsigned e = unsigned(max(error, 1));
	const int msb = 31 - __clz(e);
	const int b = 255 - min(255, msb * 8 + int((e >> (msb >= 3 ? msb - 3 : 0)) & 7u));
	const int kind = RefineKindOf(mode, opaque);
	/* the buckets of the block's kind, and in a mixed launch the half of its
	   denoise form */
	int from = 0, width = 256;
	if (stage == kStepRefine)
	{
		width = kRefineBuckets;
		from = kRefineBuckets * kind;
	}
	if (sg.mixed)
	{
		width >>= 1;
		from += denoise ? 0 : width;
	}
	return from + (b * width >> 8);
}

/* Records that position k waits for pass n (one thread). */
__device__ __forceinline__ void Publish(const Stages& sg, int k, int n, int error, int mode, bool opaque, int denoise)
{
	sg.next[k] = n;
	atomicAdd(&sg.hist[n * 256 + StageBucket(sg, n, k, error, mode, opaque, denoise)], 1);
}

__device__ __forceinline__ void SaveRecord(BlockRecord& r, const CellRegs& R, int lane)
{
	if (lane == 0)
	{
		r.best[0] = R.best[0];
		r.best[1] = R.best[1];
		r.best[2] = R.best[2];
		r.bestParam = R.bestParam;
		r.bestMode = R.bestMode;
		r.opaqueAlphaError = R.opaqueAlphaError;
		r.errAlpha = R.errAlpha;
		r.errTotal = R.errTotal;
		r.personalParam = R.personalParam;
		r.personalMode = R.personalMode;
		r.denoiseStep = R.denoiseStep;
		r.opaque = R.a1.opaque;
	}
}

/* Rebuilds a block's state: its pixels and masks, the saved scalars, the
   whole-block area (src/Bc7Core.cpp:1532-1535).  Returns the record's
   `handed`. */
__device__ __forceinline__ int RestoreBlock(WarpState& st, CellRegs& R, const BlockRef& b, const BlockRecord& record, const Params& P,
	int lane)
{
	LoadCell(st, b, R, lane);
	/* past L1: another SM may have written it within this kernel (split passes) */
	BlockRecord r;
	const uint4* from = reinterpret_cast<const uint4*>(&record);
#pragma unroll
	for (int i = 0; i < int(sizeof(BlockRecord) / 16); i++)
		reinterpret_cast<uint4*>(&r)[i] = __ldcg(from + i);
	R.best[0] = r.best[0];
	R.best[1] = r.best[1];
	R.best[2] = r.best[2];
	R.bestParam = r.bestParam;
	R.bestMode = r.bestMode;
	R.opaqueAlphaError = r.opaqueAlphaError;
	R.errAlpha = r.errAlpha;
	R.errTotal = r.errTotal;
	R.personalParam = r.personalParam;
	R.personalMode = r.personalMode;
	R.denoiseStep = r.denoiseStep;
	BuildWholeBlock(st, R, P, lane);
	return r.handed;
}

/* Shared memory of a warp of stage STAGE: the block state, and the search
   state as far as the pass uses it (SearchState).  One CTA of the precise
   mode-2 search took 53 KB with the whole of both, which left 37 KB of L1 for
   16 warps (18 % hits on the level tables). */
__host__ __device__ constexpr size_t StageWarpBytes(int stage, bool split)
{
	if (stage < kStepRefine || stage == kStepFinish)
		return sizeof(WarpState);
	const bool pca = !split && (stage == kStepFull2Mode1 || stage == kStepFull2Mode3 || stage == kStepMode7);
	const size_t search = pca ? sizeof(SearchState)
		: (stage == kStepRefine || stage == kStepMode7) ? offsetof(SearchState, table) + sizeof(SearchState::table)
		: stage == kStepMode6 ? offsetof(SearchState, plane16) + sizeof(SearchState::plane16)
		: ThreeSubsetStep(stage) ? offsetof(SearchState, three) + sizeof(SearchState::three)
		: offsetof(SearchState, three);
	return kSearchWarpBytes + ((search + 15) & ~size_t(15));
}

__host__ __device__ constexpr size_t StageSharedBytes(int stage, bool split)
{
	return kWarpsPerCta * StageWarpBytes(stage, split);
}

/* Passes whose blocks a CTA's warps search together when there are few
   (TeamBlocks): then the longest search is what the pass takes (a 1024x1024
   photo leaves the three-subset search of mode 2 eight blocks, 2.3 ms of one
   warp each; the mode 7 refinement of an alpha texture's 1200 blocks took
   5.4 ms, 0.4 ms of the GPU's warps).  Of a long refinement list the first two
   blocks per CTA, which the list's order makes the ones with long searches, and
   up to 16 per CTA of those with alpha (modes 6, 6Index2, 7): on a 1118x1105
   alpha texture one mode 6 block took a warp 33 ms, and the 56065 blocks'
   refinement 34.0 ms with 2 per CTA, 15.8 ms with 16. */
__host__ __device__ constexpr bool TeamStage(int S)
{
	return ThreeSubsetStep(S) || S == kStepRefine || S == kStepMode6;
}

__device__ __forceinline__ int TeamBlocks(int S, int n, int heavy, int ctas)
{
	if (n <= (ThreeSubsetStep(S) ? 1 : 2) * kWarpsPerCta * ctas)
		return n;
	return S == kStepRefine ? max(min(heavy, 16 * ctas), min(n, 2 * ctas)) : 0;
}

/* The refinement of a block's mode (ModeN::CompressBlock), one function per
   kind: each has registers and code of its own (inlined into one kernel body
   the kinds spilled and outgrew the instruction cache, 30 -> 38 ms on an alpha
   texture; one kernel per kind waits for the longest search of each).  The
   warp's state, the tables and the team's exchange come as shared-memory
   addresses, so that the accesses stay shared ones. */
template<int kD, int KIND>
__device__ __noinline__ void RefineOne(CellRegs& shared, unsigned stAt, unsigned tablesAt, unsigned tsAt, int size, int rank, int lane)
{
	WarpState& st = *static_cast<WarpState*>(__cvta_shared_to_generic(stAt));
	SearchState& ss = *static_cast<SearchState*>(__cvta_shared_to_generic(stAt + kSearchWarpBytes));
	const LevelTables& T = *static_cast<const LevelTables*>(__cvta_shared_to_generic(tablesAt));
	TeamState* ts = static_cast<TeamState*>(__cvta_shared_to_generic(tsAt));
	const Params& P = st.P;
	CellRegs R = shared;
	Team team{ size, rank, &ts->exchange, 0 };
	if constexpr (KIND == kRefineOpaque)
	{
		switch (R.bestMode)
		{
		case 0: RefineOpaque<kD, 0>(st, ss, R, P, T, team, ts, lane); break;
		case 1: RefineOpaque<kD, 1>(st, ss, R, P, T, team, ts, lane); break;
		case 2: RefineOpaque<kD, 2>(st, ss, R, P, T, team, ts, lane); break;
		default: RefineOpaque<kD, 3>(st, ss, R, P, T, team, ts, lane); break;
		}
	}
	else if constexpr (KIND == kRefineRot)
	{
		if (R.bestMode == 4)
			RefineMode4<kD>(st, ss, R, P, T, team, ts, lane);
		else
			RefineMode5<kD>(st, ss, R, P, T, team, ts, lane);
	}
	else if constexpr (KIND == kRefine6)
	{
		if (R.bestMode == 6)
			RefineMode6<kD, 6>(st, ss, R, P, T, team, ts, lane);
		else
			RefineMode6<kD, 9>(st, ss, R, P, T, team, ts, lane);
	}
	else
		RefineMode7<kD>(st, ss, R, P, T, team, ts, StageWarpBytes(kStepRefine, false), lane);
	shared = R;
}

/* One stage: the passes of the draft chain after the mode 6 fast pass
   (DraftChain), or one pass of the normal / slow chains (NormalPasses). */
template<int kD, int S>
__device__ __forceinline__ void RunStep(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const LevelTables& T, int lane,
	int from, Team& team, TeamState* ts)
{
	if constexpr (S == kStepDraftRest)
	{
		/* entered with errTotal > step (src/Bc7Core.cpp:1558-1597) */
		const int step = R.denoiseStep, gate = R.opaqueAlphaError + step;
		FastRot<kD, 4>(st, R, P, lane);
		if (R.errTotal > step)
		{
			FastRot<kD, 5>(st, R, P, lane);
			if (R.errTotal > step)
				FastMode7<kD>(st, R, P, T, lane);
		}
		if (int(int16_t(R.a1.minmax[0])) > 255 - 16 && R.errTotal > gate)
		{
			FastOpaque<kD, 3>(st, R, P, lane);
			if (R.errTotal > gate)
			{
				FastOpaque<kD, 1>(st, R, P, lane);
				if (R.errTotal > gate)
				{
					FastOpaque<kD, 2>(st, R, P, lane);
					if (R.errTotal > gate)
						FastOpaque<kD, 0>(st, R, P, lane);
				}
			}
		}
	}
	else if constexpr (S == kStepRefine)
	{
		if (R.errTotal > (R.bestMode < 4 ? R.opaqueAlphaError : 0))
		{
			const unsigned stAt = unsigned(__cvta_generic_to_shared(&st));
			const unsigned tablesAt = unsigned(__cvta_generic_to_shared(&T));
			const unsigned tsAt = unsigned(__cvta_generic_to_shared(ts));
			if (R.bestMode < 4)
				RefineOne<kD, kRefineOpaque>(R, stAt, tablesAt, tsAt, team.size, team.rank, lane);
			else if (R.bestMode < 6)
				RefineOne<kD, kRefineRot>(R, stAt, tablesAt, tsAt, team.size, team.rank, lane);
			else if (R.bestMode == 7)
				RefineOne<kD, kRefine7>(R, stAt, tablesAt, tsAt, team.size, team.rank, lane);
			else
				RefineOne<kD, kRefine6>(R, stAt, tablesAt, tsAt, team.size, team.rank, lane);
		}
		R.personalParam = R.bestParam;
		R.personalMode = R.bestMode;
	}
	else if constexpr (S == kStepFull2Mode1)
		FullTwoSubsets<kD, 1>(st, ss, R, P, T, lane, from);
	else if constexpr (S == kStepFull2Mode3)
		FullTwoSubsets<kD, 3>(st, ss, R, P, T, lane, from);
	else if constexpr (S == kStepRot5)
		FullRot<kD, 5>(st, ss, R, P, T, lane, from);
	else if constexpr (S == kStepRot4)
		FullRot<kD, 4>(st, ss, R, P, T, lane, from);
	else if constexpr (S == kStepMode7)
		FullMode7<kD>(st, ss, R, P, T, lane, from);
	else if constexpr (S == kStepMode6)
		FullMode6<kD>(st, ss, R, P, T, team, ts, lane);
}

__device__ __forceinline__ int AfterDraft(const Params& P)
{
	return (P.doNormal && P.doDraft != 2) ? kStepRefine : kStepFinish;
}

/* The pass after S: the nesting of the normal and slow chains in
   NormalPasses (src/Bc7Core.cpp:1677-1745), whose conditions are tested when
   each pass is reached. */
__device__ __forceinline__ int NextStep(int S, const CellRegs& R, const Params& P)
{
	const int OA = R.opaqueAlphaError, step = R.denoiseStep, e = R.errTotal;
	if (S == kStepDraftRest)
		return AfterDraft(P);
	if (R.a1.opaque)
	{
		switch (S)
		{
		case kStepRefine: return e > OA + step ? kStepFull3Mode2 : kStepFinish;
		case kStepFull3Mode2: return e > OA + step ? kStepFull3Mode0 : kStepFinish;
		case kStepFull3Mode0: return (P.doSlow && e > OA + step) ? kStepFull2Mode1 : kStepFinish;
		case kStepFull2Mode1: return e > OA + step ? kStepFull2Mode3 : kStepFinish;
		case kStepFull2Mode3: return e > step ? kStepRot5 : kStepFinish;
		case kStepRot5: return e > step ? kStepRot4 : kStepFinish;
		case kStepRot4: return e > step ? kStepMode7 : kStepFinish;
		case kStepMode7: return e > step ? kStepMode6 : kStepFinish;
		default: return kStepFinish;
		}
	}
	switch (S)
	{
	case kStepRefine: return e > step ? kStepRot5 : kStepFinish;
	case kStepRot5: return e > step ? kStepRot4 : kStepFinish;
	case kStepRot4: return e > step ? kStepMode7 : kStepFinish;
	case kStepMode7: return (P.doSlow && e > step) ? kStepMode6 : kStepFinish;
	default: return kStepFinish;
	}
}

/* Writes the block and its result (src/Bc7Core.cpp:1976-1984). */
template<int kD>
__device__ __forceinline__ void StoreBlock(const BlockRef& b, const CellRegs& R, uint64_t lo, uint64_t hi, double qa, double qc,
	int lane)
{
	if (lane == 0)
	{
		*reinterpret_cast<uint4*>(b.out) = make_uint4(unsigned(lo), unsigned(lo >> 32), unsigned(hi), unsigned(hi >> 32));
		if (b.result)
		{
			BlockResult r;
			r.errAlpha = int(unsigned(R.errAlpha) << (kD + kD));
			r.errColor = int(unsigned(R.errTotal - R.errAlpha) << (kD + kD));
			r.ssimAlpha = qa;
			r.ssimColor = qc;
			*b.result = r;
		}
	}
	__syncwarp();
}

/* The final pack when the search beat the starting block, then the
   self-check (src/Bc7Core.cpp:1799-1807) and the SSIM sums. */
template<int kD>
__device__ __forceinline__ void FinishBlock(WarpState& st, CellRegs& R, const Params& P, int water, uint64_t startLo, uint64_t startHi,
	const BlockRef& b, int lane)
{
	uint64_t lo = startLo, hi = startHi;
	if (water > R.errTotal)
		FinalPack<kD>(st, R, P, lo, hi, lane);
	Ep dummy[3];
	int dp, dm;
	DecodeToState(st, lo, hi, dummy, dp, dm, lane);
	int ea, et;
	CompareBlocks<kD>(st, P, lane, ea, et);
	if (ea != R.errAlpha || et != R.errTotal)
	{
		lo = startLo;
		hi = startHi;
	}
	double qa = 1.0, qc = 1.0;
	if (b.result)
		CompareBlocksSSIM(st, P, lane, qa, qc);
	StoreBlock<kD>(b, R, lo, hi, qa, qc, lane);
}

/* The first kernel's block: the start of EncodeBlockAt and of the draft
   chain (src/Bc7Core.cpp:1516-1556: the starting block, its error, the
   stepping values, the Mode6Index2 and mode 6 fast passes).  An exact
   starting block is written at once; every other block saves its record
   for the next stage and waits.  Returns whether the block finished. */
template<int kD>
__device__ bool DraftStage(WarpState& st, const BlockRef& b, const LevelTables& T, const Params& P, const Stages& sg, int k, int lane)
{
	CellRegs R;
	LoadCell(st, b, R, lane);
	const uint4 blk = *reinterpret_cast<const uint4*>(b.out);
	uint64_t lo = uint64_t(blk.x) | (uint64_t(blk.y) << 32);
	uint64_t hi = uint64_t(blk.z) | (uint64_t(blk.w) << 32);
	if (!(lo & 0xFF))
	{
		/* src/Bc7Core.cpp:1518-1522: an empty block starts as a zero mode 6 block */
		lo = 1u << 6;
		hi = 0;
	}
	DecodeToState(st, lo, hi, R.best, R.bestParam, R.bestMode, lane);
	CompareBlocks<kD>(st, P, lane, R.errAlpha, R.errTotal);
	if (!(R.errTotal > 0))
	{
		StoreBlock<kD>(b, R, lo, hi, 1.0, 1.0, lane);
		if (lane == 0)
			sg.next[k] = kStepNone;
		return true;
	}
	BuildWholeBlock(st, R, P, lane);
	R.personalMode = -1;
	R.personalParam = -1;
	const int water = R.errTotal;
	int n = kStepFinish;
	if (P.doDraft)
	{
		const int step = R.a1.active * ((P.denoiseStep * (R.a1.opaque ? P.wColor : P.wColorAlpha)) >> (kD + kD));
		R.denoiseStep = step;
		/* src/Bc7Core.cpp:24-50 */
		{
			int e = 0;
			if (!R.a1.opaque && lane < 16)
			{
				int da = int(st.area1.px[lane][0]) ^ 255;
				da = kD ? (da >> kD) : (da > 0x7F ? 0x7F : da);
				e = da * da;
			}
			e = int(__reduce_add_sync(kFull, unsigned(e)));
			R.opaqueAlphaError = R.a1.opaque ? 0 : e * P.wA;
		}
		if (P.doDraft == 2)
		{
			/* the "Mode6Index2 fast" run: the draft chain reduced to its
			   first pass (no counterpart in the reference) */
			if (R.errTotal > step && (kD > 0 || P.denoiseStep > 0))
				FastMode6<kD, true>(st, R, P, T, lane);
		}
		else
		{
			if (R.errTotal > step)
			{
				if (kD > 0 || P.denoiseStep > 0)
					FastMode6<kD, true>(st, R, P, T, lane);
				if (R.errTotal > step)
					FastMode6<kD, false>(st, R, P, T, lane);
			}
			n = R.errTotal > step ? int(kStepDraftRest) : AfterDraft(P);
		}
	}
	else
	{
		/* no draft chain: the starting block stands (water == errTotal) */
		R.denoiseStep = 0;
		R.opaqueAlphaError = 0;
	}
	BlockRecord& rec = sg.rec[k];
	SaveRecord(rec, R, lane);
	if (lane == 0)
	{
		rec.handed = 0;
		rec.denoise = kD;
		rec.startLo = lo;
		rec.startHi = hi;
		rec.water = water;
		Publish(sg, k, n, R.errTotal, R.bestMode, R.a1.opaque, kD);
	}
	__syncwarp();
	return false;
}

/* FullThreeSubsets of the block at position k: the estimates, then the search
   in the (team's first) warp, or its hand-over to the tasks of KEncodeSplit
   (returns true).  A block that was handed and comes back (a result that was
   not kept) goes on from candidate `from` with its estimates; `handed` is its
   record's, as every warp of the team read it before the first one clears it
   here: warps that disagree would part at the estimates' barriers. */
template<int kD, int S>
__device__ __forceinline__ bool ThreeSubsetsStage(WarpState& st, SearchState& ss, CellRegs& R, const Params& P, const LevelTables& T,
	const Stages& sg, int k, int handed, int from, bool hand, const Team& team, int lane)
{
	constexpr int MODE = SplitMode(S);
	const Spec3 sp = GetSpec3(MODE, T);
	BlockRecord& rec = sg.rec[k];
	if (handed)
	{
		if (team.rank)
			return false;
		const int* src = reinterpret_cast<const int*>(sg.estimates + (handed - 1));
		for (int i = lane; i < int(sizeof(ThreeEstimates) / 4); i += 32)
			reinterpret_cast<int*>(&ss.three)[i] = __ldcg(src + i);
		__syncwarp();
		if (lane == 0)
			rec.handed = 0;
	}
	else
	{
		ThreeSubsetsEstimates<kD, MODE>(st, ss, R, P, sp, team, StageWarpBytes(S, false), lane);
		if (team.rank)
			return false;
		/* sorted: the first ones are below the error */
		int left = 0;
		for (int i = lane; i < ss.three.count; i += 32)
			left += ss.three.order[i].x < R.errTotal;
		left = int(__reduce_add_sync(kFull, unsigned(left)));
		if (hand && left > kInlineCandidates)
		{
			SplitQueue& q = sg.split[SplitIndex(S)];
			int slot = 0;
			if (lane == 0)
				slot = atomicAdd(&q.handedCount, 1);
			slot = __shfl_sync(kFull, slot, 0);
			if (slot < sg.handedCap)
			{
				int* dst = reinterpret_cast<int*>(sg.estimates + slot);
				for (int i = lane; i < int(sizeof(ThreeEstimates) / 4); i += 32)
					dst[i] = reinterpret_cast<const int*>(&ss.three)[i];
				if (lane == 0)
				{
					rec.handed = slot + 1;
					sg.handed[slot] = k;
					sg.start[k] = 0;
					sg.firstImp[k] = kSplitNone;
					sg.pending[k] = SplitTasks(S);
				}
				__syncwarp();
				return true;
			}
		}
		from = 0;
	}
	const int count = ss.three.count;
#pragma unroll 1
	for (int i = from; i < count; i++)
	{
		const int2 o = ss.three.order[i];
		if (o.x < R.errTotal && ThreeSubsetsPartition<kD, MODE>(st, ss, R, P, sp, o.y, lane))
			break;
	}
	return false;
}

/* A pass kernel's block: runs pass S (of a split pass, the partitions from
   `from` on) and records the next one. */
template<int kD, int S>
__device__ void PassStage(WarpState& st, SearchState& ss, const BlockRef& b, const LevelTables& T, const Params& P, const Stages& sg, int k,
	int from, bool hand, Team& team, TeamState* ts, int lane)
{
	CellRegs R;
	BlockRecord& rec = sg.rec[k];
	const int handed = RestoreBlock(st, R, b, rec, P, lane);
	if (TeamStage(S) && team.size > 1)
		__syncthreads();   /* every warp has read the record before it changes */
	if constexpr (ThreeSubsetStep(S))
	{
		if (ThreeSubsetsStage<kD, S>(st, ss, R, P, T, sg, k, handed, from, hand, team, lane))
			return;   /* handed to the tasks */
	}
	else
		RunStep<kD, S>(st, ss, R, P, T, lane, from, team, ts);
	if (team.rank)
		return;
	const int n = NextStep(S, R, P);
	SaveRecord(rec, R, lane);
	if (lane == 0)
		Publish(sg, k, n, R.errTotal, R.bestMode, R.a1.opaque, kD);
	__syncwarp();
}

/* The finish kernel's block. */
template<int kD>
__device__ void FinishStage(WarpState& st, const BlockRef& b, const Params& P, const BlockRecord& rec, int lane)
{
	CellRegs R;
	RestoreBlock(st, R, b, rec, P, lane);
	FinishBlock<kD>(st, R, P, rec.water, rec.startLo, rec.startHi, b, lane);
}

/* Stage STAGE of one block at queue position k; returns whether the block
   finished (its output is written). */
template<int kD, int STAGE>
__device__ __forceinline__ bool StageBlock(WarpState& st, SearchState& ss, const BlockRef& b, const LevelTables& T, const Params& P,
	const Stages& sg, int k, bool hand, Team& team, TeamState* ts, int lane)
{
	if constexpr (STAGE == kStageDraft)
		return DraftStage<kD>(st, b, T, P, sg, k, lane);
	else if constexpr (STAGE == kStepFinish)
	{
		FinishStage<kD>(st, b, P, sg.rec[k], lane);
		return true;
	}
	else
	{
		PassStage<kD, STAGE>(st, ss, b, T, P, sg, k, SplitIndex(STAGE) >= 0 ? sg.start[k] : 0, hand, team, ts, lane);
		return false;
	}
}

/* One stage of a staged encode over a list of queue positions (`list`,
   *count entries, taken through *head): the draft kernel takes every
   position (no list); a pass or the finish kernel takes the positions
   gathered for it.  kD as for KEncode. */
template<int kD, int STAGE>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 4) KEncodeStage(Job job, Stages sg, const int* list, const int* count, int* head,
	LevelTables T0, LevelTables T1)
{
	extern __shared__ __align__(16) unsigned char encodeSmem[];
	const int lane = threadIdx.x & 31;
	const int warp = threadIdx.x >> 5;
	WarpState& st = *reinterpret_cast<WarpState*>(encodeSmem + warp * StageWarpBytes(STAGE, false));
	SearchState& ss = *reinterpret_cast<SearchState*>(reinterpret_cast<unsigned char*>(&st) + kSearchWarpBytes);
	__shared__ LevelTables tables[2];
	__shared__ TeamState ts;
	WaitForLaunch();
	const int n = list ? *count : job.total;
	if (n == 0)
		return;
	ShareTables(tables, T0, T1);
	/* the first blocks of a list a CTA each (TeamBlocks), the others a warp each */
	const int nTeam = TeamStage(STAGE) ? TeamBlocks(STAGE, n, sg.count[kNumStages], int(gridDim.x)) : 0;
	Team team{ nTeam > 0 ? kWarpsPerCta : 1, nTeam > 0 ? warp : 0, &ts.exchange, 0 };
	for (;;)
	{
		int i = 0;
		if (team.rank == 0 && lane == 0)
			i = atomicAdd(head, 1);
		if (TeamStage(STAGE) && team.size > 1)
		{
			__syncthreads();
			if (threadIdx.x == 0)
				ts.task[0] = i;
			__syncthreads();
			i = ts.task[0];
			if (i >= nTeam)
			{
				/* every warp for itself from here; the first has a block already */
				team = SingleWarp();
				if (warp && lane == 0)
					i = atomicAdd(head, 1);
				i = __shfl_sync(kFull, i, 0);
			}
		}
		else
			i = __shfl_sync(kFull, i, 0);
		if (i >= n)
			break;
		const int k = list ? list[i] : i;
		TexDesc d;
		BlockRef b;
		QueuedBlock(job, k, d, b);
		const Params& P = SharedParams(st, d, lane);
		bool finished;
		if constexpr (kD == kAnyDenoise)
		{
			if (d.denoise)
				finished = StageBlock<1, STAGE>(st, ss, b, tables[1], P, sg, k, n <= kHandOverBlocks, team, &ts, lane);
			else
				finished = StageBlock<0, STAGE>(st, ss, b, tables[0], P, sg, k, n <= kHandOverBlocks, team, &ts, lane);
		}
		else
			finished = StageBlock<kD, STAGE>(st, ss, b, tables[kD], P, sg, k, n <= kHandOverBlocks, team, &ts, lane);
		if (finished)
			BlockFinished(d, lane);
	}
}

/* One task of a split pass: candidate p of the block at position k,
   searched from the error in its record (the error at the start of the
   round).  An improving candidate before the round's first improvement so
   far keeps its result and lowers the block's firstImp; a candidate after
   it is not searched (the next round searches it again).  N warps of the CTA
   run the task together (mode 7: its four). */
template<int kD, int S, int N>
__device__ NEBC7_PASS void SplitTask(WarpState& st, SearchState& ss, TeamState* ts, const BlockRef& b, const LevelTables& T, const Params& P,
	const Stages& sg, SplitQueue& q, int k, int p, int first, int rank, int lane)
{
	constexpr int MODE = SplitMode(S);
	if ((first >> kSplitSlotBits) < p)
		return;
	CellRegs R;
	RestoreBlock(st, R, b, sg.rec[k], P, lane);
	const int E = R.errTotal, step = R.denoiseStep;
	bool end;
	int param = p;
	Team one = SingleWarp();
	/* the conditions of the candidate loops (FullTwoSubsets, FullMode7, FullRot) */
	if constexpr (MODE == 4 || MODE == 5)
	{
		const int rotation = MODE == 4 ? c_rot4[p] : c_rot5[p];
		if (MODE == 4 && R.personalMode == 4 && !((R.personalParam ^ rotation) & 3))
			return;
		if (MODE == 5 && R.personalMode == 5 && R.personalParam == rotation)
			return;
		Ep mc = 0;
		int error = step;
		if (error < E)
			error += CompressRotSubset<kD, MODE>(st, ss, R, P, T, mc, E - error, rotation, one, nullptr, lane);
		if (!(E > error))
			return;
		R.errTotal = error - step;
		R.best[0] = mc;
		end = error <= step;
		param = rotation;
	}
	else if constexpr (MODE == 0 || MODE == 2)
	{
		/* candidate p of the sorted estimates */
		const ThreeEstimates& from = sg.estimates[__ldcg(&sg.rec[k].handed) - 1];
		if (p >= __ldcg(&from.count))
			return;
		const int2 o = __ldcg(&from.order[p]);
		if (!(o.x < E))
			return;
		param = o.y;
		if (lane < 9)
			(&ss.three.est[param][0][0])[lane] = __ldcg(&from.est[param][0][0] + lane);
		else if (lane < 11)
			ss.three.lines[param][lane - 9] = __ldcg(&from.lines[param][lane - 9]);
		__syncwarp();
		end = ThreeSubsetsPartition<kD, MODE>(st, ss, R, P, GetSpec3(MODE, T), param, lane);
		if (R.errTotal == E)
			return;
	}
	else
	{
		if (R.personalMode == MODE && R.personalParam == p)
			return;
		if constexpr (MODE == 7)
		{
			if (!(0 < E - step) || !(step < E))
				return;
			if constexpr (N == 1)
				end = Mode7Partition<kD>(st, ss, R, P, T, p, 0, 0, lane);
			else
				end = Mode7PartitionTeam<kD>(st, ss, *ts, StageWarpBytes(S, true), R, P, T, p, rank, lane);
		}
		else
		{
			const int OA = R.opaqueAlphaError;
			if (!(0 < E - step - OA) || !(OA + step < E))
				return;
			end = TwoSubsetsPartition<kD, MODE>(st, ss, R, P, GetSpec3(MODE, T), p, 0, 0, lane);
		}
		if (R.errTotal == E)
			return;
	}
	if (rank != 0 || lane != 0 || (*reinterpret_cast<volatile int*>(sg.firstImp + k) >> kSplitSlotBits) < p)
		return;
	int slot = kSplitNoSlot;
	const int at = atomicAdd(&q.kept, 1);
	if (at < sg.impCap)
	{
		SplitResult r;
		r.best0 = R.best[0];
		r.best1 = R.best[1];
		r.best2 = R.best[2];
		r.error = R.errTotal;
		r.end = end;
		r.param = param;
		r.pad[0] = r.pad[1] = r.pad[2] = 0;
		sg.imp[at] = r;
		slot = at;
	}
	/* the result before the word that leads to it */
	__threadfence();
	atomicMin(sg.firstImp + k, (p << kSplitSlotBits) | slot);
}

/* Whether candidate p of the block at position k can improve on the error at
   the start of the round, as far as the line bound tells (mode 7). */
template<int kD, int S>
__device__ NEBC7_PASS bool SplitOpen(WarpState& st, const BlockRef& b, const Params& P, const Stages& sg, int k, int p, int lane)
{
	if constexpr (SplitMode(S) == 7)
	{
		CellRegs R;
		RestoreBlock(st, R, b, sg.rec[k], P, lane);
		return !(R.personalMode == 7 && R.personalParam == p) && Mode7Open<kD>(st, R, P, p, lane);
	}
	return true;
}

/* The end of a block's round of split pass S (one thread, after its last
   task): the first improving candidate f becomes the block's best and ends
   the pass, or the block goes on from f + 1 in a later round with the new
   error; a block without an improvement has finished the pass and gets its
   next one (NextStep).  Blocks whose result was not kept, and those that
   must run whole, are left to the one-warp remainder. */
template<int S>
__device__ __forceinline__ void SplitCommit(const Job& job, const Stages& sg, SplitQueue& q, int k)
{
	constexpr int MODE = SplitMode(S), NT = SplitTasks(S);
	const int f = *reinterpret_cast<volatile int*>(sg.firstImp + k);
	BlockRecord& r = sg.rec[k];
	int from = -1;
	bool rest = false;
	if (f == kSplitSerial)
	{
		from = 0;
		rest = true;
	}
	else if (f != kSplitNone)
	{
		const int p = f >> kSplitSlotBits, slot = f & kSplitNoSlot;
		if (slot >= sg.impCap)
		{
			from = p;   /* its result was not kept: search it again */
			rest = true;
		}
		else
		{
			const uint4* e = reinterpret_cast<const uint4*>(sg.imp + slot);
			SplitResult v;
#pragma unroll
			for (int i = 0; i < int(sizeof(SplitResult) / 16); i++)
				reinterpret_cast<uint4*>(&v)[i] = __ldcg(e + i);
			r.errTotal = v.error;
			r.best[0] = v.best0;
			if (MODE != 4 && MODE != 5)
				r.best[1] = v.best1;
			if (MODE == 0 || MODE == 2)
				r.best[2] = v.best2;
			r.bestParam = v.param;
			r.bestMode = MODE;
			if (!v.end && p < NT - 1)
				from = p + 1;
		}
	}
	if (from >= 0)
	{
		sg.start[k] = from;
		sg.firstImp[k] = kSplitNone;
		sg.pending[k] = NT - from;
		const int at = rest ? sg.laterCap : atomicAdd(&q.laterReserve, 1);
		if (at < sg.laterCap)
		{
			sg.later[at] = k;
			/* published in order: the entries before it are being published by
			   running warps; should that take seconds, the block (and those
			   behind it) goes to the remainder */
			__threadfence();
			for (int tries = 0; tries < kSplitPolls; tries++)
			{
				if (atomicCAS(&q.laterTail, at, at + 1) == at)
					return;
				__nanosleep(500);
			}
		}
		sg.rest[atomicAdd(&q.restCount, 1)] = k;
	}
	else
	{
		const BlockRecord now = r;
		TexDesc d;
		BlockRef b;
		QueuedBlock(job, k, d, b);
		CellRegs R;
		R.errTotal = now.errTotal;
		R.opaqueAlphaError = now.opaqueAlphaError;
		R.denoiseStep = now.denoiseStep;
		R.a1.opaque = now.opaque != 0;
		r.handed = 0;
		Publish(sg, k, NextStep(S, R, d.P), now.errTotal, now.bestMode, now.opaque != 0, now.denoise);
	}
	__threadfence();
	atomicAdd(&q.finished, 1);
}

/* The next task (one thread): of a later round if there is one, else of the
   first round (n blocks); waits while blocks of either are still running.
   firstRound: whether the caller has found no end of the first round yet.
   Returns the task's entry * NT + candidate, the later rounds' entries after
   the first round's n, or -1. */
template<int S>
__device__ __forceinline__ long long SplitTake(const Stages& sg, SplitQueue& q, int n, bool& firstRound, int grab = 1)
{
	constexpr int NT = SplitTasks(S);
	for (int polls = 0; polls < kSplitPolls;)
	{
		int4 s;
		asm volatile("ld.volatile.global.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(s.x), "=r"(s.y), "=r"(s.z), "=r"(s.w) : "l"(&q) : "memory");
		/* laterHead counts tasks, laterTail entries */
		if (s.x < s.y * NT)
		{
			if (atomicCAS(&q.laterHead, s.x, s.x + 1) == s.x)
			{
				__threadfence();   /* the block's record and start after the entry */
				return (long long)n * NT + s.x;
			}
			continue;
		}
		if (firstRound)
		{
			/* `grab` first-round tasks from here (NT is a multiple of it) */
			const int t = atomicAdd(&q.head, grab);
			if (t < n * NT)
				return t;
			firstRound = false;
		}
		if (s.z >= n)
			break;
		__nanosleep(2000);
		polls++;
	}
	return -1;
}

/* Warps of a CTA that run a task of split pass S together. */
__host__ __device__ constexpr int SplitTeam(int S)
{
	return S == kStepMode7 ? kWarpsPerCta : 1;
}

/* From this many blocks on, a team takes four mode 7 candidates at a time, whose
   bounds its warps compute beside each other: three of four candidates end
   there (1118x1105 alpha texture, 3455 blocks: 13.5 -> 11.4 ms).  A shorter list
   would leave CTAs without a task while others search four in turn.  Whole
   encodes of alpha textures one and four at a time: 64x64 5.5 and 5.9 ms, 256x256
   13.8 and 15.2, 512x512 21.7 and 20.4, 1024x1024 32.9 and 31.3; /slow 256x256
   15.6 and 17.0, 512x512 24.1 and 22.6. */
constexpr int kGrabBlocks = 1024;

/* Split pass S over the blocks list[i], i < *count (at most kSplitMaxBlocks).
   The tasks (block, candidate p) are taken block by block, so that the
   candidates of a block go to as many warps; a block's last task commits the
   round, and the next round's tasks are taken as soon as it has: the rounds
   of the hard blocks, whose tasks come first, run beside the other blocks'
   first round. */
template<int kD, int S>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 4) KEncodeSplit(Job job, Stages sg, const int* list, const int* count, LevelTables T0,
	LevelTables T1)
{
	constexpr int NT = SplitTasks(S), N = SplitTeam(S);
	extern __shared__ __align__(16) unsigned char encodeSmem[];
	__shared__ TeamState ts;
	const int lane = threadIdx.x & 31;
	const int warp = threadIdx.x >> 5;
	WarpState& st = *reinterpret_cast<WarpState*>(encodeSmem + warp * StageWarpBytes(S, true));
	SearchState& ss = *reinterpret_cast<SearchState*>(reinterpret_cast<unsigned char*>(&st) + kSearchWarpBytes);
	__shared__ LevelTables tables[2];
	SplitQueue& q = sg.split[SplitIndex(S)];
	WaitForLaunch();
	const int n = min(*count, ThreeSubsetStep(S) ? sg.handedCap : kSplitMaxBlocks);
	if (n == 0)
		return;
	ShareTables(tables, T0, T1);
	const int rank = N > 1 ? warp : 0;   /* within the task's warps */
	const int grab = N > 1 && n >= kGrabBlocks ? N : 1;
	bool firstRound = true;
	/* task t: the block's position k and candidate p (-1 if the round starts
	   after it), and the first improvement so far */
	auto task = [&](long long t, int& k, int& p, int& first) {
		const long long e = t / NT;
		p = int(t % NT);
		k = e < n ? list[e] : *reinterpret_cast<volatile int*>(sg.later + (e - n));
		if (p < *reinterpret_cast<volatile int*>(sg.start + k))
			p = -1;
		first = *reinterpret_cast<volatile int*>(sg.firstImp + k);
	};
	for (;;)
	{
		int k = -1, p = 0, first = 0, count = 1;
		if (rank == 0 && lane == 0)
		{
			const long long t = SplitTake<S>(sg, q, n, firstRound, grab);
			if (t >= 0)
				task(t, k, p, first);
			if (N > 1)
				count = grab > 1 && t >= 0 && t < (long long)n * NT ? grab : 1;
		}
		if (N > 1)
		{
			__syncthreads();   /* the last task's shared state is read */
			if (threadIdx.x == 0)
			{
				/* one read of the first improvement for all the task's warps:
				   other warps lower it meanwhile */
				ts.task[0] = k;
				ts.task[1] = p;
				ts.task[2] = first;
				ts.task[3] = count;
			}
			__syncthreads();
			k = ts.task[0];
			p = ts.task[1];
			first = ts.task[2];
			count = ts.task[3];
		}
		else
		{
			k = __shfl_sync(kFull, k, 0);
			p = __shfl_sync(kFull, p, 0);
			first = __shfl_sync(kFull, first, 0);
		}
		if (k < 0)
			break;
		if (p < 0 && count == 1)
			continue;
		TexDesc d;
		BlockRef b;
		QueuedBlock(job, k, d, b);
		const Params& P = SharedParams(st, d, lane);
		if (P.pca && (SplitMode(S) & 1) && SplitMode(S) != 5)
		{
			/* OPTION_PCA orders the partitions by their bounds first: the
			   pass runs whole, in one warp */
			if (rank == 0 && lane == 0)
				sg.firstImp[k] = kSplitSerial;
			first = kSplitSerial;
			__syncwarp();
		}
		/* of several tasks (of one block, from candidate p on), each warp
		   looks whether one is open */
		unsigned open = 1;
		if (N > 1 && count > 1)
		{
			bool mine = false;
			if ((first >> kSplitSlotBits) >= p + warp)
			{
				if constexpr (kD == kAnyDenoise)
				{
					if (d.denoise)
						mine = SplitOpen<1, S>(st, b, P, sg, k, p + warp, lane);
					else
						mine = SplitOpen<0, S>(st, b, P, sg, k, p + warp, lane);
				}
				else
					mine = SplitOpen<kD, S>(st, b, P, sg, k, p + warp, lane);
			}
			if (lane == 0)
				ts.open[warp] = mine;
			__syncthreads();
			open = 0;
			for (int j = 0; j < N; j++)
				open |= unsigned(ts.open[j]) << j;
		}
		else if (first == kSplitSerial)
			open = 0;
		while (open)
		{
			const int at = p + __ffs(open) - 1;
			open &= open - 1;
			if constexpr (kD == kAnyDenoise)
			{
				if (d.denoise)
					SplitTask<1, S, N>(st, ss, &ts, b, tables[1], P, sg, q, k, at, first, rank, lane);
				else
					SplitTask<0, S, N>(st, ss, &ts, b, tables[0], P, sg, q, k, at, first, rank, lane);
			}
			else
				SplitTask<kD, S, N>(st, ss, &ts, b, tables[kD], P, sg, q, k, at, first, rank, lane);
			/* every warp of a team has read the block's record before its round
			   can end and change it, and the task's shared state */
			if (N > 1)
				__syncthreads();
			else
				__syncwarp();
		}
		if (rank == 0 && lane == 0)
		{
			__threadfence();
			if (atomicSub(sg.pending + k, count) == count)
			{
				__threadfence();
				SplitCommit<S>(job, sg, q, k);
			}
		}
		__syncwarp();
	}
}

/* Gathers the positions whose next pass is `stage` into its list, bucket by
   bucket (StageBucket), and their number; for a split pass (tasks per block
   NT > 0) the blocks start at candidate 0, and those past kSplitMaxBlocks
   (more than the task count can number) go to the remainder at once. */
static __global__ void __launch_bounds__(1024) KStageList(Stages sg, int stage, int splitIndex, int NT)
{
	__shared__ int base[256];
	const int lane = threadIdx.x & 31;
	WaitForLaunch();
	if (threadIdx.x < 32)
	{
		/* exclusive scan of the bucket counts: 8 per lane, then the lanes */
		int c[8], run = 0;
#pragma unroll
		for (int j = 0; j < 8; j++)
		{
			c[j] = run;
			run += sg.hist[stage * 256 + lane * 8 + j];
		}
		int incl = run;
		for (int o = 1; o < 32; o <<= 1)
		{
			const int v = __shfl_up_sync(kFull, incl, o);
			if (lane >= o)
				incl += v;
		}
#pragma unroll
		for (int j = 0; j < 8; j++)
			base[lane * 8 + j] = incl - run + c[j];
		__syncwarp();   /* the first lane's entries before the mark of an empty list */
		if (blockIdx.x == 0 && lane == 31)
			sg.count[stage] = incl;
		if (stage == kStepRefine && blockIdx.x == 0 && lane == kRefineHeavy / 8)
			sg.count[kNumStages] = base[kRefineHeavy];
		if (lane == 31 && incl == 0)
			base[0] = -1;
	}
	__syncthreads();
	if (base[0] < 0)
		return;
	for (int k = blockIdx.x * 1024 + threadIdx.x; k < sg.total; k += gridDim.x * 1024)
	{
		if (sg.next[k] != stage)
			continue;
		const int b = StageBucket(sg, stage, k, sg.rec[k].errTotal, sg.rec[k].bestMode, sg.rec[k].opaque != 0, sg.rec[k].denoise);
		const int at = base[b] + atomicAdd(&sg.cursor[stage * 256 + b], 1);
		sg.list[at] = k;
		if (NT)
		{
			sg.start[k] = 0;
			sg.firstImp[k] = kSplitNone;
			sg.pending[k] = NT;
			if (at >= kSplitMaxBlocks)
				sg.rest[atomicAdd(&sg.split[splitIndex].restCount, 1)] = k;
		}
	}
}

/* Host-side launcher of a staged encode: the draft kernel, then for each
   pass its list and its kernel, then the finish kernel's list and kernel; chain:
   as programmatic dependents (WaitForLaunch).  The launches are capturable.  Compiled per kD in encode_*_staged.cu. */
template<int kD>
cudaError_t LaunchStagedEncode(int grid, cudaStream_t stream, const Job& job, const Stages& sg, bool slow, bool chain,
	const LevelTables& T0, const LevelTables& T1);

/* Raises the stage kernels' dynamic shared-memory limit (once per process
   and device, before the first launch) and reports CTAs per SM. */
template<int kD>
cudaError_t StagedEncodeOccupancy(int* ctasPerSm);

/* Bytes of the per-position state of a staged encode of n positions
   (records, next-pass words, the pass list, the split passes' words, later
   rounds and kept results; 256-byte aligned pieces), after kStagedZeroed bytes
   of counts, queues and histograms that must be zero before each launch. */
constexpr size_t kStagedZeroed = 256 + kSplitPasses * sizeof(SplitQueue) + 2 * size_t(kNumStages) * 1024;
static_assert(kStagedZeroed % 256 == 0 && kNumStages < 32, "the counts and queue heads take 128 bytes each");

/* Spare entries past one a block in the rooms of a large launch: all that the
   blocks a pass hands over can ask for. */
constexpr size_t kSplitSpare = size_t(kHandedBlocks) * kSplitMaxTasks;

constexpr size_t LeastOf(size_t a, size_t b, size_t c)
{
	return a < b ? (a < c ? a : c) : (b < c ? b : c);
}

/* Results a pass keeps: three a block of a small launch, one of a large one
   (noise and two-colour blocks keep up to 0.65 a block in a pass of modes 1, 3, 4
   or 5, photos and alpha textures 0.005; the blocks handed over by modes 2 and 0
   up to 4 each).  A slot has to fit its field of a firstImp word, below the mark:
   with more room than that, results past 2^24 ran into the candidate's bits and
   another block's was taken for them.  What finds no slot is searched again by
   the remainder. */
constexpr size_t SplitResultCap(int n)
{
	return LeastOf(3 * size_t(n) + 1024, size_t(n) + kSplitSpare, size_t(kSplitNoSlot));
}

static_assert(SplitResultCap(0x7FFFFFFF) == size_t(kSplitNoSlot) && kSplitMaxTasks << kSplitSlotBits <= kSplitNone,
	"candidates and slots fit a firstImp word");

/* Entries of a pass's later rounds (up to 0.45 a block in those textures); their
   tasks stay an int. */
constexpr size_t SplitLaterCap(int n)
{
	return LeastOf(4 * size_t(n) + 1024, size_t(n) + kSplitSpare, size_t(1) << 24);
}

constexpr size_t HandedCap(int n)
{
	return n < kHandedBlocks ? n : kHandedBlocks;
}

constexpr size_t StagedAlign(size_t v) { return (v + 255) & ~size_t(255); }

constexpr size_t StagedScratchBytes(int n)
{
	return kStagedZeroed + StagedAlign(size_t(n) * sizeof(BlockRecord)) + StagedAlign(size_t(n) * 4) * 6 + StagedAlign(SplitLaterCap(n) * 4) +
		StagedAlign(SplitResultCap(n) * sizeof(SplitResult)) + StagedAlign(HandedCap(n) * 4) + HandedCap(n) * sizeof(ThreeEstimates);
}

/* Splits a staged scratch (256-byte aligned, StagedScratchBytes(n) bytes). */
inline Stages SplitStaged(uint8_t* p, int n, bool mixed)
{
	Stages s;
	s.count = (int*)p;
	s.counters = (int*)(p + 128);
	s.split = (SplitQueue*)(p + 256);
	s.hist = (int*)(p + 256 + kSplitPasses * sizeof(SplitQueue));
	s.cursor = s.hist + kNumStages * 256;
	s.total = n;
	s.mixed = mixed;
	s.rec = (BlockRecord*)(p + kStagedZeroed);
	uint8_t* q = p + kStagedZeroed + StagedAlign(size_t(n) * sizeof(BlockRecord));
	const size_t ints = StagedAlign(size_t(n) * 4);
	s.next = (int*)q;
	s.list = (int*)(q + ints);
	s.start = (int*)(q + 2 * ints);
	s.firstImp = (int*)(q + 3 * ints);
	s.pending = (int*)(q + 4 * ints);
	s.rest = (int*)(q + 5 * ints);
	s.later = (int*)(q + 6 * ints);
	s.laterCap = int(SplitLaterCap(n));
	s.imp = (SplitResult*)(q + 6 * ints + StagedAlign(SplitLaterCap(n) * 4));
	s.impCap = int(SplitResultCap(n));
	uint8_t* h = (uint8_t*)s.imp + StagedAlign(SplitResultCap(n) * sizeof(SplitResult));
	s.handed = (int*)h;
	s.estimates = (ThreeEstimates*)(h + StagedAlign(HandedCap(n) * 4));
	s.handedCap = int(HandedCap(n));
	return s;
}

} // namespace nebc7
