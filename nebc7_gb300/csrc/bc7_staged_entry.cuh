/*
 * Definitions of the staged-encode launchers declared in bc7_staged.cuh;
 * included by the per-kDenoise translation units only.
 */
#pragma once

#include "bc7_staged.cuh"

namespace nebc7 {

/* CTAs for `tasks` tasks of `warps` warps each, at least one and at most `grid`
   (the resident ones). */
inline int StageGrid(int grid, long long tasks, int warps)
{
	const long long ctas = (tasks * warps + kWarpsPerCta - 1) / kWarpsPerCta;
	return ctas < 1 ? 1 : (ctas < grid ? int(ctas) : grid);
}

/* The list of pass STAGE and its kernels: of a split pass the tasks, of a
   three-subset pass its estimates and the tasks of the blocks they hand over;
   then a split pass's blocks that must run whole (OPTION_PCA, results not
   kept), in one warp each from their start candidates. */
template<int kD, int STAGE>
cudaError_t LaunchStage(int grid, cudaStream_t stream, const Job& job, const Stages& sg, const LevelTables& T0, const LevelTables& T1)
{
	constexpr int split = SplitIndex(STAGE);
	constexpr bool three = ThreeSubsetStep(STAGE);
	if (STAGE != kStageDraft)
	{
		const int ctas = (job.total + 1023) / 1024;
		KStageList<<<ctas < 152 ? ctas : 152, 1024, 0, stream>>>(sg, STAGE, split, split >= 0 && !three ? SplitTasks(STAGE) : 0);
	}
	const int stageGrid = StageGrid(grid, job.total, TeamStage(STAGE) ? kWarpsPerCta : 1);
	if constexpr (split < 0 || three)
	{
		const bool all = STAGE == kStageDraft;
		KEncodeStage<kD, STAGE><<<stageGrid, kWarpsPerCta * 32, StageSharedBytes(STAGE, false), stream>>>(job, sg, all ? nullptr : sg.list,
			all ? nullptr : sg.count + STAGE, sg.counters + (STAGE + 1), T0, T1);
	}
	if constexpr (split >= 0)
	{
		/* a small texture's tasks fill more SMs than its blocks */
		const int blocks = three ? sg.handedCap : job.total;
		KEncodeSplit<kD, STAGE><<<StageGrid(grid, (long long)blocks * SplitTasks(STAGE), SplitTeam(STAGE)), kWarpsPerCta * 32,
			StageSharedBytes(STAGE, true), stream>>>(job, sg, three ? sg.handed : sg.list, three ? &sg.split[split].handedCount : sg.count + STAGE,
			T0, T1);
		KEncodeStage<kD, STAGE><<<stageGrid, kWarpsPerCta * 32, StageSharedBytes(STAGE, false), stream>>>(job, sg, sg.rest,
			&sg.split[split].restCount, &sg.split[split].restHead, T0, T1);
	}
	return cudaGetLastError();
}

/* The passes from STAGE on. */
template<int kD, int STAGE>
cudaError_t LaunchStagesFrom(int grid, cudaStream_t stream, const Job& job, const Stages& sg, bool slow, const LevelTables& T0,
	const LevelTables& T1)
{
	if constexpr (STAGE < kNumStages)
	{
		if (StageLaunched(STAGE, slow))
			if (const cudaError_t e = LaunchStage<kD, STAGE>(grid, stream, job, sg, T0, T1))
				return e;
		return LaunchStagesFrom<kD, STAGE + 1>(grid, stream, job, sg, slow, T0, T1);
	}
	return cudaSuccess;
}

template<int kD>
cudaError_t LaunchStagedEncode(int grid, cudaStream_t stream, const Job& job, const Stages& sg, bool slow, const LevelTables& T0,
	const LevelTables& T1)
{
	return LaunchStagesFrom<kD, kStageDraft>(grid, stream, job, sg, slow, T0, T1);
}

template<int kD, int STAGE>
cudaError_t PrepareStage()
{
	const cudaError_t e = cudaFuncSetAttribute(KEncodeStage<kD, STAGE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		int(StageSharedBytes(STAGE, false)));
	if constexpr (SplitIndex(STAGE) >= 0)
		if (e == cudaSuccess)
			return cudaFuncSetAttribute(KEncodeSplit<kD, STAGE>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(StageSharedBytes(STAGE, true)));
	return e;
}

template<int kD, int STAGE>
cudaError_t PrepareStagesFrom()
{
	if constexpr (STAGE < kNumStages)
	{
		if (const cudaError_t e = PrepareStage<kD, STAGE>())
			return e;
		return PrepareStagesFrom<kD, STAGE + 1>();
	}
	return cudaSuccess;
}

template<int kD>
cudaError_t StagedEncodeOccupancy(int* ctasPerSm)
{
	const cudaError_t e = PrepareStagesFrom<kD, kStageDraft>();
	if (e != cudaSuccess)
		return e;
	/* every stage kernel has the refining kernel's shared memory and bounds */
	return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctasPerSm, KEncodeStage<kD, kStepFull3Mode2>, kWarpsPerCta * 32,
		StageSharedBytes(kStepFull3Mode2, false));
}

} // namespace nebc7

#define NEBC7_INSTANTIATE_STAGED(KD) \
	template cudaError_t nebc7::LaunchStagedEncode<KD>(int, cudaStream_t, const nebc7::Job&, const nebc7::Stages&, bool, \
		const nebc7::LevelTables&, const nebc7::LevelTables&); \
	template cudaError_t nebc7::StagedEncodeOccupancy<KD>(int*);
