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

/* Launches a kernel of the staged form; chain: as the programmatic dependent
   of the one before it (WaitForLaunch). */
template<class... P, class... A>
cudaError_t LaunchChained(void (*kernel)(P...), bool chain, int grid, int threads, size_t smem, cudaStream_t stream, const A&... args)
{
	cudaLaunchAttribute chained = {};
	chained.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	chained.val.programmaticStreamSerializationAllowed = 1;
	cudaLaunchConfig_t config = {};
	config.gridDim = dim3(grid);
	config.blockDim = dim3(threads);
	config.dynamicSmemBytes = smem;
	config.stream = stream;
	config.attrs = &chained;
	config.numAttrs = chain ? 1 : 0;
	return cudaLaunchKernelEx(&config, kernel, P(args)...);
}

/* The list of pass STAGE and its kernels: of a split pass the tasks, of a
   three-subset pass its estimates and the tasks of the blocks they hand over;
   then a split pass's blocks that must run whole (OPTION_PCA, results not
   kept), in one warp each from their start candidates. */
template<int kD, int STAGE>
cudaError_t LaunchStage(int grid, cudaStream_t stream, const Job& job, const Stages& sg, bool chain, const LevelTables& T0,
	const LevelTables& T1)
{
	constexpr int split = SplitIndex(STAGE), threads = kWarpsPerCta * 32;
	constexpr bool three = ThreeSubsetStep(STAGE), draft = STAGE == kStageDraft;
	cudaError_t e = cudaSuccess;
	if (!draft)
	{
		const int ctas = (job.total + 1023) / 1024;
		e = LaunchChained(KStageList, chain, ctas < 152 ? ctas : 152, 1024, 0, stream, sg, STAGE, split, split >= 0 && !three ? SplitTasks(STAGE) : 0);
	}
	const int stageGrid = StageGrid(grid, job.total, TeamStage(STAGE) ? kWarpsPerCta : 1);
	if constexpr (split < 0 || three)
	{
		if (e == cudaSuccess)
			e = LaunchChained(KEncodeStage<kD, STAGE>, chain, stageGrid, threads, StageSharedBytes(STAGE, false), stream, job, sg,
				draft ? nullptr : sg.list, draft ? nullptr : sg.count + STAGE, sg.counters + (STAGE + 1), T0, T1);
	}
	if constexpr (split >= 0)
	{
		/* a small texture's tasks fill more SMs than its blocks */
		const int blocks = three ? sg.handedCap : job.total;
		if (e == cudaSuccess)
			e = LaunchChained(KEncodeSplit<kD, STAGE>, chain, StageGrid(grid, (long long)blocks * SplitTasks(STAGE), SplitTeam(STAGE)), threads,
				StageSharedBytes(STAGE, true), stream, job, sg, three ? sg.handed : sg.list,
				three ? &sg.split[split].handedCount : sg.count + STAGE, T0, T1);
		if (e == cudaSuccess)
			e = LaunchChained(KEncodeStage<kD, STAGE>, chain, stageGrid, threads, StageSharedBytes(STAGE, false), stream, job, sg, sg.rest,
				&sg.split[split].restCount, &sg.split[split].restHead, T0, T1);
	}
	return e;
}

/* The passes from STAGE on. */
template<int kD, int STAGE>
cudaError_t LaunchStagesFrom(int grid, cudaStream_t stream, const Job& job, const Stages& sg, bool slow, bool chain,
	const LevelTables& T0, const LevelTables& T1)
{
	if constexpr (STAGE < kNumStages)
	{
		if (StageLaunched(STAGE, slow))
			if (const cudaError_t e = LaunchStage<kD, STAGE>(grid, stream, job, sg, chain, T0, T1))
				return e;
		return LaunchStagesFrom<kD, STAGE + 1>(grid, stream, job, sg, slow, chain, T0, T1);
	}
	return cudaSuccess;
}

template<int kD>
cudaError_t LaunchStagedEncode(int grid, cudaStream_t stream, const Job& job, const Stages& sg, bool slow, bool chain,
	const LevelTables& T0, const LevelTables& T1)
{
	return LaunchStagesFrom<kD, kStageDraft>(grid, stream, job, sg, slow, chain, T0, T1);
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
	/* every stage kernel is compiled for four CTAs per SM, and the 7.6 to 53 KB
	   of shared memory that one takes leave room for them */
	return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctasPerSm, KEncodeStage<kD, kStepFull3Mode2>, kWarpsPerCta * 32,
		StageSharedBytes(kStepFull3Mode2, false));
}

} // namespace nebc7

#define NEBC7_INSTANTIATE_STAGED(KD) \
	template cudaError_t nebc7::LaunchStagedEncode<KD>(int, cudaStream_t, const nebc7::Job&, const nebc7::Stages&, bool, bool, \
		const nebc7::LevelTables&, const nebc7::LevelTables&); \
	template cudaError_t nebc7::StagedEncodeOccupancy<KD>(int*);
