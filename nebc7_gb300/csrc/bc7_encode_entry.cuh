/*
 * Definitions of the KEncode launchers declared in bc7_encode.cuh; included
 * by the per-instantiation translation units only.
 */
#pragma once

#include "bc7_encode.cuh"

namespace nebc7 {

/* Lets the kernel use more than the default 48 KB of dynamic shared memory
   (once per process and device; idempotent). */
template<int kD, bool NORMAL>
cudaError_t PrepareEncodeKernel()
{
	return cudaFuncSetAttribute(KEncode<kD, NORMAL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		int(EncodeSharedBytes<NORMAL>()));
}

template<int kD, bool NORMAL>
cudaError_t LaunchEncodeKernel(int grid, cudaStream_t stream, const Job& job, const LevelTables& T0, const LevelTables& T1)
{
	KEncode<kD, NORMAL><<<grid, kWarpsPerCta * 32, EncodeSharedBytes<NORMAL>(), stream>>>(job, T0, T1);
	return cudaGetLastError();
}

template<int kD, bool NORMAL>
cudaError_t EncodeKernelOccupancy(int* ctasPerSm)
{
	const cudaError_t e = PrepareEncodeKernel<kD, NORMAL>();
	if (e != cudaSuccess)
		return e;
	return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctasPerSm, KEncode<kD, NORMAL>, kWarpsPerCta * 32,
		EncodeSharedBytes<NORMAL>());
}

} // namespace nebc7

#define NEBC7_INSTANTIATE_ENCODE(KD, NORMAL) \
	template cudaError_t nebc7::LaunchEncodeKernel<KD, NORMAL>(int, cudaStream_t, const nebc7::Job&, \
		const nebc7::LevelTables&, const nebc7::LevelTables&); \
	template cudaError_t nebc7::EncodeKernelOccupancy<KD, NORMAL>(int*);
