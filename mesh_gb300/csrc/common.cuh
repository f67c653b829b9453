// Shared infrastructure of the sm_103a library: status codes, the per-context
// state (device, stream, FP64 reduction scratch), launch sizing.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <memory>
#include <stdexcept>
#include <string>

#include "../../include/mesh_gb300.h"

namespace meshgb {

// Error carrying a C-ABI status code; every extern "C" entry point catches it
// and returns the code (no exception crosses the ABI).
struct Error : std::runtime_error
{
	int code;
	Error(int c, std::string const &m) : std::runtime_error(m), code(c) {}
};

inline void cuda_check(cudaError_t e, char const *what)
{
	if (e != cudaSuccess)
		throw Error(MESH_ERR_CUDA, std::string("cuda error: ") + what + ": " + cudaGetErrorString(e));
}
#define MESH_CUDA(x) ::meshgb::cuda_check((x), #x)
#define MESH_LAUNCH_CHECK() ::meshgb::cuda_check(cudaGetLastError(), "kernel launch")

inline void require(bool ok, char const *msg, int code = MESH_ERR_ARG)
{
	if (!ok)
		throw Error(code, msg);
}

// Number of FP64 reduction slots a context owns; slots are used for the
// scalars of one HMC trajectory (S_old, S_new, K_old, K_new, ...) and by the
// synchronous one-off reductions.
constexpr int kSlots = 64;
// Last-block counters: one per slot, then those of launches with several sums.
constexpr int kCounters = 2 * kSlots;
// Maximum number of blocks of one reduction launch (partials per slot).
constexpr int kMaxRedBlocks = 4096;

struct Context
{
	// owners: the caller's handle plus every field and chain created on it;
	// the context is torn down when the last one is released
	int refs = 1;
	int device = 0;
	cudaStream_t stream = nullptr;
	bool own_stream = false;
	int num_sms = 0;
	// reduction scratch: partials [kSlots][kMaxRedBlocks] (double),
	// results [kSlots] (double), counters [kCounters] (unsigned, zero between launches)
	double *d_partials = nullptr;
	double *d_results = nullptr;
	unsigned *d_counters = nullptr;
	// device error word: kernels with bounded waits (the TMA-staged line march)
	// write a nonzero code here when a wait gives up; zero otherwise
	int *d_err = nullptr;
	// host staging for layout conversions
	void *d_stage = nullptr;
	size_t stage_bytes = 0;

	// workspace of calls on plain fields (products of a momentum step, lines of
	// Wilson loops): on this context's stream, so calls use it one after another;
	// grown on demand, freed with the context or when an allocation wants the memory
	static constexpr size_t kWorkCap = size_t(512) << 20; // the most that is kept
	void *d_work = nullptr;
	size_t work_bytes = 0;
	// false for more than is kept, and (with no workspace) when there is no memory
	bool grow_work(size_t bytes)
	{
		if (bytes > kWorkCap)
			return false;
		if (work_bytes >= bytes)
			return true;
		// the calls that come here wait for nothing and allocate nothing else: a capture of
		// another stream, on this thread or another, must not be invalidated here
		cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
		cudaThreadExchangeStreamCaptureMode(&mode);
		if (d_work)
		{
			cudaStreamSynchronize(stream);
			cudaFree(d_work);
		}
		d_work = nullptr;
		work_bytes = 0;
		if (cudaMalloc(&d_work, bytes) == cudaSuccess)
			work_bytes = bytes;
		else
		{
			cudaGetLastError();
			d_work = nullptr;
		}
		cudaThreadExchangeStreamCaptureMode(&mode);
		return work_bytes > 0;
	}

	// scratch of the chains' molecular-dynamics steps, one for all chains of the
	// context: they run on its stream one after another and nothing stays in it
	// between steps. A chain keeps the memory it was made with (its captured
	// trajectory holds the address); a larger chain replaces what later ones share.
	std::shared_ptr<void> md_shared;
	size_t md_shared_bytes = 0;

	// frees what is kept only to be used again; false when there is nothing, or while
	// the stream is captured
	bool give_back()
	{
		cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
		bool shared = md_shared && md_shared.use_count() == 1;
		if ((!d_work && !shared) || cudaStreamIsCapturing(stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)
			return false;
		cudaStreamSynchronize(stream);
		cudaFree(d_work);
		d_work = nullptr;
		work_bytes = 0;
		if (shared)
		{
			md_shared.reset();
			md_shared_bytes = 0;
		}
		return true;
	}
	// device memory that outlives the call (async: of the stream's pool); one that the
	// kept workspaces leave no room for takes them back
	void *alloc(size_t bytes, bool async = false)
	{
		void *p = nullptr;
		auto get = [&] { return async ? cudaMallocAsync(&p, bytes, stream) : cudaMalloc(&p, bytes); };
		cudaError_t e = get();
		if (e == cudaErrorMemoryAllocation && give_back())
			e = get();
		cudaGetLastError(); // not left for the next launch's check
		MESH_CUDA(e);
		return p;
	}

	void *stage(size_t bytes)
	{
		if (bytes > stage_bytes)
		{
			void *old = d_stage;
			d_stage = nullptr;
			stage_bytes = 0;
			if (old)
				MESH_CUDA(cudaFreeAsync(old, stream));
			d_stage = alloc(bytes, true);
			stage_bytes = bytes;
		}
		return d_stage;
	}
};

// Makes the context's device current for the duration of a call.
struct DeviceGuard
{
	int prev = -1;
	explicit DeviceGuard(int dev)
	{
		cudaGetDevice(&prev);
		if (prev != dev)
			MESH_CUDA(cudaSetDevice(dev));
	}
	~DeviceGuard()
	{
		if (prev >= 0)
			cudaSetDevice(prev);
	}
};

// grid size for a grid-stride kernel over n items: at most `per_sm` resident
// blocks per SM worth of blocks, never more than needed.
inline unsigned grid_for(Context const &c, int64_t n, int block, int per_sm = 8)
{
	int64_t need = (n + block - 1) / block;
	int64_t cap = int64_t(c.num_sms) * per_sm;
	if (need < 1)
		need = 1;
	return unsigned(need < cap ? need : cap);
}

} // namespace meshgb
