// Launchers of the chunked line-solve kernels, one translation unit per (direction,
// precision) so the many template instances compile in parallel.
#pragma once

#include <cuda_runtime.h>

#include "bpm_kernels.cuh"
#include "solve_config.h"

namespace nbpm {

struct SolveLaunch {
	int M, KS, kind;           // chunk length, slots per thread, stencil kind (ST_*)
	bool dep = false;          // launch_dep: the launch before it on the stream is its only new dependency
	bool tout = false;         // k_solve_xc: transposed, component-exchanged output (ST_WOOD_X only)
	dim3 grid, block;
	size_t smem;
	cudaStream_t stream;
};

// Launches a kernel that begins with wait_predecessor(); with dep set it may be scheduled before the kernel
// launched before it on the stream has ended (that kernel must be its only unfinished dependency: nothing
// between the two on the stream but their launches). Small meshes gain the launch latency: 64x64x40
// FP32 1.21 -> 1.09 ms, FP64 4.13 -> 4.04 ms, 64x64x32 with 112 slots 3.2 -> 3.0 ms.
template <typename... P, typename... A>
inline void launch_dep(bool dep, void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
	cudaLaunchConfig_t c = {};
	c.gridDim = grid;
	c.blockDim = block;
	c.dynamicSmemBytes = smem;
	c.stream = st;
	cudaLaunchAttribute a;
	a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	a.val.programmaticStreamSerializationAllowed = 1;
	c.attrs = &a;
	c.numAttrs = dep ? 1 : 0;
	cudaLaunchKernelEx(&c, k, static_cast<P>(args)...);  // errors: cudaGetLastError at the caller
}

// Returns false if (M, KS) has no compiled instance. ai2 (xc / yc only): a second accumulator
// input, ao = (ai + ai2) + x.
template <typename R>
bool launch_solve_xc(const SolveLaunch& L, Geom G, int slot0, int nch, const cx<R>* coef, const cx<R>* fac,
	size_t plane, const cx<double>* lsc, const cx<R>* src, cx<R>* dst, const cx<R>* ai, cx<R>* ao,
	const cx<R>* ai2 = nullptr);
template <typename R>
bool launch_solve_yc(const SolveLaunch& L, Geom G, int slot0, int nch, const cx<R>* coef, const cx<R>* fac,
	size_t plane, const cx<double>* lsc, const cx<R>* src, cx<R>* dst, const cx<R>* ai, cx<R>* ao,
	const cx<R>* ai2 = nullptr);
template <typename R>
bool launch_solve_xw(const SolveLaunch& L, Geom G, int slot0, int nch, const cx<R>* coef, const cx<R>* fac,
	size_t plane, const cx<double>* lsc, const cx<R>* src, cx<R>* dst, const cx<R>* ai, cx<R>* ao, const cx<R>* ai2 = nullptr);
void set_solve_smem_xw_f32(int bytes);
void set_solve_smem_xw_f64(int bytes);
// FP32 pair solves (pair_kernels.cuh), M and warps per line W: kind ST_EXPL_Y (out PO_SAME) or ST_WOOD_X; src,
// dst, acc0: pairs; plain: the plain planes of PO_PLAIN. Returns false if there is no instance.
bool launch_solve_pair(cudaStream_t st, bool dep, int M, int W, int kind, int out, Geom G, int ng, const cx<float>* coef,
	const cx<float>* fac, size_t plane, const cx<double>* lsc, const cx<float>* src, cx<float>* dst, const cx<float>* acc0,
	cx<float>* plain);
void set_solve_smem_pair(int bytes);
template <typename R>
bool launch_solve_xs(const SolveLaunch& L, Geom G, int slot0, int nch, const cx<R>* coef, const cx<R>* fac,
	size_t plane, const cx<double>* lsc, const cx<R>* src, cx<R>* dst, const cx<R>* ai, cx<R>* ao);
void set_solve_smem_xs_f32(int bytes);
void set_solve_smem_xs_f64(int bytes);
template <typename R>
bool launch_solve_ys(const SolveLaunch& L, Geom G, int slot0, int nch, const cx<R>* coef, const cx<R>* fac,
	size_t plane, const cx<double>* lsc, const cx<R>* src, cx<R>* dst, const cx<R>* ai, cx<R>* ao, cx<R>* vbuf);
// y-line solve in the x-line form (k_solve_yt): grid (columns / LT, groups * nch * 2), block 32*LT,
// shared memory LT * KS * 32 * (M + 1) complex; (M, KS) as for k_solve_xc.
template <typename R>
bool launch_solve_yt(const SolveLaunch& L, Geom G, int nch, const cx<R>* coef, const cx<R>* fac, size_t plane,
	const cx<double>* lsc, const cx<R>* src, cx<R>* dst, const cx<R>* ai, cx<R>* ao, const cx<R>* ai2);
void set_solve_smem_yt_f32(int bytes);
void set_solve_smem_yt_f64(int bytes);
// Sequential y-line solve (k_solve_yq): grid (columns / block.x, groups * nch), KS in {1, 2, 4}.
// scr receives the forward values; it must alias none of src, ai, ai2 (it may be dst or ao).
template <typename R>
bool launch_solve_yq(const SolveLaunch& L, Geom G, int nch, const cx<R>* coef, const cx<R>* fac, size_t plane,
	const cx<double>* lsc, const cx<R>* src, cx<R>* scr, cx<R>* dst, const cx<R>* ai, cx<R>* ao, const cx<R>* ai2);
void set_solve_smem_x_f32(int bytes);
void set_solve_smem_x_f64(int bytes);
void set_solve_smem_y_f32(int bytes);
void set_solve_smem_y_f64(int bytes);

}  // namespace nbpm
