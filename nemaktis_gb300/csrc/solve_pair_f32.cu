// Instances of the FP32 solves on pairs of slots.
#include "pair_kernels.cuh"
#include "solve_dispatch.cuh"

namespace nbpm {

// one line per warp: chunk lengths 2 .. 8; several warps per line: 8
#define NBPM_XP_M(F, MM) F(MM, ST_EXPL_Y, PO_SAME) F(MM, ST_WOOD_X, PO_SAME) F(MM, ST_WOOD_X, PO_TRANS) F(MM, ST_WOOD_X, PO_PLAIN)
#define NBPM_XP_ALL(F) \
	NBPM_XP_M(F, 2) NBPM_XP_M(F, 3) NBPM_XP_M(F, 4) NBPM_XP_M(F, 5) NBPM_XP_M(F, 6) NBPM_XP_M(F, 7) NBPM_XP_M(F, 8)
#define NBPM_XWP_ALL(F) \
	F(8, ST_EXPL_Y, PO_SAME) F(8, ST_WOOD_X, PO_SAME) F(8, ST_WOOD_X, PO_TRANS) F(8, ST_WOOD_X, PO_PLAIN)

bool launch_solve_pair(cudaStream_t st, bool dep, int M, int W, int kind, int out, Geom G, int ng, const cx<float>* coef,
		const cx<float>* fac, size_t plane, const cx<double>* lsc, const cx<float>* src, cx<float>* dst, const cx<float>* acc0,
		cx<float>* plain) {
	const pr* s = reinterpret_cast<const pr*>(src);
	const pr* a = reinterpret_cast<const pr*>(acc0);
	pr* d = reinterpret_cast<pr*>(dst);
	if(W == 1) {
		const dim3 grid((unsigned)((size_t)((G.Ny + 3) / 4) * 2 * G.Nq), (unsigned)ng);
		const size_t smem = (size_t)4 * (32 * part_pitch(M) + 2) * sizeof(pr);
#define NBPM_XP(MM, KD, OO) \
		if(M == MM && kind == KD && out == OO) { \
			launch_dep(dep, k_solve_xp<MM, KD, OO>, grid, dim3(128), smem, st, G, coef, fac, plane, lsc, s, d, a, plain); \
			return true; \
		}
		NBPM_XP_ALL(NBPM_XP)
		return false;
	}
	const dim3 grid((unsigned)((size_t)((G.Ny + 1) / 2) * 2 * G.Nq), (unsigned)ng);
	const size_t smem = (size_t)2 * (32 * W * part_pitch(M) + 4 + 4 * W + 2) * sizeof(pr);
	// Registers: lines of 3 warps and more make blocks of 192 threads and more, of which 64 registers leave
	// 30 warps per SM resident (1024x1024: 83.8 ms a step with 64, 90.4 with 72); blocks of two-warp lines, 128
	// threads, take 72 as k_solve_xp, or 96 when the launch has too few warps to fill the SMs anyway
	// (512x512, one pair: 21.4 ms with 96, 23.2 with 72, 23.8 with 64).
	const int regs = W > 2 ? 64 : (size_t)grid.x * grid.y * 4 <= (size_t)152 * 20 ? 96 : 72;
#define NBPM_XWP_R(MM, KD, OO, RR) \
	if(M == MM && kind == KD && out == OO && regs == RR) { \
		launch_dep(dep, k_solve_xwp<MM, KD, OO, RR>, grid, dim3((unsigned)(64 * W)), smem, st, G, W, coef, fac, plane, lsc, s, d, a, plain); \
		return true; \
	}
#define NBPM_XWP(MM, KD, OO) NBPM_XWP_R(MM, KD, OO, 64) NBPM_XWP_R(MM, KD, OO, 72) NBPM_XWP_R(MM, KD, OO, 96)
	NBPM_XWP_ALL(NBPM_XWP)
	return false;
}

void set_solve_smem_pair(int bytes) {
#define NBPM_XPA(MM, KD, OO) cudaFuncSetAttribute(k_solve_xp<MM, KD, OO>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
	NBPM_XP_ALL(NBPM_XPA)
// 16 bytes of static shared memory beside the dynamic ones
#define NBPM_XWPA_R(MM, KD, OO, RR) cudaFuncSetAttribute(k_solve_xwp<MM, KD, OO, RR>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes - 16);
#define NBPM_XWPA(MM, KD, OO) NBPM_XWPA_R(MM, KD, OO, 64) NBPM_XWPA_R(MM, KD, OO, 72) NBPM_XWPA_R(MM, KD, OO, 96)
	NBPM_XWP_ALL(NBPM_XWPA)
}

}  // namespace nbpm
