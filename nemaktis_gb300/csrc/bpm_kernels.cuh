// sm_103a kernels of the bpm z-stepping loop.
//
// Data layout in HBM (one sample):
//   director  dir[iz][iy][ix][c]            FP64, c < 3 (director) or 6 (Q-tensor)
//   fields    F[slot][comp][iy][ix]          cx<R>; slot = pol + 2*(q + Nq*lambda): the same
//                                            order as the (Nl,Nq,4,Ny,Nx) user buffer
//   eps ring  Q[2][group][NQ][iy][ix]        FP64 per-voxel derived permittivity, planes iz
//                                            and iz+1 of every wavelength group
//   coef      C[group][p/32][..][p%32]      one point's operators in CSET scalars R: the stencils of
//                                            mu*R (DX, DY, DXDY x 4 blocks) without their parts that
//                                            are zero, and 3 complex phase-operator entries, in
//                                            tiles of 32 points (coef_v, coef_u, coef_ph)
//   factors   X/Y[group][comp][NFAC][p]      cx<R>: pre-factored periodic line solves
// A "group" is one wavelength: every (q, pol) slot of the group shares eps, R, the phase
// operator and the line-solve factorisations.
#pragma once

#include <cstdint>

#include "cplx.cuh"
#include "line_join.cuh"
#include "solve_config.h"

namespace nbpm {

// Per-voxel derived permittivity components (PermittivityTensorField.cpp:3-99).
enum { Q_XXTR = 0, Q_YYTR, Q_XYTR, Q_XXS, Q_YYS, Q_XYS, Q_VX, Q_VY, Q_IZZ, NQ };
// Line-solve factor planes.
// F_A = alpha_i = -inf_i/beta_i (forward recurrence d_i = alpha_i d_{i-1} + b_i/beta_i),
// F_RB = 1/beta_i, F_W = w_i, F_C = -gamma_i (backward recurrence), F_COR = corr_i.
enum { F_A = 0, F_RB, F_W, F_C, F_COR, NFAC };
// Factor planes of the partitioned x-line solves (k_factor_part): every chunk of M points of a line
// is factored by itself. F_A = -l_i (forward recurrence d_i = r_i - l_i d_{i-1}, l_i = a_i/beta_{i-1},
// 0 at the chunk's first point), F_DB = 1/beta_i - base, F_C = -c_i/beta_i, F_Z = (product of F_C over the
// points before i) / beta_i, so that the chunk's first unknown is sum_i F_Z d_i, and F_E = what the
// unknown before the chunk adds to point i before the backward sweep. base is 1 on lines of weak coupling,
// where the difference is rounded to its own, smaller size: in a uniform region every point of every slab repeats
// the rounding of 1/beta_i, which took 7.7e-8 of the amplitude per slab in FP32 (64 slabs 256x256: 4.9e-6, 0.8e-6
// so; the solves 324 -> 332 us; FP64, droplets of 128 and 256 points: errors of 2.7e-14, 1.8 and 1.9e-14 so, for at most
// 2 % of the step). Else 0.
// It is in the line scalar lsc[line][0].y.
enum { F_DB = F_RB, F_Z = F_W, F_E = F_COR };
// Interface coefficients per chunk of those solves (h the chunk's last unknown, g the next chunk's
// first one): h = I_HD d_last + I_HY yf' and g = I_GD d_last + I_GY yf' from the two chunks alone,
// I_PH, I_PG what the previous chunk's h adds to h and g, I_QH, I_QG what the next chunk's g adds. Lines joined
// by ring_solve (line_join.cuh) hold the node's coefficients in place of those four and after them, and the right-hand
// sides' coefficients include f2 and d; the line's closing coefficients are the first four entries of I_X.
enum { I_HD = 0, I_HY, I_GD, I_GY, I_PH, I_PG, I_QH, I_QG, I_ETA, I_KAP, I_TAU, I_X, I_UNUSED, NIF };
enum { I_F = I_PH };  // RN_F .. RN_RHO there, RN_ETA .. RN_TAU from I_ETA on
static_assert(NIF == PART_NIF, "part_plane");
// Layout of a line's factors: for each point k of a chunk the vectors {F_A, F_Z} of the CH chunks, then
// {F_DB, F_C}, then F_E; after the M points the NIF interface coefficients of the chunks.
__host__ __device__ __forceinline__ size_t part_line_size(int M, int CH) { return (size_t)CH * (M * NFAC + NIF); }
template <typename S>
struct alignas(4 * sizeof(S)) v4 {
	S x, y, z, w;
};
// Shared-memory pitch of a chunk of M points: odd, so that accesses in chunk order have no bank conflicts.
__host__ __device__ constexpr int part_pitch(int M) { return M | 1; }
template <typename S>
__device__ __forceinline__ const v4<S>& part_az(const cx<S>* Fc, int k, int CH, int ci) {
	return reinterpret_cast<const v4<S>*>(Fc + (size_t)k * NFAC * CH)[ci];
}
template <typename S>
__device__ __forceinline__ const v4<S>& part_rc(const cx<S>* Fc, int k, int CH, int ci) {
	return reinterpret_cast<const v4<S>*>(Fc + (size_t)k * NFAC * CH + 2 * CH)[ci];
}
template <typename S>
__device__ __forceinline__ const cx<S>& part_e(const cx<S>* Fc, int k, int CH, int ci) { return Fc[(size_t)k * NFAC * CH + 4 * CH + ci]; }

// Coefficient set of one point. The entries of mu*R are i*(dZ/2)*(real), but for the walk-off terms: first
// derivatives, which only the outer entries of DX blocks 0, 1, 2 and of DY blocks 1, 2, 3 have. So an
// entry is one real number (its imaginary part) except those twelve, 52 numbers in place of 80, and a
// tap with a real number costs two multiply-adds in place of four. They are kept as 12 vectors of
// four and two pairs (m, c, p: the entries of the previous point, the
// point itself and the next one; the index is the block):
//   V_DD + b   DXDY block b: (px,py), (mx,py), (px,my), (mx,my)
//   V_DX + i   DX block i = 0, 1, 2: m (complex), p (complex)       V_DX + 3: m3, p3, c3, c2    U_DX: c0, c1
//   V_DY + i   DY block 3 - i = 3, 2, 1: m (complex), p (complex)   V_DY + 3: m0, p0, c0, c1    U_DY: c3, c2
// The order of the DY blocks makes the transposed frame's DX and DY plain copies of DY and DX. Sets are
// stored in tiles of 32 points with all of a tile together, so that what a kernel reads at one point is
// at fixed distances from one address and 32 consecutive points of a vector are one contiguous segment.
enum { V_DD = 0, V_DX = 4, V_DY = 8, NV = 12, U_DX = 0, U_DY = 1, NU = 2 };
enum { CSET = 4 * NV + 2 * NU + 6 };  // scalars per point: vectors, pairs, 3 complex phase entries
// complex values per group
__host__ __device__ __forceinline__ size_t coef_set_size(int N) { return (size_t)(CSET / 2) * (((size_t)N + 31) & ~(size_t)31); }
template <typename C>
__device__ __forceinline__ C* coef_tile(C* coef, int p) { return coef + (size_t)(p >> 5) * (CSET / 2 * 32); }
// half h of vector k: a tile's halves are apart, for threads that need one of them at a time (StripRhs) and so that
// a warp's 16-byte accesses to FP64 halves are contiguous
template <typename C>
__device__ __forceinline__ C& coef_h(C* coef, int k, int h, int p) { return coef_tile(coef, p)[(2 * k + h) * 32 + (p & 31)]; }
template <typename S>
__device__ __forceinline__ v4<S> coef_v(const cx<S>* coef, int k, int p) {
	const cx<S> a = coef_h(coef, k, 0, p), b = coef_h(coef, k, 1, p);
	return v4<S>{a.x, a.y, b.x, b.y};
}
template <typename S>
__device__ __forceinline__ void coef_put(cx<S>* coef, int k, int p, v4<S> v) {
	coef_h(coef, k, 0, p) = mk(v.x, v.y);
	coef_h(coef, k, 1, p) = mk(v.z, v.w);
}
// pairs and phase entries follow the vectors
template <typename C>
__device__ __forceinline__ C& coef_u(C* coef, int u, int p) { return coef_tile(coef, p)[2 * NV * 32 + u * 32 + (p & 31)]; }
template <typename C>
__device__ __forceinline__ C& coef_ph(C* coef, int i, int p) { return coef_tile(coef, p)[(2 * NV + NU) * 32 + i * 32 + (p & 31)]; }
// Entries m, c, p of the diagonal block of component comp along direction DIRN (0: DX, 1: DY) at point p.
template <int DIRN, typename S>
__device__ __forceinline__ void coef_diag(const cx<S>* coef, int comp, int p, cx<S>& m, cx<S>& c, cx<S>& n) {
	if(comp == DIRN) {  // DX block 0, DY block 3: with walk-off
		const v4<S> v = coef_v(coef, DIRN == 0 ? V_DX : V_DY, p);
		m = mk(v.x, v.y);
		n = mk(v.z, v.w);
		c = mk((S)0, coef_u(coef, DIRN == 0 ? U_DX : U_DY, p).x);
	}
	else {
		const v4<S> v = coef_v(coef, DIRN == 0 ? V_DX + 3 : V_DY + 3, p);
		m = mk((S)0, v.x);
		n = mk((S)0, v.y);
		c = mk((S)0, v.z);
	}
}
struct GroupParams {
	double wavelength, k0, dX, dY, dZ;
	double no, ne, ne_imag, nhost, nin, nout_fresnel;
	double absorp_im;  // imaginary part of 1 + i*ne_imag/(ne-no)
	double nref;
	double rX, rY, rXX, rYY, rXY;  // 1/dX, 1/dY, 1/dX^2, 1/dY^2, 1/(dX dY)
};

struct ShiftParams {
	int active;       // 0: identity (q = 0)
	int msx, msy;     // integer parts of the shifts
	double wx[4], wy[4];
	double ph_re, ph_im;
	// the same weights and phase factor rounded to FP32 (the FP32 transition reads these instead of
	// converting the FP64 values at each use)
	float fwx[4], fwy[4];
	float fph_re, fph_im;
	// weights of one shift and of two one after the other as 7 taps, the latter sums of products of the above
	double tx[2][7], ty[2][7];
};

// Weights and phase factor in the arithmetic type R, and the filter of nsh = 1 or 2 shifts of one axis on N
// consecutive values in place, v[k] for k < N - 6. FP64: one 7-tap filter (7 (N - 6) multiply-adds in place of
// 4 (N - 3) + 4 (N - 6); the FP64 pipe bounds the transition: 1408 -> 1082 us on 256x256, 3 wavelengths, 13
// q). FP32: two 4-tap passes, which need fewer registers (473 us on 16 wavelengths, 513 with 7 taps).
template <typename R>
struct ShiftW {
	const int nsh;
	R wx[4], wy[4];
	cx<R> ph;
	__device__ __forceinline__ ShiftW(const ShiftParams& P, int n) : nsh(n) {
#pragma unroll
		for(int k = 0; k < 4; k++) { wx[k] = P.fwx[k]; wy[k] = P.fwy[k]; }
		ph = mk<R>(P.fph_re, P.fph_im);
	}
	template <int N>
	__device__ __forceinline__ void filter(const R* w, cx<R>* v) const {
#pragma unroll
		for(int k = 0; k < N - 3; k++) v[k] = w[0] * v[k] + w[1] * v[k + 1] + w[2] * v[k + 2] + w[3] * v[k + 3];
		if(nsh == 2) {
#pragma unroll
			for(int k = 0; k < N - 6; k++) v[k] = w[0] * v[k] + w[1] * v[k + 1] + w[2] * v[k + 2] + w[3] * v[k + 3];
		}
	}
};
template <>
struct ShiftW<double> {
	double wx[7], wy[7];
	cx<double> ph;
	__device__ __forceinline__ ShiftW(const ShiftParams& P, int n) {
#pragma unroll
		for(int k = 0; k < 7; k++) { wx[k] = P.tx[n - 1][k]; wy[k] = P.ty[n - 1][k]; }
		ph = mk<double>(P.ph_re, P.ph_im);
	}
	template <int N>
	__device__ __forceinline__ void filter(const double* w, cx<double>* v) const {
#pragma unroll
		for(int k = 0; k < N - 6; k++) {
			cx<double> s = w[0] * v[k];
#pragma unroll
			for(int m = 1; m < 7; m++) s = mk<double>(fma(w[m], v[k + m].x, s.x), fma(w[m], v[k + m].y, s.y));
			v[k] = s;
		}
	}
};

struct Geom {
	int Nx, Ny, N;
	int Nz;
	int spg;          // slots per group = 2*Nq
	int Nq;
};

// ---------------------------------------------------------------------------------------
// Permittivity per voxel from the director or Q-tensor (PermittivityTensorField.cpp:19-99).
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void eps_voxel(const double* __restrict__ dir, int fd, bool m,
		const GroupParams& gp, double e[6]) {
	double eps_perp = gp.no * gp.no;
	double eps_a = gp.ne * gp.ne - eps_perp;
	double eps_host = gp.nhost * gp.nhost;
	if(!m) {
		e[0] = e[1] = e[2] = eps_host;
		e[3] = e[4] = e[5] = 0;
		return;
	}
	if(fd == 3) {
		double n0 = dir[0], n1 = dir[1], n2 = dir[2];
		e[0] = eps_perp + eps_a * (n0 * n0);
		e[1] = eps_perp + eps_a * (n1 * n1);
		e[2] = eps_perp + eps_a * (n2 * n2);
		e[3] = eps_a * n0 * n1;
		e[4] = eps_a * n0 * n2;
		e[5] = eps_a * n1 * n2;
	}
	else {
		double ea = 2 * eps_a / 3, ei = eps_perp + eps_a / 3.;
		e[0] = ei + ea * dir[0];
		e[1] = ei + ea * dir[1];
		e[2] = ei + ea * dir[2];
		e[3] = ea * dir[3];
		e[4] = ea * dir[4];
		e[5] = ea * dir[5];
	}
}

__device__ __forceinline__ double neff_of(double xxtr, double yytr, double xytr) {
	double det = xxtr * yytr - xytr * xytr;
	double tr = 0.5 * (xxtr + yytr);
	if(tr * tr - det < 1e-8) return sqrt(tr);
	double r = sqrt(tr * tr - det);
	return (sqrt(tr + r) + sqrt(tr - r)) / 2.;
}

// neff of one voxel in FP32 arithmetic (the same formulas as eps_voxel + neff_of), for the nref
// mean of the FP32 mode.
__device__ __forceinline__ float neff_voxel_f(const double* __restrict__ dir, int fd, bool m, float eps_perp,
		float eps_a, float eps_host) {
	float e0, e1, e2, e3, e4, e5;
	if(!m) return sqrtf(eps_host);
	if(fd == 3) {
		float n0 = (float)dir[0], n1 = (float)dir[1], n2 = (float)dir[2];
		e0 = eps_perp + eps_a * (n0 * n0);
		e1 = eps_perp + eps_a * (n1 * n1);
		e2 = eps_perp + eps_a * (n2 * n2);
		e3 = eps_a * n0 * n1;
		e4 = eps_a * n0 * n2;
		e5 = eps_a * n1 * n2;
	}
	else {
		float ea = 2 * eps_a / 3, ei = eps_perp + eps_a / 3.f;
		e0 = ei + ea * (float)dir[0];
		e1 = ei + ea * (float)dir[1];
		e2 = ei + ea * (float)dir[2];
		e3 = ea * (float)dir[3];
		e4 = ea * (float)dir[4];
		e5 = ea * (float)dir[5];
	}
	float xx = e0 - (e4 * e4) / e2, yy = e1 - (e5 * e5) / e2, xy = e3 - e4 * e5 / e2;
	float det = xx * yy - xy * xy, tr = 0.5f * (xx + yy);
	if(tr * tr - det < 1e-8f) return sqrtf(tr);
	float r = sqrtf(tr * tr - det);
	return (sqrtf(tr + r) + sqrtf(tr - r)) / 2.f;
}

// One transverse plane of derived quantities for every group of the pass, computed and
// stored in the plan's precision Q (FP64 mode: FP64; FP32 mode: FP32).
template <typename Q>
static __global__ void k_eps_plane(const double* __restrict__ dir, int fd, const uint8_t* __restrict__ mask,
		int N, int iz, const GroupParams* __restrict__ gps, Q* __restrict__ out) {
	int p = blockIdx.x * blockDim.x + threadIdx.x;
	int g = blockIdx.y;
	if(p >= N) return;
	size_t v = (size_t)iz * N + p;
	GroupParams gp = gps[g];
	const bool m = mask ? mask[v] != 0 : true;
	Q* o = out + (size_t)g * NQ * N + p;
	if(sizeof(Q) == sizeof(float)) {
		// FP32 mode: the same formulas in FP32 arithmetic
		const float ep = (float)(gp.no * gp.no), ea = (float)(gp.ne * gp.ne - gp.no * gp.no);
		const float eh = (float)(gp.nhost * gp.nhost);
		const double* d = dir + v * fd;
		float e0, e1, e2, e3, e4, e5;
		if(!m) { e0 = e1 = e2 = eh; e3 = e4 = e5 = 0.f; }
		else if(fd == 3) {
			float n0 = (float)d[0], n1 = (float)d[1], n2 = (float)d[2];
			e0 = ep + ea * (n0 * n0); e1 = ep + ea * (n1 * n1); e2 = ep + ea * (n2 * n2);
			e3 = ea * n0 * n1; e4 = ea * n0 * n2; e5 = ea * n1 * n2;
		}
		else {
			float a = 2 * ea / 3, ei = ep + ea / 3.f;
			e0 = ei + a * (float)d[0]; e1 = ei + a * (float)d[1]; e2 = ei + a * (float)d[2];
			e3 = a * (float)d[3]; e4 = a * (float)d[4]; e5 = a * (float)d[5];
		}
		const float rz = 1.f / e2, vx = e4 * rz, vy = e5 * rz;
		float xx = e0 - e4 * vx, yy = e1 - e5 * vy, xy = e3 - e4 * vy;
		float det = xx * yy - xy * xy, tr = 0.5f * (xx + yy), ne;
		if(tr * tr - det < 1e-8f) ne = sqrtf(tr);
		else { float r = sqrtf(tr * tr - det); ne = (sqrtf(tr + r) + sqrtf(tr - r)) / 2.f; }
		const float rn = 0.25f / ne;
		o[Q_XXTR * N] = (Q)xx;
		o[Q_YYTR * N] = (Q)yy;
		o[Q_XYTR * N] = (Q)xy;
		o[Q_XXS * N] = (Q)(ne + (xx - yy) * rn);
		o[Q_YYS * N] = (Q)(ne + (yy - xx) * rn);
		o[Q_XYS * N] = (Q)(xy * (2 * rn));
		o[Q_VX * N] = (Q)vx;
		o[Q_VY * N] = (Q)vy;
		o[Q_IZZ * N] = (Q)rz;
		return;
	}
	double e[6];
	eps_voxel(dir + v * fd, fd, m, gp, e);
	// one division by eps_zz and one by neff: an FP64 division costs about ten multiplications
	const double rz = 1. / e[2], vx = e[4] * rz, vy = e[5] * rz;
	double xxtr = e[0] - e[4] * vx;
	double yytr = e[1] - e[5] * vy;
	double xytr = e[3] - e[4] * vy;
	double neff = neff_of(xxtr, yytr, xytr);
	const double rn = 0.25 / neff;
	o[Q_XXTR * N] = (Q)xxtr;
	o[Q_YYTR * N] = (Q)yytr;
	o[Q_XYTR * N] = (Q)xytr;
	o[Q_XXS * N] = (Q)(neff + (xxtr - yytr) * rn);
	o[Q_YYS * N] = (Q)(neff + (yytr - xxtr) * rn);
	o[Q_XYS * N] = (Q)(xytr * (2 * rn));
	o[Q_VX * N] = (Q)vx;
	o[Q_VY * N] = (Q)vy;
	o[Q_IZZ * N] = (Q)rz;
}

// Partial sums of neff over the volume for nref (PermittivityTensorField.cpp:183-211),
// in a fixed block order so the reduction is deterministic.
// FP32 mode (F32 = true): neff in FP32 arithmetic, summed in FP64.
template <bool F32>
static __global__ void k_neff_partial(const double* __restrict__ dir, int fd, const uint8_t* __restrict__ mask,
		size_t nvox, const GroupParams* __restrict__ gps, double* __restrict__ partial) {
	__shared__ double sh[256];
	int g = blockIdx.y;
	GroupParams gp = gps[g];
	double acc = 0;
	const float ep = (float)(gp.no * gp.no), ea = (float)(gp.ne * gp.ne - gp.no * gp.no), eh = (float)(gp.nhost * gp.nhost);
	for(size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvox; v += (size_t)gridDim.x * blockDim.x) {
		if(F32) {
			acc += (double)neff_voxel_f(dir + v * fd, fd, mask ? mask[v] != 0 : true, ep, ea, eh);
			continue;
		}
		double e[6];
		eps_voxel(dir + v * fd, fd, mask ? mask[v] != 0 : true, gp, e);
		const double rz = 1. / e[2];
		double xxtr = e[0] - (e[4] * e[4]) * rz;
		double yytr = e[1] - (e[5] * e[5]) * rz;
		double xytr = e[3] - e[4] * e[5] * rz;
		acc += neff_of(xxtr, yytr, xytr);
	}
	sh[threadIdx.x] = acc;
	__syncthreads();
	for(int s = blockDim.x / 2; s > 0; s >>= 1) {
		if(threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
		__syncthreads();
	}
	if(threadIdx.x == 0) partial[(size_t)g * gridDim.x + blockIdx.x] = sh[0];
}

// ---------------------------------------------------------------------------------------
// Per-slab operator coefficients, in the plan's precision (the phase's argument too):
//  * phase operator exp(i*a*d) (PhaseEvolutionOperator.cpp:34-63)
//  * mu*R with R = i*W + (D*S^-1 + S^-1*D)/4, D = D0 + D1*K (ParaxialPrimaryEvolution-
//    Operator.cpp:212-490), written per stencil entry: S^-1 and K at the column point for
//    D*S^-1 and D1*K, S^-1 at the row point for S^-1*D, the walk-off split between row
//    and column points. D1 uses the reference's neighbour indices (ix==Nx-1 -> 1,
//    ix==0 -> Nx-2) while the stencil columns wrap with period Nx-1.
// ---------------------------------------------------------------------------------------
// Phase operator of one point (PhaseEvolutionOperator.cpp:14-32) from eps planes A, B of the
// slab's two ends, in the arithmetic type T.
template <typename T>
__device__ __forceinline__ void phase_op(const T* A, const T* B, int N, int p, T w0, T w1, const GroupParams& gp,
		cx<T>& oxx, cx<T>& oyy, cx<T>& oxy) {
	T hz = (T)(0.5 * gp.dZ);
	T dxx = hz * (w0 * A[Q_XXS * N + p] + w1 * B[Q_XXS * N + p] - (T)gp.no);
	T dyy = hz * (w0 * A[Q_YYS * N + p] + w1 * B[Q_YYS * N + p] - (T)gp.no);
	T dxy = hz * (w0 * A[Q_XYS * N + p] + w1 * B[Q_XYS * N + p]);
	T diff = (dxx - dyy) / (T)2, tr = (dxx + dyy) / (T)2;
	T det = sqrt(dxy * dxy + diff * diff);
	cx<T> a = mk<T>((T)1, (T)gp.absorp_im);
	cx<T> sinc = mk<T>((T)1, (T)0);
	cx<T> e, c;
	if(gp.absorp_im == 0) {
		// no absorption: the imaginary parts vanish (sinh 0, cosh 0 below)
		T s, co, se, ce;
		if(sizeof(T) == sizeof(double)) { double a_, b_; sincos((double)det, &a_, &b_); s = (T)a_; co = (T)b_; sincos((double)tr, &a_, &b_); se = (T)a_; ce = (T)b_; }
		else { float a_, b_; sincosf((float)det, &a_, &b_); s = (T)a_; co = (T)b_; sincosf((float)tr, &a_, &b_); se = (T)a_; ce = (T)b_; }
		if(!(fabs(det) < (T)1e-8)) sinc = mk<T>(s / det, (T)0);
		e = mk<T>(ce, se);
		c = mk<T>(co, (T)0);
	}
	else if(sizeof(T) == sizeof(double)) {
		cx<double> ad = cvt<double>(a);
		if(!(fabs((double)det) < 1e-8)) {
			cx<double> sn = csin_d((double)det * ad);
			sinc = cvt<T>(mk(sn.x / (double)det, sn.y / (double)det));
		}
		e = cvt<T>(cexp_d(mk(-ad.y * (double)tr, ad.x * (double)tr)));  // exp(i*a*tr)
		c = cvt<T>(ccos_d((double)det * ad));
	}
	else {
		cx<float> af = cvt<float>(a);
		if(!(fabsf((float)det) < 1e-8f)) {
			cx<float> sn = csin_f((float)det * af);
			sinc = cvt<T>(mk(sn.x / (float)det, sn.y / (float)det));
		}
		e = cvt<T>(cexp_f(mk(-af.y * (float)tr, af.x * (float)tr)));
		c = cvt<T>(ccos_f((float)det * af));
	}
	cx<T> ids = mk<T>((T)0, diff) * sinc;
	oxx = e * (c + ids);
	oyy = e * (c - ids);
	oxy = ((e * mk<T>((T)0, (T)1)) * dxy) * sinc;
}

// A block takes a tile of 32 x TY points and first forms what the operators need of a point (S^-1, K, 1/eps_zz,
// walk-off) once for each point of the tile and around it, in shared memory: a point's ten neighbours would
// each form it again (a determinant and a division each). The stencil columns wrap with period N - 1 while the
// first derivatives' weights look at the natural neighbour, so column and row 0 have a place of their own past the
// tile's edge (index 32 + 2, TY + 2) for the last unknowns. TR: the tile's entries also go to the transposed
// frame's set (its DX is DY, its DY is DX, its DXDY block b is DXDY block 3 - b with the two middle corners
// exchanged), through shared memory so that TY consecutive points are written together.
// Bound: FP64 pipe (FP64), HBM (FP32, 82 % of the copy rate). With every neighbour's values formed again and the
// transposed set copied by a kernel of its own: 256x256, 16 wavelengths, FP32 88 + 87 us, 96 us so; 3
// wavelengths FP64 269 + 36 and 179 us; a 64x64 FP64 slab 31 + 8 and 25 us.
constexpr int COEF_TX = 32;
enum { CQ_CXX = 0, CQ_CYY, CQ_CXY, CQ_KXX, CQ_KYY, CQ_KXY, CQ_EZ, CQ_V0, CQ_V1, NCQ };
template <int TY>
constexpr int coef_tile_points() { return (COEF_TX + 3) * (TY + 3); }
template <typename S, int TY>
constexpr size_t coef_smem(bool tr) {
	return NCQ * coef_tile_points<TY>() * sizeof(S) + 32 + (tr ? (size_t)4 * TY * (COEF_TX + 1) * 4 * sizeof(S) : 0);
}
template <typename S, int TY, bool TR>
__global__ void __launch_bounds__(32 * TY) k_coef(const S* __restrict__ QA, const S* __restrict__ QB,
		const double* __restrict__ wts, int iz, Geom G, const GroupParams* __restrict__ gps,
		cx<S>* __restrict__ coef, cx<S>* __restrict__ coefT) {
	typedef S T;  // arithmetic type of the eps planes, the phase operator and the R coefficients
	extern __shared__ unsigned char smem_raw[];
	constexpr int LX = COEF_TX + 3, LY = TY + 3, LP = LX * LY;
	T* const sm = reinterpret_cast<T*>(smem_raw);
	const int g = blockIdx.z, N = G.N, Nx = G.Nx, Ny = G.Ny;
	const int x0 = blockIdx.x * COEF_TX, y0 = blockIdx.y * TY;
	const GroupParams& gp = gps[g];
	const T* A = QA + (size_t)g * NQ * N;
	const T* B = QB + (size_t)g * NQ * N;
	cx<S>* C = coef + (size_t)g * coef_set_size(N);
	const int tid = threadIdx.y * 32 + threadIdx.x;
	// place l of a tile's axis: l = 0 the point before the tile (period n - 1), 1 .. size + 1 the tile and the
	// natural next point, size + 2 point 0
	auto place = [](int l, int size, int o, int n) {
		const int i = l == size + 2 ? 0 : l == 0 ? (o == 0 ? n - 2 : o - 1) : o + l - 1;
		return max(0, min(i, n - 1));
	};
	for(int e = tid; e < LP; e += 32 * TY) {
		const int q = place(e % LX, COEF_TX, x0, Nx) + Nx * place(e / LX, TY, y0, Ny);
		auto avg = [&](int k) { return (A[k * N + q] + B[k * N + q]) * (T)0.5; };
		const T exx = avg(Q_XXS), eyy = avg(Q_YYS), exy = avg(Q_XYS);
		const T r = (T)1 / (exx * eyy - exy * exy);
		sm[CQ_CXX * LP + e] = eyy * r;
		sm[CQ_CYY * LP + e] = exx * r;
		sm[CQ_CXY * LP + e] = -exy * r;
		sm[CQ_KXX * LP + e] = avg(Q_XXTR);
		sm[CQ_KYY * LP + e] = avg(Q_YYTR);
		sm[CQ_KXY * LP + e] = avg(Q_XYTR);
		sm[CQ_EZ * LP + e] = avg(Q_IZZ);
		sm[CQ_V0 * LP + e] = A[Q_VX * N + q] + B[Q_VX * N + q];
		sm[CQ_V1 * LP + e] = A[Q_VY * N + q] + B[Q_VY * N + q];
	}
	__syncthreads();
	const int ix = x0 + threadIdx.x, iy = y0 + threadIdx.y, p = ix + Nx * iy;
	const bool live = ix < Nx && iy < Ny;
	if(live) {
		T w0 = (T)0.5, w1 = (T)0.5;
		if(wts) { size_t vi = (size_t)iz * N + p; w0 = (T)wts[2 * vi]; w1 = (T)wts[2 * vi + 1]; }
		cx<T> oxx, oyy, oxy;
		phase_op<T>(A, B, N, p, w0, w1, gp, oxx, oyy, oxy);
		coef_ph(C, 0, p) = oxx;
		coef_ph(C, 1, p) = oyy;
		coef_ph(C, 2, p) = oxy;
	}
	const int lx = threadIdx.x + 1, ly = threadIdx.y + 1, l0 = lx + LX * ly;
	const int lxp = ix == Nx - 2 ? COEF_TX + 2 : lx + 1, lyp = iy == Ny - 2 ? TY + 2 : ly + 1;  // next stencil column / row
	auto Q = [&](int k, int l) { return sm[k * LP + l]; };
	const T hmu = (T)(gp.dZ / 2.), q4 = (T)0.25, h4 = q4 * hmu;
	const T rX = (T)gp.rX, rY = (T)gp.rY, rXX = (T)gp.rXX, rYY = (T)gp.rYY, rXY = (T)gp.rXY;
	const T rxx = Q(CQ_CXX, l0), ryy = Q(CQ_CYY, l0), rxy = Q(CQ_CXY, l0), e0 = Q(CQ_EZ, l0);
	const T va0 = Q(CQ_V0, l0), va1 = Q(CQ_V1, l0);
	// imaginary parts of the four blocks, (dZ/2) (D S^-1 + S^-1 D) / 4 with S^-1 at the neighbour l and at the point
	auto blocks = [&](T D00, T D01, T D10, T D11, int l, T* im) {
		const T cxx = Q(CQ_CXX, l), cyy = Q(CQ_CYY, l), cxy = Q(CQ_CXY, l);
		im[0] = h4 * (D00 * cxx + D01 * cxy + rxx * D00 + rxy * D10);
		im[1] = h4 * (D00 * cxy + D01 * cyy + rxx * D01 + rxy * D11);
		im[2] = h4 * (D10 * cxx + D11 * cxy + rxy * D00 + ryy * D10);
		im[3] = h4 * (D10 * cxy + D11 * cyy + rxy * D01 + ryy * D11);
	};
	// the sets of 4 vectors as they are complete: to the point's set and, for TR, to the transposed one
	v4<S>* const st = reinterpret_cast<v4<S>*>(smem_raw + ((NCQ * LP * sizeof(S) + 31) & ~(size_t)31));
	cx<S>* CT = coefT + (TR ? (size_t)g * coef_set_size(N) : 0);
	auto put = [&](const v4<S>* v, int k, int kt, bool corners) {
		if(live) {
#pragma unroll
			for(int j = 0; j < 4; j++) coef_put(C, k + j, p, v[j]);
		}
		if(TR) {
			__syncthreads();  // the vectors before these have been written
#pragma unroll
			for(int j = 0; j < 4; j++)
				st[(j * TY + threadIdx.y) * (COEF_TX + 1) + threadIdx.x] = corners ? v4<S>{v[3 - j].x, v[3 - j].z, v[3 - j].y, v[3 - j].w} : v[j];
			__syncthreads();
			const int ty = tid % TY, tx = tid / TY;
			if(x0 + tx < Nx && y0 + ty < Ny) {
#pragma unroll
				for(int j = 0; j < 4; j++) coef_put(CT, kt + j, (x0 + tx) * Ny + y0 + ty, st[(j * TY + ty) * (COEF_TX + 1) + tx]);
			}
		}
	};
	v4<S> v[4];
	const v4<S> zero{0, 0, 0, 0};
	cx<S> ux = mk<S>(0, 0), uy = mk<S>(0, 0);
	T m[4], c[4], n[4];
	// DX: rows ix < Nx-1 when Nx > 3; m, c, n: columns ix - 1, ix, ix + 1
	v[0] = v[1] = v[2] = v[3] = zero;
	if(Nx > 3 && ix < Nx - 1) {
		const int lm = l0 - 1, ln = lxp + LX * ly;
		const T cm = (T)0.5 * (Q(CQ_EZ, lm) + e0) * rXX, cp = (T)0.5 * (Q(CQ_EZ, l0 + 1) + e0) * rXX, c0 = -cm - cp;
		blocks(cm * Q(CQ_KXX, lm), cm * Q(CQ_KXY, lm), (T)0, rXX, lm, m);
		blocks(c0 * Q(CQ_KXX, l0), c0 * Q(CQ_KXY, l0), (T)0, (T)-2 * rXX, l0, c);
		blocks(cp * Q(CQ_KXX, ln), cp * Q(CQ_KXY, ln), (T)0, rXX, ln, n);
		// walk-off: -(dZ/2) (-+ 1 / (2 dX)) / 4 times v0 twice, v1 of the neighbour, v1 of the point
		const T d = hmu * (T)0.5 * rX * q4;
		v[0] = v4<S>{d * (va0 + Q(CQ_V0, lm)), m[0], -d * (va0 + Q(CQ_V0, ln)), n[0]};
		v[1] = v4<S>{d * Q(CQ_V1, lm), m[1], -d * Q(CQ_V1, ln), n[1]};
		v[2] = v4<S>{d * va1, m[2], -d * va1, n[2]};
		v[3] = v4<S>{m[3], n[3], c[3], c[2]};
		ux = mk(c[0], c[1]);
	}
	put(v, V_DX, V_DY, false);
	// DY: rows iy < Ny-1 when Ny > 3; vectors in the order of blocks 3, 2, 1
	v[0] = v[1] = v[2] = v[3] = zero;
	if(Ny > 3 && iy < Ny - 1) {
		const int lm = l0 - LX, ln = lx + LX * lyp;
		const T cm = (T)0.5 * (Q(CQ_EZ, lm) + e0) * rYY, cp = (T)0.5 * (Q(CQ_EZ, l0 + LX) + e0) * rYY, c0 = -cm - cp;
		blocks(rYY, (T)0, cm * Q(CQ_KXY, lm), cm * Q(CQ_KYY, lm), lm, m);
		blocks((T)-2 * rYY, (T)0, c0 * Q(CQ_KXY, l0), c0 * Q(CQ_KYY, l0), l0, c);
		blocks(rYY, (T)0, cp * Q(CQ_KXY, ln), cp * Q(CQ_KYY, ln), ln, n);
		const T d = hmu * (T)0.5 * rY * q4;
		v[0] = v4<S>{d * (va1 + Q(CQ_V1, lm)), m[3], -d * (va1 + Q(CQ_V1, ln)), n[3]};
		v[1] = v4<S>{d * Q(CQ_V0, lm), m[2], -d * Q(CQ_V0, ln), n[2]};
		v[2] = v4<S>{d * va0, m[1], -d * va0, n[1]};
		v[3] = v4<S>{m[0], n[0], c[0], c[1]};
		uy = mk(c[3], c[2]);
	}
	put(v, V_DY, V_DX, false);
	// DXDY: rows ix < Nx-1, iy < Ny-1 when Nx > 3 and Ny > 3; corners pxpy, mxpy, pxmy, mxmy
	v[0] = v[1] = v[2] = v[3] = zero;
	if(Nx > 3 && Ny > 3 && ix < Nx - 1 && iy < Ny - 1) {
		const T a1 = q4 * Q(CQ_EZ, l0 + 1) * rXY, c1 = q4 * Q(CQ_EZ, l0 - 1) * rXY;
		const T a2 = q4 * Q(CQ_EZ, l0 + LX) * rXY, c2 = q4 * Q(CQ_EZ, l0 - LX) * rXY, g0 = q4 * rXY;
		auto corner = [&](int l, T d01, T d10, T gg, T* im) {
			const T kxx = Q(CQ_KXX, l), kyy = Q(CQ_KYY, l), kxy = Q(CQ_KXY, l);
			blocks(d01 * kxy, gg + d01 * kyy, gg + d10 * kxx, d10 * kxy, l, im);
		};
		T pp[4], mp[4], pm[4], mm[4];
		corner(lxp + LX * lyp, a1, a2, -g0, pp);
		corner(lx - 1 + LX * lyp, -c1, -a2, g0, mp);
		corner(lxp + LX * (ly - 1), -a1, -c2, g0, pm);
		corner(l0 - 1 - LX, c1, c2, -g0, mm);
#pragma unroll
		for(int b = 0; b < 4; b++) v[b] = v4<S>{pp[b], mp[b], pm[b], mm[b]};
	}
	put(v, V_DD, V_DD, true);
	if(live) {
		coef_u(C, U_DX, p) = ux;
		coef_u(C, U_DY, p) = uy;
	}
	if(TR) {
		__syncthreads();
		st[threadIdx.y * (COEF_TX + 1) + threadIdx.x] = v4<S>{uy.x, uy.y, ux.x, ux.y};
		__syncthreads();
		const int ty = tid % TY, tx = tid / TY;
		if(x0 + tx < Nx && y0 + ty < Ny) {
			const v4<S> u = st[ty * (COEF_TX + 1) + tx];
			const int q = (x0 + tx) * Ny + y0 + ty;
			coef_u(CT, U_DX, q) = mk(u.x, u.y);
			coef_u(CT, U_DY, q) = mk(u.z, u.w);
		}
	}
}

// ---------------------------------------------------------------------------------------
// Right-hand-side kernels over all (point, slot) pairs of a pass.
// ---------------------------------------------------------------------------------------
template <typename R>
struct Stencil {
	const cx<R>* C;
	int N, Nx, Ny;
};

// out += (i*a) f for a real entry a of an imaginary coefficient.
template <typename R>
__device__ __forceinline__ cx<R> ifma(R a, cx<R> f, cx<R> out) { return mk<R>(fmar(-a, f.y, out.x), fmar(a, f.x, out.y)); }

// Step kinds of the composite stencil kernel (ParaxialPrimaryEvolutionOperator.cpp:153-207
// with the duplicate-row/column fix-ups of BlockSparseMatrix.cpp folded in analytically).
enum { ST_EXPL_Y = 0, ST_EXPL_X = 1, ST_WOOD_X = 2, ST_WOOD_Y = 3 };

// A value at a byte offset from a field plane: the plane's address is the same for the whole block and
// the offset 32 bits wide (a plane pair of one slot is below 4 GB), so that an access costs one add at most.
template <typename R>
__device__ __forceinline__ cx<R> at_off(const cx<R>* f, unsigned o) {
	return *reinterpret_cast<const cx<R>*>(reinterpret_cast<const char*>(f) + o);
}

// One component of a composite stencil step at point (ix, iy) for KS consecutive slots at once (f0: comp-0
// plane of the first slot, slot planes 2N apart, comp-1 plane at +N); every stencil coefficient is loaded
// once. EXPL kinds return f + mu*R f (explicit half-step), WOOD kinds mu*R_offdiag t (Woodbury
// right-hand side). (xx, yy) are the indices with the duplicate column / row folded onto column / row
// 0, which is where the reference's fix-ups copy their values from. The neighbours wrap with period
// N - 1; directions of three points or fewer have no derivatives.
template <typename R, int KIND, int KS>
__device__ __forceinline__ void composite_m(const Stencil<R>& st, int comp, int ix, int iy, const cx<R>* f0,
		cx<R>* out) {
	const int Nx = st.Nx, Ny = st.Ny;
	const size_t N = st.N;
	constexpr unsigned SZ = sizeof(cx<R>);
	const bool ax = Nx > 3, ay = Ny > 3;
	const cx<R>* C = st.C;
	constexpr bool XDIR = KIND == ST_EXPL_X || KIND == ST_WOOD_X;  // derivatives along x (else along y)
	constexpr bool EXPL = KIND == ST_EXPL_X || KIND == ST_EXPL_Y;
	// the component that also takes the mixed derivatives: 0 along x, 1 along y
	const bool mixed = XDIR ? comp == 0 : comp == 1;
#pragma unroll
	for(int j = 0; j < KS; j++) out[j] = mk<R>(0, 0);
	const unsigned own = ((unsigned)iy * (unsigned)Nx + (unsigned)ix) * SZ;
	if(XDIR ? ax : ay) {
		const bool both = mixed && ax && ay;
		// the row point of the taps: folded along both directions where the mixed derivatives take part
		// (or would, without the other direction: only along this one)
		const int xx = (XDIR || both) && ix == Nx - 1 ? 0 : ix;
		const int yy = (!XDIR || both) && iy == Ny - 1 ? 0 : iy;
		const int p = xx + Nx * yy;
		const unsigned o = (unsigned)p * SZ;
		const unsigned om = XDIR ? (xx == 0 ? o + (unsigned)(Nx - 2) * SZ : o - SZ)
			: (yy == 0 ? o + (unsigned)(Ny - 2) * (unsigned)Nx * SZ : o - (unsigned)Nx * SZ);
		const unsigned op = XDIR ? (xx == Nx - 2 ? o - (unsigned)(Nx - 2) * SZ : o + SZ)
			: (yy == Ny - 2 ? o - (unsigned)(Ny - 2) * (unsigned)Nx * SZ : o + (unsigned)Nx * SZ);
		// entries (m, c, p) applied to component plane f of every slot
		auto taps = [&](v4<R> v, R c, const cx<R>* f) {
#pragma unroll
			for(int j = 0; j < KS; j++) {
				const cx<R>* fj = f + 2 * N * j;
				out[j] = cfma(mk(v.z, v.w), at_off(fj, op), ifma(c, at_off(fj, o), cfma(mk(v.x, v.y), at_off(fj, om), out[j])));
			}
		};
		auto itaps = [&](R m, R c, R n, const cx<R>* f) {  // without walk-off
#pragma unroll
			for(int j = 0; j < KS; j++) {
				const cx<R>* fj = f + 2 * N * j;
				out[j] = ifma(n, at_off(fj, op), ifma(c, at_off(fj, o), ifma(m, at_off(fj, om), out[j])));
			}
		};
		const cx<R>* f1 = f0 + N;
		// DX and DY blocks by their place in the set: D + 3 holds (m, p, c) of the block without walk-off and a
		// centre, U the centres of the two other blocks
		constexpr int D = XDIR ? V_DX : V_DY, U = XDIR ? U_DX : U_DY;
		if(XDIR) {
			if(comp == 0) {
				const cx<R> u = coef_u(C, U, p);
				if(EXPL) taps(coef_v(C, D, p), u.x, f0);
				taps(coef_v(C, D + 1, p), u.y, f1);
			}
			else {
				const v4<R> w = coef_v(C, D + 3, p);
				if(EXPL) itaps(w.x, w.z, w.y, f1);
				taps(coef_v(C, D + 2, p), w.w, f0);
			}
		}
		else {
			if(comp == 0) {
				const v4<R> w = coef_v(C, D + 3, p);
				if(EXPL) itaps(w.x, w.z, w.y, f0);
				taps(coef_v(C, D + 2, p), w.w, f1);
			}
			else {
				const cx<R> u = coef_u(C, U, p);
				if(EXPL) taps(coef_v(C, D, p), u.x, f1);
				taps(coef_v(C, D + 1, p), u.y, f0);
			}
		}
		if(both) {
			// corners: the offsets along the other direction, relative to the tap along this one
			const unsigned dm = XDIR ? (yy == 0 ? (unsigned)(Ny - 2) * (unsigned)Nx * SZ : 0u - (unsigned)Nx * SZ)
				: (xx == 0 ? (unsigned)(Nx - 2) * SZ : 0u - SZ);
			const unsigned dp = XDIR ? (yy == Ny - 2 ? 0u - (unsigned)(Ny - 2) * (unsigned)Nx * SZ : (unsigned)Nx * SZ)
				: (xx == Nx - 2 ? 0u - (unsigned)(Nx - 2) * SZ : SZ);
			const unsigned opp = op + dp, omm = om + dm, opm = XDIR ? op + dm : om + dp, omp = XDIR ? om + dp : op + dm;
			// opm: (px, my), omp: (mx, py)
			auto corners = [&](v4<R> v, const cx<R>* f) {
#pragma unroll
				for(int j = 0; j < KS; j++) {
					const cx<R>* fj = f + 2 * N * j;
					out[j] = ifma(v.w, at_off(fj, omm), ifma(v.z, at_off(fj, opm), ifma(v.y, at_off(fj, omp), ifma(v.x, at_off(fj, opp), out[j]))));
				}
			};
			if(XDIR) { corners(coef_v(C, V_DD + 0, p), f0); corners(coef_v(C, V_DD + 1, p), f1); }
			else { corners(coef_v(C, V_DD + 3, p), f1); corners(coef_v(C, V_DD + 2, p), f0); }
		}
	}
	if(EXPL) {
		const cx<R>* f = f0 + (comp == 0 ? 0 : N);
#pragma unroll
		for(int j = 0; j < KS; j++) out[j] += at_off(f + 2 * N * j, own);
	}
}

template <typename R, int KIND>
__global__ void k_stencil(Geom G, int slot0, const cx<R>* __restrict__ coef, const cx<R>* __restrict__ src,
		cx<R>* __restrict__ dst) {
	int p = blockIdx.x * blockDim.x + threadIdx.x;
	int N = G.N, Nx = G.Nx, Ny = G.Ny;
	if(p >= N) return;
	int s = blockIdx.y;
	int g = (slot0 + s) / G.spg - slot0 / G.spg;
	Stencil<R> st{coef + (size_t)g * coef_set_size(N), N, Nx, Ny};
	const cx<R>* f0 = src + (size_t)s * 2 * N;
	int ix = p % Nx, iy = p / Nx;
#pragma unroll
	for(int c = 0; c < 2; c++) {
		cx<R> r;
		composite_m<R, KIND, 1>(st, c, ix, iy, f0, &r);
		dst[(size_t)s * 2 * N + (size_t)c * N + p] = r;
	}
}

// Periodic line solve with the pre-factored Thomas/Sherman-Morrison data, sequential form:
// one thread per (line, comp, slot). Used for lines too long for the chunked kernels.
// dst may alias src. If acc_out is set: acc_out = acc_in + x.
template <typename R, int DIRN>
__global__ void k_solve(Geom G, int slot0, int nslots, const cx<R>* __restrict__ fac, size_t plane,
		const cx<double>* __restrict__ lsc, const cx<R>* src, cx<R>* dst,
		const cx<R>* acc_in, cx<R>* acc_out) {
	int Nx = G.Nx, Ny = G.Ny, N = G.N;
	int L = DIRN == 0 ? Nx : Ny;
	int nlines = DIRN == 0 ? Ny : Nx;
	int t = blockIdx.x * blockDim.x + threadIdx.x;
	if(t >= nslots * 2 * nlines) return;
	int line = t % nlines;
	int c = (t / nlines) % 2;
	int s = t / (2 * nlines);
	int g = (slot0 + s) / G.spg - slot0 / G.spg;
	size_t off = (size_t)s * 2 * N + (size_t)c * N;
	const cx<R>* S = src + off;
	cx<R>* D = dst + off;
	const int stride = DIRN == 0 ? 1 : Nx;
	const int base = DIRN == 0 ? Nx * line : line;
	if(L <= 3) {
		for(int i = 0; i < L; i++) {
			int q = base + i * stride;
			cx<R> x = S[q];
			D[q] = x;
			if(acc_out) acc_out[off + q] = acc_in[off + q] + x;
		}
		return;
	}
	const cx<R>* Fc = fac + ((size_t)g * 2 + c) * NFAC * plane;
	const cx<double>* ls = lsc + (((size_t)g * 2 + c) * nlines + line) * 2;
	int q = base;
	cx<R> d = S[q] * Fc[F_RB * plane + q];
	cx<R> acc = d;
	D[q] = d;
	for(int i = 1; i < L - 1; i++) {
		q += stride;
		d = Fc[F_A * plane + q] * d + S[q] * Fc[F_RB * plane + q];
		acc += Fc[F_W * plane + q] * d;
		D[q] = d;
	}
	cx<double> frac = (cvt<double>(acc) - ls[0] * cvt<double>(d)) * ls[1];
	cx<R> fr = cvt<R>(frac);
	cx<R> dn = d;
	cx<R> x = dn - fr * Fc[F_COR * plane + q];
	D[q] = x;
	if(acc_out) acc_out[off + q] = acc_in[off + q] + x;
	for(int i = L - 2; i > 0; i--) {
		q -= stride;
		cx<R> dp = D[q] + Fc[F_C * plane + q] * dn;
		x = dp - fr * Fc[F_COR * plane + q];
		D[q] = x;
		if(acc_out) acc_out[off + q] = acc_in[off + q] + x;
		dn = dp;
	}
	int qe = base + (L - 1) * stride;
	D[qe] = x;  // duplicate point = x_0
	if(acc_out) acc_out[off + qe] = acc_in[off + qe] + x;
}

// x-line solve fused with the right-hand side that precedes it (KIND: explicit y half-step or
// x Woodbury term), chunked parallel form: one warp per (line, comp, KS slots of one
// wavelength); lane l owns the unknowns [l*M, l*M+M) of the line. The forward and backward
// recurrences are composed per chunk, combined by warp-shuffle scans and replayed, so every
// sweep is parallel over 32 lanes. The right-hand side is formed with each stencil
// coefficient loaded once for the KS slots and staged through shared memory so that global
// accesses stay coalesced; the factor planes are stored chunk-interleaved (element l*M+k at
// k*32+l) and are also loaded once for the KS slots. Block = LT warps = LT lines.
// ---------------------------------------------------------------------------------------
// The y-line solves as x-line solves of the transposed frame (x' = y, y' = x, components
// exchanged): the stencil blocks b become 3 - b (00 <-> 11, 01 <-> 10), the DX and DY stencils
// exchange, the DXDY corners (px,py), (mx,py), (px,my), (mx,my) become corners 0, 2, 1, 3, and the
// duplicate-row/column folding and the period-(N-1) wraps map onto themselves. k_coef writes the
// transposed sets those solves read (their phase entries are not used).

// Pre-factorisation of the periodic line solves (I - mu*R_cc) x = b per (group, comp, line), in
// the plan's precision. Restates shifted_block_vmult_inv (BlockSparseMatrix.cpp:195-258 and
// 386-449): Thomas sweep with beta0 = 2*mid0 and the Sherman-Morrison corner vector corr
// (corr0 = -1/2). Everything that does not depend on the right-hand side is computed here once
// per (wavelength, slab) and shared by all (q, pol) slots:
//   F_A    alpha_i = -inf_i/beta_i   F_RB  1/beta_i        F_C   -gamma_i
//   F_COR  corr_i after back-substitution
//   F_W    w_i = prod_{j<i}(-gamma_j), so that the back-substituted x_0 = sum_i w_i d_i
//          is formed during the forward sweep
// plus per line r0 = inf0/mid0 and rden = 1/(1 + corr0 - r0*corr_{L-2}) in FP64. The forward
// sweep of a solve is then d_i = alpha_i d_{i-1} + b_i/beta_i and the backward sweep
// x_{i-1} = d_{i-1} - gamma_{i-1} x_i: both first-order affine recurrences whose coefficients
// do not depend on b, which is what the chunked solves exploit.
// Chunk-parallel form: every line is split into chunks processed by different threads. The
// pivots follow the continued fraction
// beta_i = mid'_i - inf_i sup_{i-1} / beta_{i-1}, a Moebius map: (p, q) -> M_i (p, q) with
// M_i = [[mid'_i, -inf_i sup_{i-1}], [1, 0]] and beta = p / q. Each chunk forms the product of
// its maps (rescaled to keep it bounded; the map is projective), the chunk products are
// combined with an exclusive scan, and each chunk replays its elements from the pivot before
// it. corr (forward), the back-substituted corr and w are affine recurrences combined the same
// way. x-lines: one warp per line, lanes = chunks of chunkM elements (the interleaved factor
// layout), combined with shuffles. y-lines: 32 columns per block (lanes), warps = chunks of
// rows, combined through shared memory. Intermediate values go to the output planes and are
// read back by the same thread.
template <typename T>
struct Aff {
	cx<T> A, B;  // x -> A x + B
};
template <typename T>
__device__ __forceinline__ Aff<T> aff_after(const Aff<T>& second, const Aff<T>& first) {
	return Aff<T>{second.A * first.A, second.A * first.B + second.B};
}
template <typename T>
__device__ __forceinline__ Aff<T> shfl_up_a(const Aff<T>& X, int o) { return Aff<T>{shfl_up_c(X.A, o), shfl_up_c(X.B, o)}; }
template <typename T>
__device__ __forceinline__ Aff<T> shfl_down_a(const Aff<T>& X, int o) { return Aff<T>{shfl_down_c(X.A, o), shfl_down_c(X.B, o)}; }

template <typename S, int DIRN>
__global__ void __launch_bounds__(DIRN == 1 ? 512 : 256) k_factor_chunked(Geom G, int ngroups, int chunkMx, int chunksX, int W,
		const cx<S>* __restrict__ coef, cx<S>* __restrict__ fac, size_t plane, cx<double>* __restrict__ lsc) {
	typedef S T;
	const int Nx = G.Nx, Ny = G.Ny, N = G.N;
	const int L = DIRN == 0 ? Nx : Ny;
	const int nlines = DIRN == 0 ? Ny : Nx;
	const int n = L - 1;
	const int lane = threadIdx.x, w = threadIdx.y;
	int line, gc, chunk, nchunks, M;
	if(DIRN == 0) {
		line = blockIdx.x * blockDim.y + w;
		gc = blockIdx.y;
		chunk = lane;
		nchunks = 32;
		M = (n + 31) / 32;
	}
	else {
		line = blockIdx.x * 32 + lane;
		gc = blockIdx.y;
		chunk = w;
		nchunks = W;
		M = (n + W - 1) / W;
	}
	const bool active = line < nlines && L > 3;
	const int g = gc / 2, c = gc % 2;
	const int i0 = chunk * M, i1 = min(i0 + M, n);
	const cx<T>* Cg = coef + (size_t)g * coef_set_size(N);
	cx<S>* Fc = fac + ((size_t)g * 2 + c) * NFAC * plane;
	const int stride = DIRN == 0 ? 1 : Nx;
	const int base = DIRN == 0 ? Nx * line : line;
	auto P = [&](int i) { return base + i * stride; };
	// storage of factor f of element i: natural layout (plane f, point P(i)), or the solves'
	// chunk-interleaved x layout: chunksX chunks of chunkMx elements per line, element
	// i = ci*chunkMx + k of factor f at ((line*chunkMx + k)*NFAC + f)*chunksX + ci, so that the
	// factors a lane reads for one element are compile-time offsets from one address
	auto Q = [&](int f, int i) -> size_t {
		if(DIRN == 1 || chunkMx <= 0) return (size_t)f * plane + P(i);
		return (((size_t)line * chunkMx + i % chunkMx) * NFAC + f) * chunksX + (i / chunkMx);
	};
	const cx<T> one = mk<T>(1, 0), zero = mk<T>(0, 0);
	auto sup = [&](int i) { cx<T> m, cc, n; coef_diag<DIRN>(Cg, c, P(i), m, cc, n); return -n; };
	auto mid = [&](int i) { cx<T> m, cc, n; coef_diag<DIRN>(Cg, c, P(i), m, cc, n); return one - cc; };
	auto inf = [&](int i) { cx<T> m, cc, n; coef_diag<DIRN>(Cg, c, P(i), m, cc, n); return -m; };
	cx<T> m0 = zero, a0 = zero, corner = zero;
	if(active) {
		m0 = mid(0);
		a0 = inf(0);
		corner = cdiv(sup(n - 1) * a0, m0);
	}
	auto midp = [&](int i) { return i == n - 1 ? mid(i) + corner : mid(i); };
	// shared memory for the y combine: [W][32] per quantity
	extern __shared__ unsigned char smem_raw[];
	Mob<T>* shM = reinterpret_cast<Mob<T>*>(smem_raw);
	Aff<T>* shA = reinterpret_cast<Aff<T>*>(shM + (DIRN == 1 ? W * 32 : 0));
	Aff<T>* shB = shA + (DIRN == 1 ? W * 32 : 0);
	cx<T>* shX = reinterpret_cast<cx<T>*>(shB + (DIRN == 1 ? W * 32 : 0));  // [2][32] corr_last, cv0

	// ---- 1. pivots: chunk product of the Moebius maps ----
	Mob<T> Pm{one, zero, zero, one};
	if(active) {
		for(int i = i0; i < i1; i++) {
			Mob<T> Mi;
			if(i == 0) Mi = Mob<T>{zero, (T)2 * m0, zero, one};
			else Mi = Mob<T>{midp(i), -(inf(i) * sup(i - 1)), one, zero};
			Pm = mob_mul(Mi, Pm);
			mob_norm(Pm);
		}
	}
	// exclusive scan over chunks in order: Sx = P_{c-1} ... P_0
	Mob<T> Sx{one, zero, zero, one};
	if(DIRN == 0) {
		Mob<T> X = Pm;
#pragma unroll
		for(int o = 1; o < 32; o <<= 1) {
			Mob<T> Y = shfl_up_m(X, o);
			if(lane >= o) { X = mob_mul(X, Y); mob_norm(X); }
		}
		Mob<T> E = shfl_up_m(X, 1);
		if(lane > 0) Sx = E;
	}
	else {
		shM[w * 32 + lane] = Pm;
		__syncthreads();
		if(w == 0) {
			Mob<T> acc{one, zero, zero, one};
			for(int k = 0; k < W; k++) {
				Mob<T> pk = shM[k * 32 + lane];
				shM[k * 32 + lane] = acc;
				acc = mob_mul(pk, acc);
				mob_norm(acc);
			}
		}
		__syncthreads();
		Sx = shM[w * 32 + lane];
	}
	// replay: beta, and the chunk maps of corr (forward) and w
	// (the divisions by the previous pivot are multiplications by its reciprocal, computed one step
	// earlier)
	Aff<T> Fcorr{one, zero}, Fw{one, zero};
	cx<T> rb_prev = zero;
	if(active && i0 < i1) {
		if(i0 > 0) rb_prev = crecip(cdiv(Sx.b, Sx.d));  // state before the chunk: Sx . (0, 1)
		for(int i = i0; i < i1; i++) {
			cx<T> beta = i == 0 ? (T)2 * m0 : midp(i) - (inf(i) * sup(i - 1)) * rb_prev;
			cx<T> rb = crecip(beta);
			cx<T> alpha = i == 0 ? zero : -(inf(i) * rb);
			Fc[Q(F_RB, i)] = cvt<S>(rb);
			Fc[Q(F_A, i)] = cvt<S>(alpha);
			Fc[Q(F_C, i)] = i < n - 1 ? cvt<S>(-(sup(i) * rb)) : mk<S>(0, 0);
			// corr_0 = -1/2, corr_i = alpha_i corr_{i-1} (+ sup_{n-1} rb_{n-1} on the last row)
			Aff<T> ec = i == 0 ? Aff<T>{zero, mk<T>(-0.5, 0)} : Aff<T>{alpha, i == n - 1 ? sup(i) * rb : zero};
			Fcorr = aff_after(ec, Fcorr);
			// w_0 = 1, w_i = -gamma_{i-1} w_{i-1}, gamma_{i-1} = sup_{i-1} / beta_{i-1}
			Aff<T> ew = i == 0 ? Aff<T>{zero, one} : Aff<T>{-(sup(i - 1) * rb_prev), zero};
			Fw = aff_after(ew, Fw);
			rb_prev = rb;
		}
	}
	// ---- 2. exclusive scans of the corr and w maps, replay ----
	Aff<T> Ec{one, zero}, Ew{one, zero};
	if(DIRN == 0) {
		Aff<T> Xc = Fcorr, Xw = Fw;
#pragma unroll
		for(int o = 1; o < 32; o <<= 1) {
			Aff<T> Yc = shfl_up_a(Xc, o), Yw = shfl_up_a(Xw, o);
			if(lane >= o) { Xc = aff_after(Xc, Yc); Xw = aff_after(Xw, Yw); }
		}
		Aff<T> Pc = shfl_up_a(Xc, 1), Pw = shfl_up_a(Xw, 1);
		if(lane > 0) { Ec = Pc; Ew = Pw; }
	}
	else {
		__syncthreads();
		shA[w * 32 + lane] = Fcorr;
		shB[w * 32 + lane] = Fw;
		__syncthreads();
		if(w == 0) {
			Aff<T> ac{one, zero}, aw{one, zero};
			for(int k = 0; k < W; k++) {
				Aff<T> fc = shA[k * 32 + lane], fw = shB[k * 32 + lane];
				shA[k * 32 + lane] = ac;
				shB[k * 32 + lane] = aw;
				ac = aff_after(fc, ac);
				aw = aff_after(fw, aw);
			}
		}
		__syncthreads();
		Ec = shA[w * 32 + lane];
		Ew = shB[w * 32 + lane];
	}
	if(DIRN == 0) __syncwarp();  // F_C of the previous chunk, written by another lane
	cx<T> corr_last = zero;
	bool own_last = active && i0 <= n - 1 && n - 1 < i1;
	if(active && i0 < i1) {
		cx<T> cr = Ec.B, wv = Ew.B;  // values before the chunk (maps applied to 0)
		for(int i = i0; i < i1; i++) {
			cx<T> alpha = cvt<T>(Fc[Q(F_A, i)]);
			cx<T> rb = cvt<T>(Fc[Q(F_RB, i)]);
			if(i == 0) { cr = mk<T>(-0.5, 0); wv = one; }
			else {
				cx<T> gm = -cvt<T>(Fc[Q(F_C, i - 1)]);  // gamma_{i-1}
				cr = cfma(alpha, cr, (i == n - 1 ? sup(i) * rb : zero));
				wv = -(gm * wv);
			}
			Fc[Q(F_COR, i)] = cvt<S>(cr);  // forward corr, replaced below
			Fc[Q(F_W, i)] = cvt<S>(wv);
			if(i == n - 1) corr_last = cr;
		}
	}
	// broadcast corr_last to the line
	if(DIRN == 0) {
		corr_last = shfl_idx_c(corr_last, (n - 1) / M);
	}
	else {
		__syncthreads();
		if(own_last) shX[lane] = corr_last;
		__syncthreads();
		corr_last = shX[lane];
	}
	// ---- 3. back-substituted corr: cv_{n-1} = corr_last, cv_j = -gamma_j cv_{j+1} + corr_j ----
	Aff<T> Bm{one, zero};
	if(active && i0 < i1) {
		for(int j = i1 - 1; j >= i0; j--) {
			Aff<T> e = j == n - 1 ? Aff<T>{zero, corr_last}
				: Aff<T>{cvt<T>(Fc[Q(F_C, j)]), cvt<T>(Fc[Q(F_COR, j)])};
			Bm = aff_after(e, Bm);
		}
	}
	Aff<T> Eb{one, zero};
	if(DIRN == 0) {
		Aff<T> X = Bm;
#pragma unroll
		for(int o = 1; o < 32; o <<= 1) {
			Aff<T> Y = shfl_down_a(X, o);
			if(lane + o < 32) X = aff_after(X, Y);
		}
		Aff<T> Nn = shfl_down_a(X, 1);
		if(lane < 31) Eb = Nn;
	}
	else {
		__syncthreads();
		shA[w * 32 + lane] = Bm;
		__syncthreads();
		if(w == 0) {
			Aff<T> acc{one, zero};
			for(int k = W - 1; k >= 0; k--) {
				Aff<T> f = shA[k * 32 + lane];
				shA[k * 32 + lane] = acc;
				acc = aff_after(f, acc);
			}
		}
		__syncthreads();
		Eb = shA[w * 32 + lane];
	}
	cx<T> cv0 = zero;
	if(active && i0 < i1) {
		cx<T> cv = Eb.B;  // cv of the element after the chunk
		for(int j = i1 - 1; j >= i0; j--) {
			cv = j == n - 1 ? corr_last
				: cvt<T>(Fc[Q(F_C, j)]) * cv + cvt<T>(Fc[Q(F_COR, j)]);
			Fc[Q(F_COR, j)] = cvt<S>(cv);
		}
		if(i0 == 0) cv0 = cv;
	}
	// padding of the interleaved x layout: identity maps
	if(DIRN == 0 && chunkMx > 0 && active) {
		for(int i = n + lane; i < chunksX * chunkMx; i += 32) {
			Fc[Q(F_A, i)] = mk<S>(0, 0);
			Fc[Q(F_RB, i)] = mk<S>(0, 0);
			Fc[Q(F_W, i)] = mk<S>(0, 0);
			Fc[Q(F_C, i)] = mk<S>(0, 0);
			Fc[Q(F_COR, i)] = mk<S>(0, 0);
		}
	}
	// Sherman-Morrison scalars in FP64
	if(active && chunk == 0) {
		cx<double>* ls = lsc + (((size_t)g * 2 + c) * nlines + line) * 2;
		cx<double> r0 = cdiv(cvt<double>(a0), cvt<double>(m0));
		ls[0] = r0;
		ls[1] = crecip(mk(1.0, 0.0) + cvt<double>(cv0) - r0 * cvt<double>(corr_last));
	}
}

// Pre-factorisation for the partitioned x-line solves (k_solve_xc, k_solve_xw): CH = 32 * W chunks
// of M points per line, one thread per chunk. Every chunk is factored by itself (LU without pivoting
// of a principal submatrix of I - mu*R_cc), so there is no scan along the line; what couples the
// chunks is the 2x2 interface system of neighbouring chunks' border unknowns (I_* above). The line
// scalar lsc[line][0].x receives the number of Jacobi steps K that the interface system needs to
// reach rounding: a step multiplies the error by rho, the largest row sum of the interface couplings,
// about the M-th power of the decay from point to point (K = 0 for 8-point chunks at the usual mesh
// spacings in FP32, 1 in FP64). Where that would be more than PART_KMAX steps (spacings far below a
// wavelength, a last chunk of few points) and on lines of one chunk K is -1 and the line is joined exactly by
// ring_solve, which costs about as much as PART_KMAX steps at any coupling.
// Bound: HBM and the latency of the reciprocals (M in a row). The scans over Moebius and affine maps
// of k_factor_chunked it replaces here took 107 us per launch on the 256x256, 16-wavelength FP32 case
// and 47 us on a 64x64 FP64 one.
constexpr int PART_KMAX = 10;
// a function of its own, so that it takes no registers from the other lines
template <bool MULTI, typename S>
__device__ __noinline__ RingNode<S> part_ring_factor(LineThreads T, cx<S> ph, cx<S> pg, cx<S> qh, cx<S> qg, cx<S>* sh) {
	return ring_factor<MULTI>(T, ph, pg, qh, qg, sh);
}
// Registers: 64 in FP64 and 48 in FP32, what the chunks' sweeps take (without the bound ring_factor's make it 102 and
// 63: a 128x128x64 FP64 step 8.8 -> 10.0 ms).
template <typename S>
__global__ void __launch_bounds__(256, sizeof(S) == sizeof(double) ? 4 : 5) k_factor_part(Geom G, int M, const cx<S>* __restrict__ coef,
		cx<S>* __restrict__ fac, size_t plane, cx<double>* __restrict__ lsc) {
	const int N = G.N, nlines = G.Ny, n = G.Nx - 1;
	const int CH = blockDim.x, t = threadIdx.x;
	const int line = blockIdx.x * blockDim.y + threadIdx.y;
	const int gc = blockIdx.y, g = gc / 2, c = gc % 2;
	const bool active = line < nlines && G.Nx > 3;
	const int nchk = (n + M - 1) / M;
	const cx<S>* Cg = coef + (size_t)g * coef_set_size(N);
	const int p0 = line * G.Nx;
	cx<S>* Fc = fac + (size_t)gc * NFAC * plane + (size_t)line * part_line_size(M, CH);
	cx<S>* If = Fc + (size_t)M * NFAC * CH;
	cx<double>* ls = lsc + ((size_t)gc * nlines + line) * 2;
	const cx<S> one = mk<S>(1, 0), zero = mk<S>(0, 0);
	// border responses to the unknowns before (v) and after (w) the chunk, and the last 1/beta
	cx<S> vf = zero, vl = zero, wf = zero, wl = zero, rbl = zero;
	// 1 / b with one division: the pivots are 1 + O(dz / (k0 n dx^2)), far from the ends of the range
	auto recip = [](cx<S> b) {
		const S r = (S)1 / (b.x * b.x + b.y * b.y);
		return mk(b.x * r, -b.y * r);
	};
	const int i0 = t * M;
	const bool own = active && i0 < n;
	// base: lines of weak coupling (|1/beta| > 0.6), by their chunks' first points
	cx<S> em = zero, ec = zero, en = zero;
	if(own) coef_diag<0>(Cg, c, p0 + i0, em, ec, en);
	const bool weak = l1abs(ec) < (S)1;
	const S base = (CH > 32 ? __syncthreads_and(weak) : __all_sync(0xffffffffu, weak)) ? 1 : 0;
	if(own) {
		const int m = min(M, n - i0);
		cx<S> rb = zero, cprev = zero, ev = zero, cpz = one;
		for(int k = 0; k < m; k++) {
			if(k) coef_diag<0>(Cg, c, p0 + i0 + k, em, ec, en);
			const cx<S> a = -em, cs = -en;
			cx<S> al = zero;  // -l
			if(k == 0) ev = -a;
			else {
				al = -(a * rb);
				ev = al * ev;
			}
			const cx<S> b1 = k == 0 ? -ec : cfma(al, cprev, -ec);  // beta - 1
			rb = recip(one + b1);
			cprev = cs;
			const cx<S> db = base != 0 ? -(rb * b1) : rb, cc = -(rb * cs), z = cpz * rb, e = rb * ev;
			cx<S>* F = Fc + (size_t)k * NFAC * CH;
			reinterpret_cast<v4<S>*>(F)[t] = v4<S>{al.x, al.y, z.x, z.y};
			reinterpret_cast<v4<S>*>(F + 2 * CH)[t] = v4<S>{db.x, db.y, cc.x, cc.y};
			F[4 * CH + t] = e;
			vf = cfma(z, ev, vf);
			cpz = cpz * cc;
			vl = e;
			wl = cc;
		}
		wf = cpz;
		rbl = rb;
	}
	if(active) {
		// past the line's end: entries that leave the sweeps' values as they are, so that the solves need no
		// condition at every point (a branch there makes each point wait for its own factors)
		for(int k = max(0, min(M, n - i0)); k < M; k++) {
			cx<S>* F = Fc + (size_t)k * NFAC * CH;
			reinterpret_cast<v4<S>*>(F)[t] = v4<S>{1, 0, 0, 0};
			reinterpret_cast<v4<S>*>(F + 2 * CH)[t] = v4<S>{-base, 0, 1, 0};
			F[4 * CH + t] = zero;
		}
	}
	// the next chunk's responses (cyclic), through shared memory
	__shared__ cx<S> shv[256], shw[256];
	__shared__ S shr[8];
	const int tid = threadIdx.y * CH + t;
	shv[tid] = vf;
	shw[tid] = wf;
	__syncthreads();
	S rho = 0;
	cx<S> ph = zero, pg = zero, qh = zero, qg = zero, hd = zero, hy = zero, gd = zero, gy = zero;
	if(own) {
		const int nx = threadIdx.y * CH + (t == nchk - 1 ? 0 : t + 1);
		const cx<S> vfn = shv[nx], wfn = shw[nx];
		const cx<S> m = recip(cfnma(wl, vfn, one));
		const cx<S> mw = m * wl, mv = m * vfn;
		ph = m * vl; pg = mv * vl; qh = mw * wfn; qg = m * wfn;
		hd = m * rbl; hy = mw; gd = mv * rbl; gy = m;
		rho = fmax(l1abs(ph) + l1abs(qh), l1abs(pg) + l1abs(qg));
		if(!(rho < (S)1)) rho = 1;  // NaN too
	}
	// largest rho of the line
#pragma unroll
	for(int o = 16; o > 0; o >>= 1) rho = fmax(rho, __shfl_xor_sync(0xffffffffu, rho, o));
	if(CH > 32) {
		if(t % 32 == 0) shr[tid / 32] = rho;
		__syncthreads();
		for(int w = 0; w < CH / 32; w++) rho = fmax(rho, shr[w]);
	}
	const S lt = sizeof(S) == sizeof(float) ? (S)-18.7 : (S)-39.5;  // ln of 2^-27, 2^-57
	int K = 0;
	if(nchk < 2 || !(rho < (S)1)) K = -1;
	else if(rho > (S)0 && log(rho) > lt) {
		const S k = ceil(lt / log(rho)) - 1;
		K = k <= (S)PART_KMAX ? (int)k : -1;
	}
	if(active && t == 0) ls[0] = mk((double)K, (double)base);
	auto put = [&](int f, cx<S> v) { if(own) If[f * CH + t] = v; };
	if(K >= 0) {
		put(I_PH, ph); put(I_PG, pg); put(I_QH, qh); put(I_QG, qg);
	}
	else {
		// the same for all threads of a line: a warp, or the block
		const LineThreads T{CH / 32, 0, t / 32, t % 32, t, nchk - 1};
		__shared__ cx<S> shf[ring_factor_shared(8)];
		const RingNode<S> r = CH > 32 ? part_ring_factor<true>(T, ph, pg, qh, qg, shf) : part_ring_factor<false>(T, ph, pg, qh, qg, shf);
		hd = cfma(r.f2, gd, hd); hy = cfma(r.f2, gy, hy);
		gd = r.d * gd; gy = r.d * gy;
		#pragma unroll
		for(int k = 0; k < RN_ALL; k++) put(k < 4 ? I_F + k : I_ETA + k - 4, r.v[k]);
		if(active && t < 4) If[I_X * CH + t] = r.X[t];
	}
	put(I_HD, hd); put(I_HY, hy); put(I_GD, gd); put(I_GY, gy);
}

// v / beta from F_DB. FP64, whose pipe is the bound, takes a sweep for each base (ONE) and no product with it.
template <bool B>
struct Flag {
	static constexpr bool on = B;
};
template <bool ONE, typename R>
__device__ __forceinline__ cx<R> from_base(cx<R> db, R base, cx<R> v) {
	if(sizeof(R) == sizeof(double)) return ONE ? cfma(db, v, v) : db * v;
	return cfma(db, v, mk<R>(base * v.x, base * v.y));
}
template <typename R, typename F>
__device__ __forceinline__ void with_base(R base, F sweep) {
	if(sizeof(R) == sizeof(float) || base != 0) sweep(Flag<true>());
	else sweep(Flag<false>());
}

// The node coefficients of a thread's chunk on a line flagged -1 by k_factor_part (If: its interface coefficients, CH
// apart), read when they are used.
template <typename R>
struct PartNode {
	const cx<R>*If, *close0;
	int CH;
	__device__ __forceinline__ cx<R> get(int k) const { return If[(k < 4 ? I_F + k : I_ETA + k - 4) * CH]; }
	__device__ __forceinline__ cx<R> close(int k) const { return close0[k]; }
};
// Border unknowns of a chunk: on entry h and g from the two chunks alone, on return what the backward sweep
// takes, the previous chunk's last unknown and the next one's first.
template <typename V, int KS>
struct Border {
	V h[KS], x[KS];
};
// Such a line's join. A function of its own, so that it takes no registers from the other lines.
template <bool MULTI, int KS, typename R, typename V>
__device__ __noinline__ Border<V, KS> part_ring(LineThreads T, const cx<R>* If, int CH, Border<V, KS> b, V* s) {
	V hl[KS];
	ring_solve<MULTI, KS, R>(T, PartNode<R>{If, If - T.ci + I_X * CH, CH}, b.h, b.x, hl, s);
#pragma unroll
	for(int j = 0; j < KS; j++) b.h[j] = hl[j];
	return b;
}

// One combine of the chunk maps of a line whose chunks sit on the 32 lanes of a warp (chunk =
// lane; lanes past the line carry identity maps). Inputs per lane: forward map (P, d0[j]),
// sum terms (S0[j], S1), backward terms (Cp, G0[j], G1). Outputs per lane: din = the forward
// value entering the chunk, xin = the backward value entering it from the line's end, and
// fr = (sum_i w_i d_i - r0 * d_last) * rden, the Sherman-Morrison factor (same on all lanes).
template <typename R, int KS>
__device__ __forceinline__ void line_combine(cx<R> P, const cx<R>* d0, const cx<R>* S0, cx<R> S1, const cx<R>* G0,
		cx<R> G1, cx<R> Cp, cx<double> r0, cx<double> rden, int lane, cx<R>* din, cx<R>* xin, cx<R>* fr) {
	const cx<R> zero = mk<R>(0, 0);
	cx<R> B[KS];
#pragma unroll
	for(int j = 0; j < KS; j++) B[j] = d0[j];
#pragma unroll
	for(int o = 1; o < 32; o <<= 1) {
		const cx<R> Pp = shfl_up_c(P, o);
#pragma unroll
		for(int j = 0; j < KS; j++) {
			const cx<R> Bp = shfl_up_c(B[j], o);
			if(lane >= o) B[j] = cfma(P, Bp, B[j]);
		}
		if(lane >= o) P = P * Pp;
	}
	cx<R> G[KS];
	cx<R> tsel = zero, dsel = zero;  // lane j < KS keeps slot j's sum and last value
#pragma unroll
	for(int j = 0; j < KS; j++) {
		din[j] = shfl_up_c(B[j], 1);
		if(lane == 0) din[j] = zero;
		cx<R> t = cfma(S1, din[j], S0[j]);
#pragma unroll
		for(int o = 16; o > 0; o >>= 1) t += shfl_xor_c(t, o);
		const cx<R> dl = shfl_idx_c(B[j], 31);
		if(lane == j) { tsel = t; dsel = dl; }
		G[j] = cfma(G1, din[j], G0[j]);
	}
	// the FP64 factor once per slot (lane j), then broadcast
	cx<R> f = zero;
	if(lane < KS) f = cvt<R>((cvt<double>(tsel) - r0 * cvt<double>(dsel)) * rden);
#pragma unroll
	for(int j = 0; j < KS; j++) fr[j] = shfl_idx_c(f, j);
#pragma unroll
	for(int o = 1; o < 32; o <<= 1) {
		const cx<R> Cn = shfl_down_c(Cp, o);
#pragma unroll
		for(int j = 0; j < KS; j++) {
			const cx<R> Gn = shfl_down_c(G[j], o);
			if(lane + o < 32) G[j] = cfma(Cp, Gn, G[j]);
		}
		if(lane + o < 32) Cp = Cp * Cn;
	}
#pragma unroll
	for(int j = 0; j < KS; j++) {
		xin[j] = shfl_down_c(G[j], 1);
		if(lane == 31) xin[j] = zero;
	}
}

// Programmatic dependent launch: the solves that follow each other on a slab's main stream are launched
// while their predecessor still runs (solve_dispatch.cuh) and wait here for its end, before they touch
// any field; then they let their own successor be launched. Saves the launch latency between them. Without
// the launch attribute both do nothing.
__device__ __forceinline__ void wait_predecessor() {
	asm volatile("griddepcontrol.wait;" ::: "memory");
	asm volatile("griddepcontrol.launch_dependents;");
}

// x-line solve fused with its right-hand side (KIND: explicit y half-step or x Woodbury term):
// a warp per line (4 lines per block) for KS slots of one wavelength. The right-hand sides are
// computed with coalesced loads into the warp's shared buffer in the lane-chunk layout (lane l
// holds points [l M, l M + M)); every lane sweeps forward through its chunk, the lanes join through
// the border unknowns of neighbouring chunks (k_factor_part), and a backward sweep with those known
// finishes the line, which goes back out coalesced.
// Bound: L1 wavefronts (73 %) and load latency (issue active 50 %). Partitioning in place of forward,
// sum and backward maps joined by shuffle scans: 20 instead of 28 multiply-adds per point and slot, 5
// instead of 7 factor loads, and no scans (5 shuffle steps each over 3 quantities) but on strongly coupled lines (part_ring). 256x256, 16
// wavelengths, 13 q, FP32: Woodbury solves 552 -> 490 us, explicit step 499 -> 476 us; the same mesh
// with 3 wavelengths in FP64 (bound by the FP64 pipe) 1351 -> 962 and 1540 -> 1162 us. With the real
// entries of the coefficient set (4 x-taps and 10 with one real number each in place of 14 complex
// ones for the Woodbury term): FP32 490 -> 477 and 476 -> 491 us, FP64 962 -> 785 and 1162 -> 923 us.
template <typename R, int M, int KIND, int KS, bool TOUT = false>
// Resident blocks per SM requested from the compiler: 8 (64 registers) for the instances
// whose chunk values fit, measured faster on GB300; the larger instances keep their registers.
#ifndef NBPM_XC_MINB
#define NBPM_XC_MINB(MK) ((MK) <= 16 ? 8 : 1)
#endif
#ifndef NBPM_YC_MINB
#define NBPM_YC_MINB 1
#endif
// TOUT: the results go out transposed with the two components exchanged ((c, iy, e) -> (1 - c,
// e, iy) of an Ny x Nx plane), written by the whole block so that each (point, LT lines) group
// is one 32-byte segment: the hand-over between the x-line frame and the transposed frame in
// which the y-lines are solved as x-lines (ADI with transposed y solves).
__global__ void __launch_bounds__(128, NBPM_XC_MINB(M * KS)) k_solve_xc(Geom G, int slot0, int nch, const cx<R>* __restrict__ coef,
		const cx<R>* __restrict__ fac, size_t plane, const cx<double>* __restrict__ lsc,
		const cx<R>* __restrict__ src, cx<R>* __restrict__ dst, const cx<R>* acc_in, cx<R>* acc_out,
		const cx<R>* acc_in2) {
	extern __shared__ unsigned char smem_raw[];
	wait_predecessor();
	constexpr int LT = 4;  // lines (warps) per block: launched with 128 threads
	const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
	const int Nx = G.Nx, Ny = G.Ny, N = G.N;
	const int iy = blockIdx.x * LT + warp;
	if(!TOUT && iy >= Ny) return;
	const int c = blockIdx.y % 2, bc = blockIdx.y / 2;
	const int g = bc / nch, ch = bc % nch;
	const int s0 = g * G.spg + ch * KS;  // first slot (pass-relative)
	const int n_unk = Nx - 1;
	const int PITCH = 32 * part_pitch(M);
	cx<R>* buf = reinterpret_cast<cx<R>*>(smem_raw) + (size_t)warp * KS * PITCH;
	if(iy < Ny) {  // always true unless TOUT (whose block writes together after a barrier)
	const cx<R>* Fc = fac + ((size_t)g * 2 + c) * NFAC * plane + (size_t)iy * part_line_size(M, 32);
	const cx<double> kb = lsc[(((size_t)g * 2 + c) * Ny + iy) * 2];
	const int K = (int)kb.x;
	const R base = (R)kb.y;
	const cx<R> zero = mk<R>(0, 0);
	const Stencil<R> st{coef + (size_t)g * coef_set_size(N), N, Nx, Ny};
	const cx<R>* f0 = src + (size_t)s0 * 2 * N;
	// right-hand sides, coalesced (point e = lane + 32 t), into the lane-chunk layout of buf; the
	// fixed trip count (rolled, unroll 2 and 4 measured slower on GB300) beats a loop to n_unk
#pragma unroll 1
	for(int t = 0; t < M; t++) {
		const int e = lane + 32 * t;
		cx<R> r[KS];
		if(e < n_unk) composite_m<R, KIND, KS>(st, c, e, iy, f0, r);
		else {
#pragma unroll
			for(int j = 0; j < KS; j++) r[j] = zero;
		}
#pragma unroll
		for(int j = 0; j < KS; j++) buf[j * PITCH + (e / M) * part_pitch(M) + e % M] = r[j];
	}
	__syncwarp();
	{
		// forward sweep of the lane's chunk (written back over the right-hand sides) and its first
		// unknown yf with nothing outside the chunk
		cx<R> d[KS], yf[KS];
		cx<R>* vb = buf + lane * part_pitch(M);
#pragma unroll
		for(int j = 0; j < KS; j++) d[j] = yf[j] = zero;
#pragma unroll
		for(int k = 0; k < M; k++) {
			const v4<R> az = part_az(Fc, k, 32, lane);
			const cx<R> z = mk(az.z, az.w);
			if(k == 0) {
#pragma unroll
				for(int j = 0; j < KS; j++) { d[j] = vb[j * PITCH]; yf[j] = z * d[j]; }
			}
			else {
				const cx<R> a = mk(az.x, az.y);
#pragma unroll
				for(int j = 0; j < KS; j++) {
					d[j] = cfma(a, d[j], vb[j * PITCH + k]);
					vb[j * PITCH + k] = d[j];
					yf[j] = cfma(z, d[j], yf[j]);
				}
			}
		}
		// interface unknowns: h (the chunk's last) and g (the next chunk's first)
		const int last = (n_unk - 1) / M;  // last chunk
		const int left = lane == 0 ? last : lane - 1, right = lane == last ? 0 : (lane + 1) & 31;
		const cx<R>* If = Fc + (size_t)M * NFAC * 32 + lane;
		cx<R> h[KS], x[KS];
		{
			const cx<R> hd = If[I_HD * 32], hy = If[I_HY * 32], gd = If[I_GD * 32], gy = If[I_GY * 32];
#pragma unroll
			for(int j = 0; j < KS; j++) {
				const cx<R> yn = shfl_idx_c(yf[j], right);
				h[j] = cfma(hy, yn, hd * d[j]);
				x[j] = cfma(gy, yn, gd * d[j]);
			}
		}
		if(K > 0) {
			const cx<R> ph = If[I_PH * 32], pg = If[I_PG * 32], qh = If[I_QH * 32], qg = If[I_QG * 32];
			cx<R> bh[KS], bg[KS];
#pragma unroll
			for(int j = 0; j < KS; j++) { bh[j] = h[j]; bg[j] = x[j]; }
#pragma unroll 1
			for(int k = 0; k < K; k++) {
#pragma unroll
				for(int j = 0; j < KS; j++) {
					const cx<R> hl = shfl_idx_c(h[j], left), gr = shfl_idx_c(x[j], right);
					h[j] = cfma(qh, gr, cfma(ph, hl, bh[j]));
					x[j] = cfma(qg, gr, cfma(pg, hl, bg[j]));
				}
			}
		}
		if(K >= 0) {
#pragma unroll
			for(int j = 0; j < KS; j++) h[j] = shfl_idx_c(h[j], left);
		}
		else {
			Border<cx<R>, KS> b;
#pragma unroll
			for(int j = 0; j < KS; j++) { b.h[j] = h[j]; b.x[j] = x[j]; }
			b = part_ring<false, KS, R>(LineThreads{1, 0, 0, lane, lane, last}, If, 32, b, (cx<R>*)nullptr);
#pragma unroll
			for(int j = 0; j < KS; j++) { h[j] = b.h[j]; x[j] = b.x[j]; }
		}
		// backward sweep from the next chunk's first unknown, with the previous chunk's last one
		with_base(base, [&](auto one) {
#pragma unroll
			for(int k = M - 1; k >= 0; k--) {
				const v4<R> rc = part_rc(Fc, k, 32, lane);
				const cx<R> db = mk(rc.x, rc.y), cc = mk(rc.z, rc.w), ee = part_e(Fc, k, 32, lane);
#pragma unroll
				for(int j = 0; j < KS; j++) {
					x[j] = cfma(cc, x[j], cfma(ee, h[j], from_base<decltype(one)::on>(db, base, vb[j * PITCH + k])));
					vb[j * PITCH + k] = x[j];
				}
			}
		});
	}
	// the explicit-step solves never accumulate; the accumulating ones load the accumulator inputs
	// of several points before storing any (their latency would otherwise be paid point by point)
	const bool acc = KIND != ST_EXPL_Y && acc_out;
	if(!TOUT) {
	__syncwarp();
	constexpr int U = 3;
#pragma unroll 1
	for(int t0 = 0; t0 <= M; t0 += U) {
		cx<R> a[U][KS];
		if(acc) {
#pragma unroll
			for(int u = 0; u < U; u++) {
				const int e = lane + 32 * (t0 + u);
				if(t0 + u <= M && e < Nx)
#pragma unroll
					for(int j = 0; j < KS; j++) {
						const size_t o = (size_t)(s0 + j) * 2 * N + (size_t)c * N + (size_t)iy * Nx + e;
						a[u][j] = acc_in2 ? acc_in[o] + acc_in2[o] : acc_in[o];
					}
			}
		}
#pragma unroll
		for(int u = 0; u < U; u++) {
			const int e = lane + 32 * (t0 + u);
			if(t0 + u <= M && e < Nx) {
				const int ee = e == Nx - 1 ? 0 : e;
#pragma unroll
				for(int j = 0; j < KS; j++) {
					const size_t o = (size_t)(s0 + j) * 2 * N + (size_t)c * N + (size_t)iy * Nx + e;
					const cx<R> x = buf[j * PITCH + (ee / M) * part_pitch(M) + ee % M];
					if(dst) dst[o] = x;
					if(acc) acc_out[o] = a[u][j] + x;
				}
			}
		}
	}
	}
	}  // iy < Ny
	if(TOUT) {
		__syncthreads();
		const cx<R>* bufs = reinterpret_cast<const cx<R>*>(smem_raw);
		const bool acc = KIND != ST_EXPL_Y && acc_out;
		constexpr int U = 4, BT = 32 * LT;
		for(int t0 = threadIdx.x; t0 < Nx * LT; t0 += U * BT) {
			cx<R> a[U][KS];
			if(acc) {
#pragma unroll
				for(int u = 0; u < U; u++) {
					const int t = t0 + u * BT, e = t / LT, line = blockIdx.x * LT + t % LT;
					if(t < Nx * LT && line < Ny)
#pragma unroll
						for(int j = 0; j < KS; j++) {
							const size_t in = (size_t)(s0 + j) * 2 * N + (size_t)c * N + (size_t)line * Nx + e;
							a[u][j] = acc_in2 ? acc_in[in] + acc_in2[in] : acc_in[in];
						}
				}
			}
#pragma unroll
			for(int u = 0; u < U; u++) {
				const int t = t0 + u * BT, e = t / LT, w = t % LT, line = blockIdx.x * LT + w;
				if(t < Nx * LT && line < Ny) {
					const int ee = e == Nx - 1 ? 0 : e;
					const cx<R>* bw = bufs + (size_t)w * KS * PITCH + (ee / M) * part_pitch(M) + ee % M;
#pragma unroll
					for(int j = 0; j < KS; j++) {
						const size_t out = (size_t)(s0 + j) * 2 * N + (size_t)(1 - c) * N + (size_t)e * Ny + line;
						const cx<R> x = bw[j * PITCH];
						if(dst) dst[out] = x;
						if(acc) acc_out[out] = a[u][j] + x;
					}
				}
			}
		}
	}
}

// y-line solve in the x-line form: one warp per (column, comp, KS slots of one wavelength), lane l
// owning the rows [l*M, l*M+M) of the column, the chunk maps combined by warp shuffles
// (line_combine) as in k_solve_xc, so that no barrier joins the warps of a line. A block of LT
// warps takes LT adjacent columns: its threads form the right-hand sides of every (row, column)
// pair of those columns together (consecutive threads take the columns of a row, so a warp's
// loads are 32-byte row segments of eight rows) into the warps' shared buffers in the lane-chunk
// layout, each warp solves its column, and the block writes the results back row by row. The
// factor planes keep the plain [row][column] layout (each 32-byte sector of a row serves the LT
// warps of the block). KIND: ST_EXPL_X (explicit x half-step) or ST_WOOD_Y (Woodbury term).
// Restates BlockSparseMatrixDY::shifted_block_vmult_inv (BlockSparseMatrix.cpp:386-451) with the
// right-hand sides of ParaxialPrimaryEvolutionOperator::apply (ParaxialPrimaryEvolutionOperator.
// cpp:153-209). Outputs: dst = x (may be null), acc_out = (acc_in [+ acc_in2]) + x (may be null).
template <typename R, int M, int KIND, int KS>
__global__ void __launch_bounds__(128, NBPM_XC_MINB(M * KS)) k_solve_yt(Geom G, int nch, const cx<R>* __restrict__ coef,
		const cx<R>* __restrict__ fac, size_t plane, const cx<double>* __restrict__ lsc,
		const cx<R>* __restrict__ src, cx<R>* __restrict__ dst, const cx<R>* acc_in, cx<R>* acc_out,
		const cx<R>* acc_in2) {
	extern __shared__ unsigned char smem_raw[];
	const int LT = blockDim.x / 32;
	const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
	const int Nx = G.Nx, Ny = G.Ny, N = G.N;
	const int x0 = blockIdx.x * LT;
	const int c = blockIdx.y % 2, bc = blockIdx.y / 2;
	const int g = bc / nch, ch = bc % nch;
	const int s0 = g * G.spg + ch * KS;
	const int n_unk = Ny - 1;
	const int PITCH = 32 * (M + 1);
	cx<R>* const bufs = reinterpret_cast<cx<R>*>(smem_raw);
	const Stencil<R> st{coef + (size_t)g * coef_set_size(N), N, Nx, Ny};
	const cx<R>* f0 = src + (size_t)s0 * 2 * N;
	const cx<R> one = mk<R>(1, 0), zero = mk<R>(0, 0);
	// right-hand sides of every (row, column) pair of the block's columns
	for(int e = threadIdx.x; e < n_unk * LT; e += blockDim.x) {
		const int i = e / LT, w = e % LT, x = x0 + w;
		if(x < Nx) {
			cx<R> r[KS];
			composite_m<R, KIND, KS>(st, c, x, i, f0, r);
			cx<R>* b = bufs + (size_t)w * KS * PITCH + (i / M) * (M + 1) + i % M;
#pragma unroll
			for(int j = 0; j < KS; j++) b[j * PITCH] = r[j];
		}
	}
	__syncthreads();
	const int x = x0 + warp;
	if(x < Nx) {
		cx<R>* buf = bufs + (size_t)warp * KS * PITCH;
		const cx<R>* Fc = fac + ((size_t)g * 2 + c) * NFAC * plane + x;
		const cx<double>* ls = lsc + (((size_t)g * 2 + c) * Nx + x) * 2;
		const cx<double> r0 = ls[0], rden = ls[1];
		const int i0 = lane * M;
		cx<R> d0[KS], S0[KS], G0[KS];
		cx<R> P = one, S1 = zero, G1 = zero, Cp = one;
#pragma unroll
		for(int j = 0; j < KS; j++) { d0[j] = zero; S0[j] = zero; G0[j] = zero; }
		cx<R>* vb = buf + lane * (M + 1);
#pragma unroll
		for(int k = 0; k < M; k++) {
			if(i0 + k < n_unk) {
				const size_t q = (size_t)(i0 + k) * Nx;
				const cx<R> a = Fc[F_A * plane + q], rb = Fc[F_RB * plane + q];
				const cx<R> w = Fc[F_W * plane + q], cc = Fc[F_C * plane + q];
				P = a * P;
				S1 = cfma(w, P, S1);
				G1 = cfma(Cp, P, G1);
#pragma unroll
				for(int j = 0; j < KS; j++) {
					const cx<R> b = vb[j * PITCH + k] * rb;
					vb[j * PITCH + k] = b;
					d0[j] = cfma(a, d0[j], b);
					S0[j] = cfma(w, d0[j], S0[j]);
					G0[j] = cfma(Cp, d0[j], G0[j]);
				}
				Cp = Cp * cc;
			}
		}
		cx<R> din[KS], xin[KS], fr[KS];
		line_combine<R, KS>(P, d0, S0, S1, G0, G1, Cp, r0, rden, lane, din, xin, fr);
#pragma unroll
		for(int k = 0; k < M; k++) {
			if(i0 + k < n_unk) {
				const cx<R> a = Fc[F_A * plane + (size_t)(i0 + k) * Nx];
#pragma unroll
				for(int j = 0; j < KS; j++) { din[j] = cfma(a, din[j], vb[j * PITCH + k]); vb[j * PITCH + k] = din[j]; }
			}
		}
#pragma unroll
		for(int k = M - 1; k >= 0; k--) {
			if(i0 + k < n_unk) {
				const size_t q = (size_t)(i0 + k) * Nx;
				const cx<R> cc = Fc[F_C * plane + q], cr = Fc[F_COR * plane + q];
#pragma unroll
				for(int j = 0; j < KS; j++) {
					xin[j] = cfma(cc, xin[j], vb[j * PITCH + k]);
					vb[j * PITCH + k] = cfnma(fr[j], cr, xin[j]);
				}
			}
		}
	}
	__syncthreads();
	// results, row by row (row Ny-1 repeats row 0)
	for(int e = threadIdx.x; e < Ny * LT; e += blockDim.x) {
		const int i = e / LT, w = e % LT, xo = x0 + w;
		if(xo >= Nx) continue;
		const int ii = i == Ny - 1 ? 0 : i;
		const cx<R>* b = bufs + (size_t)w * KS * PITCH + (ii / M) * (M + 1) + ii % M;
#pragma unroll
		for(int j = 0; j < KS; j++) {
			const size_t off = (size_t)(s0 + j) * 2 * N + (size_t)c * N + (size_t)i * Nx + xo;
			const cx<R> v = b[j * PITCH];
			if(dst) dst[off] = v;
			if(KIND != ST_EXPL_X && acc_out) acc_out[off] = (acc_in2 ? acc_in[off] + acc_in2[off] : acc_in[off]) + v;
		}
	}
}

// Whether k_solve_yc<M, KS, MAXT> keeps its chunk values in shared memory: the values
// (KS*M*MAXT complex) and the combine arrays ((4 + 3 KS)*MAXT + 32 KS complex) within 224 KiB.
__host__ __device__ constexpr bool yc_values_in_smem(int M, int KS, int MAXT, int csize) {
	return ((long)KS * M * MAXT + (4L + 3L * KS) * MAXT + 32L * KS) * csize <= 224L * 1024;
}

// Combine of the y-chunk maps of a block (32 columns x WY chunks; shared arrays at
// [chunk][column], per-slot arrays at [slot][chunk][column]): warp w combines columns
// w, w + WY, ... with its lanes indexing the chunks (line_combine), and leaves per chunk the
// forward and backward entering values in sD0 / sG0 and per column the Sherman-Morrison
// factor in sF.
template <typename R, int KS>
__device__ __forceinline__ void ycol_combine(const cx<R>* sP, const cx<R>* sS1, const cx<R>* sG1, const cx<R>* sCp,
		cx<R>* sD0, const cx<R>* sS0, cx<R>* sG0, cx<R>* sF, int WY, int w, int lane, int ix0, int Nx,
		const cx<double>* ls) {
	const int SZ = WY * 32;
	const cx<R> one = mk<R>(1, 0), zero = mk<R>(0, 0);
	for(int col = w; col < 32; col += WY) {
		if(ix0 + col >= Nx) continue;  // uniform across the warp
		const bool ok = lane < WY;
		const int e = lane * 32 + col;
		const cx<R> P = ok ? sP[e] : one, S1 = ok ? sS1[e] : zero, G1 = ok ? sG1[e] : zero, Cp = ok ? sCp[e] : one;
		cx<R> d0[KS], S0[KS], G0[KS], din[KS], xin[KS], fr[KS];
#pragma unroll
		for(int j = 0; j < KS; j++) {
			d0[j] = ok ? sD0[j * SZ + e] : zero;
			S0[j] = ok ? sS0[j * SZ + e] : zero;
			G0[j] = ok ? sG0[j * SZ + e] : zero;
		}
		const cx<double> r0 = ls[(size_t)(ix0 + col) * 2], rden = ls[(size_t)(ix0 + col) * 2 + 1];
		line_combine<R, KS>(P, d0, S0, S1, G0, G1, Cp, r0, rden, lane, din, xin, fr);
		if(ok) {
#pragma unroll
			for(int j = 0; j < KS; j++) { sD0[j * SZ + e] = din[j]; sG0[j * SZ + e] = xin[j]; }
		}
		if(lane == 0) {
#pragma unroll
			for(int j = 0; j < KS; j++) sF[j * 32 + col] = fr[j];
		}
	}
}

// y-line solve fused with its right-hand side (KIND: explicit x half-step or y Woodbury term),
// chunked parallel form: block = 32 adjacent columns (lanes, coalesced) x WY warps for KS
// slots of one wavelength; warp w owns the rows [w*M, w*M+M) of the 32 lines for all KS
// slots. One pass builds the chunk maps, one combine (ycol_combine) joins them across the
// warps, one pass finishes the lines. MAXT: block size the instance is compiled for (512, or
// 1024 for 32 warps of short chunks).
template <typename R, int M, int KIND, int KS, int MAXT = 512>
__global__ void __launch_bounds__(MAXT, NBPM_YC_MINB) k_solve_yc(Geom G, int slot0, int nch, const cx<R>* __restrict__ coef,
		const cx<R>* __restrict__ fac, size_t plane, const cx<double>* __restrict__ lsc,
		const cx<R>* __restrict__ src, cx<R>* __restrict__ dst, const cx<R>* acc_in, cx<R>* acc_out,
		const cx<R>* acc_in2) {
	extern __shared__ unsigned char smem_raw[];
	const int WY = blockDim.y;
	const int lane = threadIdx.x, w = threadIdx.y;
	const int Nx = G.Nx, Ny = G.Ny, N = G.N;
	const int ix = blockIdx.x * 32 + lane;
	const bool col = ix < Nx;
	const int c = blockIdx.y % 2, bc = blockIdx.y / 2;
	const int g = bc / nch, ch = bc % nch;
	const int s0 = g * G.spg + ch * KS;
	const int n_unk = Ny - 1;
	const int SZ = WY * 32;
	cx<R>* sP = reinterpret_cast<cx<R>*>(smem_raw);  // [WY][32] each
	cx<R>* sS1 = sP + SZ;
	cx<R>* sG1 = sS1 + SZ;
	cx<R>* sCp = sG1 + SZ;
	cx<R>* sD0 = sCp + SZ;                            // [KS][WY][32] each
	cx<R>* sS0 = sD0 + KS * SZ;
	cx<R>* sG0 = sS0 + KS * SZ;
	cx<R>* sF = sG0 + KS * SZ;                        // [KS][32]
	// chunk values in shared memory ([KS][M][WY][32]) when they fit beside the combine arrays,
	// else in registers
	constexpr bool VS = yc_values_in_smem(M, KS, MAXT, (int)sizeof(cx<R>));
	cx<R>* sV = sF + KS * 32;
	const cx<R>* Fc = fac + ((size_t)g * 2 + c) * NFAC * plane;
	const int i0 = w * M;
	const cx<R> one = mk<R>(1, 0), zero = mk<R>(0, 0);
	const Stencil<R> st{coef + (size_t)g * coef_set_size(N), N, Nx, Ny};
	const cx<R>* f0 = src + (size_t)s0 * 2 * N;
	// chunk pass: right-hand sides b (kept in v) and the chunk maps of line_combine
	cx<R> v[VS ? 1 : KS][VS ? 1 : M];
	auto V = [&](int j, int k) -> cx<R>& { return VS ? sV[((j * M + k) * WY + w) * 32 + lane] : v[VS ? 0 : j][VS ? 0 : k]; };
	cx<R> d0[KS], S0[KS], G0[KS];
	cx<R> P = one, S1 = zero, G1 = zero, Cp = one;
#pragma unroll
	for(int j = 0; j < KS; j++) { d0[j] = zero; S0[j] = zero; G0[j] = zero; }
	// chunk values in shared memory need no compile-time row index: unroll by 2 in the 16-warp
	// blocks (measured faster on GB300), fully in the 32-warp ones
	constexpr int U1 = (VS && MAXT <= 512 && M >= 2) ? 2 : M;
#pragma unroll U1
	for(int k = 0; k < M; k++) {
		const int i = i0 + k;
#pragma unroll
		for(int j = 0; j < KS; j++) V(j, k) = zero;
		if(col && i < n_unk) {
			const size_t q = (size_t)ix + (size_t)Nx * i;
			const cx<R> a = Fc[F_A * plane + q], rb = Fc[F_RB * plane + q];
			const cx<R> wv = Fc[F_W * plane + q], cc = Fc[F_C * plane + q];
			cx<R> r[KS];
			composite_m<R, KIND, KS>(st, c, ix, i, f0, r);
			P = a * P;
			S1 = cfma(wv, P, S1);
			G1 = cfma(Cp, P, G1);
#pragma unroll
			for(int j = 0; j < KS; j++) {
				const cx<R> b = r[j] * rb;
				V(j, k) = b;
				d0[j] = cfma(a, d0[j], b);
				S0[j] = cfma(wv, d0[j], S0[j]);
				G0[j] = cfma(Cp, d0[j], G0[j]);
			}
			Cp = Cp * cc;
		}
	}
	{
		const int e = w * 32 + lane;
		sP[e] = P; sS1[e] = S1; sG1[e] = G1; sCp[e] = Cp;
#pragma unroll
		for(int j = 0; j < KS; j++) { sD0[j * SZ + e] = d0[j]; sS0[j * SZ + e] = S0[j]; sG0[j * SZ + e] = G0[j]; }
	}
	__syncthreads();
	ycol_combine<R, KS>(sP, sS1, sG1, sCp, sD0, sS0, sG0, sF, WY, w, lane, blockIdx.x * 32, Nx,
		lsc + ((size_t)g * 2 + c) * Nx * 2);
	__syncthreads();
	if(!col) return;
	cx<R> d[KS], x[KS], fr[KS];
#pragma unroll
	for(int j = 0; j < KS; j++) {
		d[j] = sD0[j * SZ + w * 32 + lane];
		x[j] = sG0[j * SZ + w * 32 + lane];
		fr[j] = sF[j * 32 + lane];
	}
#pragma unroll
	for(int k = 0; k < M; k++) {
		const int i = i0 + k;
		if(i < n_unk) {
			const cx<R> a = Fc[F_A * plane + (size_t)ix + (size_t)Nx * i];
#pragma unroll
			for(int j = 0; j < KS; j++) { d[j] = cfma(a, d[j], V(j, k)); V(j, k) = d[j]; }
		}
	}
#pragma unroll
	for(int k = M - 1; k >= 0; k--) {
		const int i = i0 + k;
		if(i < n_unk) {
			const size_t q = (size_t)ix + (size_t)Nx * i;
			const cx<R> cc = Fc[F_C * plane + q], cr = Fc[F_COR * plane + q];
#pragma unroll
			for(int j = 0; j < KS; j++) {
				x[j] = cfma(cc, x[j], V(j, k));
				const cx<R> y = cfnma(fr[j], cr, x[j]);
				const size_t off = (size_t)(s0 + j) * 2 * N + (size_t)c * N;
				if(dst) dst[off + q] = y;
				// the explicit-step solves never accumulate
				if(KIND != ST_EXPL_X && acc_out)
					acc_out[off + q] = (acc_in2 ? acc_in[off + q] + acc_in2[off + q] : acc_in[off + q]) + y;
				if(i == 0) {
					const size_t qe = (size_t)ix + (size_t)Nx * (Ny - 1);
					if(dst) dst[off + qe] = y;
					if(KIND != ST_EXPL_X && acc_out)
						acc_out[off + qe] = (acc_in2 ? acc_in[off + qe] + acc_in2[off + qe] : acc_in[off + qe]) + y;
				}
			}
		}
	}
}

// y-line solve fused with its right-hand side, sequential form: one thread per (column, KS
// slots of one wavelength), both field components. Consecutive threads take consecutive columns,
// so every load and store of a row is coalesced. The forward sweep
//   d_i = alpha_i d_{i-1} + b_i / beta_i,   S = sum_i w_i d_i
// stores d_i in scr (a field-sized buffer that none of the inputs alias: the output buffer
// itself when there is one), the Sherman-Morrison factor f = (S - r0 d_{n-1}) rden is formed in
// FP64, and the backward sweep x_i = d_i - gamma_i x_{i+1} turns d into the solution
// x_i - f corr_i in place. Every thread is independent: no barriers, no cross-chunk combine,
// and a tenth of the instructions per point of the chunked form (the stencil taps of the
// neighbouring columns come from L1). Restates BlockSparseMatrixDY::shifted_block_vmult_inv
// (BlockSparseMatrix.cpp:386-451) with the right-hand side of ParaxialPrimaryEvolutionOperator::
// apply (ParaxialPrimaryEvolutionOperator.cpp:153-209) for KIND = ST_EXPL_X (explicit x
// half-step) or ST_WOOD_Y (Woodbury term). Outputs: dst = x (may be null), acc_out =
// (acc_in [+ acc_in2]) + x (may be null); row Ny-1 receives row 0 (period Ny-1).
template <typename R, int KIND, int KS>
__global__ void __launch_bounds__(128) k_solve_yq(Geom G, int nch, const cx<R>* __restrict__ coef,
		const cx<R>* __restrict__ fac, size_t plane, const cx<double>* __restrict__ lsc,
		const cx<R>* __restrict__ src, cx<R>* scr, cx<R>* dst, const cx<R>* acc_in, cx<R>* acc_out,
		const cx<R>* acc_in2) {
	const int Nx = G.Nx, Ny = G.Ny, N = G.N;
	const int ix = blockIdx.x * blockDim.x + threadIdx.x;
	if(ix >= Nx) return;
	const int g = blockIdx.y / nch, ch = blockIdx.y % nch;
	const int s0 = g * G.spg + ch * KS;
	const int n = Ny - 1;
	const size_t ss = 2 * (size_t)N;
	const Stencil<R> st{coef + (size_t)g * coef_set_size(N), N, Nx, Ny};
	const cx<R>* f0 = src + (size_t)s0 * ss;
	const cx<R>* F0 = fac + ((size_t)g * 2 + 0) * NFAC * plane;
	const cx<R>* F1 = fac + ((size_t)g * 2 + 1) * NFAC * plane;
	cx<R>* sc = scr + (size_t)s0 * ss;
	const cx<R> zero = mk<R>(0, 0);
	cx<R> d0[KS], d1[KS], a0[KS], a1[KS];
#pragma unroll
	for(int j = 0; j < KS; j++) { d0[j] = zero; d1[j] = zero; a0[j] = zero; a1[j] = zero; }
#pragma unroll 2
	for(int i = 0; i < n; i++) {
		const size_t q = (size_t)ix + (size_t)Nx * i;
		cx<R> r0[KS], r1[KS];
		composite_m<R, KIND, KS>(st, 0, ix, i, f0, r0);
		composite_m<R, KIND, KS>(st, 1, ix, i, f0, r1);
		const cx<R> A0 = F0[F_A * plane + q], B0 = F0[F_RB * plane + q], W0 = F0[F_W * plane + q];
		const cx<R> A1 = F1[F_A * plane + q], B1 = F1[F_RB * plane + q], W1 = F1[F_W * plane + q];
#pragma unroll
		for(int j = 0; j < KS; j++) {
			const cx<R> b0 = r0[j] * B0, b1 = r1[j] * B1;
			d0[j] = cfma(A0, d0[j], b0);
			d1[j] = cfma(A1, d1[j], b1);
			a0[j] = cfma(W0, d0[j], a0[j]);
			a1[j] = cfma(W1, d1[j], a1[j]);
			sc[j * ss + q] = d0[j];
			sc[j * ss + N + q] = d1[j];
		}
	}
	const cx<double>* l0 = lsc + (((size_t)g * 2 + 0) * Nx + ix) * 2;
	const cx<double>* l1 = lsc + (((size_t)g * 2 + 1) * Nx + ix) * 2;
	const cx<double> r00 = l0[0], rd0 = l0[1], r01 = l1[0], rd1 = l1[1];
	cx<R> fr0[KS], fr1[KS], x0[KS], x1[KS];
#pragma unroll
	for(int j = 0; j < KS; j++) {
		fr0[j] = cvt<R>((cvt<double>(a0[j]) - r00 * cvt<double>(d0[j])) * rd0);
		fr1[j] = cvt<R>((cvt<double>(a1[j]) - r01 * cvt<double>(d1[j])) * rd1);
		x0[j] = zero;
		x1[j] = zero;
	}
	const size_t qe = (size_t)ix + (size_t)Nx * n;
#pragma unroll 2
	for(int i = n - 1; i >= 0; i--) {
		const size_t q = (size_t)ix + (size_t)Nx * i;
		const cx<R> C0 = F0[F_C * plane + q], K0 = F0[F_COR * plane + q];
		const cx<R> C1 = F1[F_C * plane + q], K1 = F1[F_COR * plane + q];
#pragma unroll
		for(int j = 0; j < KS; j++) {
			const size_t o0 = (size_t)(s0 + j) * ss + q, o1 = o0 + N;
			x0[j] = cfma(C0, x0[j], sc[j * ss + q]);
			x1[j] = cfma(C1, x1[j], sc[j * ss + N + q]);
			const cx<R> y0 = x0[j] - fr0[j] * K0, y1 = x1[j] - fr1[j] * K1;
			if(dst) { dst[o0] = y0; dst[o1] = y1; }
			if(KIND != ST_EXPL_X && acc_out) {
				acc_out[o0] = (acc_in2 ? acc_in[o0] + acc_in2[o0] : acc_in[o0]) + y0;
				acc_out[o1] = (acc_in2 ? acc_in[o1] + acc_in2[o1] : acc_in[o1]) + y1;
			}
			if(i == 0) {
				const size_t e0 = (size_t)(s0 + j) * ss + qe, e1 = e0 + N;
				if(dst) { dst[e0] = y0; dst[e1] = y1; }
				if(KIND != ST_EXPL_X && acc_out) {
					acc_out[e0] = (acc_in2 ? acc_in[e0] + acc_in2[e0] : acc_in[e0]) + y0;
					acc_out[e1] = (acc_in2 ? acc_in[e1] + acc_in2[e1] : acc_in[e1]) + y1;
				}
			}
		}
	}
}

// x-line solve for long lines: one block of W warps per line, 32*W chunks of M points (the
// partitioned layout with 32*W chunks), solved as in k_solve_xc; neighbouring chunks in different
// warps exchange their border unknowns through shared memory (2 + K barriers a line, 6 with part_ring).
// acc_in2 (may be null): a second accumulator input, acc_out = (acc_in + acc_in2) + x. TOUT: the
// results go out transposed with the components exchanged ((c, iy, e) -> (1 - c, e, iy) of an
// Ny x Nx plane), as in k_solve_xc.
template <typename R, int M, int KIND, int KS, bool TOUT = false>
__global__ void __launch_bounds__(256) k_solve_xw(Geom G, int slot0, int nch, const cx<R>* __restrict__ coef,
		const cx<R>* __restrict__ fac, size_t plane, const cx<double>* __restrict__ lsc,
		const cx<R>* __restrict__ src, cx<R>* __restrict__ dst, const cx<R>* acc_in, cx<R>* acc_out,
		const cx<R>* acc_in2) {
	extern __shared__ unsigned char smem_raw[];
	wait_predecessor();
	const int W = blockDim.x / 32;
	const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
	const int Nx = G.Nx, Ny = G.Ny, N = G.N;
	const int iy = blockIdx.x;
	const int c = blockIdx.y % 2, bc = blockIdx.y / 2;
	const int g = bc / nch, ch = bc % nch;
	const int s0 = g * G.spg + ch * KS;
	const int n_unk = Nx - 1;
	const int CH = 32 * W;
	const int ci = warp * 32 + lane;
	const int PITCH = CH * part_pitch(M);
	cx<R>* buf = reinterpret_cast<cx<R>*>(smem_raw);  // [KS][CH][M+1]
	cx<R>* sG = buf + KS * PITCH;                     // [2][KS][W]: g (first yf) of the warps' first chunks
	cx<R>* sH = sG + 2 * KS * W;                      // [2][KS][W + 1]: h of the warps' last chunks, then of the line's
	const cx<R>* Fc = fac + ((size_t)g * 2 + c) * NFAC * plane + (size_t)iy * part_line_size(M, CH);
	const cx<double> kb = lsc[(((size_t)g * 2 + c) * Ny + iy) * 2];
	const int K = (int)kb.x;
	const R base = (R)kb.y;
	const int last = (n_unk - 1) / M;  // last chunk
	const cx<R> zero = mk<R>(0, 0);
	const Stencil<R> st{coef + (size_t)g * coef_set_size(N), N, Nx, Ny};
	const cx<R>* f0 = src + (size_t)s0 * 2 * N;
#pragma unroll 1
	for(int t = 0; t < M; t++) {
		const int e = threadIdx.x + CH * t;
		cx<R> r[KS];
		if(e < n_unk) composite_m<R, KIND, KS>(st, c, e, iy, f0, r);
		else {
#pragma unroll
			for(int j = 0; j < KS; j++) r[j] = zero;
		}
#pragma unroll
		for(int j = 0; j < KS; j++) buf[j * PITCH + (e / M) * part_pitch(M) + e % M] = r[j];
	}
	__syncthreads();
	{
		// forward sweep of the thread's chunk and its first unknown with nothing outside the chunk
		cx<R> d[KS], yf[KS];
		cx<R>* vb = buf + ci * part_pitch(M);
#pragma unroll
		for(int j = 0; j < KS; j++) d[j] = yf[j] = zero;
#pragma unroll
		for(int k = 0; k < M; k++) {
			const v4<R> az = part_az(Fc, k, CH, ci);
			const cx<R> z = mk(az.z, az.w);
			if(k == 0) {
#pragma unroll
				for(int j = 0; j < KS; j++) { d[j] = vb[j * PITCH]; yf[j] = z * d[j]; }
			}
			else {
				const cx<R> a = mk(az.x, az.y);
#pragma unroll
				for(int j = 0; j < KS; j++) {
					d[j] = cfma(a, d[j], vb[j * PITCH + k]);
					vb[j * PITCH + k] = d[j];
					yf[j] = cfma(z, d[j], yf[j]);
				}
			}
		}
		// interface unknowns as in k_solve_xc; neighbours in other warps through shared memory
		const cx<R>* If = Fc + (size_t)M * NFAC * CH + ci;
		const bool edge_r = lane == 31 || ci == last;   // the next chunk is in another warp (or the first)
		const int wr = ci == last ? 0 : (warp + 1) % W;
		auto next = [&](cx<R> v, const cx<R>* s, int j) {
			const cx<R> n = shfl_down_c(v, 1);
			return edge_r ? s[j * W + wr] : n;
		};
		if(lane == 0) {
#pragma unroll
			for(int j = 0; j < KS; j++) sG[j * W + warp] = yf[j];
		}
		__syncthreads();
		cx<R> h[KS], x[KS], hl[KS];
		{
			const cx<R> hd = If[I_HD * CH], hy = If[I_HY * CH], gd = If[I_GD * CH], gy = If[I_GY * CH];
#pragma unroll
			for(int j = 0; j < KS; j++) {
				const cx<R> yn = next(yf[j], sG, j);
				h[j] = cfma(hy, yn, hd * d[j]);
				x[j] = cfma(gy, yn, gd * d[j]);
			}
		}
		cx<R> bh[KS], bg[KS];
#pragma unroll
		for(int j = 0; j < KS; j++) { bh[j] = h[j]; bg[j] = x[j]; }
		if(K < 0) {
			Border<cx<R>, KS> b;
#pragma unroll
			for(int j = 0; j < KS; j++) { b.h[j] = h[j]; b.x[j] = x[j]; }
			b = part_ring<true, KS, R>(LineThreads{W, 0, warp, lane, ci, last}, If, CH, b, sG);
#pragma unroll
			for(int j = 0; j < KS; j++) { hl[j] = b.h[j]; x[j] = b.x[j]; }
		}
		else
#pragma unroll 1
		for(int it = 0;; it++) {
			// two buffers in turn: the one written here was last read two barriers ago
			cx<R>* H = sH + (it & 1) * KS * (W + 1);
			cx<R>* Gn = sG + ((it + 1) & 1) * KS * W;
#pragma unroll
			for(int j = 0; j < KS; j++) {
				if(lane == 31) H[j * (W + 1) + warp] = h[j];
				if(ci == last) H[j * (W + 1) + W] = h[j];
			}
			if(lane == 0) {
#pragma unroll
				for(int j = 0; j < KS; j++) Gn[j * W + warp] = x[j];
			}
			__syncthreads();
#pragma unroll
			for(int j = 0; j < KS; j++) {
				const cx<R> up = shfl_up_c(h[j], 1);
				hl[j] = lane > 0 ? up : H[j * (W + 1) + (warp > 0 ? warp - 1 : W)];
			}
			if(it >= K) break;
			const cx<R> ph = If[I_PH * CH], pg = If[I_PG * CH], qh = If[I_QH * CH], qg = If[I_QG * CH];
#pragma unroll
			for(int j = 0; j < KS; j++) {
				const cx<R> gr = next(x[j], Gn, j);
				h[j] = cfma(qh, gr, cfma(ph, hl[j], bh[j]));
				x[j] = cfma(qg, gr, cfma(pg, hl[j], bg[j]));
			}
		}
		// backward sweep from the next chunk's first unknown, with the previous chunk's last one
		with_base(base, [&](auto one) {
#pragma unroll
			for(int k = M - 1; k >= 0; k--) {
				const v4<R> rc = part_rc(Fc, k, CH, ci);
				const cx<R> db = mk(rc.x, rc.y), cc = mk(rc.z, rc.w), ee = part_e(Fc, k, CH, ci);
#pragma unroll
				for(int j = 0; j < KS; j++) {
					x[j] = cfma(cc, x[j], cfma(ee, hl[j], from_base<decltype(one)::on>(db, base, vb[j * PITCH + k])));
					vb[j * PITCH + k] = x[j];
				}
			}
		});
	}
	__syncthreads();
	// write-out: the accumulator inputs of several points are loaded before any store
	constexpr int U = 4;
	for(int e0 = threadIdx.x; e0 < Nx; e0 += U * blockDim.x) {
		cx<R> a[U][KS];
		if(acc_out) {
#pragma unroll
			for(int u = 0; u < U; u++) {
				const int e = e0 + u * blockDim.x;
				if(e < Nx)
#pragma unroll
					for(int j = 0; j < KS; j++) {
						const size_t o = (size_t)(s0 + j) * 2 * N + (size_t)c * N + (size_t)iy * Nx + e;
						a[u][j] = acc_in2 ? acc_in[o] + acc_in2[o] : acc_in[o];
					}
			}
		}
#pragma unroll
		for(int u = 0; u < U; u++) {
			const int e = e0 + u * blockDim.x;
			if(e < Nx) {
				const int ee = e == Nx - 1 ? 0 : e;
#pragma unroll
				for(int j = 0; j < KS; j++) {
					const cx<R> x = buf[j * PITCH + (ee / M) * part_pitch(M) + ee % M];
					const size_t o = TOUT ? (size_t)(s0 + j) * 2 * N + (size_t)(1 - c) * N + iy + (size_t)e * Ny
						: (size_t)(s0 + j) * 2 * N + (size_t)c * N + (size_t)iy * Nx + e;
					if(dst) dst[o] = x;
					if(acc_out) acc_out[o] = a[u][j] + x;
				}
			}
		}
	}
}

// x-line solve with the chunk values in the warp's shared-memory buffer instead of registers
// (same algorithm and layout as k_solve_xc): for long lines (large M) the per-thread state
// stays small, so more warps stay resident.
template <typename R, int KIND, int KS>
__global__ void __launch_bounds__(128) k_solve_xs(Geom G, int slot0, int nch, int M, const cx<R>* __restrict__ coef,
		const cx<R>* __restrict__ fac, size_t plane, const cx<double>* __restrict__ lsc,
		const cx<R>* __restrict__ src, cx<R>* __restrict__ dst, const cx<R>* acc_in, cx<R>* acc_out) {
	extern __shared__ unsigned char smem_raw[];
	const int LT = blockDim.x / 32;
	const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
	const int Nx = G.Nx, Ny = G.Ny, N = G.N;
	const int iy = blockIdx.x * LT + warp;
	if(iy >= Ny) return;
	const int c = blockIdx.y % 2, bc = blockIdx.y / 2;
	const int g = bc / nch, ch = bc % nch;
	const int s0 = g * G.spg + ch * KS;
	const int n_unk = Nx - 1;
	const int PITCH = 32 * (M + 1);
	cx<R>* buf = reinterpret_cast<cx<R>*>(smem_raw) + (size_t)warp * KS * PITCH;
	const cx<R>* Fc = fac + ((size_t)g * 2 + c) * NFAC * plane + (size_t)iy * 32 * M * NFAC;
	const cx<double>* ls = lsc + (((size_t)g * 2 + c) * Ny + iy) * 2;
	const cx<double> r0 = ls[0], rden = ls[1];
	const int i0 = lane * M;
	const int last = n_unk - 1, lane_last = last / M, k_last = last % M;
	const cx<R> one = mk<R>(1, 0), zero = mk<R>(0, 0);
	const Stencil<R> st{coef + (size_t)g * coef_set_size(N), N, Nx, Ny};
	const cx<R>* f0 = src + (size_t)s0 * 2 * N;
	for(int e = lane; e < n_unk; e += 32) {
		cx<R> r[KS];
		composite_m<R, KIND, KS>(st, c, e, iy, f0, r);
#pragma unroll
		for(int j = 0; j < KS; j++) buf[j * PITCH + (e / M) * (M + 1) + e % M] = r[j];
	}
	__syncwarp();
	auto V = [&](int j, int k) -> cx<R>& { return buf[j * PITCH + lane * (M + 1) + k]; };
	cx<R> A[KS], B[KS];
#pragma unroll
	for(int j = 0; j < KS; j++) { A[j] = one; B[j] = zero; }
	for(int k = 0; k < M; k++) {
		if(i0 + k < n_unk) {
			cx<R> a = Fc[(k * NFAC + F_A) * 32 + lane], rb = Fc[(k * NFAC + F_RB) * 32 + lane];
#pragma unroll
			for(int j = 0; j < KS; j++) {
				cx<R> b = V(j, k) * rb;
				V(j, k) = b;
				B[j] = cfma(a, B[j], b);
				A[j] = a * A[j];
			}
		}
	}
#pragma unroll
	for(int o = 1; o < 32; o <<= 1) {
#pragma unroll
		for(int j = 0; j < KS; j++) {
			cx<R> Ap = shfl_up_c(A[j], o), Bp = shfl_up_c(B[j], o);
			if(lane >= o) { B[j] = A[j] * Bp + B[j]; A[j] = A[j] * Ap; }
		}
	}
	cx<R> d[KS], acc[KS], dl[KS];
#pragma unroll
	for(int j = 0; j < KS; j++) {
		d[j] = shfl_up_c(B[j], 1);
		if(lane == 0) d[j] = zero;
		acc[j] = zero;
		dl[j] = zero;
	}
	for(int k = 0; k < M; k++) {
		if(i0 + k < n_unk) {
			cx<R> a = Fc[(k * NFAC + F_A) * 32 + lane], w = Fc[(k * NFAC + F_W) * 32 + lane];
#pragma unroll
			for(int j = 0; j < KS; j++) {
				d[j] = cfma(a, d[j], V(j, k));
				V(j, k) = d[j];
				acc[j] = cfma(w, d[j], acc[j]);
			}
		}
		if(k == k_last) {
#pragma unroll
			for(int j = 0; j < KS; j++) dl[j] = d[j];
		}
	}
	cx<R> fr[KS];
#pragma unroll
	for(int j = 0; j < KS; j++) {
#pragma unroll
		for(int o = 16; o > 0; o >>= 1) acc[j] += shfl_xor_c(acc[j], o);
		dl[j] = shfl_idx_c(dl[j], lane_last);
		fr[j] = cvt<R>((cvt<double>(acc[j]) - r0 * cvt<double>(dl[j])) * rden);
		A[j] = one;
		B[j] = zero;
	}
	for(int k = M - 1; k >= 0; k--) {
		if(i0 + k < n_unk) {
			cx<R> cc = Fc[(k * NFAC + F_C) * 32 + lane];
#pragma unroll
			for(int j = 0; j < KS; j++) { B[j] = cfma(cc, B[j], V(j, k)); A[j] = cc * A[j]; }
		}
	}
#pragma unroll
	for(int o = 1; o < 32; o <<= 1) {
#pragma unroll
		for(int j = 0; j < KS; j++) {
			cx<R> An = shfl_down_c(A[j], o), Bn = shfl_down_c(B[j], o);
			if(lane + o < 32) { B[j] = A[j] * Bn + B[j]; A[j] = A[j] * An; }
		}
	}
#pragma unroll
	for(int j = 0; j < KS; j++) {
		d[j] = shfl_down_c(B[j], 1);
		if(lane == 31) d[j] = zero;
	}
	for(int k = M - 1; k >= 0; k--) {
		if(i0 + k < n_unk) {
			cx<R> cc = Fc[(k * NFAC + F_C) * 32 + lane], cr = Fc[(k * NFAC + F_COR) * 32 + lane];
#pragma unroll
			for(int j = 0; j < KS; j++) {
				d[j] = cfma(cc, d[j], V(j, k));
				V(j, k) = cfnma(fr[j], cr, d[j]);
			}
		}
	}
	__syncwarp();
	for(int j = 0; j < KS; j++) {
		const size_t off = (size_t)(s0 + j) * 2 * N + (size_t)c * N + (size_t)iy * Nx;
		for(int e = lane; e < Nx; e += 32) {
			int ee = e == Nx - 1 ? 0 : e;
			cx<R> x = buf[j * PITCH + (ee / M) * (M + 1) + ee % M];
			if(dst) dst[off + e] = x;
			if(acc_out) acc_out[off + e] = acc_in[off + e] + x;
		}
	}
}

// y-line solve for any Ny (same algorithm as k_solve_yc): block = 32 columns x W warps,
// warp w owns rows [w*M, w*M+M) with M = ceil((Ny-1)/W); the chunk values are kept in the
// scratch array vbuf (field layout, L2-resident while the block runs) instead of registers,
// so neither Ny nor the chunk length is bounded by the register file.
template <typename R, int KIND, int KS>
__global__ void __launch_bounds__(256) k_solve_ys(Geom G, int slot0, int nch, const cx<R>* __restrict__ coef,
		const cx<R>* __restrict__ fac, size_t plane, const cx<double>* __restrict__ lsc,
		const cx<R>* __restrict__ src, cx<R>* __restrict__ dst, const cx<R>* acc_in, cx<R>* acc_out,
		cx<R>* __restrict__ vbuf) {
	extern __shared__ unsigned char smem_raw[];
	const int WY = blockDim.y;
	const int lane = threadIdx.x, w = threadIdx.y;
	const int Nx = G.Nx, Ny = G.Ny, N = G.N;
	const int ix = blockIdx.x * 32 + lane;
	const bool col = ix < Nx;
	const int c = blockIdx.y % 2, bc = blockIdx.y / 2;
	const int g = bc / nch, ch = bc % nch;
	const int s0 = g * G.spg + ch * KS;
	const int n_unk = Ny - 1;
	const int M = (n_unk + WY - 1) / WY;
	const int i0 = w * M, i1 = min(i0 + M, n_unk);
	const int SZ = WY * 32;
	cx<R>* sA = reinterpret_cast<cx<R>*>(smem_raw);  // [KS][WY][32]
	cx<R>* sB = sA + KS * SZ;
	cx<R>* sD = sB + KS * SZ;
	cx<R>* sP = sD + KS * SZ;
	cx<R>* sL = sP + KS * SZ;                         // [KS][32]
	cx<R>* sF = sL + KS * 32;                         // [KS][32]
	const cx<R>* Fc = fac + ((size_t)g * 2 + c) * NFAC * plane;
	const cx<R> one = mk<R>(1, 0), zero = mk<R>(0, 0);
	cx<double> r0 = mk(0.0, 0.0), rden = mk(0.0, 0.0);
	if(col) {
		const cx<double>* ls = lsc + (((size_t)g * 2 + c) * Nx + ix) * 2;
		r0 = ls[0];
		rden = ls[1];
	}
	const Stencil<R> st{coef + (size_t)g * coef_set_size(N), N, Nx, Ny};
	const cx<R>* f0 = src + (size_t)s0 * 2 * N;
	auto va = [&](int j, int i) { return (size_t)(s0 + j) * 2 * N + (size_t)c * N + (size_t)ix + (size_t)Nx * i; };
	cx<R> A[KS], B[KS];
#pragma unroll
	for(int j = 0; j < KS; j++) { A[j] = one; B[j] = zero; }
	if(col) {
		for(int i = i0; i < i1; i++) {
			size_t q = (size_t)ix + (size_t)Nx * i;
			cx<R> a = Fc[F_A * plane + q], rb = Fc[F_RB * plane + q];
			cx<R> r[KS];
			composite_m<R, KIND, KS>(st, c, ix, i, f0, r);
#pragma unroll
			for(int j = 0; j < KS; j++) {
				cx<R> b = r[j] * rb;
				vbuf[va(j, i)] = b;
				B[j] = cfma(a, B[j], b);
				A[j] = a * A[j];
			}
		}
	}
#pragma unroll
	for(int j = 0; j < KS; j++) { sA[j * SZ + w * 32 + lane] = A[j]; sB[j * SZ + w * 32 + lane] = B[j]; }
	__syncthreads();
	if(w == 0) {
		for(int j = 0; j < KS; j++) {
			cx<R> D = zero;
			for(int ww = 0; ww < WY; ww++) {
				sD[j * SZ + ww * 32 + lane] = D;
				D = sA[j * SZ + ww * 32 + lane] * D + sB[j * SZ + ww * 32 + lane];
			}
		}
	}
	__syncthreads();
	cx<R> d[KS], acc[KS];
#pragma unroll
	for(int j = 0; j < KS; j++) { d[j] = sD[j * SZ + w * 32 + lane]; acc[j] = zero; }
	if(col) {
		for(int i = i0; i < i1; i++) {
			size_t q = (size_t)ix + (size_t)Nx * i;
			cx<R> a = Fc[F_A * plane + q], wv = Fc[F_W * plane + q];
#pragma unroll
			for(int j = 0; j < KS; j++) {
				d[j] = cfma(a, d[j], vbuf[va(j, i)]);
				vbuf[va(j, i)] = d[j];
				acc[j] = cfma(wv, d[j], acc[j]);
				if(i == n_unk - 1) sL[j * 32 + lane] = d[j];
			}
		}
	}
#pragma unroll
	for(int j = 0; j < KS; j++) sP[j * SZ + w * 32 + lane] = acc[j];
	__syncthreads();
	if(w == 0) {
		for(int j = 0; j < KS; j++) {
			cx<R> tot = zero;
			for(int ww = 0; ww < WY; ww++) tot += sP[j * SZ + ww * 32 + lane];
			sF[j * 32 + lane] = cvt<R>((cvt<double>(tot) - r0 * cvt<double>(sL[j * 32 + lane])) * rden);
		}
	}
#pragma unroll
	for(int j = 0; j < KS; j++) { A[j] = one; B[j] = zero; }
	if(col) {
		for(int i = i1 - 1; i >= i0; i--) {
			cx<R> cc = Fc[F_C * plane + (size_t)ix + (size_t)Nx * i];
#pragma unroll
			for(int j = 0; j < KS; j++) { B[j] = cfma(cc, B[j], vbuf[va(j, i)]); A[j] = cc * A[j]; }
		}
	}
#pragma unroll
	for(int j = 0; j < KS; j++) { sA[j * SZ + w * 32 + lane] = A[j]; sB[j * SZ + w * 32 + lane] = B[j]; }
	__syncthreads();
	if(w == 0) {
		for(int j = 0; j < KS; j++) {
			cx<R> D = zero;
			for(int ww = WY - 1; ww >= 0; ww--) {
				sD[j * SZ + ww * 32 + lane] = D;
				D = sA[j * SZ + ww * 32 + lane] * D + sB[j * SZ + ww * 32 + lane];
			}
		}
	}
	__syncthreads();
	cx<R> fr[KS];
#pragma unroll
	for(int j = 0; j < KS; j++) { fr[j] = sF[j * 32 + lane]; d[j] = sD[j * SZ + w * 32 + lane]; }
	if(col) {
		for(int i = i1 - 1; i >= i0; i--) {
			size_t q = (size_t)ix + (size_t)Nx * i;
			cx<R> cc = Fc[F_C * plane + q], cr = Fc[F_COR * plane + q];
#pragma unroll
			for(int j = 0; j < KS; j++) {
				d[j] = cfma(cc, d[j], vbuf[va(j, i)]);
				cx<R> x = cfnma(fr[j], cr, d[j]);
				size_t off = (size_t)(s0 + j) * 2 * N + (size_t)c * N;
				if(dst) dst[off + q] = x;
				if(acc_out) acc_out[off + q] = acc_in[off + q] + x;
				if(i == 0) {
					size_t qe = (size_t)ix + (size_t)Nx * (Ny - 1);
					if(dst) dst[off + qe] = x;
					if(acc_out) acc_out[off + qe] = acc_in[off + qe] + x;
				}
			}
		}
	}
}

// Transverse translation for tilted incidence (SimpleShiftOperator.cpp:52-93): 4-tap cubic
// interpolation with period Nx-1 / Ny-1 (wrap rule SimpleShiftOperator.h:24-39).
__device__ __forceinline__ int ref_wrap(int i, int n) {
	if(i > n - 2) return i % (n - 1);
	if(i < 0) return i + (1 - i / (n - 1)) * (n - 1);
	return i;
}

template <typename R>
__device__ __forceinline__ void phase_apply(const cx<R>* C, size_t N, int p, cx<R>& a, cx<R>& b) {
	cx<R> oxx = coef_ph(C, 0, p), oyy = coef_ph(C, 1, p), oxy = coef_ph(C, 2, p);
	cx<R> u = cfma(oxy, b, oxx * a), v = cfma(oyy, b, oxy * a);
	a = u;
	b = v;
}

// x pass of the shift operator for every slot (q = 0 slots included: their weights are
// exactly 0/1/0/0 and the pass reduces to the duplicate-column copy), optionally preceded by
// the phase operator of coefficient set CA applied at each tap: T = X(phase_A(F)).
template <typename R>
__global__ void k_shift_x(Geom G, int slot0, const ShiftParams* __restrict__ sp, const cx<R>* __restrict__ CA,
		const cx<R>* __restrict__ F, cx<R>* __restrict__ T) {
	int p = blockIdx.x * blockDim.x + threadIdx.x;
	if(p >= G.N) return;
	int s = blockIdx.y;
	int gs = slot0 + s;
	int g = gs / G.spg - slot0 / G.spg;
	int gq = (gs / G.spg) * G.Nq + (gs / 2) % G.Nq;
	const ShiftParams P = sp[gq];
	const size_t N = G.N;
	const int Nx = G.Nx;
	int ix = p % Nx, iy = p / Nx;
	const cx<R>* f = F + (size_t)s * 2 * N;
	const cx<R>* Cg = CA ? CA + (size_t)g * coef_set_size(N) : nullptr;
	cx<R> v0, v1;
	if(Nx > 3) {
		v0 = mk<R>(0, 0);
		v1 = mk<R>(0, 0);
#pragma unroll
		for(int k = 0; k < 4; k++) {
			int q = ref_wrap(ix + P.msx - 1 + k, Nx) + Nx * iy;
			cx<R> a = f[q], b = f[N + q];
			if(Cg) phase_apply(Cg, N, q, a, b);
			v0 += (R)P.wx[k] * a;
			v1 += (R)P.wx[k] * b;
		}
	}
	else {
		v0 = f[p];
		v1 = f[N + p];
		if(Cg) phase_apply(Cg, N, p, v0, v1);
	}
	T[(size_t)s * 2 * N + p] = v0;
	T[(size_t)s * 2 * N + N + p] = v1;
}

// y pass and phase factor of the shift operator, optionally followed by the phase operator
// of coefficient set CB: F = phase_B(ph * Y(T)).
template <typename R>
__global__ void k_shift_y(Geom G, int slot0, const ShiftParams* __restrict__ sp, const cx<R>* __restrict__ CB,
		const cx<R>* __restrict__ T, cx<R>* __restrict__ F) {
	int p = blockIdx.x * blockDim.x + threadIdx.x;
	if(p >= G.N) return;
	int s = blockIdx.y;
	int gs = slot0 + s;
	int g = gs / G.spg - slot0 / G.spg;
	int gq = (gs / G.spg) * G.Nq + (gs / 2) % G.Nq;
	const ShiftParams P = sp[gq];
	const size_t N = G.N;
	const int Nx = G.Nx, Ny = G.Ny;
	int ix = p % Nx, iy = p / Nx;
	const cx<R>* t = T + (size_t)s * 2 * N;
	cx<R> ph = mk<R>((R)P.ph_re, (R)P.ph_im);
	cx<R> v0, v1;
	if(Ny > 3) {
		v0 = mk<R>(0, 0);
		v1 = mk<R>(0, 0);
#pragma unroll
		for(int k = 0; k < 4; k++) {
			int q = ix + Nx * ref_wrap(iy + P.msy - 1 + k, Ny);
			v0 += (R)P.wy[k] * t[q];
			v1 += (R)P.wy[k] * t[N + q];
		}
	}
	else {
		v0 = t[p];
		v1 = t[N + p];
	}
	v0 = v0 * ph;
	v1 = v1 * ph;
	if(CB) phase_apply(CB + (size_t)g * coef_set_size(N), N, p, v0, v1);
	F[(size_t)s * 2 * N + p] = v0;
	F[(size_t)s * 2 * N + N + p] = v1;
}

// Whole transition between two slabs in one pass (replaces shift_x(A), shift_y, shift_x,
// shift_y(B)): F_out = phase_B(ph^n * Y^n X^n (phase_A(F))), n = nshift (1 or 2). X and Y are
// the circulant cubic shifts of SimpleShiftOperator (period Nx-1 / Ny-1; they act on rows and
// columns and commute, so Y X Y X = Y Y X X). For a tile of 32 x 32 outputs of one slot the
// block stages the input window (phase_A applied) in shared memory; each thread then filters
// 8 consecutive outputs of a window row in registers (the 8 + 3n inputs read once) into a second
// buffer, then 4 consecutive rows of an output column, and writes the tile. Indices wrap with
// i mod (N-1), which equals the reference's wrap rule for every index above -(N-1) (the composition
// of two wrapped passes then also reduces to one mod); a slot whose integer shift reaches -(N-2) or
// below takes the exact per-point path instead. The duplicate row and column of F are never read, as
// in the separate passes. Bound: the FP64 pipe; in FP32 instruction issue (59 % active).
constexpr int SHT = 32;  // tile edge

__device__ __forceinline__ int pmod(int i, int n) {
	int r = i % n;
	return r < 0 ? r + n : r;
}

template <typename R>
__device__ __forceinline__ void tap_in(const cx<R>* f, const cx<R>* Ca, size_t N, int q, cx<R>& a, cx<R>& b) {
	a = f[q];
	b = f[N + q];
	if(Ca) phase_apply(Ca, N, q, a, b);
}

// Exact composition with the reference's wrap rule, one output point (rarely used).
template <typename R>
__device__ void shift_point_exact(const Geom& G, const ShiftParams& P, const cx<R>* f, const cx<R>* Ca, int nsh,
		int ix, int iy, cx<R>& o0, cx<R>& o1) {
	const size_t N = G.N;
	const int Nx = G.Nx, Ny = G.Ny;
	const bool ax = Nx > 3, ay = Ny > 3;
	auto xrow = [&](int r, int x, cx<R>& a, cx<R>& b) {  // X^n of row r at column x
		if(!ax) { tap_in(f, Ca, N, x + Nx * r, a, b); return; }
		a = b = mk<R>(0, 0);
		for(int k1 = 0; k1 < 4; k1++) {
			int j = ref_wrap(x + P.msx - 1 + k1, Nx);
			cx<R> u0 = mk<R>(0, 0), u1 = mk<R>(0, 0);
			if(nsh == 2) {
				for(int k0 = 0; k0 < 4; k0++) {
					cx<R> t0, t1;
					tap_in(f, Ca, N, ref_wrap(j + P.msx - 1 + k0, Nx) + Nx * r, t0, t1);
					u0 += (R)P.wx[k0] * t0;
					u1 += (R)P.wx[k0] * t1;
				}
			}
			else tap_in(f, Ca, N, j + Nx * r, u0, u1);
			a += (R)P.wx[k1] * u0;
			b += (R)P.wx[k1] * u1;
		}
	};
	if(!ay) { xrow(iy, ix, o0, o1); return; }
	o0 = o1 = mk<R>(0, 0);
	for(int l1 = 0; l1 < 4; l1++) {
		int r1 = ref_wrap(iy + P.msy - 1 + l1, Ny);
		cx<R> u0 = mk<R>(0, 0), u1 = mk<R>(0, 0);
		if(nsh == 2) {
			for(int l0 = 0; l0 < 4; l0++) {
				cx<R> t0, t1;
				xrow(ref_wrap(r1 + P.msy - 1 + l0, Ny), ix, t0, t1);
				u0 += (R)P.wy[l0] * t0;
				u1 += (R)P.wy[l0] * t1;
			}
		}
		else xrow(r1, ix, u0, u1);
		o0 += (R)P.wy[l1] * u0;
		o1 += (R)P.wy[l1] * u1;
	}
}

// The window of a transition tile: the tile's points inside the plane and, along a filtered axis, 3 more per
// shift; phase_A is applied as it is loaded. Its points are dealt out to the 256 threads one after the other: a
// warp per row of 38 points took two rounds, the second with 6 lanes, and the loads of a point waited for those of
// the point before. Here the loads of U points are in flight together. 256x256: FP32 pairs, 16
// wavelengths, 13 q, 472 us as rows, 364 us so; FP64, 3 wavelengths, 13 q, 1082 and 957 us. The clipping to the plane
// spares a 97x75 mesh a third of its window points (FP64, 3 wavelengths, 7 q: 137 and 110 us).
template <typename R>
struct ShiftWindow {
	static constexpr int U = sizeof(R) == 4 ? 3 : 2, PA = SHT + 7;
	int wx, wy, magic;
	int* at;  // [2][SHT + 6]: the columns, and the first points of the rows
	// places: shared memory for 2 * (SHT + 6) numbers. By all threads of the block, with a barrier.
	__device__ __forceinline__ ShiftWindow(const Geom& G, const ShiftParams& P, int nsh, int x0, int y0, int* places) : at(places) {
		const bool ax = G.Nx > 3, ay = G.Ny > 3;
		wx = min(SHT, G.Nx - x0) + (ax ? 3 * nsh : 0);
		wy = min(SHT, G.Ny - y0) + (ay ? 3 * nsh : 0);
		magic = 65536 / wx + 1;  // e / wx = e * magic >> 16 for e < 38 * wx, wx <= 38
		const int u = threadIdx.x, v = threadIdx.x - 64;
		if(u < wx) at[u] = ax ? pmod(x0 + nsh * (P.msx - 1) + u, G.Nx - 1) : x0 + u;
		if(v >= 0 && v < wy) at[SHT + 6 + v] = G.Nx * (ay ? pmod(y0 + nsh * (P.msy - 1) + v, G.Ny - 1) : y0 + v);
		__syncthreads();
	}
	// f: component planes of a slot; A: [2][SHT + 6][PA]. All threads of the block; the caller's barrier follows.
	__device__ __forceinline__ void load(const cx<R>* f, const cx<R>* Ca, size_t N, cx<R>* A) const {
		if(Ca) points<true>(f, Ca, N, A);
		else points<false>(f, Ca, N, A);
	}
	template <bool PHASE>
	__device__ __forceinline__ void points(const cx<R>* f, const cx<R>* Ca, size_t N, cx<R>* A) const {
		const int cnt = wx * wy;
#pragma unroll 1
		for(int e0 = threadIdx.x; e0 < cnt; e0 += U * 256) {
			cx<R> a[U], b[U];
			int to[U];
#pragma unroll
			for(int j = 0; j < U; j++) {
				// past the end: the last point once more, the same value
				const int e = min(e0 + 256 * j, cnt - 1), v = e * magic >> 16, u = e - v * wx, q = at[u] + at[SHT + 6 + v];
				to[j] = v * PA + u;
				a[j] = f[q];
				b[j] = f[N + q];
				if(PHASE) phase_apply(Ca, N, q, a[j], b[j]);
			}
#pragma unroll
			for(int j = 0; j < U; j++) {
				A[to[j]] = a[j];
				A[(SHT + 6) * PA + to[j]] = b[j];
			}
		}
	}
};

template <typename R>
__global__ void __launch_bounds__(256) k_shift_fused(Geom G, int slot0, const ShiftParams* __restrict__ sp,
		const cx<R>* __restrict__ CA, const cx<R>* __restrict__ CB, int nsh, const cx<R>* __restrict__ F,
		cx<R>* __restrict__ Fo) {
	extern __shared__ unsigned char smem_raw[];
	const int s = blockIdx.z;
	const int gs = slot0 + s;
	const int g = gs / G.spg - slot0 / G.spg;
	const int gq = (gs / G.spg) * G.Nq + (gs / 2) % G.Nq;
	const ShiftParams& P = sp[gq];
	const ShiftW<R> W(P, nsh);
	const size_t N = G.N;
	const int Nx = G.Nx, Ny = G.Ny;
	const bool ax = Nx > 3, ay = Ny > 3;
	const int x0 = blockIdx.x * SHT, y0 = blockIdx.y * SHT;
	const int tid = threadIdx.x;
	const cx<R>* f = F + (size_t)s * 2 * N;
	cx<R>* fo = Fo + (size_t)s * 2 * N;
	const cx<R>* Ca = CA ? CA + (size_t)g * coef_set_size(N) : nullptr;
	const cx<R>* Cb = CB ? CB + (size_t)g * coef_set_size(N) : nullptr;
	const int Px = Nx - 1, Py = Ny - 1;
	cx<R> ph = W.ph;
	if(nsh == 2) ph = ph * ph;
	// every tap index of both passes stays above -(N-1): mod arithmetic equals the wrap rule
	const bool regular = (!ax || P.msx - 1 > -Px) && (!ay || P.msy - 1 > -Py);
	if(!regular) {
		for(int e = tid; e < SHT * SHT; e += blockDim.x) {
			int ix = x0 + e % SHT, iy = y0 + e / SHT;
			if(ix >= Nx || iy >= Ny) continue;
			cx<R> o0, o1;
			shift_point_exact(G, P, f, Ca, nsh, ix, iy, o0, o1);
			o0 = o0 * ph;
			o1 = o1 * ph;
			int p = ix + Nx * iy;
			if(Cb) phase_apply(Cb, N, p, o0, o1);
			fo[p] = o0;
			fo[N + p] = o1;
		}
		return;
	}
	// 1. input window, phase_A applied
	constexpr int PA = SHT + 7, PB = SHT + 1;  // odd pitches (8-byte words): no bank conflicts
	cx<R>* A = reinterpret_cast<cx<R>*>(smem_raw);  // [2][wy][PA]: the window
	cx<R>* B = A + 2 * (SHT + 6) * PA;             // [2][wy][PB]: the window after the x-passes
	__shared__ int places[2 * (SHT + 6)];
	const ShiftWindow<R> win(G, P, nsh, x0, y0, places);
	const int wy = win.wy, nseg = (min(SHT, Nx - x0) + 7) / 8;
	win.load(f, Ca, N, A);
	__syncthreads();
	// 2. the n x-passes of one component over 8 consecutive outputs of a window row per thread, in
	// registers (consecutive threads take consecutive rows)
	const cx<R>* Y = A;  // what the y-passes read, with its pitch
	int PY = PA;
	if(ax) {
		for(int t = tid; t < 2 * nseg * wy; t += blockDim.x) {
			const int v = t % wy, r = t / wy, c = r >= nseg, seg = r - c * nseg;
			// past the window shared memory is not initialised: FP64's one filter for both shifts (ShiftW) takes
			// seven values with zero weights among them, the 4-tap passes none that is not in the window
			const int nin = sizeof(R) == 8 ? min(8 + 3 * nsh, win.wx - seg * 8) : 8 + 3 * nsh;
			const cx<R>* in = A + c * (SHT + 6) * PA + v * PA + seg * 8;
			cx<R> w[14];
#pragma unroll
			for(int k = 0; k < 14; k++) w[k] = k < nin ? in[k] : mk<R>(0, 0);
			W.template filter<14>(W.wx, w);
			cx<R>* out = B + c * (SHT + 6) * PB + v * PB + seg * 8;
#pragma unroll
			for(int k = 0; k < 8; k++) out[k] = w[k];
		}
		__syncthreads();
		Y = B;
		PY = PB;
	}
	// 3. the n y-passes over 4 consecutive output rows of one column per thread (both components),
	// then the phase factor, phase_B and the store (consecutive threads take consecutive columns)
	for(int t = tid; t < SHT * (SHT / 4); t += blockDim.x) {
		const int u = t % SHT, seg = t / SHT;
		const int ix = x0 + u;
		if(ix >= Nx || y0 + seg * 4 >= Ny) continue;
		cx<R> o[2][4];
#pragma unroll
		for(int c = 0; c < 2; c++) {
			const cx<R>* in = Y + c * (SHT + 6) * PY + seg * 4 * PY + u;
			if(ay) {
				const int nin = sizeof(R) == 8 ? min(4 + 3 * nsh, wy - seg * 4) : 4 + 3 * nsh;
				cx<R> w[10];
#pragma unroll
				for(int k = 0; k < 10; k++) w[k] = k < nin ? in[k * PY] : mk<R>(0, 0);
				W.template filter<10>(W.wy, w);
#pragma unroll
				for(int k = 0; k < 4; k++) o[c][k] = w[k];
			}
			else {
#pragma unroll
				for(int k = 0; k < 4; k++) o[c][k] = in[k * PY];
			}
		}
		if(ix >= Nx) continue;
#pragma unroll
		for(int k = 0; k < 4; k++) {
			const int iy = y0 + seg * 4 + k;
			if(iy < Ny) {
				cx<R> o0 = o[0][k] * ph, o1 = o[1][k] * ph;
				const int p = ix + Nx * iy;
				if(Cb) phase_apply(Cb, N, p, o0, o1);
				fo[p] = o0;
				fo[N + p] = o1;
			}
		}
	}
}

// All slots at q = 0: phase_A, then the shift operator's duplicate-border copy (column 0 ->
// column Nx-1, then row 0 -> row Ny-1), then phase_B, in one in-place pass. The thread of a
// source point also writes the border points copied from it, so no thread reads a value
// another thread writes.
template <typename R>
__global__ void k_phase_sync(Geom G, int slot0, const cx<R>* __restrict__ CA, const cx<R>* __restrict__ CB,
		cx<R>* F) {
	int p = blockIdx.x * blockDim.x + threadIdx.x;
	if(p >= G.N) return;
	int s = blockIdx.y;
	int g = (slot0 + s) / G.spg - slot0 / G.spg;
	const size_t N = G.N;
	const int Nx = G.Nx, Ny = G.Ny;
	const bool ax = Nx > 3, ay = Ny > 3;
	int ix = p % Nx, iy = p / Nx;
	if((ax && ix == Nx - 1) || (ay && iy == Ny - 1)) return;
	cx<R>* f = F + (size_t)s * 2 * N;
	const cx<R>* Ca = CA ? CA + (size_t)g * coef_set_size(N) : nullptr;
	const cx<R>* Cb = CB ? CB + (size_t)g * coef_set_size(N) : nullptr;
	cx<R> u0 = f[p], u1 = f[N + p];
	if(Ca) phase_apply(Ca, N, p, u0, u1);
	auto put = [&](int d) {
		cx<R> a = u0, b = u1;
		if(Cb) phase_apply(Cb, N, d, a, b);
		f[d] = a;
		f[N + d] = b;
	};
	put(p);
	if(ax && ix == 0) put((Nx - 1) + Nx * iy);
	if(ay && iy == 0) put(ix + Nx * (Ny - 1));
	if(ax && ay && ix == 0 && iy == 0) put((Nx - 1) + Nx * (Ny - 1));
}

// k_shift_fused for the two slots of a (wavelength, q) (FP32): the same window passes, one slot after the
// other through the same shared memory, the results written as pairs (pair_kernels.cuh). The phase entries
// and the window's indices are the same for both. blockIdx.z: pair of the pass; pair0: the pass's first one.
static __global__ void __launch_bounds__(256, 4) k_shift_pair(Geom G, int pair0, const ShiftParams* __restrict__ sp,
		const cx<float>* __restrict__ CA, const cx<float>* __restrict__ CB, int nsh, const cx<float>* __restrict__ F,
		v4<float>* __restrict__ Fo) {
	typedef float R;
	extern __shared__ unsigned char smem_raw[];
	const int z = blockIdx.z, g = z / G.Nq;
	const ShiftParams& P = sp[pair0 + z];
	const ShiftW<R> W(P, nsh);
	const size_t N = G.N;
	const int Nx = G.Nx, Ny = G.Ny;
	const bool ax = Nx > 3, ay = Ny > 3;
	const int x0 = blockIdx.x * SHT, y0 = blockIdx.y * SHT;
	const int tid = threadIdx.x;
	const cx<R>* f = F + (size_t)z * 4 * N;
	v4<float>* fo = Fo + (size_t)z * 2 * N;
	const cx<R>* Ca = CA ? CA + (size_t)g * coef_set_size(N) : nullptr;
	const cx<R>* Cb = CB + (size_t)g * coef_set_size(N);
	const int Px = Nx - 1, Py = Ny - 1;
	cx<R> ph = W.ph;
	if(nsh == 2) ph = ph * ph;
	const bool regular = (!ax || P.msx - 1 > -Px) && (!ay || P.msy - 1 > -Py);  // see k_shift_fused
	if(!regular) {
		for(int e = tid; e < SHT * SHT; e += blockDim.x) {
			int ix = x0 + e % SHT, iy = y0 + e / SHT;
			if(ix >= Nx || iy >= Ny) continue;
			cx<R> o[2][2];
			for(int pol = 0; pol < 2; pol++) {
				shift_point_exact(G, P, f + pol * 2 * N, Ca, nsh, ix, iy, o[pol][0], o[pol][1]);
				o[pol][0] = o[pol][0] * ph;
				o[pol][1] = o[pol][1] * ph;
				phase_apply(Cb, N, ix + Nx * iy, o[pol][0], o[pol][1]);
			}
			for(int c = 0; c < 2; c++) fo[c * N + ix + Nx * iy] = v4<float>{o[0][c].x, o[0][c].y, o[1][c].x, o[1][c].y};
		}
		return;
	}
	constexpr int PA = SHT + 7, PB = SHT + 1;
	cx<R>* A = reinterpret_cast<cx<R>*>(smem_raw);  // [2][wy][PA]: the window
	cx<R>* B = A + 2 * (SHT + 6) * PA;             // [2][wy][PB]: the window after the x-passes
	__shared__ int places[2 * (SHT + 6)];
	const ShiftWindow<R> win(G, P, nsh, x0, y0, places);
	const int wy = win.wy, nseg = (min(SHT, Nx - x0) + 7) / 8;
	// the thread's outputs: 4 rows of one column (SHT * SHT / 4 threads)
	const int ix = x0 + tid % SHT, iy0 = y0 + tid / SHT * 4;
	cx<R> keep[2][4];
	for(int pol = 0; pol < 2; pol++) {
		if(pol) __syncthreads();  // the first slot's window has been read
		win.load(f + pol * 2 * N, Ca, N, A);
		__syncthreads();
		const cx<R>* Y = A;
		int PY = PA;
		if(ax) {
			for(int t = tid; t < 2 * nseg * wy; t += blockDim.x) {
				const int v = t % wy, r = t / wy, c = r >= nseg, seg = r - c * nseg;
				const int nin = 8 + 3 * nsh;
				const cx<R>* in = A + c * (SHT + 6) * PA + v * PA + seg * 8;
				cx<R> w[14];
#pragma unroll
				for(int k = 0; k < 14; k++) w[k] = k < nin ? in[k] : mk<R>(0, 0);
				W.template filter<14>(W.wx, w);
				cx<R>* out = B + c * (SHT + 6) * PB + v * PB + seg * 8;
#pragma unroll
				for(int k = 0; k < 8; k++) out[k] = w[k];
			}
			__syncthreads();
			Y = B;
			PY = PB;
		}
		cx<R> o[2][4];
#pragma unroll
		for(int c = 0; c < 2; c++) {
			const cx<R>* in = Y + c * (SHT + 6) * PY + (tid / SHT) * 4 * PY + tid % SHT;
			if(ay) {
				const int nin = 4 + 3 * nsh;
				cx<R> w[10];
#pragma unroll
				for(int k = 0; k < 10; k++) w[k] = k < nin ? in[k * PY] : mk<R>(0, 0);
				W.template filter<10>(W.wy, w);
#pragma unroll
				for(int k = 0; k < 4; k++) o[c][k] = w[k];
			}
			else {
#pragma unroll
				for(int k = 0; k < 4; k++) o[c][k] = in[k * PY];
			}
		}
		if(pol == 0) {
#pragma unroll
			for(int k = 0; k < 4; k++) { keep[0][k] = o[0][k]; keep[1][k] = o[1][k]; }
		}
		else if(ix < Nx) {
#pragma unroll
			for(int k = 0; k < 4; k++) {
				const int iy = iy0 + k;
				if(iy < Ny) {
					cx<R> a0 = keep[0][k] * ph, a1 = keep[1][k] * ph, b0 = o[0][k] * ph, b1 = o[1][k] * ph;
					const int p = ix + Nx * iy;
					phase_apply(Cb, N, p, a0, a1);
					phase_apply(Cb, N, p, b0, b1);
					fo[p] = v4<float>{a0.x, a0.y, b0.x, b0.y};
					fo[N + p] = v4<float>{a1.x, a1.y, b1.x, b1.y};
				}
			}
		}
	}
}

// k_phase_sync for the two slots of a (wavelength, q) (FP32), out of place: plain planes in, pairs out.
static __global__ void k_phase_sync_pair(Geom G, const cx<float>* __restrict__ CA, const cx<float>* __restrict__ CB,
		const cx<float>* __restrict__ F, v4<float>* __restrict__ Fo) {
	int p = blockIdx.x * blockDim.x + threadIdx.x;
	if(p >= G.N) return;
	const int z = blockIdx.y, g = z / G.Nq;
	const size_t N = G.N;
	const int Nx = G.Nx, Ny = G.Ny;
	const bool ax = Nx > 3, ay = Ny > 3;
	int ix = p % Nx, iy = p / Nx;
	if((ax && ix == Nx - 1) || (ay && iy == Ny - 1)) return;
	const cx<float>* f = F + (size_t)z * 4 * N + p;
	v4<float>* fo = Fo + (size_t)z * 2 * N;
	const cx<float>* Cb = CB + (size_t)g * coef_set_size(N);
	cx<float> u0 = f[0], u1 = f[N], v0 = f[2 * N], v1 = f[3 * N];
	if(CA) {
		const cx<float>* Ca = CA + (size_t)g * coef_set_size(N);
		phase_apply(Ca, N, p, u0, u1);
		phase_apply(Ca, N, p, v0, v1);
	}
	auto put = [&](int d) {
		cx<float> a = u0, b = u1, c = v0, e = v1;
		phase_apply(Cb, N, d, a, b);
		phase_apply(Cb, N, d, c, e);
		fo[d] = v4<float>{a.x, a.y, c.x, c.y};
		fo[N + d] = v4<float>{b.x, b.y, e.x, e.y};
	};
	put(p);
	if(ax && ix == 0) put((Nx - 1) + Nx * iy);
	if(ay && iy == 0) put(ix + Nx * (Ny - 1));
	if(ax && ay && ix == 0 && iy == 0) put((Nx - 1) + Nx * (Ny - 1));
}

// Entrance field: beam profile with polarisation angle pi/2*pol (BPMIteration.cpp:87-109,
// BeamProfile.cpp:17-39) followed by the input Fresnel operator (FresnelOperator.cpp:16-38)
// built on sqrt(eps_tr) at iz = 0.
template <typename R>
__global__ void k_init_fields(Geom G, int slot0, const GroupParams* __restrict__ gps, const R* __restrict__ Q0,
		int beam_type, double waist, double dx, double dy, double cpol1, double spol1, cx<R>* F) {
	// arithmetic in the plan's precision (FP32 mode: FP32, within its error budget)
	using T = R;
	int p = blockIdx.x * blockDim.x + threadIdx.x;
	if(p >= G.N) return;
	int s = blockIdx.y;
	int N = G.N, Nx = G.Nx, Ny = G.Ny;
	int gs = slot0 + s;
	int g = gs / G.spg - slot0 / G.spg;
	int pol = gs % 2;
	// polarisation (cos, sin)(pi/2 * pol); the pol = 1 values come from the host's libm
	const T cth = pol ? (T)cpol1 : (T)1, sth = pol ? (T)spol1 : (T)0;
	T amp = 1;
	if(beam_type == 1) {
		const T x = (T)(((p % Nx) - (Nx - 1) / 2.) * dx), y = (T)(((p / Nx) - (Ny - 1) / 2.) * dy), w = (T)waist;
		amp = exp(-(x * x + y * y) / (2 * w * w));
	}
	const T ex = cth * amp, ey = sth * amp;
	const R* Q = Q0 + (size_t)g * NQ * N;
	const T nxx = Q[Q_XXS * N + p], nyy = Q[Q_YYS * N + p], nxy = Q[Q_XYS * N + p];
	const T n = (T)gps[g].nin;
	const T det = (n + nxx) * (n + nyy) - nxy * nxy;
	const T a = 2 * n * (n + nyy) / det * ex - 2 * n * nxy / det * ey;
	const T b = -2 * n * nxy / det * ex + 2 * n * (n + nxx) / det * ey;
	F[(size_t)s * 2 * N + p] = mk<R>((R)a, 0);
	F[(size_t)s * 2 * N + N + p] = mk<R>((R)b, 0);
}

// Output Fresnel operator at iz = Nz-1 (FresnelOperator.cpp:45-69), in the plan's precision.
template <typename R>
__global__ void k_fresnel_out(Geom G, int slot0, const GroupParams* __restrict__ gps, const R* __restrict__ QL,
		cx<R>* F) {
	using T = R;
	int p = blockIdx.x * blockDim.x + threadIdx.x;
	if(p >= G.N) return;
	int s = blockIdx.y;
	int N = G.N;
	int g = (slot0 + s) / G.spg - slot0 / G.spg;
	const R* Q = QL + (size_t)g * NQ * N;
	const T nxx = Q[Q_XXS * N + p], nyy = Q[Q_YYS * N + p], nxy = Q[Q_XYS * N + p];
	const T n = (T)gps[g].nout_fresnel;
	const T det = (n + nxx) * (n + nyy) - nxy * nxy;
	const T axx = 2 * (1 - n * (n + nyy) / det), ayy = 2 * (1 - n * (n + nxx) / det), axy = 2 * (n * nxy / det);
	cx<R>* f = F + (size_t)s * 2 * N + p;
	const cx<R> a = f[0], b = f[N];
	f[0] = axx * a + axy * b;
	f[N] = ayy * b + axy * a;
}

template <typename R>
__global__ void k_copy(size_t n, const cx<R>* __restrict__ a, cx<R>* __restrict__ b) {
	size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if(i < n) b[i] = a[i];
}

template <typename R>
__global__ void k_widen(size_t n, const cx<R>* __restrict__ a, cx<double>* __restrict__ b) {
	size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if(i < n) b[i] = cvt<double>(a[i]);
}

template <typename R>
__global__ void k_narrow(size_t n, const cx<double>* __restrict__ a, cx<R>* __restrict__ b) {
	size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if(i < n) b[i] = cvt<R>(a[i]);
}

}  // namespace nbpm
