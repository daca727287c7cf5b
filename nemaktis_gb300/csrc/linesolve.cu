// Batched periodic tridiagonal line solves as a standalone C-ABI primitive.
//
// Restates BlockSparseMatrixDX/DY::shifted_block_vmult_inv (BeamPropagationSolver/src/
// BeamPropagationLib/BlockSparseMatrix.cpp:195-258, 386-449): each line has L points of which
// the last duplicates the first (period L-1); row i of the system is
//   inf_i x_{i-1} + mid_i x_i + sup_i x_{i+1} = b_i   (indices modulo L-1),  x_{L-1} = x_0,
// solved by a Thomas sweep with beta_0 = 2*mid_0 plus the Sherman-Morrison corner correction.
// Complex FP64 throughout. Lines that fit in shared memory: one block per line, chunks factored and
// solved side by side (k_pt_part, no scratch). Longer ones: one thread per line, factorisation into
// scratch, then solve (k_pt_factor, k_pt_solve).
#include <cuda_runtime.h>

#include <mutex>
#include <string>

#include "../../include/nbpm.h"
#include "cplx.cuh"
#include "line_join.cuh"

namespace nbpm {

void set_last_error(const std::string& m);

// Scratch per line element: 5 complex planes (alpha, 1/beta, w, -gamma, corr), plus 2 complex
// scalars per line (r0, 1/den). The forward pass keeps gamma in the -gamma plane and the
// forward corr in the corr plane; the backward pass overwrites them in place.
__global__ void k_pt_factor(int L, int nlines, const cx<double>* __restrict__ inf, const cx<double>* __restrict__ mid,
		const cx<double>* __restrict__ sup, long long ls_in, cx<double>* __restrict__ scr) {
	int line = blockIdx.x * blockDim.x + threadIdx.x;
	if(line >= nlines) return;
	const int n = L - 1;  // unknowns per line
	const size_t P = (size_t)nlines * n;
	cx<double>* FA = scr;
	cx<double>* FRB = FA + P;
	cx<double>* FW = FRB + P;
	cx<double>* FC = FW + P;
	cx<double>* FCOR = FC + P;
	cx<double>* LS = FCOR + P + (size_t)line * 2;
	const size_t o = (size_t)line * n;
	auto I = [&](int i) { return inf[line * ls_in + i]; };
	auto Mi = [&](int i) { return mid[line * ls_in + i]; };
	auto S = [&](int i) { return sup[line * ls_in + i]; };
	const cx<double> one = mk(1.0, 0.0);
	cx<double> beta = 2.0 * Mi(0);
	cx<double> rb = crecip(beta);
	FRB[o] = rb;
	FA[o] = mk(0.0, 0.0);
	cx<double> corr = mk(-0.5, 0.0);
	FCOR[o] = corr;
	for(int i = 1; i < n - 1; i++) {
		cx<double> gam = S(i - 1) * rb;
		FC[o + i - 1] = gam;
		beta = Mi(i) - I(i) * gam;
		rb = crecip(beta);
		FRB[o + i] = rb;
		FA[o + i] = -(I(i) * rb);
		corr = -(I(i) * corr) * rb;
		FCOR[o + i] = corr;
	}
	cx<double> gl = S(n - 2) * rb;
	FC[o + n - 2] = gl;
	beta = Mi(n - 1) + cdiv(S(n - 1) * I(0), Mi(0)) - I(n - 1) * gl;
	rb = crecip(beta);
	FRB[o + n - 1] = rb;
	FA[o + n - 1] = -(I(n - 1) * rb);
	cx<double> corr_last = (S(n - 1) - I(n - 1) * corr) * rb;
	// w_i = prod_{j<i}(-gamma_j) from the forward gammas, before they are negated
	cx<double> w = one;
	FW[o] = w;
	for(int i = 1; i < n; i++) {
		w = -(w * FC[o + i - 1]);
		FW[o + i] = w;
	}
	FCOR[o + n - 1] = corr_last;
	cx<double> cn = corr_last;
	for(int i = n - 1; i > 0; i--) {
		cx<double> g = FC[o + i - 1];
		cx<double> cv = FCOR[o + i - 1] - g * cn;
		FCOR[o + i - 1] = cv;
		FC[o + i - 1] = -g;
		cn = cv;
	}
	FC[o + n - 1] = mk(0.0, 0.0);
	cx<double> r0 = cdiv(I(0), Mi(0));
	LS[0] = r0;
	LS[1] = crecip(one + cn - r0 * corr_last);
}

__global__ void k_pt_solve(int L, int nlines, long long ls_b, const cx<double>* __restrict__ scr,
		const cx<double>* __restrict__ b, cx<double>* __restrict__ x) {
	int line = blockIdx.x * blockDim.x + threadIdx.x;
	if(line >= nlines) return;
	const int n = L - 1;
	const size_t P = (size_t)nlines * n;
	const cx<double>* FA = scr;
	const cx<double>* FRB = FA + P;
	const cx<double>* FW = FRB + P;
	const cx<double>* FC = FW + P;
	const cx<double>* FCOR = FC + P;
	const cx<double>* LS = FCOR + P + (size_t)line * 2;
	const size_t o = (size_t)line * n;
	const cx<double>* bb = b + line * ls_b;
	cx<double>* xx = x + line * ls_b;
	cx<double> d = bb[0] * FRB[o];
	cx<double> acc = d;
	xx[0] = d;
	for(int i = 1; i < n; i++) {
		d = FA[o + i] * d + bb[i] * FRB[o + i];
		acc += FW[o + i] * d;
		xx[i] = d;
	}
	cx<double> fr = (acc - LS[0] * d) * LS[1];
	cx<double> dn = d;
	cx<double> v = dn - fr * FCOR[o + n - 1];
	xx[n - 1] = v;
	for(int i = n - 1; i > 0; i--) {
		cx<double> dp = xx[i - 1] + FC[o + i - 1] * dn;
		v = dp - fr * FCOR[o + i - 1];
		xx[i - 1] = v;
		dn = dp;
	}
	xx[n] = v;  // duplicate point
}

// Largest smaller-than-rounding coupling: ln of 2^-57; Jacobi steps beyond which the chunks are joined by
// ring_solve, which with its factorisation costs about as much (700 lines of 199 unknowns, 8 steps: 56 us, 83 us
// joined by ring_solve); and the change of a border unknown, relative to itself, that one more
// step may make.
constexpr double PT_LN_TOL = -39.5;
constexpr int PT_KMAX = 24;
constexpr double PT_CHANGE = 1.0 / (1ll << 50);

__device__ __forceinline__ double pt_l1(cx<double> z) { return l1abs(z); }
// 1 / b; clears ok where |b|^2 leaves the range of doubles.
__device__ __forceinline__ cx<double> pt_recip(cx<double> b, bool& ok) {
	const double d = b.x * b.x + b.y * b.y;
	ok = ok && d > 1e-280 && d < 1e280;
	const double r = 1.0 / d;
	return mk(b.x * r, -b.y * r);
}

// One block per line of n = L - 1 unknowns, thread t its points [t M, t M + M). The line's four arrays are
// staged in shared memory (coalesced) and overwritten in place. Every chunk is swept by itself (LU
// without pivoting): d the forward values, ev what the unknown before the chunk adds to them, rb = 1/pivot,
// cc = -sup * rb; yf, vf and wf are the responses of its first unknown to the right-hand sides, the
// unknown before and the one after the chunk, yl, vl and wl those of its last one. Neighbouring chunks
// then join through their border unknowns: h (a chunk's last) and g (the next one's first) from the two
// chunks alone, corrected by K Jacobi steps for the chunks beyond, K from the couplings so that what is
// left is below rounding. Lines that would need many steps, and those where one step more changes an unknown
// noticeably against its own size (right-hand sides of very different magnitudes along the line, NaN and
// infinities) are joined by ring_solve instead: its scans keep small unknowns beside large ones as exact as
// a sweep along the line does. A line whose multipliers or join pivots are large (not diagonally dominant) is
// solved again from its inputs by one thread, as k_pt_factor and k_pt_solve do.
// Bound: the FP64 pipe, about 58 multiply-adds per point plus the reciprocal. 2048 lines of 512: one
// thread per line with strided loads took 3.02 ms, this kernel 0.18 ms. 2000 lines of 249 unknowns (last chunk of
// one point, some joined by ring_solve): 1.51 ms, 0.19 ms here (2.12 ms where such lines were swept by one thread).
__global__ void __launch_bounds__(256) k_pt_part(int L, int M, const cx<double>* __restrict__ inf,
		const cx<double>* __restrict__ mid, const cx<double>* __restrict__ sup, const cx<double>* rhs, cx<double>* x) {
	extern __shared__ unsigned char smem_raw[];
	__shared__ int sK;
	const int n = L - 1, T = blockDim.x, t = threadIdx.x;
	const int Mp = M | 1;  // odd chunk pitch: no bank conflicts of the chunk-ordered accesses
	const int nchk = (n + M - 1) / M, CH = nchk * Mp;
	cx<double>* sA = reinterpret_cast<cx<double>*>(smem_raw);
	cx<double>* sB = sA + CH;
	cx<double>* sC = sB + CH;
	cx<double>* sD = sC + CH;
	cx<double>* sv = sD + CH;  // [T] each: vf, wf, yf; then h and g, two buffers
	cx<double>* sw = sv + T;
	cx<double>* sy = sw + T;
	cx<double>* sH = sy + T;
	cx<double>* sG = sH + 2 * T;
	const size_t o = (size_t)blockIdx.x * L;
	auto at = [&](int i) { const int c = i / M; return c * Mp + (i - c * M); };
	auto stage = [&] {
		for(int i = t; i < n; i += T) {
			const int q = at(i);
			sA[q] = inf[o + i];
			sB[q] = mid[o + i];
			sC[q] = sup[o + i];
			sD[q] = rhs[o + i];
		}
	};
	if(t == 0) sK = 0;
	stage();
	__syncthreads();
	const cx<double> one = mk(1.0, 0.0), zero = mk(0.0, 0.0);
	const int m = min(M, n - t * M), q0 = t * Mp;  // m <= 0: no chunk
	const int next = t >= nchk - 1 ? 0 : t + 1, prev = t == 0 ? nchk - 1 : t - 1;
	cx<double> rb = zero, ev = zero, d = zero, cc = zero, cpz = one, vf = zero, yf = zero, cs = zero;
	bool ok = true;
	for(int k = 0; k < m; k++) {
		const cx<double> a = sA[q0 + k], b = sB[q0 + k], c = sC[q0 + k], r = sD[q0 + k];
		cx<double> beta = b;
		if(k == 0) { ev = -a; d = r; }
		else {
			const cx<double> l = a * rb;
			ok = ok && pt_l1(l) <= 2.0;
			beta = cfnma(l, cs, b);
			ev = -(l * ev);
			d = cfnma(l, d, r);
		}
		rb = pt_recip(beta, ok);
		cs = c;
		cc = -(rb * c);
		ok = ok && pt_l1(cc) <= 2.0;
		const cx<double> z = cpz * rb;
		vf = cfma(z, ev, vf);
		yf = cfma(z, d, yf);
		cpz = cpz * cc;
		sA[q0 + k] = ev;
		sB[q0 + k] = rb;
		sC[q0 + k] = cc;
		sD[q0 + k] = d;
	}
	if(m > 0) { sv[t] = vf; sw[t] = cpz; sy[t] = yf; }
	__syncthreads();
	cx<double> h = zero, g = zero, ph = zero, pg = zero, qh = zero, qg = zero;
	if(m > 0) {
		const cx<double> vl = rb * ev, yl = rb * d, vn = sv[next], wn = sw[next], yn = sy[next];
		const cx<double> p = pt_recip(cfnma(cc, vn, one), ok);
		ok = ok && pt_l1(p) <= 4.0;
		const cx<double> pw = p * cc, pv = p * vn;
		h = cfma(p, yl, pw * yn);
		g = cfma(pv, yl, p * yn);
		ph = p * vl; pg = pv * vl; qh = pw * wn; qg = p * wn;
		const float rho = (float)fmax(pt_l1(ph) + pt_l1(qh), pt_l1(pg) + pt_l1(qg));
		int K = PT_KMAX + 1;
		if(rho < 1.f) {
			const float lr = logf(rho);  // -inf for rho = 0
			K = lr < (float)PT_LN_TOL ? 0 : (int)fminf(ceilf((float)PT_LN_TOL / lr) - 1.f, PT_KMAX + 1.f);
		}
		if(!ok) K = PT_KMAX + 2;
		if(K) atomicMax(&sK, K);
	}
	__syncthreads();
	const int K = nchk < 2 ? PT_KMAX + 2 : sK;
	bool seq = K > PT_KMAX + 1;
	if(!seq) {
		const cx<double> bh = h, bg = g;
		cx<double> hl;
		bool done = K <= PT_KMAX;
		if(done)
		for(int it = 0;; it++) {
			// two buffers in turn: the one written here was last read two barriers ago
			cx<double>* H = sH + (it & 1) * T;
			cx<double>* Gb = sG + (it & 1) * T;
			H[t] = h;
			Gb[t] = g;
			__syncthreads();
			hl = H[prev];
			const cx<double> gr = Gb[next], hn = cfma(qh, gr, cfma(ph, hl, bh)), gn = cfma(qg, gr, cfma(pg, hl, bg));
			if(it == K) {
				done = __syncthreads_and(m <= 0 || pt_l1(hn - h) + pt_l1(gn - g) <= PT_CHANGE * fmin(pt_l1(h), pt_l1(g)));
				break;
			}
			h = hn;
			g = gn;
		}
		if(!done) {
			const LineThreads lt{T / 32, 0, t / 32, t % 32, t, nchk - 1};
			RingNode<double> r;
			if(T > 32) r = ring_factor<true>(lt, ph, pg, qh, qg, sv);
			else r = ring_factor<false>(lt, ph, pg, qh, qg, sv);
			seq = !__syncthreads_and(m <= 0 || pt_l1(r.d) <= 4.0);
			if(!seq) {
				h = cfma(r.f2, bg, bh);
				g = r.d * bg;
				if(T > 32) ring_solve<true, 1, double>(lt, r, &h, &g, &hl, sw);
				else ring_solve<false, 1, double>(lt, r, &h, &g, &hl, sw);
			}
		}
		if(!seq) {
			cx<double> v = g;
			for(int k = m - 1; k >= 0; k--) {
				v = cfma(sC[q0 + k], v, sB[q0 + k] * cfma(sA[q0 + k], hl, sD[q0 + k]));
				sD[q0 + k] = v;
			}
		}
	}
	if(seq) {
		__syncthreads();
		stage();
		__syncthreads();
		if(t == 0) {
			// forward: d, corr (in sA), gamma (in sC) and the sums that give the back-substituted first
			// unknowns; see k_pt_factor
			const cx<double> a0 = sA[0], m0 = sB[0];
			cx<double> r = crecip(2.0 * m0);
			cx<double> dv = sD[0] * r, corr = mk(-0.5, 0.0), w = one, gam = sC[0] * r;
			cx<double> acc = dv, cv0 = corr;
			sD[0] = dv; sA[0] = corr; sC[0] = gam;
			for(int i = 1; i < n; i++) {
				const int q = at(i);
				const cx<double> a = sA[q], s = sC[q];
				cx<double> beta = sB[q] - a * gam;
				if(i == n - 1) beta = beta + cdiv(s * a0, m0);
				r = crecip(beta);
				dv = (sD[q] - a * dv) * r;
				corr = ((i == n - 1 ? s : zero) - a * corr) * r;
				w = -(w * gam);
				gam = s * r;
				acc += w * dv;
				cv0 += w * corr;
				sD[q] = dv; sA[q] = corr; sC[q] = gam;
			}
			const cx<double> r0 = cdiv(a0, m0);
			const cx<double> fr = (acc - r0 * dv) * crecip(one + cv0 - r0 * corr);
			cx<double> dn = dv, cn = corr;
			sD[at(n - 1)] = dn - fr * cn;
			for(int i = n - 2; i >= 0; i--) {
				const int q = at(i);
				dn = sD[q] - sC[q] * dn;
				cn = sA[q] - sC[q] * cn;
				sD[q] = dn - fr * cn;
			}
		}
	}
	__syncthreads();
	for(int i = t; i < L; i += T) x[o + i] = sD[at(i == n ? 0 : i)];
}

// Threads and chunk length of k_pt_part for a line of n unknowns, and its shared memory; false if the line
// does not fit (above 2750 unknowns). One warp a line as long as several lines share an SM (512 points: 35
// KB); more for longer lines, and when the lines are too few to give every SM four warps. Chunks of at
// least 4 points: shorter ones need more steps to join than they save.
static bool pt_part_shape(int n, int nlines, int& T, int& M, size_t& smem) {
	T = n <= 512 ? 32 : n <= 1024 ? 64 : n <= 2048 ? 128 : 256;
	while(T < 128 && (long long)nlines * (T / 32) < 4 * 152 && n >= 8 * T) T *= 2;
	M = (n + T - 1) / T;
	if(M < 4) M = 4;
	for(int k = 0; k < 2; k++, M++) {
		const int nchk = (n + M - 1) / M;
		smem = ((size_t)4 * nchk * (M | 1) + (size_t)7 * T) * sizeof(cx<double>);
		// an even length is padded to the next odd one, which may fit where it does not
		if(smem <= 200 * 1024) return true;
	}
	return false;
}

// Whether a call needs the scratch of pt_scratch_elems.
bool pt_needs_scratch(int L, int nlines) {
	int T, M;
	size_t smem;
	return !pt_part_shape(L - 1, nlines, T, M, smem);
}

size_t pt_scratch_elems(int L, int nlines) { return (size_t)nlines * (L - 1) * 5 + (size_t)nlines * 2; }

int pt_check(int L, int nlines, const void* a, const void* b, const void* c, const void* d, const void* e,
		std::string& err) {
	if(L < 4) { err = "line length must be >= 4 (period L-1 >= 3)"; return NBPM_ERR_ARG; }
	if(nlines < 1) { err = "nlines must be >= 1"; return NBPM_ERR_ARG; }
	if(!a || !b || !c || !d || !e) { err = "null device pointer"; return NBPM_ERR_ARG; }
	return 0;
}

int pt_run(int L, int nlines, const double* inf, const double* mid, const double* sup, const double* rhs,
		double* x, cudaStream_t st, cx<double>* scr, std::string& err) {
	int Tp, M;
	size_t smem;
	if(pt_part_shape(L - 1, nlines, Tp, M, smem)) {
		if(smem > 48 * 1024) {
			const cudaError_t e = cudaFuncSetAttribute(k_pt_part, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
			if(e != cudaSuccess) { err = cudaGetErrorString(e); return NBPM_ERR_CUDA; }
		}
		k_pt_part<<<(unsigned)nlines, Tp, smem, st>>>(L, M, reinterpret_cast<const cx<double>*>(inf),
			reinterpret_cast<const cx<double>*>(mid), reinterpret_cast<const cx<double>*>(sup),
			reinterpret_cast<const cx<double>*>(rhs), reinterpret_cast<cx<double>*>(x));
		const cudaError_t e = cudaGetLastError();
		if(e != cudaSuccess) { err = cudaGetErrorString(e); return NBPM_ERR_CUDA; }
		return 0;
	}
	const int T = 128;
	const unsigned blocks = (unsigned)((nlines + T - 1) / T);
	k_pt_factor<<<blocks, T, 0, st>>>(L, nlines, reinterpret_cast<const cx<double>*>(inf),
		reinterpret_cast<const cx<double>*>(mid), reinterpret_cast<const cx<double>*>(sup), (long long)L, scr);
	k_pt_solve<<<blocks, T, 0, st>>>(L, nlines, (long long)L, scr, reinterpret_cast<const cx<double>*>(rhs),
		reinterpret_cast<cx<double>*>(x));
	cudaError_t e = cudaGetLastError();
	if(e != cudaSuccess) { err = cudaGetErrorString(e); return NBPM_ERR_CUDA; }
	return 0;
}

}  // namespace nbpm

using namespace nbpm;


extern "C" {

int nbpm_periodic_tridiag_solve(int L, int nlines, const double* inf, const double* mid, const double* sup,
		const double* rhs, double* x, void* stream) {
	std::string err;
	int rc = pt_check(L, nlines, inf, mid, sup, rhs, x, err);
	if(rc) { set_last_error(err); return rc; }
	cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
	cx<double>* scr = nullptr;
	cudaError_t e = cudaSuccess;
	if(pt_needs_scratch(L, nlines)) {
		e = cudaMallocAsync(reinterpret_cast<void**>(&scr), pt_scratch_elems(L, nlines) * sizeof(cx<double>), st);
		if(e != cudaSuccess) {
			set_last_error(cudaGetErrorString(e));
			return e == cudaErrorMemoryAllocation ? NBPM_ERR_MEMORY : NBPM_ERR_CUDA;
		}
	}
	rc = pt_run(L, nlines, inf, mid, sup, rhs, x, st, scr, err);
	if(scr) cudaFreeAsync(scr, st);
	if(rc) { set_last_error(err); return rc; }
	e = cudaStreamSynchronize(st);
	if(e != cudaSuccess) { set_last_error(cudaGetErrorString(e)); return NBPM_ERR_CUDA; }
	return 0;
}

}  // extern "C"
