// Batched 2-D complex FFTs and the screen-plane Fourier filter.
//
// The reference transforms each wavelength's 4*Nq planes (Ny, Nx) with FFTW
// (OpticalFieldCollection.cpp:62-71: unnormalised, full Nx including the duplicated
// periodic column) and multiplies by the 2x2 transfer filter of ScreenOutput.cpp:226-302.
// Here a line FFT is a shared-memory Stockham autosort transform, mixed radix: stages of
// radix 4, 2, 3, 5, 7 and a generic prime radix. A block transforms `lpb` lines; rows
// (stride 1) load with the element index fastest, columns (stride Nx) load adjacent columns
// together so global accesses stay coalesced. Twiddles W_n^k = exp(-2*pi*i*k/n) come from a
// table computed on the host in FP64 with std::cos/std::sin.
#pragma once

#include <algorithm>

#include "cplx.cuh"

namespace nbpm {

constexpr int FFT_MAX_STAGES = 24;

struct FftPlan1D {
	int n;
	int nst;
	int radix[FFT_MAX_STAGES];
	// e / d as umulhi(e, m), m = ceil(2^32 / d) (exact while e * d < 2^32), 0 for d = 1: for d = the
	// butterflies per line n / radix and the stage's Ns
	unsigned m_nb[FFT_MAX_STAGES], m_ns[FFT_MAX_STAGES];
	int pmax;  // entries of the shared DFT table of the largest radix above 8; 0: none, or read from tw
};

// Radix sequence for a length-n line: 4s, then 2s, then odd primes in increasing order.
// Returns false when n needs more than FFT_MAX_STAGES stages.
inline bool fft_plan_1d(int n, FftPlan1D& P) {
	P.n = n;
	P.nst = 0;
	auto push = [&](int r) {
		if(P.nst >= FFT_MAX_STAGES) return false;
		P.radix[P.nst++] = r;
		return true;
	};
	while(n % 4 == 0 && n > 1) { if(!push(4)) return false; n /= 4; }
	while(n % 2 == 0) { if(!push(2)) return false; n /= 2; }
	for(int p = 3; n > 1 && p * p <= n; p += 2)
		while(n % p == 0) { if(!push(p)) return false; n /= p; }
	if(n > 1 && !push(n)) return false;
	auto magic = [](int d) { return d == 1 ? 0u : (unsigned)((0x100000000ull + (unsigned)d - 1) / (unsigned)d); };
	P.pmax = 0;
	int Ns = 1;
	for(int i = 0; i < P.nst; i++) {
		P.m_nb[i] = magic(P.n / P.radix[i]);
		P.m_ns[i] = magic(Ns);
		Ns *= P.radix[i];
		if(P.radix[i] > 8) P.pmax = std::max(P.pmax, P.radix[i]);
	}
	return true;
}
__device__ __forceinline__ int fdiv(int e, unsigned m) { return m ? (int)__umulhi((unsigned)e, m) : e; }
// Leaves the DFT table out where a line and the table do not fit.
template <typename R>
inline void fft_fit(FftPlan1D& P, size_t smem_limit) {
	if(((size_t)2 * (P.n + 1) + P.pmax) * sizeof(cx<R>) > smem_limit) P.pmax = 0;
}
// Shared memory of nl lines: two buffers of pitch n + 1, and the DFT table of a large prime factor.
template <typename R>
inline size_t fft_smem(const FftPlan1D& P, int nl) { return ((size_t)2 * nl * (P.n + 1) + P.pmax) * sizeof(cx<R>); }

template <typename R>
__device__ __forceinline__ cx<R> tw_get(const cx<R>* tw, int idx, int sign) {
	cx<R> w = tw[idx];
	return sign > 0 ? conj(w) : w;
}

// Mixed-radix Stockham stages on nl lines held in shared memory (pitch n+1): `in` holds the
// input; returns the buffer (in or out) that holds the transform. wp: P.pmax entries for the DFT table
// of a large prime factor. Ends with __syncthreads().
template <typename R>
__device__ cx<R>* fft_stages(cx<R>* in, cx<R>* out, const FftPlan1D& P, int nl, const cx<R>* __restrict__ tw,
		int sign, cx<R>* wp) {
	const int n = P.n, pitch = n + 1;
	int Ns = 1;
	for(int st = 0; st < P.nst; st++) {
		const int p = P.radix[st];
		const int nb = n / p;  // butterflies per line
		const int span = n / (Ns * p);  // twiddle index scale
		const unsigned mnb = P.m_nb[st], mns = P.m_ns[st];
		if(p <= 8) {
			for(int e = threadIdx.x; e < nl * nb; e += blockDim.x) {
				const int li = fdiv(e, mnb), j = e - li * nb;
				const cx<R>* I = in + li * pitch;
				cx<R>* O = out + li * pitch;
				const int jq = fdiv(j, mns), k = j - jq * Ns;
				const int obase = jq * Ns * p + k;
				cx<R> v[8];
				for(int r = 0; r < p; r++) {
					cx<R> x = I[j + r * nb];
					if(r && k) x = x * tw_get(tw, r * k * span, sign);
					v[r] = x;
				}
				if(p == 2) {
					O[obase] = v[0] + v[1];
					O[obase + Ns] = v[0] - v[1];
				}
				else if(p == 4) {
					cx<R> a = v[0] + v[2], b = v[0] - v[2];
					cx<R> c = v[1] + v[3], d = v[1] - v[3];
					// multiply d by -i (forward) or +i (backward)
					cx<R> dj = sign > 0 ? mk<R>(-d.y, d.x) : mk<R>(d.y, -d.x);
					O[obase] = a + c;
					O[obase + Ns] = b + dj;
					O[obase + 2 * Ns] = a - c;
					O[obase + 3 * Ns] = b - dj;
				}
				else {
					int wstep = n / p;
					for(int s = 0; s < p; s++) {
						cx<R> acc = v[0];
						for(int r = 1; r < p; r++)
							acc += v[r] * tw_get(tw, ((r * s) % p) * wstep, sign);
						O[obase + s * Ns] = acc;
					}
				}
			}
		}
		else {
			// large prime: with a_r = x_r + x_{p-r}, b_r = x_r - x_{p-r} the outputs s and p - s are
			// x_0 + sum_r a_r cos(2 pi r s / p) -+ i sum_r b_r sin(2 pi r s / p), p multiply-adds per output
			// in place of 4 p. One pass forms the twiddled a_r and b_r in place (b_r where x_{p-r} was),
			// then a thread takes one pair of outputs. 97-point rows of 84 planes, FP64: 3630 us with one thread per
			// line and every product complex, 122 us so.
			const int hp = (p - 1) / 2, wstep = n / p;
			const bool table = P.pmax > 0;
			if(table)
				for(int i = threadIdx.x; i < p; i += blockDim.x) wp[i] = conj(tw[i * wstep]);  // cos, sin
			for(int e = threadIdx.x; e < nl * nb * hp; e += blockDim.x) {
				const int f = e / hp, r = e - f * hp + 1;
				const int li = fdiv(f, mnb), j = f - li * nb;
				cx<R>* I = in + li * pitch + j;
				const int jq = fdiv(j, mns), k = j - jq * Ns;
				cx<R> x = I[r * nb], y = I[(p - r) * nb];
				if(k) {
					x = x * tw_get(tw, r * k * span, sign);
					y = y * tw_get(tw, (p - r) * k * span, sign);
				}
				I[r * nb] = x + y;
				I[(p - r) * nb] = x - y;
			}
			__syncthreads();
			for(int e = threadIdx.x; e < nl * nb * (hp + 1); e += blockDim.x) {
				// pair s = 0 .. hp of butterfly f (s = 0: the sum alone)
				const int f = e / (hp + 1), s = e - f * (hp + 1);
				const int li = fdiv(f, mnb), j = f - li * nb;
				const cx<R>* I = in + li * pitch + j;
				const int jq = fdiv(j, mns), k = j - jq * Ns;
				cx<R>* O = out + li * pitch + jq * Ns * p + k;
				cx<R> A = I[0], B = mk<R>(0, 0);
				int idx = 0;
				for(int r = 1; r <= hp; r++) {
					idx += s;
					if(idx >= p) idx -= p;
					const cx<R> w = table ? wp[idx] : conj(tw[idx * wstep]), a = I[r * nb], b = I[(p - r) * nb];
					A = mk<R>(fmar(w.x, a.x, A.x), fmar(w.x, a.y, A.y));
					B = mk<R>(fmar(w.y, b.x, B.x), fmar(w.y, b.y, B.y));
				}
				if(s == 0) O[0] = A;
				else {
					const cx<R> iB = sign > 0 ? mk<R>(-B.y, B.x) : mk<R>(B.y, -B.x);  // +-i B
					O[s * Ns] = A + iB;
					O[(p - s) * Ns] = A - iB;
				}
			}
		}
		__syncthreads();
		cx<R>* t = in; in = out; out = t;
		Ns *= p;
	}
	return in;
}

// Transform `nlines` lines of length P.n. Line l starts at base(l) = (l / lines_per_plane)
// * plane_stride + (l % lines_per_plane) * line_stride and its elements are elem_stride apart.
// Reads from `src` (data when null) and writes to `data`. keep (may be null): one byte per element for
// every 4 planes; elements whose byte is 0 are taken as zero and not read.
template <typename R>
static __global__ void k_fft_lines(cx<R>* data, const cx<R>* src, FftPlan1D P, int nlines, int lines_per_plane,
		long long plane_stride, long long line_stride, long long elem_stride, int lpb,
		const cx<R>* __restrict__ tw, int sign, const unsigned char* __restrict__ keep = nullptr) {
	extern __shared__ unsigned char smem_raw[];
	cx<R>* sA = reinterpret_cast<cx<R>*>(smem_raw);
	const int n = P.n, pitch = n + 1;
	cx<R>* sB = sA + (size_t)lpb * pitch;
	cx<R>* wp = sB + (size_t)lpb * pitch;
	const int l0 = blockIdx.x * lpb;
	const int nl = min(lpb, nlines - l0);
	if(nl <= 0) return;
	const cx<R>* in_data = src ? src : data;
	auto base = [&](int l) {
		return (long long)(l / lines_per_plane) * plane_stride + (long long)(l % lines_per_plane) * line_stride;
	};
	const int tot = nl * n;
	if(elem_stride == 1) {
		// a warp per line
		for(int li = threadIdx.x / 32; li < nl; li += blockDim.x / 32) {
			const cx<R>* q = in_data + base(l0 + li);
			const unsigned char* kp = keep ? keep + (size_t)((l0 + li) / lines_per_plane / 4) * n : nullptr;
			for(int i = threadIdx.x % 32; i < n; i += 32) sA[li * pitch + i] = !kp || kp[i] ? q[i] : mk<R>(0, 0);
		}
	}
	else {
		for(int e = threadIdx.x; e < tot; e += blockDim.x) {
			int li = e % nl, i = e / nl;
			sA[li * pitch + i] = in_data[base(l0 + li) + (long long)i * elem_stride];
		}
	}
	__syncthreads();
	cx<R>* in = fft_stages<R>(sA, sB, P, nl, tw, sign, wp);
	if(elem_stride == 1) {
		for(int li = threadIdx.x / 32; li < nl; li += blockDim.x / 32) {
			cx<R>* q = data + base(l0 + li);
			for(int i = threadIdx.x % 32; i < n; i += 32) q[i] = in[li * pitch + i];
		}
	}
	else {
		for(int e = threadIdx.x; e < tot; e += blockDim.x) {
			int li = e % nl, i = e / nl;
			data[base(l0 + li) + (long long)i * elem_stride] = in[li * pitch + i];
		}
	}
}

// Screen filter of ScreenOutput::assemble_fourier_filter (ScreenOutput.cpp:226-302), FP64,
// applied to both polarisation slots of every (group, q) with the 1/(Nx*Ny) scaling of
// apply_no_export (:212-219). q0_sqr is |q0| as in :252.
struct ScreenParams {
	int Nx, Ny, Nq, n_iso;
	double dx, dy, NA, z_foc;
	double thick[8];
	double index[9];  // iso layer indices; last entry replaced per group by nout(lambda)
};

// Transverse wavevector of Fourier mode i of n (spacing d) over k0, plus q (ScreenOutput.cpp:226-302).
__device__ __forceinline__ double screen_q(int i, int n, double d, double lambda, double q) {
	const double PI_REF = 3.1415926535897932;
	const double k = (i < double(n / 2.)) ? 2 * PI_REF * i / (d * n) : -2 * PI_REF * (n - i) / (d * n);
	return k / (2 * PI_REF / lambda) + q;
}

// The transfer matrix M (2x2, scaled by 1 / (Nx Ny)) of the mode of wavevector (q0d, q1d) for illumination
// (qx, qy); zero outside the aperture.
template <typename R>
__device__ void screen_matrix(const ScreenParams& sp, double q0d, double q1d, double lambda, double nout_, double qx, double qy,
		cx<R> M[2][2]) {
	// transfer matrices in the plan's precision (FP32 mode: FP32, within its error budget)
	using T = R;
	const double PI_REF = 3.1415926535897932;
	const T k0 = (T)(2 * PI_REF / lambda);
	// the aperture test |q| < NA in FP64 in both modes, so that no mode near its edge flips in or out; the
	// square root decides only within rounding of the edge
	const double qsq = q0d * q0d + q1d * q1d, na2 = sp.NA * sp.NA;
	const bool inside = sp.NA > 0 && (qsq < na2 * (1 - 1e-12) || (qsq < na2 * (1 + 1e-12) && sqrt(qsq) < sp.NA));
	const cx<T> zero = mk<T>(0, 0);
	M[0][0] = M[0][1] = M[1][0] = M[1][1] = zero;
	if(inside) {
		const T qx0 = (T)qx, qy0 = (T)qy;
		const T q0 = (T)q0d, q1 = (T)q1d;
		const T qn2 = (T)qsq;
		const T q0s = sqrt(qx0 * qx0 + qy0 * qy0);
		const T inv = (T)(1.0 / ((double)sp.Nx * sp.Ny));
		if(sp.n_iso == 0) {
			// no layers: the focal phase alone
			const T ph = (sqrt((T)nout_ * (T)nout_ - qn2) - sqrt((T)nout_ * (T)nout_ - q0s)) * k0 * (T)sp.z_foc;
			if(ph == (T)0) M[0][0] = mk<T>(inv, 0);
			else M[0][0] = mk<T>(cos(ph) * inv, sin(ph) * inv);
			M[1][1] = M[0][0];
			return;
		}
		const T n_out = (T)nout_;
		cx<T> TM[4][4];
		for(int a = 0; a < 4; a++) for(int b = 0; b < 4; b++) TM[a][b] = mk<T>(a == b ? 1 : 0, 0);
		for(int l = 0; l < sp.n_iso; l++) {
			const T np = (T)sp.index[l];
			const T nn = (l + 1 < sp.n_iso) ? (T)sp.index[l + 1] : n_out;
			const T neff = sqrt(np * np - qn2), nneff = sqrt(nn * nn - qn2);
			const T im[2][2] = {{neff + q0 * q0 / neff, q0 * q1 / neff}, {q0 * q1 / neff, neff + q1 * q1 / neff}};
			const T ni[2][2] = {{(1 - (q0 / nn) * (q0 / nn)) / nneff, -q0 * q1 / (nn * nn * nneff)},
				{-q0 * q1 / (nn * nn * nneff), (1 - (q1 / nn) * (q1 / nn)) / nneff}};
			T tp[2][2], tm[2][2];
			for(int a = 0; a < 2; a++) for(int b = 0; b < 2; b++)
				tp[a][b] = (T)0.5 * ((a == b ? (T)1 : (T)0) + ni[a][0] * im[0][b] + ni[a][1] * im[1][b]);
			for(int a = 0; a < 2; a++) for(int b = 0; b < 2; b++) tm[a][b] = (a == b ? (T)1 : (T)0) - tp[a][b];
			const T ph = (neff - sqrt(np * np - q0s)) * k0 * (T)sp.thick[l];
			const cx<T> gg = mk<T>(cos(ph), sin(ph)), gc = conj(gg);
			cx<T> Lm[4][4];
			for(int a = 0; a < 2; a++) for(int b = 0; b < 2; b++) {
				Lm[a][b] = tp[a][b] * gg;
				Lm[a][b + 2] = tm[a][b] * gc;
				Lm[a + 2][b] = tm[a][b] * gg;
				Lm[a + 2][b + 2] = tp[a][b] * gc;
			}
			cx<T> T2[4][4];
			for(int a = 0; a < 4; a++) for(int b = 0; b < 4; b++) {
				cx<T> s = zero;
				for(int c = 0; c < 4; c++) s += Lm[a][c] * TM[c][b];
				T2[a][b] = s;
			}
			for(int a = 0; a < 4; a++) for(int b = 0; b < 4; b++) TM[a][b] = T2[a][b];
		}
		const cx<T> det = TM[2][2] * TM[3][3] - TM[2][3] * TM[3][2];
		const cx<T> tmp[2][2] = {{cdiv(TM[3][3], det), cdiv(-TM[2][3], det)}, {cdiv(-TM[3][2], det), cdiv(TM[2][2], det)}};
		const T ph = (sqrt(n_out * n_out - qn2) - sqrt(n_out * n_out - q0s)) * k0 * (T)sp.z_foc;
		const cx<T> e = mk<T>(cos(ph), sin(ph));
		for(int a = 0; a < 2; a++) for(int b = 0; b < 2; b++) {
			cx<T> s = zero;
			for(int c = 0; c < 2; c++) for(int d = 0; d < 2; d++) s += TM[a][c + 2] * tmp[c][d] * TM[d + 2][b];
			M[a][b] = ((TM[a][b] - s) * e) * inv;
		}
	}
}

template <typename R>
__global__ void k_screen_filter(cx<R>* F, ScreenParams sp, int g0, const double* __restrict__ wl,
		const double* __restrict__ nout, const double* __restrict__ qv) {
	int p = blockIdx.x * blockDim.x + threadIdx.x;
	const int Nx = sp.Nx, N = Nx * sp.Ny;
	if(p >= N) return;
	int gq = blockIdx.y;            // group-local (g, q)
	int g = gq / sp.Nq, q = gq % sp.Nq;
	cx<R> M[2][2];
	const double la = wl[g0 + g], qx = qv[2 * q], qy = qv[2 * q + 1];
	screen_matrix<R>(sp, screen_q(p % Nx, Nx, sp.dx, la, qx), screen_q(p / Nx, sp.Ny, sp.dy, la, qy), la, nout[g0 + g], qx, qy, M);
	for(int pol = 0; pol < 2; pol++) {
		size_t slot = (size_t)pol + 2 * ((size_t)q + (size_t)sp.Nq * g);
		cx<R>* f = F + slot * 2 * N + p;
		const cx<R> a = f[0], b = f[N];
		f[0] = M[0][0] * a + M[0][1] * b;
		f[N] = M[1][0] * a + M[1][1] * b;
	}
}

// Which Fourier columns of a (wavelength, q) reach the aperture: |kx / k0 + qx| < NA. Outside, the matrix of every
// mode of the column is zero: sqrt(q0^2 + q1^2) is not below |q0| in floating point either.
static __global__ void k_screen_keep(ScreenParams sp, size_t n, const double* __restrict__ wl, const double* __restrict__ qv,
		unsigned char* __restrict__ keep) {
	const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if(t >= n) return;
	const int ix = (int)(t % sp.Nx), gq = (int)(t / sp.Nx);
	const double q0 = screen_q(ix, sp.Nx, sp.dx, wl[gq / sp.Nq], qv[2 * (gq % sp.Nq)]);
	keep[t] = fabs(q0) < sp.NA;
}

// The y half of the screen filter in one pass, after the row transforms: forward transform of `nc` columns of both
// components of a slot, transfer matrices, backward transform. Column groups outside the aperture are left
// alone; the backward row transforms take them as zero.
// Bound: FP64 pipe (FP64), HBM and shared memory (FP32). In place of the column transforms, the filter
// pass and the column transforms back (5 reads and writes of the fields, about a third of whose columns are inside
// the aperture at spacings of half a wavelength): 256x256, 832 planes FP32 3.7 ms in three launches, 1.24 ms here;
// 156 planes FP64 2.8 and 0.78 ms.
template <typename R>
__global__ void __launch_bounds__(512) k_screen_cols(cx<R>* F, ScreenParams sp, FftPlan1D P, int nc, const cx<R>* __restrict__ tw,
		const double* __restrict__ wl, const double* __restrict__ nout, const double* __restrict__ qv,
		const unsigned char* __restrict__ keep) {
	extern __shared__ unsigned char smem_raw[];
	cx<R>* sA = reinterpret_cast<cx<R>*>(smem_raw);
	const int Nx = sp.Nx, n = P.n, pitch = n + 1;
	const size_t N = (size_t)Nx * n;
	cx<R>* sB = sA + (size_t)2 * nc * pitch;
	cx<R>* wp = sB + (size_t)2 * nc * pitch;
	double* sq = reinterpret_cast<double*>(wp + P.pmax + (P.pmax & 1));  // [n] q1 of the modes, [nc] q0 of the columns
	// blocks: the column groups of a slot, then the slots (more of them than a grid's y may hold)
	const int ncg = (Nx + nc - 1) / nc, slot = blockIdx.x / ncg, x0 = (blockIdx.x - slot * ncg) * nc, m = min(nc, Nx - x0), gq = slot / 2;
	const unsigned char* kp = keep + (size_t)gq * Nx + x0;
	bool any = false;
	for(int i = 0; i < m; i++) any |= kp[i] != 0;
	if(!any) return;
	const int g = gq / sp.Nq, q = gq % sp.Nq;
	const double la = wl[g], qx = qv[2 * q], qy = qv[2 * q + 1];
	for(int e = threadIdx.x; e < n + m; e += blockDim.x)
		sq[e] = e < n ? screen_q(e, n, sp.dy, la, qy) : screen_q(x0 + e - n, Nx, sp.dx, la, qx);
	cx<R>* f = F + (size_t)slot * 2 * N + x0;
	// lines: component c of column i at c * nc + i
	for(int e = threadIdx.x; e < 2 * n * nc; e += blockDim.x) {
		const int i = e % nc, r = e / nc, c = r >= n, y = r - c * n;
		if(i < m) sA[(c * nc + i) * pitch + y] = f[c * N + (size_t)y * Nx + i];
	}
	__syncthreads();
	cx<R>* s = fft_stages<R>(sA, sB, P, 2 * nc, tw, -1, wp);
	for(int e = threadIdx.x; e < n * nc; e += blockDim.x) {
		const int i = e / n, y = e - i * n;
		if(i < m) {
			cx<R> M[2][2];
			screen_matrix<R>(sp, sq[n + i], sq[y], la, nout[g], qx, qy, M);
			cx<R>&u = s[i * pitch + y], &v = s[(nc + i) * pitch + y];
			const cx<R> a = u, b = v;
			u = M[0][0] * a + M[0][1] * b;
			v = M[1][0] * a + M[1][1] * b;
		}
	}
	__syncthreads();
	s = fft_stages<R>(s, s == sA ? sB : sA, P, 2 * nc, tw, +1, wp);
	for(int e = threadIdx.x; e < 2 * n * nc; e += blockDim.x) {
		const int i = e % nc, r = e / nc, c = r >= n, y = r - c * n;
		if(i < m) f[c * N + (size_t)y * Nx + i] = s[(c * nc + i) * pitch + y];
	}
}

}  // namespace nbpm
