// FP32 propagation kernels on pairs of slots: the two polarisations of a (wavelength, q), which every
// sample has, side by side. Between the transition and the last y solve of a slab the fields are kept as
//   F2[pair][comp][iy][ix] = {slot 2*pair, slot 2*pair + 1}    (16 bytes, pair = q + Nq*lambda)
// so that one 16-byte access brings a point of both slots: half the loads and address arithmetic per
// value, unaligned neighbour accesses that touch 5 instead of 2 x 3 lines, conflict-free 16-byte
// accesses to shared memory. The transition reads the plain planes and writes pairs, the last y solve
// writes plain planes again, both at no extra pass. Same operators, same order of operations per slot as the
// general kernels of bpm_kernels.cuh.
#pragma once

#include "bpm_kernels.cuh"

namespace nbpm {

typedef v4<float> pr;  // {re, im} of the first slot, {re, im} of the second one

__device__ __forceinline__ cx<float> lo(pr a) { return mk(a.x, a.y); }
__device__ __forceinline__ cx<float> hi(pr a) { return mk(a.z, a.w); }
__device__ __forceinline__ pr join(cx<float> a, cx<float> b) { return pr{a.x, a.y, b.x, b.y}; }
// c + a * b for both slots, a complex (pfma), a = i*s imaginary (pifma)
__device__ __forceinline__ pr pfma(cx<float> a, pr b, pr c) { return join(cfma(a, lo(b), lo(c)), cfma(a, hi(b), hi(c))); }
__device__ __forceinline__ pr pifma(float s, pr b, pr c) { return join(ifma(s, lo(b), lo(c)), ifma(s, hi(b), hi(c))); }
__device__ __forceinline__ pr pmul(cx<float> a, pr b) { return join(a * lo(b), a * hi(b)); }
__device__ __forceinline__ pr padd(pr a, pr b) { return pr{a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w}; }
__device__ __forceinline__ pr pshfl(pr v, int l) {
	return pr{__shfl_sync(0xffffffffu, v.x, l), __shfl_sync(0xffffffffu, v.y, l), __shfl_sync(0xffffffffu, v.z, l),
		__shfl_sync(0xffffffffu, v.w, l)};
}
// for ring_solve
__device__ __forceinline__ pr vfma(cx<float> a, pr b, pr c) { return pfma(a, b, c); }
__device__ __forceinline__ pr vshfl(pr v, int l) { return pshfl(v, l); }
__device__ __forceinline__ pr at_byte(const pr* f, unsigned o) {
	return *reinterpret_cast<const pr*>(reinterpret_cast<const char*>(f) + o);
}

// Right-hand sides of x-lines (composite_m with KIND ST_EXPL_Y or ST_WOOD_X) of one component for a pair, at
// column x < Nx - 1 of the L lines iy0, iy0 + 1, ... (pairs have Nx, Ny > 3); f0, f1: the pair's component planes. A
// field row is loaded once and used by the up to three lines it touches: 4 lines with corners take 24 instead of 32
// corner loads, and 6 instead of 12 in the column itself. Each case is straight-line code, so that the loads of later
// rows are issued before the first are used: with the component and the corners as branches inside the row loop the
// explicit step at 256x256 took 508 us, 324 us without. Coefficients come by halves, as a row needs them: whole
// vectors held for three rows spilled (explicit step 515 us). Rows of lines past Ny - 1 are held inside the
// plane; their results are not used. The row offsets are bytes.
template <int KIND, int L>
struct StripRhs {
	const cx<float>* C;
	const pr *f0, *f1;
	int Nx, Ny, iy0, comp;
	__device__ __forceinline__ StripRhs(const cx<float>* C_, const pr* f, const Geom& G, int comp_, int iy0_) : C(C_), f0(f), f1(f + G.N),
			Nx(G.Nx), Ny(G.Ny), iy0(iy0_), comp(comp_) {}
	// row iy0 - 1 + k on the periodic lines 0 .. Ny - 2
	__device__ __forceinline__ int row(int k) const {
		const int P = Ny - 1, r = iy0 - 1 + k;
		return r < 0 ? r + P : r < P ? r : min(r - P, P);
	}
	// the two corners of a row
	static __device__ __forceinline__ pr corners(cx<float> v, pr m, pr p, pr c) { return pifma(v.y, m, pifma(v.x, p, c)); }
	__device__ __forceinline__ void operator()(int x, pr (&out)[L]) const {
		constexpr unsigned SZ = sizeof(pr);
		const unsigned o = (unsigned)x * SZ, w = (unsigned)Nx * SZ;
		const unsigned om = x == 0 ? (unsigned)(Nx - 2) * SZ : o - SZ, op = x == Nx - 2 ? 0u : o + SZ;
#pragma unroll
		for(int l = 0; l < L; l++) out[l] = pr{0, 0, 0, 0};
		if(KIND == ST_WOOD_X) {
			if(comp == 0) wood0(x, o, om, op, w, out);
			else wood1(x, o, om, op, w, out);
		}
		else if(comp == 0) expl<0>(x, o, om, op, w, out);
		else expl<1>(x, o, om, op, w, out);
	}
	__device__ __forceinline__ void wood0(int x, unsigned o, unsigned om, unsigned op, unsigned w, pr (&out)[L]) const {
#pragma unroll
		for(int k = 0; k < L + 2; k++) {
			const int yr = row(k), q = x + Nx * yr;
			const unsigned r = (unsigned)yr * w;
			const pr am = at_byte(f0, r + om), ap = at_byte(f0, r + op), bm = at_byte(f1, r + om), bp = at_byte(f1, r + op);
			if(k >= 2) {
				const int qp = x + Nx * row(k - 1);
				out[k - 2] = corners(coef_h(C, V_DD + 0, 0, qp), am, ap, corners(coef_h(C, V_DD + 1, 0, qp), bm, bp, out[k - 2]));
			}
			if(k >= 1 && k <= L) {
				const v4<float> v = coef_v(C, V_DX + 1, q);
				pr& t = out[k - 1];
				t = pfma(mk(v.z, v.w), bp, pifma(coef_u(C, U_DX, q).y, at_byte(f1, r + o), pfma(mk(v.x, v.y), bm, t)));
			}
			if(k < L) {
				const int qn = x + Nx * row(k + 1);
				out[k] = corners(coef_h(C, V_DD + 0, 1, qn), am, ap, corners(coef_h(C, V_DD + 1, 1, qn), bm, bp, out[k]));
			}
		}
	}
	__device__ __forceinline__ void wood1(int x, unsigned o, unsigned om, unsigned op, unsigned w, pr (&out)[L]) const {
#pragma unroll
		for(int l = 0; l < L; l++) {
			const int yy = min(iy0 + l, Ny - 1), q = x + Nx * yy;
			const unsigned r = (unsigned)yy * w;
			const v4<float> v = coef_v(C, V_DX + 2, q);
			out[l] = pfma(mk(v.z, v.w), at_byte(f0, r + op), pifma(coef_h(C, V_DX + 3, 1, q).y, at_byte(f0, r + o),
				pmul(mk(v.x, v.y), at_byte(f0, r + om))));
		}
	}
	template <int COMP>
	__device__ __forceinline__ void expl(int x, unsigned o, unsigned om, unsigned op, unsigned w, pr (&out)[L]) const {
		const pr *fa = COMP == 0 ? f0 : f1, *fb = COMP == 0 ? f1 : f0;  // this component, the other one
		pr own[L];
#pragma unroll
		for(int k = 0; k < L + 2; k++) {
			const unsigned r = (unsigned)row(k) * w;
			const pr a = at_byte(fa, r + o), b = at_byte(fb, r + o);
			pr am, ap, bm, bp;
			if(COMP == 1) {
				am = at_byte(fa, r + om);
				ap = at_byte(fa, r + op);
				bm = at_byte(fb, r + om);
				bp = at_byte(fb, r + op);
			}
			if(k >= 2) {
				const int q = x + Nx * row(k - 1);
				pr& t = out[k - 2];
				if(COMP == 0) t = pfma(coef_h(C, V_DY + 2, 1, q), b, pifma(coef_h(C, V_DY + 3, 0, q).y, a, t));
				else t = pfma(coef_h(C, V_DY + 1, 1, q), b, pfma(coef_h(C, V_DY + 0, 1, q), a, t));
				if(COMP == 1) t = corners(coef_h(C, V_DD + 2, 0, q), bm, bp, corners(coef_h(C, V_DD + 3, 0, q), am, ap, t));
				t = padd(t, own[k - 2]);
			}
			if(k >= 1 && k <= L) {
				const int q = x + Nx * row(k);
				const cx<float> u = COMP == 0 ? coef_h(C, V_DY + 3, 1, q) : coef_u(C, U_DY, q);
				out[k - 1] = pifma(u.y, b, pifma(u.x, a, out[k - 1]));
				own[k - 1] = iy0 + k - 1 == Ny - 1 ? at_byte(fa, (unsigned)(Ny - 1) * w + o) : a;
			}
			if(k < L) {
				const int q = x + Nx * row(k + 1);
				pr& t = out[k];
				if(COMP == 0) t = pfma(coef_h(C, V_DY + 2, 0, q), b, pifma(coef_h(C, V_DY + 3, 0, q).x, a, t));
				else t = pfma(coef_h(C, V_DY + 1, 0, q), b, pfma(coef_h(C, V_DY + 0, 0, q), a, t));
				if(COMP == 1) t = corners(coef_h(C, V_DD + 2, 1, q), bm, bp, corners(coef_h(C, V_DD + 3, 1, q), am, ap, t));
			}
		}
	}
};

// Where a pair solve writes: pairs in its own frame, pairs in the transposed frame with the components
// exchanged, or the two slots' plain planes in the transposed frame with the components exchanged. With t0 the
// explicit solve and S the Woodbury solve the direction's result t0 + S t0 + S S t0 is formed as t0 + S (t0 + S t0):
// the first Woodbury solve adds its source (PO_SAME), the second one adds t0 (acc0).
enum { PO_SAME = 0, PO_TRANS = 1, PO_PLAIN = 2 };

// The chunk sweeps of one thread (chunk ci of CH) on shared pairs vb, as in k_solve_xc.
template <int M>
__device__ __forceinline__ void pair_forward(pr* vb, const cx<float>* Fc, int CH, int ci, pr& d, pr& yf) {
#pragma unroll
	for(int k = 0; k < M; k++) {
		const v4<float> az = part_az(Fc, k, CH, ci);
		if(k == 0) {
			d = vb[0];
			yf = pmul(mk(az.z, az.w), d);
		}
		else {
			d = pfma(mk(az.x, az.y), d, vb[k]);
			vb[k] = d;
			yf = pfma(mk(az.z, az.w), d, yf);
		}
	}
}
template <int M>
__device__ __forceinline__ void pair_backward(pr* vb, const cx<float>* Fc, int CH, int ci, float base, pr h, pr x) {
#pragma unroll
	for(int k = M - 1; k >= 0; k--) {
		const v4<float> rc = part_rc(Fc, k, CH, ci);
		const cx<float> e = part_e(Fc, k, CH, ci);
		x = pfma(mk(rc.z, rc.w), x, pfma(e, h, pfma(mk(rc.x, rc.y), vb[k], pr{base * vb[k].x, base * vb[k].y, base * vb[k].z, base * vb[k].w})));
		vb[k] = x;
	}
}

// Partitioned x-line solve with its right-hand side (k_solve_xc) for a pair of slots: a warp per line, 4
// lines per block; the blocks of a line group, both components and all pairs of the wavelength follow each
// other, so that they find its coefficients and factors in L2.
// Bound: L1 wavefronts and load latency. 7 blocks per SM: at 8 the 64 registers spill (206 against 195 ms
// for the whole step), at 6 too few warps wait for loads (205 ms). Right-hand sides: a thread takes a column of
// the block's 4 lines (StripRhs), for short lines (M < 6) a point of one line, where a column per thread leaves warps
// without work (64x64: explicit step 16.6 us, with 2 lines per thread 18.3 us, with 4 lines 22.6 us; 224x224: 55.0
// us with 1 or 2 lines, 50.7 us with 4). 256x256, 16 wavelengths, 13 q: Woodbury solves 477 us as k_solve_xc with
// two slots per thread, 402 us here with a line per warp for the right-hand sides too, 332 us with strips;
// explicit step 491, 378 and 330 us. The rows of a block staged in shared memory (cp.async) gave 438 and
// 415 us, x neighbours from lane shuffles 478 and 498 us.
template <int M, int KIND, int OUT>
__global__ void __launch_bounds__(128, 7) k_solve_xp(Geom G, const cx<float>* __restrict__ coef,
		const cx<float>* __restrict__ fac, size_t plane, const cx<double>* __restrict__ lsc, const pr* __restrict__ src,
		pr* __restrict__ dst, const pr* __restrict__ acc0, cx<float>* __restrict__ plain) {
	extern __shared__ unsigned char smem_raw[];
	wait_predecessor();
	constexpr int LT = 4;
	// 16-byte entries per warp; the warps' buffers 2 entries apart modulo 8: no bank conflicts when the
	// block reads one point of its 4 lines
	constexpr int PM = part_pitch(M), WS = 32 * PM + 2;
	pr* const bufs = reinterpret_cast<pr*>(smem_raw);
	const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
	const int Nx = G.Nx, Ny = G.Ny, N = G.N, nch = G.Nq;
	const int ch = blockIdx.x % nch, c = blockIdx.x / nch % 2, line0 = blockIdx.x / nch / 2 * LT, g = blockIdx.y;
	const int iy = line0 + warp;
	const int n = Nx - 1;
	const size_t pair = (size_t)g * nch + ch;
	const pr* f = src + pair * 2 * N;
	{
		constexpr int L = M >= 6 ? 4 : 1, COLS = 128 * L / LT;
		const int l0 = threadIdx.x / COLS * L;
		const StripRhs<KIND, L> rhs(coef + (size_t)g * coef_set_size(N), f, G, c, line0 + l0);
		if(line0 + l0 < Ny) {
#pragma unroll 1
			for(int e = threadIdx.x % COLS; e < 32 * M; e += COLS) {
				pr v[L];
				if(e < n) rhs(e, v);
#pragma unroll
				for(int l = 0; l < L; l++) bufs[(l0 + l) * WS + e / M * PM + e % M] = e < n ? v[l] : pr{0, 0, 0, 0};  // chunk e / M
			}
		}
		__syncthreads();
	}
	if(iy < Ny) {
		const cx<float>* Fc = fac + ((size_t)g * 2 + c) * NFAC * plane + (size_t)iy * part_line_size(M, 32);
		const cx<double> kb = lsc[(((size_t)g * 2 + c) * Ny + iy) * 2];
		const int K = (int)kb.x;
		const float base = (float)kb.y;
		pr* buf = bufs + warp * WS;
		{
			pr* vb = buf + lane * PM;
			pr d, yf;
			pair_forward<M>(vb, Fc, 32, lane, d, yf);
			const int last = (n - 1) / M;
			const int left = lane == 0 ? last : lane - 1, right = lane == last ? 0 : (lane + 1) & 31;
			const cx<float>* If = Fc + (size_t)M * NFAC * 32 + lane;
			const pr yn = pshfl(yf, right);
			pr h = pfma(If[I_HY * 32], yn, pmul(If[I_HD * 32], d)), x = pfma(If[I_GY * 32], yn, pmul(If[I_GD * 32], d));
			if(K > 0) {
				const cx<float> ph = If[I_PH * 32], pg = If[I_PG * 32], qh = If[I_QH * 32], qg = If[I_QG * 32];
				const pr bh = h, bg = x;
#pragma unroll 1
				for(int k = 0; k < K; k++) {
					const pr hl = pshfl(h, left), gr = pshfl(x, right);
					h = pfma(qh, gr, pfma(ph, hl, bh));
					x = pfma(qg, gr, pfma(pg, hl, bg));
				}
			}
			if(K >= 0) h = pshfl(h, left);
			else {
				const Border<pr, 1> b = part_ring<false, 1, float>(LineThreads{1, 0, 0, lane, lane, last}, If, 32, Border<pr, 1>{{h}, {x}}, (pr*)nullptr);
				h = b.h[0];
				x = b.x[0];
			}
			pair_backward<M>(vb, Fc, 32, lane, base, h, x);
		}
		__syncwarp();
		// out, or for the transposed outputs the sums into the buffer, where the added field comes with
		// aligned loads (point n repeats point 0; its entry is free or padding)
		const pr first = buf[0];
		__syncwarp();
		const pr* add = (OUT == PO_SAME ? f : acc0 + pair * 2 * N) + (size_t)c * N + (size_t)iy * Nx;
		pr* o = dst + (pair * 2 + c) * N + (size_t)iy * Nx;
		constexpr int U = 4;
#pragma unroll 1
		for(int t0 = 0; t0 <= M; t0 += U) {
			pr a[U];
			if(KIND == ST_WOOD_X) {
#pragma unroll
				for(int u = 0; u < U; u++) {
					const int e = lane + 32 * (t0 + u);
					if(t0 + u <= M && e < Nx) a[u] = add[e];
				}
			}
#pragma unroll
			for(int u = 0; u < U; u++) {
				const int e = lane + 32 * (t0 + u);
				if(t0 + u <= M && e < Nx) {
					pr x = e == n ? first : buf[e / M * PM + e % M];
					if(KIND == ST_WOOD_X) x = padd(a[u], x);
					if(OUT == PO_SAME) o[e] = x;
					else buf[e / M * PM + e % M] = x;
				}
			}
		}
	}
	if(OUT != PO_SAME) {
		__syncthreads();
		// consecutive threads take the 4 lines of a point: one 64-byte segment of the transposed plane
		const int w = threadIdx.x % LT;
		const pr* b = bufs + w * WS;
		if(w < Ny - line0) {
#pragma unroll 4
			for(int e = threadIdx.x / LT; e < Nx; e += 128 / LT) {
				const pr x = b[e / M * PM + e % M];
				const size_t q = (size_t)e * Ny + line0 + w;
				if(OUT == PO_TRANS) dst[(pair * 2 + (1 - c)) * N + q] = x;
				else {
					plain[(pair * 4 + (1 - c)) * N + q] = lo(x);
					plain[(pair * 4 + 2 + (1 - c)) * N + q] = hi(x);
				}
			}
		}
	}
}

// The same for long lines: W warps per line and 2 lines per block (32-byte segments of the transposed plane), 32*W
// chunks of M points, border unknowns of chunks in different warps through shared memory as in k_solve_xw.
// REGS: registers per thread, by the launch (launch_solve_pair).
// 1024x1024, 2 wavelengths, 7 q: Woodbury solves 1007 us as k_solve_xw (a line's coefficients and factors, 190 MB
// per wavelength, were read again from DRAM for every two slots), 508 us here, 462 us with the right-hand
// sides of both lines from one thread (StripRhs); explicit step 810, 503 and 425 us. 4 lines per block: 461 and 491
// us; 512x512, 14 pairs: 14.4 ms a step with 2 lines, 16.2 ms with 4.
template <int M, int KIND, int OUT, int REGS>
__global__ void __maxnreg__(REGS) k_solve_xwp(Geom G, int W, const cx<float>* __restrict__ coef,
		const cx<float>* __restrict__ fac, size_t plane, const cx<double>* __restrict__ lsc, const pr* __restrict__ src,
		pr* __restrict__ dst, const pr* __restrict__ acc0, cx<float>* __restrict__ plain) {
	extern __shared__ unsigned char smem_raw[];
	wait_predecessor();
	constexpr int LT = 2;
	constexpr int PM = part_pitch(M);
	const int CH = 32 * W, WS = CH * PM + 4;  // the two lines' buffers 4 entries apart modulo 8
	pr* const bufs = reinterpret_cast<pr*>(smem_raw);
	const int ln = threadIdx.x / CH, ci = threadIdx.x % CH, warp = ci / 32, lane = ci % 32;
	pr* sG = bufs + LT * WS + ln * (4 * W + 2);  // [2][W]: g (first yf) of the warps' first chunks
	pr* sH = sG + 2 * W;                         // [2][W + 1]: h of the warps' last chunks, then of the line's
	const int Nx = G.Nx, Ny = G.Ny, N = G.N, nch = G.Nq;
	const int ch = blockIdx.x % nch, c = blockIdx.x / nch % 2, lb = blockIdx.x / nch / 2, g = blockIdx.y;
	const int iy = lb * LT + ln;
	const bool live = iy < Ny;
	const int n = Nx - 1;
	const size_t pair = (size_t)g * nch + ch;
	const pr* f = src + pair * 2 * N;
	const cx<float>* Fc = fac + ((size_t)g * 2 + c) * NFAC * plane + (size_t)iy * part_line_size(M, CH);
	const cx<double> kb = live ? lsc[(((size_t)g * 2 + c) * Ny + iy) * 2] : mk(0., 0.);
	const int K = (int)kb.x;
	const float base = (float)kb.y;
	pr* buf = bufs + ln * WS;
	{
		const StripRhs<KIND, LT> rhs(coef + (size_t)g * coef_set_size(N), f, G, c, lb * LT);
#pragma unroll 1
		for(int e = threadIdx.x; e < M * CH; e += LT * CH) {
			pr v[LT];
			if(e < n) rhs(e, v);
#pragma unroll
			for(int l = 0; l < LT; l++) bufs[l * WS + e / M * PM + e % M] = e < n ? v[l] : pr{0, 0, 0, 0};
		}
	}
	// the barriers are the block's: both lines take the larger number of steps
	__shared__ int sK;
	if(threadIdx.x == 0) sK = 0;
	__syncthreads();
	if(ci == 0 && K > 0) atomicMax(&sK, K);
	pr d, yf;
	pr* vb = buf + ci * PM;
	if(live) pair_forward<M>(vb, Fc, CH, ci, d, yf);
	else d = yf = pr{0, 0, 0, 0};
	const int last = (n - 1) / M;
	const bool edge_r = lane == 31 || ci == last;
	const int wr = ci == last ? 0 : (warp + 1) % W;
	auto next = [&](pr v, const pr* s) {
		const pr m = pshfl(v, (lane + 1) & 31);
		return edge_r ? s[wr] : m;
	};
	if(lane == 0) sG[warp] = yf;
	__syncthreads();
	const int Kb = sK;
	const cx<float>* If = Fc + (size_t)M * NFAC * CH + ci;
	const pr yn = next(yf, sG);
	pr h{0, 0, 0, 0}, x{0, 0, 0, 0}, hl;
	if(live) {
		h = pfma(If[I_HY * CH], yn, pmul(If[I_HD * CH], d));
		x = pfma(If[I_GY * CH], yn, pmul(If[I_GD * CH], d));
	}
	// a line without Jacobi steps is joined by its own threads, at a barrier of theirs; it only waits in the loop below
	const bool part = live && K >= 0;
	if(live && K < 0) {
		const Border<pr, 1> b = part_ring<true, 1, float>(LineThreads{W, 1 + ln, warp, lane, ci, last}, If, CH, Border<pr, 1>{{h}, {x}}, sG);
		hl = b.h[0];
		x = b.x[0];
	}
	const pr bh = h, bg = x;
#pragma unroll 1
	for(int it = 0;; it++) {
		// two buffers in turn: the one written here was last read two barriers ago
		pr* H = sH + (it & 1) * (W + 1);
		pr* Gn = sG + ((it + 1) & 1) * W;
		if(part) {
			if(lane == 31) H[warp] = h;
			if(ci == last) H[W] = h;
			if(lane == 0) Gn[warp] = x;
		}
		__syncthreads();
		const pr up = pshfl(h, (lane + 31) & 31);
		if(part) hl = lane > 0 ? up : H[warp > 0 ? warp - 1 : W];
		if(it >= Kb) break;
		const pr gr = next(x, Gn);
		if(part) {
			const cx<float> ph = If[I_PH * CH], pg = If[I_PG * CH], qh = If[I_QH * CH], qg = If[I_QG * CH];
			h = pfma(qh, gr, pfma(ph, hl, bh));
			x = pfma(qg, gr, pfma(pg, hl, bg));
		}
	}
	if(live) pair_backward<M>(vb, Fc, CH, ci, base, hl, x);
	__syncthreads();
	if(OUT == PO_SAME) {
		if(!live) return;
		pr* o = dst + (pair * 2 + c) * N + (size_t)iy * Nx;
		const pr* own = f + (size_t)c * N + (size_t)iy * Nx;
#pragma unroll 4
		for(int e = ci; e < Nx; e += CH) {
			const int ee = e == n ? 0 : e;
			const pr x = buf[ee / M * PM + ee % M];
			o[e] = KIND == ST_WOOD_X ? padd(own[e], x) : x;
		}
	}
	else {
		const int line0 = lb * LT, nl = min(LT, Ny - line0);
		const pr* a0 = acc0 + (pair * 2 + c) * N + (size_t)line0 * Nx;
		const int w = threadIdx.x % LT;
		constexpr int U = 4;
		const int BE = CH;  // points per round: LT * CH threads
#pragma unroll 1
		for(int e0 = threadIdx.x / LT; e0 < Nx; e0 += U * BE) {
			pr a[U];
#pragma unroll
			for(int u = 0; u < U; u++) {
				const int e = e0 + u * BE;
				if(e < Nx && w < nl) a[u] = a0[w * Nx + e];
			}
#pragma unroll
			for(int u = 0; u < U; u++) {
				const int e = e0 + u * BE;
				if(e < Nx && w < nl) {
					const int ee = e == n ? 0 : e;
					const pr v = padd(a[u], bufs[w * WS + ee / M * PM + ee % M]);
					const size_t q = (size_t)e * Ny + line0 + w;
					if(OUT == PO_TRANS) dst[(pair * 2 + (1 - c)) * N + q] = v;
					else {
						plain[(pair * 4 + (1 - c)) * N + q] = lo(v);
						plain[(pair * 4 + 2 + (1 - c)) * N + q] = hi(v);
					}
				}
			}
		}
	}
}

}  // namespace nbpm
