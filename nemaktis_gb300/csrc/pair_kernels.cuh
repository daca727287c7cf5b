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
__device__ __forceinline__ pr at_byte(const pr* f, unsigned o) {
	return *reinterpret_cast<const pr*>(reinterpret_cast<const char*>(f) + o);
}

// Right-hand side of x-lines (composite_m with KIND ST_EXPL_Y or ST_WOOD_X) of one component at point
// (x, iy), x < Nx - 1, for a pair; f0, f1: the pair's component planes. The row offsets are bytes.
template <int KIND>
struct PairRhs {
	const cx<float>* C;
	const pr *f0, *f1;
	int Nx, Ny, iy, yy, comp;
	bool both;
	unsigned r0, rm, rp, ro;  // rows of the point, of its y neighbours, and iy itself
	__device__ __forceinline__ PairRhs(const cx<float>* C_, const pr* f, const Geom& G, int comp_, int iy_) : C(C_), f0(f), f1(f + G.N),
			Nx(G.Nx), Ny(G.Ny), iy(iy_), comp(comp_) {
		constexpr bool XDIR = KIND == ST_WOOD_X;
		const bool mixed = XDIR ? comp == 0 : comp == 1;
		both = mixed && Nx > 3 && Ny > 3;
		yy = (!XDIR || both) && iy == Ny - 1 ? 0 : iy;
		const unsigned w = (unsigned)Nx * (unsigned)sizeof(pr);
		ro = (unsigned)iy * w;
		r0 = (unsigned)yy * w;
		rm = yy == 0 ? (unsigned)max(Ny - 2, 0) * w : r0 - w;
		rp = yy == Ny - 2 ? 0u : r0 + w;
	}
	__device__ __forceinline__ pr operator()(int x) const {
		constexpr unsigned SZ = sizeof(pr);
		const unsigned o = (unsigned)x * SZ;
		const unsigned om = x == 0 ? (unsigned)(Nx - 2) * SZ : o - SZ, op = x == Nx - 2 ? 0u : o + SZ;
		const int p = x + Nx * yy;
		pr out{0, 0, 0, 0};
		auto corners = [&](v4<float> v, const pr* f) {
			out = pifma(v.w, at_byte(f, rm + om), pifma(v.z, at_byte(f, rm + op), pifma(v.y, at_byte(f, rp + om),
				pifma(v.x, at_byte(f, rp + op), out))));
		};
		if(KIND == ST_WOOD_X) {
			auto taps = [&](v4<float> v, float c, const pr* f) {
				out = pfma(mk(v.z, v.w), at_byte(f, r0 + op), pifma(c, at_byte(f, r0 + o), pfma(mk(v.x, v.y), at_byte(f, r0 + om), out)));
			};
			if(comp == 0) {
				taps(coef_v(C, V_DX + 1, p), coef_u(C, U_DX, p).y, f1);
				if(both) { corners(coef_v(C, V_DD + 0, p), f0); corners(coef_v(C, V_DD + 1, p), f1); }
			}
			else taps(coef_v(C, V_DX + 2, p), coef_v(C, V_DX + 3, p).w, f0);
			return out;
		}
		if(Ny > 3) {
			auto taps = [&](v4<float> v, float c, const pr* f) {
				out = pfma(mk(v.z, v.w), at_byte(f, rp + o), pifma(c, at_byte(f, r0 + o), pfma(mk(v.x, v.y), at_byte(f, rm + o), out)));
			};
			if(comp == 0) {
				const v4<float> w = coef_v(C, V_DY + 3, p);
				out = pifma(w.y, at_byte(f0, rp + o), pifma(w.z, at_byte(f0, r0 + o), pifma(w.x, at_byte(f0, rm + o), out)));
				taps(coef_v(C, V_DY + 2, p), w.w, f1);
			}
			else {
				const cx<float> u = coef_u(C, U_DY, p);
				taps(coef_v(C, V_DY + 0, p), u.x, f1);
				taps(coef_v(C, V_DY + 1, p), u.y, f0);
				if(both) { corners(coef_v(C, V_DD + 3, p), f1); corners(coef_v(C, V_DD + 2, p), f0); }
			}
		}
		return padd(out, at_byte(comp == 0 ? f0 : f1, ro + o));
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
__device__ __forceinline__ void pair_backward(pr* vb, const cx<float>* Fc, int CH, int ci, pr h, pr x) {
#pragma unroll
	for(int k = M - 1; k >= 0; k--) {
		const v4<float> rc = part_rc(Fc, k, CH, ci);
		const cx<float> e = part_e(Fc, k, CH, ci);
		x = pfma(mk(rc.z, rc.w), x, pfma(e, h, pmul(mk(rc.x, rc.y), vb[k])));
		vb[k] = x;
	}
}

// Partitioned x-line solve with its right-hand side (k_solve_xc) for a pair of slots: a warp per line, 4
// lines per block; the blocks of a line group, both components and all pairs of the wavelength follow each
// other, so that they find its coefficients and factors in L2.
// Bound: L1 wavefronts (70 %) and load latency. 7 blocks per SM: at 8 the 64 registers spill (206 against
// 195 ms for the whole step), at 6 too few warps wait for loads (205 ms). 256x256, 16 wavelengths, 13 q: Woodbury
// solves 477 us as k_solve_xc with two slots per thread, 402 us here; explicit step 491 and 378 us. The rows of
// a block staged in shared memory (cp.async) gave 438 and 415 us, x neighbours from lane shuffles 478 and
// 498 us.
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
	if(iy < Ny) {
		const cx<float>* Fc = fac + ((size_t)g * 2 + c) * NFAC * plane + (size_t)iy * part_line_size(M, 32);
		const int K = (int)lsc[(((size_t)g * 2 + c) * Ny + iy) * 2].x;
		pr* buf = bufs + warp * WS;
		const PairRhs<KIND> rhs(coef + (size_t)g * coef_set_size(N), f, G, c, iy);
#pragma unroll 1
		for(int t = 0; t < M; t++) {
			const int e = lane + 32 * t;
			buf[e / M * PM + e % M] = e < n ? rhs(e) : pr{0, 0, 0, 0};  // chunk e / M
		}
		__syncwarp();
		if(K >= 0) {
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
			h = pshfl(h, left);
			pair_backward<M>(vb, Fc, 32, lane, h, x);
		}
		else if(lane == 0) part_solve_seq<float, M, 2, 2>(reinterpret_cast<cx<float>*>(buf), 1, Fc, 32, n);
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
// 1024x1024, 2 wavelengths, 7 q: Woodbury solves 1007 us as k_solve_xw, 508 us here (a line's coefficients and
// factors, 190 MB per wavelength, were read again from DRAM for every two slots), explicit step 810 and 503 us.
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
	const int K = live ? (int)lsc[(((size_t)g * 2 + c) * Ny + iy) * 2].x : 0;
	pr* buf = bufs + ln * WS;
	if(live) {
		const PairRhs<KIND> rhs(coef + (size_t)g * coef_set_size(N), f, G, c, iy);
#pragma unroll 1
		for(int t = 0; t < M; t++) {
			const int e = ci + CH * t;
			buf[e / M * PM + e % M] = e < n ? rhs(e) : pr{0, 0, 0, 0};
		}
	}
	// the barriers are the block's: both lines take the larger number of steps
	__shared__ int sK;
	if(threadIdx.x == 0) sK = 0;
	__syncthreads();
	if(ci == 0 && K > 0) atomicMax(&sK, K);
	pr d, yf;
	const bool part = live && K >= 0;
	pr* vb = buf + ci * PM;
	if(part) pair_forward<M>(vb, Fc, CH, ci, d, yf);
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
	if(part) {
		h = pfma(If[I_HY * CH], yn, pmul(If[I_HD * CH], d));
		x = pfma(If[I_GY * CH], yn, pmul(If[I_GD * CH], d));
	}
	const pr bh = h, bg = x;
#pragma unroll 1
	for(int it = 0;; it++) {
		// two buffers in turn: the one written here was last read two barriers ago
		pr* H = sH + (it & 1) * (W + 1);
		pr* Gn = sG + ((it + 1) & 1) * W;
		if(lane == 31) H[warp] = h;
		if(ci == last) H[W] = h;
		if(lane == 0) Gn[warp] = x;
		__syncthreads();
		const pr up = pshfl(h, (lane + 31) & 31);
		hl = lane > 0 ? up : H[warp > 0 ? warp - 1 : W];
		if(it >= Kb) break;
		const pr gr = next(x, Gn);
		if(part) {
			const cx<float> ph = If[I_PH * CH], pg = If[I_PG * CH], qh = If[I_QH * CH], qg = If[I_QG * CH];
			h = pfma(qh, gr, pfma(ph, hl, bh));
			x = pfma(qg, gr, pfma(pg, hl, bg));
		}
	}
	if(part) pair_backward<M>(vb, Fc, CH, ci, hl, x);
	else if(live && ci == 0) part_solve_seq<float, M, 2, 2>(reinterpret_cast<cx<float>*>(buf), 1, Fc, CH, n);
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
