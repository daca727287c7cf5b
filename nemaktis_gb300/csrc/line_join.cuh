// Joining the chunks of a periodic line through their border unknowns, exactly. A line is cut into m chunks that
// are solved by themselves; node t of a closed chain stands between chunk t and the next one, with h_t the
// last unknown of chunk t and g_t the first one of chunk t + 1:
//   h_t = bh_t + ph_t h_{t-1} + qh_t g_{t+1},   g_t = bg_t + pg_t h_{t-1} + qg_t g_{t+1}   (t modulo m).
// Weakly coupled lines take a few Jacobi steps (the kernels themselves do them). For the others the chain is
// eliminated from node 0 on, with H = h_{m-1} and G = g_0 carried along:
//   h_t = alpha_t + rho_t g_{t+1} + eta_t H,   g_t = gamma_t + kappa_t H + tau_t G.
// rho is a Moebius recurrence and alpha, gamma, eta, kappa, tau are affine ones, so that every one is a scan over
// the threads of the line, one node per thread; rho, eta, kappa, tau and the closing 2x2 system do not
// depend on the right-hand side (ring_factor), and a solve is one scan forward and one backward (ring_solve).
// Threads past the line's last chunk take part with neutral maps.
#pragma once

#include "cplx.cuh"

namespace nbpm {

template <typename R>
__device__ __forceinline__ cx<R> shfl_up_c(cx<R> v, int d) {
	return mk<R>(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}
template <typename R>
__device__ __forceinline__ cx<R> shfl_down_c(cx<R> v, int d) {
	return mk<R>(__shfl_down_sync(0xffffffffu, v.x, d), __shfl_down_sync(0xffffffffu, v.y, d));
}
template <typename R>
__device__ __forceinline__ cx<R> shfl_idx_c(cx<R> v, int l) {
	return mk<R>(__shfl_sync(0xffffffffu, v.x, l), __shfl_sync(0xffffffffu, v.y, l));
}
template <typename R>
__device__ __forceinline__ cx<R> shfl_xor_c(cx<R> v, int m) {
	return mk<R>(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}
template <typename T>
__device__ __forceinline__ T l1abs(cx<T> z) { return fabs(z.x) + fabs(z.y); }

// Moebius maps z -> (a z + b) / (c z + d), scaled at will.
template <typename T>
struct Mob {
	cx<T> a, b, c, d;  // [[a, b], [c, d]]
};
template <typename T>
__device__ __forceinline__ Mob<T> mob_mul(const Mob<T>& X, const Mob<T>& Y) {  // X . Y
	return Mob<T>{X.a * Y.a + X.b * Y.c, X.a * Y.b + X.b * Y.d, X.c * Y.a + X.d * Y.c, X.c * Y.b + X.d * Y.d};
}
template <typename T>
__device__ __forceinline__ void mob_norm(Mob<T>& X) {
	T m = fmax(fmax(l1abs(X.a), l1abs(X.b)), fmax(l1abs(X.c), l1abs(X.d)));
	if(m > (T)0) {
		T r = (T)1 / m;
		X.a = X.a * r; X.b = X.b * r; X.c = X.c * r; X.d = X.d * r;
	}
}
template <typename T>
__device__ __forceinline__ Mob<T> shfl_up_m(const Mob<T>& X, int o) {
	return Mob<T>{shfl_up_c(X.a, o), shfl_up_c(X.b, o), shfl_up_c(X.c, o), shfl_up_c(X.d, o)};
}

// The threads of one line: W warps; a line of several warps meets at barrier `bar` of its block.
struct LineThreads {
	int W, bar, warp, lane;
	int ci, last;  // this thread's chunk, the line's last chunk
	// barrier numbers 0, 1 and 2 as constants: a number in a register makes the block hold all 16, which leaves fewer
	// blocks resident (pair solves of 300x300 lines 161 -> 254 us)
	__device__ __forceinline__ void sync() const {
		if(bar == 0) asm volatile("bar.sync 0, %0;" ::"r"(32 * W) : "memory");
		else if(bar == 1) asm volatile("bar.sync 1, %0;" ::"r"(32 * W) : "memory");
		else asm volatile("bar.sync 2, %0;" ::"r"(32 * W) : "memory");
	}
};

// What a solve needs of node t besides its right-hand sides: f and b1, b2 (the maps of alpha and gamma), rho, eta,
// kappa, tau, and the closing coefficients X (the same in every node): H = X0 alpha_{m-1} + X1 gamma_0, G = X2 .. + X3 ...
// The scans take the right-hand sides bh + f2 bg and d bg.
enum { RN_F = 0, RN_B1, RN_B2, RN_RHO, RN_ETA, RN_KAP, RN_TAU, RN_ALL };
template <typename S>
struct RingNode {
	cx<S> v[RN_ALL], f2, d, X[4];
	__device__ __forceinline__ cx<S> get(int k) const { return v[k]; }
	__device__ __forceinline__ cx<S> close(int k) const { return X[k]; }
};
__host__ __device__ constexpr int ring_factor_shared(int W) { return 7 * W + 4; }

// sh: ring_factor_shared(W) values of shared memory (MULTI: lines of several warps; else unused).
template <bool MULTI, typename S>
__device__ __forceinline__ RingNode<S> ring_factor(const LineThreads& T, cx<S> ph, cx<S> pg, cx<S> qh, cx<S> qg, cx<S>* sh) {
	const cx<S> one = mk<S>(1, 0), zero = mk<S>(0, 0);
	const bool in = T.ci <= T.last;
	if(!in) ph = pg = qh = qg = zero;
	RingNode<S> r;
	// rho_t = (ph qg - qh pg) rho + qh over 1 - pg rho
	Mob<S> X{one, zero, zero, one};
	if(in) X = Mob<S>{cfnma(qh, pg, ph * qg), qh, -pg, one};
#pragma unroll 1
	for(int o = 1; o < 32; o <<= 1) {
		const Mob<S> Y = shfl_up_m(X, o);
		if(T.lane >= o) { X = mob_mul(X, Y); mob_norm(X); }
	}
	cx<S> p = zero, q = one;  // rho of the chunk before the warp's first, as p / q
	if(MULTI) {
		Mob<S>* sm = reinterpret_cast<Mob<S>*>(sh);
		if(T.lane == 31) sm[T.warp] = X;
		T.sync();
		for(int w = 0; w < T.warp; w++) {
			const Mob<S> Y = sm[w];
			const cx<S> t = cfma(Y.a, p, Y.b * q);
			q = cfma(Y.c, p, Y.d * q);
			p = t;
		}
	}
	cx<S> prev = shfl_up_c(cdiv(cfma(X.a, p, X.b * q), cfma(X.c, p, X.d * q)), 1);
	if(T.lane == 0) prev = cdiv(p, q);
	r.d = crecip(cfnma(pg, prev, one));
	r.v[RN_F] = ph * r.d;
	r.f2 = r.v[RN_F] * prev;
	r.v[RN_RHO] = cfma(r.f2, qg, qh);
	r.v[RN_B1] = r.d * pg;
	r.v[RN_B2] = in ? r.d * qg : one;
	// eta: products of f from node 0 on
	cx<S> e = in ? r.v[RN_F] : one;
#pragma unroll 1
	for(int o = 1; o < 32; o <<= 1) {
		const cx<S> y = shfl_up_c(e, o);
		if(T.lane >= o) e = e * y;
	}
	cx<S> e0 = one;
	if(MULTI) {
		cx<S>* se = sh + 4 * T.W;
		if(T.lane == 31) se[T.warp] = e;
		T.sync();
		for(int w = 0; w < T.warp; w++) e0 = e0 * se[w];
		e = e * e0;
	}
	cx<S> eprev = shfl_up_c(e, 1);
	if(T.lane == 0) eprev = e0;
	r.v[RN_ETA] = e;
	// kappa, tau: from the last node back
	cx<S> A = r.v[RN_B2], B = in ? r.v[RN_B1] * eprev : zero;
#pragma unroll 1
	for(int o = 1; o < 32; o <<= 1) {
		const cx<S> a = shfl_down_c(A, o), b = shfl_down_c(B, o);
		if(T.lane + o < 32) { B = cfma(A, b, B); A = A * a; }
	}
	r.v[RN_TAU] = A;
	r.v[RN_KAP] = B;
	cx<S> rl, el, k0, t0;  // rho and eta of the last node, kappa and tau of the first one
	if(MULTI) {
		cx<S>*sa = sh + 5 * T.W, *sb = sa + T.W, *sc = sh + 7 * T.W;
		if(T.lane == 0) { sa[T.warp] = A; sb[T.warp] = B; }
		if(T.ci == T.last) { sc[0] = r.v[RN_RHO]; sc[1] = r.v[RN_ETA]; }
		T.sync();
		cx<S> k = zero, t = one;
		for(int w = T.W - 1; w > T.warp; w--) { k = cfma(sa[w], k, sb[w]); t = sa[w] * t; }
		r.v[RN_KAP] = cfma(A, k, B);
		r.v[RN_TAU] = A * t;
		if(T.ci == 0) { sc[2] = r.v[RN_KAP]; sc[3] = r.v[RN_TAU]; }
		T.sync();
		rl = sc[0]; el = sc[1]; k0 = sc[2]; t0 = sc[3];
	}
	else {
		rl = shfl_idx_c(r.v[RN_RHO], T.last); el = shfl_idx_c(r.v[RN_ETA], T.last);
		k0 = shfl_idx_c(r.v[RN_KAP], 0); t0 = shfl_idx_c(r.v[RN_TAU], 0);
	}
	const cx<S> u = one - el, v = one - t0, det = crecip(cfnma(rl, k0, u * v));
	r.X[0] = v * det;
	r.X[1] = rl * det;
	r.X[2] = k0 * det;
	r.X[3] = u * det;
	return r;
}

// Values V of a solve: cx<S>, or several right-hand sides side by side with overloads of these.
template <typename S>
__device__ __forceinline__ cx<S> vfma(cx<S> a, cx<S> b, cx<S> c) { return cfma(a, b, c); }
template <typename S>
__device__ __forceinline__ cx<S> vshfl(cx<S> v, int l) { return shfl_idx_c(v, l); }

// The border unknowns of a line's chunks for KS right-hand sides. h, x: bh + f2 bg and d bg of the thread's node on
// entry, h_t and g_t on return; hl receives h_{t-1}. s (MULTI): KS (2 W + 1) values V and 2 W values cx<S> of
// shared memory; the first KS W values V are written after the first barrier only.
// Node: RingNode, or where the coefficients lie, with the same functions.
template <bool MULTI, int KS, typename S, typename Node, typename V>
__device__ __forceinline__ void ring_solve(const LineThreads& T, const Node& r, V* h, V* x, V* hl, V* s) {
	const V zero{};
	const int lane = T.lane, W = T.W;
	const bool in = T.ci <= T.last;
	V *sB = s, *sF = s + KS * W, *sL = sF + KS * W;
	cx<S>* sA = reinterpret_cast<cx<S>*>(sL + KS);
	const cx<S> one = mk<S>(1, 0);
	// alpha forward; the coefficients of threads past the last chunk may never have been written
	cx<S> A = in ? r.get(RN_F) : one;
#pragma unroll 1
	for(int o = 1; o < 32; o <<= 1) {
		const cx<S> a = shfl_up_c(A, o);
		const bool on = lane >= o;
#pragma unroll
		for(int j = 0; j < KS; j++) {
			const V b = vshfl(h[j], lane - o);
			if(on) h[j] = vfma(A, b, h[j]);
		}
		if(on) A = A * a;
	}
	V c[KS];  // alpha of the chunk before the warp's first, later gamma of the one after its last
#pragma unroll
	for(int j = 0; j < KS; j++) c[j] = zero;
	if(MULTI) {
		if(lane == 31) {
			sA[T.warp] = A;
#pragma unroll
			for(int j = 0; j < KS; j++) sF[j * W + T.warp] = h[j];
		}
		T.sync();
		for(int w = 0; w < T.warp; w++) {
#pragma unroll
			for(int j = 0; j < KS; j++) c[j] = vfma(sA[w], c[j], sF[j * W + w]);
		}
#pragma unroll
		for(int j = 0; j < KS; j++) h[j] = vfma(A, c[j], h[j]);
		if(T.ci == T.last) {
#pragma unroll
			for(int j = 0; j < KS; j++) sL[j] = h[j];
		}
	}
	// gamma back
#pragma unroll
	for(int j = 0; j < KS; j++) {
		const V up = vshfl(h[j], lane - 1);
		x[j] = in ? vfma(r.get(RN_B1), lane > 0 ? up : c[j], x[j]) : zero;
	}
	A = in ? r.get(RN_B2) : one;
#pragma unroll 1
	for(int o = 1; o < 32; o <<= 1) {
		const cx<S> a = shfl_down_c(A, o);
		const bool on = lane + o < 32;
#pragma unroll
		for(int j = 0; j < KS; j++) {
			const V b = vshfl(x[j], lane + o);
			if(on) x[j] = vfma(A, b, x[j]);
		}
		if(on) A = A * a;
	}
	if(MULTI) {
		if(lane == 0) {
			sA[W + T.warp] = A;
#pragma unroll
			for(int j = 0; j < KS; j++) sB[j * W + T.warp] = x[j];
		}
		T.sync();
	}
	V H[KS];
#pragma unroll
	for(int j = 0; j < KS; j++) {
		V al, g0 = zero;
		if(MULTI) {
			al = sL[j];
			V mine = zero;
			for(int w = W - 1; w >= 0; w--) {
				if(w == T.warp) mine = g0;
				g0 = vfma(sA[W + w], g0, sB[j * W + w]);
			}
			x[j] = vfma(A, mine, x[j]);
		}
		else {
			al = vshfl(h[j], T.last);
			g0 = vshfl(x[j], 0);
		}
		H[j] = vfma(r.close(0), al, vfma(r.close(1), g0, zero));
		const V G = vfma(r.close(2), al, vfma(r.close(3), g0, zero));
		x[j] = vfma(r.get(RN_KAP), H[j], vfma(r.get(RN_TAU), G, x[j]));
		c[j] = G;
	}
	// h_t = alpha_t + rho_t g_{t+1} + eta_t H, and the neighbour's
	if(MULTI) {
		if(lane == 0) {
#pragma unroll
			for(int j = 0; j < KS; j++) sF[j * W + T.warp] = x[j];
		}
		T.sync();
	}
#pragma unroll
	for(int j = 0; j < KS; j++) {
		V g = vshfl(x[j], lane + 1);
		if(MULTI && lane == 31 && T.warp + 1 < W) g = sF[j * W + T.warp + 1];
		if(T.ci == T.last) g = c[j];
		h[j] = vfma(r.get(RN_RHO), g, vfma(r.get(RN_ETA), H[j], h[j]));
	}
	if(MULTI) {
		if(lane == 31) {
#pragma unroll
			for(int j = 0; j < KS; j++) sB[j * W + T.warp] = h[j];
		}
		T.sync();
	}
#pragma unroll
	for(int j = 0; j < KS; j++) {
		hl[j] = vshfl(h[j], lane - 1);
		if(MULTI && lane == 0 && T.warp > 0) hl[j] = sB[j * W + T.warp - 1];
		if(T.ci == 0) hl[j] = H[j];
	}
}

}  // namespace nbpm
