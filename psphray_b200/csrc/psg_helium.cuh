// Helium and secondary ionisation on the device (psphray.HOnly = false,
// psphray.secondaryIonization): the cross sections of the three species,
// the secondary-ionisation table lookup, and the update of one particle
// over the four variables (lambdaH, lambdaHeI, lambdaHeII, ie) of
// function() solve.c:76-141.
//
// The isothermal closed form does not apply once helium's electrons enter
// ye, so every helium update is integrated: Dormand-Prince 5(4) (rtol 1e-6)
// for up to HE_SWITCH steps, then a Rosenbrock W-method (ode23s, rtol 1e-5,
// LU with partial pivoting of the 4x4 W) for particles stiffer than that;
// or, with the explicit build, step_evolve_euler() solve.c:225-316.
#pragma once

#include "psg_div3.h"
#include "psg_solve.cuh"

// xs_get() atomic-rate.c:126-131 for species s (0 HI, 1 HeI, 2 HeII)
__device__ __forceinline__ double xs_get_s(const PhysParams &P, int s, double freq) {
	const double cut = s == 0 ? P.xs_cut_HI : (s == 1 ? P.xs_cut_HeI : P.xs_cut_HeII);
	if (freq < cut) return 0.0;
	return tab_get(P.xs_nrows, P.xs_min, P.xs_step_inv, P.xs, P.xs + (size_t)(1 + s) * P.xs_nrows, freq);
}

// secion_get() secion.c:100-103 = tabfun2_get() tabfun.c:173-222 on column
// col (0 PhiHI, 1 PhiHeI, 2 Eh): clamped rows or columns interpolate along
// the other axis, inside the table bilinear; the grid values are
// min + i*step as tabfun2 stores them.
__device__ inline double secion_get(const PhysParams &P, int col, double E, double y) {
	const int n1 = PSG_SECION_NE, n2 = PSG_SECION_NX;
	const double *d = P.si + (size_t)col * n1 * n2;
	const int xind = (int)((E - P.si_min1) * P.si_step1_inv);
	const int yind = (int)((y - P.si_min2) * P.si_step2_inv);
	int lo = -1;
	if (xind < 0) lo = 0;
	if (xind >= n1 - 1) lo = (n1 - 1) * n2;
	if (lo != -1) {
		if (yind < 0) return d[lo];
		if (yind >= n2 - 1) return d[lo + n2 - 1];
		const double left = P.si_min2 + yind * P.si_step2, right = P.si_min2 + (yind + 1) * P.si_step2;
		return ((right - y) * d[lo + yind] + (y - left) * d[lo + yind + 1]) * P.si_step2_inv;
	}
	int lin = -1;
	if (yind < 0) lin = 0;
	if (yind >= n2 - 1) lin = n2 - 1;
	if (lin != -1) {
		const double left = P.si_min1 + xind * P.si_step1, right = P.si_min1 + (xind + 1) * P.si_step1;
		return ((right - E) * d[(size_t)xind * n2 + lin] + (E - left) * d[(size_t)(xind + 1) * n2 + lin]) *
				P.si_step1_inv;
	}
	const double x1 = P.si_min1 + xind * P.si_step1, x2 = P.si_min1 + (xind + 1) * P.si_step1;
	const double y1 = P.si_min2 + yind * P.si_step2, y2 = P.si_min2 + (yind + 1) * P.si_step2;
	const double fac = P.si_step1_inv * P.si_step2_inv;
	const double f11 = d[(size_t)xind * n2 + yind], f12 = d[(size_t)xind * n2 + yind + 1];
	const double f21 = d[(size_t)(xind + 1) * n2 + yind], f22 = d[(size_t)(xind + 1) * n2 + yind + 1];
	return fac * (f11 * (x2 - E) * (y2 - y) + f21 * (E - x1) * (y2 - y) + f12 * (x2 - E) * (y - y1) +
			f22 * (E - x1) * (y - y1));
}

// lambda_to_ye() psystem.h:134-138 (without yeMET)
__device__ __forceinline__ double ye_he(const PhysParams &P, double lamH, double l1, double l2) {
	return (1.0 - lamH) + P.hemf / P.hmf * 0.25 * (l2 + 2 * (1.0 - l2 - l1));
}

// One helium step: the Step fields the right-hand side reads.
struct HeStep {
	double yeMET, gHI, gHeI, gHeII, heat, time, nH, T;
};

// What the right-hand side needs of it, with what does not change along the
// step taken out of it (the divisions by the step length).
struct HeCtx {
	double yeMET, g0, g1, g2, heat, nH, t, T;      // g, heat: per unit time, the photons negative
};

__device__ __forceinline__ HeCtx make_he_ctx(const HeStep &s) {
	HeCtx c;
	c.yeMET = s.yeMET;
	c.g0 = -s.gHI / s.time;
	c.g1 = -s.gHeI / s.time;
	c.g2 = -s.gHeII / s.time;
	c.heat = s.heat / s.time;
	c.nH = s.nH;
	c.t = s.time;
	c.T = s.T;
	return c;
}

// Where rhs_he reads its rate rows (7 float4 of the table's 8 hold columns):
// in device memory, or those of log T from PSG_WIN_LOGT on in the block's
// shared memory, the others in device memory.
struct HeRows {
	const float4 *row;
	__device__ __forceinline__ HeRows at(const PhysParams &P, int idx) const { return {P.ar_he + 8 * (size_t)idx}; }
	__device__ __forceinline__ float4 operator[](int c) const { return row[c]; }
};
#define HE_WIN_F4 7
struct HeWindowRow {
	const float4 *sm, *gl;
	bool in;
	__device__ __forceinline__ float4 operator[](int c) const {
		float4 v;
		if (in) v = sm[c];
		else v = gl[c];
		return v;
	}
};
struct HeWindow {
	const float4 *sm;
	int lo, n;
	// The block copies the rows into buf, 112 bytes each (an odd number of
	// 16-byte banks), and every thread waits for bar before its first row.
	__device__ __forceinline__ void start(const PhysParams &P, float4 *buf, int rows, uint64_t *bar) {
		sm = buf;
		lo = P.ar_win_lo;
		n = min(rows, P.ar_nrows - lo);
		const uint32_t b = (uint32_t)__cvta_generic_to_shared(bar), d = (uint32_t)__cvta_generic_to_shared(buf);
		const uint32_t row = HE_WIN_F4 * sizeof(float4);
		if (threadIdx.x == 0) rate_bar_arm(b, n * row);
		__syncthreads();      // (armed before a copy ends or anyone waits)
		for (int j = threadIdx.x; j < n; j += blockDim.x)
			rate_bar_copy(d + j * row, P.ar_he + 8 * (size_t)(lo + j), row, b);
	}
	__device__ __forceinline__ HeWindowRow at(const PhysParams &P, int idx) const {
		const int w = idx - lo;
		return {sm + HE_WIN_F4 * w, P.ar_he + 8 * (size_t)idx, (unsigned)w < (unsigned)n};
	}
};

// function() solve.c:76-141 with helium (the rates of FETCH_VARS
// solve.c:42-73); x = (lambdaH, lambdaHeI, lambdaHeII, ie), the derivative
// per unit normalised time. On the spot (case B) the helium equations use
// x_HI where solve.c:94-95 writes it; not on the spot (case A) rec[3]
// receives the recombination photons' rates d(yGrecHII, yGrecHeII,
// yGrecHeIII)/ds of solve.c:84-91. The products and sums are those of
// solve.c, each rounded; the rates come two columns to a 16-byte load from
// the row of tabfun_get() tabfun.c:38-58 (clamped rows, a NaN temperature
// included: offset 0), FP32 value + slope * offset in FP64.
template <typename ROWS = HeRows>
__device__ __forceinline__ void rhs_he(const PhysParams &P, const HeCtx &c, const double x[4], double dx[4],
		double *rec = nullptr, const ROWS &rows = ROWS()) {
	const double xHI = x[0], xHII = 1.0 - x[0], xHeII = x[2];
	const double xHeIII = 1.0 - x[2] - x[1];
	const double ye = (xHII + P.he_f * (xHeII + 2 * xHeIII)) + c.yeMET;
	const double T = P.isothermal ? c.T
			: psg_div3(rn_dmul(__ddiv_rn(rn_dmul(P.MPROTON_OVER_BOLTZMANN, x[3]), rn_dadd(P.T_den0, rn_dmul(P.hmf, ye))), 2.0));
	const double logT = log10(T);
	const double u = (logT - P.ar_min) * P.ar_step_inv;
	int idx = 0;
	double du = 0.0;
	if (u > -1.0) {
		idx = P.ar_nrows - 1;
		if (u < (double)(P.ar_nrows - 1)) {
			idx = (int)u;
			du = logT - __fma_rn((double)idx, P.ar_step, P.ar_min);
		}
	}
	const auto row = rows.at(P, idx);
	const float4 q0 = row[0], q1 = row[1], q2 = row[2];
#define PSG_RATE(v, s, col) (__fma_rn((double)(s), du, (double)(v)) * P.ar_he_scale[col])
	const double nH = c.nH, t = c.t;
	const double ci0 = PSG_RATE(q0.x, q0.y, PSG_HE_CI0) * nH, rc0 = PSG_RATE(q0.z, q0.w, PSG_HE_RC0) * nH;
	const double ci1 = PSG_RATE(q1.x, q1.y, PSG_HE_CI1) * nH, rc1 = PSG_RATE(q1.z, q1.w, PSG_HE_RC1) * nH;
	const double ci2 = PSG_RATE(q2.x, q2.y, PSG_HE_CI2) * nH, rc2 = PSG_RATE(q2.z, q2.w, PSG_HE_RC2) * nH;
	const bool ots = P.on_the_spot;
	const double i1 = ots ? xHI : x[1], i2 = ots ? xHI : xHeII;      // what ionisation multiplies
	dx[0] = (c.g0 + (-ci0 * ye * xHI + rc0 * ye * xHII)) * t;
	dx[1] = (c.g1 + (-ci1 * ye * i1 + rc1 * ye * xHeII)) * t;
	dx[2] = (c.g2 + (-ci2 * ye * i2 - rc1 * ye * xHeII + rc2 * ye * xHeIII)) * t;
	if (!ots && rec) {
		const float4 q5 = row[5], q6 = row[6];
		const double b0 = PSG_RATE(q5.z, q5.w, PSG_HE_RCB0) * nH, b1 = PSG_RATE(q6.x, q6.y, PSG_HE_RCB1) * nH;
		const double b2 = PSG_RATE(q6.z, q6.w, PSG_HE_RCB2) * nH;
		rec[0] = fdim(rc0, b0) * ye * xHII * t;
		rec[1] = fdim(rc1, b1) * ye * xHeII * t;
		rec[2] = fdim(rc2, b2) * ye * xHeIII * t;
	}
	if (P.isothermal || P.adiabatic) {
		dx[3] = 0.0;
	} else {
		const float4 q3 = row[3], q4 = row[4], q5 = row[5];
		const double eta = PSG_RATE(q3.x, q3.y, PSG_HE_RCC) * nH, beta = PSG_RATE(q3.z, q3.w, PSG_HE_BREM) * nH;
		const double zeta = PSG_RATE(q4.x, q4.y, PSG_HE_CIC) * nH, psi = PSG_RATE(q4.z, q4.w, PSG_HE_CEC) * nH;
		const double chi = PSG_RATE(q5.x, q5.y, PSG_HE_COMP);
		const double L = P.H_PER_MASS * ((zeta + psi) * ye * xHI + (eta * ye * xHII) + beta * ye * xHII + chi * ye);
		dx[3] = (c.heat - L) * t;
	}
#undef PSG_RATE
}

#define HE_SWITCH 32

__device__ __forceinline__ double he_err_norm(const double e[4], const double x[4], const double y[4], double atol3,
		double rtol) {
	double err = 0.0;
	for (int i = 0; i < 4; i++) {
		const double sc = (i < 3 ? DP_ATOL0 : atol3) + rtol * fmax(fabs(x[i]), fabs(y[i]));
		err += (e[i] / sc) * (e[i] / sc);
	}
	return sqrt(0.25 * err);
}

// Rosenbrock ode23s over the four variables, a step at a time. With QUAD
// four neighbouring lanes hold the same integration and evaluate a column of
// the Jacobian each (a forward difference), the rest alike: a step is then
// three right-hand sides long instead of six. The loops over W are unrolled
// and its row swaps selected, so that it stays in registers. Not on the spot
// (REC) the three recombination-photon counts are carried as extra
// components whose Jacobian columns are zero: W's extra rows add
// h*d*(J_r . k) to their stage values; they stay out of the error norm.
struct HeRbState {
	double x[4], F0[4], t, h, atol3;
	double rec[3], R0[3];
};

template <bool REC>
__device__ __forceinline__ void he_rb_init(const PhysParams &P, const HeCtx &c, HeRbState &S, const double x[4],
		double t, double h, const double *rec) {
#pragma unroll
	for (int i = 0; i < 4; i++) S.x[i] = x[i];
	S.t = t;
	S.h = fmin(fmax(h, 1e-10), 1.0);
	S.atol3 = DP_ATOL1_REL * fabs(x[3]) + 1e-300;
#pragma unroll
	for (int i = 0; i < 3; i++) {
		S.rec[i] = REC ? rec[i] : 0.0;
		S.R0[i] = 0.0;
	}
	rhs_he(P, c, S.x, S.F0, REC ? S.R0 : nullptr);
}

// One attempted step from S.t < 1: 1 once s = 1 is reached, 0 before, -1
// where W is singular. mask: the lanes that call (whole groups of four).
template <bool REC, bool QUAD>
__device__ __forceinline__ int he_rb_step(const PhysParams &P, const HeCtx &c, HeRbState &S, unsigned mask = 0) {
	const double d = 1.0 / (2.0 + 1.4142135623730951), e32 = 6.0 + 1.4142135623730951;
	double h = S.h;
	if (S.t + h > 1.0) h = 1.0 - S.t;
	double W[4][4], JR[3][4];
	if (QUAD) {
		const int q = threadIdx.x & 3;
		double y[4], Fj[4], Rj[3] = {0.0, 0.0, 0.0}, wcol[4], jcol[3], del = 0.0;
#pragma unroll
		for (int j = 0; j < 4; j++) {
			const double dj = 1e-7 * fmax(fabs(S.x[j]), (j < 3 ? DP_ATOL0 : S.atol3) / RB_RTOL);
			y[j] = j == q ? S.x[j] + dj : S.x[j];
			del = j == q ? dj : del;
		}
		rhs_he(P, c, y, Fj, REC ? Rj : nullptr);
#pragma unroll
		for (int i = 0; i < 4; i++) wcol[i] = (i == q ? 1.0 : 0.0) - h * d * (Fj[i] - S.F0[i]) / del;
		if (REC)
#pragma unroll
			for (int i = 0; i < 3; i++) jcol[i] = (Rj[i] - S.R0[i]) / del;
#pragma unroll
		for (int j = 0; j < 4; j++) {
			const int src = (threadIdx.x & 28) + j;
#pragma unroll
			for (int i = 0; i < 4; i++) W[i][j] = __shfl_sync(mask, wcol[i], src);
			if (REC)
#pragma unroll
				for (int i = 0; i < 3; i++) JR[i][j] = __shfl_sync(mask, jcol[i], src);
		}
	} else {
#pragma unroll
		for (int j = 0; j < 4; j++) {
			const double del = 1e-7 * fmax(fabs(S.x[j]), (j < 3 ? DP_ATOL0 : S.atol3) / RB_RTOL);
			double y[4] = {S.x[0], S.x[1], S.x[2], S.x[3]}, Fj[4], Rj[3] = {0.0, 0.0, 0.0};
			y[j] += del;
			rhs_he(P, c, y, Fj, REC ? Rj : nullptr);
#pragma unroll
			for (int i = 0; i < 4; i++) W[i][j] = (i == j ? 1.0 : 0.0) - h * d * (Fj[i] - S.F0[i]) / del;
			if (REC)
#pragma unroll
				for (int i = 0; i < 3; i++) JR[i][j] = (Rj[i] - S.R0[i]) / del;
		}
	}
	// LU with partial pivoting, in place
	int piv[4];
	bool sing = false;
#pragma unroll
	for (int k = 0; k < 4; k++) {
		int m = k;
		double best = fabs(W[k][k]);
#pragma unroll
		for (int i = k + 1; i < 4; i++) {
			const bool up = fabs(W[i][k]) > best;
			m = up ? i : m;
			best = up ? fabs(W[i][k]) : best;
		}
		piv[k] = m;
#pragma unroll
		for (int i = k + 1; i < 4; i++) {
			const bool sw = m == i;
#pragma unroll
			for (int j = 0; j < 4; j++) {
				const double a = W[k][j], b = W[i][j];
				W[k][j] = sw ? b : a;
				W[i][j] = sw ? a : b;
			}
		}
		sing = sing || W[k][k] == 0.0;
#pragma unroll
		for (int i = k + 1; i < 4; i++) {
			W[i][k] /= W[k][k];
#pragma unroll
			for (int j = k + 1; j < 4; j++) W[i][j] -= W[i][k] * W[k][j];
		}
	}
	if (sing) return -1;
	auto solve = [&](const double b[4], double v[4]) {
#pragma unroll
		for (int i = 0; i < 4; i++) v[i] = b[i];
#pragma unroll
		for (int k = 0; k < 3; k++)
#pragma unroll
			for (int i = k + 1; i < 4; i++) {
				const bool sw = piv[k] == i;
				const double a = v[k], q = v[i];
				v[k] = sw ? q : a;
				v[i] = sw ? a : q;
			}
#pragma unroll
		for (int i = 1; i < 4; i++)
#pragma unroll
			for (int j = 0; j < i; j++) v[i] -= W[i][j] * v[j];
#pragma unroll
		for (int i = 3; i >= 0; i--) {
#pragma unroll
			for (int j = i + 1; j < 4; j++) v[i] -= W[i][j] * v[j];
			v[i] /= W[i][i];
		}
	};
	auto rdot = [&](int i, const double k[4]) {
		return JR[i][0] * k[0] + JR[i][1] * k[1] + JR[i][2] * k[2] + JR[i][3] * k[3];
	};
	double k1[4], k2[4], k3[4], F1[4], F2[4], y[4], yn[4], b[4], e[4];
	double R1[3] = {0.0, 0.0, 0.0}, R2[3] = {0.0, 0.0, 0.0}, kr1[3], kr2[3];
	solve(S.F0, k1);
	if (REC)
#pragma unroll
		for (int i = 0; i < 3; i++) kr1[i] = S.R0[i] + h * d * rdot(i, k1);
#pragma unroll
	for (int i = 0; i < 4; i++) y[i] = S.x[i] + 0.5 * h * k1[i];
	rhs_he(P, c, y, F1, REC ? R1 : nullptr);
#pragma unroll
	for (int i = 0; i < 4; i++) b[i] = F1[i] - k1[i];
	solve(b, k2);
	if (REC)
#pragma unroll
		for (int i = 0; i < 3; i++) kr2[i] = (R1[i] - kr1[i]) + h * d * rdot(i, k2) + kr1[i];
#pragma unroll
	for (int i = 0; i < 4; i++) {
		k2[i] += k1[i];
		yn[i] = S.x[i] + h * k2[i];
	}
	rhs_he(P, c, yn, F2, REC ? R2 : nullptr);
#pragma unroll
	for (int i = 0; i < 4; i++) b[i] = F2[i] - e32 * (k2[i] - F1[i]) - 2.0 * (k1[i] - S.F0[i]);
	solve(b, k3);
#pragma unroll
	for (int i = 0; i < 4; i++) e[i] = h / 6.0 * (k1[i] - 2.0 * k2[i] + k3[i]);
	const double err = he_err_norm(e, S.x, yn, S.atol3, RB_RTOL);
	if (err <= 1.0 && isfinite(err)) {
		S.t += h;
#pragma unroll
		for (int i = 0; i < 4; i++) {
			S.x[i] = yn[i];
			S.F0[i] = F2[i];
		}
		if (REC)
#pragma unroll
			for (int i = 0; i < 3; i++) {
				S.rec[i] += h * kr2[i];
				S.R0[i] = R2[i];
			}
	}
	const double fac = (err > 0.0 && isfinite(err)) ? fmin(5.0, fmax(0.2, 0.9 * pow(err, -1.0 / 3.0)))
			: (isfinite(err) ? 5.0 : 0.2);
	S.h = fmax(h * fac, 1e-14);
	return S.t >= 1.0 ? 1 : 0;
}

// The whole finish on one thread; false if the step limit is reached or W
// is singular.
template <bool REC>
__device__ inline bool rosenbrock_he(const PhysParams &P, const HeCtx &c, double x[4], double t, double h,
		int max_steps, double *rec) {
	HeRbState S;
	he_rb_init<REC>(P, c, S, x, t, h, rec);
	int done = t >= 1.0;
	for (int it = 0; it < max_steps && done == 0; it++) done = he_rb_step<REC, false>(P, c, S);
	for (int i = 0; i < 4; i++) x[i] = S.x[i];
	if (REC)
		for (int i = 0; i < 3; i++) rec[i] = S.rec[i];
	return done == 1;
}

// Dormand-Prince 5(4) over the four variables: the coefficients of the
// stages' arguments, row 5 those of the solution, and of the error (the
// second stage enters neither).
static __constant__ double kHeA[6][6] = {{1. / 5, 0, 0, 0, 0, 0}, {3. / 40, 9. / 40, 0, 0, 0, 0},
	{44. / 45, -56. / 15, 32. / 9, 0, 0, 0}, {19372. / 6561, -25360. / 2187, 64448. / 6561, -212. / 729, 0, 0},
	{9017. / 3168, -355. / 33, 46732. / 5247, 49. / 176, -5103. / 18656, 0},
	{35. / 384, 0, 500. / 1113, 125. / 192, -2187. / 6784, 11. / 84}};
static __constant__ double kHeE[6] = {71. / 57600, 0, -71. / 16695, 71. / 1920, -17253. / 339200, 22. / 525};

// One integration; its stages' slopes live in k (a thread's own column of
// 6 x 4 doubles, stride apart): a step then loops over its stages with one
// copy of the right-hand side, which needs half the registers and a seventh
// of the instructions that the unrolled form took. With REC (not on the
// spot) the recombination photons are a quadrature over the same stages.
struct HeDp {
	double x[4], t, h, atol3;
	double gain[3], r1[3];
	int steps;
};

// Starts the integration at x: the first slope and step. Evaluates nothing
// but the right-hand side at x.
template <bool REC>
__device__ __forceinline__ void he_dp_start(HeDp &S, const double k1[4], const double r1[3], double *k, int stride) {
	S.t = 0.0;
	S.steps = 0;
	S.atol3 = DP_ATOL1_REL * fabs(S.x[3]) + 1e-300;
	double h = 1.0;
#pragma unroll
	for (int i = 0; i < 4; i++) {
		const double scale = fabs(S.x[i]) + (i < 3 ? DP_ATOL0 : S.atol3) / DP_RTOL;
		if (fabs(k1[i]) > 0.0) h = fmin(h, 0.01 * scale / fabs(k1[i]));
		k[i * stride] = k1[i];
	}
	S.h = fmax(h, 1e-8);
	if (REC)
#pragma unroll
		for (int i = 0; i < 3; i++) {
			S.gain[i] = 0.0;
			S.r1[i] = r1[i];
		}
}

// One pass over the lanes' next work: for fresh lanes the slope at x first,
// then for all lanes one attempted step. fresh must be the warp's when other
// lanes call too: anyfresh says whether any lane's is set. UNROLLED: the
// stages one after another, so that slopes in an array of the thread's own
// (stride 1) stay in registers; the same sums.
template <bool REC, bool UNROLLED = false, typename ROWS = HeRows>
__device__ __forceinline__ void he_dp_step(const PhysParams &P, const HeCtx &c, HeDp &S, bool fresh, bool anyfresh,
		double *k, int stride, const ROWS &rows = ROWS()) {
	double e[4], y[4], q[3], h = 0.0;
	if (UNROLLED && fresh) {
		double dx[4], r[3];
		rhs_he(P, c, S.x, dx, REC ? r : nullptr, rows);
		he_dp_start<REC>(S, dx, r, k, stride);
	}
	constexpr int U = UNROLLED ? 6 : 1;
#pragma unroll U
	for (int st = !UNROLLED && anyfresh ? -1 : 0; st < 6; st++) {
		if (st < 0 && !fresh) continue;
		if (st <= 0) {
			if (st == 0) {
				if (S.t + S.h > 1.0) S.h = 1.0 - S.t;
				h = S.h;
			}
#pragma unroll
			for (int i = 0; i < 4; i++) y[i] = S.x[i];
			if (REC)
#pragma unroll
				for (int i = 0; i < 3; i++) q[i] = kHeA[5][0] * S.r1[i];
		}
		if (st >= 0) {
#pragma unroll
			for (int i = 0; i < 4; i++) {
				const double k1 = k[i * stride];
				double s = kHeA[st][0] * k1;
				if (st == 5) e[i] = kHeE[0] * k1;
#pragma unroll
				for (int j = 1; j < 6; j++)
					if (j <= st && (st < 5 || j != 1)) {
						const double kj = k[(4 * j + i) * stride];
						s += kHeA[st][j] * kj;
						if (st == 5) e[i] += kHeE[j] * kj;
					}
				y[i] = S.x[i] + h * s;
			}
		}
		double dx[4], r[3];
		rhs_he(P, c, y, dx, REC ? r : nullptr, rows);
		if (st < 0) {
			he_dp_start<REC>(S, dx, r, k, stride);
		} else if (st < 5) {
#pragma unroll
			for (int i = 0; i < 4; i++) k[(4 * (st + 1) + i) * stride] = dx[i];
			if (REC && st > 0)
#pragma unroll
				for (int i = 0; i < 3; i++) q[i] += kHeA[5][st + 1] * r[i];
		} else {
#pragma unroll
			for (int i = 0; i < 4; i++) e[i] = h * (e[i] + (-1. / 40) * dx[i]);
			const double err = he_err_norm(e, S.x, y, S.atol3, DP_RTOL);
			if (err <= 1.0) {
				S.t += h;
#pragma unroll
				for (int i = 0; i < 4; i++) {
					S.x[i] = y[i];
					k[i * stride] = dx[i];
				}
				if (REC)
#pragma unroll
					for (int i = 0; i < 3; i++) {
						S.gain[i] += h * q[i];
						S.r1[i] = r[i];
					}
			}
			const double fac = err > 0.0 ? fmin(5.0, fmax(0.2, 0.9 * pow(err, -0.2))) : 5.0;
			S.h = fmax(h * fac, 1e-14);
			S.steps++;
		}
	}
}

// Up to HE_SWITCH steps from s = 0 on one thread; returns true once s = 1
// is reached, else leaves the time reached and the next step size in *t_out,
// *h_out. With rec, rec[3] accumulates the recombination photons. The slopes
// stay in registers: psg_step_evolve of 300 records 271 -> 237 us (case A
// 318 -> 254 us) against the loop over slopes in the thread's stack.
template <bool REC>
__device__ inline bool dopri_he_explicit(const PhysParams &P, const HeCtx &c, double x[4], double *rec,
		double *t_out, double *h_out) {
	double k[24];
	HeDp S;
#pragma unroll
	for (int i = 0; i < 4; i++) S.x[i] = x[i];
	bool fresh = true;
	do {
		he_dp_step<REC, true>(P, c, S, fresh, fresh, k, 1);
		fresh = false;
	} while (S.t < 1.0 && S.steps < HE_SWITCH);
#pragma unroll
	for (int i = 0; i < 4; i++) x[i] = S.x[i];
	if (REC)
#pragma unroll
		for (int i = 0; i < 3; i++) rec[i] += S.gain[i];
	*t_out = S.t;
	*h_out = S.h;
	return S.t >= 1.0;
}

// Dormand-Prince 5(4) over the four variables, then the Rosenbrock finish.
__device__ inline bool dopri_he(const PhysParams &P, const HeCtx &s, double x[4], int max_steps,
		double *rec = nullptr) {
	double t = 0.0, h = 0.0;
	if (rec)
		return dopri_he_explicit<true>(P, s, x, rec, &t, &h) || rosenbrock_he<true>(P, s, x, t, h, max_steps, rec);
	return dopri_he_explicit<false>(P, s, x, rec, &t, &h) || rosenbrock_he<false>(P, s, x, t, h, max_steps, rec);
}

// step_evolve_euler() solve.c:225-316 with helium: the internal step a
// 200th of the shortest recombination and ionisation time at the start,
// at most 10000 steps, stopping one step after a fraction leaves [0, 1] or
// x_HeIII turns negative. Returns PSG_ST_* bits.
__device__ inline uint32_t euler_he(const PhysParams &P, const HeStep &s, double x[4], double &step_remain,
		int &refined, double *rec = nullptr) {
	const double ye = (1.0 - x[0] + P.hemf / P.hmf * 0.25 * (x[2] + 2 * (1.0 - x[2] - x[1]))) + s.yeMET;
	const double T = P.isothermal ? s.T : ieye2T(P, x[3], ye);
	const RateAt R = rates_at(P, log10(T));
	double rectime = 1.0 / (R(PSG_AR_HII_RC_A) * s.nH);
	double iontime = 1.0 / (R(PSG_AR_HI_CI) * s.nH);
	rectime = fmin(rectime, 1.0 / (R(PSG_AR_HEII_RC_A) * s.nH));
	rectime = fmin(rectime, 1.0 / (R(PSG_AR_HEIII_RC_A) * s.nH));
	iontime = fmin(iontime, 1.0 / (R(PSG_AR_HEI_CI) * s.nH));
	iontime = fmin(iontime, 1.0 / (R(PSG_AR_HEII_CI) * s.nH));
	double internal = fmin(rectime, iontime) / 200.;
	internal = fmin(internal, s.time);
	int nsteps = (int)(s.time / internal);
	if (nsteps > 10000) nsteps = 10000;
	if (nsteps < 1) nsteps = 1;
	const double h = 1.0 / nsteps;
	refined = nsteps > 1;
	const HeCtx cx = make_he_ctx(s);
	uint32_t st = 0;
	int k;
	for (k = 0; k < nsteps; k++) {
		double dx[4], r[3] = {0.0, 0.0, 0.0};
		rhs_he(P, cx, x, dx, rec ? r : nullptr);
		if (!(x[3] + dx[3] >= 0.0)) st |= PSG_ST_IE_NEG;
		for (int i = 0; i < 4; i++) x[i] += dx[i] * h;
		if (rec)
			for (int i = 0; i < 3; i++) rec[i] += r[i] * h;
		if (!isfinite(x[0]) || !isfinite(x[1]) || !isfinite(x[2]) || !isfinite(x[3])) {
			st |= PSG_ST_NAN;
			k++;
			break;
		}
		bool out = false;
		for (int i = 0; i < 3; i++) out |= (x[i] < 0.0 || x[i] > 1.0);
		if (out || 1.0 - x[1] - x[2] < 0.0) {
			k++;
			break;
		}
	}
	step_remain = 1.0 - (double)((float)k / (float)nsteps);
	return st;
}

// LSODA's exit clamps of the fractions (solve.c:208-210).
__device__ __forceinline__ void clamp_he(double x[4]) {
	x[0] = fmin(1., fmax(0., x[0]));
	x[1] = fmin(1., fmax(0., x[1]));
	x[2] = fmin(1. - x[1], fmax(0., x[2]));
}

// One helium step of step_evolve() (LSODA's exit clamps, solve.c:208-213):
// x = (lambdaH, lambdaHeI, lambdaHeII, ie) in and out; with rec (not on the
// spot) the three recombination-photon counts in and out. Returns PSG_ST_*
// bits.
__device__ inline uint32_t solve_step_he(const PhysParams &P, const HeStep &s, double x[4],
		double *rec = nullptr) {
	uint32_t st = 0;
	double gain[3] = {0.0, 0.0, 0.0};
	if (!dopri_he(P, make_he_ctx(s), x, 200000, rec ? gain : nullptr)) st |= PSG_ST_SOLVER;
	if (rec)
		for (int i = 0; i < 3; i++) rec[i] = fmax(0.0, rec[i] + gain[i]);
	if (!(x[3] >= 0.0)) st |= PSG_ST_IE_NEG;
	for (int i = 0; i < 4; i++)
		if (!isfinite(x[i])) st |= PSG_ST_NAN;
	x[0] = fmin(1., fmax(0., x[0]));
	x[1] = fmin(1., fmax(0., x[1]));
	x[2] = fmin(1. - x[1], fmax(0., x[2]));
	return st;
}
