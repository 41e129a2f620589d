// The dense factorisations of the stabilised equal-time Green's function
// (reference src/greens.c:69-208, calc_eq_g), one CTA of 16 warps per
// (chain, spin) matrix, the N x N working matrix in shared memory (or, where
// it does not fit, in a per-item global workspace):
//
// k_qrp   Householder QR with column pivoting by the largest remaining
//         partial column norm, downdated and recomputed as LAPACK geqp3 does
//         (greens.c:89, QR_PIVOT);
// k_qrb   Householder QR of the columns in order of decreasing norm, computed
//         once after scaling by d (the norm pre-pivoting of greens.c:112-135,
//         QR_PRESORT), blocked by 8 with DMMA block-reflector updates;
//         both form Q explicitly (so that a later g*Q is a plain GEMM and
//         diag(v) Q^H is elementwise), with the phase of det Q;
// k_qrc   k_qrb's factorisation with the matrix over a cluster's shared memory;
// k_recb  G = (D_b^-1 Q^H + D_s T)^-1 D_b^-1 Q^H (greens.c:157-178) by LU
//         with partial row pivoting and two triangular solves, plus the
//         phase of det G (greens.c:194-207); or the two-sided form of it for
//         a product given as Q D T on its left and T_L^H D_L Q_L^H on its right.
#pragma once

#include "common.cuh"

namespace dq {

enum : int { QR_PIVOT = 1, QR_PRESORT = 2 };

template <typename T>
struct QrArgs {
	int N, batch, mode;
	const T *X; long long x_stride;       // input matrices (ld N)
	int trans;                            // PRESORT: factor X^H instead of X
	const double *dcol; long long d_stride; // PRESORT: columns scaled by d on load (null: 1)
	T *Q; long long q_stride;             // explicit Q out
	T *Tout; long long t_stride;          // T = D^-1 R P^T (PRESORT: or Rs)
	T *Rs; long long r_stride;            // PRESORT: D^-1 R in pivot order
	int *pvt; long long p_stride;         // pivot order (column chosen at step j)
	double *dout; long long dout_stride;  // diag(R), 0 -> 1 (real: Householder beta)
	T *qdet;                              // phase of det Q per item
	T *work; long long w_stride;          // N x N per item: working matrix of the
	                                      // shared-memory kernels' global-memory form
	unsigned *err;
};

// ----------------------------------------------- blocked QR, pre-sorted
//
// The QR_PRESORT factorisation (greens.c:119-146: columns scaled by
// the previous D, ordered by descending norm, then geqrf and the explicit
// Q), with the matrix in shared memory and the reflectors taken NBK = 8 at
// a time.  Warps 0-3 carry the block reflector I - V T^H V^H of a panel to the
// next panel's columns and factor that panel (qr_panel8); the other 12 take it to
// the remaining columns meanwhile (reflect8, FP64 tensor-core tiles).
// Q is then accumulated backwards, block by block, in the same memory.
// Outputs: Q, D^-1 R in position order (Rs), diag(R) and the order.

// leading dimension: N rounded so that ld = 4 (mod 16) doubles, which keeps
// the 8 x 4 DMMA fragment loads of neighbouring columns bank-conflict free
__host__ __device__ inline int qrb_ld(int N) { return (N + 11) / 16 * 16 + 4; }

// In the global-memory form (GM) the N x N working matrix lives in the
// caller's per-item workspace with leading dimension N, and shared memory
// keeps only the small arrays; otherwise it is the first part of shared memory.
template <typename T, int NBK>
size_t qrb_smem_bytes(int N, bool gm = false)
{
	const int np = (N + NBK - 1) / NBK, ld = gm ? N : qrb_ld(N);
	return sizeof(T) * ((gm ? (size_t)ld * NBK : (size_t)ld * N) + (size_t)ld * NBK + N
	                    + (size_t)np * NBK * NBK)
	       + sizeof(double) * 3 * (size_t)N + sizeof(int) * (size_t)N + 64;
}

// warps that factor a panel, and rows of it per lane: two while the panel's
// rows fit a thread's registers, else four (us a launch of two items, with one /
// two / four warps: N = 64 106 / 72 / 72, N = 144 281 / 201 / 205)
template <typename T, int RPL>
struct QrbPanel {
	static constexpr int PW = (!is_cplx<T>::value && RPL <= 5) ? 2 : 4;
	static constexpr int RP = (RPL + PW - 1) / PW;
};

// C layout -> B layout of an 8 x 8 tile: element (row r, col c) sits in lane
// 4 c + r % 4, k-step r / 4; lane (lq, lr) of the C layout holds row lq, columns
// 2 lr + e
template <typename T>
__device__ inline void tile_c_to_b(const T (&x)[2], T (&b)[2], int lane)
{
	const int lr = lane & 3, lq = lane >> 2;
#pragma unroll
	for (int s = 0; s < 2; s++) {
		const int src = 4 * (4 * s + lr) + (lq >> 1);
		const T v0 = shfl(x[0], src), v1 = shfl(x[1], src);
		b[s] = (lq & 1) ? v1 : v0;
	}
}

template <typename T>
__device__ inline void tile_b_to_c(const T (&b)[2], T (&x)[2], int lane)
{
	// C lane (lq, lr), element e: row lq, column 2 lr + e, held by B lane
	// 4 (2 lr + e) + lq % 4 in k-step lq / 4
	const int lr = lane & 3, lq = lane >> 2;
#pragma unroll
	for (int e = 0; e < 2; e++) {
		const int src = 4 * (2 * lr + e) + (lq & 3);
		const T v0 = shfl(b[0], src), v1 = shfl(b[1], src);
		x[e] = (lq < 4) ? v0 : v1;
	}
}

// c (8 x 8 accumulators) += a b, one k-step
__device__ inline void tile_mma(double (&c)[2], double a, double b) { dmma(c[0], c[1], a, b); }
__device__ inline void tile_mma(zd (&c)[2], zd a, zd b)
{
	dmma(c[0].x, c[1].x, a.x, b.x);
	dmma(c[0].x, c[1].x, -a.y, b.y);
	dmma(c[0].y, c[1].y, a.x, b.y);
	dmma(c[0].y, c[1].y, a.y, b.x);
}

// reflector k of a panel at its row r: unit diagonal, zero above; V keeps R there
template <typename T>
__device__ inline T qr_v8(const T *V, size_t ldv, int r, int k, int mr, int nb)
{
	if (k >= nb || r < k || r >= mr) return zero<T>();
	return (r == k) ? one<T>() : V[r + ldv * k];
}

// The block reflector of 8 reflectors on the 8 columns of C (ncol of them
// present) on the FP64 tensor cores, one warp: W = V^H C, W' = op(T) W (T^H
// when HERM), C -= V W'.  V and C from the panel's first row on, mr rows; the
// first 8 rows of V hold R on and above the diagonal (qr_v8), the others
// are read as they are, so columns k >= nb hold zeros there.  Fragment layouts
// of m8n8k4: lane l holds A[l/4][l%4], B[l%4][l/4] and C[l/4][2(l%4) + {0,1}];
// W moves from the C to the B layout by shuffles.  Absent columns are computed
// on the last present one and not stored.  W's row quads go round AC
// accumulators, whose number alone sets the order of the sum; LD quads and RT row
// tiles are in flight at a time, more when C lies in global memory.
// Bound by the FP64 tensor pipe (16 cycles a DMMA and SM quarter) when all
// warps have columns, else by the chain load - product - store; the full row
// groups carry no row or column test, which cost more issue slots than the
// products.
template <typename T, bool HERM, int AC, int LD, int RT>
__device__ inline void reflect8(T *C, size_t ldc, int ncol, const T *V, size_t ldv, const T *Tp, int mr,
		int nb, int lane)
{
	const int lr = lane & 3, lq = lane >> 2;
	T w[AC][2];
#pragma unroll
	for (int u = 0; u < AC; u++) w[u][0] = w[u][1] = zero<T>();
	const T *cb = C + ldc * min(lq, ncol - 1), *vb = V + ldv * lq;
	{
		T av[2], bv[2];
#pragma unroll
		for (int u = 0; u < 2; u++) {
			const int q = 4 * u + lr;
			av[u] = conjv(qr_v8(V, ldv, q, lq, mr, nb));
			bv[u] = q < mr ? cb[q] : zero<T>();
		}
#pragma unroll
		for (int u = 0; u < 2; u++) tile_mma(w[u % AC], av[u], bv[u]);
	}
	// quad q to accumulator q % AC, loads LD at a time
	constexpr int B = AC > LD ? AC : LD;
	static_assert(B % AC == 0 && B % LD == 0, "whole rounds");
	int r = 8;
#pragma unroll 2
	for (; r + 4 * B <= mr; r += 4 * B) {
#pragma unroll
		for (int g = 0; g < B; g += LD) {
			T av[LD], bv[LD];
#pragma unroll
			for (int u = 0; u < LD; u++) {
				av[u] = conjv(vb[r + 4 * (g + u) + lr]);
				bv[u] = cb[r + 4 * (g + u) + lr];
			}
#pragma unroll
			for (int u = 0; u < LD; u++) tile_mma(w[(g + u) % AC], av[u], bv[u]);
		}
	}
#pragma unroll
	for (int u = 0; u < B; u++) {
		if (r + 4 * u >= mr) break;
		const bool ok = r + 4 * u + lr < mr;
		tile_mma(w[u % AC], ok ? conjv(vb[r + 4 * u + lr]) : zero<T>(), ok ? cb[r + 4 * u + lr] : zero<T>());
	}
#pragma unroll
	for (int u = AC / 2; u > 0; u /= 2)
#pragma unroll
		for (int k = 0; k < u; k++)
#pragma unroll
			for (int e = 0; e < 2; e++) w[k][e] += w[k + u][e];
	T b[2], x[2] = {zero<T>(), zero<T>()};
	tile_c_to_b(w[0], b, lane);
#pragma unroll
	for (int s = 0; s < 2; s++) {
		const int kk = 4 * s + lr;
		T a;
		if (HERM) a = (kk <= lq && lq < nb) ? conjv(Tp[kk + 8 * lq]) : zero<T>();
		else a = (lq <= kk && kk < nb) ? Tp[lq + 8 * kk] : zero<T>();
		tile_mma(x, a, b[s]);
	}
	tile_c_to_b(x, b, lane);
	b[0] = -b[0];
	b[1] = -b[1];
	const bool st[2] = {2 * lr < ncol, 2 * lr + 1 < ncol};
	T *ce[2] = {C + ldc * min(2 * lr, ncol - 1) + lq, C + ldc * min(2 * lr + 1, ncol - 1) + lq};
	const T *vs[2] = {V + ldv * lr + lq, V + ldv * (4 + lr) + lq};
	// one row tile with every test
	auto edge = [&](int r, bool top) {
		const bool ok = r + lq < mr;
		T y[2];
#pragma unroll
		for (int e = 0; e < 2; e++) y[e] = ok ? ce[e][r] : zero<T>();
#pragma unroll
		for (int s = 0; s < 2; s++)
			tile_mma(y, top ? qr_v8(V, ldv, lq, 4 * s + lr, mr, nb) : (ok ? vs[s][r] : zero<T>()), b[s]);
#pragma unroll
		for (int e = 0; e < 2; e++)
			if (ok && st[e]) ce[e][r] = y[e];
	};
	edge(0, true);
	r = 8;
	for (; r + 8 * RT <= mr; r += 8 * RT) {
		T y[RT][2], va[RT][2];
#pragma unroll
		for (int u = 0; u < RT; u++)
#pragma unroll
			for (int e = 0; e < 2; e++) {
				y[u][e] = ce[e][r + 8 * u];
				va[u][e] = vs[e][r + 8 * u];
			}
#pragma unroll
		for (int s = 0; s < 2; s++)
#pragma unroll
			for (int u = 0; u < RT; u++) tile_mma(y[u], va[u][s], b[s]);
#pragma unroll
		for (int u = 0; u < RT; u++)
#pragma unroll
			for (int e = 0; e < 2; e++)
				if (st[e]) ce[e][r + 8 * u] = y[u][e];
	}
	for (; r < mr; r += 8) edge(r, false);
}

// depths of reflect8 for columns in shared and in global memory: the same
// accumulators in both, so that a QR gives the same bits wherever its matrix
// lies (the form goes by the items of a launch, which a lane count changes).
// Eight for complex scalars, whose terms are two products each: with two, G of
// complex Hubbard clusters was 12 to 18% further from the exact one (N = 64 to
// 144) than with the shuffled sums that the tiles replaced, with eight 4 to 5%, at
// the same time a launch.
template <typename T, bool GMEM>
struct ReflectDepth {
	static constexpr int AC = is_cplx<T>::value ? 8 : 4;
	static constexpr int LD = is_cplx<T>::value ? (GMEM ? 4 : 2) : (GMEM ? 8 : 4);
	static constexpr int RT = is_cplx<T>::value ? (GMEM ? 4 : 2) : (GMEM ? 8 : 3);
};

// depths of reflect_next for up to 32 RPL rows
template <typename T, int RPL>
struct NextDepth {
	static constexpr int AC = is_cplx<T>::value ? (RPL > 2 ? 4 : 2) : (RPL > 4 ? 8 : RPL > 1 ? 4 : 2);
	static constexpr int RT = is_cplx<T>::value ? (RPL < 3 ? RPL : 3) : (RPL < 6 ? RPL : (RPL + 1) / 2);
};

// columns [cfirst, cend) of A in groups of 8, group g taken by warp `slot` when
// g % nslots == slot; Vp and A from row j0 on
template <typename T, bool HERM, bool GMEM>
__device__ inline void reflect_cols(T *A, size_t lda, int cfirst, int cend, const T *Vp, size_t ldv,
		const T *Tp, int mr, int nb, int slot, int nslots, int lane)
{
	using D = ReflectDepth<T, GMEM>;
	for (int c = cfirst + 8 * slot; c < cend; c += 8 * nslots)
		reflect8<T, HERM, D::AC, D::LD, D::RT>(A + lda * c, lda, min(8, cend - c), Vp, ldv, Tp, mr, nb, lane);
}

// ----------------------------------------------- panel of 8 columns
//
// Householder QR of mr x nb (nb <= 8) by PW warps, each lane holding its rows
// lane + 32 (w + PW t), t < RP, of all 8 columns in registers, and the block's
// T (larft, forward columnwise).  Per reflector k one reduction gives
// x_k^H x_c below row k for every column c: the norm (c = k), v_k^H x_c of the
// later columns and v_c^H v_k of the earlier ones, with v_k = scal x_k below the
// diagonal and 1 on it (zlarfg convention).  The 8 sums are folded onto the
// lanes, lane 4 s + {0..3} ending up with slot s, and each lane forms its
// slot's coefficient: one barrier per reflector and no second reduction.  Bound
// by that chain of latencies (about 1000 cycles a reflector, 300 of them the
// square root and the division), so
// - the columns rotate through the slots and the loop is not unrolled,
// - each lane forms one of the quotients 1 / (alpha - beta) and tau, and
// - T is solved for at the end, one column a lane.
// One column per warp with two barriers and two reductions per reflector before:
// k_qrb 275 -> 201 us at N = 144 x 2, 1050 -> 800 us at N = 144 x 512, complex
// N = 100 x 64 320 -> 238 us, with the products of reflect8.
// load(r, c): the panel's entries; store(r, c, v) for all 8 columns: R on and
// above the diagonal, V below, zero for c >= nb.
template <typename T, int PW>
struct PanelShared {
	T red[2][PW][8], xrow[2][8], g[PW][8], y[8][8];
	T wred[4][64];
};

template <int NWARP>
__device__ inline void bar_panel()
{
	asm volatile("barrier.sync 1, %0;\n" ::"n"(NWARP * 32) : "memory");
}

template <typename T, int PW, int RP, typename L, typename S>
__device__ inline void qr_panel8(PanelShared<T, PW> &sh, int mr, int nb, int w, int lane, T *Tp, T *tau,
		double *beta_out, double *vv, const L &load, const S &store)
{
	const int r0 = lane + 32 * w, cl = lane >> 2;
	if (nb < 8 && w == PW - 1) sh.y[lane >> 3][lane & 7] = sh.y[4 + (lane >> 3)][lane & 7] = zero<T>();
	T x[8][RP];
#pragma unroll
	for (int c = 0; c < 8; c++)
#pragma unroll
		for (int t = 0; t < RP; t++) {
			const int r = r0 + 32 * PW * t;
			x[c][t] = (c < nb && r < mr) ? load(r, c) : zero<T>();
		}
	// slot s holds column (k + s) mod 8
	auto rotate = [&]() {
#pragma unroll
		for (int t = 0; t < RP; t++) {
			const T first = x[0][t];
#pragma unroll
			for (int s = 0; s < 7; s++) x[s][t] = x[s + 1][t];
			x[7][t] = first;
		}
	};
#pragma unroll 1
	for (int k = 0; k < nb; k++) {
		T *xr = sh.xrow[k & 1];
		if (r0 == k) {
#pragma unroll
			for (int s = 0; s < 8; s++) xr[s] = x[s][0];
		}
		T d[8];
#pragma unroll
		for (int s = 0; s < 8; s++) d[s] = zero<T>();
#pragma unroll
		for (int t = 0; t < RP; t++) {
			const T xk = (t == 0 && r0 <= k) ? zero<T>() : conjv(x[0][t]);
#pragma unroll
			for (int s = 0; s < 8; s++) d[s] += xk * x[s][t];
		}
#pragma unroll
		for (int o = 16, n = 4; n > 0; o >>= 1, n >>= 1) {
			const bool up = lane & o;
#pragma unroll
			for (int i = 0; i < n; i++) {
				const T send = up ? d[i] : d[i + n];
				d[i] = (up ? d[i + n] : d[i]) + shfl_xor(send, o);
			}
		}
		T sm = d[0];
		sm += shfl_xor(sm, 2);
		sm += shfl_xor(sm, 1);
		double sig;
		if (PW > 1) {
			if ((lane & 3) == 0) sh.red[k & 1][w][cl] = sm;
			bar_panel<PW>();
			sm = sh.red[k & 1][0][cl];
			sig = re(sh.red[k & 1][0][0]);
#pragma unroll
			for (int q = 1; q < PW; q++) {
				sm += sh.red[k & 1][q][cl];
				sig += re(sh.red[k & 1][q][0]);
			}
		} else {
			__syncwarp();
			sig = re(shfl(sm, 0));
		}
		const T alpha = xr[0], xc = xr[cl];
		const bool none = sig == 0.0 && im(alpha) == 0.0;
		const double beta = none ? re(alpha) : -copysign(sqrt(abs2(alpha) + sig), re(alpha));
		const T del = alpha - beta;
		// scal = 1 / del and tau = -del / beta, one quotient a lane
		T tk, scal;
		if constexpr (is_cplx<T>::value) {
			const double q = ((lane & 1) ? im(del) : re(del)) / ((lane & 2) ? -beta : ((lane & 1) ? -abs2(del) : abs2(del)));
			scal = T{__shfl_sync(0xffffffffu, q, 0), __shfl_sync(0xffffffffu, q, 1)};
			tk = T{__shfl_sync(0xffffffffu, q, 2), __shfl_sync(0xffffffffu, q, 3)};
		} else {
			const double q = ((lane & 1) ? -del : 1.0) / ((lane & 1) ? beta : del);
			const double o = shfl_xor(q, 1);
			scal = (lane & 1) ? o : q;
			tk = (lane & 1) ? q : o;
		}
		if (none) scal = tk = zero<T>();
		// v_k^H x_c; later columns: x_c -= v_k g; earlier ones hold v_c already
		const T dk = xc + conjv(scal) * sm;
		const T g = (cl > 0 && cl < 8 - k) ? conjv(tk) * dk : zero<T>();
		if ((lane & 3) == 0) sh.g[w][cl] = g;
		__syncwarp();
#pragma unroll
		for (int t = 0; t < RP; t++)
			if (t > 0 || r0 > k) x[0][t] *= scal;
		T u[RP];
#pragma unroll
		for (int t = 0; t < RP; t++) u[t] = (t == 0 && r0 <= k) ? (r0 == k ? one<T>() : zero<T>()) : x[0][t];
		if (r0 == k) x[0][0] = from_re<T>(beta);
#pragma unroll
		for (int s = 1; s < 8; s++) {
			const T gs = sh.g[w][s];
#pragma unroll
			for (int t = 0; t < RP; t++) x[s][t] -= u[t] * gs;
		}
		if (w == PW - 1) {
			if (lane == 0) {
				tau[k] = tk;
				beta_out[k] = beta;
				vv[k] = 1.0 + sig * abs2(scal);
			}
			if (cl >= 8 - k && (lane & 3) == 0) sh.y[k + cl - 8][k] = conjv(dk);
		}
		rotate();
	}
	for (int k = nb; k < 8; k++) rotate();
	__syncwarp();
	if (PW > 1) bar_panel<PW>();
	if (w == PW - 1 && lane < nb) {
		// column `lane` of T upwards from its diagonal:
		// T[i, c] = -tau_i (y_i,i+1 T[i+1, c] + ... + y_ic T[c, c])
		T tc[8];
#pragma unroll
		for (int i = 7; i >= 0; i--) {
			T ts = zero<T>();
#pragma unroll
			for (int m = 7; m > i; m--) ts += sh.y[i][m] * tc[m];
			const T ti = i < nb ? tau[i] : zero<T>();
			tc[i] = (i > lane) ? zero<T>() : (i == lane) ? ti : -(ti * ts);
			if (i <= lane) Tp[i + 8 * lane] = tc[i];
		}
	}
#pragma unroll
	for (int c = 0; c < 8; c++) {
#pragma unroll
		for (int t = 0; t < RP; t++) {
			const int r = r0 + 32 * PW * t;
			if (r < mr) store(r, c, x[c][t]);
		}
	}
}

// the block reflector (V, Tp) on the next panel's columns (ncol <= 8), the rows
// over GW warps; C(r, c) is read through load, written through store
template <typename T, int GW, int AC, int RT, int PW, typename L, typename S>
__device__ inline void reflect_next(PanelShared<T, PW> &sh, int ncol, const T *V, size_t ldv, const T *Tp,
		int mr, int nb, int w, int lane, const L &load, const S &store)
{
	const int lr = lane & 3, lq = lane >> 2;
	T wv[AC][2];
#pragma unroll
	for (int u = 0; u < AC; u++) wv[u][0] = wv[u][1] = zero<T>();
	const int cb = min(lq, ncol - 1);
	const T *vb = V + ldv * lq;
	for (int r = 4 * w; r < mr; r += 4 * GW * AC) {
		T av[AC], bv[AC];
#pragma unroll
		for (int u = 0; u < AC; u++) {
			const int q = r + 4 * GW * u + lr;
			bv[u] = q < mr ? load(q, cb) : zero<T>();
			av[u] = q < mr ? conjv(vb[q]) : zero<T>();
		}
		if (r < 8) av[0] = conjv(qr_v8(V, ldv, r + lr, lq, mr, nb));
#pragma unroll
		for (int u = 0; u < AC; u++) tile_mma(wv[u], av[u], bv[u]);
	}
#pragma unroll
	for (int u = AC / 2; u > 0; u /= 2)
#pragma unroll
		for (int k = 0; k < u; k++)
#pragma unroll
			for (int e = 0; e < 2; e++) wv[k][e] += wv[k + u][e];
	sh.wred[w][8 * lq + 2 * lr] = wv[0][0];
	sh.wred[w][8 * lq + 2 * lr + 1] = wv[0][1];
	bar_panel<GW>();
	T y[2] = {zero<T>(), zero<T>()}, b[2];
#pragma unroll
	for (int h = 0; h < 2; h++) {
		const int kk = 4 * h + lr;
		T bs = sh.wred[0][8 * kk + lq];
#pragma unroll
		for (int q = 1; q < GW; q++) bs += sh.wred[q][8 * kk + lq];
		tile_mma(y, (kk <= lq && lq < nb) ? conjv(Tp[kk + 8 * lq]) : zero<T>(), bs);
	}
	tile_c_to_b(y, b, lane);
	b[0] = -b[0];
	b[1] = -b[1];
	const int c0 = min(2 * lr, ncol - 1), c1 = min(2 * lr + 1, ncol - 1);
	for (int r = 8 * w; r < mr; r += 8 * GW * RT) {
		T z[RT][2], va[RT][2];
#pragma unroll
		for (int u = 0; u < RT; u++) {
			const int q = r + 8 * GW * u + lq;
			const bool ok = q < mr;
			z[u][0] = ok ? load(q, c0) : zero<T>();
			z[u][1] = ok ? load(q, c1) : zero<T>();
#pragma unroll
			for (int h = 0; h < 2; h++) va[u][h] = ok ? V[q + ldv * (4 * h + lr)] : zero<T>();
		}
		if (r == 0) {
#pragma unroll
			for (int h = 0; h < 2; h++) va[0][h] = qr_v8(V, ldv, lq, 4 * h + lr, mr, nb);
		}
#pragma unroll
		for (int h = 0; h < 2; h++)
#pragma unroll
			for (int u = 0; u < RT; u++) tile_mma(z[u], va[u][h], b[h]);
#pragma unroll
		for (int u = 0; u < RT; u++) {
			const int q = r + 8 * GW * u + lq;
#pragma unroll
			for (int e = 0; e < 2; e++)
				if (q < mr && 2 * lr + e < ncol) store(q, 2 * lr + e, z[u][e]);
		}
	}
}

// T of the block of reflectors j0 .. j0+nb-1 stored below the diagonal of
// A (larft, forward columnwise): one warp
template <typename T, int NBK>
__device__ inline void qrb_block_t(const T *A, int ld, const T *tau, T *Tp, int N, int j0, int nb,
		int lane)
{
	for (int k = 0; k < nb; k++) {
		const int jk = j0 + k;
		T y[NBK];
#pragma unroll
		for (int m = 0; m < NBK; m++) y[m] = zero<T>();
		for (int r = jk + lane; r < N; r += 32) {
			const T vk = (r == jk) ? one<T>() : A[r + (size_t)ld * jk];
#pragma unroll
			for (int m = 0; m < NBK; m++)
				if (m < k) y[m] += conjv(A[r + (size_t)ld * (j0 + m)]) * vk;
		}
#pragma unroll
		for (int o = 16; o > 0; o >>= 1)
#pragma unroll
			for (int m = 0; m < NBK; m++) y[m] += shfl_xor(y[m], o);
		const T tk = tau[jk];
		if (lane < k) {
			T sm = zero<T>();
#pragma unroll
			for (int m = 0; m < NBK; m++)
				if (m >= lane && m < k) sm += Tp[lane + NBK * m] * y[m];
			Tp[lane + NBK * k] = -tk * sm;
		}
		if (lane == k) Tp[k + NBK * k] = tk;
		__syncwarp();
	}
}

// Q = H_0 ... H_{N-1} from the reflectors below the diagonal of A and the
// block factors Ts, accumulated backwards by blocks in place of A (block p
// acts on rows and columns >= j0 of the partial product, whose panel
// columns are still e_c there and whose rows j0..j1-1 are zero), then Q to
// global memory and the phase of det Q.  All warps of the CTA.  Per block:
// each thread moves its elements of the block's reflectors into Vb and
// resets them to e_c in the same pass; one barrier; the apply; one barrier.
// (A second buffer, filled while the previous block is applied, saves the
// first barrier but takes 9.5 KB more shared memory, which keeps a GEMM CTA
// of another lane from sharing the SM.)
template <typename T, int NW, int NBK, bool GM>
__device__ inline void qrb_form_q(const QrArgs<T> &a, int item, T *A, int ld, T *Vb, const T *Ts,
		const T *tau, const double *vv, int N)
{
	const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
	const int np = (N + NBK - 1) / NBK;
	for (int p = np - 1; p >= 0; p--) {
		const int j0 = p * NBK, nb = min(NBK, N - j0), j1 = j0 + nb, mr = N - j0;
		// element (j0 + q % mr, j0 + q / mr) of the panel, copied then reset
		for (int q = tid; q < nb * mr; q += blockDim.x) {
			const int k = q / mr, r = j0 + q - k * mr;
			T *e = A + r + (size_t)ld * (j0 + k);
			Vb[r - j0 + (size_t)ld * k] = *e;
			*e = (r == j0 + k) ? one<T>() : zero<T>();
		}
		for (int q = tid; q < nb * (N - j1); q += blockDim.x) {
			const int c = q / nb;
			A[j0 + q - c * nb + (size_t)ld * (j1 + c)] = zero<T>();
		}
		__syncthreads();
		reflect_cols<T, false, GM>(A + j0, ld, j0, N, Vb, ld, Ts + (size_t)p * NBK * NBK, mr, nb, w, NW, lane);
		__syncthreads();
	}
	T *Q = a.Q + (size_t)item * a.q_stride;
	for (int c = w; c < N; c += NW)
		for (int r = lane; r < N; r += 32) Q[r + (size_t)N * c] = A[r + (size_t)ld * c];
	if (w == 0 && a.qdet) {
		T ph = one<T>();
		for (int j = lane; j < N; j += 32) ph = ph * phase_of(one<T>() - tau[j] * vv[j]);
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) ph = ph * shfl_xor(ph, o);
		if (lane == 0) a.qdet[item] = ph;
	}
}

// pvt: the columns of X (rows when a.trans) in stable descending order of
// their norms, scaled by dc (greens.c:123-129); the ranks in (int *)Vb when
// a.trans.  vn: N doubles, Vb: 8 N elements of scratch.  All warps.
template <typename T, int NW, int RPL>
__device__ inline void qr_order(const QrArgs<T> &a, const T *X, const double *dc, int N, double *vn, int *pvt, T *Vb)
{
	constexpr int NBK = 8;
	const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
	if (a.trans) {
		// norms of X's rows: a warp's lanes take 32 rows, a warp every NW-th column,
		// the partial sums meet in Vb
		const int nrow = (N + 31) / 32, g = w / nrow, ng = min(NW / nrow, NBK);
		double *ps = (double *)Vb;
		const int c = (w - g * nrow) * 32 + lane;
		if (g < ng && c < N) {
			double s = 0.0;
#pragma unroll 4
			for (int r = g; r < N; r += ng) s += abs2(X[c + (size_t)N * r]);
			ps[g * N + c] = s;
		}
		__syncthreads();
		for (int q = tid; q < N; q += blockDim.x) {
			double s = 0.0;
			for (int k = 0; k < ng; k++) s += ps[k * N + q];
			vn[q] = dc ? s * dc[q] * dc[q] : s;
		}
	} else {
#pragma unroll 2
		for (int c = w; c < N; c += NW) {
			const double sc = dc ? dc[c] : 1.0;
			T e[RPL];
#pragma unroll
			for (int t = 0; t < RPL; t++) e[t] = lane + 32 * t < N ? X[lane + 32 * t + (size_t)N * c] : zero<T>();
			double s = 0.0;
#pragma unroll
			for (int t = 0; t < RPL; t++) s += abs2(e[t] * sc);
			s = warp_sum(s);
			if (lane == 0) vn[c] = s;
		}
	}
	__syncthreads();
	// stable descending order of the squared norms (greens.c:123-129); a NaN
	// norm ranks last so that the order stays a permutation
	for (int c = tid; c < N; c += blockDim.x) {
		double v = vn[c];
		if (!(v >= 0.0)) {
			v = -1.0;
			if (a.err) atomicOr(a.err, DQ_ERR_NAN);
		}
		int rank = 0;
#pragma unroll 4
		for (int o = 0; o < N; o++) {
			double u = vn[o];
			if (!(u >= 0.0)) u = -1.0;
			rank += (u > v) || (u == v && o < c);
		}
		pvt[rank] = c;
		if (a.trans) ((int *)Vb)[c] = rank;
	}
	__syncthreads();
}

template <typename T, int NW, int NBK, int RPL, bool GM>
__global__ void __launch_bounds__(NW * 32) k_qrb(QrArgs<T> a)
{
	const int item = blockIdx.x;
	if (item >= a.batch) return;
	const int N = a.N, ld = GM ? N : qrb_ld(N);
	const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
	const int np = (N + NBK - 1) / NBK;
	extern __shared__ __align__(16) unsigned char smraw[];
	// N columns, leading dimension ld, position order
	T *A = GM ? a.work + (size_t)item * a.w_stride : (T *)smraw;
	// copies of a panel's V (ld x NBK): one, in the global-memory form two
	T *Vb = GM ? (T *)smraw : A + (size_t)ld * N;
	T *tau = Vb + (GM ? 2 : 1) * (size_t)ld * NBK;   // N
	T *Ts = tau + N;                            // np blocks of NBK x NBK
	double *dsh = (double *)(Ts + (size_t)np * NBK * NBK);
	double *vv = dsh + N;                       // v^H v
	double *vn = vv + N;                        // squared column norms
	int *pvt = (int *)(vn + N);
	if (N > 32 * RPL) {
		if (tid == 0 && a.err) atomicOr(a.err, DQ_ERR_SIZE);
		return;
	}
	const T *X = a.X + (size_t)item * a.x_stride;
	const double *dc = a.dcol ? a.dcol + (size_t)item * a.d_stride : nullptr;

	qr_order<T, NW, RPL>(a, X, dc, N, vn, pvt, Vb);
	if (a.trans) {
		const int *rk = (const int *)Vb;
		for (int r = w; r < N; r += NW)
			for (int c = lane; c < N; c += 32)
				A[r + (size_t)ld * rk[c]] = conjv(X[c + (size_t)N * r]) * (dc ? dc[c] : 1.0);
	} else {
#pragma unroll 2
		for (int j = w; j < N; j += NW) {
			const int c = pvt[j];
			const double sc = dc ? dc[c] : 1.0;
			T e[RPL];
#pragma unroll
			for (int t = 0; t < RPL; t++) e[t] = lane + 32 * t < N ? X[lane + 32 * t + (size_t)N * c] : zero<T>();
#pragma unroll
			for (int t = 0; t < RPL; t++)
				if (lane + 32 * t < N) A[lane + 32 * t + (size_t)ld * j] = e[t] * sc;
		}
	}
	__syncthreads();

	// Panel p by warps 0..PW-1; then warps 0..GW-1 take its block reflector to
	// the next panel's columns and factor that panel while the other warps
	// take it to the rest.  In the global-memory form the next panel and the
	// reflectors pass through shared memory (two buffers).
	using ND = NextDepth<T, RPL>;
	constexpr int PW = QrbPanel<T, RPL>::PW, RP = QrbPanel<T, RPL>::RP, GW = 4;
	static_assert(NBK == 8 && PW <= GW && GW < NW, "panels of 8 columns, panel warps among the look-ahead's");
	__shared__ PanelShared<T, PW> sh;
	auto panel = [&](int p) {
		const int j0 = p * NBK, nb = min(NBK, N - j0);
		T *Aj = A + j0 + (size_t)ld * j0;
		T *Vj = GM ? Vb + (size_t)(p & 1) * ld * NBK : Aj;
		qr_panel8<T, PW, RP>(
			sh, N - j0, nb, w, lane, Ts + (size_t)p * NBK * NBK, tau + j0, dsh + j0, vv + j0,
			[&](int r, int c) { return (GM && p) ? Vj[r + (size_t)ld * c] : Aj[r + (size_t)ld * c]; },
			[&](int r, int c, T v) {
				if (c >= nb) return;
				Aj[r + (size_t)ld * c] = v;
				if (GM) Vj[r + (size_t)ld * c] = v;
			});
	};
	if (w < PW) panel(0);
	__syncthreads();
	for (int p = 0; p < np; p++) {
		const int j0 = p * NBK, nb = min(NBK, N - j0), j1 = j0 + nb, mr = N - j0;
		const T *Vp = GM ? Vb + (size_t)(p & 1) * ld * NBK : A + j0 + (size_t)ld * j0;
		const T *Tp = Ts + (size_t)p * NBK * NBK;
		if (w < GW) {
			if (j1 < N) {
				T *C = A + j0 + (size_t)ld * j1, *Vn = Vb + (size_t)((p + 1) & 1) * ld * NBK;
				reflect_next<T, GW, ND::AC, ND::RT>(
					sh, min(NBK, N - j1), Vp, ld, Tp, mr, nb, w, lane,
					[&](int r, int c) { return C[r + (size_t)ld * c]; },
					[&](int r, int c, T v) {
						if (GM && r >= NBK) Vn[r - NBK + (size_t)ld * c] = v;
						else C[r + (size_t)ld * c] = v;
					});
				bar_panel<GW>();
				if (w < PW) panel(p + 1);
			}
		} else {
			reflect_cols<T, true, GM>(A + j0, ld, j1 + NBK, N, Vp, ld, Tp, mr, nb, w - GW, NW - GW, lane);
		}
		__syncthreads();
	}

	// D^-1 R in position order (Rs) or in the original one (Tout), diag(R)
	// (0 -> 1) and the order
	for (int j = w; j < N; j += NW) {
		T *out = a.Tout ? a.Tout + (size_t)item * a.t_stride + (size_t)N * pvt[j]
		                : a.Rs + (size_t)item * a.r_stride + (size_t)N * j;
		for (int r = lane; r < N; r += 32) {
			const double dr = dsh[r] == 0.0 ? 1.0 : dsh[r];
			out[r] = (r <= j) ? A[r + (size_t)ld * j] / dr : zero<T>();
		}
	}
	for (int r = tid; r < N; r += blockDim.x) {
		a.dout[(size_t)item * a.dout_stride + r] = dsh[r] == 0.0 ? 1.0 : dsh[r];
		if (a.pvt) a.pvt[(size_t)item * a.p_stride + r] = pvt[r];
	}
	__syncthreads();

	qrb_form_q<T, NW, NBK, GM>(a, item, A, ld, Vb, Ts, tau, vv, N);
}

// ----------------------------------------------- the same over a cluster
//
// Few matrices that do not fit one SM's shared memory: the columns' 8-column
// blocks lie round robin over the shared memory of a cluster of P CTAs (block b
// in CTA b mod P).  A panel's owner factors it and writes its reflectors and T
// to every CTA; each takes them to its own columns, the next panel's owner
// with its first four warps on that panel; one cluster barrier per panel.  Q
// backwards: each CTA copies the next block's reflectors from their owner
// while the present block's are applied.
// Bound by the panels' chain of latencies; with the matrix in L2 one SM's traffic
// (64 bytes a cycle, three passes over the trailing columns per panel) is.  The
// launcher's rule carries both sides' times.

template <typename T>
size_t qrc_smem_bytes(int N, int P)
{
	const int np = (N + 7) / 8, ld = qrb_ld(N), nl = (np + P - 1) / P;
	return sizeof(T) * ((size_t)ld * 8 * nl + 2 * (size_t)ld * 8 + 2 * 64 + N) + sizeof(double) * 3 * (size_t)N
	       + sizeof(int) * (size_t)N + 64;
}

// p of CTA `rank` of the cluster
template <typename T>
__device__ inline T *cluster_peer(T *p, int rank)
{
	unsigned long long r;
	asm volatile("mapa.u64 %0, %1, %2;" : "=l"(r) : "l"((unsigned long long)p), "r"(rank));
	return (T *)r;
}

template <typename T, int NW, int RPL>
__global__ void __launch_bounds__(NW * 32) k_qrc(QrArgs<T> a, int P)
{
	constexpr int NBK = 8;
	const int item = blockIdx.x / P, rank = blockIdx.x % P;
	const int N = a.N, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
	const size_t ld = qrb_ld(N);
	const int np = (N + NBK - 1) / NBK, nl = (np + P - 1) / P;
	extern __shared__ __align__(16) unsigned char smraw[];
	T *A = (T *)smraw;                          // own blocks, 8 columns each
	T *Vb = A + ld * NBK * nl;                  // two panels' reflectors from their first row on
	T *Tb = Vb + 2 * ld * NBK;                  // their T
	T *tau = Tb + 2 * NBK * NBK;                // N
	double *dsh = (double *)(tau + N), *vv = dsh + N, *vn = vv + N;
	int *pvt = (int *)(vn + N);
	T *Tg = a.work + (size_t)item * a.w_stride; // every panel's T
	const T *X = a.X + (size_t)item * a.x_stride;
	const double *dc = a.dcol ? a.dcol + (size_t)item * a.d_stride : nullptr;
	auto cluster_sync = []() {
		asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
	};
	// first own block >= b; local column of a global one
	auto first = [&](int b) { return b <= rank ? 0 : (b - rank + P - 1) / P; };
	auto block = [&](int b) { return A + ld * NBK * (b / P); };

	qr_order<T, NW, RPL>(a, X, dc, N, vn, pvt, Vb);
	if (a.trans) {
		const int *rk = (const int *)Vb;
		for (int c = lane; c < N; c += 32) {
			const int j = rk[c], b = j / NBK;
			if (b % P != rank) continue;
			T *Aj = block(b) + ld * (j - b * NBK);
			const double sc = dc ? dc[c] : 1.0;
#pragma unroll 4
			for (int r = w; r < N; r += NW) Aj[r] = conjv(X[c + (size_t)N * r]) * sc;
		}
	} else {
#pragma unroll 2
		for (int lc = w; lc < NBK * nl; lc += NW) {
			const int j = (lc / NBK * P + rank) * NBK + lc % NBK;
			if (j >= N) continue;
			const int c = pvt[j];
			const double sc = dc ? dc[c] : 1.0;
			T e[RPL];
#pragma unroll
			for (int t = 0; t < RPL; t++) e[t] = lane + 32 * t < N ? X[lane + 32 * t + (size_t)N * c] : zero<T>();
#pragma unroll
			for (int t = 0; t < RPL; t++)
				if (lane + 32 * t < N) A[lane + 32 * t + ld * lc] = e[t] * sc;
		}
	}
	// also: every CTA of the cluster runs before the first remote write
	cluster_sync();

	using ND = NextDepth<T, RPL>;
	using D = ReflectDepth<T, false>;
	constexpr int PW = QrbPanel<T, RPL>::PW, RP = QrbPanel<T, RPL>::RP, GW = 4;
	static_assert(PW <= GW && GW < NW, "panel warps among the look-ahead's");
	__shared__ PanelShared<T, PW> sh;
	auto panel = [&](int p) {
		const int j0 = p * NBK, nb = min(NBK, N - j0);
		T *Aj = block(p) + j0, *V = Vb + (p & 1) * ld * NBK, *Tp = Tb + (p & 1) * NBK * NBK;
		qr_panel8<T, PW, RP>(
			sh, N - j0, nb, w, lane, Tp, tau + j0, dsh + j0, vv + j0,
			[&](int r, int c) { return Aj[r + ld * c]; },
			[&](int r, int c, T v) {
				if (c >= nb) return;
				Aj[r + ld * c] = v;
				for (int q = 0; q < P; q++) cluster_peer(V, q)[r + ld * c] = v;
			});
		if (w == PW - 1) {
			__syncwarp();
			for (int e = lane; e < NBK * NBK; e += 32) {
				if (e % NBK > e / NBK || e / NBK >= nb) continue;
				Tg[p * NBK * NBK + e] = Tp[e];
				for (int q = 0; q < P; q++)
					if (q != rank) cluster_peer(Tp, q)[e] = Tp[e];
			}
			if (lane < nb)
				for (int q = 0; q < P; q++)
					if (q != rank) {
						cluster_peer(tau, q)[j0 + lane] = tau[j0 + lane];
						cluster_peer(dsh, q)[j0 + lane] = dsh[j0 + lane];
						cluster_peer(vv, q)[j0 + lane] = vv[j0 + lane];
					}
		}
	};
	if (rank == 0 && w < PW) panel(0);
	cluster_sync();
	for (int p = 0; p < np; p++) {
		const int j0 = p * NBK, nb = min(NBK, N - j0), j1 = j0 + nb, mr = N - j0;
		const T *V = Vb + (p & 1) * ld * NBK, *Tp = Tb + (p & 1) * NBK * NBK;
		const bool next = j1 < N && (p + 1) % P == rank;
		if (next && w < GW) {
			T *C = block(p + 1) + j0;
			reflect_next<T, GW, ND::AC, ND::RT>(
				sh, min(NBK, N - j1), V, ld, Tp, mr, nb, w, lane,
				[&](int r, int c) { return C[r + ld * c]; },
				[&](int r, int c, T v) { C[r + ld * c] = v; });
			bar_panel<GW>();
			if (w < PW) panel(p + 1);
		} else {
			const int ns = next ? NW - GW : NW;
			for (int l = first(p + 2) + (next ? w - GW : w); l * P + rank < np; l += ns)
				reflect8<T, true, D::AC, D::LD, D::RT>(A + j0 + ld * NBK * l, ld, min(NBK, N - NBK * (l * P + rank)), V,
				                                ld, Tp, mr, nb, lane);
		}
		cluster_sync();
	}

	// D^-1 R in position order (Rs) or in the original one (Tout), diag(R)
	// (0 -> 1) and the order
	for (int lc = w; lc < NBK * nl; lc += NW) {
		const int j = (lc / NBK * P + rank) * NBK + lc % NBK;
		if (j >= N) continue;
		T *out = a.Tout ? a.Tout + (size_t)item * a.t_stride + (size_t)N * pvt[j]
		                : a.Rs + (size_t)item * a.r_stride + (size_t)N * j;
		for (int r = lane; r < N; r += 32) {
			const double dr = dsh[r] == 0.0 ? 1.0 : dsh[r];
			out[r] = (r <= j) ? A[r + ld * lc] / dr : zero<T>();
		}
	}
	if (rank == 0)
		for (int r = tid; r < N; r += NW * 32) {
			a.dout[(size_t)item * a.dout_stride + r] = dsh[r] == 0.0 ? 1.0 : dsh[r];
			if (a.pvt) a.pvt[(size_t)item * a.p_stride + r] = pvt[r];
		}

	// Q = H_0 ... H_{N-1} backwards in place of A (qrb_form_q)
	auto fetch = [&](int p) {
		const int j0 = p * NBK, nb = min(NBK, N - j0);
		const T *Aj = cluster_peer(block(p) + j0, p % P);
		T *V = Vb + (p & 1) * ld * NBK;
		for (int k = w & 7; k < nb; k += 8)
#pragma unroll 4
			for (int r = j0 + lane + 32 * (w >> 3); r < N; r += 64) V[r - j0 + ld * k] = Aj[r - j0 + ld * k];
		if (tid < NBK * NBK) Tb[(p & 1) * NBK * NBK + tid] = Tg[p * NBK * NBK + tid];
	};
	fetch(np - 1);
	cluster_sync();
	for (int p = np - 1; p >= 0; p--) {
		const int j0 = p * NBK, nb = min(NBK, N - j0), mr = N - j0;
		if (p % P == rank) {
			T *Aj = block(p) + j0;
			for (int k = w; k < nb; k += NW)
				for (int r = lane; r < mr; r += 32) Aj[r + ld * k] = (r == k) ? one<T>() : zero<T>();
		}
		for (int lc = NBK * first(p + 1) + w; lc < NBK * nl; lc += NW)
			if (lane < nb) A[j0 + lane + ld * lc] = zero<T>();
		if (p > 0) fetch(p - 1);
		__syncthreads();
		for (int l = first(p) + w; l * P + rank < np; l += NW)
			reflect8<T, false, D::AC, D::LD, D::RT>(A + j0 + ld * NBK * l, ld, min(NBK, N - NBK * (l * P + rank)),
			                                 Vb + (p & 1) * ld * NBK, ld, Tb + (p & 1) * NBK * NBK, mr, nb, lane);
		cluster_sync();
	}
	T *Q = a.Q + (size_t)item * a.q_stride;
	for (int lc = w; lc < NBK * nl; lc += NW) {
		const int j = (lc / NBK * P + rank) * NBK + lc % NBK;
		if (j >= N) continue;
		for (int r = lane; r < N; r += 32) Q[r + (size_t)N * j] = A[r + ld * lc];
	}
	if (rank == 0 && w == 0 && a.qdet) {
		T ph = one<T>();
		for (int j = lane; j < N; j += 32) ph = ph * phase_of(one<T>() - tau[j] * vv[j]);
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) ph = ph * shfl_xor(ph, o);
		if (lane == 0) a.qdet[item] = ph;
	}
}

// ----------------------------------------------- column-pivoted QR
//
// The QR_PIVOT factorisation (geqp3 as greens.c:97-101 calls it:
// column pivoting by the largest partial column norm, norms downdated as
// LAPACK dlaqp2 does and recomputed when cancellation makes the downdate
// unreliable), with the matrix in shared memory and columns swapped in
// place so that column j holds pivot position j.  Step j: warp 0 picks
// the pivot (first largest norm in position order, as idamax) from the
// per-warp first largest norms of the last update, exchanges the two
// columns with the pivot column kept in registers and forms the reflector
// there; all warps then update the remaining columns and their norms
// (qrp_update) and leave their own first largest norm for the next step.
// Q is formed from blocks of NBK reflectors as in k_qrb.
// Outputs: Q, T = D^-1 R P^T, diag(R) and the pivot order.

template <typename T, int NBK>
size_t qrp_smem_bytes(int N, bool gm = false)
{
	return qrb_smem_bytes<T, NBK>(N, gm) + sizeof(double) * (size_t)N + 16;
}

// Householder step j of the pivoted QR on the columns j+1 .. N-1: one column
// per 8 lanes, 4 columns per warp at a time (lane = 4 g + s: column slot s,
// rows j + g + 8 i), so that a column's products need three exchange levels;
// then each column's partial norm is downdated from its updated row j as
// LAPACK dlaqp2 does, or recomputed below row j when the downdate has lost
// too much.  The downdate n1 sqrt(1 - (|a_j| / n1)^2) is taken as
// sqrt((n1 - |a_j|)(n1 + |a_j|)) and its test tt (n1 / n2)^2 <= tol3z as
// (n1 - |a_j|)(n1 + |a_j|) <= tol3z n2^2: the same quantities without a
// division.  The loops over a lane's rows stop at the last row (a
// warp-uniform test), so late steps issue only the rows that remain.
// Returns this warp's first largest new norm among its columns (NaN ranks
// below every number, as -0.5) and its position, in every lane.
// MAXI >= ceil(N / 8); the real shared-memory forms keep the column in
// registers between the two passes (v is read again: its loads are shared by
// the four column slots of a warp).
template <typename T, int NW, int MAXI>
__device__ inline void qrp_update(T *A, int ld, int N, int j, T ct, double *vn1, double *vn2,
		double tol3z, double &best, int &bi, bool &nan_seen)
{
	constexpr bool CACHE = !is_cplx<T>::value && MAXI <= 20;
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, s = lane & 3, g = lane >> 2;
	const T *vj = A + (size_t)ld * j;
	auto vrow = [&](int r) { return (r < N) ? ((r == j) ? one<T>() : vj[r]) : zero<T>(); };
	best = -1.0;
	bi = N;
	const int nc = N - j - 1;
	for (int q0 = 4 * w; q0 < nc; q0 += 4 * NW) {
		const int q = q0 + s, c = j + 1 + q;
		const bool act = q < nc;
		// an idle slot reads column j+1 and writes nothing
		T *col = A + (size_t)ld * (act ? c : j + 1);
		T d0 = zero<T>(), d1 = zero<T>(), aj;
		double s2a = 0.0, s2b = 0.0;
		if constexpr (CACHE) {
			T x[MAXI];
#pragma unroll
			for (int i = 0; i < MAXI; i++) {
				if (j + 8 * i >= N) break;
				const int r = j + g + 8 * i;
				x[i] = (r < N) ? col[r] : zero<T>();
				if (i & 1) d1 += conjv(vrow(r)) * x[i];
				else d0 += conjv(vrow(r)) * x[i];
			}
			T d = d0 + d1;
			d += shfl_xor(d, 4);
			d += shfl_xor(d, 8);
			d += shfl_xor(d, 16);
			const T f = ct * d;
#pragma unroll
			for (int i = 0; i < MAXI; i++) {
				if (j + 8 * i >= N) break;
				const int r = j + g + 8 * i;
				x[i] -= vrow(r) * f;
				if (r < N) {
					if (act) col[r] = x[i];
					if (r > j) {
						if (i & 1) s2b += abs2(x[i]);
						else s2a += abs2(x[i]);
					}
				}
			}
			aj = shfl(x[0], s);
		} else {
			for (int r = j + g; r < N; r += 8) d0 += conjv(vrow(r)) * col[r];
			T d = d0;
			d += shfl_xor(d, 4);
			d += shfl_xor(d, 8);
			d += shfl_xor(d, 16);
			const T f = ct * d;
			T x0 = zero<T>();
			for (int r = j + g; r < N; r += 8) {
				const T y = col[r] - vrow(r) * f;
				if (act) col[r] = y;
				if (r > j) s2a += abs2(y);
				else x0 = y;
			}
			aj = shfl(x0, s);
		}
		double s2 = s2a + s2b;
		s2 += __shfl_xor_sync(0xffffffffu, s2, 4);
		s2 += __shfl_xor_sync(0xffffffffu, s2, 8);
		s2 += __shfl_xor_sync(0xffffffffu, s2, 16);
		if (act) {
			// every lane of the column computes the new norm; lane g = 0 stores it
			const double n1 = vn1[c], n2 = vn2[c];
			double nv = n1;
			if (n1 != 0.0) {
				const double aa = absv(aj);
				const double d2 = fmax(0.0, (n1 - aa) * (n1 + aa));
				if (d2 <= tol3z * n2 * n2) {
					nv = sqrt(s2);
					if (g == 0) vn2[c] = nv;
				} else {
					nv = sqrt(d2);
				}
				if (g == 0) vn1[c] = nv;
			}
			if (!(nv >= 0.0)) {
				nv = -0.5;
				nan_seen = true;
			}
			if (nv > best) {
				best = nv;
				bi = c;
			}
		}
	}
	// first largest over the warp's four column slots
#pragma unroll
	for (int o = 1; o <= 2; o <<= 1) {
		const double ob = __shfl_xor_sync(0xffffffffu, best, o);
		const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
		if (ob > best || (ob == best && oi < bi)) {
			best = ob;
			bi = oi;
		}
	}
}

// at most 96 registers a thread (48 K of the SM's 64 K for 512 threads), so
// that a GEMM CTA of another lane can share the SM with this one
template <typename T, int NW, int NBK, int RPL, bool GM>
__global__ void __maxnreg__(96) k_qrp(QrArgs<T> a)
{
	const int item = blockIdx.x;
	if (item >= a.batch) return;
	const int N = a.N, ld = GM ? N : qrb_ld(N);
	const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
	const int np = (N + NBK - 1) / NBK;
	extern __shared__ __align__(16) unsigned char smraw[];
	T *A = GM ? a.work + (size_t)item * a.w_stride : (T *)smraw;
	T *Vb = GM ? (T *)smraw : A + (size_t)ld * N;
	T *tau = Vb + (size_t)ld * NBK;
	T *Ts = tau + N;
	double *dsh = (double *)(Ts + (size_t)np * NBK * NBK);
	double *vv = dsh + N;
	double *vn1 = vv + N;                       // partial column norms
	int *pvt = (int *)(vn1 + N);                // original column at each position
	const size_t o2 = ((size_t)((unsigned char *)(pvt + N) - smraw) + 15) & ~(size_t)15;
	double *vn2 = (double *)(smraw + o2);       // norms at the last recompute
	if (N > 32 * RPL) {
		if (tid == 0 && a.err) atomicOr(a.err, DQ_ERR_SIZE);
		return;
	}
	// per warp: first largest candidate norm of its columns and its position
	__shared__ double s_best[NW];
	__shared__ int s_bi[NW];
	bool nan_seen = false;
	const T *X = a.X + (size_t)item * a.x_stride;
	{
		double best = -1.0;
		int bi = N;
		for (int c = w; c < N; c += NW) {
			double s = 0.0;
			for (int r = lane; r < N; r += 32) {
				const T v = X[r + (size_t)N * c];
				A[r + (size_t)ld * c] = v;
				s += abs2(v);
			}
			s = sqrt(warp_sum(s));
			if (lane == 0) {
				vn1[c] = s;
				vn2[c] = s;
				pvt[c] = c;
			}
			if (!(s >= 0.0)) {
				s = -0.5;
				nan_seen = true;
			}
			if (s > best) {
				best = s;
				bi = c;
			}
		}
		if (lane == 0) {
			s_best[w] = best;
			s_bi[w] = bi;
		}
	}
	__syncthreads();
	const double tol3z = sqrt(2.220446049250313e-16);
	for (int j = 0; j < N; j++) {
		if (w == 0) {
			// pivot: the first largest partial norm among positions j..N-1 (a
			// NaN norm ranks below every number but stays a candidate), from
			// the warps' partial results of the last update
			double best = lane < NW ? s_best[lane] : -1.0;
			int bi = lane < NW ? s_bi[lane] : N;
#pragma unroll
			for (int o = 16; o > 0; o >>= 1) {
				const double ob = __shfl_xor_sync(0xffffffffu, best, o);
				const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
				if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
			}
			const int pj = bi;
			// columns pj and j exchange places; the pivot column stays in
			// registers and becomes the reflector (dlarfg convention)
			T xp[RPL], xj[RPL];
#pragma unroll
			for (int t = 0; t < RPL; t++) {
				const int r = lane + 32 * t;
				xp[t] = (r < N) ? A[r + (size_t)ld * pj] : zero<T>();
				xj[t] = (r < N) ? A[r + (size_t)ld * j] : zero<T>();
			}
			if (pj != j) {
#pragma unroll
				for (int t = 0; t < RPL; t++) {
					const int r = lane + 32 * t;
					if (r < N) A[r + (size_t)ld * pj] = xj[t];
				}
				if (lane == 0) {
					const double t1 = vn1[j]; vn1[j] = vn1[pj]; vn1[pj] = t1;
					const double t2 = vn2[j]; vn2[j] = vn2[pj]; vn2[pj] = t2;
					const int t3 = pvt[j]; pvt[j] = pvt[pj]; pvt[pj] = t3;
				}
			}
			double sig = 0.0;
			T al = zero<T>();
#pragma unroll
			for (int t = 0; t < RPL; t++) {
				const int r = lane + 32 * t;
				if (r > j && r < N) sig += abs2(xp[t]);
				if (t == (j >> 5)) al = xp[t];
			}
			sig = warp_sum(sig);
			const T alpha = shfl(al, j & 31);
			T tj, scal;
			double beta;
			if (sig == 0.0 && im(alpha) == 0.0) {
				tj = zero<T>();
				beta = re(alpha);
				scal = zero<T>();
			} else {
				beta = -copysign(sqrt(abs2(alpha) + sig), re(alpha));
				tj = (from_re<T>(beta) - alpha) / beta;
				scal = one<T>() / (alpha - beta);
			}
			T *vj = A + (size_t)ld * j;
#pragma unroll
			for (int t = 0; t < RPL; t++) {
				const int r = lane + 32 * t;
				if (r < N) vj[r] = (r > j) ? xp[t] * scal : ((r == j) ? from_re<T>(beta) : xp[t]);
			}
			if (lane == 0) {
				tau[j] = tj;
				dsh[j] = beta;
				vv[j] = 1.0 + sig * abs2(scal);
			}
		}
		__syncthreads();
		// H_j^H = I - conj(tau) v v^H on every remaining column, then the
		// norm downdate from the updated row j
		double best;
		int bi;
		qrp_update<T, NW, 4 * RPL>(A, ld, N, j, conjv(tau[j]), vn1, vn2, tol3z, best, bi, nan_seen);
		if (lane == 0) {
			s_best[w] = best;
			s_bi[w] = bi;
		}
		__syncthreads();
	}
	if (nan_seen && a.err) atomicOr(a.err, DQ_ERR_NAN);
	// T = D^-1 R P^T: position j is original column pvt[j]
	for (int j = w; j < N; j += NW) {
		const int c = pvt[j];
		for (int r = lane; r < N; r += 32) {
			const double dr = dsh[r] == 0.0 ? 1.0 : dsh[r];
			a.Tout[(size_t)item * a.t_stride + r + (size_t)N * c] =
				(r <= j) ? A[r + (size_t)ld * j] / dr : zero<T>();
		}
	}
	for (int r = tid; r < N; r += blockDim.x) {
		a.dout[(size_t)item * a.dout_stride + r] = dsh[r] == 0.0 ? 1.0 : dsh[r];
		if (a.pvt) a.pvt[(size_t)item * a.p_stride + r] = pvt[r];
	}
	for (int p = w; p < np; p += NW)
		qrb_block_t<T, NBK>(A, ld, tau, Ts + (size_t)p * NBK * NBK, N, p * NBK, min(NBK, N - p * NBK), lane);
	__syncthreads();
	qrb_form_q<T, NW, NBK, GM>(a, item, A, ld, Vb, Ts, tau, vv, N);
}

template <typename T>
struct RecArgs {
	int N, batch;
	const T *Q; long long q_stride;
	const T *Tm; long long t_stride;
	const double *d; long long d_stride;
	const T *qdet;
	// two-sided form: the product is Q D T (T_L^H D_L Q_L^H); Wl = Q^H Q_L, Tm =
	// T T_L^H, dl = D_L, and G receives D_Lb^-1 Z (the Q_L on its left follows)
	const T *Wl; long long wl_stride;
	const double *dl; long long dl_stride;
	const T *qdetl;
	T *G; long long g_stride;
	T *phase;                 // per item: 1 / phase(det G)
	double *logdet;           // per item, optional: log |det(I + B...B)| = -log |det G|
	T *work; long long w_stride;   // N x N per item, global-memory form only
	unsigned *err;
};

// ----------------------------------------------- recombine
//
// G = (D_b^-1 Q^H + D_s T)^-1 D_b^-1 Q^H (greens.c:157-178), or its two-sided
// form, one CTA per item with M in shared memory (GM: in global memory):
//   * LU with partial pivoting in panels of 8 columns (getrf; the pivot is the
//     first largest entry, see pivot_mag).  The panel's warps hold it in registers,
//     rows in place with their positions beside them.  A column costs one
//     barrier among them: each warp leaves its candidate row in shared memory
//     before it, and takes the winner's row from there after it.  They write
//     the panel back in pivoted order and list the rows that moved.  The other
//     warps meanwhile apply the previous panel to their tiles of 8 columns: the
//     moved rows, the rows of U (substitution), the trailing rows by DMMA
//     (one-panel look-ahead: the panel's warps bring its columns up to date in
//     registers);
//   * the 8 x 8 diagonal blocks of L and U are inverted in place, so that the
//     solves have no divisions and no substitution;
//   * each warp solves for 8 right-hand sides at a time, L and U by DMMA on
//     tiles of 8 rows, solved tiles in a slab of shared memory (rec_solve8);
//   * the phase 1/phase(det G) = phase(det Q) phase(det M) sign(prod v).
// What bounds it: the panels' chain (N columns in turn), then the solve's
// chains, of which the slabs that fit beside M limit how many run at once.
// Two items, N = 144: 175 us a launch (LU 183k cycles, solves 130k), against 419 us
// for an unblocked LU with a barrier per column and solves with substitution
// in the diagonal blocks; 512 items 0.75 ms against 1.77; N = 256 (M in L2)
// 1.09 ms against 6.0; complex N = 100 0.27 ms for 128 items
// against 0.59.

// The magnitude a pivot is chosen by: the modulus, for complex scalars within 8%
// of it (the octagon's norm; an infinity or a NaN stays one).  |re| + |im|, up to
// 41% off, lets multipliers grow to 1.41: G of well-conditioned complex products 1
// to 2% further from the exact one.  hypot as in the unblocked LU costs 10% of
// the launch at N = 64.
__device__ inline double pivot_mag(double a) { return fabs(a); }
__device__ inline double pivot_mag(zd a)
{
	const double x = fabs(a.x), y = fabs(a.y);
	const bool xl = x >= y;
	return fma(0.41421356, xl ? y : x, xl ? x : y);
}

// the warps of a panel: one up to N = 64, else four; up to two rows a lane
template <int RPL>
struct LuPanel {
	static constexpr int PW = RPL <= 2 ? 1 : 4;
	static constexpr int RP = (RPL + PW - 1) / PW;
};
constexpr int LU_PB = 8;

// the rows a panel moved: row src of the other columns goes to row dst
struct LuMoves {
	int n;
	int src[16], dst[16];
};

// what a panel's warps share: the rows of U above it, their candidate rows
// (two buffers)
template <typename T>
struct __align__(16) LuCand {
	T u[LU_PB][LU_PB];              // rows of U in a panel's columns
	T row[2][4][LU_PB];
	unsigned long long key[2][4];
	int pos[2][4];
};

// a panel's moved rows in the columns c0 .. c0+7 (those < cend), one warp
template <typename T>
__device__ inline void lu_move_tile(T *M, int ld, int c0, int cend, const LuMoves &mv, int lane)
{
	const int c = c0 + (lane & 7), n = mv.n;
	T v[4];
#pragma unroll
	for (int i = 0; i < 4; i++) {
		const int m = (lane >> 3) + 4 * i;
		if (m < n && c < cend) v[i] = M[mv.src[m] + (size_t)ld * c];
	}
	__syncwarp();
#pragma unroll
	for (int i = 0; i < 4; i++) {
		const int m = (lane >> 3) + 4 * i;
		if (m < n && c < cend) M[mv.dst[m] + (size_t)ld * c] = v[i];
	}
	__syncwarp();
}

// named barrier 1 of the panel's warps
template <int PW>
__device__ inline void bar_lu()
{
	if (PW > 1) asm volatile("barrier.sync 1, %0;\n" ::"n"(PW * 32) : "memory");
	else __syncwarp();
}

// LU of the panel of columns j0 .. j0+pb-1 (pb <= 8), rows j0 .. N-1, by the
// warps w < PW: lane l of warp w holds the rows j0 + l + 32 (w + PW t).  With
// mp (the moved rows of the panel before, 8 columns from j0 - 8) its columns
// are brought up to date first, in the registers that then hold the panel.
template <typename T, int RPL>
__device__ inline void lu_panel(T *M, int ld, int N, int j0, int pb, int *ipiv, LuMoves &mv,
		const LuMoves *mp, LuCand<T> &cd, int w, int lane, bool &nan_seen, bool &sing)
{
	constexpr int PW = LuPanel<RPL>::PW, RP = LuPanel<RPL>::RP, PB = LU_PB;
	T x[RP][PB];
	int pos[RP];
	unsigned used = 0;
	// the row slots that reach into the matrix (the same for the whole warp)
	const int nslot = min(RP, (N - j0 - 32 * w + 32 * PW - 1) / (32 * PW));
	if (w == 0 && lane == 0) mv.n = 0;
	if (mp) {
		if (w == 0) {
			lu_move_tile(M, ld, j0, j0 + pb, *mp, lane);
			// the rows of U: lane c column j0 + c
			const int i0 = j0 - PB, c = lane & 7;
			T u[PB];
#pragma unroll
			for (int i = 0; i < PB; i++) u[i] = c < pb ? M[i0 + i + (size_t)ld * (j0 + c)] : zero<T>();
#pragma unroll
			for (int k = 0; k < PB - 1; k++)
#pragma unroll
				for (int i = k + 1; i < PB; i++) u[i] -= M[i0 + i + (size_t)ld * (i0 + k)] * u[k];
			if (lane < 8) {
#pragma unroll
				for (int i = 0; i < PB; i++) {
					cd.u[i][c] = u[i];
					if (c < pb) M[i0 + i + (size_t)ld * (j0 + c)] = u[i];
				}
			}
		}
		bar_lu<PW>();
	}
#pragma unroll
	for (int t = 0; t < RP; t++) {
		const int r = j0 + lane + 32 * (w + PW * t);
		pos[t] = r;
		if (r >= N) used |= 1u << t;
#pragma unroll
		for (int c = 0; c < PB; c++) x[t][c] = (r < N && c < pb) ? M[r + (size_t)ld * (j0 + c)] : zero<T>();
		if (mp && t < nslot) {
			T l[PB];
#pragma unroll
			for (int k = 0; k < PB; k++) l[k] = r < N ? M[r + (size_t)ld * (j0 - PB + k)] : zero<T>();
#pragma unroll
			for (int k = 0; k < PB; k++)
#pragma unroll
				for (int c = 0; c < PB; c++) x[t][c] -= l[k] * cd.u[k][c];
		}
	}
#pragma unroll
	for (int k = 0; k < PB; k++) {
		if (k >= pb) break;
		// first largest of this warp's unused rows: by the bits of the magnitude
		// (a NaN ranks last), then by position
		unsigned long long best = 0;
		int bp = 0x7fffffff, bt = 0;
#pragma unroll
		for (int t = 0; t < RP; t++) {
			if (t >= nslot) break;
			const double m = pivot_mag(x[t][k]);
			const bool num = m >= 0.0, ok = !(used >> t & 1u);
			if (ok && !num) nan_seen = true;
			const unsigned long long key = num ? (unsigned long long)__double_as_longlong(m) : 0ull;
			if (ok && (key > best || (key == best && pos[t] < bp))) {
				best = key;
				bp = pos[t];
				bt = t;
			}
		}
		const unsigned hi = (unsigned)(best >> 32), lo = (unsigned)best;
		const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
		const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
		int q = __reduce_min_sync(0xffffffffu, (hi == mh && lo == ml) ? bp : 0x7fffffff);
		if (bp == q) {
			// its owner (every lane without rows when the warp has none left)
#pragma unroll
			for (int c = 0; c < PB; c++)
				if (c >= k) cd.row[k & 1][w][c] = (RP > 1 && bt) ? x[RP - 1][c] : x[0][c];
			cd.key[k & 1][w] = best;
			cd.pos[k & 1][w] = bp;
		}
		bar_lu<PW>();
		int ww = 0;
		unsigned long long bk = cd.key[k & 1][0];
		q = cd.pos[k & 1][0];
#pragma unroll
		for (int v = 1; v < PW; v++) {
			const unsigned long long kv = cd.key[k & 1][v];
			const int pv_ = cd.pos[k & 1][v];
			if (kv > bk || (kv == bk && pv_ < q)) {
				bk = kv;
				q = pv_;
				ww = v;
			}
		}
		T pv[PB];
#pragma unroll
		for (int c = 0; c < PB; c++)
			if (c >= k) pv[c] = cd.row[k & 1][ww][c];
		T piv = pv[k];
		if (re(piv) == 0.0 && im(piv) == 0.0) {
			sing = true;
			piv = one<T>();
		}
		const T ip = one<T>() / piv;
		// positions: the pivot row to j, the row that was there to the pivot's
		const int j = j0 + k;
		if (w == 0 && lane == 0) ipiv[j] = q;
#pragma unroll
		for (int t = 0; t < RP; t++) {
			if (t >= nslot) break;
			const bool mine = pos[t] == q;
			if (pos[t] == j) pos[t] = q;
			if (mine) {
				pos[t] = j;
				used |= 1u << t;
			}
			if (!(used >> t & 1u)) {
				x[t][k] = x[t][k] * ip;
#pragma unroll
				for (int c = 0; c < PB; c++)
					if (c > k) x[t][c] -= x[t][k] * pv[c];
			}
		}
	}
#pragma unroll
	for (int t = 0; t < RP; t++) {
		if (t >= nslot) break;
		const int r = j0 + lane + 32 * (w + PW * t);
		if (r < N) {
#pragma unroll
			for (int c = 0; c < PB; c++)
				if (c < pb) M[pos[t] + (size_t)ld * (j0 + c)] = x[t][c];
		}
		const bool moved = r < N && pos[t] != r;
		const unsigned m = __ballot_sync(0xffffffffu, moved);
		int i = 0;
		if (m && lane == 0) i = atomicAdd(&mv.n, __popc(m));
		i = __shfl_sync(0xffffffffu, i, 0) + __popc(m & ((1u << lane) - 1u));
		if (moved) {
			mv.src[i] = r;
			mv.dst[i] = pos[t];
		}
	}
}

// the rows j0 .. j0+pb-1 of U in the columns c0 .. c0+7 (those < N) right of
// the panel, from the moved rows by substitution, one warp; returns them as a
// B operand
template <typename T>
__device__ inline void lu_u_rows(T *M, int ld, int N, int j0, int pb, int c0, int lane, T (&b)[2])
{
	constexpr int PB = LU_PB;
	const int lr = lane & 3, lq = lane >> 2, cc = c0 + 2 * lr;
	const bool in = lq < pb;
	T l[PB - 1], u[2];
#pragma unroll
	for (int q = 0; q < PB - 1; q++) l[q] = (in && q < lq) ? M[j0 + lq + (size_t)ld * (j0 + q)] : zero<T>();
#pragma unroll
	for (int e = 0; e < 2; e++) u[e] = (in && cc + e < N) ? M[j0 + lq + (size_t)ld * (cc + e)] : zero<T>();
#pragma unroll
	for (int q = 0; q < PB - 1; q++) {
		const T y0 = shfl(u[0], 4 * q + lr), y1 = shfl(u[1], 4 * q + lr);
		u[0] -= l[q] * y0;
		u[1] -= l[q] * y1;
	}
#pragma unroll
	for (int e = 0; e < 2; e++)
		if (in && cc + e < N) M[j0 + lq + (size_t)ld * (cc + e)] = u[e];
	tile_c_to_b(u, b, lane);
}

// M -= L U on the rows from j0 + pb on of the columns c0 .. c0+7, one warp.  A
// complex term adds its two real products one after the other, two roundings at
// M's size where a scalar update has one, so a complex tile sums L U by itself and
// adds it to M once (N = 100 x 128 257 -> 273 us a launch; G of well-conditioned
// complex products 3 to 5% closer to the exact one).
template <typename T>
__device__ inline void lu_trail(T *M, int ld, int N, int j0, int pb, int c0, const T (&b)[2], int lane)
{
	constexpr bool SUM = is_cplx<T>::value;
	constexpr int RT = is_cplx<T>::value ? 2 : 3;   // row tiles at a time
	const int lr = lane & 3, lq = lane >> 2, cc = c0 + 2 * lr;
	for (int r0 = j0 + pb; r0 < N; r0 += 8 * RT) {
		T x[RT][2], a[RT][2];
		T *Mx = M + r0 + lq + (size_t)ld * cc;
		const T *Ma = M + r0 + lq + (size_t)ld * (j0 + lr);
#pragma unroll
		for (int i = 0; i < RT; i++) {
			const bool in = r0 + 8 * i + lq < N;
#pragma unroll
			for (int e = 0; e < 2; e++) x[i][e] = (!SUM && in && cc + e < N) ? Mx[8 * i + ld * e] : zero<T>();
#pragma unroll
			for (int s = 0; s < 2; s++) a[i][s] = (in && 4 * s + lr < pb) ? -Ma[8 * i + ld * 4 * s] : zero<T>();
		}
#pragma unroll
		for (int s = 0; s < 2; s++)
#pragma unroll
			for (int i = 0; i < RT; i++) tile_mma(x[i], a[i][s], b[s]);
#pragma unroll
		for (int i = 0; i < RT; i++) {
			const bool in = r0 + 8 * i + lq < N;
#pragma unroll
			for (int e = 0; e < 2; e++)
				if (in && cc + e < N) Mx[8 * i + ld * e] = SUM ? Mx[8 * i + ld * e] + x[i][e] : x[i][e];
		}
	}
	__syncwarp();
}

// inverse in place of an 8 x 8 diagonal block: of unit lower L (below the
// diagonal) or of U (on and above it), one warp, lane c < 8 column c
template <typename T, bool LOWER>
__device__ inline void tri_invert8(T *M, int ld, int N, int j0, int lane)
{
	const int c = lane & 7;
	T x[8];
	if (LOWER) {
#pragma unroll
		for (int i = 0; i < 8; i++) {
			T v = (i == c) ? one<T>() : zero<T>();
#pragma unroll
			for (int k = 0; k < i; k++) {
				const T l = (j0 + i < N) ? M[j0 + i + (size_t)ld * (j0 + k)] : zero<T>();
				v -= l * x[k];
			}
			x[i] = v;
		}
	} else {
		T d = (j0 + c < N) ? M[j0 + c + (size_t)ld * (j0 + c)] : one<T>();
		if (re(d) == 0.0 && im(d) == 0.0) d = one<T>();
		d = one<T>() / d;
#pragma unroll
		for (int i = 7; i >= 0; i--) {
			T v = (i == c) ? one<T>() : zero<T>();
#pragma unroll
			for (int k = 7; k > i; k--) {
				const T u = (j0 + k < N) ? M[j0 + i + (size_t)ld * (j0 + k)] : zero<T>();
				v -= u * x[k];
			}
			x[i] = v * shfl(d, i);
		}
	}
	__syncwarp();
#pragma unroll
	for (int i = 0; i < 8; i++)
		if (lane < 8 && j0 + i < N && j0 + c < N && (LOWER ? i > c : i <= c)) M[j0 + i + (size_t)ld * (j0 + c)] = x[i];
}

// The two triangular solves for the right-hand sides c0 .. c0+7 (those < N),
// one warp: Y = D_b^-1 Q^H with the LU's row order (perm), then L and U from M,
// whose 8 x 8 diagonal blocks are inverted.  Rows go by tiles of 8: the
// product of a tile's row of L (or U) with the tiles already solved is a chain
// of DMMAs (two accumulators), the diagonal block one product more.  Solved
// tiles are kept in the B-fragment layout (lane: rows 4s + l%4, column l/4)
// in ys, this warp's slab of 64 ceil(N/8) numbers in shared memory, each lane
// reading back only what it wrote.  osc: factors of the solution's rows on
// output (null: none).  UN: tiles whose loads are on their way together.
template <typename T, int UN>
__device__ inline void rec_solve8(const T *M, int ld, const int *perm, const double *vsh, const T *Q,
		T *G, int N, int c0, int lane, T *ys, const double *osc)
{
	const int lr = lane & 3, lq = lane >> 2, cc = c0 + 2 * lr;
	const int nt = (N + 7) / 8;
	auto yb = [&](int u, int s) -> T & { return ys[64 * u + 32 * s + lane]; };
	// rows past N take row N - 1's entries of M: their results stay finite and
	// are not used (their columns of L and U count as zero)
	T xn[2];
	double vn;
	auto rhs = [&](int t) {
		const int pr = perm[min(8 * t + lq, N - 1)];
		vn = vsh[pr];
#pragma unroll
		for (int e = 0; e < 2; e++) xn[e] = Q[min(cc + e, N - 1) + (size_t)N * pr];
	};
	rhs(0);
#pragma unroll 1
	for (int t = 0; t < nt; t++) {
		const T *Mr = M + min(8 * t + lq, N - 1) + (size_t)ld * lr;
		const T x0 = conjv(xn[0]) * vn, x1 = conjv(xn[1]) * vn;
		T a0[2] = {zero<T>(), zero<T>()}, a1[2] = {zero<T>(), zero<T>()}, b[2];
		T y[2] = {zero<T>(), zero<T>()};
		if (t + 1 < nt) rhs(t + 1);
		// the diagonal block's inverse, on its way meanwhile
		const T *Md = Mr + (size_t)ld * 8 * t;
		const bool in = 8 * t + lq < N;
		T ld0 = (in && lr < lq) ? Md[0] : zero<T>(), ld1 = (in && lr + 4 < lq) ? Md[(size_t)ld * 4] : zero<T>();
		if (lr == lq) ld0 = one<T>();
		if (lr + 4 == lq) ld1 = one<T>();
#pragma unroll UN
		for (int u = 0; u < t; u++) {
			const T l0 = Mr[0], l1 = Mr[(size_t)ld * 4];
			Mr += (size_t)ld * 8;
			tile_mma(a0, l0, yb(u, 0));
			tile_mma(a1, l1, yb(u, 1));
		}
		a0[0] = x0 - (a0[0] + a1[0]);
		a0[1] = x1 - (a0[1] + a1[1]);
		tile_c_to_b(a0, b, lane);
		tile_mma(y, ld0, b[0]);
		tile_mma(y, ld1, b[1]);
		tile_c_to_b(y, b, lane);
		yb(t, 0) = b[0];
		yb(t, 1) = b[1];
	}
#pragma unroll 1
	for (int t = nt - 1; t >= 0; t--) {
		const int r = 8 * t + lq;
		const T *Md = M + min(r, N - 1) + (size_t)ld * (8 * t + lr), *Mr = Md + (size_t)ld * 8;
		T a0[2] = {zero<T>(), zero<T>()}, a1[2] = {zero<T>(), zero<T>()}, b[2] = {yb(t, 0), yb(t, 1)};
		T y[2] = {zero<T>(), zero<T>()}, x[2];
		const T ud0 = (lr >= lq && 8 * t + lr < N) ? Md[0] : zero<T>();
		const T ud1 = (lr + 4 >= lq && 8 * t + lr + 4 < N) ? Md[(size_t)ld * 4] : zero<T>();
		tile_b_to_c(b, x, lane);
		// columns past N: only in the last tile
#pragma unroll UN
		for (int u = t + 1; u < nt - 1; u++) {
			const T u0 = Mr[0], u1 = Mr[(size_t)ld * 4];
			Mr += (size_t)ld * 8;
			tile_mma(a0, u0, yb(u, 0));
			tile_mma(a1, u1, yb(u, 1));
		}
		if (t + 1 < nt) {
			const int k = 8 * (nt - 1) + lr;
			const T u0 = k < N ? Mr[0] : zero<T>(), u1 = k + 4 < N ? Mr[(size_t)ld * 4] : zero<T>();
			tile_mma(a0, u0, yb(nt - 1, 0));
			tile_mma(a1, u1, yb(nt - 1, 1));
		}
		a0[0] = x[0] - (a0[0] + a1[0]);
		a0[1] = x[1] - (a0[1] + a1[1]);
		tile_c_to_b(a0, b, lane);
		tile_mma(y, ud0, b[0]);
		tile_mma(y, ud1, b[1]);
		if (r < N) {
			const double f = osc ? osc[r] : 1.0;
			if (cc < N) G[r + (size_t)N * cc] = y[0] * f;
			if (cc + 1 < N) G[r + (size_t)N * (cc + 1)] = y[1] * f;
		}
		tile_c_to_b(y, b, lane);
		yb(t, 0) = b[0];
		yb(t, 1) = b[1];
	}
}

// shared memory: M (unless in global memory), the scale vectors, pivots, row
// order and move lists, then the solve slabs of rec_solve_warps warps, as many
// as fit under RECB_SMEM_CAP, at least one
constexpr size_t RECB_SMEM_CAP = 226 * 1024;

template <typename T>
__host__ __device__ inline size_t recb_base_bytes(int N, bool gm)
{
	// a multiple of 16 bytes, where the solve slabs start
	return ((gm ? 0 : sizeof(T) * (size_t)qrb_ld(N) * N) + sizeof(double) * 2 * (size_t)N
	        + sizeof(int) * 2 * (size_t)N + 2 * sizeof(LuMoves) + sizeof(LuCand<T>) + 64 + 31) & ~(size_t)15;
}

template <typename T>
__host__ __device__ inline size_t recb_slab_bytes(int N) { return sizeof(T) * 64 * (size_t)((N + 7) / 8); }

template <typename T>
__host__ __device__ inline int recb_solve_warps(int N, bool gm)
{
	const size_t base = recb_base_bytes<T>(N, gm), slab = recb_slab_bytes<T>(N);
	const size_t fit = base < RECB_SMEM_CAP ? (RECB_SMEM_CAP - base) / slab : 0;
	return fit < 1 ? 1 : (fit > 16 ? 16 : (int)fit);
}

template <typename T>
size_t recb_smem_bytes(int N, bool gm = false)
{
	return recb_base_bytes<T>(N, gm) + recb_slab_bytes<T>(N) * recb_solve_warps<T>(N, gm);
}

template <typename T, int NW, int RPL, bool GM>
__global__ void __launch_bounds__(NW * 32) k_recb(RecArgs<T> a)
{
	constexpr int PB = LU_PB, PW = LuPanel<RPL>::PW;
	const int item = blockIdx.x;
	if (item >= a.batch) return;
	const int N = a.N, ld = GM ? N : qrb_ld(N);
	const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
	extern __shared__ __align__(16) unsigned char smraw[];
	// N columns, leading dimension ld
	T *M = GM ? a.work + (size_t)item * a.w_stride : (T *)smraw;
	double *vsh = GM ? (double *)smraw : (double *)((T *)smraw + (size_t)ld * N);   // D_b^-1
	double *dss = vsh + N;                      // D_s, then (two-sided) D_Lb^-1
	int *ipiv = (int *)(dss + N);               // row swapped with row j at step j
	int *perm = ipiv + N;                       // row r of P Y is row perm[r] of Y
	LuMoves *mv = (LuMoves *)(perm + N);        // of panel p, by parity
	LuCand<T> &cd = *(LuCand<T> *)(((size_t)(mv + 2) + 15) & ~(size_t)15);
	if (N > 32 * RPL) {
		if (tid == 0 && a.err) atomicOr(a.err, DQ_ERR_SIZE);
		return;
	}
	const T *Q = a.Q + (size_t)item * a.q_stride;
	const T *Tm = a.Tm + (size_t)item * a.t_stride;
	const double *d = a.d + (size_t)item * a.d_stride;
	for (int r = tid; r < N; r += blockDim.x) {
		const double dr = d[r];
		if (fabs(dr) > 1.0) { vsh[r] = 1.0 / dr; dss[r] = 1.0; }
		else { vsh[r] = 1.0; dss[r] = dr; }
		perm[r] = r;
	}
	__syncthreads();
	const double *osc = nullptr;
	if (a.Wl) {
		// D_b^-1 (Q^H Q_L) D_Lb^-1 + D_s (T T_L^H) D_Ls
		const T *Wl = a.Wl + (size_t)item * a.wl_stride;
		const double *dl = a.dl + (size_t)item * a.dl_stride;
		for (int c = w; c < N; c += NW) {
			const double x = dl[c], vl = fabs(x) > 1.0 ? 1.0 / x : 1.0, sl = fabs(x) > 1.0 ? 1.0 : x;
			for (int r = lane; r < N; r += 32)
				M[r + (size_t)ld * c] = Wl[r + (size_t)N * c] * (vsh[r] * vl) + Tm[r + (size_t)N * c] * (dss[r] * sl);
		}
		__syncthreads();
		// D_s is spent: its place takes D_Lb^-1
		for (int r = tid; r < N; r += blockDim.x) dss[r] = fabs(dl[r]) > 1.0 ? 1.0 / dl[r] : 1.0;
		osc = dss;
	} else {
		for (int c = w; c < N; c += NW)
			for (int r = lane; r < N; r += 32)
				M[r + (size_t)ld * c] = conjv(Q[c + (size_t)N * r]) * vsh[r] + Tm[r + (size_t)N * c] * dss[r];
	}
	__syncthreads();

	bool nan_seen = false, sing = false;
	if (w < PW) lu_panel<T, RPL>(M, ld, N, 0, min(PB, N), ipiv, mv[0], nullptr, cd, w, lane, nan_seen, sing);
	__syncthreads();
	for (int j0 = 0, p = 0; j0 < N; j0 += PB, p++) {
		const int pb = min(PB, N - j0), j1 = j0 + pb;
		const LuMoves &m = mv[p & 1];
		if (w < PW) {
			if (j1 < N)
				lu_panel<T, RPL>(M, ld, N, j1, min(PB, N - j1), ipiv, mv[(p + 1) & 1], &m, cd, w, lane, nan_seen,
				                 sing);
		} else {
			if (w == NW - 1) {
				const int v = lane < m.n ? perm[m.src[lane & 15]] : 0;
				__syncwarp();
				if (lane < m.n) perm[m.dst[lane]] = v;
			}
			// tiles right of the next panel, then the columns left of this one
			const int nr = max(0, (N - (j1 + 8) + 7) / 8), nl = m.n ? (j0 + 7) / 8 : 0;
			for (int t = w - PW; t < nr + nl; t += NW - PW) {
				if (t < nr) {
					const int c0 = j1 + 8 + 8 * t;
					T b[2];
					lu_move_tile(M, ld, c0, N, m, lane);
					lu_u_rows<T>(M, ld, N, j0, pb, c0, lane, b);
					lu_trail<T>(M, ld, N, j0, pb, c0, b, lane);
				} else {
					lu_move_tile(M, ld, 8 * (t - nr), j0, m, lane);
				}
			}
		}
		__syncthreads();
	}
	// any panel warp may have met a NaN or a zero pivot
	if (w < PW) {
		nan_seen = __any_sync(0xffffffffu, nan_seen);
		sing = __any_sync(0xffffffffu, sing);
		if (lane == 0 && nan_seen && a.err) atomicOr(a.err, DQ_ERR_NAN);
		if (w == 0 && lane == 0 && sing && a.err) atomicOr(a.err, DQ_ERR_SINGULAR);
	}
	if (w == 0) {
		// phase(det) = phase(det Q) prod phase(U_jj) sign(prod v_j) (-1)^swaps,
		// each lane taking every 32nd j, then a butterfly over the warp
		T ph = one<T>();
		int neg = 0;
		double l = 0.0;
		for (int j = lane; j < N; j += 32) {
			const T u = M[j + (size_t)ld * j];
			ph = ph * phase_of(u);
			neg ^= (vsh[j] < 0.0) ^ (ipiv[j] != j) ^ (osc && osc[j] < 0.0);
			// G = M^-1 diag(v) Q^H: log |det G| = sum log |v_j| - sum log |U_jj|
			// (two-sided: and sum log |v_L,j|)
			if (a.logdet) l += log(absv(u)) - log(fabs(vsh[j])) - (osc ? log(fabs(osc[j])) : 0.0);
		}
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) {
			ph = ph * shfl_xor(ph, o);
			neg ^= __shfl_xor_sync(0xffffffffu, neg, o);
			l += __shfl_xor_sync(0xffffffffu, l, o);
		}
		if (lane == 0) {
			if (a.qdet) ph = a.qdet[item] * ph;
			if (osc && a.qdetl) ph = ph * conjv(a.qdetl[item]);
			a.phase[item] = neg ? ph * -1.0 : ph;
			if (a.logdet) a.logdet[item] = l;
		}
	}
	__syncthreads();
	const int nt = (N + 7) / 8;
	for (int t = w; t < 2 * nt; t += NW) {
		if (t < nt) tri_invert8<T, true>(M, ld, N, 8 * t, lane);
		else tri_invert8<T, false>(M, ld, N, 8 * (t - nt), lane);
	}
	__syncthreads();
	// right-hand sides Y = D_b^-1 Q^H, 8 columns per pass of a warp
	T *G = a.G + (size_t)item * a.g_stride;
	const int nws = min(NW, recb_solve_warps<T>(N, GM));
	T *ys = (T *)(smraw + recb_base_bytes<T>(N, GM)) + (size_t)64 * nt * w;
	for (int c0 = 8 * w; w < nws && c0 < N; c0 += 8 * nws)
		rec_solve8<T, GM ? 8 : 4>(M, ld, perm, vsh, Q, G, N, c0, lane, ys, osc);
}

}  // namespace dq
