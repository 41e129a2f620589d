// Unequal-time Green's functions G(0,t), G(t,t), G(t,0) for every slice t
// (reference src/greens.c:247-494, calc_ue_g), batched over the (chain,
// spin) items of a group.
//
//   calc_o   (greens.c:247-264)  block-cyclic O of the E = 1 + (F-1)/2
//                                pair products of the cluster matrices
//   bsofi    (greens.c:266-337)  O = Q R by Householder QRs of 2N-row
//                                panels, R^-1 by blocks, O^-1 = R^-1 Q^H
//   expand_g (greens.c:339-469)  the E x E blocks of O^-1 seed G at every
//                                2 n_matmul-th slice; chains of B_l / B_l^-1
//                                products fill the slices between
//
// Layouts: O and O^-1 are NE x NE per item (NE = N E), column-major.  The
// slice stacks (G0t, Gtt, Gt0 and the materialised B_l, B_l^-1) are
// slice-major, stack[l][item] N x N, so that one launch can take the same
// step of every group's chain through a table of slice indices.
#pragma once

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "gemm.cuh"
#include "qr.cuh"

namespace dq {

// B_l = exp_K diag(d_l) and B_l^-1 = diag(1/d_l) inv_exp_K for every slice
// and item (reference calcBu/iBu, dqmc.c:29-59); d per item [L][N]
template <typename T>
__global__ void k_build_bib(int N, int L, int NB, const T *expK, const T *iexpK,
		const double *dv, const double *dvi, T *Bs, T *iBs)
{
	const long long NN = (long long)N * N, tot = NN * NB * L;
	for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < tot;
	     q += (long long)gridDim.x * blockDim.x) {
		const long long e = q % NN, sb = q / NN;
		const int item = (int)(sb % NB), l = (int)(sb / NB);
		const int r = (int)(e % N), c = (int)(e / N);
		const long long s = (long long)(item & 1) * NN;
		const size_t dof = ((size_t)item * L + l) * N;
		Bs[q] = expK[s + e] * dv[dof + c];
		iBs[q] = iexpK[s + e] * dvi[dof + r];
	}
}

// dst_b = alpha src_b (rows x cols, leading dimensions lds / ldd), or the
// identity when src is null
template <typename T>
__global__ void k_copy2d(int rows, int cols, int NB, const T *src, long long ss, int lds, T *dst,
		long long ds, int ldd, T alpha)
{
	const long long per = (long long)rows * cols, tot = per * NB;
	for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < tot;
	     q += (long long)gridDim.x * blockDim.x) {
		const int b = (int)(q / per);
		const long long e = q % per;
		const int r = (int)(e % rows), c = (int)(e / rows);
		T v;
		if (src) v = alpha * src[b * ss + r + (long long)lds * c];
		else v = (r == c) ? one<T>() : zero<T>();
		dst[b * ds + r + (long long)ldd * c] = v;
	}
}

// diag += 1 on NB matrices n x n, item stride s
template <typename T>
__global__ void k_add_diag(int n, int NB, T *A, long long s)
{
	const long long tot = (long long)n * NB;
	for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < tot;
	     q += (long long)gridDim.x * blockDim.x) {
		const int b = (int)(q / n), i = (int)(q % n);
		T *p = A + b * s + i + (long long)n * i;
		*p = *p + 1.0;
	}
}

// ------------------------------------------------ Householder QR with Q^H
//
// One CTA per item factors an M x n panel (M >= n) in place, A = Q R,
// leaving R in the top n rows (zeros below), writing Q^H (M x M) and
// applying Q^H to `nx1` columns right of the panel and `nx2` columns at X
// (rows of the panel).  The reflectors are LAPACK's geqrf convention
// (zgeqr2/zlarfg: beta = -sign(Re alpha) ||x||); NBK of them at a time are
// factored in shared memory and applied to the trailing columns as one
// block reflector I - V T^H V^H (larft forward, columnwise), 8 columns per warp
// by DMMA (reflect8), so every trailing column is read twice and written once
// per block.
// Warps 0-3 take a panel's reflector to the next panel and factor that one
// (qr_panel8) while the others take it to the remaining columns.  Bound by
// latency: one CTA per item, M / 8 panels in series.  The class of one
// unequal-time measurement, one column per warp at first: 8x8, one chain, 1.58 ms
// with tiles alone, 0.77 ms with the register panels beside them; complex 10x10
// x 64 16.6 -> 11.0 ms.

template <typename T>
struct HqrArgs {
	int M, n, batch;
	T *A; Addr aA; int lda;
	int nx1, nx2;
	T *X; Addr aX;            // nx2 extra columns, leading dimension lda
	T *Qh; Addr aQ;           // M x M, leading dimension M
	unsigned *err;
};

// warps of a panel and the look-ahead's; leading dimension of the reflectors
// (4 mod 16: conflict-free tiles)
constexpr int HQR_PW = 4;
__host__ __device__ inline int hqr_ld(int M) { return (M + 11) / 16 * 16 + 4; }

template <typename T, int NBK>
size_t hqr_smem_bytes(int M)
{
	return sizeof(T) * (2 * (size_t)hqr_ld(M) * NBK + 2 * NBK * NBK + NBK) + sizeof(double) * 2 * NBK;
}

template <typename T, int NBK, int NW, int RP>
__global__ void __launch_bounds__(NW * 32) k_hqr(HqrArgs<T> a)
{
	const int item = blockIdx.x;
	if (item >= a.batch) return;
	const int M = a.M, n = a.n, ldv = hqr_ld(M);
	const size_t lda = a.lda;
	const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
	extern __shared__ __align__(16) unsigned char smraw[];
	T *Vb = (T *)smraw;                   // two panels from their first row on, ld ldv
	T *Tb = Vb + 2 * (size_t)ldv * NBK;   // their NBK x NBK block-reflector factors
	T *tau = Tb + 2 * NBK * NBK;
	double *beta = (double *)(tau + NBK), *vv = beta + NBK;
	__shared__ PanelShared<T, HQR_PW> sh;
	T *A = a.A + a.aA.off(item);
	T *Q = a.Qh + a.aQ.off(item);
	T *X2 = a.nx2 ? a.X + a.aX.off(item) : nullptr;
	if (n > M || M > 32 * HQR_PW * RP) {
		if (tid == 0) atomicOr(a.err, DQ_ERR_SIZE);
		return;
	}
	for (int q = tid; q < M * M; q += NW * 32) Q[q] = (q / M == q % M) ? one<T>() : zero<T>();
	// panel p from Vb, where the look-ahead left it (p > 0), or from A: V stays in
	// Vb, R goes to A with zeros below
	bool bad = false;
	auto panel = [&](int p) {
		const int j0 = p * NBK, nb = min(NBK, n - j0);
		T *Aj = A + j0 + lda * j0, *V = Vb + (size_t)(p & 1) * ldv * NBK;
		qr_panel8<T, HQR_PW, RP>(
			sh, M - j0, nb, w, lane, Tb + (p & 1) * NBK * NBK, tau, beta, vv,
			[&](int r, int c) { return p ? V[r + (size_t)ldv * c] : Aj[r + lda * c]; },
			[&](int r, int c, T v) {
				V[r + (size_t)ldv * c] = v;
				if (c < nb) Aj[r + lda * c] = (r <= c) ? v : zero<T>();
			});
		if (tid < nb && !(beta[tid] == beta[tid])) bad = true;
	};
	__syncthreads();
	if (w < HQR_PW) panel(0);
	__syncthreads();
	const int np = (n + NBK - 1) / NBK;
	for (int p = 0; p < np; p++) {
		const int j0 = p * NBK, nb = min(NBK, n - j0), j1 = j0 + nb, mr = M - j0;
		const T *V = Vb + (size_t)(p & 1) * ldv * NBK, *Tp = Tb + (p & 1) * NBK * NBK;
		const bool next = j1 < n;
		if (next && w < HQR_PW) {
			// the next panel's columns and that panel
			T *C = A + j0 + lda * j1, *Vn = Vb + (size_t)((p + 1) & 1) * ldv * NBK;
			using ND = NextDepth<T, 4 * RP>;
			reflect_next<T, HQR_PW, ND::AC, ND::RT>(
				sh, min(NBK, n - j1), V, ldv, Tp, mr, nb, w, lane,
				[&](int r, int c) { return C[r + lda * c]; },
				[&](int r, int c, T v) {
					if (r >= NBK) Vn[r - NBK + (size_t)ldv * c] = v;
					else C[r + lda * c] = v;
				});
			bar_panel<HQR_PW>();
			panel(p + 1);
		} else {
			// all other columns: of the panel and the nx1 right of it, X, Q
			const int slot = next ? w - HQR_PW : w, ns = next ? NW - HQR_PW : NW;
			const int c1 = min(j1 + NBK, n), n1 = n + a.nx1 - c1;
			const int t1 = (n1 + 7) / 8, t2 = (a.nx2 + 7) / 8, t3 = (M + 7) / 8;
			using D = ReflectDepth<T, true>;
			constexpr int AC = 8;          // of W: M = 2 N rows a sum
			for (int t = slot; t < t1 + t2 + t3; t += ns) {
				T *C;
				size_t ldc = lda;
				int left;
				if (t < t1) {
					C = A + j0 + lda * (c1 + 8 * t);
					left = n1 - 8 * t;
				} else if (t < t1 + t2) {
					C = X2 + j0 + lda * (8 * (t - t1));
					left = a.nx2 - 8 * (t - t1);
				} else {
					ldc = M;
					C = Q + j0 + ldc * (8 * (t - t1 - t2));
					left = M - 8 * (t - t1 - t2);
				}
				reflect8<T, true, AC, D::LD, D::RT>(C, ldc, min(8, left), V, ldv, Tp, mr, nb, lane);
			}
		}
		__syncthreads();
	}
	if (bad) atomicOr(a.err, DQ_ERR_NAN);
}

// ------------------------------------------------ triangular block inverse
//
// One CTA per (item, diagonal block e): X_ee = R_ee^-1 for the N x N upper
// triangular diagonal blocks of R (NE x NE per item, leading dimension NE),
// column by column: X[0:j, j] = -X[0:j, 0:j] R[0:j, j] / R[j, j].

template <typename T>
struct TriArgs {
	int N, NE, E, batch;
	const T *R;
	T *X;
	unsigned *err;
};

template <typename T>
size_t trtri_smem_bytes(int N)
{
	return sizeof(T) * ((size_t)N * N + N) + 64;
}

template <typename T>
__global__ void __launch_bounds__(256) k_trtri(TriArgs<T> a)
{
	const int item = blockIdx.x / a.E, e = blockIdx.x % a.E;
	if (item >= a.batch) return;
	const int N = a.N;
	const long long NE = a.NE;
	const size_t off = (size_t)item * NE * NE + (size_t)e * N * (1 + NE);
	const T *R = a.R + off;
	T *X = a.X + off;
	extern __shared__ __align__(16) unsigned char smraw[];
	T *S = (T *)smraw;
	T *rc = S + (size_t)N * N;
	bool bad = false;
	for (int j = 0; j < N; j++) {
		for (int i = threadIdx.x; i <= j; i += blockDim.x) rc[i] = R[i + NE * j];
		__syncthreads();
		const T xjj = one<T>() / rc[j];
		for (int i = threadIdx.x; i < N; i += blockDim.x) {
			T v;
			if (i < j) {
				T s = zero<T>();
				for (int k = i; k < j; k++) s += S[i + (size_t)N * k] * rc[k];
				v = -s * xjj;
			} else {
				v = (i == j) ? xjj : zero<T>();
			}
			S[i + (size_t)N * j] = v;
		}
		__syncthreads();
	}
	for (int q = threadIdx.x; q < N * N; q += blockDim.x) {
		const T v = S[q];
		if (!(abs2(v) == abs2(v)) || abs2(v) > 1e300) bad = true;
		X[(q % N) + NE * (q / N)] = v;
	}
	if (bad) atomicOr(a.err, DQ_ERR_SINGULAR);
}

// the blocks of O^-1 that seed the slice stacks (greens.c:353-357, 404-409,
// 437-442): G0t[e nme] = (0, e), Gtt[e nme] = (e, e), Gt0[e nme] = (e, 0)
template <typename T>
__global__ void k_ue_seed(int N, int E, int NB, int nme, const T *Gred, T *G0t, T *Gtt, T *Gt0)
{
	const long long NN = (long long)N * N, NE = (long long)N * E, tot = NN * E * NB;
	for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < tot;
	     q += (long long)gridDim.x * blockDim.x) {
		const long long el = q % NN;
		const int item = (int)((q / NN) % NB), e = (int)(q / (NN * NB));
		const int r = (int)(el % N), c = (int)(el / N);
		const T *g = Gred + (size_t)item * NE * NE;
		const size_t d = ((size_t)e * nme * NB + item) * NN + el;
		G0t[d] = g[r + NE * (c + (long long)N * e)];
		Gtt[d] = g[(r + (long long)N * e) + NE * (c + (long long)N * e)];
		Gt0[d] = g[(r + (long long)N * e) + NE * c];
	}
}

// ------------------------------------------------ the expand_g step plan
//
// Six chain kinds, each a sequence of (m, next) slice pairs per group:
//   0 G0t left   G0t[n] = a G0t[m] B[n]               a = -1 at m = 0
//   1 G0t right  G0t[n] = a G0t[m] iB[m] + b iB[m]     b = -1 at m = 0
//   2 Gtt up     Gtt[n] = iB[n] (Gtt[m] B[n])
//   3 Gtt down   Gtt[n] = B[m] (Gtt[m] iB[m])
//   4 Gt0 up     Gt0[n] = a iB[n] Gt0[m] + b iB[n]     a = -1, b = 1 at m = 0
//   5 Gt0 down   Gt0[n] = a B[m] Gt0[m] (+ I)          a = -1, + I at n = 0
// The steps with the ordinary coefficients of all groups go in one batched
// launch per (step, kind), through tables of slice indices; the few steps
// with other coefficients get launches of their own.

struct UeOp {
	int kind, nact;     // nact groups in this launch (1 for a special step)
	int tab;            // offset of 4 * nact ints: slices of A, B, C, D (D: 2nd GEMM's A)
	bool special;
	int m, next;
	double alpha, beta; // special steps only
	int prefill;        // special: 0 none, 1 iB[m], 2 iB[next], 3 identity
};

struct UePlan {
	int E = 0, nme = 0;
	std::vector<UeOp> ops;
	std::vector<int> tabs;

	static void coef(int kind, int m, int next, double &alpha, double &beta, int &prefill)
	{
		alpha = 1.0; beta = 0.0; prefill = 0;
		switch (kind) {
		case 0: if (m == 0) alpha = -1.0; break;
		case 1:
			if (next == 0) alpha = -1.0;
			if (m == 0) { beta = -alpha; prefill = 1; }
			break;
		case 4:
			if (m == 0) { alpha = -1.0; beta = 1.0; prefill = 2; }
			break;
		case 5:
			if (next == 0) { alpha = -1.0; beta = 1.0; prefill = 3; }
			break;
		default: break;
		}
	}

	// reference expand_g bounds (greens.c:339-352), with E = 1 + (F-1)/2
	// groups of nme = 2 L/F slices
	void build(int L, int F)
	{
		E = 1 + (F - 1) / 2;
		nme = (L / F) * 2;
		const int n_left = (nme - 1) / 2, n_right = nme / 2;
		const int rstop_last = ((E - 1) * nme + L) / 2;
		const int lstop_first = (rstop_last + 1) % L;
		// chains[kind][group] = (m, next) pairs
		std::vector<std::vector<std::pair<int, int>>> ch[6];
		int maxlen = 0;
		for (int kind = 0; kind < 6; kind++) {
			ch[kind].resize(E);
			const bool left = (kind % 2 == 0);
			for (int f = 0; f < E; f++) {
				const int l = f * nme;
				const int stop = left ? ((f == 0) ? lstop_first : l - n_left)
				                      : ((f == E - 1) ? rstop_last : l + n_right);
				int m = l;
				for (int it = 0; it < L && m != stop; it++) {
					const int nx = left ? (m - 1 + L) % L : (m + 1) % L;
					ch[kind][f].push_back({m, nx});
					m = nx;
				}
				maxlen = std::max(maxlen, (int)ch[kind][f].size());
			}
		}
		ops.clear();
		tabs.clear();
		for (int s = 0; s < maxlen; s++)
			for (int kind = 0; kind < 6; kind++) {
				std::vector<std::pair<int, int>> norm, spec;
				for (int f = 0; f < E; f++) {
					if ((int)ch[kind][f].size() <= s) continue;
					const auto pr = ch[kind][f][s];
					double al, be;
					int pf;
					coef(kind, pr.first, pr.second, al, be, pf);
					((al == 1.0 && be == 0.0) ? norm : spec).push_back(pr);
				}
				if (!norm.empty()) {
					UeOp o{};
					o.kind = kind; o.nact = (int)norm.size(); o.tab = (int)tabs.size();
					o.special = false;
					for (int k = 0; k < 4; k++)
						for (const auto &pr : norm) tabs.push_back(slice_of(kind, k, pr.first, pr.second));
					ops.push_back(o);
				}
				for (const auto &pr : spec) {
					UeOp o{};
					o.kind = kind; o.nact = 1; o.tab = -1; o.special = true;
					o.m = pr.first; o.next = pr.second;
					coef(kind, o.m, o.next, o.alpha, o.beta, o.prefill);
					ops.push_back(o);
				}
			}
	}

	// slice of operand k (0 A, 1 B, 2 C, 3 D) of a step of this kind
	static int slice_of(int kind, int k, int m, int nx)
	{
		switch (kind) {
		case 0: { const int s[4] = {m, nx, nx, 0}; return s[k]; }
		case 1: { const int s[4] = {m, m, nx, 0}; return s[k]; }
		case 2: { const int s[4] = {m, nx, nx, nx}; return s[k]; }
		case 3: { const int s[4] = {m, m, nx, m}; return s[k]; }
		case 4: { const int s[4] = {nx, m, nx, 0}; return s[k]; }
		default: { const int s[4] = {m, m, nx, 0}; return s[k]; }
		}
	}
};

// device buffers of the unequal-time computation of one group
template <typename T>
struct UneqState {
	// sizes the kernels here take: trtri keeps an N x N block in shared
	// memory, k_hqr a panel of 2N x 8
	static bool supported(int N, int F, int L)
	{
		const int nmax = is_cplx<T>::value ? 112 : 160;
		return N >= 1 && N <= nmax && F >= 1 && L >= 2 && L % F == 0;
	}
	struct Buf {
		T *p = nullptr;
		int alloc(size_t n)
		{
			if (cudaMalloc(&p, sizeof(T) * (n ? n : 1)) != cudaSuccess) { p = nullptr; return 1; }
			return 0;
		}
		void release() { if (p) cudaFree(p); p = nullptr; }
	};
	Buf G0t, Gtt, Gt0, Bs, iBs, O, Gr, Qh, Tw, Rw, Cw;
	int *dtab = nullptr;
	UePlan plan;
	int N = 0, L = 0, F = 0, NB = 0, E = 0, NE = 0;

	int alloc(int N_, int L_, int F_, int NB_)
	{
		N = N_; L = L_; F = F_; NB = NB_;
		plan.build(L, F);
		E = plan.E;
		NE = N * E;
		const size_t NN = (size_t)N * N, st = (size_t)L * NB * NN;
		int rc = 0;
		rc |= G0t.alloc(st); rc |= Gtt.alloc(st); rc |= Gt0.alloc(st);
		rc |= Bs.alloc(st); rc |= iBs.alloc(st);
		rc |= O.alloc((size_t)NB * NE * NE); rc |= Gr.alloc((size_t)NB * NE * NE);
		rc |= Qh.alloc((size_t)NB * std::max(E - 1, 1) * 4 * NN);
		rc |= Tw.alloc((size_t)NB * E * NN);
		rc |= Rw.alloc((size_t)NB * NE * 2 * N);
		rc |= Cw.alloc((size_t)NB * E * NN);
		if (rc) return 1;
		const size_t nt = plan.tabs.size();
		if (cudaMalloc(&dtab, sizeof(int) * (nt ? nt : 1)) != cudaSuccess) { dtab = nullptr; return 1; }
		if (nt && cudaMemcpy(dtab, plan.tabs.data(), sizeof(int) * nt, cudaMemcpyHostToDevice) != cudaSuccess)
			return 1;
		return 0;
	}
	void release()
	{
		Buf *b[] = {&G0t, &Gtt, &Gt0, &Bs, &iBs, &O, &Gr, &Qh, &Tw, &Rw, &Cw};
		for (Buf *x : b) x->release();
		if (dtab) cudaFree(dtab);
		dtab = nullptr;
	}
};

}  // namespace dq
