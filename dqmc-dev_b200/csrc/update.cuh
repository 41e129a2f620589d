// Delayed rank-k Sherman-Morrison Metropolis updates of one imaginary-time
// slice (reference src/updates.c:7-84, with the shuffle of src/rand.h:25-31
// and the draws of rand.h:6-22 that dqmc.c:249-253 makes before it).
//
// The slice's N sequential tests only ever look at G on the sites still to be
// visited, so the sites are taken in windows of 16 in visiting order:
//   * gather: the window's 16 x 16 entries of both spins' G (all threads);
//   * decide: one warp, a half per spin, one window site per lane.  Every lane
//     evaluates its own site's accept test (the spins' ratios cross by a
//     shuffle), and the first accepting site is the next accept: the sites
//     before it are rejected by the very same numbers.  Its row and column,
//     the window sites' panel entries and diagonals follow, and the tests are
//     evaluated again.  A rejected site costs nothing, an accept no barrier
//     (metro_window);
//   * panels: meanwhile the other warps, one row of G per thread, form the new
//     columns of the panels A, B, following the accepts as they are published
//     (panel_row);
//   * the panels are flushed, G += A B^T, with FP64 tensor-core MMAs
//     (flush_panels).
// A window ends early after n_delay accepts (its panels' columns).
// An entry (i, j) of the updated G is G[i, j] + A_0[i] B_0[j] + ..., each term
// one fma_(A, B, .) in ascending order, whichever thread forms it; the flush
// adds the products of the same panels in the same order wherever G lies.
//
// What bounds it: the decide step is a latency chain (a division, a ballot
// and a dot product of the panel depth per accept), the flush tensor and
// memory work (L2 when G stays in device memory).
// One test at a time over all of the chain's threads, two CTA-wide barriers
// per accept (about 1700 cycles) and a row and a column of G fetched per
// accept, took 255 us a slice at N = 144 and 68 us at N = 64 (one real chain);
// in windows 234 and 64 us with G in device memory, where the flushes' L2
// traffic is left, and 84 and 38 us with G on chip (update_cl.cuh), of which
// the decisions take about 0.55 us an accept.
//
// The number of draws of a slice depends only on its fields at slice start
// (one uniform per site whose delta is non-zero), so the site permutation and
// uniforms of slice l+1 are drawn by one more warp while slice l is being
// updated, and the next kernel reads them.  rng_ckpt keeps the state as it was
// before the look-ahead, which is the state the reference has at that point
// (dqmc.c:249).
#pragma once

#include "common.cuh"
#include "gemm.cuh"
#include "mbar.cuh"

namespace dq {

template <typename T>
struct UpdArgs {
	int N, L, n_delay;     // n_delay: flush period used by the kernel
	int nchain;
	int slice;
	int ldp;               // panel leading dimension in shared memory
	const double *del;     // [chain][2][N]
	const double *exp_lambda; // [chain][2][N]
	uint64_t *rng;         // [chain][17] working state (ahead by the look-ahead draws)
	uint64_t *rng_ckpt;    // [chain][17] state before the look-ahead draws
	int *hs;               // [chain][L][N]
	T *G;                  // [chain][2][N*N]
	T *phase;              // [chain]
	double *dv, *dvi;      // [chain][2][L][N]: d_l and 1/d_l of every slice (optional)
	int *n_accept;         // [chain] running accept count (optional)
	int *order;            // [chain][2][N] site permutations, by slice parity
	double *u;             // [chain][2][N] uniforms in visiting order (2: never accept)
	int next_slice;        // slice whose draws the look-ahead warp takes (-1: none)
	unsigned *err;
};

// x mod m for x < 2^61 and m < 2^10, with 32-bit divisions only
__device__ inline unsigned mod_small(uint64_t x, unsigned m)
{
	unsigned r = (unsigned)(x >> 44) % m;
	r = ((r << 22) | (unsigned)((x >> 22) & 0x3FFFFFu)) % m;
	r = ((r << 22) | (unsigned)(x & 0x3FFFFFu)) % m;
	return r;
}

__device__ inline double u01_from(uint64_t r)
{
	return __longlong_as_double((long long)((0x3FFULL << 52) | (r >> 12))) - 1.0;
}

// The draws of one slice, in the reference's order: the inside-out
// Fisher-Yates permutation (rand.h:25-31), then one uniform per visited site
// whose delta is non-zero (updates.c:19-26).  One warp: the generator steps
// are a serial chain on lane 0, which leaves the raw words in `raw`; the
// remainders, the fields' look-up and the conversions go over the lanes.
// rs (17 words), order_s (N) and raw (N) in shared memory; order and u receive
// the result in device memory.
__device__ inline void xs1024_fill(uint64_t *rs, int n, uint64_t *raw)
{
	int p = (int)rs[16];
	uint64_t a = rs[p];
	for (int i = 0; i < n; i++) {
		p = (p + 1) & 15;
		uint64_t b = rs[p];
		b ^= b << 31;
		a = b ^ a ^ (b >> 11) ^ (a >> 30);
		rs[p] = a;
		raw[i] = a * 1181783497276652981ULL;
	}
	rs[16] = (uint64_t)p;
}

__device__ inline void draw_slice_warp(uint64_t *rs, int N, const int *hs_row, const double *del,
		int *order_s, uint64_t *raw, int *order, double *u, int lane)
{
	__syncwarp();
	if (lane == 0) xs1024_fill(rs, N, raw);
	__syncwarp();
	for (int i = lane; i < N; i += 32) raw[i] = mod_small(raw[i] >> 3, (unsigned)(i + 1));
	__syncwarp();
	if (lane == 0)
		for (int i = 0; i < N; i++) {
			const int jj = (int)raw[i];
			if (jj != i) order_s[i] = order_s[jj];
			order_s[jj] = i;
		}
	__syncwarp();
	// visited sites that draw, packed: their count, then their words
	int n = 0;
	for (int i0 = 0; i0 < N; i0 += 32) {
		const int ii = i0 + lane;
		bool d = false;
		if (ii < N) {
			const int i = order_s[ii], h = hs_row[i];
			d = !(del[i + N * h] == 0.0 && del[i + N * (1 - h)] == 0.0);
			order[ii] = i;
		}
		const unsigned m = __ballot_sync(0xffffffffu, d);
		// the position of each site's word, or -1
		if (ii < N) order_s[ii] = d ? n + __popc(m & ((1u << lane) - 1u)) : -1;
		n += __popc(m);
	}
	if (lane == 0) xs1024_fill(rs, n, raw);
	__syncwarp();
	for (int ii = lane; ii < N; ii += 32) u[ii] = order_s[ii] < 0 ? 2.0 : u01_from(raw[order_s[ii]]);
	__syncwarp();
}

// draws of slice `slice` for every chain, one warp per chain (start of a run);
// shared memory draws_smem_bytes(N)
inline size_t draws_smem_bytes(int N)
{
	return sizeof(uint64_t) * (18 + (size_t)N) + sizeof(int) * (size_t)N;
}

__global__ void k_draws(int N, int L, int nchain, int slice, const double *del, uint64_t *rng,
		uint64_t *rng_ckpt, const int *hs, int *order, double *u)
{
	extern __shared__ __align__(16) unsigned char smraw[];
	const int c = blockIdx.x, lane = threadIdx.x;
	if (c >= nchain) return;
	uint64_t *s = (uint64_t *)smraw, *raw = s + 18;
	int *os = (int *)(raw + N);
	if (lane < 17) {
		s[lane] = rng[(size_t)c * 17 + lane];
		rng_ckpt[(size_t)c * 17 + lane] = s[lane];
	}
	const int par = slice & 1;
	draw_slice_warp(s, N, hs + ((size_t)c * L + slice) * N, del + (size_t)c * 2 * N, os, raw,
	                order + ((size_t)c * 2 + par) * N, u + ((size_t)c * 2 + par) * N, lane);
	if (lane < 17) rng[(size_t)c * 17 + lane] = s[lane];
}

// ------------------------------------------------------------- one window

constexpr int WIN = 16;             // window sites: half a warp
constexpr int WIN_LD = WIN + 1;     // leading dimension of a window's block of G: rows and
                                    // columns are read without bank conflicts
constexpr int WIN_DONE = 1 << 16;   // added to the published count at the window's end

// a and b of one window site for one accept of the window
template <typename T>
struct __align__(16) Ab {
	T a, b;
};

// shared memory of a window
template <typename T>
struct __align__(16) WinShared {
	Ab<T> w[2][WIN][WIN];   // [spin][accept][site]: the window sites' panel entries
	T sc[2][WIN];           // [spin][accept]: the scales
	T prob[WIN];            // [accept]: r_up r_down
	int site[WIN], lane[WIN];   // [accept]: the accepted site, its window position
	int cnt;                // accepts published
	int kw, used;           // at the end: accepts, sites consumed
};

// start of a window, by nthr threads: nothing published, all entries zero
template <typename T>
__device__ inline void win_clear(WinShared<T> &ws, int tid, int nthr)
{
	if (tid == 0) ws.cnt = 0;
	double2 *z = (double2 *)ws.w;
	for (int q = tid; q < (int)(sizeof(ws.w) / 16); q += nthr) z[q] = make_double2(0.0, 0.0);
}

__device__ inline double unit_phase(double prob) { return copysign(1.0, prob); }
__device__ inline zd unit_phase(zd prob) { return prob / absv(prob); }

// Named barrier 1: the working threads (the look-ahead warp never joins it);
// the non-aligned form, since lanes may arrive apart.
__device__ inline void bar_metro(int nthreads)
{
	asm volatile("barrier.sync 1, %0;\n" ::"r"(nthreads) : "memory");
}

__device__ inline void st_release_cta(int *p, int v)
{
	asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
__device__ inline int ld_acquire_cta(const int *p)
{
	int v;
	asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
	return v;
}

// The sequential decisions of the window sites order[0 .. W), one warp: lanes
// 0-15 hold the sites for spin up, 16-31 for spin down.  S: this lane's spin's
// block of G, up to date.  Stops after kmax accepts.  Publishes each accept in
// ws (position, scale, the window sites' panel entries) and leaves the totals;
// returns the product of the accepts' phases.
template <typename T>
__device__ inline T metro_window(int W, int kmax, const T *S, WinShared<T> &ws, const int *order,
		const double *u, const int *hsl, const double *dl, int N)
{
	const int lane = threadIdx.x & 31, r = lane & (WIN - 1), sp = lane >> 4;
	const bool in = r < W;
	const int site = order[in ? r : 0], h = hsl[site];
	const double ur = u[in ? r : 0];
	const double del = dl[site + N * (h ^ sp)];
	const T *srow = S + r, *scol = S + WIN_LD * r;
	T d = scol[r];
	Ab<T> *wo = ws.w[sp][0] + r;
	const Ab<T> *wp = ws.w[sp][0];
	T *sco = ws.sc[sp];
	unsigned live = __ballot_sync(0xffffffffu, in && ur < 1.0) & 0xffffu;
	int used = W, kw = 0;
	while (true) {
		const T ro = 1.0 + (1.0 - d) * del;
		const T rx = shfl_xor(ro, 16);
		// the factors in one order, so that both halves see the same bits
		const T prob = (sp ? rx : ro) * (sp ? ro : rx);
		const unsigned acc = __ballot_sync(0xffffffffu, ur < absv(prob)) & live;
		if (!acc) break;
		const int p = __ffs(acc) - 1;
		live &= 0xfffffffeu << p;
		// the loads run a step ahead of the products (the first ones while the
		// division runs); entries from kw on are zero, so that whole steps of
		// four are taken
		T av = srow[WIN_LD * p], bv = scol[p];
		const Ab<T> *xo = wo, *xp = wp + p;
		Ab<T> x[4], y[4];
#pragma unroll
		for (int t = 0; t < 4; t++) {
			x[t] = xo[t * WIN];
			y[t] = xp[t * WIN];
		}
		const T sc = shfl(del / ro, p + (lane & 16));
#pragma unroll
		for (int m = 0; m < WIN; m += 4) {
			if (m >= kw) break;
			Ab<T> xn[4], yn[4];
			if (m + 4 < WIN) {
#pragma unroll
				for (int t = 0; t < 4; t++) {
					xn[t] = xo[(m + 4 + t) * WIN];
					yn[t] = xp[(m + 4 + t) * WIN];
				}
			}
#pragma unroll
			for (int t = 0; t < 4; t++) {
				av = fma_(x[t].a, y[t].b, av);
				bv = fma_(y[t].a, x[t].b, bv);
			}
#pragma unroll
			for (int t = 0; t < 4; t++) {
				x[t] = xn[t];
				y[t] = yn[t];
			}
		}
		av = av - (r == p ? 1.0 : 0.0);
		av = av * sc;
		d = fma_(av, bv, d);
		wo[kw * WIN] = Ab<T>{av, bv};
		sco[kw] = sc;
		if (lane == p) {
			ws.prob[kw] = prob;
			ws.site[kw] = site;
			ws.lane[kw] = p;
		}
		kw++;
		__syncwarp();
		if (lane == 0) st_release_cta(&ws.cnt, kw);
		if (kw == kmax) {
			used = p + 1;
			break;
		}
	}
	__syncwarp();
	T ph = lane < kw ? unit_phase(ws.prob[lane & (WIN - 1)]) : one<T>();
#pragma unroll
	for (int o = 8; o > 0; o >>= 1) ph = ph * shfl_xor(ph, o);
	if (lane == 0) {
		ws.kw = kw;
		ws.used = used;
		st_release_cta(&ws.cnt, kw + WIN_DONE);
	}
	return shfl(ph, 0);
}

// accepts published so far: waits for `need` of them or for the window's end
// (the decision warps always reach it: every wait of theirs is bounded), with
// a limit after which it gives up
__device__ inline int win_wait(const int *cnt, int need, unsigned *err)
{
	for (int it = 0; it < (1 << 24); it++) {
		const int v = ld_acquire_cta(cnt);
		if (v >= need) return v & (WIN_DONE - 1);   // WIN_DONE exceeds every need
	}
	if (err) atomicOr(err, DQ_ERR_TIMEOUT);
	return 0;
}

// one panel element of the split planes (complex: re and im in planes)
template <typename T>
struct Panel {
	double *re, *im;
	int ld;
	__device__ T get(int j, int m) const
	{
		if constexpr (is_cplx<T>::value) return mkz(re[j + ld * m], im[j + ld * m]);
		else return re[j + ld * m];
	}
	__device__ void set(int j, int m, const T &v) const
	{
		double x, y;
		split(v, x, y);
		re[j + ld * m] = x;
		if (is_cplx<T>::value) im[j + ld * m] = y;
	}
};

// Row j of a window's panels:
// A_m = (G[:, i_m] + sum_{m'<m} A_m' B_m'[i_m] - e_{i_m}) sc_m     (PA)
// B_m = G[i_m, :] + sum_{m'<m} B_m' A_m'[i_m]                      (!PA)
// g(i) is G's entry (j, i) for A and (i, j) for B; the coefficients are the
// window sites' entries, so the rows are independent of one another.  As many
// accepts at a time as have been published, at most four, so that the entries
// of a row that lags behind (G in device memory) are fetched together.
template <typename T, int NBM, bool PA, typename GET>
__device__ __forceinline__ void panel_step(const GET &g, int j, int jo, int m0, int nb,
		const WinShared<T> &ws, int s, const Panel<T> &own)
{
	T v[NBM];
	int it[NBM], lt[NBM];
#pragma unroll
	for (int t = 0; t < NBM; t++) {
		const int m = m0 + min(t, nb - 1);
		lt[t] = ws.lane[m];
		it[t] = ws.site[m];
		v[t] = g(it[t]);
	}
#pragma unroll 4
	for (int q = 0; q < m0; q++) {
		const T a = own.get(jo, q);
#pragma unroll
		for (int t = 0; t < NBM; t++) {
			const Ab<T> &y = ws.w[s][q][lt[t]];
			v[t] = PA ? fma_(a, y.b, v[t]) : fma_(y.a, a, v[t]);
		}
	}
#pragma unroll
	for (int t = 0; t < NBM; t++) {
		if (t >= nb) break;
		if (PA) {
			v[t] = v[t] - (j == it[t] ? 1.0 : 0.0);
			v[t] = v[t] * ws.sc[s][m0 + t];
		}
		own.set(jo, m0 + t, v[t]);
#pragma unroll
		for (int t2 = t + 1; t2 < NBM; t2++) {
			const Ab<T> &y = ws.w[s][m0 + t][lt[t2]];
			v[t2] = PA ? fma_(v[t], y.b, v[t2]) : fma_(y.a, v[t], v[t2]);
		}
	}
}

template <typename T, bool PA, typename GET>
__device__ inline void panel_row(const GET &g, int j, int jo, int s, const WinShared<T> &ws,
		const Panel<T> &own, unsigned *err)
{
	for (int m = 0;;) {
		const int nb = min(4, win_wait(&ws.cnt, m + 1, err) - m);
		if (nb <= 0) return;
		if (nb == 1) panel_step<T, 1, PA>(g, j, jo, m, 1, ws, s, own);
		else panel_step<T, 4, PA>(g, j, jo, m, nb, ws, s, own);
		m += nb;
	}
}

// one spin's panels by nwarp warps, 32 rows of A (all N) or of B (rows j0 ..
// j0 + nj - 1, stored from 0) at a time; ga(j, i) and gb(i, j): G's entries
template <typename T, typename GA, typename GB>
__device__ inline void panel_rows(const GA &ga, const GB &gb, int N, int j0, int nj, int s,
		const WinShared<T> &ws, const Panel<T> &A, const Panel<T> &B, int warp, int nwarp, int lane,
		unsigned *err)
{
	const int na = (N + 31) / 32, nt = na + (nj + 31) / 32;
	for (int t = warp; t < nt; t += nwarp) {
		if (t < na) {
			const int j = t * 32 + lane;
			if (j < N) panel_row<T, true>([&](int i) { return ga(j, i); }, j, j, s, ws, A, err);
		} else {
			const int jo = (t - na) * 32 + lane;
			if (jo < nj) panel_row<T, false>([&](int i) { return gb(i, j0 + jo); }, j0 + jo, jo, s, ws, B, err);
		}
	}
}

// G (N rows, NC columns) += A B^T by nwarp warps: each warp takes R x C tiles of 8 x 8
// at a time, G's entries as the DMMA accumulators, ascending k.  A fragment is
// read from shared memory once per C (B: R) tiles; one column of
// tiles at a time the fragment reads alone took longer than the DMMAs.
template <typename T> struct FlushTile { static constexpr int R = 3, C = 2; };
template <> struct FlushTile<zd> { static constexpr int R = 2, C = 2; };

template <typename T>
__device__ inline void flush_panels(T *G, size_t ldg, int N, int NC, int kc, const Panel<T> &A,
		const Panel<T> &B, int warp, int nwarp, int lane)
{
	constexpr bool CX = is_cplx<T>::value;
	constexpr int FLUSH_R = FlushTile<T>::R, FLUSH_C = FlushTile<T>::C;
	const int gq = lane >> 2, tq = lane & 3;
	const int nr = (N + 8 * FLUSH_R - 1) / (8 * FLUSH_R), nc = (NC + 8 * FLUSH_C - 1) / (8 * FLUSH_C);
	int cg = warp / nr, rg = warp - cg * nr;
	const int dc = nwarp / nr, dr = nwarp - dc * nr;
	T g[FLUSH_R][FLUSH_C][2];
	auto load = [&](int cg_, int rg_) {
		const int r0 = rg_ * 8 * FLUSH_R + gq, c0 = cg_ * 8 * FLUSH_C + 2 * tq;
		const T *Gt = G + r0 + ldg * c0;
#pragma unroll
		for (int v = 0; v < FLUSH_C; v++)
#pragma unroll
			for (int h = 0; h < 2; h++)
#pragma unroll
				for (int u = 0; u < FLUSH_R; u++)
					g[u][v][h] = (r0 + 8 * u < N && c0 + 8 * v + h < NC) ? Gt[8 * u + ldg * (8 * v + h)] : zero<T>();
	};
	if (cg < nc) load(cg, rg);
	while (cg < nc) {
		const int r0 = rg * 8 * FLUSH_R + gq, c0 = cg * 8 * FLUSH_C;
		double cr[FLUSH_R][FLUSH_C][2], ci[CX ? FLUSH_R : 1][CX ? FLUSH_C : 1][2];
#pragma unroll
		for (int v = 0; v < FLUSH_C; v++)
#pragma unroll
			for (int h = 0; h < 2; h++)
#pragma unroll
				for (int u = 0; u < FLUSH_R; u++) {
					double gi;
					split(g[u][v][h], cr[u][v][h], gi);
					if constexpr (CX) ci[u][v][h] = gi;
				}
		int cn = cg + dc, rn = rg + dr;
		if (rn >= nr) {
			rn -= nr;
			cn++;
		}
		if (!CX && cn < nc) load(cn, rn);     // the next tiles, while these are multiplied
		const double *Ar = A.re + r0 + A.ld * tq, *Br = B.re + c0 + gq + B.ld * tq;
		const double *Ai = A.im + r0 + A.ld * tq, *Bi = B.im + c0 + gq + B.ld * tq;
#pragma unroll 2
		for (int k0 = 0; k0 < kc; k0 += 4) {
			const bool okk = k0 + tq < kc;
			double br[FLUSH_C], bi[FLUSH_C], ar[FLUSH_R], ai[FLUSH_R];
#pragma unroll
			for (int v = 0; v < FLUSH_C; v++) {
				const bool ok = okk && c0 + 8 * v + gq < NC;
				br[v] = ok ? Br[8 * v + B.ld * k0] : 0.0;
				bi[v] = (CX && ok) ? Bi[8 * v + B.ld * k0] : 0.0;
			}
#pragma unroll
			for (int u = 0; u < FLUSH_R; u++) {
				const bool ok = okk && r0 + 8 * u < N;
				ar[u] = ok ? Ar[8 * u + A.ld * k0] : 0.0;
				ai[u] = (CX && ok) ? Ai[8 * u + A.ld * k0] : 0.0;
			}
#pragma unroll
			for (int u = 0; u < FLUSH_R; u++)
#pragma unroll
				for (int v = 0; v < FLUSH_C; v++) {
					dmma(cr[u][v][0], cr[u][v][1], ar[u], br[v]);
					if constexpr (CX) {
						dmma(cr[u][v][0], cr[u][v][1], -ai[u], bi[v]);
						dmma(ci[u][v][0], ci[u][v][1], ar[u], bi[v]);
						dmma(ci[u][v][0], ci[u][v][1], ai[u], br[v]);
					}
				}
		}
		T *Gt = G + r0 + ldg * (c0 + 2 * tq);
#pragma unroll
		for (int v = 0; v < FLUSH_C; v++)
#pragma unroll
			for (int h = 0; h < 2; h++)
#pragma unroll
				for (int u = 0; u < FLUSH_R; u++)
					if (r0 + 8 * u < N && c0 + 8 * v + 2 * tq + h < NC) {
						if constexpr (CX) {
							Gt[8 * u + ldg * (8 * v + h)] = mkz(cr[u][v][h], ci[u][v][h]);
						} else {
							Gt[8 * u + ldg * (8 * v + h)] = cr[u][v][h];
						}
					}
		cg = cn;
		rg = rn;
		if (CX && cg < nc) load(cg, rg);
	}
}

// leading dimension of G in shared memory: >= N with ld = 2 (mod 4), so
// that the flush's accumulator fragments (rows gq, columns 2 tq + h) of a
// half-warp fall in distinct banks
__host__ __device__ inline int cl_ldg(int N) { return N + ((6 - N % 4) % 4); }

// whether columns of a real G (N rows) can move 16 bytes at a time: every column
// starts on 16 bytes.  G is the caller's in dqmc_gpu_update_delayed and need
// only be aligned to its 8-byte numbers there.
__host__ __device__ inline bool g_wide(const void *Gg, int N)
{
	return (N & 1) == 0 && ((uintptr_t)Gg & 15) == 0;
}

// nc columns of G (N rows) between device memory and shared memory (leading dimension
// cl_ldg(N), even), by nwarp warps: 16 bytes at a time where g_wide allows.  The
// load is asynchronous (cp.async): commit and wait follow.
template <typename T>
__device__ inline void g_load(T *Gs, const T *Gg, int N, int nc, int warp, int nwarp, int lane)
{
	const int ldg = cl_ldg(N);
	const bool wide = g_wide(Gg, N);
	for (int col = warp; col < nc; col += nwarp) {
		T *dst = Gs + (size_t)ldg * col;
		const T *src = Gg + (size_t)N * col;
		if (is_cplx<T>::value || !wide)
			for (int r = lane; r < N; r += 32) cp_async_el<T>(dst + r, src + r, true);
		else
			for (int r = 2 * lane; r < N; r += 64) cp_async16(dst + r, src + r, true);
	}
}

template <typename T>
__device__ inline void g_store(T *Gg, const T *Gs, int N, int nc, int warp, int nwarp, int lane)
{
	const int ldg = cl_ldg(N);
	const bool wide = g_wide(Gg, N);
	for (int col = warp; col < nc; col += nwarp) {
		T *dst = Gg + (size_t)N * col;
		const T *src = Gs + (size_t)ldg * col;
		if (!is_cplx<T>::value && wide)
			for (int r = 2 * lane; r < N; r += 64) *(double2 *)(dst + r) = *(const double2 *)(src + r);
		else
			for (int r = lane; r < N; r += 32) dst[r] = src[r];
	}
}

// ------------------------------------------- one CTA per chain, both spins

// shared memory: rng, order, hsl, u, del, the next slice's order and raw
// words, each padded to 16 bytes, the panels of both spins, the window and its
// blocks of G
template <typename T>
size_t update_smem_bytes(int N, int kd, int ldp)
{
	const int planes = is_cplx<T>::value ? 2 : 1;
	return sizeof(uint64_t) * 17 + sizeof(int) * 3 * (size_t)N + sizeof(double) * 4 * (size_t)N + 8 * 16
	       + sizeof(double) * planes * 4 * (size_t)ldp * kd + sizeof(WinShared<T>) + 2 * sizeof(T) * WIN * WIN_LD;
}

// the accepts a window takes before its flush: the file's n_delay, at most a
// window's sites, and at most what shared memory has panel columns for
template <typename T>
int update_delay(int N, int n_delay, int ldp)
{
	int kd = n_delay < 1 ? 1 : (n_delay < WIN ? n_delay : WIN);
	if (kd > N) kd = N;
	while (kd > 1 && update_smem_bytes<T>(N, kd, ldp) > 226 * 1024) kd /= 2;
	return kd;
}

// working warps, beside the look-ahead warp: two per 32 rows, four to
// fourteen; an even number, since half of them flush each spin
__host__ __device__ inline int update_warps(int N)
{
	const int n = 2 * ((N + 31) / 32);
	return n < 4 ? 4 : (n > 14 ? 14 : n);
}

// the delayed update with G in device memory, one CTA per chain
template <typename T>
__device__ __forceinline__ void update_chain(const UpdArgs<T> &a)
{
	constexpr bool CX = is_cplx<T>::value;
	constexpr int PL = CX ? 2 : 1;
	const int c = blockIdx.x;
	if (c >= a.nchain) return;
	const int N = a.N, KD = a.n_delay, LDP = a.ldp;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int NT = (int)blockDim.x - 32, NWK = NT >> 5;   // working threads; the last warp draws ahead
	const size_t NN = (size_t)N * N;
	const int par = a.slice & 1;

	extern __shared__ __align__(16) unsigned char smraw[];
	auto al16 = [](size_t b) { return (b + 15) & ~(size_t)15; };
	size_t off = 0;
	uint64_t *rs = (uint64_t *)(smraw + off);  off = al16(off + 17 * sizeof(uint64_t));
	int *order = (int *)(smraw + off);         off = al16(off + N * sizeof(int));
	int *hsl = (int *)(smraw + off);           off = al16(off + N * sizeof(int));
	double *u = (double *)(smraw + off);       off = al16(off + N * sizeof(double));
	double *dl = (double *)(smraw + off);      off = al16(off + 2 * N * sizeof(double));
	int *ord_n = (int *)(smraw + off);         off = al16(off + N * sizeof(int));
	uint64_t *raw = (uint64_t *)(smraw + off); off = al16(off + N * sizeof(uint64_t));
	WinShared<T> &ws = *(WinShared<T> *)(smraw + off);   off += sizeof(WinShared<T>);
	T *S = (T *)(smraw + off);                 // [spin][WIN * WIN_LD]
	off += 2 * sizeof(T) * WIN * WIN_LD;
	double *pan = (double *)(smraw + off);     // [spin][A/B][plane][LDP*KD]
	auto P = [&](int sp, int ab) {
		double *b = pan + (size_t)((sp * 2 + ab) * PL) * LDP * KD;
		return Panel<T>{b, b + (size_t)(PL - 1) * LDP * KD, LDP};
	};
	T *Gc = a.G + (size_t)(2 * c) * NN;
	int *hs = a.hs + ((size_t)c * a.L + a.slice) * N;

	for (int q = tid; q < N; q += blockDim.x) {
		hsl[q] = hs[q];
		order[q] = a.order[((size_t)c * 2 + par) * N + q];
		u[q] = a.u[((size_t)c * 2 + par) * N + q];
	}
	for (int q = tid; q < 2 * N; q += blockDim.x) dl[q] = a.del[(size_t)c * 2 * N + q];
	if (tid < 17) rs[tid] = a.rng[(size_t)c * 17 + tid];
	T phase = a.phase[c];                      // warp 0's is the running one
	int nacc = 0;
	__syncthreads();

	if (tid >= NT) {
		// look-ahead warp: the draws of the next slice
		if (a.next_slice >= 0) {
			if (lane < 17) a.rng_ckpt[(size_t)c * 17 + lane] = rs[lane];
			const int np = a.next_slice & 1;
			draw_slice_warp(rs, N, a.hs + ((size_t)c * a.L + a.next_slice) * N, dl, ord_n, raw,
			                a.order + ((size_t)c * 2 + np) * N, a.u + ((size_t)c * 2 + np) * N, lane);
			if (lane < 17) a.rng[(size_t)c * 17 + lane] = rs[lane];
		}
	} else {
		for (int pos = 0; pos < N;) {
			const int w = min(WIN, N - pos);
			win_clear(ws, tid, NT);
			for (int q = tid; q < 2 * WIN * WIN; q += NT) {
				const int sp = q / (WIN * WIN), r = q % WIN, cc = q / WIN % WIN;
				if (r < w && cc < w)
					S[sp * WIN * WIN_LD + r + WIN_LD * cc] = Gc[sp * NN + order[pos + r] + (size_t)N * order[pos + cc]];
			}
			bar_metro(NT);
			// one spin per half of the warps
			const int nh = NWK / 2, sp = warp >= nh;
			T *G = Gc + sp * NN;
			if (warp == 0) {
				phase = phase * metro_window<T>(w, KD, S + (lane >> 4) * WIN * WIN_LD, ws, order + pos, u + pos,
				                                hsl, dl, N);
			} else {
				panel_rows<T>([&](int j, int i) { return G[j + (size_t)N * i]; },
				              [&](int i, int j) { return G[i + (size_t)N * j]; }, N, 0, N, sp, ws, P(sp, 0),
				              P(sp, 1), warp - (sp ? nh : 1), sp ? NWK - nh : nh - 1, lane, a.err);
			}
			bar_metro(NT);
			const int kw = ws.kw;
			if (tid < kw) {
				int *h = hsl + ws.site[tid];
				*h = 1 - *h;
			}
			pos += ws.used;
			nacc += kw;
			if (kw) flush_panels<T>(G, (size_t)N, N, N, kw, P(sp, 0), P(sp, 1), warp - sp * nh, nh, lane);
			bar_metro(NT);
		}
	}
	__syncthreads();
	for (int q = tid; q < N; q += blockDim.x) {
		const int hq = hsl[q];
		hs[q] = hq;
		if (!a.dv) continue;
		for (int sp = 0; sp < 2; sp++) {
			const double el = a.exp_lambda[(size_t)c * 2 * N + q + N * (hq ^ sp)];
			const size_t o = (((size_t)c * 2 + sp) * a.L + a.slice) * N + q;
			a.dv[o] = el;
			a.dvi[o] = 1.0 / el;
		}
	}
	if (tid == 0) {
		a.phase[c] = phase;
		if (a.n_accept) a.n_accept[c] += nacc;
	}
}

// MAXT threads, MINB CTAs on an SM.  While every chain has an SM to itself, CTAs
// take the registers they want; with more chains than SMs the small ones leave
// room for a second CTA as long as that does not cost many spills (real N <= 128; with
// room for two CTAs of 352 threads the bound is 80 registers).  Microseconds a
// slice, one CTA / two: real N = 64 x 256 chains - / 77 (154 registers either way),
// N = 81 x 128 97 / 109, x 256 186 / 136, N = 100 x 128 117 / 154, x 256 229 / 204,
// N = 144 x 32 234 / 359, x 256 477 / 577; complex N = 64 x 128 112 / 123, x 256
// 227 / 151.
template <typename T, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) k_update(UpdArgs<T> a)
{
	update_chain(a);
}

// k_update's instance for N's CTA; chains: those of the whole engine, whose lanes
// share the SMs
template <typename T>
auto update_kernel(int N, int chains)
{
	const int t = update_warps(N) * 32 + 32;
	const bool one = chains <= 148;
	if constexpr (is_cplx<T>::value) {
		if (t <= 160 && one) return k_update<T, 160, 1>;
		// 168 registers: two CTAs of 160 threads fit as well
		return t <= 352 ? k_update<T, 352, 1> : k_update<T, 480, 1>;
	} else {
		if (t <= 160) return k_update<T, 160, 2>;
		if (t <= 224 && !one) return k_update<T, 224, 2>;
		if (t <= 288 && !one) return k_update<T, 288, 2>;
		return t <= 352 ? k_update<T, 352, 1> : k_update<T, 480, 1>;
	}
}

}  // namespace dq
