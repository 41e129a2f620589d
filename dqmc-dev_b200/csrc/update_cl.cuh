// Delayed rank-k Metropolis updates of one slice with the Green's function
// held on chip (reference src/updates.c:7-84; draws of src/rand.h:6-31 as in
// update.cuh).
//
// A chain's two spins are spread over a cluster of 2 P CTAs, P = 1, 2 or 4 per
// spin, each holding the slab of N / P columns of its spin's G in shared
// memory for the whole slice: the flushes G += A B^T and the row and column
// reads of every accept stay on chip instead of going through L2.
//
// The sites are decided in windows as in update.cuh, by every CTA from the
// same numbers:
//   * each CTA sends the window entries of its columns to all CTAs of the
//     cluster (st.async onto the receivers' mbarriers): one exchange per window
//     where an exchange per accept would need a dozen.  The received blocks are
//     double-buffered by window parity: a CTA sends window n + 2 only after it
//     has received n + 1 from everyone, who sent it after reading n;
//   * the panels: A's rows need column i_m of G, read from the CTA that holds
//     it through distributed shared memory (P > 1), B's rows only the CTA's own
//     columns;
//   * the flush of a CTA's slab must neither run before all CTAs of the spin
//     have read its columns (an mbarrier they all arrive on after their
//     panels), nor be read before it is complete (each CTA arrives on everyone's
//     window mbarrier after its flush).
// Every wait on another CTA is an mbarrier wait with a time limit, so a CTA
// whose peers stop answering sets DQ_ERR_TIMEOUT and finishes in bounded time
// instead of hanging.
//
// The arithmetic is that of k_update in update.cuh, operation for operation,
// so both kernels give bit-identical fields, RNG states and G.
//
// What bounds it: the decisions (a latency chain, about 60k of 165k cycles a
// slice at N = 144, one CTA per spin) and the flushes' DMMAs and shared-memory
// traffic (65k).  One chain, microseconds per slice, P = 1 / 2 / 4: N = 144
// 101 / 91 / 84 (one exchange per accept and P = 1: 186), N = 196 - / 157 / 135
// (G in device memory 468), N = 256 - / - / 182 (935).
#pragma once

#include <cstdlib>
#include <cstring>

#include "mbar.cuh"
#include "update.cuh"

namespace dq {

// ------------------------------------------------------------ PTX helpers

__device__ inline uint32_t cluster_rank()
{
	uint32_t r;
	asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
	return r;
}

// address of the same shared-memory location in CTA `rank` of the cluster
__device__ inline uint32_t peer_smem(uint32_t a, uint32_t rank)
{
	uint32_t r;
	asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
	return r;
}

// asynchronous 8-byte store into a peer CTA's shared memory, completing 8
// transaction bytes on the peer's mbarrier at `mbar`
__device__ inline void st_async_f64(uint32_t a, double v, uint32_t mbar)
{
	asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];"
	             ::"r"(a), "d"(v), "r"(mbar) : "memory");
}

__device__ inline uint32_t cluster_ctas()
{
	uint32_t r;
	asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(r));
	return r;
}

// one arrival on a CTA's mbarrier (cluster address), releasing what this CTA
// has done so far to the cluster
__device__ inline void mbar_arrive_cluster(uint32_t mbar)
{
	asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(mbar) : "memory");
}

__device__ inline double ld_cluster(uint32_t a, const double *)
{
	double v;
	asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
	return v;
}
__device__ inline zd ld_cluster(uint32_t a, const zd *)
{
	zd v;
	asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
	return v;
}

// cluster-wide barrier of all threads of all CTAs, with release/acquire
// ordering of shared-memory accesses across the cluster
__device__ inline void cluster_sync_all()
{
	asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// ------------------------------------------------------ shared-memory plan

// panel leading dimension: >= n, = 4 (mod 16) for conflict-free fragments
__host__ __device__ inline int cl_ldp(int n) { return n + ((20 - n % 16) % 16); }
// columns of one CTA's slab: N / P rounded up to whole 8-column tiles
__host__ __device__ inline int cl_slab(int N, int P) { return P == 1 ? N : (N + 8 * P - 1) / (8 * P) * 8; }

struct ClPlan {
	size_t mb, rs, order, hsl, u, dl, ordn, raw, win, s, pana, panb, g, total;
};

template <typename T>
__host__ __device__ inline ClPlan cl_plan(int N, int P, int kd)
{
	const int planes = is_cplx<T>::value ? 2 : 1, nc = cl_slab(N, P);
	auto al = [](size_t b) { return (b + 15) & ~(size_t)15; };
	ClPlan p;
	size_t off = 0;
	p.mb = off;    off = al(off + 3 * sizeof(uint64_t));
	p.rs = off;    off = al(off + 17 * sizeof(uint64_t));
	p.order = off; off = al(off + (size_t)N * sizeof(int));
	p.hsl = off;   off = al(off + (size_t)N * sizeof(int));
	p.u = off;     off = al(off + (size_t)N * sizeof(double));
	p.dl = off;    off = al(off + 2 * (size_t)N * sizeof(double));
	p.ordn = off;  off = al(off + (size_t)N * sizeof(int));
	p.raw = off;   off = al(off + (size_t)N * sizeof(uint64_t));
	p.win = off;   off = al(off + sizeof(WinShared<T>));
	p.s = off;     off = al(off + 4 * sizeof(T) * WIN * WIN_LD);       // [buffer][spin]
	p.pana = off;  off = al(off + sizeof(double) * planes * (size_t)cl_ldp(N) * kd);
	p.panb = off;  off = al(off + sizeof(double) * planes * (size_t)cl_ldp(nc) * kd);
	p.g = off;     off = al(off + sizeof(T) * (size_t)nc * cl_ldg(N));
	p.total = off;
	return p;
}

constexpr size_t CL_SMEM = 227 * 1024 - 64;   // beside the few bytes of static shared memory

// working warps, beside the look-ahead warp: one that decides, the others for
// the panel rows and the flush's tiles
__host__ __device__ inline int cl_warps(int N) { return (N + 7) / 8 < 3 ? 3 : ((N + 7) / 8 > 15 ? 15 : (N + 7) / 8); }

// ------------------------------------------------------------------ kernel

template <typename T>
__global__ void __launch_bounds__(512, 1) k_update_cl(UpdArgs<T> a)
{
	constexpr bool CX = is_cplx<T>::value;
	constexpr int PL = CX ? 2 : 1;
	const int ncta = (int)cluster_ctas(), P = ncta >> 1, rank = (int)cluster_rank();
	const int c = blockIdx.x / ncta;           // chain
	const int s = rank / P, slab = rank - s * P;   // spin, slab of its columns
	const int N = a.N, KD = a.n_delay, SW = cl_slab(N, P);
	const int j0 = slab * SW, nc = max(0, min(SW, N - j0));
	const int LDG = cl_ldg(N);
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int NT = (int)blockDim.x - 32, NWK = NT >> 5;   // working threads; the last warp draws ahead
	const size_t NN = (size_t)N * N;
	const int par = a.slice & 1;
	const ClPlan pl = cl_plan<T>(N, P, KD);

	extern __shared__ __align__(16) unsigned char smraw[];
	uint64_t *mb = (uint64_t *)(smraw + pl.mb);     // window blocks of parity 0, 1; panels read
	uint64_t *rs = (uint64_t *)(smraw + pl.rs);
	int *order = (int *)(smraw + pl.order);
	int *hsl = (int *)(smraw + pl.hsl);
	double *u = (double *)(smraw + pl.u);
	double *dl = (double *)(smraw + pl.dl);
	WinShared<T> &ws = *(WinShared<T> *)(smraw + pl.win);
	T *S = (T *)(smraw + pl.s);                     // [buffer][spin][WIN * WIN_LD]
	double *pa = (double *)(smraw + pl.pana), *pb = (double *)(smraw + pl.panb);
	T *Gs = (T *)(smraw + pl.g);                    // this slab's columns, ld LDG
	const Panel<T> A{pa, pa + (size_t)(PL - 1) * cl_ldp(N) * KD, cl_ldp(N)};
	const Panel<T> B{pb, pb + (size_t)(PL - 1) * cl_ldp(SW) * KD, cl_ldp(SW)};
	__shared__ volatile int s_abort;

	T *Gg = a.G + (size_t)(2 * c + s) * NN + (size_t)N * j0;
	int *hs = a.hs + ((size_t)c * a.L + a.slice) * N;
	g_load<T>(Gs, Gg, N, nc, warp, NWK + 1, lane);
	cp_commit();
	for (int q = tid; q < N; q += blockDim.x) {
		hsl[q] = hs[q];
		order[q] = a.order[((size_t)c * 2 + par) * N + q];
		u[q] = a.u[((size_t)c * 2 + par) * N + q];
	}
	for (int q = tid; q < 2 * N; q += blockDim.x) dl[q] = a.del[(size_t)c * 2 * N + q];
	if (rank == 0 && tid < 17) rs[tid] = a.rng[(size_t)c * 17 + tid];
	if (tid == 0) {
		s_abort = 0;
		mbar_init(smem_u32(&mb[0]), 1 + ncta);
		mbar_init(smem_u32(&mb[1]), 1 + ncta);
		mbar_init(smem_u32(&mb[2]), P);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	T phase = a.phase[c];                      // warp 0's is the running one
	int nacc = 0;
	cp_wait<0>();
	__syncthreads();
	cluster_sync_all();

	if (tid >= NT) {
		// look-ahead warp of the first CTA: the draws of the next slice
		if (rank == 0 && a.next_slice >= 0) {
			if (lane < 17) a.rng_ckpt[(size_t)c * 17 + lane] = rs[lane];
			const int np = a.next_slice & 1;
			draw_slice_warp(rs, N, a.hs + ((size_t)c * a.L + a.next_slice) * N, dl,
			                (int *)(smraw + pl.ordn), (uint64_t *)(smraw + pl.raw),
			                a.order + ((size_t)c * 2 + np) * N, a.u + ((size_t)c * 2 + np) * N, lane);
			if (lane < 17) a.rng[(size_t)c * 17 + lane] = rs[lane];
		}
	} else {
		int n = 0;
		const uint32_t mb0 = smem_u32(mb), s0 = smem_u32(S), g0 = smem_u32(Gs);
		for (int pos = 0; pos < N; n++) {
			const int w = min(WIN, N - pos), buf = n & 1;
			const uint32_t mbw = mb0 + 8 * buf;
			win_clear(ws, tid, NT);
			if (tid == 0) mbar_arrive_tx(mbw, (uint32_t)(2 * w * w * sizeof(T)));
			// tid < ncta: this CTA's flush is complete (and so are its sends)
			if (tid < ncta) mbar_arrive_cluster(peer_smem(mbw, (uint32_t)tid));
			for (int q = tid; q < WIN * WIN * ncta; q += NT) {
				const int r = q % WIN, cc = q / WIN % WIN, to = q / (WIN * WIN);
				if (r >= w || cc >= w) continue;
				const int ic = order[pos + cc] - j0;
				if (ic < 0 || ic >= nc) continue;
				const T v = Gs[order[pos + r] + (size_t)LDG * ic];
				const uint32_t ra = peer_smem(s0 + (uint32_t)(((buf * 2 + s) * WIN * WIN_LD + r + WIN_LD * cc) * sizeof(T)),
				                              (uint32_t)to);
				const uint32_t rb = peer_smem(mbw, (uint32_t)to);
				double xr, xi;
				split(v, xr, xi);
				st_async_f64(ra, xr, rb);
				if (CX) st_async_f64(ra + 8, xi, rb);
			}
			bar_metro(NT);
			mbar_wait_bounded(mbw, (uint32_t)((n >> 1) & 1), &s_abort, a.err);
			__syncwarp();
			if (warp == 0) {
				phase = phase * metro_window<T>(w, KD, S + (buf * 2 + (lane >> 4)) * WIN * WIN_LD, ws, order + pos,
				                                u + pos, hsl, dl, N);
			} else if (P == 1) {
				panel_rows<T>([&](int j, int i) { return Gs[j + (size_t)LDG * i]; },
				              [&](int i, int j) { return Gs[i + (size_t)LDG * j]; }, N, 0, N, s, ws, A, B, warp - 1,
				              NWK - 1, lane, a.err);
			} else {
				panel_rows<T>(
					[&](int j, int i) {
						const int o = i / SW;      // the slab of column i
						return ld_cluster(peer_smem(g0 + (uint32_t)((j + (size_t)LDG * (i - o * SW)) * sizeof(T)),
						                            (uint32_t)(s * P + o)), (const T *)nullptr);
					},
					[&](int i, int j) { return Gs[i + (size_t)LDG * (j - j0)]; }, N, j0, nc, s, ws, A, B, warp - 1,
					NWK - 1, lane, a.err);
			}
			bar_metro(NT);
			const int kw = ws.kw;
			if (tid < kw) {
				int *h = hsl + ws.site[tid];
				*h = 1 - *h;
			}
			pos += ws.used;
			nacc += kw;
			if (P > 1) {
				// every CTA of the spin has read the columns it needs
				if (tid < P) mbar_arrive_cluster(peer_smem(mb0 + 16, (uint32_t)(s * P + tid)));
				mbar_wait_bounded(mb0 + 16, (uint32_t)(n & 1), &s_abort, a.err);
				__syncwarp();
			}
			if (kw) flush_panels<T>(Gs, (size_t)LDG, N, nc, kw, A, B, warp, NWK, lane);
			bar_metro(NT);
		}
	}
	__syncthreads();
	g_store<T>(Gg, Gs, N, nc, warp, NWK + 1, lane);
	if (rank == 0) {
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
	// no CTA leaves while another may still address its shared memory
	cluster_sync_all();
}

// CTAs per spin (1, 2 or 4; at least p) that hold one spin's G and panels; 0
// when none does
template <typename T>
inline int update_cl_split(int N, int kd, int p)
{
	for (; p <= 4; p *= 2)
		if (cl_plan<T>(N, p, kd).total <= CL_SMEM) return p;
	return 0;
}

template <typename T>
size_t update_cl_smem_bytes(int N, int P, int kd)
{
	return cl_plan<T>(N, P, kd).total;
}

// The form of the delayed update: 0 for one CTA per chain with G in device memory
// (k_update), else the CTAs per spin P of k_update_cl.  Both do the same arithmetic
// in the same order.  The on-chip form shortens a slice but a chain then holds 2 P
// SMs (74, 36 and 15 clusters run at once for P = 1, 2, 4), so the rule goes by what
// runs at once and by how much that gains.  launch: the chains of the largest
// launch, chains: those of all lanes.  Milliseconds a sweep of L = 10 in the
// default lanes, device memory / the fewest SMs that hold G:
//                    32        64       100       128       192       256 chains
//   real  N = 36  .66/.55   .70/.59   .76/.66   .84/.72  1.00/.93  1.28/1.21
//             64 1.06/.78  1.11/.84  1.33/1.37 1.36/1.26 1.76/1.74 2.30/2.52
//            100 2.03/1.59 2.27/1.84 3.09/3.32 3.15/3.12 4.67/4.49 5.71/6.03
//            121 2.94/2.07 3.42/2.56 4.47/4.41 4.62/4.25 7.14/6.26 8.86/8.36
//            144 3.90/2.56 4.32/3.00 5.80/5.45 5.97/5.28 8.42/7.75 11.3/10.3
//   P = 2    156 5.13/3.57 5.63/5.07 7.90/9.32 8.54/9.82 12.3/14.4 19.6/21.9
//            196 8.13/5.18 9.60/8.20 13.4/15.0 15.4/16.3 22.5/24.1 31.8/32.7
//   P = 4    225 14.0/11.4 16.6/17.0 23.7/27.3 26.8/31.2 39.8/46.3 52.4/61.0
//            256 17.6/13.6 20.5/20.1 29.6/31.9 33.6/36.0 48.7/53.3 65.8/70.7
//   cplx      32  .67/.69   .71/.74   .83/.88   .93/.98  1.21/1.26 1.52/1.58
//             36 1.02/.91  1.12/.98  1.32/1.26 1.51/1.42 1.99/1.97 2.44/2.50
//             64 1.88/1.54 2.12/1.77 2.52/2.41 2.85/2.95 3.91/4.40 4.63/5.72
//             81 3.45/2.57 3.91/3.07 4.62/4.18 5.16/5.12 7.10/7.57 9.28/10.0
//   P = 2    100 4.66/3.56 5.34/5.43 6.47/8.18 7.61/10.2 11.0/15.4 14.6/20.4
//            121 6.62/4.81 8.31/7.93 9.74/11.6 12.5/15.2 16.7/21.4 21.9/28.4
//   P = 4    144 9.20/9.97 11.5/15.1 (16 chains 8.34/7.24)
//            169 16.1/14.7 20.0/21.6
// More than one CTA per spin where one would do pays from N = 90 up (complex: 64)
// while the clusters run at once: 8 chains real N = 100 1.39 / 1.32 / 1.28 ms for P
// = 1 / 2 / 4, 32 chains 1.59 / 1.52 / 2.55.  DQMC_UPDATE=cluster or =global
// overrides the choice between the two forms (read when an engine is created, or a
// seam called).
template <typename T>
int update_split(int N, int kd, int launch, int chains)
{
	constexpr bool CX = is_cplx<T>::value;
	const char *v = getenv("DQMC_UPDATE");
	const bool forced = v && *v;
	if (N > 480 || (forced ? strcmp(v, "cluster") != 0 : N < (CX ? 33 : 25))) return 0;
	const int pmin = update_cl_split<T>(N, kd, 1);
	if (!pmin) return 0;
	if (!forced) {
		int limit;      // chains beyond which G in device memory is faster
		if (pmin == 1) limit = CX ? (N < 56 ? 222 : 110) : (N < 64 || N >= 112) ? chains : launch <= 74 ? 222 : 74;
		else if (pmin == 2) limit = CX && N < 112 ? 36 : 72;
		else limit = !CX ? 60 : N < 160 ? 30 : 45;
		if (chains > limit) return 0;
	}
	const int p = (N >= 90 && chains <= 8) ? 4 : (N >= (CX ? 64 : 90) && chains <= 32) ? 2 : 1;
	return update_cl_split<T>(N, kd, p);
}

}  // namespace dq
