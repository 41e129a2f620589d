// Launcher of the batched GEMM kernel (gemm.cuh): mode dispatch and tile
// choice.  Included by launch_gemm_r.cu and launch_gemm_c.cu only.
#pragma once

#include <cstdlib>

#include "dqmc_b200.h"
#include "launch.cuh"

namespace dq {

template <typename T, int BM, int BN, int BK, int WM, int WN, int ST, int MODE, bool TMA>
static int launch_gemm_form(const GemmArgs<T> &g, cudaStream_t st)
{
	using Cfg = GemmCfg<T, BM, BN, BK, WM, WN, ST, MODE>;
	if (raise_smem(k_gemm<T, BM, BN, BK, WM, WN, ST, MODE, TMA>, Cfg::SMEM_MAX, true) != cudaSuccess)
		return DQMC_E_ARG;
	// the grid's z extent is at most 65535: larger batches take several launches
	for (int b0 = 0; b0 < g.batch; b0 += 65535) {
		GemmArgs<T> gc = g;
		gc.b0 = b0;
		dim3 grid((g.M + BM - 1) / BM, (g.N + BN - 1) / BN, min(65535, g.batch - b0));
		k_gemm<T, BM, BN, BK, WM, WN, ST, MODE, TMA>
			<<<grid, Cfg::THREADS, Cfg::smem_bytes(MODE, g.K, TMA), st>>>(gc);
	}
	return 0;
}

// the TMA form wherever tensor maps describe both operands (not the row
// gather, whose rows come from a table); the element-wise form otherwise.
// DQMC_GEMM_TMA=0 in the environment selects the element-wise form always.
template <typename T, int BM, int BN, int BK, int WM, int WN, int ST, int MODE>
static int launch_gemm_mode(const GemmArgs<T> &g, cudaStream_t st)
{
	using Cfg = GemmCfg<T, BM, BN, BK, WM, WN, ST, MODE>;
	if constexpr (!(MODE & GM_B_GATHER)) {
		static const bool off = [] {
			const char *e = getenv("DQMC_GEMM_TMA");
			return e && e[0] == '0';
		}();
		constexpr int ED = is_cplx<T>::value ? 2 : 1;
		GemmArgs<T> gt = g;
		if (!off &&
		    tma_map_operand(&gt.tmA, &gt.tzA, &gt.twA, g.A, ED, Cfg::A_CT ? g.K : g.M, Cfg::A_CT ? g.M : g.K, g.lda,
		                    g.aA, g.batch, Cfg::SA, Cfg::NA) &&
		    ((MODE & GM_B_IDENT) ||
		     tma_map_operand(&gt.tmB, &gt.tzB, &gt.twB, g.B, ED, Cfg::B_CT ? g.N : g.K, Cfg::B_CT ? g.K : g.N, g.ldb,
		                     g.aB, g.batch, Cfg::SB, Cfg::NBOX)))
			return launch_gemm_form<T, BM, BN, BK, WM, WN, ST, MODE, true>(gt, st);
	}
	return launch_gemm_form<T, BM, BN, BK, WM, WN, ST, MODE, false>(g, st);
}

template <typename T, int BM, int BN, int BK, int WM, int WN, int ST>
static int launch_gemm_cfg(const GemmArgs<T> &g, cudaStream_t st)
{
	switch (g.mode) {
	case 0: return launch_gemm_mode<T, BM, BN, BK, WM, WN, ST, 0>(g, st);
	case GM_A_DD: return launch_gemm_mode<T, BM, BN, BK, WM, WN, ST, GM_A_DD>(g, st);
	case GM_B_ROWD: return launch_gemm_mode<T, BM, BN, BK, WM, WN, ST, GM_B_ROWD>(g, st);
	case GM_B_COLD: return launch_gemm_mode<T, BM, BN, BK, WM, WN, ST, GM_B_COLD>(g, st);
	case GM_B_IDENT: return launch_gemm_mode<T, BM, BN, BK, WM, WN, ST, GM_B_IDENT>(g, st);
	case GM_A_CT: return launch_gemm_mode<T, BM, BN, BK, WM, WN, ST, GM_A_CT>(g, st);
	case GM_B_CT: return launch_gemm_mode<T, BM, BN, BK, WM, WN, ST, GM_B_CT>(g, st);
	case GM_A_UPPER | GM_B_GATHER:
		return launch_gemm_mode<T, BM, BN, BK, WM, WN, ST, GM_A_UPPER | GM_B_GATHER>(g, st);
	default: return DQMC_E_ARG;
	}
}

// Tile choice.  A launch that leaves SMs idle is bound by one CTA's chain
// (launch, first TMA round trip, K in steps), so few matrices take the smallest
// tiles, whose CTAs have one 8 x 8 DMMA per warp and step: us a launch in a
// graph, 16 / 32 / 48-64 tiles, real: N = 64 x 2 2.5 / 3.6 / 6.6, N = 144 x 2
// 3.8 / 5.6 / 9.5, x 16 8.7 / 7.1 / 9.6, x 64 21.7 / 20.7 / 16.3; complex
// N = 100 x 2 4.8 / 8.8 / 19.3, x 32 15.4 / 18.6 / 19.4.  The lines lie where
// the next tile overtakes: about 1000 CTAs of 16 x 16 (complex 1600), 600 of
// 32 x 32 (real).  Beyond, the whole CTAs per SM count, times what a CTA of the tile
// takes (gemm_tile_cost), larger tiles on ties: N = 100 x 512 53 us with 56 (64: 69),
// N = 196 x 256 137 with 40 (32: 178), N = 75 x 512 31 with 40 (48: 35), complex N =
// 100 x 512 191 with 56 (64: 217); 1000 x 1000 70 with 48 (40, the least padded area:
// 99), complex N = 156 x 512 488 with 32 (40: 550).  Over 410 launches of 16 to 4000
// rows the choice takes 2.7% more than the fastest tile, the least padded area 5%, with
// 64, 48 and 32 alone 13%.

// a CTA of tile t at depth K, per entry of the tile: fitted to those launches with more
// than 900 CTAs (relative units; slope in K, and what the prologue and the stores
// add)
inline long long gemm_tile_cost(bool cplx, int t, int K)
{
	switch (t) {
	case 64: return cplx ? 228ll * K + 3400 : 61ll * K + 2500;
	case 56: return cplx ? 262ll * K + 3550 : 74ll * K + 1600;
	case 48: return cplx ? 227ll * K + 3800 : 66ll * K + 1950;
	case 40: return cplx ? 274ll * K + 1950 : 75ll * K + 1850;
	default: return cplx ? 236ll * K + 3150 : 70ll * K + 3150;
	}
}

inline int gemm_tile(bool cplx, int batch, int M, int N, int K)
{
	auto ctas = [&](int t) { return (long long)batch * ((M + t - 1) / t) * ((N + t - 1) / t); };
	if (ctas(16) <= (cplx ? 1600 : 1024)) return 16;
	if (!cplx && ctas(32) <= 600) return 32;
	auto cost = [&](int t) { return (ctas(t) + 147) / 148 * t * t * gemm_tile_cost(cplx, t, K); };
	int best = 64;
	for (int t : {56, 48, 40, 32})
		if (cost(t) < cost(best)) best = t;
	return best;
}

template <typename T>
int launch_gemm(const GemmArgs<T> &g, cudaStream_t st)
{
	// the scale vectors and gather indices of these modes are staged per K
	const bool k_staged = g.mode & (GM_A_DD | GM_B_ROWD | GM_B_GATHER);
	if ((k_staged && g.K > 512) || g.M < 1 || g.N < 1 || g.K < 1 || g.batch < 1) return DQMC_E_ARG;
	const int best = gemm_tile(is_cplx<T>::value, g.batch, g.M, g.N, g.K);
	if constexpr (is_cplx<T>::value) {
		switch (best) {
		case 64: return launch_gemm_cfg<T, 64, 64, 8, 4, 2, 3>(g, st);
		case 56: return launch_gemm_cfg<T, 56, 56, 8, 1, 7, 3>(g, st);
		case 48: return launch_gemm_cfg<T, 48, 48, 8, 2, 2, 3>(g, st);
		case 40: return launch_gemm_cfg<T, 40, 40, 8, 1, 5, 3>(g, st);
		case 16: return launch_gemm_cfg<T, 16, 16, 16, 2, 2, 3>(g, st);
		default: return launch_gemm_cfg<T, 32, 32, 8, 2, 2, 3>(g, st);
		}
	} else {
		switch (best) {
		case 64: return launch_gemm_cfg<T, 64, 64, 16, 2, 2, 3>(g, st);
		case 56: return launch_gemm_cfg<T, 56, 56, 8, 1, 7, 3>(g, st);
		// k-depth 8: 24-28 KB per CTA, 7-8 CTAs per SM (2-5% over k-depth 16
		// with its 4-5 CTAs at 512 x 144^3)
		case 48: return launch_gemm_cfg<T, 48, 48, 8, 2, 2, 3>(g, st);
		case 40: return launch_gemm_cfg<T, 40, 40, 8, 1, 5, 3>(g, st);
		case 16: return launch_gemm_cfg<T, 16, 16, 32, 2, 2, 3>(g, st);
		default: return launch_gemm_cfg<T, 32, 32, 16, 2, 2, 4>(g, st);
		}
	}
}

}  // namespace dq
