// Launchers of the dense per-matrix kernels (qr.cuh): the shared-memory or
// global-memory form by N, and the rows-per-lane instantiation.  Included by
// the launch_{qrb,qrp,rec}_{r,c}.cu translation units only.
#pragma once

#include "dqmc_b200.h"
#include "launch.cuh"

namespace dq {

// rows per lane of a warp column: 32 * RPL >= N
#define DQ_RPL(X) X(32, 1) X(64, 2) X(96, 3) X(128, 4) X(160, 5) X(192, 6) X(224, 7) X(256, 8)

// for matrices beyond one SM's shared memory (N > 100)
#define DQ_RPL_BIG(X) X(128, 4) X(160, 5) X(192, 6) X(224, 7) X(256, 8)

// 226 KB leaves room for the kernels' static shared memory
static const size_t SMEM_FIT = 226 * 1024;
// beside the panel's shared variables
template <typename T>
constexpr size_t qr_panel_fit() { return 227 * 1024 - sizeof(PanelShared<T, 4>) - 256; }

// carve: the shared-memory forms take the largest shared-memory carveout
// (room for a GEMM CTA beside them); the global-memory forms keep the
// default, whose L1 serves their working matrix
template <typename K, typename Args>
static int launch_dense(K kern, const Args &a, size_t sm, cudaStream_t st, bool carve)
{
	if (raise_smem(kern, sm, carve) != cudaSuccess) return DQMC_E_ARG;
	kern<<<a.batch, 512, sm, st>>>(a);
	return 0;
}

template <typename T, int RPL, bool GM>
static int launch_qrb_rpl(const QrArgs<T> &a, cudaStream_t st)
{
	return launch_dense(k_qrb<T, 16, 8, RPL, GM>, a, qrb_smem_bytes<T, 8>(a.N, GM), st, !GM);
}

// CTAs of the cluster form: as few as hold the matrix (two items of
// N = 196 on 2 / 4 / 8: 384 / 345 / 352 us, 128 items 788 / 1403 / 3195)
template <typename T>
static int qrc_ctas(int N)
{
	int P = 2;
	while (P < 8 && qrc_smem_bytes<T>(N, P) > qr_panel_fit<T>()) P *= 2;
	return P;
}

template <typename T, int RPL>
static int launch_qrc_rpl(const QrArgs<T> &a, cudaStream_t st)
{
	const int P = qrc_ctas<T>(a.N);
	const size_t sm = qrc_smem_bytes<T>(a.N, P);
	auto kern = k_qrc<T, 16, RPL>;
	if (sm > qr_panel_fit<T>() || raise_smem(kern, sm, true) != cudaSuccess) return DQMC_E_ARG;
	cudaLaunchConfig_t cfg = {};
	cudaLaunchAttribute at = {};
	at.id = cudaLaunchAttributeClusterDimension;
	at.val.clusterDim.x = P;
	at.val.clusterDim.y = at.val.clusterDim.z = 1;
	cfg.gridDim = dim3(P * a.batch);
	cfg.blockDim = dim3(512);
	cfg.dynamicSmemBytes = sm;
	cfg.stream = st;
	cfg.attrs = &at;
	cfg.numAttrs = 1;
	return cudaLaunchKernelEx(&cfg, kern, a, P) == cudaSuccess ? 0 : DQMC_E_CUDA;
}

template <typename T, int RPL, bool GM>
static int launch_qrp_rpl(const QrArgs<T> &a, cudaStream_t st)
{
	return launch_dense(k_qrp<T, 16, 8, RPL, GM>, a, qrp_smem_bytes<T, 8>(a.N, GM), st, !GM);
}

template <typename T, bool GM>
static int launch_qrp_gm(const QrArgs<T> &a, cudaStream_t st)
{
#define X(NMAX, R) if (a.N <= NMAX) return launch_qrp_rpl<T, R, GM>(a, st);
	DQ_RPL(X)
#undef X
	return DQMC_E_ARG;
}

template <typename T>
int launch_qr_presort(const QrArgs<T> &a, cudaStream_t st)
{
	if (a.N < 1 || a.N > max_dense_n<T>()) return DQMC_E_ARG;
	if (qrb_smem_bytes<T, 8>(a.N) <= qr_panel_fit<T>()) {
#define X(NMAX, R) if (a.N <= NMAX) return launch_qrb_rpl<T, R, false>(a, st);
		DQ_RPL(X)
#undef X
	}
	if (!a.work) return DQMC_E_ARG;
	// A cluster per item while all of them run at once, else one SM per item with
	// the matrix in L2 (us a launch, cluster / L2: N = 196 x 4 384 / 442, x 128
	// 788 / 461; N = 256 x 8 484 / 1210, x 32 507 / 1204, x 128 1978 / 1397; complex
	// N = 144 x 4 438 / 557, x 64 457 / 565, x 128 911 / 592;
	// N = 256 x 4 888 / 2063)
	const bool cl = (long long)qrc_ctas<T>(a.N) * a.batch <= 128;
#define X(NMAX, R) if (a.N <= NMAX) return cl ? launch_qrc_rpl<T, R>(a, st) : launch_qrb_rpl<T, R, true>(a, st);
	DQ_RPL_BIG(X)
#undef X
	return DQMC_E_ARG;
}

template <typename T>
int launch_qr_pivot(const QrArgs<T> &a, cudaStream_t st)
{
	if (a.N < 1 || a.N > max_dense_n<T>()) return DQMC_E_ARG;
	if (qrp_smem_bytes<T, 8>(a.N) <= SMEM_FIT) return launch_qrp_gm<T, false>(a, st);
	if (!a.work) return DQMC_E_ARG;
	return launch_qrp_gm<T, true>(a, st);
}

template <typename T, int RPL, bool GM>
static int launch_rec_rpl(const RecArgs<T> &a, cudaStream_t st)
{
	return launch_dense(k_recb<T, 16, RPL, GM>, a, recb_smem_bytes<T>(a.N, GM), st, !GM);
}

template <typename T, bool GM>
static int launch_rec_gm(const RecArgs<T> &a, cudaStream_t st)
{
#define X(NMAX, R) if (a.N <= NMAX) return launch_rec_rpl<T, R, GM>(a, st);
	DQ_RPL(X)
#undef X
	return DQMC_E_ARG;
}

template <typename T>
int launch_rec(const RecArgs<T> &a, cudaStream_t st)
{
	if (a.N < 1 || a.N > max_dense_n<T>()) return DQMC_E_ARG;
	if (recb_smem_bytes<T>(a.N) <= SMEM_FIT) return launch_rec_gm<T, false>(a, st);
	if (!a.work) return DQMC_E_ARG;
	return launch_rec_gm<T, true>(a, st);
}

}  // namespace dq
