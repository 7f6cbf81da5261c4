// Launch of the sweep kernels; included by the nine translation units
// sweep_<descriptor>_<fast|exact|fp16s>.cu, each of which instantiates one
// part (sweep_dispatch.cuh picks the part at run time).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "sweep.cuh"
#include "launch_util.cuh"
#include "sweep_dispatch.cuh"
#include "sweep_rows.cuh"
#include "sweep_tile.cuh"

namespace kel {
namespace gb {

// Row pipeline: persistent grid of (resident CTAs per SM) x SMs, capped at the
// row count.  The shared-memory opt-in and the occupancy query run once per
// kernel variant, device, row length and stage count (one cached entry).
// Any grid size is correct (rows are dealt round-robin to the CTAs); the
// occupancy only makes all CTAs resident at once.
template <class L, int STORE, bool ODD, int COLL, bool EXACT>
static cudaError_t launch_rows(const SweepParams &p, cudaStream_t st) {
	auto kern = sweep_rows_kernel<L, STORE, ODD, COLL, EXACT>;
	const int smem = rows_smem_bytes(L::Q, p.nxp, (int)sizeof(typename Store<STORE>::T), p.stages);
	const int threads = ((p.nxp + 31) & ~31) + 32; // consumers (one per cell) + the producer warp
	// one atomic word: device + 1 (bits 48-63), stages (40-47), nxp (16-39), CTAs per SM (0-15)
	static std::atomic<uint64_t> cached{0};
	int dev = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e != cudaSuccess) return e;
	const uint64_t key = (static_cast<uint64_t>(dev + 1) << 48) | (static_cast<uint64_t>(p.stages & 0xff) << 40) |
						 (static_cast<uint64_t>(p.nxp & 0xffffff) << 16);
	const uint64_t hit = cached.load();
	int per_sm = 0;
	if ((hit & ~static_cast<uint64_t>(0xffff)) == key) {
		per_sm = static_cast<int>(hit & 0xffff);
	} else {
		// opt in to the device's whole per-block shared memory, so that no
		// later call with a smaller footprint can lower it under another thread
		int optin = 0;
		if ((e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
		if (smem > optin) return cudaErrorInvalidConfiguration;
		if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin)) != cudaSuccess) return e;
		if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem)) != cudaSuccess) return e;
		if (per_sm < 1) return cudaErrorInvalidConfiguration;
		cached.store(key | static_cast<uint64_t>(per_sm & 0xffff));
	}
	const int64_t rows = static_cast<int64_t>(p.ny) * p.nz;
	const int64_t slots = static_cast<int64_t>(per_sm) * (p.sms > 0 ? p.sms : 1);
	const unsigned grid = static_cast<unsigned>(rows < slots ? rows : slots);
	kern<<<grid, threads, smem, st>>>(p);
	return cudaGetLastError();
}

// Whether a one-cell sweep overlaps its neighbours on the stream.  It saves about 2 us
// per launch, but not for free:
//  - a block's griddepcontrol instructions go through a unit that serves about 1,000
//    blocks per us, so many blocks of little work each are bound by it (D2Q9 FP32, 32 x
//    65,000: 66 us overlapped, 41 without the instructions; 64 x 39,062 41 and 34;
//    128 x 19,531 25.6 and 29.0; D3Q19 32 x 280 x 280 82 and 73, D3Q27 32 x 177 x 177, of
//    27 populations a cell, 40 and 46);
//  - inside a graph, where a launch costs little, a 3D grid of whole blocks that fills
//    half to three quarters of the SMs' slots lets the next grid's first blocks take
//    the free ones unevenly (D3Q19 FP32 512 x 14 x 14, 784 blocks on 152 SMs of 8: 5.3 us
//    per step overlapped, 5.0 without; fuller grids gain: 128 x 33 x 33 4.9 and 5.6).
static bool sweep1_overlaps(const SweepParams &p, int Q, int D, int block) {
	const int64_t rows = (int64_t)p.ny * p.nz, blocks = (p.nxp + block - 1) / block * rows;
	if (blocks > 16384 && p.nxp * rows * Q < 650 * blocks) return false;
	const int slots = p.sms * (1024 / block); // 64 registers per thread
	return !(p.overlap == OVERLAP_GRAPH && D == 3 && p.nxp % block == 0 && blocks > slots / 2 && blocks <= slots * 3 / 4);
}

// One cell per thread: the grid, and the prefetch distance -- the block one
// resident wave later (32 warps per SM at most: 1024 / block blocks on each
// SM; measured at 256^3: D3Q19 FP32 0.92 -> 0.97 of HBM, FP16S 0.50 -> 0.55,
// D3Q27 FP32 0.88 -> 0.95; two or three waves ahead gained less) -- in the
// grid's coordinates.
template <class L, int STORE, bool ODD, int COLL, bool EXACT, bool HW = false>
static cudaError_t launch_sweep1(SweepParams p, int block, cudaStream_t st) {
	const dim3 grid((p.nxp + block - 1) / block, p.ny, p.nz);
	const bool overlap = p.overlap && sweep1_overlaps(p, L::Q, L::D, block);
	const int ahead = p.sms * (1024 / block);
	p.pf_x = ahead % (int)grid.x;
	p.pf_y = ahead / (int)grid.x % (int)grid.y;
	p.pf_z = ahead / (int)grid.x / (int)grid.y;
	const int lines = block * (int)sizeof(typename Store<STORE>::T) / 128;
	p.pf_shift = lines >= 8 ? 3 : (lines >= 4 ? 2 : (lines >= 2 ? 1 : 0));
	auto go = [&](auto kern) { return launch_overlapped(kern, grid, block, 0, st, overlap, p); };
	if (!p.idx32) return go(sweep1_kernel<L, STORE, ODD, COLL, EXACT, HW, false>);
	if constexpr (!HW)
		if (!overlap) return go(sweep1_kernel<L, STORE, ODD, COLL, EXACT, false, true, false>);
	return go(sweep1_kernel<L, STORE, ODD, COLL, EXACT, HW, true>);
}

template <class L, int STORE, bool ODD, int COLL, bool EXACT>
static cudaError_t launch_variant(const SweepParams &p, cudaStream_t st) {
	const int block = p.block > 0 ? p.block : 256;
	if (p.hw_mask) { // half-way walls: the one-cell sweep only (other shapes fall back to it)
		return launch_sweep1<L, STORE, ODD, COLL, EXACT, true>(p, p.cpt == 1 ? block : 256, st);
	}
	if (p.cpt == CPT_ROWS) return launch_rows<L, STORE, ODD, COLL, EXACT>(p, st);
	if (p.cpt == 2) {
		const int64_t threads = static_cast<int64_t>(p.ny) * p.nz * p.wpr2 * 32;
		const int64_t blocks = (threads + block - 1) / block;
		if constexpr (STORE == STORE_FP16S) // nxp is even in FP16S storage
			sweep2h_kernel<L, ODD, COLL, EXACT><<<static_cast<unsigned>(blocks), block, 0, st>>>(p);
		else
			sweep2_kernel<L, STORE, ODD, COLL, EXACT><<<static_cast<unsigned>(blocks), block, 0, st>>>(p);
		return cudaGetLastError();
	}
	if constexpr (COLL == COLL_HLBM) { // one cell per thread only
		return launch_sweep1<L, STORE, ODD, COLL, EXACT>(p, block, st);
	} else if (p.cpt == 1) {
		return launch_sweep1<L, STORE, ODD, COLL, EXACT>(p, block, st);
	} else {
		const int64_t threads = static_cast<int64_t>(p.ny) * p.nz * p.wpr * 32;
		const int64_t blocks = (threads + block - 1) / block;
		sweep_kernel<L, STORE, ODD, COLL, EXACT><<<static_cast<unsigned>(blocks), block, 0, st>>>(p);
	}
	return cudaGetLastError();
}

template <class L, int STORE, bool ODD, bool EXACT>
static cudaError_t launch_coll(const SweepParams &p, int coll, cudaStream_t st) {
	switch (coll) {
	case COLL_BGK: return launch_variant<L, STORE, ODD, COLL_BGK, EXACT>(p, st);
	case COLL_BGK_GUO: return launch_variant<L, STORE, ODD, COLL_BGK_GUO, EXACT>(p, st);
	case COLL_PSM: return launch_variant<L, STORE, ODD, COLL_PSM, EXACT>(p, st);
	case COLL_PSM_GUO: return launch_variant<L, STORE, ODD, COLL_PSM_GUO, EXACT>(p, st);
	case COLL_HLBM:
		if constexpr (L::Q == 9) return launch_variant<L, STORE, ODD, COLL_HLBM, EXACT>(p, st);
		return cudaErrorInvalidValue;
	}
	return cudaErrorInvalidValue;
}

// One part of the variant set (the translation units compile one part each,
// in parallel): FP32 fast arithmetic, FP32 reference arithmetic, FP16S.
template <class L, int PART>
cudaError_t launch_sweep_part(const SweepParams &p, bool odd, int coll, cudaStream_t st) {
	if constexpr (PART == PART_FAST32)
		return odd ? launch_coll<L, STORE_FP32, true, false>(p, coll, st) : launch_coll<L, STORE_FP32, false, false>(p, coll, st);
	else if constexpr (PART == PART_EXACT32)
		return odd ? launch_coll<L, STORE_FP32, true, true>(p, coll, st) : launch_coll<L, STORE_FP32, false, true>(p, coll, st);
	else
		return odd ? launch_coll<L, STORE_FP16S, true, false>(p, coll, st)
				   : launch_coll<L, STORE_FP16S, false, false>(p, coll, st);
}

template <int STORE, int COLL, class TS>
static cudaError_t launch_tile_variant(const TileParams &q, cudaStream_t st) {
	static std::atomic<uint64_t> done{0};
	auto kern = sweep_tile_kernel<STORE, COLL, TS>;
	const int smem = tile_smem(TS::W, TS::K, q.ty, (int)sizeof(typename TileStore<STORE>::T));
	cudaError_t e = allow_smem(kern, smem, done);
	if (e != cudaSuccess) return e;
	constexpr int TX = TS::W - 2 * TS::K;
	const dim3 grid((q.p.nxp + TX - 1) / TX, (q.p.ny + q.ty - 1) / q.ty);
	return launch_overlapped(kern, grid, TS::NT, smem, st, q.p.overlap != 0, q);
}

template <int PART>
cudaError_t launch_tile_part(const TileParams &q, int coll, bool wide, cudaStream_t st) {
	constexpr int STORE = PART == PART_FP16S ? STORE_FP16S : STORE_FP32;
	auto go = [&](auto c) -> cudaError_t { // wide tiles: FP32, and not with PSM and a force (plan_tiles)
		constexpr int C = decltype(c)::value;
		if constexpr (STORE == STORE_FP32 && C != COLL_PSM_GUO)
			if (wide) return launch_tile_variant<STORE, C, TileWide>(q, st);
		return wide ? cudaErrorInvalidValue : launch_tile_variant<STORE, C, TileSmall>(q, st);
	};
	switch (coll) {
	case COLL_BGK: return go(std::integral_constant<int, COLL_BGK>());
	case COLL_BGK_GUO: return go(std::integral_constant<int, COLL_BGK_GUO>());
	case COLL_PSM: return go(std::integral_constant<int, COLL_PSM>());
	case COLL_PSM_GUO: return go(std::integral_constant<int, COLL_PSM_GUO>());
	}
	return cudaErrorInvalidValue;
}

} // namespace gb
} // namespace kel
