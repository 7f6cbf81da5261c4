// Several time steps of a D2Q9 lattice per launch, on tiles in shared memory.
//
// A block loads its tile and a ring of K cells around it, runs K steps
// on it and writes the tile's populations of K steps later to a
// second array.  Each step's valid region is one ring smaller than the one
// before, so the rings hold copies of cells that the neighbouring blocks
// compute too (the same operations on the same values: the same bits).
//
// Why: a 2D sweep moves 73 bytes per cell and step and is over in a few
// microseconds.  Small lattices are bound by one launch per step, lattices
// beyond the L2 by HBM.  Here a cell is read and written once per K steps and
// the steps between find their populations at constant offsets from one
// shared-memory address; the price is the ring, computed redundantly (1.3 to
// 1.6 times the tile's cells, by tile height) and, for boundary steps other than
// bounce-back, a call per cell.  Tiles and the one-step sweep, us per step of 20 in
// FP32 (x periodic between walls; a channel with Zou-He ends in brackets):
//   BGK   256x64 1.3 / 2.1 (1.9 / 2.3), 512x128 1.6 / 2.7 (2.4 / 2.9), 400x240 1.9 / 3.0
//         (333x290 2.9 / 3.0), 1900x1752 27 / 32 (30 / 33), 2048^2 33 / 42 (37 / 43),
//         4096^2 129 / 188 (135 / 189); between the last small and the first large one
//         the L2 holds the lattice and the one-step sweep is the faster one;
//   a force costs the tiles more: 0.72 of the one-step sweep's time at 256x64 (0.95), 0.84
//         at 400x240 (1.14 at 333x290), 1.04 at 1900x1752, 0.90 at 2640x2600 (0.95);
//   PSM   0.66 at 256x64 (0.95), 0.92 at 1900x1752 (1.01), 0.84 at 4096^2 (0.86); with a
//         force 0.76 (1.03) at 256x64, 1.02 to 1.07 beyond the L2;
//   columns that a row fills badly: 200x24000 0.72 (1.04), 120x50000 0.83 (1.26);
//   FP16S beyond its L2 size (2640x2600 and more) 1.04 to 1.38: none there.
// In the reference's arithmetic the one-step sweep is faster at every size from
// 256x64 up (3.2 / 3.1 there, 4096^2 438 / 300: the ring repeats an expensive collision).
//
// Inside the tile the populations are in the AA layout of sweep.cuh (one copy
// in shared memory, each slot read and written by the same cell within a
// step, one barrier between steps): an even step reads slot i and writes slot
// opp i of its own cell, an odd step reads slot opp i of x - c_i and writes
// slot i of x + c_i.  K is even and a launch starts at an even time step,
// so both arrays are in the even-step layout.  Cells outside the lattice are
// flag-0 cells, which emit the ghost ring's zeros.
#pragma once

#include "sweep.cuh"

namespace kel {
namespace gb {

// A tile shape: W cells of a region row, K steps per launch (the ring), R rows
// per thread, NT threads per block, BPS blocks per SM the registers allow.
template <int W_, int K_, int R_, int NT_, int BPS_>
struct TileShape {
	static constexpr int W = W_, K = K_, R = R_, NT = NT_, BPS = BPS_;
};
constexpr int TILE_K = 4;
// Wide, for lattices beyond the L2: the least redundant work, two cells per
// instruction (120 instructions per cell and step; 4096^2 118 us per step,
// Small 129).  Small, for small lattices: one cell per thread, more blocks
// (256x64 in an earlier form 1.5 us per step, Wide 2.3).  Eight steps per launch lose
// more to the ring than they save in launches (1.8 there).
using TileWide = TileShape<64, TILE_K, 2, 384, 2>;
using TileSmall = TileShape<32, TILE_K, 1, 512, 2>;

// Populations of a tile in shared memory: [row][direction][W] in the
// lattice's storage type, so that every offset from a cell is a constant.
template <int STORE>
struct TileStore;

template <>
struct TileStore<STORE_FP32> {
	using T = float;
	__device__ static __forceinline__ float ld(const T *a, float) { return *a; }
	__device__ static __forceinline__ void st(T *a, float v, float) { *a = v; }
};

// FP16S: every step's populations pass through the half storage, as they do
// in global memory (the same rounding).
template <>
struct TileStore<STORE_FP16S> {
	using T = __half;
	__device__ static __forceinline__ float ld(const T *a, float s) {
		float r;
		asm("add.rn.f32.f16 %0, %1, %2;" : "=f"(r) : "h"(__half_as_ushort(*a)), "f"(s));
		return r;
	}
	__device__ static __forceinline__ void st(T *a, float v, float s) { *a = __float2half_rn(v - s); }
};

// Where a tile lies in the arrays it is read from and written to.
struct TileGeom {
	const void *in;
	void *out;
	int off[9];      // index of a cell's slot in plane i (9 planes < 2^31 cells)
	int base;        // index of the lattice's (channel's) first cell in plane 0
	int nxp, ny;     // its extents
	int periodic;
	int x0, y0;      // lattice coordinates of the region's first cell (the tile's minus K)
	int rows;        // rows of the region, even: tile rows + 2 K
	int t_end;       // the tile's rows: [K, t_end) of the region
	const uint8_t *flags;
};

// Two cells' values in one register pair: sm_103a's two-wide FP32 operations
// round each half as the scalar ones do.
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }
// A product that no later sum may absorb: a two-wide product (__fmul2_rn, and
// mul.rn.f32x2 too) may be fused into the two-wide sum that takes its result, one
// rounding less than the scalar operations have.  As two scalar products 0.5 % slower
// at 2048^2.
__device__ __forceinline__ float2 mul2_alone(float2 a, float2 b) { return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)); }

// collide<D2Q9, COLL_BGK, false> on two cells: the same operations in the
// same order, two cells per instruction.  The tile's steps are bound by
// instruction issue once their addresses are constants.
__device__ __forceinline__ void collide_bgk2(float (&fa)[9], float (&fb)[9], float omega) {
	using L = D2Q9;
	float2 f[9];
#pragma unroll
	for (int i = 0; i < 9; ++i) f[i] = make_float2(fa[i], fb[i]);
	float2 r = f[0], jx = neg2(f[1]), jy = neg2(f[3]);
#pragma unroll
	for (int j = 1; j < 9; ++j) {
		r = __fadd2_rn(r, f[j]);
		if (j > 1 && L::cx(j) != 0) jx = __fadd2_rn(jx, L::cx(j) > 0 ? f[j] : neg2(f[j]));
		if (j > 3 && L::cy(j) != 0) jy = __fadd2_rn(jy, L::cy(j) > 0 ? f[j] : neg2(f[j]));
	}
	const float2 ir = make_float2(__frcp_rn(r.x), __frcp_rn(r.y));
	const float2 ux = mul2_alone(jx, ir), uy = mul2_alone(jy, ir);
	const float2 vv = __fadd2_rn(mul2_alone(ux, ux), mul2_alone(uy, uy));
	const float2 nh = __fmul2_rn(both(-1.5f), vv), om = both(omega);
	auto relax = [&](float2 v, float2 eq) { return __ffma2_rn(om, __fadd2_rn(eq, neg2(v)), v); };
	const float2 w0 = __fmul2_rn(both((float)L::w(0)), r);
	f[0] = relax(f[0], __ffma2_rn(w0, nh, w0));
#pragma unroll
	for (int i = 1; i < 9; i += 2) { // opp(i) = i + 1
		const float2 cu = i == 1 ? neg2(ux) : (i == 3 ? neg2(uy) : __fadd2_rn(neg2(ux), i == 5 ? neg2(uy) : uy));
		const float2 vcc = mul2_alone(both(3.0f), cu);
		const float2 sym = __ffma2_rn(__fmul2_rn(both(0.5f), vcc), vcc, nh);
		const float2 wr = __fmul2_rn(both((float)L::w(i)), r);
		f[i] = relax(f[i], __ffma2_rn(wr, __fadd2_rn(vcc, sym), wr));
		f[i + 1] = relax(f[i + 1], __ffma2_rn(wr, __fadd2_rn(sym, neg2(vcc)), wr));
	}
#pragma unroll
	for (int i = 0; i < 9; ++i) {
		fa[i] = f[i].x;
		fb[i] = f[i].y;
	}
}

// A wall cell's full-way bounce-back, or (not a wall) a cell outside the lattice.
__device__ __forceinline__ void bounce_or_zero(float (&f)[9], bool wall) {
#pragma unroll
	for (int i = 1; i < 9; i += 2) { // opp(i) = i + 1
		const float t = f[i];
		f[i] = wall ? f[i + 1] : 0.f;
		f[i + 1] = wall ? t : 0.f;
	}
	f[0] = wall ? f[0] : 0.f;
}

// A cell's populations after its boundary step, and whether it collides then.
struct Bounded {
	float f[9];
	int collides;
};

// Out of line: the boundary kinds besides walls, which few cells have and
// whose code would otherwise be in every step of the tile.
static __device__ __noinline__ Bounded tile_boundary(const OpEntry *ops, const float *profile, float f0, float f1, float f2,
											  float f3, float f4, float f5, float f6, float f7, float f8, int flag, int y) {
	float f[9] = {f0, f1, f2, f3, f4, f5, f6, f7, f8};
	CellCtx ctx;
	ctx.ops = ops;
	ctx.profile = profile;
	Bounded r;
	r.collides = boundary_step<D2Q9, false>(f, flag, y, ctx);
#pragma unroll
	for (int i = 0; i < 9; ++i) r.f[i] = f[i];
	return r;
}

// The steps of one tile (a warp's lanes are neighbours in a row; a thread has
// the cells of its column in R consecutive rows at a time).  up.cells(f, c0,
// c1) collides R cells (c0, c1: their indices in plane 0); up.boundary(f,
// flag, y) is one cell's boundary step (flag 0: outside the lattice) and tells
// whether it collides; up.is_plain(flag): no boundary step.
// A cell that does not collide is stored straight after its boundary step (its
// slots are its own) and follows the others through the collision at rest.
template <int STORE, class TS, class Shift, class Cells>
__device__ __forceinline__ void tile_steps(const TileGeom &g, const Shift &shift, typename TileStore<STORE>::T *sm,
										   uint32_t *bnd, uint8_t *fl, const Cells &up) {
	using L = D2Q9;
	using S = TileStore<STORE>;
	using T = typename S::T;
	constexpr int K = TS::K, W = TS::W, R = TS::R, RS = R * TS::NT / W, PITCH = 9 * W, WPR = W / 32;
	constexpr unsigned FULL = 0xffffffffu;
	const int rx = (int)threadIdx.x % W, r0 = R * ((int)threadIdx.x / W), wx = rx >> 5;
	const int lx = g.x0 + rx;
	int gx = lx;
	if (g.periodic) { // the images of a cell evolve alike
		gx %= g.nxp;
		if (gx < 0) gx += g.nxp;
	}
	const bool x_in = gx >= 0 && gx < g.nxp;
	const T *const A = static_cast<const T *>(g.in);
	const int tx_end = min(W - K, g.nxp - g.x0);
	auto at = [&](int gy) { return x_in && gy >= 0 && gy < g.ny ? g.base + gy * g.nxp + gx : g.base; };

	// step 0 reads global memory, R rows ahead of the ones it collides
	float nf[R][9];
	int nfl[R]; // their flags
	auto fetch = [&](int ry) {
#pragma unroll
		for (int k = 0; k < R; ++k) {
			const int gy = g.y0 + ry + k, c = at(gy);
			const bool in = x_in && gy >= 0 && gy < g.ny;
			nfl[k] = in ? (int)g.flags[c] : 0;
#pragma unroll
			for (int i = 0; i < 9; ++i) nf[k][i] = in ? S::ld(A + (c + g.off[i]), shift(i)) : 0.f;
		}
	};
	// step m of row ry's R cells; rim[k]: lanes of row ry + k with a boundary step
	auto store = [&](int m, const float (&f)[9], int ry) {
		T *const s = sm + ry * PITCH + rx;
		if (m + 1 < K) {
#pragma unroll
			for (int i = 0; i < 9; ++i)
				S::st(s + ((m & 1) ? L::cy(i) * PITCH + i * W + L::cx(i) : L::opp(i) * W), f[i], shift(i));
		} else {
			// last step (odd): straight to the tile's cells in the other array
			// (from lx, not wrapped: a tile's cells lie in [0, nxp))
			T *const B = static_cast<T *>(g.out);
			const int to = g.base + (g.y0 + ry) * g.nxp + lx;
#pragma unroll
			for (int i = 0; i < 9; ++i) {
				const int tx = rx + L::cx(i), ty = ry + L::cy(i);
				if (tx >= K && tx < tx_end && ty >= K && ty < g.t_end)
					S::st(B + (to + g.off[i] + L::cx(i) + L::cy(i) * g.nxp), f[i], shift(i));
			}
		}
	};
	auto step = [&](int m, float (&f)[R][9], int ry, bool mine, const unsigned (&rim)[R]) {
		bool go[R];
#pragma unroll
		for (int k = 0; k < R; ++k) {
			go[k] = mine;
			if (rim[k]) {
				if (mine) go[k] = up.boundary(f[k], (int)fl[(ry + k) * W + rx], g.y0 + ry + k);
				if (mine && !go[k]) store(m, f[k], ry + k);
#pragma unroll
				for (int i = 0; i < 9; ++i) f[k][i] = go[k] ? f[k][i] : (float)L::w(i);
			}
		}
		const int gy = g.y0 + ry;
		up.cells(f, at(gy), at(gy + R - 1));
#pragma unroll
		for (int k = 0; k < R; ++k)
			if (go[k]) store(m, f[k], ry + k);
	};

	grid_dependency_wait(); // the launch before wrote the populations
	if (r0 < g.rows) fetch(r0);
#pragma unroll 1
	for (int ry = r0; ry < g.rows; ry += RS) { // step 0: every cell of the region
		float f[R][9];
		unsigned rim[R];
#pragma unroll
		for (int k = 0; k < R; ++k) {
#pragma unroll
			for (int i = 0; i < 9; ++i) f[k][i] = nf[k][i];
			fl[(ry + k) * W + rx] = (uint8_t)nfl[k];
			rim[k] = __ballot_sync(FULL, !up.is_plain(nfl[k]));
			if ((threadIdx.x & 31) == 0) bnd[(ry + k) * WPR + wx] = rim[k];
		}
		if (ry + RS < g.rows) fetch(ry + RS);
		step(0, f, ry, true, rim);
	}
	__syncthreads();
#pragma unroll
	for (int m = 1; m < K; ++m) { // step m: the cells at least m from the region's rim
		const bool mine = rx >= m && rx < W - m;
		const unsigned lanes = __ballot_sync(FULL, mine);
#pragma unroll 1
		for (int ry = m + r0; ry < g.rows - m; ry += RS) {
			// a rim lane's slots are other cells', which may be storing to them: it
			// reads nothing and follows the others at rest
			T *const s = sm + ry * PITCH + rx;
			float f[R][9];
			unsigned rim[R];
#pragma unroll
			for (int k = 0; k < R; ++k) {
				rim[k] = bnd[(ry + k) * WPR + wx] & lanes;
#pragma unroll
				for (int i = 0; i < 9; ++i)
					f[k][i] = mine ? S::ld(s + (k * PITCH + ((m & 1) ? -L::cy(i) * PITCH + L::opp(i) * W - L::cx(i) : i * W)),
										   shift(i))
								   : (float)L::w(i);
			}
			step(m, f, ry, mine, rim);
		}
		if (m + 1 < K) __syncthreads();
	}
}

struct TileParams {
	SweepParams p;
	void *out;
	int ty; // tile rows (a multiple of R)
};

// Shared memory of a tile of ty rows: populations, boundary bits, flags.
constexpr int tile_smem(int w, int k, int ty, int elem) { return (ty + 2 * k) * (w * (9 * elem + 1) + w / 32 * 4); }

template <int COLL>
struct LatticeCells {
	const SweepParams &p;
	__device__ __forceinline__ bool is_plain(int flag) const { return flag < MAX_FLAGS && ((p.plain >> flag) & 1u); }
	__device__ __forceinline__ bool boundary(float (&f)[9], int flag, int y) const {
		if (is_plain(flag)) return true;
		const bool wall = flag < MAX_FLAGS && ((p.bounce >> flag) & 1u);
		if (flag == 0 || wall) {
			bounce_or_zero(f, wall);
			return false;
		}
		const Bounded r = tile_boundary(p.ops, p.profile, f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7], f[8], flag, y);
#pragma unroll
		for (int i = 0; i < 9; ++i) f[i] = r.f[i];
		return r.collides != 0;
	}
	template <int R>
	__device__ __forceinline__ void cells(float (&f)[R][9], int c0, int c1) const {
		if constexpr (COLL == COLL_BGK && R == 2) {
			collide_bgk2(f[0], f[1], p.omega);
		} else {
#pragma unroll
			for (int k = 0; k < R; ++k) {
				const int c = k ? c1 : c0;
				float por = 1.f, Fc[3] = {0.f, 0.f, 0.f}, rho, u[3];
				if (COLL == COLL_PSM || COLL == COLL_PSM_GUO) por = p.por[c];
				if ((COLL == COLL_BGK_GUO || COLL == COLL_PSM_GUO) && p.force) {
					Fc[0] = p.force[c];
					Fc[1] = p.force[p.plane + c];
				}
				collide<D2Q9, COLL, false>(f[k], cell_ctx(p), por, Fc, rho, u);
			}
		}
	}
};

template <int STORE, int COLL, class TS>
__global__ void __launch_bounds__(TS::NT, TS::BPS) sweep_tile_kernel(const __grid_constant__ TileParams q) {
	using T = typename TileStore<STORE>::T;
	extern __shared__ __align__(16) unsigned char tile_mem[];
	const SweepParams &p = q.p;
	grid_dependents_launch();
	TileGeom g;
	g.in = p.f;
	g.out = q.out;
#pragma unroll
	for (int i = 0; i < 9; ++i) g.off[i] = p.off_even[i];
	g.base = 0;
	g.nxp = p.nxp;
	g.ny = p.ny;
	g.periodic = p.periodic;
	g.x0 = (int)blockIdx.x * (TS::W - 2 * TS::K) - TS::K;
	g.y0 = (int)blockIdx.y * q.ty - TS::K;
	// the last tiles' rows end at the lattice's (rounded up to whole R)
	const int left = p.ny - (int)blockIdx.y * q.ty;
	g.rows = min(q.ty, (left + TS::R - 1) / TS::R * TS::R) + 2 * TS::K;
	g.t_end = min(q.ty, left) + TS::K;
	g.flags = p.flags;
	const int cells = (q.ty + 2 * TS::K) * TS::W;
	T *const sm = reinterpret_cast<T *>(tile_mem);
	uint32_t *const bnd = reinterpret_cast<uint32_t *>(sm + 9 * cells);
	uint8_t *const fl = reinterpret_cast<uint8_t *>(bnd + cells / 32);
	tile_steps<STORE, TS>(g, [&](int i) { return p.wshift[i]; }, sm, bnd, fl, LatticeCells<COLL>{p});
}

} // namespace gb
} // namespace kel
