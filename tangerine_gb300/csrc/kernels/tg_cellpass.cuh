// The cell pass of one brick (surface nets' active cells) and the brick geometry it shares
// with the brick evaluation.
#pragma once

#include "tg_device.cuh"
#include "tg_kernels.hpp"
#include "tg_surface.cuh"

namespace tg
{
	struct BrickGrid
	{
		int B;                  // cells per brick edge
		int NBX, NBY, NBZ;      // bricks per axis
	};

	// The cells of listed bricks, a CTA per brick with a grid stride over the list.
	// Cells of unlisted bricks hold no surface and are never visited: the active-cell
	// bitmask starts zeroed and only listed cells can set their bit.
	struct BrickCells
	{
		int64_t i0, j0, k0;
		int nx, ny, nz;
	};

	__device__ __forceinline__ BrickCells CellsOf(uint32_t b, const BrickGrid& bg, const CellGeom& cg)
	{
		const int bx = (int)(b % (uint32_t)bg.NBX), by = (int)((b / (uint32_t)bg.NBX) % (uint32_t)bg.NBY);
		const int bz = (int)(b / ((uint32_t)bg.NBX * (uint32_t)bg.NBY));
		BrickCells bc;
		bc.i0 = (int64_t)bx * bg.B; bc.j0 = (int64_t)by * bg.B; bc.k0 = (int64_t)bz * bg.B;
		bc.nx = (int)min((int64_t)bg.B, cg.sx - bc.i0);
		bc.ny = (int)min((int64_t)bg.B, cg.sy - bc.j0);
		bc.nz = (int)min((int64_t)bg.B, cg.sz - bc.k0);
		return bc;
	}

	constexpr int kTiledBox = 8;
	constexpr int kTiledThreads = 128;
	constexpr int kTiledRounds = 3;   // 7^3 = 343 cells <= 3 x 128

	// BT: the brick edge in cells when known at compile time (the cell coordinates then
	// come from constant divisions, edge bricks masking their missing cells), or 0.
	// The cell pass of one kept brick from its corner box in shared memory (kTiledBox^3,
	// x fastest): every cell with corners of both signs sets its bit in `words` and is
	// appended to `cells` (one atomic per brick).  Called by the whole CTA (it
	// synchronises); `warpBase` is shared scratch, one word per warp.
	template<int BT, int Threads = kTiledThreads>
	__device__ __forceinline__ void BrickCellFlags(const float* box, const BrickCells& bc, const CellGeom& cg, uint32_t* __restrict__ words,
		uint32_t* __restrict__ cells, uint32_t* __restrict__ cell_count, uint32_t* warpBase)
	{
		constexpr int kRounds = (7 * 7 * 7 + Threads - 1) / Threads;
		const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
		const int ex = BT ? BT : bc.nx, ey = BT ? BT : bc.ny;
		const int total = BT ? BT * BT * BT : bc.nx * bc.ny * bc.nz;
		const int64_t sxy = cg.sx * cg.sy;
		const int64_t c0 = bc.i0 + bc.j0 * cg.sx + bc.k0 * sxy;
		unsigned ballots[kRounds];
		uint32_t cellOf[kRounds];
		uint32_t mine = 0;
#pragma unroll
		for (int r = 0; r < kRounds; ++r)
		{
			const int t = r * Threads + (int)threadIdx.x;
			bool active = false;
			cellOf[r] = 0;
			const int x = t % ex, y = (t / ex) % ey, z = t / (ex * ey);
			if (t < total && x < bc.nx && y < bc.ny && z < bc.nz)
			{
				const float* b = box + (z * kTiledBox + y) * kTiledBox + x;
				constexpr int dy = kTiledBox, dz = kTiledBox * kTiledBox;
				const float v[8] = { b[0], b[1], b[dy + 1], b[dy], b[dz], b[dz + 1], b[dz + dy + 1], b[dz + dy] };
				unsigned pos = 0;
#pragma unroll
				for (int q = 0; q < 8; ++q) pos |= (v[q] >= 0.0f ? 1u : 0u) << q;
				active = pos != 0u && pos != 0xFFu;
				const int64_t c = c0 + x + y * cg.sx + z * sxy;
				cellOf[r] = (uint32_t)c;
				if (active) atomicOr(words + (c >> 5), 1u << (c & 31));
			}
			ballots[r] = __ballot_sync(0xFFFFFFFFu, active);
			mine += (uint32_t)__popc(ballots[r]);
		}
		if (lane == 0) warpBase[warp] = mine;
		__syncthreads();
		if (threadIdx.x == 0)
		{
			uint32_t sum = 0;
			uint32_t counts[Threads / 32];
#pragma unroll
			for (int w = 0; w < Threads / 32; ++w) { counts[w] = warpBase[w]; sum += counts[w]; }
			uint32_t at = sum ? atomicAdd(cell_count, sum) : 0u;
#pragma unroll
			for (int w = 0; w < Threads / 32; ++w) { warpBase[w] = at; at += counts[w]; }
		}
		__syncthreads();
		uint32_t at = warpBase[warp];
		const unsigned below = (1u << lane) - 1u;
#pragma unroll
		for (int r = 0; r < kRounds; ++r)
		{
			if ((ballots[r] >> lane) & 1u) cells[at + __popc(ballots[r] & below)] = cellOf[r];
			at += (uint32_t)__popc(ballots[r]);
		}
	}

	inline BrickGrid MakeBrickGrid(const GridSpec& g, int B)
	{
		return { B, (g.NX - 1 + B - 1) / B, (g.NY - 1 + B - 1) / B, (g.NZ - 1 + B - 1) / B };
	}
}
