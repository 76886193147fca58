// The mesh export's 7^3-cell bricks through shortened programs (tg_parts.cuh): in a 512^3
// export of a 256-primitive tree the cells' programs hold a dozen records on average and a
// part's tape two or three.
#include "tg_device.cuh"
#include "tg_kernels.hpp"
#include "tg_surface.cuh"
#include "tg_tape.cuh"
#include "tg_parts.cuh"

namespace tg
{
	namespace
	{
		using namespace parts;
		constexpr int kCells = kBox - 1;
		constexpr int kEvalCtasPerSm = 8;

		// The export lattice in bricks of 7^3 cells: a brick's corner points, the last of an axis
		// shared with the next brick.
		struct MeshLattice
		{
			static constexpr int kStride = kCells;
			static constexpr int kBox = parts::kBox, kMost = 24;
			static constexpr bool kOutside = false, kBetween = true, kAbove = false;
			static constexpr int kShortest = 0;
			GridSpec Grid;
			__device__ __forceinline__ float Coord(int a, int i) const
			{
				return a == 0 ? LatticeCoord(Grid.X0, i, Grid.DX) : a == 1 ? LatticeCoord(Grid.Y0, i, Grid.DY) : LatticeCoord(Grid.Z0, i, Grid.DZ);
			}
			__host__ __device__ __forceinline__ int Points(int a) const { return a == 0 ? Grid.NX : a == 1 ? Grid.NY : Grid.NZ; }
			__host__ __device__ __forceinline__ int Bricks(int a) const { return (Points(a) - 1 + kCells - 1) / kCells; }
			__device__ __forceinline__ float Keep() const { return 0.0f; }
		};

		// The evaluation with the cell pass folded in: a warp draws a brick from a counter and
		// evaluates its points (BrickPoints), writing the lattice and the brick's 8^3 corner box
		// in shared memory; it then flags and lists the brick's active cells from the signs of that box:
		// eight corners of a row make a byte, four rows' bytes the seven cells between them.
		__global__ void __launch_bounds__(kThreads, kEvalCtasPerSm) EvalBrickTapesKernel(DeviceProgram prog, MeshLattice lat,
			const uint32_t* __restrict__ list, const uint32_t* __restrict__ count, BrickTapes tapes, float* __restrict__ lattice,
			uint32_t* __restrict__ words, uint32_t* __restrict__ cells, uint32_t* __restrict__ cell_count)
		{
			extern __shared__ __align__(16) float2 spill2[];
			__shared__ __align__(16) float boxes[kWarps][kBox * kBox * kBox];
			__shared__ float axes[kWarps][3][kBox];
			const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
			float* box = boxes[warp];
			float (*axis)[kBox] = axes[warp];
			const GridSpec& g = lat.Grid;
			const PairUnits units = LoadPairUnits();
			const uint32_t n = *count;
			const uint32_t plane = (uint32_t)g.NX * (uint32_t)g.NY;
			for (;;)
			{
				uint32_t item = 0;
				if (lane == 0) item = atomicAdd(tapes.Counters + 3, 1u);
				item = __shfl_sync(0xFFFFFFFFu, item, 0);
				if (item >= n) break;
				const uint32_t b = __ldg(list + item);
				const uint2 own = __ldg(tapes.Bricks + b);
				int first[3], extent[3];
				BrickSpan(lat, b, first, extent);
				const int i0 = first[0], j0 = first[1], k0 = first[2], ex = extent[0], ey = extent[1], ez = extent[2];
				// All parts of one sign: the brick has no active cell, and nobody reads its values.
				uint32_t sign = kBoxPositive | kBoxNegative;
				for (uint32_t p = 0; p < own.y; ++p) sign &= __ldg(&tapes.Parts[own.x + p].Box);
				if (own.y && sign) continue;
				float* corner = lattice + ((int64_t)k0 * g.NY + j0) * g.NX + i0;
				__syncwarp();       // the previous brick is done with the box and the axes
				if (lane < 24)
				{
					const int a = lane >> 3, q = lane & 7;
					axis[a][q] = lat.Coord(a, first[a] + q);
				}
				__syncwarp();
				BrickPoints<false>(prog, tapes, own, extent, axis, units, spill2 + threadIdx.x, [&](int at, float v, bool live)
				{
					if (!live) return;
					corner[(int64_t)(at >> 6) * plane + ((at >> 3) & 7) * g.NX + (at & 7)] = v;
					box[at] = v;
				});
				__syncwarp();
				// The cell pass.  Lane l has rows 2l and 2l + 1 of the box (row = z * 8 + y).
				uint32_t signs = 0;
#pragma unroll
				for (int q = 0; q < 4; ++q)
				{
					const float4 v = reinterpret_cast<const float4*>(box)[lane * 4 + q];
					// "Positive" is >= isovalue (0).
					signs |= ((v.x >= 0.0f ? 1u : 0u) | (v.y >= 0.0f ? 2u : 0u) | (v.z >= 0.0f ? 4u : 0u) | (v.w >= 0.0f ? 8u : 0u)) << (4 * q);
				}
				const uint32_t beside = __shfl_down_sync(0xFFFFFFFFu, signs, 1), above = __shfl_down_sync(0xFFFFFFFFu, signs, 4);
				const uint32_t both = __shfl_down_sync(0xFFFFFFFFu, signs, 5);
				const int z = lane >> 2, y = 2 * (lane & 3);
				const uint32_t wide = (1u << ex) - 1u;
				auto cellsOf = [&](uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) -> uint32_t
				{
					const uint32_t any = (r0 | r1 | r2 | r3) & 0xFFu, all = (r0 & r1 & r2 & r3) & 0xFFu;
					return (any | (any >> 1)) & ~(all & (all >> 1)) & wide;
				};
				uint32_t active[2];
				active[0] = z < ez && y < ey ? cellsOf(signs, signs >> 8, above, above >> 8) : 0u;
				active[1] = z < ez && y + 1 < ey ? cellsOf(signs >> 8, beside, above >> 8, both) : 0u;
				const int64_t sx = g.NX - 1, sy = g.NY - 1;
				const int64_t c0 = i0 + sx * ((j0 + y) + sy * (k0 + z));
#pragma unroll
				for (int q = 0; q < 2; ++q)
				{
					if (!active[q]) continue;
					const int64_t c = c0 + q * sx;
					const int shift = (int)(c & 31);
					atomicOr(words + (c >> 5), active[q] << shift);
					if (shift > 32 - kBox && (active[q] >> (32 - shift))) atomicOr(words + (c >> 5) + 1, active[q] >> (32 - shift));
				}
				const uint32_t total = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)(__popc(active[0]) + __popc(active[1])));
				uint32_t to = 0;
				if (lane == 0 && total) to = atomicAdd(cell_count, total);
				to = __shfl_sync(0xFFFFFFFFu, to, 0);
				// The cells by part (that of the cell's first corner), so that the vertices of a
				// part, which run one tape, follow each other.
				for (uint32_t p = 0; p < max(own.y, 1u) && total; ++p)
				{
					const uint32_t span = own.y ? __ldg(&tapes.Parts[own.x + p].Box) : PackBox(0, ex, 0, ey, 0, ez);
					const int x0 = (int)(span & 15u), x1 = (int)((span >> 4) & 15u);
					const uint32_t columns = (2u << x1) - (1u << x0);
					const bool inZ = z >= (int)((span >> 16) & 15u) && z <= (int)((span >> 20) & 15u);
					uint32_t bits[2];
#pragma unroll
					for (int q = 0; q < 2; ++q)
						bits[q] = inZ && y + q >= (int)((span >> 8) & 15u) && y + q <= (int)((span >> 12) & 15u) ? active[q] & columns : 0u;
					const uint32_t mine = (uint32_t)(__popc(bits[0]) + __popc(bits[1]));
					uint32_t upTo = mine;
#pragma unroll
					for (int o = 1; o < 32; o <<= 1)
					{
						const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, upTo, o);
						if (lane >= o) upTo += v;
					}
					uint32_t at = to + upTo - mine;
					to += __shfl_sync(0xFFFFFFFFu, upTo, 31);
#pragma unroll
					for (int q = 0; q < 2; ++q)
					{
						while (bits[q])
						{
							const int x = __ffs((int)bits[q]) - 1;
							bits[q] &= bits[q] - 1u;
							cells[at++] = (uint32_t)(c0 + q * sx + x);
						}
					}
				}
			}
		}

		// Normals and colours of the export's vertices, a thread per vertex in the active-cell
		// list's order (cells grouped by brick, so a warp's vertices mostly run one tape).
		__global__ void __launch_bounds__(kThreads, 8) BrickAttributesKernel(DeviceProgram prog, MeshLattice lat, BrickTapes tapes,
			const uint32_t* __restrict__ cells, const uint32_t* __restrict__ words, const uint32_t* __restrict__ word_base,
			const float* __restrict__ vertices, uint32_t n, float* __restrict__ normals, uint8_t* __restrict__ colors)
		{
			extern __shared__ __align__(16) float2 spill2[];
			const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
			if (t >= n) return;
			const uint32_t c = __ldg(cells + t);
			const uint32_t w = __ldg(words + (c >> 5)), before = __ldg(word_base + (c >> 5));
			const uint32_t sx = (uint32_t)(lat.Grid.NX - 1), sy = (uint32_t)(lat.Grid.NY - 1);
			const uint32_t row = c / sx, k = row / sy, i = c - row * sx, j = row - k * sy;
			const uint32_t b = i / kCells + (uint32_t)lat.Bricks(0) * (j / kCells + (uint32_t)lat.Bricks(1) * (k / kCells));
			const uint2 own = __ldg(tapes.Bricks + b);
			const uint32_t v = before + __popc(w & ((1u << (c & 31)) - 1u));
			const Vec3 p(__ldg(vertices + (int64_t)v * 3), __ldg(vertices + (int64_t)v * 3 + 1), __ldg(vertices + (int64_t)v * 3 + 2));
			float2* spill = spill2 + threadIdx.x;
			PointRun run;
			if (!FindPart(tapes, own, p, run)) RunWhole(prog, p, run);
			const PairUnits units = LoadPairUnits();
			float none;
			const Vec3 normal = RunGradient<false>(prog, tapes, run, p, units, spill, false, none);
			normals[(int64_t)v * 3 + 0] = normal.x;
			normals[(int64_t)v * 3 + 1] = normal.y;
			normals[(int64_t)v * 3 + 2] = normal.z;
			if (!colors) return;
			const uchar4 color = RunColor(prog, tapes, run, p, units, spill);
			colors[(int64_t)v * 3 + 0] = color.x;
			colors[(int64_t)v * 3 + 1] = color.y;
			colors[(int64_t)v * 3 + 2] = color.z;
		}
	}

	// Parts and events are bounded by the bricks of the grid: a fine export keeps one brick in
	// ten or twenty, with two or three parts each; a coarse one keeps more, with up to a dozen.
	// What does not fit is evaluated without (BrickPartsKernel, BuildPartTapesKernel).
	size_t BrickPartCapacity(int64_t bricks) { return (size_t)bricks / 2 + 65536; }
	size_t BrickEventCapacity(size_t parts) { return parts * 12; }

	cudaError_t LaunchBrickTapes(const DeviceProgram& prog, const GridSpec& g, int B, const uint32_t* list, const uint32_t* count,
		const uint32_t* tops, const BrickTapes& tapes, int sms, cudaStream_t stream)
	{
		if (B != kCells) return cudaErrorInvalidValue;
		return LaunchParts(prog, MeshLattice{ g }, list, count, tops, tapes, sms, stream);
	}

	cudaError_t LaunchEvalBrickTapes(const DeviceProgram& prog, const GridSpec& g, int B, const uint32_t* list, const uint32_t* count,
		const BrickTapes& tapes, float* lattice, uint32_t* words, uint32_t* cells, uint32_t* cell_count, int sms, cudaStream_t stream)
	{
		if (B != kCells) return cudaErrorInvalidValue;
		const int64_t total = (int64_t)(g.NX - 1) * (g.NY - 1) * (g.NZ - 1);
		cudaError_t e = cudaMemsetAsync(words, 0, (size_t)((total + 31) / 32) * 4, stream);
		if (e == cudaSuccess) e = cudaMemsetAsync(cell_count, 0, sizeof(uint32_t), stream);
		if (e != cudaSuccess) return e;
		const size_t smem = SpillPairs(prog, 1) * kThreads * sizeof(float2);
		if (smem > 39 * 1024)
		{
			e = cudaFuncSetAttribute(EvalBrickTapesKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		EvalBrickTapesKernel<<<sms * kEvalCtasPerSm, kThreads, smem, stream>>>(prog, MeshLattice{ g }, list, count, tapes, lattice, words, cells, cell_count);
		return cudaGetLastError();
	}

	cudaError_t LaunchBrickAttributes(const DeviceProgram& prog, const GridSpec& g, int B, const BrickTapes& tapes, const uint32_t* cells,
		const uint32_t* words, const uint32_t* word_base, const float* vertices, uint32_t vertex_count, float* normals, uint8_t* colors,
		cudaStream_t stream)
	{
		if (vertex_count == 0) return cudaSuccess;
		if (B != kCells) return cudaErrorInvalidValue;
		// The walk takes two words a level, the gradient one pair.
		const size_t smem = SpillPairs(prog, 2) * kThreads * sizeof(float2);
		if (smem > 48 * 1024)
		{
			const cudaError_t e = cudaFuncSetAttribute(BrickAttributesKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		BrickAttributesKernel<<<(vertex_count + kThreads - 1) / kThreads, kThreads, smem, stream>>>(prog, MeshLattice{ g }, tapes, cells, words, word_base, vertices, vertex_count, normals, colors);
		return cudaGetLastError();
	}
}
