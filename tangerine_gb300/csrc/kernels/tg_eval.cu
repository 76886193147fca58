// Distance evaluation over the export lattice.
//
// Small lattices run the cells' whole programs: one CTA covers an 8 x 16 patch of lattice
// columns and K consecutive z levels; every thread evaluates its K points with one pass over
// the record stream of the octree cell they fall in (the common case: K points, one cell).
// Records are read through the read-only cache with warp-uniform addresses, so each record
// quad is one broadcast load per warp.  Operands below the top of the postfix stack spill to
// shared memory in a thread-interleaved layout (no bank conflicts).  Large ones go by
// shortened programs, at the end of this file.
#include "tg_device.cuh"
#include "tg_kernels.hpp"
#include "tg_pair.cuh"
#include "tg_parts.cuh"

namespace tg
{
	namespace
	{
		constexpr int kTileX = 8;
		constexpr int kTileY = 16;
		constexpr int kThreads = kTileX * kTileY;

		template<int K>
		__global__ void __launch_bounds__(kThreads) EvalGridKernel(DeviceProgram prog, GridSpec g, float* __restrict__ out)
		{
			extern __shared__ float spill[];
			const int tx = threadIdx.x % kTileX;
			const int ty = threadIdx.x / kTileX;
			const int ix = blockIdx.x * kTileX + tx;
			const int iy = blockIdx.y * kTileY + ty;
			const int iz0 = blockIdx.z * K;
			const bool inPlane = ix < g.NX && iy < g.NY;
			const float x = LatticeCoord(g.X0, ix < g.NX ? ix : g.NX - 1, g.DX);
			const float y = LatticeCoord(g.Y0, iy < g.NY ? iy : g.NY - 1, g.DY);

			float px[K], py[K], pz[K], res[K];
			int cell[K];
			unsigned todo = 0;
#pragma unroll
			for (int k = 0; k < K; ++k)
			{
				const int iz = iz0 + k;
				px[k] = x;
				py[k] = y;
				pz[k] = LatticeCoord(g.Z0, iz < g.NZ ? iz : g.NZ - 1, g.DZ);
				cell[k] = DescendOctree(prog.Nodes, px[k], py[k], pz[k]);
				res[k] = 0.0f;
				if (inPlane && iz < g.NZ) todo |= 1u << k;
			}

			// Evaluate once per distinct octree cell among this thread's points.
			while (todo)
			{
				int c = -1;
#pragma unroll
				for (int k = 0; k < K; ++k)
					if (c < 0 && ((todo >> k) & 1u)) c = cell[k];
				float r[K];
				if constexpr (K % 2 == 0)
				{
					// Points in pairs through the paired FP32 instructions (tg_pair.cuh).
					const float4* code = prog.Code;
					RunDistancePaired<K>([&](int q) { return __ldg(code + q); }, __ldg(&prog.Nodes[c].DistanceCode), px, py, pz, r,
						spill + 2 * threadIdx.x, kThreads);
				}
				else
				{
					RunDistance<K>(prog.Code, __ldg(&prog.Nodes[c].DistanceCode), px, py, pz, r, spill + threadIdx.x, kThreads);
				}
#pragma unroll
				for (int k = 0; k < K; ++k)
				{
					if (((todo >> k) & 1u) && cell[k] == c)
					{
						res[k] = r[k];
						todo &= ~(1u << k);
					}
				}
			}

			if (inPlane)
			{
#pragma unroll
				for (int k = 0; k < K; ++k)
				{
					const int iz = iz0 + k;
					if (iz < g.NZ) out[((int64_t)iz * g.NY + iy) * g.NX + ix] = res[k];
				}
			}
		}
	}

	namespace
	{
		template<int K>
		cudaError_t LaunchEvalGridK(const DeviceProgram& prog, const GridSpec& grid, float* out, cudaStream_t stream)
		{
			const int depth = prog.MaxStack > 1 ? prog.MaxStack - 1 : 1;
			const size_t smem = (size_t)depth * K * kThreads * sizeof(float);
			if (smem > 48 * 1024)
			{
				cudaError_t e = cudaFuncSetAttribute(EvalGridKernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
				if (e != cudaSuccess) return e;
			}
			const dim3 blocks((grid.NX + kTileX - 1) / kTileX, (grid.NY + kTileY - 1) / kTileY, (grid.NZ + K - 1) / K);
			EvalGridKernel<K><<<blocks, kThreads, smem, stream>>>(prog, grid, out);
			return cudaGetLastError();
		}
	}

	cudaError_t LaunchEvalGrid(const DeviceProgram& prog, const GridSpec& grid, float* out, cudaStream_t stream, int lanes)
	{
		switch (lanes)
		{
		case 1: return LaunchEvalGridK<1>(prog, grid, out, stream);
		case 2: return LaunchEvalGridK<2>(prog, grid, out, stream);
		default: return LaunchEvalGridK<4>(prog, grid, out, stream);
		}
	}

	namespace
	{
		// Levels of a brick that a warp takes at a time: two, one where there are few bricks.  At four
		// a warp whose part has no tape (a long program, a coarse lattice) ran the whole program 16
		// times over, longer than all others took together: 512 primitives at 110^3 2764 us by whole
		// programs, 5310 at four levels, 3077 at two, 2175 at one; 32 primitives at 190^3 710, 201, 173,
		// 162, at 300^3 2639, 334, 321, 332.
		constexpr int64_t kFewBricks = 2000;
		constexpr int64_t kSlabBricks = 16384;
		constexpr int kDenseCtasPerSm = 8;

		// The lattice by shortened programs: a brick's parts each get a tape (tg_parts.cuh), and
		// almost all of a part's up to 4096 points' passes over its cell's program become passes
		// over the two or three operands that matter there.  Bricks of 16^3: at 8^3 the building
		// (a pass of the whole program per part) took 375 of 500 us for 301 x 257 x 193 points of
		// 64 primitives, at 16^3 93 of 225, and the evaluation 108 for 98.  That lattice: 1401 ->
		// 243 us (another tree: 463 -> 220); 320^3 of 256 primitives 5500 -> 608.
		// Bound by the interpreter's issue; the writes take 9 us of the 108.

		// A slab of the lattice, Levels levels from level K0 on, in bricks of 16^3 points.
		struct DenseLattice
		{
			static constexpr int kBox = 16, kStride = 16, kMost = 96;
			static constexpr bool kOutside = false, kBetween = false, kAbove = false;
			static constexpr int kShortest = 0;
			GridSpec Grid;
			int K0, Levels;
			__device__ __forceinline__ float Coord(int a, int i) const
			{
				return a == 0 ? LatticeCoord(Grid.X0, i, Grid.DX) : a == 1 ? LatticeCoord(Grid.Y0, i, Grid.DY) : LatticeCoord(Grid.Z0, K0 + i, Grid.DZ);
			}
			__host__ __device__ __forceinline__ int Points(int a) const { return a == 0 ? Grid.NX : a == 1 ? Grid.NY : Levels; }
			__host__ __device__ __forceinline__ int Bricks(int a) const { return (Points(a) + kStride - 1) / kStride; }
			__device__ __forceinline__ float Keep() const { return INFINITY; }
		};

		// A warp per slice of a brick, drawn from a counter.
		template<int Slice>
		__global__ void __launch_bounds__(parts::kThreads, kDenseCtasPerSm) EvalGridTapesKernel(DeviceProgram prog, DenseLattice lat, BrickTapes tapes,
			float* __restrict__ out)
		{
			extern __shared__ __align__(16) float2 spill2[];
			__shared__ float axes[parts::kWarps][3][DenseLattice::kBox];
			constexpr int kSlices = DenseLattice::kBox / Slice;
			const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
			float (*axis)[DenseLattice::kBox] = axes[warp];
			const PairUnits units = LoadPairUnits();
			const uint32_t n = (uint32_t)lat.Bricks(0) * (uint32_t)lat.Bricks(1) * (uint32_t)lat.Bricks(2);
			const int64_t plane = (int64_t)lat.Grid.NX * lat.Grid.NY;
			for (;;)
			{
				uint32_t item = 0;
				if (lane == 0) item = atomicAdd(tapes.Counters + 3, 1u);
				item = __shfl_sync(0xFFFFFFFFu, item, 0);
				if (item >= n * kSlices) break;
				const uint32_t b = item / kSlices;
				const int lowest = (int)(item % kSlices) * Slice;
				int first[3], extent[3];
				parts::BrickSpan(lat, b, first, extent);
				if (lowest > extent[2]) continue;
				__syncwarp();       // the previous slice is done with the axes
				for (int q = lane; q < 48; q += 32) axis[q >> 4][q & 15] = lat.Coord(q >> 4, first[q >> 4] + (q & 15));
				__syncwarp();
				float* corner = out + (lat.K0 + first[2]) * plane + (int64_t)first[1] * lat.Grid.NX + first[0];
				parts::BrickPoints<false, DenseLattice::kBox>(prog, tapes, __ldg(tapes.Bricks + b), extent, axis, units, spill2 + threadIdx.x,
					[&](int at, float v, bool live)
					{
						if (live) corner[(at >> 8) * plane + ((at >> 4) & 15) * lat.Grid.NX + (at & 15)] = v;
					}, lowest, lowest + Slice - 1);
			}
		}

		int64_t DensePlane(const GridSpec& g)
		{
			constexpr int B = DenseLattice::kBox;
			return (int64_t)((g.NX + B - 1) / B) * ((g.NY + B - 1) / B);
		}
	}

	// Slabs bound the tapes' memory: kSlabBricks bricks, or one layer of them where that is more.
	int64_t DenseSlabBricks(const GridSpec& g)
	{
		const int64_t plane = DensePlane(g), layers = (g.NZ + DenseLattice::kBox - 1) / DenseLattice::kBox;
		const int64_t most = plane >= kSlabBricks ? 1 : kSlabBricks / plane;
		return plane * (layers < most ? layers : most);
	}

	cudaError_t LaunchEvalGridTapes(const DeviceProgram& prog, const GridSpec& g, const BrickTapes& tapes, float* out, int sms, cudaStream_t stream)
	{
		const size_t smem = parts::SpillPairs(prog, 1) * parts::kThreads * sizeof(float2);
		const int64_t bricks = DensePlane(g) * ((g.NZ + DenseLattice::kBox - 1) / DenseLattice::kBox);
		auto* kernel = bricks <= kFewBricks ? EvalGridTapesKernel<1> : EvalGridTapesKernel<2>;
		if (smem > 46 * 1024)
		{
			const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		const int levels = (int)(DenseSlabBricks(g) / DensePlane(g)) * DenseLattice::kBox;
		for (int k0 = 0; k0 < g.NZ; k0 += levels)
		{
			const DenseLattice lat{ g, k0, g.NZ - k0 < levels ? g.NZ - k0 : levels };
			cudaError_t e = parts::LaunchParts(prog, lat, nullptr, nullptr, nullptr, tapes, sms, stream);
			if (e != cudaSuccess) return e;
			kernel<<<sms * kDenseCtasPerSm, parts::kThreads, smem, stream>>>(prog, lat, tapes, out);
			e = cudaGetLastError();
			if (e != cudaSuccess) return e;
		}
		return cudaSuccess;
	}
}
