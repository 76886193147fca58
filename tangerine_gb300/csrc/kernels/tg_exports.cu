// The reference's other two lattice exports on the GPU:
//  * PointCloudExportThread (tangerine/export.cpp:384-480): voxel centres whose octree
//    distance is within the half-voxel diagonal, then gradient steps toward the surface
//    kept inside the voxel;
//  * VoxExport (tangerine/magica.cpp:27-72): voxels whose centre's full-tree distance is
//    within the half-voxel radius.
// Both keep the reference's float operation order, so the kept cells and refined points are
// the reference's bit for bit; the kept cells become an index-ordered list through the
// bitmask + scan of the brick lists.
#include "tg_device.cuh"
#include "tg_kernels.hpp"
#include "tg_surface.cuh"
#include "tg_tape.cuh"
#include "tg_parts.cuh"

namespace tg
{
	namespace
	{
		inline unsigned Blocks(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

		// Cell i's centre: float(i / slice) * step.z + start.z (and so on), then + half.
		__device__ __forceinline__ Vec3 CloudCentre(const CloudSpec& s, int i)
		{
			const int slice = s.IX * s.IY;
			const float Z = (float)(i / slice) * s.Step[2] + s.Start[2];
			const float Y = (float)((i % slice) / s.IX) * s.Step[1] + s.Start[1];
			const float X = (float)(i % s.IX) * s.Step[0] + s.Start[0];
			return Vec3(X, Y, Z) + Vec3(s.Half[0], s.Half[1], s.Half[2]);
		}

		// `spill`: this thread's column of the operand stack in shared memory (stride
		// `stride`), as the interpreters lay it out.
		__device__ __forceinline__ float OctreeDistance(const DeviceProgram& prog, Vec3 p, float* spill, int stride)
		{
			const float px[1] = { p.x }, py[1] = { p.y }, pz[1] = { p.z };
			float r[1];
			const int cell = DescendOctree(prog.Nodes, p.x, p.y, p.z);
			RunDistance<1>(prog.Code, __ldg(&prog.Nodes[cell].DistanceCode), px, py, pz, r, spill, stride);
			return r[0];
		}

		// Voxel bricks: 8^3 voxels whose tests are decided together when a bound proves that
		// none of them can pass.  The distance functions are 1-Lipschitz (or the test is not
		// made), so |f(c)| > r + threshold + margin at the centre c of the ball (radius r)
		// through the brick's voxel centres means |f| > threshold at every one of them; the
		// margin covers the rounding of f at c and at the voxel (as in the export's bricks).
		constexpr int kVoxelBrick = 8;

		struct VoxelBricks
		{
			int NX, NY, NZ;     // bricks per axis
		};

		__device__ __forceinline__ void BrickRange(int b, const VoxelBricks& vb, int sx, int sy, int sz, int (&lo)[3], int (&hi)[3])
		{
			const int bx = b % vb.NX, by = (b / vb.NX) % vb.NY, bz = b / (vb.NX * vb.NY);
			lo[0] = bx * kVoxelBrick; hi[0] = min(lo[0] + kVoxelBrick - 1, sx - 1);
			lo[1] = by * kVoxelBrick; hi[1] = min(lo[1] + kVoxelBrick - 1, sy - 1);
			lo[2] = bz * kVoxelBrick; hi[2] = min(lo[2] + kVoxelBrick - 1, sz - 1);
		}

		__device__ __forceinline__ int BrickOfVoxel(int x, int y, int z, const VoxelBricks& vb)
		{
			return x / kVoxelBrick + vb.NX * (y / kVoxelBrick + vb.NY * (z / kVoxelBrick));
		}

		// The ball through the box [lo, hi] of voxel centres, and the margin for rounding.
		__device__ __forceinline__ void BallOf(const float (&lo)[3], const float (&hi)[3], float (&c)[3], float& r, float& margin,
			float scale)
		{
			float e2 = 0.0f;
#pragma unroll
			for (int a = 0; a < 3; ++a)
			{
				c[a] = 0.5f * (lo[a] + hi[a]);
				const float e = 0.5f * (hi[a] - lo[a]);
				e2 += e * e;
			}
			r = sqrtf(e2) * 1.0001f + 1e-6f;
			margin = 1e-4f * (1.0f + fabsf(c[0]) + fabsf(c[1]) + fabsf(c[2]) + scale);
		}

		// One thread per brick of the point cloud's voxels: when the bricks' voxel centres
		// all descend to one octree cell, that cell's program at the ball's centre decides.
		__global__ void __launch_bounds__(128) CloudBricksKernel(DeviceProgram prog, CloudSpec s, VoxelBricks vb,
			uint32_t* __restrict__ brick_bits)
		{
			extern __shared__ float spill[];
			const int b = (int)(blockIdx.x * blockDim.x + threadIdx.x);
			if (b >= vb.NX * vb.NY * vb.NZ) return;
			int lo[3], hi[3];
			BrickRange(b, vb, s.IX, s.IY, s.IZ, lo, hi);
			// Voxel centres float(i) * step + start + half: monotone in i.
			float clo[3], chi[3];
#pragma unroll
			for (int a = 0; a < 3; ++a)
			{
				clo[a] = ((float)lo[a] * s.Step[a] + s.Start[a]) + s.Half[a];
				chi[a] = ((float)hi[a] * s.Step[a] + s.Start[a]) + s.Half[a];
			}
			bool keep = true;
			bool shared;
			const int cell = DescendBox(prog.Nodes, clo[0], chi[0], clo[1], chi[1], clo[2], chi[2], shared);
			const float clip = __ldg(&prog.Nodes[cell].ClipRadius);
			if (shared && clip >= 0.0f && !(__ldg(&prog.Nodes[cell].Flags) & kNodeNoEvaluator))
			{
				float c[3], r, margin;
				BallOf(clo, chi, c, r, margin, fabsf(__ldg(&prog.Nodes[0].ClipRadius)));
				const float px[1] = { c[0] }, py[1] = { c[1] }, pz[1] = { c[2] };
				float f[1];
				RunDistance<1>(prog.Code, __ldg(&prog.Nodes[cell].DistanceCode), px, py, pz, f, spill + threadIdx.x, 128);
				keep = !(fabsf(f[0]) > r + s.Diagonal + margin);
			}
			if (keep) atomicOr(brick_bits + (b >> 5), 1u << (b & 31));
		}

		// abs(Octree->Eval(Cursor)) < Diagonal per voxel centre (export.cpp:404-423).
		__global__ void __launch_bounds__(128) CloudFlagsKernel(DeviceProgram prog, CloudSpec s, VoxelBricks vb,
			const uint32_t* __restrict__ brick_bits, uint32_t* __restrict__ words)
		{
			extern __shared__ float spill[];
			const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
			bool keep = false;
			bool live = false;
			if (t < s.Total)
			{
				const int i = (int)t;
				const int slice = s.IX * s.IY;
				const int b = BrickOfVoxel(i % s.IX, (i % slice) / s.IX, i / slice, vb);
				live = (__ldg(brick_bits + (b >> 5)) >> (b & 31)) & 1u;
			}
			if (live)
			{
				const float d = OctreeDistance(prog, CloudCentre(s, (int)t), spill + threadIdx.x, 128);
				keep = fabsf(d) < s.Diagonal;
			}
			const unsigned ballot = __ballot_sync(0xFFFFFFFFu, keep);
			if ((threadIdx.x & 31) == 0 && t < s.Total) words[t >> 5] = ballot;
		}

		// SDFOctree::Gradient (the selected cell's SDFNode::Gradient, sdf_evaluator.cpp:298-333)
		// at p: the four tetrahedral evaluations share one pass over the cell's surface
		// program; the evaluation at p itself is needed only when they cancel.
		__device__ __forceinline__ Vec3 OctreeGradient(const DeviceProgram& prog, Vec3 p, float* spill, int stride)
		{
			const int cell = DescendOctree(prog.Nodes, p.x, p.y, p.z);
			const int pc = __ldg(&prog.Nodes[cell].SurfaceCode);
			float px[4], py[4], pz[4];
#pragma unroll
			for (int k = 0; k < 4; ++k)
			{
				const Vec3 q = TetraPoint(p, k);
				px[k] = q.x; py[k] = q.y; pz[k] = q.z;
			}
			float e[5];
			float r4[4];
			RunSurfaceBatch<4>(prog.Code, pc, px, py, pz, r4, -1, nullptr, spill, stride);
#pragma unroll
			for (int k = 0; k < 4; ++k) e[k] = r4[k];
			e[4] = 0.0f;
			const float h = 0.0001f;
			const Vec3 xyy(h, -h, -h), yyx(-h, -h, h), yxy(-h, h, -h), xxx(h, h, h);
			Vec3 g = xyy * e[0];
			g = g + yyx * e[1];
			g = g + yxy * e[2];
			g = g + xxx * e[3];
			if ((g.x * g.x + g.y * g.y) + g.z * g.z == 0.0f)
			{
				const float qx[1] = { p.x }, qy[1] = { p.y }, qz[1] = { p.z };
				float r1[1];
				RunSurfaceBatch<1>(prog.Code, pc, qx, qy, qz, r1, -1, nullptr, spill, stride);
				e[4] = r1[0];
			}
			return GradientOf(e);
		}

		// The refinement (export.cpp:434-465): `iterations` steps of Cursor += Gradient *
		// -Eval, clamped to the voxel; the point moves only if it stays within the diagonal.
		// Compiled for 12 resident CTAs per SM (the default took 80 registers, 6 CTAs): the
		// refinement of the 0.01-voxel cloud measured 4.17 ms at 6, 3.85 at 8, 3.58 at 10,
		// 3.47 at 12 and 4.13 at 16.
		__global__ void __launch_bounds__(128, 12) CloudRefineKernel(DeviceProgram prog, CloudSpec s, const uint32_t* __restrict__ cells,
			const uint32_t* __restrict__ count, int iterations, float* __restrict__ points)
		{
			extern __shared__ float spill[];
			const uint32_t n = __ldg(count);
			const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
			if (v >= n) return;
			const Vec3 vertex = CloudCentre(s, (int)__ldg(cells + v));
			const Vec3 half(s.Half[0], s.Half[1], s.Half[2]);
			Vec3 cursor = vertex;
			if (iterations > 0)
			{
				const Vec3 low = vertex - half, high = vertex + half;
				for (int r = 0; r < iterations; ++r)
				{
					const Vec3 dir = OctreeGradient(prog, cursor, spill + threadIdx.x, 128);
					// Octree->Eval(Cursor) * -1.0 rounds back to float exactly: a negation.
					const float dist = -OctreeDistance(prog, cursor, spill + threadIdx.x, 128);
					cursor = cursor + dir * dist;
				}
				cursor = TernaryMin(TernaryMax(cursor, low), high);
				const Vec3 d = vertex - cursor;
				if (!(sqrtf(Dot(d, d)) <= s.Diagonal)) cursor = vertex;
			}
			points[(int64_t)v * 3 + 0] = cursor.x;
			points[(int64_t)v * 3 + 1] = cursor.y;
			points[(int64_t)v * 3 + 2] = cursor.z;
		}

		// The point cloud by shortened programs (tg_parts.cuh): bricks of 8^3 voxel centres.  A
		// voxel's refined point may leave its brick by half a voxel.
		struct CloudLattice
		{
			static constexpr int kStride = parts::kBox;
			static constexpr int kBox = parts::kBox, kMost = 24;
			static constexpr bool kOutside = true, kBetween = true, kAbove = false;
			static constexpr int kShortest = 0;
			CloudSpec Spec;
			__device__ __forceinline__ float Coord(int a, int i) const { return ((float)i * Spec.Step[a] + Spec.Start[a]) + Spec.Half[a]; }
			__host__ __device__ __forceinline__ int Points(int a) const { return a == 0 ? Spec.IX : a == 1 ? Spec.IY : Spec.IZ; }
			__host__ __device__ __forceinline__ int Bricks(int a) const { return (Points(a) + parts::kBox - 1) / parts::kBox; }
			__device__ __forceinline__ float Keep() const { return Spec.Diagonal; }
			__device__ __forceinline__ int IndexAt(int a, float p) const
			{
				// In float until clamped: a wandering point may be far away, or not a number.
				return (int)fminf(fmaxf((p - Coord(a, 0)) / Spec.Step[a], 0.0f), (float)(Points(a) - 1)) / parts::kBox;
			}
			__device__ __forceinline__ uint32_t BrickAt(Vec3 p) const
			{
				return (uint32_t)min(IndexAt(0, p.x), Bricks(0) - 1) + (uint32_t)Bricks(0) * ((uint32_t)min(IndexAt(1, p.y), Bricks(1) - 1) +
					(uint32_t)Bricks(1) * (uint32_t)min(IndexAt(2, p.z), Bricks(2) - 1));
			}
		};

		// CloudBricksKernel's test, with the kept bricks listed and their descents stored.
		__global__ void __launch_bounds__(128) CloudListKernel(DeviceProgram prog, CloudLattice lat, uint32_t* __restrict__ list,
			uint32_t* __restrict__ count, uint32_t* __restrict__ tops)
		{
			extern __shared__ float spill[];
			const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
			const int lane = (int)(threadIdx.x & 31);
			bool keep = false;
			if (b < (int64_t)lat.Bricks(0) * lat.Bricks(1) * lat.Bricks(2))
			{
				int first[3], extent[3];
				parts::BrickSpan(lat, (uint32_t)b, first, extent);
				const uint32_t packed = parts::DescendBrick(prog, lat, first, extent);
				const int cell = (int)(packed & 0x7FFFFFFFu);
				keep = true;
				if ((packed >> 31) && __ldg(&prog.Nodes[cell].ClipRadius) >= 0.0f)
				{
					float lo[3], hi[3], c[3], r, margin;
#pragma unroll
					for (int a = 0; a < 3; ++a) { lo[a] = lat.Coord(a, first[a]); hi[a] = lat.Coord(a, first[a] + extent[a]); }
					BallOf(lo, hi, c, r, margin, fabsf(__ldg(&prog.Nodes[0].ClipRadius)));
					const float px[1] = { c[0] }, py[1] = { c[1] }, pz[1] = { c[2] };
					float f[1];
					RunDistance<1>(prog.Code, __ldg(&prog.Nodes[cell].DistanceCode), px, py, pz, f, spill + threadIdx.x, 128);
					keep = !(fabsf(f[0]) > r + lat.Spec.Diagonal + margin);
				}
				if (keep) tops[b] = packed;
			}
			const unsigned kept = __ballot_sync(0xFFFFFFFFu, keep);
			uint32_t at = 0;
			if (lane == 0 && kept) at = atomicAdd(count, (uint32_t)__popc(kept));
			at = __shfl_sync(0xFFFFFFFFu, at, 0);
			if (keep) list[at + (uint32_t)__popc(kept & ((1u << lane) - 1u))] = (uint32_t)b;
		}

		// abs(Octree->Eval(Cursor)) < Diagonal for the voxels of the listed bricks, a warp per
		// brick; the kept ones set their bits and are listed by brick and part, so that points
		// running one tape follow each other.
		__global__ void __launch_bounds__(parts::kThreads, 8) CloudVoxelsKernel(DeviceProgram prog, CloudLattice lat, const uint32_t* __restrict__ list,
			const uint32_t* __restrict__ count, BrickTapes tapes, uint32_t* __restrict__ words, uint32_t* __restrict__ voxels,
			uint32_t* __restrict__ voxel_count)
		{
			using namespace parts;
			extern __shared__ __align__(16) float2 spill2[];
			__shared__ uint16_t found[kWarps][kBox * kBox * kBox];
			__shared__ float axes[kWarps][3][kBox];
			const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
			float (*axis)[kBox] = axes[warp];
			uint16_t* kept = found[warp];
			const PairUnits units = LoadPairUnits();
			const uint32_t n = *count;
			for (;;)
			{
				uint32_t item = 0;
				if (lane == 0) item = atomicAdd(tapes.Counters + 3, 1u);
				item = __shfl_sync(0xFFFFFFFFu, item, 0);
				if (item >= n) break;
				const uint32_t b = __ldg(list + item);
				const uint2 own = __ldg(tapes.Bricks + b);
				bool far = own.y != 0;
				for (uint32_t p = 0; p < own.y; ++p) far = far && (__ldg(&tapes.Parts[own.x + p].Box) & (kBoxPositive | kBoxNegative));
				if (far) continue;
				int first[3], extent[3];
				BrickSpan(lat, b, first, extent);
				__syncwarp();       // the previous brick is done with the axes and the list
				if (lane < 24) axis[lane >> 3][lane & 7] = lat.Coord(lane >> 3, first[lane >> 3] + (lane & 7));
				__syncwarp();
				uint32_t total = 0;
				BrickPoints<true>(prog, tapes, own, extent, axis, units, spill2 + threadIdx.x, [&](int at, float v, bool live)
				{
					const unsigned keep = __ballot_sync(0xFFFFFFFFu, live && fabsf(v) < lat.Spec.Diagonal);
					if ((keep >> lane) & 1u) kept[total + (uint32_t)__popc(keep & ((1u << lane) - 1u))] = (uint16_t)at;
					total += (uint32_t)__popc(keep);
				});
				uint32_t to = 0;
				if (lane == 0 && total) to = atomicAdd(voxel_count, total);
				to = __shfl_sync(0xFFFFFFFFu, to, 0);
				__syncwarp();
				for (uint32_t i = (uint32_t)lane; i < total; i += 32)
				{
					const int at = kept[i];
					const int64_t t = first[0] + (at & 7) + (int64_t)lat.Spec.IX * ((first[1] + ((at >> 3) & 7)) + (int64_t)lat.Spec.IY * (first[2] + (at >> 6)));
					atomicOr(words + (t >> 5), 1u << (t & 31));
					voxels[to + i] = (uint32_t)t;
				}
			}
		}

		// The refinement (export.cpp:434-465): `iterations` steps of Cursor += Gradient * -Eval,
		// clamped to the voxel (the point moves only if it stays within the diagonal), then the
		// point's normal and colour; a thread per voxel in the bricks' order, each point by its
		// part's tape while it is in the part's box.
		__global__ void __launch_bounds__(parts::kThreads, 6) CloudPointsKernel(DeviceProgram prog, CloudLattice lat, BrickTapes tapes,
			const uint32_t* __restrict__ voxels, uint32_t n, const uint32_t* __restrict__ words, const uint32_t* __restrict__ word_base, int iterations,
			uint32_t* __restrict__ cubes, float* __restrict__ points, float* __restrict__ normals, uint8_t* __restrict__ colors)
		{
			using namespace parts;
			extern __shared__ __align__(16) float2 spill2[];
			const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
			if (t >= n) return;
			const CloudSpec& s = lat.Spec;
			const uint32_t c = __ldg(voxels + t);
			const uint32_t w = __ldg(words + (c >> 5));
			const uint32_t v = __ldg(word_base + (c >> 5)) + __popc(w & ((1u << (c & 31)) - 1u));
			const uint32_t row = c / (uint32_t)s.IX, k = row / (uint32_t)s.IY, i = c - row * (uint32_t)s.IX, j = row - k * (uint32_t)s.IY;
			const uint2 own = __ldg(tapes.Bricks + i / kBox + (uint32_t)lat.Bricks(0) * (j / kBox + (uint32_t)lat.Bricks(1) * (k / kBox)));
			const Vec3 vertex = CloudCentre(s, (int)c);
			const PairUnits units = LoadPairUnits();
			float2* spill = spill2 + threadIdx.x;
			Vec3 cursor = vertex;
			PointRun run;
			run.Lo[0] = 1.0f; run.Hi[0] = 0.0f;
			Vec3 normal(0.0f, 0.0f, 0.0f);
			for (int r = 0; r <= iterations; ++r)
			{
				if (r == iterations)
				{
					if (iterations > 0)
					{
						const Vec3 half(s.Half[0], s.Half[1], s.Half[2]);
						const Vec3 low = vertex - half, high = vertex + half;
						cursor = TernaryMin(TernaryMax(cursor, low), high);
						const Vec3 d = vertex - cursor;
						if (!(sqrtf(Dot(d, d)) <= s.Diagonal)) cursor = vertex;
					}
					if (!normals) break;
				}
				if (!InRun(run, cursor))
				{
					// The voxel's own brick, then the one the point is in now (one that was not kept
					// has no parts).  A point that runs whole programs holds up its warp: looked for in
					// its own brick alone, a few in a hundred did, and two warps in three.
					bool found = FindPart(tapes, own, cursor, run);
					if (!found)
					{
						const uint32_t b = lat.BrickAt(cursor);
						found = FindPart(tapes, __ldg(tapes.Bricks + b), cursor, run);
					}
					if (!found) RunWhole(prog, cursor, run);
				}
				float d = 0.0f;
				normal = RunGradient<true>(prog, tapes, run, cursor, units, spill, r < iterations, d);
				if (r == iterations) break;
				// Octree->Eval(Cursor) * -1.0 rounds back to float exactly: a negation.
				cursor = cursor + normal * -d;
			}
			cubes[v] = c;
			points[(int64_t)v * 3 + 0] = cursor.x;
			points[(int64_t)v * 3 + 1] = cursor.y;
			points[(int64_t)v * 3 + 2] = cursor.z;
			if (!normals) return;
			normals[(int64_t)v * 3 + 0] = normal.x;
			normals[(int64_t)v * 3 + 1] = normal.y;
			normals[(int64_t)v * 3 + 2] = normal.z;
			if (!colors) return;
			const uchar4 color = RunColor(prog, tapes, run, cursor, units, spill);
			colors[(int64_t)v * 3 + 0] = color.x;
			colors[(int64_t)v * 3 + 1] = color.y;
			colors[(int64_t)v * 3 + 2] = color.z;
		}

		// glm::mix(x, y, a) = x * (1 - a) + y * a, per component.
		__device__ __forceinline__ float Mix(float x, float y, float a)
		{
			return x * (1.0f - a) + y * a;
		}

		// VoxExport's voxel centre on one axis: mix(Min, Max, (x + .5) / Size), where
		// vec3(x + .5, ...) converts the double sums to float.
		__device__ __forceinline__ float VoxCentre(float lo, float hi, int x, int size)
		{
			return Mix(lo, hi, (float)((double)x + 0.5) / (float)size);
		}

		// The ball through the voxel centres [lo, hi], and the margin for rounding.  mix()
		// rounds each centre separately, so the box is widened by a relative 1e-6 of its
		// coordinates.
		__device__ __forceinline__ void VoxBall(const VoxSpec& s, const int (&lo)[3], const int (&hi)[3], float scale, float (&c)[3], float& r,
			float& margin)
		{
			const int size[3] = { s.SX, s.SY, s.SZ };
			float clo[3], chi[3];
#pragma unroll
			for (int a = 0; a < 3; ++a)
			{
				const float u = VoxCentre(s.Min[a], s.Max[a], lo[a], size[a]);
				const float v = VoxCentre(s.Min[a], s.Max[a], hi[a], size[a]);
				const float slack = 1e-6f * (fabsf(u) + fabsf(v) + fabsf(s.Min[a]) + fabsf(s.Max[a]));
				clo[a] = fminf(u, v) - slack;
				chi[a] = fmaxf(u, v) + slack;
			}
			BallOf(clo, chi, c, r, margin, scale);
		}

		// VoxExport's test (magica.cpp:52-64) is on the whole tree (SDFNode::Eval), some
		// hundreds of records.  Blocks of 64^3 voxels, then the 16^3 blocks in them that may
		// hold a kept voxel, then the 4^3 boxes in those, are decided by a ball each, and every
		// level shortens the tree's surface program for the next (tg_tape.cuh): a warp per
		// block runs the program it was given at its 64 parts' centres.
		constexpr int kVoxCoarse = 64, kVoxBlock = 16, kVoxFine = 4;
		constexpr int kVoxCoarseCap = 2048, kVoxBlockCap = 192;
		constexpr int kVoxWarps = 4, kVoxCtasPerSm = 6, kVoxEvalCtasPerSm = 8;
		constexpr int kVoxDirectBlocks = 1000;
		constexpr int kVoxWholeBoxes = 4096;

		// A warp's scratch while it builds a 16^3 block's tape.
		struct VoxScratch
		{
			float4 Window[64];
			uint2 Heads[16], Value[kVoxBlockCap], Start[kMaxStack + 2];
		};

		struct VoxGrid
		{
			int NX, NY, NZ;         // 64^3 blocks per axis
		};

		struct VoxState
		{
			uint2* Events;          // kVoxCoarseCap per 64^3 block: its tape; then the 16^3 blocks' tapes
			uint32_t* Counts;       // per 64^3 block: its tape's length (kNoTape: none)
			uint32_t* List;         // 16^3 blocks to look at: 64^3 block * 64 + part
			uint2* Tapes;           // per listed 16^3 block: first event and length of the tape it goes by
			uint32_t* Boxes;        // 4^3 boxes to test: listed block * 64 + part
			uint32_t* Counters;     // blocks listed, blocks taken, events of the 16^3 blocks, boxes listed, boxes taken
			uint32_t EventBase, EventCap;   // where the 16^3 blocks' events begin, and how many fit
		};
		constexpr int kVoxCounters = 5;

		// The first voxel of a listed 16^3 block.
		__device__ __forceinline__ void VoxBlockStart(const VoxGrid& vg, uint32_t entry, int (&from)[3])
		{
			const int b = (int)(entry >> 6), part = (int)(entry & 63u);
			from[0] = (b % vg.NX) * kVoxCoarse + (part & 3) * kVoxBlock;
			from[1] = ((b / vg.NX) % vg.NY) * kVoxCoarse + ((part >> 2) & 3) * kVoxBlock;
			from[2] = (b / (vg.NX * vg.NY)) * kVoxCoarse + (part >> 4) * kVoxBlock;
		}

		// Part `part` (0..63, x fastest) of a block that starts at voxel `from` and has 4 x 4 x 4
		// parts of `edge` voxels an axis; false when it lies outside the lattice (the box is then
		// the nearest voxel).
		__device__ __forceinline__ bool VoxPart(const VoxSpec& s, const int (&from)[3], int part, int edge, int (&lo)[3], int (&hi)[3])
		{
			const int size[3] = { s.SX, s.SY, s.SZ };
			const int at[3] = { part & 3, (part >> 2) & 3, part >> 4 };
			bool in = true;
#pragma unroll
			for (int a = 0; a < 3; ++a)
			{
				lo[a] = from[a] + at[a] * edge;
				in = in && lo[a] < size[a];
				lo[a] = min(lo[a], size[a] - 1);
				hi[a] = min(lo[a] + edge - 1, size[a] - 1);
			}
			return in;
		}

		// The two balls of this lane in a block: parts lane and lane + 32.
		struct VoxLane
		{
			float2 X, Y, Z, R, Margin;
			bool In[2];
		};

		__device__ __forceinline__ VoxLane VoxLaneOf(const VoxSpec& s, const int (&from)[3], int edge, float scale)
		{
			VoxLane l;
			float c[2][3], r[2], m[2];
#pragma unroll
			for (int j = 0; j < 2; ++j)
			{
				int lo[3], hi[3];
				l.In[j] = VoxPart(s, from, (int)(threadIdx.x & 31) + 32 * j, edge, lo, hi);
				VoxBall(s, lo, hi, scale, c[j], r[j], m[j]);
			}
			l.X = make_float2(c[0][0], c[1][0]);
			l.Y = make_float2(c[0][1], c[1][1]);
			l.Z = make_float2(c[0][2], c[1][2]);
			l.R = make_float2(r[0], r[1]);
			l.Margin = make_float2(m[0], m[1]);
			return l;
		}

		__device__ __forceinline__ float VoxReach(const VoxLane& l, float rootClip)
		{
			return fmaxf(TapeReach(l.R.x, l.X.x, l.Y.x, l.Z.x, rootClip), TapeReach(l.R.y, l.X.y, l.Y.y, l.Z.y, rootClip));
		}

		// One warp per 64^3 block: bound by the latency of one pass over the whole tree.
		__global__ void __launch_bounds__(32) VoxCoarseKernel(DeviceProgram prog, VoxSpec s, VoxGrid vg, VoxState st, int spill_pairs)
		{
			extern __shared__ __align__(16) uint8_t shared[];
			float4* window = reinterpret_cast<float4*>(shared);
			uint2* value = reinterpret_cast<uint2*>(window + 64);
			uint2* start = value + kVoxCoarseCap;
			float2* spill = reinterpret_cast<float2*>(start + kMaxStack + 2) + threadIdx.x;
			const int lane = (int)threadIdx.x, b = (int)blockIdx.x;
			const int from[3] = { (b % vg.NX) * kVoxCoarse, ((b / vg.NX) % vg.NY) * kVoxCoarse, (b / (vg.NX * vg.NY)) * kVoxCoarse };
			const float rootClip = fabsf(__ldg(&prog.Nodes[0].ClipRadius));
			const VoxLane l = VoxLaneOf(s, from, kVoxBlock, rootClip);
			SurfaceSource src;
			src.In.Open(prog.Code + prog.FullSurfaceCode, prog.CodeQuads - prog.FullSurfaceCode, window);
			TapeCounts counts;
			const bool ok = BuildTape<false, true>(src, l.X, l.Y, l.Z, VoxReach(l, rootClip), kRoundingSlack, prog.Widths, LoadPairUnits(), spill, 32,
				TapeLists{ value, nullptr, start, kVoxCoarseCap }, counts);
			if (ok)
				for (int i = lane; i < counts.Value; i += 32) st.Events[(int64_t)b * kVoxCoarseCap + i] = value[i];
			if (lane == 0) st.Counts[b] = ok ? (uint32_t)counts.Value : kNoTape;
#pragma unroll
			for (int j = 0; j < 2; ++j)
			{
				const float d = j ? counts.Distance.y : counts.Distance.x, r = j ? l.R.y : l.R.x;
				const float margin = (j ? l.Margin.y : l.Margin.x) + (j ? counts.Error.y : counts.Error.x);
				const bool keep = l.In[j] && !(fabsf(d) > r + s.Radius + margin);
				const unsigned kept = __ballot_sync(0xFFFFFFFFu, keep);
				uint32_t at = 0;
				if (lane == 0 && kept) at = atomicAdd(st.Counters, (uint32_t)__popc(kept));
				at = __shfl_sync(0xFFFFFFFFu, at, 0);
				if (keep) st.List[at + (uint32_t)__popc(kept & ((1u << lane) - 1u))] = (uint32_t)b * 64u + (uint32_t)(lane + 32 * j);
			}
		}

		// A list that finds no room still leaves the distances, which drop the boxes out of reach: 2000
		// primitives at 92^3 voxels 4933 us a call with every box of such a block kept, 3377 so; at 230^3
		// 11033 and 5306.
		//
		// One warp per listed 16^3 block, drawn from a counter: its tape from its 64^3 block's,
		// and the 4^3 boxes in it that may hold a kept voxel.  Direct: every 16^3 block, from the
		// whole tree's program (as where the 64^3 block's tape had no room).
		template<bool Direct>
		__global__ void __launch_bounds__(kVoxWarps * 32, kVoxCtasPerSm) VoxBlockKernel(DeviceProgram prog, VoxSpec s, VoxGrid vg, VoxState st,
			int spill_pairs)
		{
			extern __shared__ __align__(16) uint8_t shared[];
			const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
			VoxScratch& sc = reinterpret_cast<VoxScratch*>(shared)[warp];
			float2* spill = reinterpret_cast<float2*>(shared + kVoxWarps * sizeof(VoxScratch)) + warp * spill_pairs * 32 + lane;
			const float rootClip = fabsf(__ldg(&prog.Nodes[0].ClipRadius));
			const PairUnits units = LoadPairUnits();
			const uint32_t n = Direct ? (uint32_t)(vg.NX * vg.NY * vg.NZ) * 64u : st.Counters[0];
			for (;;)
			{
				uint32_t item = 0;
				if (lane == 0) item = atomicAdd(st.Counters + 1, 1u);
				item = __shfl_sync(0xFFFFFFFFu, item, 0);
				if (item >= n) break;
				const uint32_t entry = Direct ? item : __ldg(st.List + item);
				int from[3];
				VoxBlockStart(vg, entry, from);
				if (Direct && (from[0] >= s.SX || from[1] >= s.SY || from[2] >= s.SZ)) continue;
				const uint32_t given = Direct ? kNoTape : __ldg(st.Counts + (entry >> 6));
				const uint32_t first = Direct ? 0u : (entry >> 6) * (uint32_t)kVoxCoarseCap;
				const VoxLane l = VoxLaneOf(s, from, kVoxFine, rootClip);
				const TapeLists lists{ sc.Value, nullptr, sc.Start, kVoxBlockCap };
				bool ok;
				TapeCounts counts;
				__syncwarp();       // the previous block's events have been copied out
				if (Direct || given == kNoTape)
				{
					SurfaceSource src;
					src.In.Open(prog.Code + prog.FullSurfaceCode, prog.CodeQuads - prog.FullSurfaceCode, sc.Window);
					ok = BuildTape<false, true>(src, l.X, l.Y, l.Z, VoxReach(l, rootClip), kRoundingSlack, prog.Widths, units, spill, 32, lists, counts);
				}
				else
				{
					SurfaceEventSource src;
					src.Open(prog.Code + prog.FullSurfaceCode, st.Events + first, (int)given, sc.Window, sc.Heads);
					ok = BuildTape<false, true>(src, l.X, l.Y, l.Z, VoxReach(l, rootClip), kRoundingSlack, prog.Widths, units, spill, 32, lists, counts);
				}
				// The box goes by its own tape, where there is room for it.
				uint2 tape = make_uint2(first, given);
				if (ok)
				{
					uint32_t at = 0;
					if (lane == 0) at = atomicAdd(st.Counters + 2, (uint32_t)counts.Value);
					at = __shfl_sync(0xFFFFFFFFu, at, 0);
					if (at <= st.EventCap && st.EventCap - at >= (uint32_t)counts.Value)
					{
						tape = make_uint2(st.EventBase + at, (uint32_t)counts.Value);
						for (int i = lane; i < counts.Value; i += 32) st.Events[tape.x + i] = sc.Value[i];
					}
				}
				if (lane == 0) st.Tapes[item] = tape;
#pragma unroll
				for (int j = 0; j < 2; ++j)
				{
					const float d = j ? counts.Distance.y : counts.Distance.x, r = j ? l.R.y : l.R.x;
					const float margin = (j ? l.Margin.y : l.Margin.x) + (j ? counts.Error.y : counts.Error.x);
					const bool keep = l.In[j] && !(fabsf(d) > r + s.Radius + margin);
					const unsigned kept = __ballot_sync(0xFFFFFFFFu, keep);
					uint32_t at = 0;
					if (lane == 0 && kept) at = atomicAdd(st.Counters + 3, (uint32_t)__popc(kept));
					at = __shfl_sync(0xFFFFFFFFu, at, 0);
					if (keep) st.Boxes[at + (uint32_t)__popc(kept & ((1u << lane) - 1u))] = item * 64u + (uint32_t)(lane + 32 * j);
				}
			}
		}

		// The kept ones of a 4^3 box's voxels, by a warp: lane l has (x, y, z) and the voxel two above
		// it, with their distances.
		__device__ __forceinline__ void PutVoxBits(const VoxSpec& s, int x, int y, int z, float2 d, uint32_t* __restrict__ words)
		{
			const int lane = (int)(threadIdx.x & 31);
#pragma unroll
			for (int j = 0; j < 2; ++j)
			{
				const bool keep = x < s.SX && y < s.SY && z + 2 * j < s.SZ && fabsf(j ? d.y : d.x) <= s.Radius;
				const unsigned bits = __ballot_sync(0xFFFFFFFFu, keep);
				// A row of four voxels of the box is four neighbouring lanes.
				const uint32_t row = (bits >> (lane & 28)) & 15u;
				if ((lane & 3) == 0 && row)
				{
					const int64_t t = x + (int64_t)s.SX * (y + (int64_t)s.SY * (z + 2 * j));
					const int shift = (int)(t & 31);
					atomicOr(words + (t >> 5), row << shift);
					if (shift > 28 && (row >> (32 - shift))) atomicOr(words + (t >> 5) + 1, row >> (32 - shift));
				}
			}
		}

		// One warp per listed 4^3 box, drawn from a counter: its voxels, two a lane.
		__global__ void __launch_bounds__(kVoxWarps * 32, kVoxEvalCtasPerSm) VoxBoxKernel(DeviceProgram prog, VoxSpec s, VoxGrid vg, VoxState st,
			bool direct, uint32_t* __restrict__ words)
		{
			extern __shared__ __align__(16) float2 spill2[];
			const int lane = (int)(threadIdx.x & 31);
			const float4* code = prog.Code + prog.FullSurfaceCode;
			auto load = [&](int q) { return __ldg(code + q); };
			const PairUnits units = LoadPairUnits();
			const uint32_t n = st.Counters[3];
			for (;;)
			{
				uint32_t item = 0;
				if (lane == 0) item = atomicAdd(st.Counters + 4, 1u);
				item = __shfl_sync(0xFFFFFFFFu, item, 0);
				if (item >= n) break;
				const uint32_t entry = __ldg(st.Boxes + item);
				const uint32_t block = direct ? entry >> 6 : __ldg(st.List + (entry >> 6));
				const uint2 tape = __ldg(st.Tapes + (entry >> 6));
				int from[3];
				VoxBlockStart(vg, block, from);
				const int part = (int)(entry & 63u);
				const int x = from[0] + (part & 3) * kVoxFine + (lane & 3), y = from[1] + ((part >> 2) & 3) * kVoxFine + ((lane >> 2) & 3);
				const int z = from[2] + (part >> 4) * kVoxFine + (lane >> 4);
				const float cx = VoxCentre(s.Min[0], s.Max[0], x, s.SX), cy = VoxCentre(s.Min[1], s.Max[1], y, s.SY);
				const float2 px[1] = { make_float2(cx, cx) }, py[1] = { make_float2(cy, cy) };
				const float2 pz[1] = { make_float2(VoxCentre(s.Min[2], s.Max[2], z, s.SZ), VoxCentre(s.Min[2], s.Max[2], z + 2, s.SZ)) };
				float2 d[1];
				const uint2* events = st.Events + tape.x;
				if (tape.y == kNoTape) d[0] = RunWholeSurfacePair(prog.Code, prog.FullSurfaceCode, px[0], py[0], pz[0], spill2 + threadIdx.x, kVoxWarps * 32);
				else
					RunSurfaceTapePairs<1>(load, 0, [&](uint32_t e) { return __ldg(events + e); }, tape.y, px, py, pz, units, d, spill2 + threadIdx.x,
						kVoxWarps * 32);
				PutVoxBits(s, x, y, z, d[0], words);
			}
		}

		// Small lattices: every 4^3 box by the whole tree's program, one warp each.  A pass over the
		// blocks first is as long as that by itself, and leaves few of so few boxes out.
		__global__ void __launch_bounds__(kVoxWarps * 32) VoxWholeKernel(DeviceProgram prog, VoxSpec s, int nx, int ny, int nz, int spill_pairs,
			uint32_t* __restrict__ words)
		{
			extern __shared__ __align__(16) float4 shared4[];
			const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
			const int box = (int)blockIdx.x * kVoxWarps + warp;
			if (box >= nx * ny * nz) return;
			const int x = box % nx * kVoxFine + (lane & 3), y = box / nx % ny * kVoxFine + ((lane >> 2) & 3);
			const int z = box / (nx * ny) * kVoxFine + (lane >> 4);
			const float cx = VoxCentre(s.Min[0], s.Max[0], x, s.SX), cy = VoxCentre(s.Min[1], s.Max[1], y, s.SY);
			SurfaceSource src;
			src.In.Open(prog.Code + prog.FullSurfaceCode, prog.CodeQuads - prog.FullSurfaceCode, shared4 + warp * 64);
			const float2 d = RunSourcePair(src, make_float2(cx, cx), make_float2(cy, cy),
				make_float2(VoxCentre(s.Min[2], s.Max[2], z, s.SZ), VoxCentre(s.Min[2], s.Max[2], z + 2, s.SZ)), LoadPairUnits(),
				reinterpret_cast<float2*>(shared4 + kVoxWarps * 64) + warp * spill_pairs * 32 + lane, 32);
			PutVoxBits(s, x, y, z, d, words);
		}

		// Trees whose programs cannot be shortened (a brush that is not 1-Lipschitz, rotations that
		// are not unit quaternions): one thread per brick of VoxExport's voxels: the whole tree's program at the centre
		// of the ball through the brick's voxel centres decides (a tree with a brush that is
		// not 1-Lipschitz keeps every brick).  mix() rounds each centre separately, so the
		// box is widened by a relative 1e-6 of its coordinates.
		__global__ void __launch_bounds__(128) VoxBricksKernel(DeviceProgram prog, VoxSpec s, VoxelBricks vb,
			uint32_t* __restrict__ brick_bits)
		{
			extern __shared__ float spill[];
			const int b = (int)(blockIdx.x * blockDim.x + threadIdx.x);
			if (b >= vb.NX * vb.NY * vb.NZ) return;
			bool keep = true;
			if (prog.Lipschitz)
			{
				int lo[3], hi[3];
				BrickRange(b, vb, s.SX, s.SY, s.SZ, lo, hi);
				const int size[3] = { s.SX, s.SY, s.SZ };
				float clo[3], chi[3];
#pragma unroll
				for (int a = 0; a < 3; ++a)
				{
					const float u = VoxCentre(s.Min[a], s.Max[a], lo[a], size[a]);
					const float v = VoxCentre(s.Min[a], s.Max[a], hi[a], size[a]);
					const float slack = 1e-6f * (fabsf(u) + fabsf(v) + fabsf(s.Min[a]) + fabsf(s.Max[a]));
					clo[a] = fminf(u, v) - slack;
					chi[a] = fmaxf(u, v) + slack;
				}
				float c[3], r, margin;
				BallOf(clo, chi, c, r, margin, fabsf(__ldg(&prog.Nodes[0].ClipRadius)));
				const float px[1] = { c[0] }, py[1] = { c[1] }, pz[1] = { c[2] };
				float f[1];
				RunSurfaceBatch<1>(prog.Code, prog.FullSurfaceCode, px, py, pz, f, -1, nullptr, spill + threadIdx.x, 128);
				keep = !(fabsf(f[0]) > r + s.Radius + margin);
			}
			if (keep) atomicOr(brick_bits + (b >> 5), 1u << (b & 31));
		}

		// VoxExport's test at every voxel of the bricks kept: the voxel centre mix(Min, Max, (x + .5) / Size)
		// on the whole tree (SDFNode::Eval), kept when |d| <= Radius.
		__global__ void __launch_bounds__(128) VoxFlagsKernel(DeviceProgram prog, VoxSpec s, VoxelBricks vb,
			const uint32_t* __restrict__ brick_bits, uint32_t* __restrict__ words)
		{
			extern __shared__ float spill[];
			const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
			bool keep = false;
			int x = 0, y = 0, z = 0;
			bool live = false;
			if (t < s.Total)
			{
				const int i = (int)t;
				const int slice = s.SX * s.SY;
				z = i / slice; y = (i % slice) / s.SX; x = i % s.SX;
				const int b = BrickOfVoxel(x, y, z, vb);
				live = (__ldg(brick_bits + (b >> 5)) >> (b & 31)) & 1u;
			}
			if (live)
			{
				const float px[1] = { VoxCentre(s.Min[0], s.Max[0], x, s.SX) };
				const float py[1] = { VoxCentre(s.Min[1], s.Max[1], y, s.SY) };
				const float pz[1] = { VoxCentre(s.Min[2], s.Max[2], z, s.SZ) };
				float r[1];
				RunSurfaceBatch<1>(prog.Code, prog.FullSurfaceCode, px, py, pz, r, -1, nullptr, spill + threadIdx.x, 128);
				keep = fabsf(r[0]) <= s.Radius;
			}
			const unsigned ballot = __ballot_sync(0xFFFFFFFFu, keep);
			if ((threadIdx.x & 31) == 0 && t < s.Total) words[t >> 5] = ballot;
		}

		__global__ void __launch_bounds__(128) VoxListKernel(VoxSpec s, const uint32_t* __restrict__ words, const uint32_t* __restrict__ base,
			int64_t n, int color, int4* __restrict__ out)
		{
			const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
			if (w >= n) return;
			uint32_t m = __ldg(words + w);
			if (!m) return;
			uint32_t at = __ldg(base + w);
			const int slice = s.SX * s.SY;
			while (m)
			{
				const int i = (int)(w * 32) + __ffs((int)m) - 1;
				m &= m - 1u;
				out[at++] = make_int4(i % s.SX, (i % slice) / s.SX, i / slice, color);
			}
		}
	}

	namespace
	{
		VoxelBricks BricksOf(int sx, int sy, int sz)
		{
			return { (sx + kVoxelBrick - 1) / kVoxelBrick, (sy + kVoxelBrick - 1) / kVoxelBrick, (sz + kVoxelBrick - 1) / kVoxelBrick };
		}

		size_t DistanceSpillBytes(const DeviceProgram& prog, int threads)
		{
			const int depth = prog.MaxStack > 1 ? prog.MaxStack - 1 : 1;
			return (size_t)depth * 2 * threads * sizeof(float);
		}
	}

	size_t VoxelBrickWords(int sx, int sy, int sz)
	{
		const VoxelBricks vb = BricksOf(sx, sy, sz);
		return ((size_t)vb.NX * vb.NY * vb.NZ + 31) / 32;
	}

	cudaError_t LaunchCloudFlags(const DeviceProgram& prog, const CloudSpec& s, uint32_t* brick_bits, uint32_t* words, cudaStream_t stream)
	{
		if (s.Total <= 0) return cudaSuccess;
		const VoxelBricks vb = BricksOf(s.IX, s.IY, s.IZ);
		const int nb = vb.NX * vb.NY * vb.NZ;
		cudaError_t e = cudaMemsetAsync(brick_bits, 0, VoxelBrickWords(s.IX, s.IY, s.IZ) * 4, stream);
		if (e != cudaSuccess) return e;
		const size_t smem = DistanceSpillBytes(prog, 128);
		if (smem > 48 * 1024)
		{
			e = cudaFuncSetAttribute(CloudBricksKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e == cudaSuccess) e = cudaFuncSetAttribute(CloudFlagsKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		CloudBricksKernel<<<Blocks(nb, 128), 128, smem, stream>>>(prog, s, vb, brick_bits);
		e = cudaGetLastError();
		if (e != cudaSuccess) return e;
		CloudFlagsKernel<<<Blocks(s.Total, 128), 128, smem, stream>>>(prog, s, vb, brick_bits, words);
		return cudaGetLastError();
	}

	int64_t CloudBricks(const CloudSpec& s)
	{
		const CloudLattice lat{ s };
		return (int64_t)lat.Bricks(0) * lat.Bricks(1) * lat.Bricks(2);
	}

	cudaError_t LaunchCloudVoxels(const DeviceProgram& prog, const CloudSpec& s, uint32_t* list, uint32_t* tops, const BrickTapes& tapes,
		uint32_t* words, uint32_t* voxels, uint32_t* counts, int sms, cudaStream_t stream)
	{
		const CloudLattice lat{ s };
		cudaError_t e = cudaMemsetAsync(counts, 0, 2 * sizeof(uint32_t), stream);
		if (e == cudaSuccess) e = cudaMemsetAsync(words, 0, (size_t)((s.Total + 31) / 32) * 4, stream);
		// Bricks that are not listed are looked up too, by points that wander: no parts there.
		if (e == cudaSuccess) e = cudaMemsetAsync(tapes.Bricks, 0, (size_t)CloudBricks(s) * sizeof(uint2), stream);
		if (e != cudaSuccess) return e;
		size_t smem = DistanceSpillBytes(prog, 128);
		if (smem > 48 * 1024)
		{
			e = cudaFuncSetAttribute(CloudListKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		CloudListKernel<<<Blocks(CloudBricks(s), 128), 128, smem, stream>>>(prog, lat, list, counts, tops);
		e = cudaGetLastError();
		if (e == cudaSuccess) e = parts::LaunchParts(prog, lat, list, counts, tops, tapes, sms, stream);
		if (e != cudaSuccess) return e;
		smem = parts::SpillPairs(prog, 1) * parts::kThreads * sizeof(float2);
		if (smem > 39 * 1024)
		{
			e = cudaFuncSetAttribute(CloudVoxelsKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		CloudVoxelsKernel<<<sms * 8, parts::kThreads, smem, stream>>>(prog, lat, list, counts, tapes, words, voxels, counts + 1);
		return cudaGetLastError();
	}

	cudaError_t LaunchCloudPoints(const DeviceProgram& prog, const CloudSpec& s, const BrickTapes& tapes, const uint32_t* voxels, uint32_t n,
		const uint32_t* words, const uint32_t* word_base, int iterations, uint32_t* cubes, float* points, float* normals, uint8_t* colors,
		cudaStream_t stream)
	{
		if (n == 0) return cudaSuccess;
		// The colour's walk takes two words a level, the gradient one pair.
		const size_t smem = parts::SpillPairs(prog, 2) * parts::kThreads * sizeof(float2);
		if (smem > 48 * 1024)
		{
			const cudaError_t e = cudaFuncSetAttribute(CloudPointsKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		CloudPointsKernel<<<Blocks(n, parts::kThreads), parts::kThreads, smem, stream>>>(prog, CloudLattice{ s }, tapes, voxels, n, words, word_base,
			iterations, cubes, points, normals, colors);
		return cudaGetLastError();
	}

	cudaError_t LaunchCloudRefine(const DeviceProgram& prog, const CloudSpec& s, const uint32_t* cells, const uint32_t* count,
		uint32_t capacity, int iterations, float* points, cudaStream_t stream)
	{
		if (capacity == 0) return cudaSuccess;
		// The gradient's four-point surface pass: four distances and a material slot per
		// depth (RunSurfaceBatch<4>'s layout), enough for the distance pass too.
		const int depth = prog.MaxStack > 1 ? prog.MaxStack - 1 : 1;
		const size_t smem = (size_t)depth * 5 * 128 * sizeof(float);
		if (smem > 48 * 1024)
		{
			const cudaError_t e = cudaFuncSetAttribute(CloudRefineKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		CloudRefineKernel<<<Blocks(capacity, 128), 128, smem, stream>>>(prog, s, cells, count, iterations, points);
		return cudaGetLastError();
	}

	static VoxGrid VoxGridOf(const VoxSpec& s)
	{
		return { (s.SX + kVoxCoarse - 1) / kVoxCoarse, (s.SY + kVoxCoarse - 1) / kVoxCoarse, (s.SZ + kVoxCoarse - 1) / kVoxCoarse };
	}

	// Lattices so thin that most of their blocks lie outside keep the general path: the blocks'
	// scratch would outgrow the lattice's own.
	static bool VoxByBlocks(const DeviceProgram& prog, const VoxSpec& s)
	{
		const VoxGrid vg = VoxGridOf(s);
		return prog.Lipschitz && (prog.Form & kFormPrunable) && (int64_t)vg.NX * vg.NY * vg.NZ <= 64 + s.Total / 16384;
	}

	// The scratch's parts, 16-byte aligned one after the other; the bytes they take.
	static size_t VoxLayout(const VoxSpec& s, void* scratch, VoxState& st)
	{
		const VoxGrid vg = VoxGridOf(s);
		const size_t blocks = (size_t)vg.NX * vg.NY * vg.NZ, boxes = blocks * 64;
		size_t at = 0;
		auto take = [&](size_t bytes) { uint8_t* p = static_cast<uint8_t*>(scratch) + at; at += (bytes + 15) / 16 * 16; return p; };
		// Events of the 16^3 blocks' own tapes: 16 on average, one block in four or five listed.
		st.EventBase = (uint32_t)(blocks * kVoxCoarseCap);
		st.EventCap = (uint32_t)(boxes * 16);
		st.Events = reinterpret_cast<uint2*>(take(((size_t)st.EventBase + st.EventCap) * sizeof(uint2)));
		st.Counts = reinterpret_cast<uint32_t*>(take(blocks * sizeof(uint32_t)));
		st.List = reinterpret_cast<uint32_t*>(take(boxes * sizeof(uint32_t)));
		st.Tapes = reinterpret_cast<uint2*>(take(boxes * sizeof(uint2)));
		st.Boxes = reinterpret_cast<uint32_t*>(take(boxes * 64 * sizeof(uint32_t)));
		st.Counters = reinterpret_cast<uint32_t*>(take(kVoxCounters * sizeof(uint32_t)));
		return at;
	}

	static int VoxBoxes(int voxels) { return (voxels + kVoxFine - 1) / kVoxFine; }

	// Lattices whose 4^3 boxes the GPU runs at once go without blocks.  Measured on a GB300, with
	// blocks / without, us a call: 60 primitives 6^3 voxels 144 / 84, 48^3 122 / 94, 80^3 115 / 170;
	// 400 primitives 15^3 653 / 285, 60^3 683 / 416; 2000 primitives 13^3 2979 / 1192, 55^3 3186 / 1613.
	static bool VoxWhole(const VoxSpec& s)
	{
		return (int64_t)VoxBoxes(s.SX) * VoxBoxes(s.SY) * VoxBoxes(s.SZ) <= kVoxWholeBoxes;
	}

	size_t VoxBlockBytes(const DeviceProgram& prog, const VoxSpec& s)
	{
		if (s.Total <= 0 || !VoxByBlocks(prog, s)) return 0;
		if (VoxWhole(s)) return 16;
		VoxState st;
		return VoxLayout(s, nullptr, st);
	}

	cudaError_t LaunchVoxFlags(const DeviceProgram& prog, const VoxSpec& s, uint32_t* brick_bits, uint32_t* words, cudaStream_t stream)
	{
		if (s.Total <= 0) return cudaSuccess;
		const VoxelBricks vb = BricksOf(s.SX, s.SY, s.SZ);
		const int nb = vb.NX * vb.NY * vb.NZ;
		cudaError_t e = cudaMemsetAsync(brick_bits, 0, VoxelBrickWords(s.SX, s.SY, s.SZ) * 4, stream);
		if (e != cudaSuccess) return e;
		const size_t smem = DistanceSpillBytes(prog, 128);
		if (smem > 48 * 1024)
		{
			e = cudaFuncSetAttribute(VoxFlagsKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e == cudaSuccess) e = cudaFuncSetAttribute(VoxBricksKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		VoxBricksKernel<<<Blocks(nb, 128), 128, smem, stream>>>(prog, s, vb, brick_bits);
		e = cudaGetLastError();
		if (e != cudaSuccess) return e;
		VoxFlagsKernel<<<Blocks(s.Total, 128), 128, smem, stream>>>(prog, s, vb, brick_bits, words);
		return cudaGetLastError();
	}

	cudaError_t LaunchVoxBlocks(const DeviceProgram& prog, const VoxSpec& s, void* scratch, uint32_t most_events, uint32_t* words, int sms,
		cudaStream_t stream)
	{
		const int depth = prog.MaxStack > 1 ? prog.MaxStack - 1 : 1;
		cudaError_t e = cudaMemsetAsync(words, 0, (size_t)((s.Total + 31) / 32) * 4, stream);
		if (e != cudaSuccess) return e;
		if (VoxWhole(s))
		{
			const int nx = VoxBoxes(s.SX), ny = VoxBoxes(s.SY), nz = VoxBoxes(s.SZ);
			const size_t smem = kVoxWarps * (64 * sizeof(float4) + (size_t)depth * 32 * sizeof(float2));
			VoxWholeKernel<<<(unsigned)((nx * ny * nz + kVoxWarps - 1) / kVoxWarps), kVoxWarps * 32, smem, stream>>>(prog, s, nx, ny, nz, depth, words);
			return cudaGetLastError();
		}
		const VoxGrid vg = VoxGridOf(s);
		VoxState st;
		VoxLayout(s, scratch, st);
		if (st.EventCap > most_events) st.EventCap = most_events;
		e = cudaMemsetAsync(st.Counters, 0, kVoxCounters * sizeof(uint32_t), stream);
		if (e != cudaSuccess) return e;
		const size_t coarse = 64 * sizeof(float4) + (kVoxCoarseCap + kMaxStack + 2) * sizeof(uint2) + (size_t)depth * 32 * sizeof(float2);
		const size_t fine = kVoxWarps * (sizeof(VoxScratch) + (size_t)depth * 32 * sizeof(float2));
		const size_t eval = kVoxWarps * (size_t)depth * 32 * sizeof(float2);
		// The first level costs a pass over the whole tree by itself: lattices whose 16^3 blocks
		// the GPU runs at once go without it.
		const int64_t small = (int64_t)((s.SX + kVoxBlock - 1) / kVoxBlock) * ((s.SY + kVoxBlock - 1) / kVoxBlock) * ((s.SZ + kVoxBlock - 1) / kVoxBlock);
		const bool direct = small <= kVoxDirectBlocks;
		auto* block = direct ? VoxBlockKernel<true> : VoxBlockKernel<false>;
		if (coarse > 48 * 1024) e = cudaFuncSetAttribute(VoxCoarseKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)coarse);
		if (e == cudaSuccess && fine > 48 * 1024) e = cudaFuncSetAttribute(block, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fine);
		if (e != cudaSuccess) return e;
		if (!direct)
		{
			VoxCoarseKernel<<<(unsigned)(vg.NX * vg.NY * vg.NZ), 32, coarse, stream>>>(prog, s, vg, st, depth);
			e = cudaGetLastError();
			if (e != cudaSuccess) return e;
		}
		block<<<sms * kVoxCtasPerSm, kVoxWarps * 32, fine, stream>>>(prog, s, vg, st, depth);
		e = cudaGetLastError();
		if (e != cudaSuccess) return e;
		VoxBoxKernel<<<sms * kVoxEvalCtasPerSm, kVoxWarps * 32, eval, stream>>>(prog, s, vg, st, direct, words);
		return cudaGetLastError();
	}

	cudaError_t LaunchVoxList(const VoxSpec& s, const uint32_t* words, const uint32_t* word_base, int color, int4* out, cudaStream_t stream)
	{
		const int64_t n = (s.Total + 31) / 32;
		if (n <= 0) return cudaSuccess;
		VoxListKernel<<<Blocks(n, 128), 128, 0, stream>>>(s, words, word_base, n, color, out);
		return cudaGetLastError();
	}
}
