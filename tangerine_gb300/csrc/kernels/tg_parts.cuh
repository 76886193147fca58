// Bricks of up to 8^3 points of a lattice, evaluated through shortened programs (tg_tape.cuh).
//
// A brick's points fall in one octree cell or, where it straddles pivots, in a few: its parts
// are the boxes of points that share one cell (BrickPartsKernel).  Each part gets a tape of
// its cell's program (BuildPartTapesKernel, one pass of the program at 64 points by a warp),
// which the part's points and the vertices in it then run.
//
// A lattice L says where its points lie: Coord(axis, index), Points(axis), Bricks(axis),
// kStride (points from one brick to the next), kBox (points of a brick per axis, at most 16),
// kMost (parts of a brick, at most), kOutside (vertices may leave their brick by up to a step),
// kBetween (points between the lattice's look for their part, too), kShortest (quads of the
// programs that get a tape, at least; not 0: the tapes are there to build finer ones from),
// kAbove (there may be such coarser tapes: those of brick Above(b) for brick b), and Keep(): the
// distance beyond which a part's points are of no interest.
#pragma once

#include "tg_device.cuh"
#include "tg_kernels.hpp"
#include "tg_surface.cuh"
#include "tg_tape.cuh"

namespace tg
{
	namespace parts
	{
		constexpr int kThreads = 128;
		constexpr int kWarps = kThreads / 32;
		constexpr int kPartCtasPerSm = 12;
		constexpr int kBuildCtasPerSm = 8;
		constexpr int kBox = 8;             // points per axis of most lattices' bricks
		constexpr int kLongQuads = 96;      // programs from this long are built first
		constexpr int kAboveQuads = 48;     // and from this long by way of a coarser brick's tape

		__device__ __forceinline__ uint32_t PackBox(int x0, int x1, int y0, int y1, int z0, int z1)
		{
			return (uint32_t)(x0 | (x1 << 4) | (y0 << 8) | (y1 << 12) | (z0 << 16) | (z1 << 20));
		}

		constexpr uint32_t kBoxLong = 0x80000000u;     // the part is in the list of long ones
		constexpr uint32_t kBoxPositive = 0x40000000u; // the distance stays above the lattice's Keep() in the part,
		constexpr uint32_t kBoxNegative = 0x20000000u; // or below its negative

		// Last index in [lo, hi] of axis a whose coordinate is not above the pivot (lo - 1: none).
		template<typename L>
		__device__ __forceinline__ int LastAtMost(const L& lat, int a, int first, int lo, int hi, float pivot)
		{
			int in = lo - 1, out = hi + 1;
#pragma unroll
			for (int step = 0; step < (L::kBox > 8 ? 5 : 4); ++step)
			{
				const int mid = (in + out) >> 1;
				if (out - in < 2) break;
				if (!(lat.Coord(a, first + mid) > pivot)) in = mid;
				else out = mid;
			}
			return in;
		}

		// The first point of brick b per axis, and how many points follow it in the brick.
		template<typename L>
		__device__ __forceinline__ void BrickSpan(const L& lat, uint32_t b, int (&first)[3], int (&extent)[3])
		{
			const uint32_t nx = (uint32_t)lat.Bricks(0), ny = (uint32_t)lat.Bricks(1);
			const uint32_t row = b / nx, bz = row / ny;
			first[0] = (int)(b - row * nx) * L::kStride;
			first[1] = (int)(row - bz * ny) * L::kStride;
			first[2] = (int)bz * L::kStride;
#pragma unroll
			for (int a = 0; a < 3; ++a) extent[a] = min(L::kBox - 1, lat.Points(a) - 1 - first[a]);
		}

		// A brick's box as DescendBox's answer: the cell reached, bit 31 set when every point of
		// the box descends to it.
		template<typename L>
		__device__ __forceinline__ uint32_t DescendBrick(const DeviceProgram& prog, const L& lat, const int (&first)[3], const int (&extent)[3])
		{
			bool shared;
			const int top = DescendBox(prog.Nodes, lat.Coord(0, first[0]), lat.Coord(0, first[0] + extent[0]), lat.Coord(1, first[1]),
				lat.Coord(1, first[1] + extent[1]), lat.Coord(2, first[2]), lat.Coord(2, first[2] + extent[2]), shared);
			return (uint32_t)top | (shared ? 0x80000000u : 0u);
		}

		template<typename L>
		__device__ __forceinline__ void PutPart(const DeviceProgram& prog, const L& lat, const BrickTapes& tapes, uint32_t slot, int cell, uint32_t b,
			uint32_t box)
		{
			BrickPart out;
			out.Cell = cell;
			out.Box = box;
			out.Value = out.Material = 0;
			out.Counts = kNoTape | (kNoTape << 16);
			out.Distance = out.Surface = 0;
			out.Brick = b;
			out.First = make_uint2(0u, 0u);
#pragma unroll
			for (int a = 0; a < 3; ++a) { out.Lo[a] = 1.0f; out.Hi[a] = 0.0f; }
			if (cell >= 0)
			{
				out.Distance = __ldg(&prog.Nodes[cell].DistanceCode);
				out.Surface = __ldg(&prog.Nodes[cell].SurfaceCode);
				if (out.Surface - out.Distance >= kLongQuads)
				{
					const uint32_t at = atomicAdd(tapes.Counters + 4, 1u);
					if (at < kLongParts)
					{
						tapes.Long[at] = slot;
						out.Box |= kBoxLong;
					}
				}
				int first[3], extent[3];
				BrickSpan(lat, b, first, extent);
				if constexpr (!L::kBetween)
				{
#pragma unroll
					for (int a = 0; a < 3; ++a)
					{
						out.Lo[a] = lat.Coord(a, first[a] + (int)((box >> (8 * a)) & 15u));
						out.Hi[a] = lat.Coord(a, first[a] + (int)((box >> (8 * a + 4)) & 15u));
					}
				}
				else
				{
					float p[3];
#pragma unroll
					for (int a = 0; a < 3; ++a)
					{
						const int x0 = (int)((box >> (8 * a)) & 15u), x1 = (int)((box >> (8 * a + 4)) & 15u);
						p[a] = lat.Coord(a, first[a] + x0);
						out.Lo[a] = lat.Coord(a, first[a] + (L::kOutside ? x0 - 1 : max(x0 - 1, 0)));
						out.Hi[a] = lat.Coord(a, first[a] + (L::kOutside ? x1 + 1 : min(x1 + 1, extent[a])));
					}
					// The pivots passed on the way to the cell bound it (DescendOctree's `p > pivot`).
					int at = 0;
					for (int guard = 0; guard < 64; ++guard)
					{
						const float4 n = __ldg(reinterpret_cast<const float4*>(prog.Nodes + at));
						if (__float_as_int(n.w) & kNodeTerminus) break;
						const float pivot[3] = { n.x, n.y, n.z };
						int octant = 0;
#pragma unroll
						for (int a = 0; a < 3; ++a)
						{
							if (p[a] > pivot[a]) { octant |= 1 << a; out.Lo[a] = fmaxf(out.Lo[a], nextafterf(pivot[a], INFINITY)); }
							else out.Hi[a] = fminf(out.Hi[a], pivot[a]);
						}
						const int child = __ldg(&prog.Nodes[at].Child[octant]);
						if (child < 0) break;
						at = child;
					}
				}
			}
			const uint4* from = reinterpret_cast<const uint4*>(&out);
			uint4* to = reinterpret_cast<uint4*>(tapes.Parts + slot);
#pragma unroll
			for (int q = 0; q < (int)(sizeof(BrickPart) / sizeof(uint4)); ++q) to[q] = from[q];
		}

		// The parts of a brick of any size against the cells, by one thread: its box of corner
		// points is split at the pivots it straddles until each piece is in one cell.
		template<typename L>
		__device__ __noinline__ void SplitBrick(const DeviceProgram& prog, const L& lat, const BrickTapes& tapes, uint32_t b, int i0, int j0, int k0,
			int top, uint32_t whole)
		{
			constexpr int kMost = L::kMost, kStack = kMost > 24 ? 48 : 24;
			uint2 found[kMost], stack[kStack];
			int parts = 0, depth = 0;
			bool fits = true;
			stack[depth++] = make_uint2((uint32_t)top, whole);
			for (int guard = 0; guard < 512 && depth > 0; ++guard)
			{
				const uint2 s = stack[--depth];
				const int node = (int)s.x;
				const int lo[3] = { (int)(s.y & 15u), (int)((s.y >> 8) & 15u), (int)((s.y >> 16) & 15u) };
				const int hi[3] = { (int)((s.y >> 4) & 15u), (int)((s.y >> 12) & 15u), (int)((s.y >> 20) & 15u) };
				const float4 a = __ldg(reinterpret_cast<const float4*>(prog.Nodes + node));
				if (__float_as_int(a.w) & kNodeTerminus)
				{
					if (parts < kMost) found[parts++] = s;
					else fits = false;
					continue;
				}
				const int cut[3] = { LastAtMost(lat, 0, i0, lo[0], hi[0], a.x), LastAtMost(lat, 1, j0, lo[1], hi[1], a.y),
					LastAtMost(lat, 2, k0, lo[2], hi[2], a.z) };
				for (int octant = 0; octant < 8; ++octant)
				{
					const int x0 = (octant & 1) ? cut[0] + 1 : lo[0], x1 = (octant & 1) ? hi[0] : cut[0];
					const int y0 = (octant & 2) ? cut[1] + 1 : lo[1], y1 = (octant & 2) ? hi[1] : cut[1];
					const int z0 = (octant & 4) ? cut[2] + 1 : lo[2], z1 = (octant & 4) ? hi[2] : cut[2];
					if (x1 < x0 || y1 < y0 || z1 < z0) continue;
					const int child = __ldg(&prog.Nodes[node].Child[octant]);
					const uint32_t box = PackBox(x0, x1, y0, y1, z0, z1);
					if (child < 0)
					{
						// The octant has no cell of its own: this cell's evaluator.
						if (parts < kMost) found[parts++] = make_uint2((uint32_t)node, box);
						else fits = false;
					}
					else if (depth < kStack) stack[depth++] = make_uint2((uint32_t)child, box);
					else fits = false;
				}
			}
			if (depth > 0 || !fits)
			{
				tapes.Bricks[b] = make_uint2(0u, 0u);
				return;
			}
			const uint32_t first = atomicAdd(tapes.Counters, (uint32_t)parts);
			const uint32_t room = first < tapes.PartCapacity ? tapes.PartCapacity - first : 0u;
			fits = room >= (uint32_t)parts;
			tapes.Bricks[b] = make_uint2(first, fits ? (uint32_t)parts : 0u);
			// Slots taken without room for all of the brick's parts stay in the list as dead ones.
			for (int p = 0; p < parts && (uint32_t)p < room; ++p)
				PutPart(prog, lat, tapes, first + (uint32_t)p, fits ? (int)found[p].x : -1, b, found[p].y);
		}

		// The parts of each kept brick.  Where cells are larger than the brick (fine grids: most
		// bricks), every part holds a corner of it: eight threads per brick each descend one
		// corner, cutting the brick's index ranges at the pivots passed (DescendOctree's rule,
		// `p > pivot`, on whole ranges), and a part is emitted by the lowest corner in it.  A
		// brick that this does not cover is split by SplitBrick; one that has no room gets no
		// parts, and its points then descend one by one.  Latency-bound: the descents are chains
		// of two loads a level.
		template<typename L>
		__global__ void __launch_bounds__(kThreads) BrickPartsKernel(DeviceProgram prog, L lat, const uint32_t* __restrict__ list,
			const uint32_t* __restrict__ count, const uint32_t* __restrict__ tops, BrickTapes tapes)
		{
			const uint32_t n = count ? *count : (uint32_t)lat.Bricks(0) * (uint32_t)lat.Bricks(1) * (uint32_t)lat.Bricks(2);
			const int lane = (int)(threadIdx.x & 31), corner = lane & 7;
			for (uint32_t base = (blockIdx.x * kWarps + (threadIdx.x >> 5)) * 4u; base < n; base += gridDim.x * kWarps * 4u)
			{
				const uint32_t item = base + (uint32_t)(lane >> 3);
				const bool live = item < n;
				const uint32_t b = live ? (list ? __ldg(list + item) : item) : 0u;
				int first3[3], extent[3];
				BrickSpan(lat, b, first3, extent);
				const int i0 = first3[0], j0 = first3[1], k0 = first3[2], ex = extent[0], ey = extent[1], ez = extent[2];
				int top = 0, cell = -1;
				int x0 = 0, x1 = ex, y0 = 0, y1 = ey, z0 = 0, z1 = ez;
				bool emit = false;
				if (live)
				{
					const uint32_t packed = tops ? __ldg(tops + b) : DescendBrick(prog, lat, first3, extent);
					cell = top = (int)(packed & 0x7FFFFFFFu);
					if (packed >> 31) emit = corner == 0;
					else
					{
						const float x = lat.Coord(0, i0 + ((corner & 1) ? ex : 0));
						const float y = lat.Coord(1, j0 + ((corner & 2) ? ey : 0));
						const float z = lat.Coord(2, k0 + ((corner & 4) ? ez : 0));
						for (int guard = 0; guard < 64; ++guard)
						{
							const float4 a = __ldg(reinterpret_cast<const float4*>(prog.Nodes + cell));
							if (__float_as_int(a.w) & kNodeTerminus) break;
							const bool hx = x > a.x, hy = y > a.y, hz = z > a.z;
							const int child = __ldg(&prog.Nodes[cell].Child[(hx ? 1 : 0) | (hy ? 2 : 0) | (hz ? 4 : 0)]);
							const int cx = LastAtMost(lat, 0, i0, x0, x1, a.x), cy = LastAtMost(lat, 1, j0, y0, y1, a.y);
							const int cz = LastAtMost(lat, 2, k0, z0, z1, a.z);
							if (hx) x0 = cx + 1; else x1 = cx;
							if (hy) y0 = cy + 1; else y1 = cy;
							if (hz) z0 = cz + 1; else z1 = cz;
							if (child < 0) break;
							cell = child;
						}
						emit = (!(corner & 1) || x0 > 0) && (!(corner & 2) || y0 > 0) && (!(corner & 4) || z0 > 0);
					}
				}
				int covered = emit ? (x1 - x0 + 1) * (y1 - y0 + 1) * (z1 - z0 + 1) : 0;
#pragma unroll
				for (int o = 1; o < 8; o <<= 1) covered += __shfl_xor_sync(0xFFFFFFFFu, covered, o);
				const bool all = covered == (ex + 1) * (ey + 1) * (ez + 1);
				const bool mine = emit && all;
				const unsigned emits = __ballot_sync(0xFFFFFFFFu, mine);
				uint32_t start = 0;
				if (lane == 0 && emits) start = atomicAdd(tapes.Counters, (uint32_t)__popc(emits));
				start = __shfl_sync(0xFFFFFFFFu, start, 0);
				const unsigned group = 0xFFu << (lane & 24);
				const uint32_t first = start + (uint32_t)__popc(emits & ((1u << (lane & 24)) - 1u));
				const uint32_t parts = (uint32_t)__popc(emits & group);
				const uint32_t room = first < tapes.PartCapacity ? tapes.PartCapacity - first : 0u;
				const bool fits = room >= parts;
				if (mine)
				{
					const uint32_t at = (uint32_t)__popc(emits & group & ((1u << lane) - 1u));
					if (at < room) PutPart(prog, lat, tapes, first + at, fits ? cell : -1, b, PackBox(x0, x1, y0, y1, z0, z1));
				}
				if (live && corner == 0)
				{
					if (all) tapes.Bricks[b] = make_uint2(first, fits ? parts : 0u);
					else SplitBrick(prog, lat, tapes, b, i0, j0, k0, top, PackBox(0, ex, 0, ey, 0, ez));
				}
			}
		}

		// A warp's scratch while it builds a part's tape.
		template<int Cap>
		struct TapeScratch
		{
			uint2 Value[Cap], Material[Cap];
			uint2 Start[kMaxStack + 2];
			uint2 Heads[8];
			float4 Window[64];
		};

		// The part of a coarser lattice's brick that holds this one, with a material list: that
		// list leaves out nothing that any point of it needs, for the distance or for the material.
		__device__ __forceinline__ int PartAround(const BrickTapes& above, uint2 own, int cell, const float (&lo)[3], const float (&hi)[3])
		{
			const uint32_t q = threadIdx.x & 31;
			bool mine = false;
			if (q < own.y)
			{
				const BrickPart& p = above.Parts[own.x + q];
				mine = p.Cell == cell && (p.Counts >> 16) != kNoTape;
#pragma unroll
				for (int a = 0; a < 3; ++a) mine = mine && p.Lo[a] <= lo[a] && p.Hi[a] >= hi[a];
			}
			const unsigned which = __ballot_sync(0xFFFFFFFFu, mine);
			return which ? (int)own.x + __ffs((int)which) - 1 : -1;
		}

		// One warp per part, drawn from a counter, those with long programs first (a single one
		// of several hundred records keeps a warp busy longer than the whole launch otherwise
		// takes).  Bound by issue and by the latency of the one pass over the cell's program.
		template<typename L>
		__global__ void __launch_bounds__(kThreads, kBuildCtasPerSm) BuildPartTapesKernel(DeviceProgram prog, L lat, BrickTapes tapes,
			BrickTapes above, int spill_pairs)
		{
			extern __shared__ __align__(16) uint8_t shared[];
			const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
			using Scratch = TapeScratch<L::kShortest ? 2 * kTapeCap : kTapeCap>;
			Scratch& ts = reinterpret_cast<Scratch*>(shared)[warp];
			const TapeLists lists{ ts.Value, ts.Material, ts.Start, L::kShortest ? 2 * kTapeCap : kTapeCap };
			float2* spill = reinterpret_cast<float2*>(shared + kWarps * sizeof(Scratch)) + warp * spill_pairs * 32 + lane;
			const uint32_t n = min(tapes.Counters[0], tapes.PartCapacity), longs = min(tapes.Counters[4], kLongParts);
			const float rootClip = __ldg(&prog.Nodes[0].ClipRadius);
			const PairUnits units = LoadPairUnits();
			const float4* code = prog.Code;
			for (;;)
			{
				uint32_t item = 0;
				if (lane == 0) item = atomicAdd(tapes.Counters + 1, 1u);
				item = __shfl_sync(0xFFFFFFFFu, item, 0);
				if (item >= n + longs) break;
				const uint32_t slot = item < longs ? tapes.Long[item] : item - longs;
				BrickPart& part = tapes.Parts[slot];
				const int cell = part.Cell;
				const uint32_t box = part.Box;
				if (cell < 0 || (item >= longs && (box & kBoxLong))) continue;
				if (__ldg(&prog.Nodes[cell].ClipRadius) < 0.0f) continue;    // not 1-Lipschitz: no tape
				const int base = part.Distance, quads = part.Surface - base;
				if (quads < L::kShortest) continue;
				TapeCounts counts;
				float reach;
				__syncwarp();       // the previous part's lists have been copied out
				bool ok;
				{
					const float lo[3] = { part.Lo[0], part.Lo[1], part.Lo[2] }, hi[3] = { part.Hi[0], part.Hi[1], part.Hi[2] };
					// 4 x 4 x 4 sub-boxes: x and y from the lane, z from the lane and the pair.
					const float wx = 0.25f * (hi[0] - lo[0]), wy = 0.25f * (hi[1] - lo[1]), wz = 0.25f * (hi[2] - lo[2]);
					const float cx = lo[0] + ((float)(lane & 3) + 0.5f) * wx;
					const float cy = lo[1] + ((float)((lane >> 2) & 3) + 0.5f) * wy;
					const float cz = lo[2] + ((float)(lane >> 4) + 0.5f) * wz;
					const float r = 0.5f * sqrtf(wx * wx + wy * wy + wz * wz) + kTetraReach;
					reach = TapeReach(r, fmaxf(fabsf(lo[0]), fabsf(hi[0])), fmaxf(fabsf(lo[1]), fabsf(hi[1])),
						fmaxf(fabsf(lo[2]), fabsf(hi[2])), rootClip);
					int around = -1;
					if constexpr (L::kAbove)
						if (above.Bricks && quads >= kAboveQuads) around = PartAround(above, above.Bricks[lat.Above(part.Brick)], cell, lo, hi);
					if (L::kAbove && around >= 0)
					{
						const BrickPart& p = above.Parts[around];
						DistanceEventSource src;
						src.Open(code + base, above.Events + p.Material, (int)(p.Counts >> 16), ts.Window, ts.Heads);
						ok = BuildTape<true>(src, make_float2(cx, cx), make_float2(cy, cy), make_float2(cz, cz + 2.0f * wz), reach, prog.Slack, prog.Widths, units,
							spill, 32, lists, counts);
					}
					else
					{
						DistanceSource src;
						src.In.Open(code + base, quads, ts.Window);
						ok = quads <= 0xFFF0 && BuildTape<true>(src, make_float2(cx, cx), make_float2(cy, cy), make_float2(cz, cz + 2.0f * wz), reach,
							prog.Slack, prog.Widths, units, spill, 32, lists, counts);
					}
				}
				if (!ok) continue;
				// |f| beyond a ball's radius (half the reach covers it) and Keep() at every centre.
				const float far = 0.5f * reach + lat.Keep();
				const bool above = __all_sync(0xFFFFFFFFu, counts.Distance.x > far + counts.Error.x && counts.Distance.y > far + counts.Error.y);
				const bool below = __all_sync(0xFFFFFFFFu, counts.Distance.x < -far - counts.Error.x && counts.Distance.y < -far - counts.Error.y);
				if (lane == 0 && (above || below)) part.Box = box | (above ? kBoxPositive : kBoxNegative);
				const int material = counts.Same ? 0 : counts.Material;
				uint32_t at = 0;
				if (lane == 0) at = atomicAdd(tapes.Counters + 2, (uint32_t)(counts.Value + material));
				at = __shfl_sync(0xFFFFFFFFu, at, 0);
				if (at > tapes.EventCapacity || tapes.EventCapacity - at < (uint32_t)(counts.Value + material)) continue;
				for (int i = lane; i < counts.Value; i += 32) tapes.Events[at + i] = ts.Value[i];
				for (int i = lane; i < material; i += 32) tapes.Events[at + counts.Value + i] = ts.Material[i];
				if (lane == 0)
				{
					part.Value = at;
					part.First = ts.Value[0];
					part.Material = counts.Same ? at : at + (uint32_t)counts.Value;
					part.Counts = (uint32_t)counts.Value |
						((prog.Form & kFormPainted) || L::kShortest ? (uint32_t)(counts.Same ? counts.Value : counts.Material) << 16 : kNoTape << 16);
				}
			}
		}

		// n / d for n < 4096 and 1 <= d <= 16 as a product and a shift, from over = OverSixteenBits(d):
		// over exceeds 65536 / d by less than 1, n over / 65536 exceeds n / d by less than 1 / 16.
		__device__ __forceinline__ uint32_t OverSixteenBits(int d) { return 65535u / (uint32_t)d + 1u; }
		__device__ __forceinline__ int SmallDivide(int n, uint32_t over) { return (int)(((uint32_t)n * over) >> 16); }

		// The distances of one brick's points, by a warp: its parts in 64-point passes (a part's
		// points numbered x fastest, two per lane, all lanes on one tape); the warp calls
		// visit(at, value, live) with each lane's point, at = x + Box (y + Box z) in the brick.  `axis`:
		// the points' coordinates per axis; levels [lowest, highest] only.  SkipFar: parts that stay
		// beyond the lattice's Keep() are left out.
		template<bool SkipFar, int Box = kBox, typename Visit>
		__device__ __forceinline__ void BrickPoints(const DeviceProgram& prog, const BrickTapes& tapes, uint2 own, const int (&extent)[3],
			const float (*axis)[Box], const PairUnits& units, float2* spill, Visit visit, int lowest = 0, int highest = Box - 1)
		{
			constexpr int kShift = Box == 16 ? 4 : 3;
			static_assert(Box == 1 << kShift, "bricks of 8 or 16 points an axis");
			const float4* code = prog.Code;
			auto load = [&](int q) { return __ldg(code + q); };
			const int lane = (int)(threadIdx.x & 31);
			const bool loose = own.y == 0u;       // no parts: every point descends
			const int partCount = loose ? 1 : (int)own.y;
			for (int p = 0; p < partCount; ++p)
			{
				uint32_t span = PackBox(0, extent[0], 0, extent[1], 0, extent[2]), tape = 0, events = kNoTape;
				int base = 0;
				if (!loose)
				{
					const uint4 q = __ldg(reinterpret_cast<const uint4*>(tapes.Parts + own.x + p));
					base = __ldg(&tapes.Parts[own.x + p].Distance);
					span = q.y;
					tape = q.z;
					events = q.w & 0xFFFFu;
				}
				if (SkipFar && (span & (kBoxPositive | kBoxNegative))) continue;
				const int x0 = (int)(span & 15u), y0 = (int)((span >> 8) & 15u), z0 = max((int)((span >> 16) & 15u), lowest);
				const int nx = (int)((span >> 4) & 15u) - x0 + 1, ny = (int)((span >> 12) & 15u) - y0 + 1;
				const int nz = min((int)((span >> 20) & 15u), highest) - z0 + 1;
				const int points = nx * ny * nz;
				const uint32_t overX = OverSixteenBits(nx), overY = OverSixteenBits(ny);
				const uint2* ev = tapes.Events + tape;
				for (int first = 0; first < points; first += 64)
				{
					float2 px[1], py[1], pz[1], d[1];
					int at[2];
#pragma unroll
					for (int k = 0; k < 2; ++k)
					{
						const int t = min(first + lane + 32 * k, points - 1);
						const int r = SmallDivide(t, overX);
						const int z = SmallDivide(r, overY);
						at[k] = x0 + (t - r * nx) + ((y0 + (r - z * ny)) << kShift) + ((z0 + z) << (2 * kShift));
						const float x = axis[0][at[k] & (Box - 1)], y = axis[1][(at[k] >> kShift) & (Box - 1)], zz = axis[2][at[k] >> (2 * kShift)];
						if (k & 1) { px[0].y = x; py[0].y = y; pz[0].y = zz; }
						else { px[0].x = x; py[0].x = y; pz[0].x = zz; }
					}
					if (events != kNoTape)
						RunTapePairs<1, false>(load, base, [&](uint32_t e) { return __ldg(ev + e); }, events, px, py, pz, units, d, spill,
							kThreads);
					else
					{
						const int ca = loose ? __ldg(&prog.Nodes[DescendOctree(prog.Nodes, px[0].x, py[0].x, pz[0].x)].DistanceCode) : base;
						const int cb = loose ? __ldg(&prog.Nodes[DescendOctree(prog.Nodes, px[0].y, py[0].y, pz[0].y)].DistanceCode) : base;
						d[0] = RunWholePair(code, ca, px[0], py[0], pz[0], spill, kThreads);
						if (cb != ca) d[0].y = RunWholePair(code, cb, px[0], py[0], pz[0], spill, kThreads).y;
					}
#pragma unroll
					for (int k = 0; k < 2; ++k) visit(at[k], (k & 1) ? d[0].y : d[0].x, first + lane + 32 * k < points);
				}
			}
		}

		// What a point runs: its part's lists over its cell's surface and distance programs.
		struct PointRun
		{
			int Cell;
			int Surface, Distance;          // first quads
			uint32_t Value, Material;       // first events
			uint32_t Events, Walk;          // events of the two lists (kNoTape: the whole program)
			uint2 First;                    // the first list's first event
			float Lo[3], Hi[3];             // the points known to run the same
		};

		__device__ __forceinline__ bool InRun(const PointRun& run, Vec3 p)
		{
			return p.x >= run.Lo[0] && p.x <= run.Hi[0] && p.y >= run.Lo[1] && p.y <= run.Hi[1] && p.z >= run.Lo[2] && p.z <= run.Hi[2];
		}

		// Looks for point p among the parts of a brick.
		__device__ __forceinline__ bool FindPart(const BrickTapes& tapes, uint2 own, Vec3 p, PointRun& run)
		{
			for (uint32_t q = 0; q < own.y; ++q)
			{
				const uint4* part = reinterpret_cast<const uint4*>(tapes.Parts + own.x + q);
				// The whole part at once: a march is a chain of such loads.
				const uint4 c = __ldg(part), d = __ldg(part + 1), a = __ldg(part + 2), b = __ldg(part + 3);
				run.Lo[0] = __uint_as_float(a.x); run.Lo[1] = __uint_as_float(a.y); run.Lo[2] = __uint_as_float(a.z);
				run.Hi[0] = __uint_as_float(a.w); run.Hi[1] = __uint_as_float(b.x); run.Hi[2] = __uint_as_float(b.y);
				if (!InRun(run, p)) continue;
				run.Cell = (int)c.x;
				run.Value = c.z;
				run.Events = c.w & 0xFFFFu;
				run.Walk = c.w >> 16;
				run.Distance = (int)d.x;
				run.Surface = (int)d.y;
				run.Material = d.z;
				run.First = make_uint2(b.z, b.w);
				return true;
			}
			return false;
		}

		// A point that is in no part: its cell's whole programs, and no other point with it.
		__device__ __forceinline__ void RunWhole(const DeviceProgram& prog, Vec3 p, PointRun& run)
		{
			const int cell = DescendOctree(prog.Nodes, p.x, p.y, p.z);
			run.Cell = cell;
			run.Surface = __ldg(&prog.Nodes[cell].SurfaceCode);
			run.Distance = __ldg(&prog.Nodes[cell].DistanceCode);
			run.Events = run.Walk = kNoTape;
			run.Value = run.Material = 0;
			run.Lo[0] = 1.0f; run.Hi[0] = 0.0f;
		}

		// SDFNode::Gradient at p (the four points as two pairs) and, with Distance, the cell's
		// distance program there.  `spill`: this thread's column, Stride
		// pairs apart.
		template<bool Distance, int Stride = kThreads>
		__device__ __forceinline__ Vec3 RunGradient(const DeviceProgram& prog, const BrickTapes& tapes, const PointRun& run, Vec3 p,
			const PairUnits& units, float2* spill, bool wanted, float& distance)
		{
			const float4* code = prog.Code;
			auto load = [&](int q) { return __ldg(code + q); };
			const uint2* ev = tapes.Events + run.Value;
			auto event = [&](uint32_t e) { return __ldg(ev + e); };
			const bool plain = (prog.Form & kFormPlain) != 0;
			float2 d[2];
#pragma unroll 1
			for (int q = 0; q < (Distance && wanted ? 3 : 2); ++q)
			{
				const bool surface = !Distance || q < 2;
				const Vec3 a = surface ? TetraPoint(p, 2 * q) : p, b = surface ? TetraPoint(p, 2 * q + 1) : p;
				const float2 px[1] = { make_float2(a.x, b.x) }, py[1] = { make_float2(a.y, b.y) }, pz[1] = { make_float2(a.z, b.z) };
				float2 r[1];
				if (run.Events != kNoTape && (plain || !surface))
				{
					if constexpr (Distance)
						r[0] = RunEitherTapePair(surface, load, surface ? run.Surface : run.Distance, event, run.Events, px[0], py[0], pz[0], units, spill,
							Stride);
					else RunSurfaceTapePairs<1>(load, run.Surface, event, run.Events, px, py, pz, units, r, spill, Stride);
				}
				else if (surface) r[0] = RunWholeSurfacePair(code, run.Surface, px[0], py[0], pz[0], spill, Stride);
				else r[0] = RunWholePair(code, run.Distance, px[0], py[0], pz[0], spill, Stride);
				if (q == 0) d[0] = r[0]; else if (q == 1) d[1] = r[0]; else distance = r[0].x;
			}
			float e[5] = { d[0].x, d[0].y, d[1].x, d[1].y, 0.0f };
			const float h = 0.0001f;
			const Vec3 xyy(h, -h, -h), yyx(-h, -h, h), yxy(-h, h, -h), xxx(h, h, h);
			Vec3 sum = xyy * e[0];
			sum = sum + yyx * e[1];
			sum = sum + yxy * e[2];
			sum = sum + xxx * e[3];
			if ((sum.x * sum.x + sum.y * sum.y) + sum.z * sum.z == 0.0f)
				e[4] = RunWholeSurfacePair(code, run.Surface, make_float2(p.x, p.x), make_float2(p.y, p.y), make_float2(p.z, p.z), spill, Stride).x;
			return GradientOf(e);
		}

		// The vertex's colour bytes (GetMaterial), white where it has no material.
		template<int Stride = kThreads>
		__device__ __forceinline__ uchar4 RunColor(const DeviceProgram& prog, const BrickTapes& tapes, const PointRun& run, Vec3 p,
			const PairUnits& units, float2* spill)
		{
			const float4* code = prog.Code;
			// The walk's operands in the first halves of this thread's pairs: other threads of the
			// block may still be in their gradients.
			float* walk = reinterpret_cast<float*>(spill);
			int m;
			// The lists name surface records by the order of the distance program's: not with stencils.
			if (run.Walk != kNoTape && (prog.Form & kFormPlain))
			{
				const uint2* ev = tapes.Events + run.Material;
				m = RunMaterialTape([&](int q) { return __ldg(code + q); }, run.Surface, [&](uint32_t q) { return __ldg(ev + q); }, run.Walk, p,
					units, walk, 2 * Stride);
			}
			else m = RunWholeMaterial(code, run.Surface, p, walk, 2 * Stride);
			return m >= 0 ? prog.Colors[m] : make_uchar4(255, 255, 255, 255);
		}

		// Pairs of the operand stack below its top, for `pairs` pairs of points a thread.
		inline size_t SpillPairs(const DeviceProgram& prog, int pairs)
		{
			return (size_t)(prog.MaxStack > 1 ? prog.MaxStack - 1 : 1) * pairs;
		}

		// Parts and tapes of the listed bricks of a lattice (list and count null: of all bricks).
		template<typename L>
		inline cudaError_t LaunchParts(const DeviceProgram& prog, const L& lat, const uint32_t* list, const uint32_t* count, const uint32_t* tops,
			const BrickTapes& tapes, int sms, cudaStream_t stream, const BrickTapes& above = BrickTapes{})
		{
			cudaError_t e = cudaMemsetAsync(tapes.Counters, 0, kBrickTapeCounters * sizeof(uint32_t), stream);
			if (e != cudaSuccess) return e;
			const int64_t bricks = (int64_t)lat.Bricks(0) * lat.Bricks(1) * lat.Bricks(2);
			const int64_t blocks = (bricks * 8 + kThreads - 1) / kThreads, most = (int64_t)sms * kPartCtasPerSm;
			BrickPartsKernel<L><<<(unsigned)(blocks < most ? blocks : most), kThreads, 0, stream>>>(prog, lat, list, count, tops, tapes);
			e = cudaGetLastError();
			if (e != cudaSuccess || !(prog.Form & kFormPrunable)) return e;
			const size_t pairs = SpillPairs(prog, 1);
			const size_t smem = kWarps * (sizeof(TapeScratch<L::kShortest ? 2 * kTapeCap : kTapeCap>) + pairs * 32 * sizeof(float2));
			if (smem > 48 * 1024)
			{
				e = cudaFuncSetAttribute(BuildPartTapesKernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
				if (e != cudaSuccess) return e;
			}
			BuildPartTapesKernel<L><<<sms * kBuildCtasPerSm, kThreads, smem, stream>>>(prog, lat, tapes, above, (int)pairs);
			return cudaGetLastError();
		}
	}
}
