// Brick evaluation through shortened programs (tg_tape.cuh), for bricks of 7^3 cells.
//
// A kept brick's corner points fall in one octree cell or, where it straddles pivots, in a
// few: its parts are the boxes of points that share one cell (BrickPartsKernel).  Each part
// gets a tape of its cell's program (BuildPartTapesKernel, one pass of the program at 64
// points by a warp), and the part's points, then the normals and colours of the vertices in
// it, run the tape: in a 512^3 export of a 256-primitive tree the cells' programs hold some
// tens of brushes and a part's tape a few.
#include "tg_device.cuh"
#include "tg_kernels.hpp"
#include "tg_surface.cuh"
#include "tg_cull.cuh"
#include "tg_tape.cuh"
#include "tg_cellpass.cuh"

namespace tg
{
	namespace
	{
		constexpr int kThreads = 128;
		constexpr int kWarps = kThreads / 32;
		constexpr int kPartCtasPerSm = 12;
		constexpr int kBuildCtasPerSm = 8;
		constexpr int kEvalCtasPerSm = 8;
		constexpr int kBox = kTiledBox;
		constexpr int kLongQuads = 96;      // programs from this long are built first

		__device__ __forceinline__ uint32_t PackBox(int x0, int x1, int y0, int y1, int z0, int z1)
		{
			return (uint32_t)(x0 | (x1 << 4) | (y0 << 8) | (y1 << 12) | (z0 << 16) | (z1 << 20));
		}

		constexpr uint32_t kBoxBits = 0xFFFFFFu;
		constexpr uint32_t kBoxLong = 0x80000000u;     // the part is in the list of long ones
		constexpr uint32_t kBoxPositive = 0x40000000u; // the distance keeps this sign over the part
		constexpr uint32_t kBoxNegative = 0x20000000u;

		// Last index in [lo, hi] whose coordinate is not above the pivot (lo - 1: none).
		__device__ __forceinline__ int LastAtMost(float origin, float step, int first, int lo, int hi, float pivot)
		{
			int i = lo - 1;
			while (i < hi && !(LatticeCoord(origin, first + i + 1, step) > pivot)) ++i;
			return i;
		}

		__device__ __forceinline__ void PutPart(const DeviceProgram& prog, const BrickTapes& tapes, uint32_t slot, int cell, uint32_t b, uint32_t box)
		{
			BrickPart out;
			out.Cell = cell;
			out.Box = box;
			out.Value = out.Material = 0;
			out.Counts = kNoTape | (kNoTape << 16);
			out.Distance = out.Surface = 0;
			out.Brick = b;
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
			}
			const uint4* from = reinterpret_cast<const uint4*>(&out);
			uint4* to = reinterpret_cast<uint4*>(tapes.Parts + slot);
			to[0] = from[0];
			to[1] = from[1];
		}

		// The parts of a brick of any size against the cells, by one thread: its box of corner
		// points is split at the pivots it straddles until each piece is in one cell.
		__device__ __noinline__ void SplitBrick(const DeviceProgram& prog, const GridSpec& g, const BrickTapes& tapes, uint32_t b, int i0, int j0,
			int k0, int top, uint32_t whole)
		{
			constexpr int kStack = 24, kMost = 24;
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
				const int cut[3] = { LastAtMost(g.X0, g.DX, i0, lo[0], hi[0], a.x), LastAtMost(g.Y0, g.DY, j0, lo[1], hi[1], a.y),
					LastAtMost(g.Z0, g.DZ, k0, lo[2], hi[2], a.z) };
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
				PutPart(prog, tapes, first + (uint32_t)p, fits ? (int)found[p].x : -1, b, found[p].y);
		}

		// The parts of each kept brick.  Where cells are larger than the brick (fine grids: most
		// bricks), every part holds a corner of it: eight threads per brick each descend one
		// corner, cutting the brick's index ranges at the pivots passed (DescendOctree's rule,
		// `p > pivot`, on whole ranges), and a part is emitted by the lowest corner in it.  A
		// brick that this does not cover is split by SplitBrick; one that has no room gets no
		// parts, and its points then descend one by one.  Latency-bound: the descents are chains
		// of two loads a level.
		__global__ void __launch_bounds__(kThreads) BrickPartsKernel(DeviceProgram prog, GridSpec g, BrickGrid bg, const uint32_t* __restrict__ list,
			const uint32_t* __restrict__ count, const uint32_t* __restrict__ tops, BrickTapes tapes)
		{
			const uint32_t n = *count;
			const int lane = (int)(threadIdx.x & 31), corner = lane & 7;
			for (uint32_t base = (blockIdx.x * kWarps + (threadIdx.x >> 5)) * 4u; base < n; base += gridDim.x * kWarps * 4u)
			{
				const uint32_t item = base + (uint32_t)(lane >> 3);
				const bool live = item < n;
				const uint32_t b = live ? __ldg(list + item) : 0u;
				const int bx = (int)(b % (uint32_t)bg.NBX), by = (int)((b / (uint32_t)bg.NBX) % (uint32_t)bg.NBY);
				const int bz = (int)(b / ((uint32_t)bg.NBX * (uint32_t)bg.NBY));
				const int i0 = bx * bg.B, j0 = by * bg.B, k0 = bz * bg.B;
				const int ex = min(bg.B, g.NX - 1 - i0), ey = min(bg.B, g.NY - 1 - j0), ez = min(bg.B, g.NZ - 1 - k0);
				int top = 0, cell = -1;
				int x0 = 0, x1 = ex, y0 = 0, y1 = ey, z0 = 0, z1 = ez;
				bool emit = false;
				if (live)
				{
					const uint32_t packed = tops ? __ldg(tops + b) : BrickTop(prog, g, i0, i0 + ex, j0, j0 + ey, k0, k0 + ez);
					cell = top = (int)(packed & 0x7FFFFFFFu);
					if (packed >> 31) emit = corner == 0;
					else
					{
						const float x = LatticeCoord(g.X0, i0 + ((corner & 1) ? ex : 0), g.DX);
						const float y = LatticeCoord(g.Y0, j0 + ((corner & 2) ? ey : 0), g.DY);
						const float z = LatticeCoord(g.Z0, k0 + ((corner & 4) ? ez : 0), g.DZ);
						for (int guard = 0; guard < 64; ++guard)
						{
							const float4 a = __ldg(reinterpret_cast<const float4*>(prog.Nodes + cell));
							if (__float_as_int(a.w) & kNodeTerminus) break;
							const bool hx = x > a.x, hy = y > a.y, hz = z > a.z;
							const int child = __ldg(&prog.Nodes[cell].Child[(hx ? 1 : 0) | (hy ? 2 : 0) | (hz ? 4 : 0)]);
							const int cx = LastAtMost(g.X0, g.DX, i0, x0, x1, a.x), cy = LastAtMost(g.Y0, g.DY, j0, y0, y1, a.y);
							const int cz = LastAtMost(g.Z0, g.DZ, k0, z0, z1, a.z);
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
					if (at < room) PutPart(prog, tapes, first + at, fits ? cell : -1, b, PackBox(x0, x1, y0, y1, z0, z1));
				}
				if (live && corner == 0)
				{
					if (all) tapes.Bricks[b] = make_uint2(first, fits ? parts : 0u);
					else SplitBrick(prog, g, tapes, b, i0, j0, k0, top, PackBox(0, ex, 0, ey, 0, ez));
				}
			}
		}

		// A warp's scratch while it builds a part's tape.
		struct TapeScratch
		{
			uint2 Value[kTapeCap], Material[kTapeCap];
			uint2 Start[kMaxStack + 2];
			float4 Window[64];
		};

		// One warp per part, drawn from a counter, those with long programs first (a single one
		// of several hundred records keeps a warp busy longer than the whole launch otherwise
		// takes).  Bound by issue and by the latency of the one pass over the cell's program.
		__global__ void __launch_bounds__(kThreads, kBuildCtasPerSm) BuildPartTapesKernel(DeviceProgram prog, GridSpec g, BrickGrid bg,
			BrickTapes tapes, int spill_pairs)
		{
			extern __shared__ __align__(16) uint8_t shared[];
			const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
			TapeScratch& ts = reinterpret_cast<TapeScratch*>(shared)[warp];
			const TapeLists lists{ ts.Value, ts.Material, ts.Start, kTapeCap };
			float2* spill = reinterpret_cast<float2*>(shared + kWarps * sizeof(TapeScratch)) + warp * spill_pairs * 32 + lane;
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
				const int base = part.Distance;
				TapeCounts counts;
				__syncwarp();       // the previous part's lists have been copied out
				bool ok;
				{
					float lo[3], hi[3];
					PartRegion(g, bg, part.Brick, box, lo, hi);
					// 4 x 4 x 4 sub-boxes: x and y from the lane, z from the lane and the pair.
					const float wx = 0.25f * (hi[0] - lo[0]), wy = 0.25f * (hi[1] - lo[1]), wz = 0.25f * (hi[2] - lo[2]);
					const float cx = lo[0] + ((float)(lane & 3) + 0.5f) * wx;
					const float cy = lo[1] + ((float)((lane >> 2) & 3) + 0.5f) * wy;
					const float cz = lo[2] + ((float)(lane >> 4) + 0.5f) * wz;
					const float r = 0.5f * sqrtf(wx * wx + wy * wy + wz * wz) + kTetraReach;
					const float reach = TapeReach(r, fmaxf(fabsf(lo[0]), fabsf(hi[0])), fmaxf(fabsf(lo[1]), fabsf(hi[1])),
						fmaxf(fabsf(lo[2]), fabsf(hi[2])), rootClip);
					DistanceSource src;
					const int quads = part.Surface - base;
					src.In.Open(code + base, quads, ts.Window);
					ok = quads <= 0xFFF0 && BuildTape<true>(src, make_float2(cx, cx), make_float2(cy, cy), make_float2(cz, cz + 2.0f * wz), reach,
						units, spill, 32, lists, counts);
				}
				if (!ok) continue;
				if (lane == 0 && counts.Sign) part.Box = box | (counts.Sign > 0 ? kBoxPositive : kBoxNegative);
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
					part.Material = counts.Same ? at : at + (uint32_t)counts.Value;
					part.Counts = (uint32_t)counts.Value |
						((prog.Form & kFormPainted) ? (uint32_t)(counts.Same ? counts.Value : counts.Material) << 16 : kNoTape << 16);
				}
			}
		}

		// n / d for n < 512 and 1 <= d <= 8, as a product and a shift.
		__device__ __forceinline__ int SmallDivide(int n, int d)
		{
			constexpr uint32_t kOver[9] = { 0, 65536, 32768, 21846, 16384, 13108, 10923, 9363, 8192 };
			uint32_t over = kOver[1];
#pragma unroll
			for (int q = 2; q <= 8; ++q) over = d == q ? kOver[q] : over;
			return (int)(((uint32_t)n * over) >> 16);
		}

		// The evaluation with the cell pass folded in: a warp draws a brick from a counter and
		// takes its parts in 32 NP x 2-point passes (a part's points numbered x fastest, all
		// lanes on one tape), writing the lattice and the brick's 8^3 corner box in shared
		// memory; it then flags and lists the brick's active cells from the signs of that box:
		// eight corners of a row make a byte, four rows' bytes the seven cells between them.
		template<int NP>
		__global__ void __launch_bounds__(kThreads, kEvalCtasPerSm) EvalBrickTapesKernel(DeviceProgram prog, GridSpec g, BrickGrid bg,
			const uint32_t* __restrict__ list, const uint32_t* __restrict__ count, BrickTapes tapes, float* __restrict__ lattice,
			uint32_t* __restrict__ words, uint32_t* __restrict__ cells, uint32_t* __restrict__ cell_count)
		{
			extern __shared__ __align__(16) float2 spill2[];
			__shared__ __align__(16) float boxes[kWarps][kBox * kBox * kBox];
			__shared__ float axes[kWarps][3][kBox];
			const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
			float* box = boxes[warp];
			float (*axis)[kBox] = axes[warp];
			const float4* code = prog.Code;
			auto load = [&](int q) { return __ldg(code + q); };
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
				const uint32_t row = b / (uint32_t)bg.NBX, bz = row / (uint32_t)bg.NBY;
				const int i0 = (int)(b - row * (uint32_t)bg.NBX) * bg.B, j0 = (int)(row - bz * (uint32_t)bg.NBY) * bg.B, k0 = (int)bz * bg.B;
				const int ex = min(bg.B, g.NX - 1 - i0), ey = min(bg.B, g.NY - 1 - j0), ez = min(bg.B, g.NZ - 1 - k0);
				// All parts of one sign: the brick has no active cell, and nobody reads its values.
				uint32_t sign = kBoxPositive | kBoxNegative;
				for (uint32_t p = 0; p < own.y; ++p) sign &= __ldg(&tapes.Parts[own.x + p].Box);
				if (own.y && sign) continue;
				float* corner = lattice + ((int64_t)k0 * g.NY + j0) * g.NX + i0;
				__syncwarp();       // the previous brick is done with the box and the axes
				if (lane < 24)
				{
					const int a = lane >> 3, q = lane & 7;
					axis[a][q] = a == 0 ? LatticeCoord(g.X0, i0 + q, g.DX) : a == 1 ? LatticeCoord(g.Y0, j0 + q, g.DY) : LatticeCoord(g.Z0, k0 + q, g.DZ);
				}
				__syncwarp();
				const bool loose = own.y == 0u;       // no parts: every point descends
				const int partCount = loose ? 1 : (int)own.y;
				for (int p = 0; p < partCount; ++p)
				{
					uint32_t span = PackBox(0, ex, 0, ey, 0, ez), tape = 0, events = kNoTape;
					int base = 0;
					if (!loose)
					{
						const uint4 q = __ldg(reinterpret_cast<const uint4*>(tapes.Parts + own.x + p));
						base = __ldg(&tapes.Parts[own.x + p].Distance);
						span = q.y;
						tape = q.z;
						events = q.w & 0xFFFFu;
					}
					const int x0 = (int)(span & 15u), y0 = (int)((span >> 8) & 15u), z0 = (int)((span >> 16) & 15u);
					const int nx = (int)((span >> 4) & 15u) - x0 + 1, ny = (int)((span >> 12) & 15u) - y0 + 1, nz = (int)((span >> 20) & 15u) - z0 + 1;
					const int points = nx * ny * nz;
					const uint2* ev = tapes.Events + tape;
					for (int first = 0; first < points; first += 64 * NP)
					{
						float2 px[NP], py[NP], pz[NP], d[NP];
						int at[2 * NP];
#pragma unroll
						for (int k = 0; k < 2 * NP; ++k)
						{
							const int t = min(first + lane + 32 * k, points - 1);
							const int r = SmallDivide(t, nx);
							const int z = SmallDivide(r, ny);
							at[k] = x0 + (t - r * nx) + ((y0 + (r - z * ny)) << 3) + ((z0 + z) << 6);
							const float x = axis[0][at[k] & 7], y = axis[1][(at[k] >> 3) & 7], zz = axis[2][at[k] >> 6];
							if (k & 1) { px[k / 2].y = x; py[k / 2].y = y; pz[k / 2].y = zz; }
							else { px[k / 2].x = x; py[k / 2].x = y; pz[k / 2].x = zz; }
						}
						if (events != kNoTape)
							RunTapePairs<NP>(load, base, [&](uint32_t e) { return __ldg(ev + e); }, events, px, py, pz, units, d, spill2 + threadIdx.x,
								kThreads);
						else
						{
#pragma unroll
							for (int j = 0; j < NP; ++j)
							{
								const int ca = loose ? __ldg(&prog.Nodes[DescendOctree(prog.Nodes, px[j].x, py[j].x, pz[j].x)].DistanceCode) : base;
								const int cb = loose ? __ldg(&prog.Nodes[DescendOctree(prog.Nodes, px[j].y, py[j].y, pz[j].y)].DistanceCode) : base;
								d[j] = RunWholePair(code, ca, px[j], py[j], pz[j], spill2 + threadIdx.x, kThreads);
								if (cb != ca) d[j].y = RunWholePair(code, cb, px[j], py[j], pz[j], spill2 + threadIdx.x, kThreads).y;
							}
						}
#pragma unroll
						for (int k = 0; k < 2 * NP; ++k)
						{
							if (first + lane + 32 * k < points)
							{
								const float v = (k & 1) ? d[k / 2].y : d[k / 2].x;
								corner[(int64_t)(at[k] >> 6) * plane + ((at[k] >> 3) & 7) * g.NX + (at[k] & 7)] = v;
								box[at[k]] = v;
							}
						}
					}
				}
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
				const uint32_t mine = (uint32_t)(__popc(active[0]) + __popc(active[1]));
				uint32_t upTo = mine;
#pragma unroll
				for (int o = 1; o < 32; o <<= 1)
				{
					const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, upTo, o);
					if (lane >= o) upTo += v;
				}
				uint32_t start = 0;
				if (lane == 31 && upTo) start = atomicAdd(cell_count, upTo);
				uint32_t to = __shfl_sync(0xFFFFFFFFu, start, 31) + upTo - mine;
				const int64_t sx = g.NX - 1, sy = g.NY - 1;
#pragma unroll
				for (int q = 0; q < 2; ++q)
				{
					uint32_t bits = active[q];
					if (!bits) continue;
					const int64_t c = i0 + sx * ((j0 + y + q) + sy * (k0 + z));
					const int shift = (int)(c & 31);
					atomicOr(words + (c >> 5), bits << shift);
					if (shift > 32 - kBox && (bits >> (32 - shift))) atomicOr(words + (c >> 5) + 1, bits >> (32 - shift));
					while (bits)
					{
						const int x = __ffs((int)bits) - 1;
						bits &= bits - 1u;
						cells[to++] = (uint32_t)(c + x);
					}
				}
			}
		}

		// Normals and colours of the export's vertices, a thread per vertex in the active-cell
		// list's order (cells grouped by brick, so a warp's vertices mostly run one tape): the
		// gradient's four points as two pairs through one pass over the part's surface records,
		// then the material walk.
		__global__ void __launch_bounds__(kThreads, 8) BrickAttributesKernel(DeviceProgram prog, GridSpec g, BrickGrid bg, BrickTapes tapes,
			const uint32_t* __restrict__ cells, const uint32_t* __restrict__ words, const uint32_t* __restrict__ word_base,
			const float* __restrict__ vertices, uint32_t n, float* __restrict__ normals, uint8_t* __restrict__ colors)
		{
			extern __shared__ __align__(16) float2 spill2[];
			const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
			if (t >= n) return;
			const uint32_t c = __ldg(cells + t);
			const uint32_t w = __ldg(words + (c >> 5)), before = __ldg(word_base + (c >> 5));
			const uint32_t sx = (uint32_t)(g.NX - 1), sy = (uint32_t)(g.NY - 1), B = (uint32_t)bg.B;
			const uint32_t row = c / sx, k = row / sy, i = c - row * sx, j = row - k * sy;
			const uint32_t b = i / B + (uint32_t)bg.NBX * (j / B + (uint32_t)bg.NBY * (k / B));
			const uint2 own = __ldg(tapes.Bricks + b);
			const uint32_t v = before + __popc(w & ((1u << (c & 31)) - 1u));
			const Vec3 p(__ldg(vertices + (int64_t)v * 3), __ldg(vertices + (int64_t)v * 3 + 1), __ldg(vertices + (int64_t)v * 3 + 2));
			const float4* code = prog.Code;
			auto load = [&](int q) { return __ldg(code + q); };
			const PairUnits units = LoadPairUnits();
			float2* spill = spill2 + threadIdx.x;
			// The vertex's part.  All points of a part's box of corners descend to its cell; a
			// vertex between two parts' boxes descends itself, to a cell of one of them.
			int surface = -1;
			uint32_t counts = kNoTape | (kNoTape << 16), value = 0, material = 0;
			for (int attempt = 0; attempt < 2 && surface < 0; ++attempt)
			{
				int cell = -1;
				if (attempt)
				{
					cell = DescendOctree(prog.Nodes, p.x, p.y, p.z);
					surface = __ldg(&prog.Nodes[cell].SurfaceCode);
				}
				for (uint32_t q = 0; q < own.y; ++q)
				{
					const BrickPart* part = tapes.Parts + own.x + q;
					const uint4 a = __ldg(reinterpret_cast<const uint4*>(part));
					float lo[3], hi[3];
					if (attempt)
					{
						if ((int)a.x != cell) continue;
						PartRegion(g, bg, b, a.y, lo, hi);
					}
					else PartCorners(g, bg, b, a.y, lo, hi);
					if (!(p.x >= lo[0] && p.x <= hi[0] && p.y >= lo[1] && p.y <= hi[1] && p.z >= lo[2] && p.z <= hi[2])) continue;
					const uint4 rest = __ldg(reinterpret_cast<const uint4*>(part) + 1);
					value = a.z;
					counts = a.w;
					surface = (int)rest.y;
					material = rest.z;
					break;
				}
			}
			float2 d[2];
			const uint32_t events = counts & 0xFFFFu, walk = counts >> 16;
			if (events != kNoTape)
			{
				const uint2* ev = tapes.Events + value;
#pragma unroll 1
				for (int q = 0; q < 2; ++q)
				{
					const Vec3 a = TetraPoint(p, 2 * q), b = TetraPoint(p, 2 * q + 1);
					const float2 px[1] = { make_float2(a.x, b.x) }, py[1] = { make_float2(a.y, b.y) }, pz[1] = { make_float2(a.z, b.z) };
					float2 r[1];
					RunSurfaceTapePairs<1>(load, surface, [&](uint32_t e) { return __ldg(ev + e); }, events, px, py, pz, units, r, spill, kThreads);
					if (q == 0) d[0] = r[0]; else d[1] = r[0];
				}
			}
			else
			{
#pragma unroll
				for (int q = 0; q < 2; ++q)
				{
					const Vec3 a = TetraPoint(p, 2 * q), b = TetraPoint(p, 2 * q + 1);
					d[q] = RunWholeSurfacePair(code, surface, make_float2(a.x, b.x), make_float2(a.y, b.y), make_float2(a.z, b.z), spill, kThreads);
				}
			}
			float e[5] = { d[0].x, d[0].y, d[1].x, d[1].y, 0.0f };
			const float h = 0.0001f;
			const Vec3 xyy(h, -h, -h), yyx(-h, -h, h), yxy(-h, h, -h), xxx(h, h, h);
			Vec3 sum = xyy * e[0];
			sum = sum + yyx * e[1];
			sum = sum + yxy * e[2];
			sum = sum + xxx * e[3];
			if ((sum.x * sum.x + sum.y * sum.y) + sum.z * sum.z == 0.0f)
				e[4] = RunWholeSurfacePair(code, surface, make_float2(p.x, p.x), make_float2(p.y, p.y), make_float2(p.z, p.z), spill, kThreads).x;
			const Vec3 normal = GradientOf(e);
			normals[(int64_t)v * 3 + 0] = normal.x;
			normals[(int64_t)v * 3 + 1] = normal.y;
			normals[(int64_t)v * 3 + 2] = normal.z;
			if (!colors) return;
			// The walk's operands in the first halves of this thread's pairs: other threads of the
			// block may still be in their gradients.
			float* walkSpill = reinterpret_cast<float*>(spill);
			int m;
			if (walk != kNoTape)
			{
				const uint2* ev = tapes.Events + material;
				m = RunMaterialTape(load, surface, [&](uint32_t q) { return __ldg(ev + q); }, walk, p, walkSpill, 2 * kThreads);
			}
			else m = RunWholeMaterial(code, surface, p, walkSpill, 2 * kThreads);
			const uchar4 color = m >= 0 ? prog.Colors[m] : make_uchar4(255, 255, 255, 255);
			colors[(int64_t)v * 3 + 0] = color.x;
			colors[(int64_t)v * 3 + 1] = color.y;
			colors[(int64_t)v * 3 + 2] = color.z;
		}

		constexpr int kEvalPairs = 1;
	}

	// Parts and events are bounded by the bricks of the grid: a fine export keeps one brick in
	// ten or twenty, with two or three parts each; a coarse one keeps more, with up to a dozen.
	// What does not fit is evaluated without (BrickPartsKernel, BuildPartTapesKernel).
	size_t BrickPartCapacity(int64_t bricks) { return (size_t)bricks / 2 + 65536; }
	size_t BrickEventCapacity(int64_t bricks) { return BrickPartCapacity(bricks) * 12; }

	// Pairs of the operand stack below its top, for `pairs` pairs of points a thread.
	static size_t SpillPairs(const DeviceProgram& prog, int pairs)
	{
		return (size_t)(prog.MaxStack > 1 ? prog.MaxStack - 1 : 1) * pairs;
	}

	cudaError_t LaunchBrickTapes(const DeviceProgram& prog, const GridSpec& g, int B, const uint32_t* list, const uint32_t* count,
		const uint32_t* tops, const BrickTapes& tapes, int sms, cudaStream_t stream)
	{
		if (B + 1 != kBox) return cudaErrorInvalidValue;
		const BrickGrid bg = MakeBrickGrid(g, B);
		cudaError_t e = cudaMemsetAsync(tapes.Counters, 0, kBrickTapeCounters * sizeof(uint32_t), stream);
		if (e != cudaSuccess) return e;
		const int64_t bricks = (int64_t)bg.NBX * bg.NBY * bg.NBZ;
		const int64_t blocks = (bricks * 8 + kThreads - 1) / kThreads, most = (int64_t)sms * kPartCtasPerSm;
		BrickPartsKernel<<<(unsigned)(blocks < most ? blocks : most), kThreads, 0, stream>>>(prog, g, bg, list, count, tops, tapes);
		e = cudaGetLastError();
		if (e != cudaSuccess || !(prog.Form & kFormPrunable)) return e;
		const size_t pairs = SpillPairs(prog, 1);
		const size_t smem = kWarps * (sizeof(TapeScratch) + pairs * 32 * sizeof(float2));
		if (smem > 48 * 1024)
		{
			e = cudaFuncSetAttribute(BuildPartTapesKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		BuildPartTapesKernel<<<sms * kBuildCtasPerSm, kThreads, smem, stream>>>(prog, g, bg, tapes, (int)pairs);
		return cudaGetLastError();
	}

	cudaError_t LaunchEvalBrickTapes(const DeviceProgram& prog, const GridSpec& g, int B, const uint32_t* list, const uint32_t* count,
		const BrickTapes& tapes, float* lattice, uint32_t* words, uint32_t* cells, uint32_t* cell_count, int sms, cudaStream_t stream)
	{
		if (B + 1 != kBox) return cudaErrorInvalidValue;
		const int64_t total = (int64_t)(g.NX - 1) * (g.NY - 1) * (g.NZ - 1);
		cudaError_t e = cudaMemsetAsync(words, 0, (size_t)((total + 31) / 32) * 4, stream);
		if (e == cudaSuccess) e = cudaMemsetAsync(cell_count, 0, sizeof(uint32_t), stream);
		if (e != cudaSuccess) return e;
		const size_t smem = SpillPairs(prog, kEvalPairs) * kThreads * sizeof(float2);
		if (smem > 39 * 1024)
		{
			e = cudaFuncSetAttribute(EvalBrickTapesKernel<kEvalPairs>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		EvalBrickTapesKernel<kEvalPairs><<<sms * kEvalCtasPerSm, kThreads, smem, stream>>>(prog, g, MakeBrickGrid(g, B), list, count, tapes, lattice,
			words, cells, cell_count);
		return cudaGetLastError();
	}

	cudaError_t LaunchBrickAttributes(const DeviceProgram& prog, const GridSpec& g, int B, const BrickTapes& tapes, const uint32_t* cells,
		const uint32_t* words, const uint32_t* word_base, const float* vertices, uint32_t vertex_count, float* normals, uint8_t* colors,
		cudaStream_t stream)
	{
		if (vertex_count == 0) return cudaSuccess;
		// The walk takes two words a level, the gradient one pair.
		const size_t smem = SpillPairs(prog, 2) * kThreads * sizeof(float2);
		if (smem > 48 * 1024)
		{
			const cudaError_t e = cudaFuncSetAttribute(BrickAttributesKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		BrickAttributesKernel<<<(vertex_count + kThreads - 1) / kThreads, kThreads, smem, stream>>>(prog, g, MakeBrickGrid(g, B), tapes, cells,
			words, word_base, vertices, vertex_count, normals, colors);
		return cudaGetLastError();
	}
}
