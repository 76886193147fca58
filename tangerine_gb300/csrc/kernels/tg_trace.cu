// Sphere tracing (SDFNode::RayMarch, tangerine/sdf_evaluator.cpp:336-353) and a
// depth / normal / colour renderer built on it.
//
// Exact form: the reference's step sequence -- every step is the whole tree's distance
// (its surface program, SDFNode::Eval order) -- so hits, travel and positions are those of
// SDFNode::RayMarch bit for bit.
//
// Octree-bounded form: outside the root cube the distance to that cube is a safe step (the
// surface lies inside it).  Inside, a point lies in the cube of the octree cell Descend
// picks, and the whole tree's distance is at least min(f_cell(q), R - |q - P|): every operand
// the cell's clip dropped exceeds R - |q - P| there (1-Lipschitz), and union, diff and the
// polynomial blends cannot fall below that bound.  The cell's distance program is a few
// brushes where the full tree is hundreds.  A hit is declared when f_cell(q) <= epsilon,
// which then holds for the whole tree too.  Shading uses the cell's surface program as
// SDFOctree::Gradient / GetMaterial do.
#include <cmath>

#include "tg_device.cuh"
#include "tg_kernels.hpp"
#include "tg_trace.cuh"
#include "tg_parts.cuh"

namespace tg
{
	namespace
	{
		constexpr int kTraceThreads = 128;
		constexpr int kTileX = 8, kTileY = 4;      // pixels of a warp

		// SDFNode::RayMarch on the whole tree.
		__device__ __forceinline__ March MarchExact(const DeviceProgram& prog, Vec3 start, Vec3 dir_in, int iterations, float epsilon,
			float* spill)
		{
			return TraceExactFrom(prog, start, Normalize(dir_in), 0.0f, iterations, epsilon, spill, kTraceThreads);
		}

		__device__ __forceinline__ March MarchBounded(const DeviceProgram& prog, Vec3 start, Vec3 dir_in, int iterations, float epsilon,
			float* spill)
		{
			const Vec3 dir = Normalize(dir_in);
			const float rootClip = fabsf(__ldg(&prog.Nodes[0].ClipRadius));
			const Vec3 root(__ldg(&prog.Nodes[0].Pivot[0]), __ldg(&prog.Nodes[0].Pivot[1]), __ldg(&prog.Nodes[0].Pivot[2]));
			const float half = rootClip * 0.57735f;               // root cube half-width
			// Leaving the root sphere along the ray ends the march: nothing lies beyond.
			const Vec3 oc = start - root;
			const float b = Dot(oc, dir);
			const float c = Dot(oc, oc) - rootClip * rootClip;
			const float disc = b * b - c;
			if (disc < 0.0f) return { false, INFINITY, start };
			const float exitTravel = -b + sqrtf(disc);
			if (exitTravel < 0.0f) return { false, INFINITY, start };
			Vec3 pos = start;
			float travel = 0.0f;
			for (int i = 0; i < iterations; ++i)
			{
				const Vec3 off = pos - root;
				const float ox = fmaxf(fabsf(off.x) - half, 0.0f), oy = fmaxf(fabsf(off.y) - half, 0.0f), oz = fmaxf(fabsf(off.z) - half, 0.0f);
				float step = sqrtf(ox * ox + oy * oy + oz * oz);
				if (!(step > epsilon))
				{
					const int cell = DescendOctree(prog.Nodes, pos.x, pos.y, pos.z);
					const float px[1] = { pos.x }, py[1] = { pos.y }, pz[1] = { pos.z };
					float f[1];
					RunDistance<1>(prog.Code, __ldg(&prog.Nodes[cell].DistanceCode), px, py, pz, f, spill, kTraceThreads);
					if (f[0] <= epsilon) return { true, travel, pos };
					const Vec3 dp = pos - Vec3(__ldg(&prog.Nodes[cell].Pivot[0]), __ldg(&prog.Nodes[cell].Pivot[1]), __ldg(&prog.Nodes[cell].Pivot[2]));
					const float room = __ldg(&prog.Nodes[cell].ClipRadius) - Length(dp);
					step = fminf(f[0], fmaxf(room, epsilon));
				}
				travel = travel + step;
				if (travel > exitTravel) break;
				pos = dir * travel + start;
			}
			return { false, INFINITY, pos };
		}

		__global__ void __launch_bounds__(kTraceThreads) RayMarchKernel(DeviceProgram prog, const float* __restrict__ origins,
			const float* __restrict__ dirs, int64_t n, int iterations, float epsilon, uint8_t* __restrict__ hit,
			float* __restrict__ travel, float* __restrict__ position)
		{
			extern __shared__ float spill[];
			const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
			if (r >= n) return;
			const March m = MarchExact(prog, Vec3(origins[r * 3], origins[r * 3 + 1], origins[r * 3 + 2]),
				Vec3(dirs[r * 3], dirs[r * 3 + 1], dirs[r * 3 + 2]), iterations, epsilon, spill + threadIdx.x);
			hit[r] = m.Hit ? 1 : 0;
			travel[r] = m.Travel;
			position[r * 3] = m.Position.x;
			position[r * 3 + 1] = m.Position.y;
			position[r * 3 + 2] = m.Position.z;
		}

		// The app's framed casts (FrameRay).
		__global__ void __launch_bounds__(kTraceThreads) RayQueryKernel(DeviceProgram prog, RayFrame f, const float* __restrict__ origins,
			const float* __restrict__ dirs, int64_t n, int iterations, float epsilon, uint8_t* __restrict__ hit,
			float* __restrict__ travel, float* __restrict__ position)
		{
			extern __shared__ float spill[];
			const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
			if (r >= n) return;
			Vec3 o(origins[r * 3], origins[r * 3 + 1], origins[r * 3 + 2]);
			Vec3 d(dirs[r * 3], dirs[r * 3 + 1], dirs[r * 3 + 2]);
			FrameRay(f, o, d);
			const March m = MarchExact(prog, o, d, iterations, epsilon, spill + threadIdx.x);
			hit[r] = m.Hit ? 1 : 0;
			travel[r] = m.Travel;
			position[r * 3] = m.Position.x;
			position[r * 3 + 1] = m.Position.y;
			position[r * 3 + 2] = m.Position.z;
		}

		// SDFNode::Eval or SDFNode::Gradient on the whole tree per point, as Lua's eval / gradient
		// and EvalTree compute them (lua_sdf.cpp:386-405): a pair of evaluations a lane, two points
		// or two of a point's four (two lanes a point), all lanes of a warp on the program's one
		// walk, read through a window in shared memory.  Bound by issue.  Calls from and to the
		// host, a thread a point (one evaluation after the other) against this: gradients of 64
		// primitives 100 000 188 / 155, 30 000 142 / 84, of 256 primitives 200 000 1177 / 825, 30 000
		// 455 / 231, of 8 primitives 1000 35 / 31; values of 256 primitives 200 000 376 / 293.  A warp
		// a CTA: with four, some SMs got a quarter more of the work than others at middling counts
		// (values of 400 primitives at 120 000 321 us by a thread a point, 356 by CTAs of four, 320 so;
		// gradients 1041, 830, 743).
		constexpr int kQueryThreads = 32;

		template<bool Gradient>
		__global__ void __launch_bounds__(kQueryThreads) PointQueryKernel(DeviceProgram prog, const float* __restrict__ points, int64_t n,
			float* __restrict__ out, int spill_pairs)
		{
			extern __shared__ __align__(16) float4 shared4[];
			const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
			float4* window = shared4 + warp * 64;
			float2* spill = reinterpret_cast<float2*>(shared4 + kQueryThreads / 32 * 64) + warp * spill_pairs * 32 + lane;
			const int64_t group = (int64_t)blockIdx.x * (kQueryThreads / 32) + warp;
			const PairUnits units = LoadPairUnits();
			const float4* code = prog.Code + prog.FullSurfaceCode;
			auto at = [&](int64_t t) { t = min(t, n - 1); return Vec3(points[t * 3], points[t * 3 + 1], points[t * 3 + 2]); };
			SurfaceSource src;
			src.In.Open(code, prog.CodeQuads - prog.FullSurfaceCode, window);
			if constexpr (!Gradient)
			{
				const int64_t t = group * 64 + lane;
				const Vec3 a = at(t), b = at(t + 32);
				const float2 d = RunSourcePair(src, make_float2(a.x, b.x), make_float2(a.y, b.y), make_float2(a.z, b.z), units, spill, 32);
				if (t < n) out[t] = d.x;
				if (t + 32 < n) out[t + 32] = d.y;
			}
			else
			{
				const int64_t t = group * 16 + (lane >> 1);
				const Vec3 p = at(t), a = TetraPoint(p, 2 * (lane & 1)), b = TetraPoint(p, 2 * (lane & 1) + 1);
				const float2 d = RunSourcePair(src, make_float2(a.x, b.x), make_float2(a.y, b.y), make_float2(a.z, b.z), units, spill, 32);
				float e[5] = { d.x, d.y, __shfl_down_sync(0xFFFFFFFFu, d.x, 1), __shfl_down_sync(0xFFFFFFFFu, d.y, 1), 0.0f };
				if (t >= n || (lane & 1)) return;
				const float h = 0.0001f;
				const Vec3 xyy(h, -h, -h), yyx(-h, -h, h), yxy(-h, h, -h), xxx(h, h, h);
				Vec3 g = xyy * e[0];
				g = g + yyx * e[1];
				g = g + yxy * e[2];
				g = g + xxx * e[3];
				if ((g.x * g.x + g.y * g.y) + g.z * g.z == 0.0f)
					e[4] = RunWholeSurfacePair(prog.Code, prog.FullSurfaceCode, make_float2(p.x, p.x), make_float2(p.y, p.y), make_float2(p.z, p.z),
						spill, 32).x;
				const Vec3 v = GradientOf(e);
				out[t * 3] = v.x;
				out[t * 3 + 1] = v.y;
				out[t * 3 + 2] = v.z;
			}
		}

		// Compiled for 10 resident CTAs per SM (48 registers instead of 56): 657 -> 667 M
		// rays/s on the 1024-primitive scene; 12 (40 registers) measured 657 again.
		__global__ void __launch_bounds__(kTraceThreads, 10) RenderKernel(DeviceProgram prog, const CameraBasis* __restrict__ cams,
			int count, int width, int height, int steps, float epsilon, bool exact, float* __restrict__ depth,
			float* __restrict__ normals, uint8_t* __restrict__ colors)
		{
			extern __shared__ float spill[];
			const int64_t pixels = (int64_t)width * height;
			const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
			if (t >= pixels * count) return;
			const int c = (int)(t / pixels);
			const int64_t pix = t % pixels;
			const int x = (int)(pix % width), y = (int)(pix / width);
			const CameraBasis& cam = cams[c];
			const float u = ((2.0f * ((float)x + 0.5f) / (float)width) - 1.0f) * cam.TanHalfFov * cam.Aspect;
			const float v = (1.0f - 2.0f * ((float)y + 0.5f) / (float)height) * cam.TanHalfFov;
			const Vec3 fwd(cam.Forward[0], cam.Forward[1], cam.Forward[2]);
			const Vec3 right(cam.Right[0], cam.Right[1], cam.Right[2]);
			const Vec3 up(cam.Up[0], cam.Up[1], cam.Up[2]);
			const Vec3 dir = (fwd + right * u) + up * v;
			const Vec3 start(cam.Position[0], cam.Position[1], cam.Position[2]);
			float* my = spill + threadIdx.x;
			const March m = exact ? MarchExact(prog, start, dir, steps, epsilon, my) : MarchBounded(prog, start, dir, steps, epsilon, my);
			depth[t] = m.Travel;
			Vec3 n(0.0f, 0.0f, 0.0f);
			uchar4 col = make_uchar4(0, 0, 0, 0);
			if (m.Hit)
			{
				const int pc = exact ? prog.FullSurfaceCode
					: __ldg(&prog.Nodes[DescendOctree(prog.Nodes, m.Position.x, m.Position.y, m.Position.z)].SurfaceCode);
				int mat = -1;
				n = TraceShade(prog, pc, m.Position, colors != nullptr, &mat, my, kTraceThreads);
				col = mat >= 0 ? prog.Colors[mat] : make_uchar4(255, 255, 255, 255);
			}
			normals[t * 3] = n.x;
			normals[t * 3 + 1] = n.y;
			normals[t * 3 + 2] = n.z;
			if (colors)
			{
				colors[t * 3] = col.x;
				colors[t * 3 + 1] = col.y;
				colors[t * 3 + 2] = col.z;
			}
		}

		// The root cube in bricks for the renderer's tapes: 8^3 points a brick at the centres of
		// the cube's (8 N)^3 cells.  The octree halves the cube, so a brick lies in one cell where
		// the cells are no smaller.
		// Level 1: bricks of 4^3 of those, for the tapes that theirs are built from: 32 768 passes of
		// programs of several hundred records took longer than the rays (2364 of 2550 us for 512
		// primitives at 2 x 300 x 200, 1811 of 5920 for 1024 at 2 x 1920 x 1080); by way of 512
		// larger bricks' tapes the images take 738 and 5011.
		template<int Level>
		struct RenderBricksOf
		{
			static constexpr int kStride = parts::kBox;
			static constexpr int kBox = parts::kBox, kMost = 24;
			static constexpr bool kOutside = true, kBetween = true, kAbove = Level == 0;
			static constexpr int kShortest = Level == 0 ? 0 : parts::kAboveQuads;
			float Origin[3];
			float Step;
			int N;
			__device__ __forceinline__ float Coord(int a, int i) const { return Origin[a] + ((float)i + 0.5f) * Step; }
			__host__ __device__ __forceinline__ int Points(int) const { return N * parts::kBox; }
			__host__ __device__ __forceinline__ int Bricks(int) const { return N; }
			__device__ __forceinline__ float Keep() const { return INFINITY; }
			__device__ __forceinline__ uint32_t BrickAt(Vec3 p) const
			{
				const float over = 1.0f / (Step * (float)parts::kBox);
				const float most = (float)(N - 1);
				const uint32_t x = (uint32_t)fminf(fmaxf((p.x - Origin[0]) * over, 0.0f), most);
				const uint32_t y = (uint32_t)fminf(fmaxf((p.y - Origin[1]) * over, 0.0f), most);
				const uint32_t z = (uint32_t)fminf(fmaxf((p.z - Origin[2]) * over, 0.0f), most);
				return x + (uint32_t)N * (y + (uint32_t)N * z);
			}
			__device__ __forceinline__ uint32_t Above(uint32_t b) const
			{
				const uint32_t n = (uint32_t)N, coarse = n / 4;
				return b % n / 4 + coarse * (b / n % n / 4 + coarse * (b / (n * n) / 4));
			}
		};
		using RenderLattice = RenderBricksOf<0>;

		// MarchBounded by the bricks' tapes: the same distances, and so the same steps.
		__device__ __forceinline__ March MarchTapes(const DeviceProgram& prog, const RenderLattice& lat, const BrickTapes& tapes, Vec3 start,
			Vec3 dir_in, int iterations, float epsilon, float* spill, parts::PointRun& run)
		{
			const Vec3 dir = Normalize(dir_in);
			const float rootClip = fabsf(__ldg(&prog.Nodes[0].ClipRadius));
			const Vec3 root(__ldg(&prog.Nodes[0].Pivot[0]), __ldg(&prog.Nodes[0].Pivot[1]), __ldg(&prog.Nodes[0].Pivot[2]));
			const float half = rootClip * 0.57735f;               // root cube half-width
			// Leaving the root sphere along the ray ends the march: nothing lies beyond.
			const Vec3 oc = start - root;
			const float b = Dot(oc, dir);
			const float c = Dot(oc, oc) - rootClip * rootClip;
			const float disc = b * b - c;
			if (disc < 0.0f) return { false, INFINITY, start };
			const float exitTravel = -b + sqrtf(disc);
			if (exitTravel < 0.0f) return { false, INFINITY, start };
			const float4* code = prog.Code;
			Vec3 pos = start;
			float travel = 0.0f;
			run.Lo[0] = 1.0f; run.Hi[0] = 0.0f;
			Vec3 pivot(0.0f, 0.0f, 0.0f);
			float clip = 0.0f;
			for (int i = 0; i < iterations; ++i)
			{
				const Vec3 off = pos - root;
				const float ox = fmaxf(fabsf(off.x) - half, 0.0f), oy = fmaxf(fabsf(off.y) - half, 0.0f), oz = fmaxf(fabsf(off.z) - half, 0.0f);
				float step = sqrtf(ox * ox + oy * oy + oz * oz);
				if (!(step > epsilon))
				{
					if (!parts::InRun(run, pos))
					{
						if (!parts::FindPart(tapes, __ldg(tapes.Bricks + lat.BrickAt(pos)), pos, run)) parts::RunWhole(prog, pos, run);
						const OctNode* n = prog.Nodes + run.Cell;
						pivot = Vec3(__ldg(&n->Pivot[0]), __ldg(&n->Pivot[1]), __ldg(&n->Pivot[2]));
						clip = __ldg(&n->ClipRadius);
					}
					float f;
					if (run.Events != kNoTape)
					{
						const uint2* ev = tapes.Events + run.Value;
						f = RunTapePoint([&](int q) { return __ldg(code + q); }, run.Distance, run.First.x, [&](uint32_t e) { return __ldg(ev + e); }, run.Events,
							pos.x, pos.y, pos.z, spill, 2 * 32);
					}
					else f = RunWholePoint(code, run.Distance, pos.x, pos.y, pos.z, spill, 2 * 32);
					if (f <= epsilon) return { true, travel, pos };
					const float room = clip - Length(pos - pivot);
					step = fminf(f, fmaxf(room, epsilon));
				}
				travel = travel + step;
				if (travel > exitTravel) break;
				pos = dir * travel + start;
			}
			return { false, INFINITY, pos };
		}

		__device__ __forceinline__ Vec3 PixelRay(const CameraBasis& cam, int x, int y, int width, int height)
		{
			const float u = ((2.0f * ((float)x + 0.5f) / (float)width) - 1.0f) * cam.TanHalfFov * cam.Aspect;
			const float v = (1.0f - 2.0f * ((float)y + 0.5f) / (float)height) * cam.TanHalfFov;
			const Vec3 fwd(cam.Forward[0], cam.Forward[1], cam.Forward[2]);
			const Vec3 right(cam.Right[0], cam.Right[1], cam.Right[2]);
			const Vec3 up(cam.Up[0], cam.Up[1], cam.Up[2]);
			return (fwd + right * u) + up * v;
		}

		// RenderKernel's octree-bounded form by tapes.  A block is one warp of 8 x 4 pixels:
		// neighbouring rays mostly share bricks (in a row of 32 they part sooner), and rays that
		// graze the surface for a hundred steps and more hold up no other warp's place.
		__global__ void __launch_bounds__(32, 32) RenderTapesKernel(DeviceProgram prog, RenderLattice lat, BrickTapes tapes,
			const CameraBasis* __restrict__ cams, int count, int width, int height, int steps, float epsilon, float* __restrict__ depth,
			float* __restrict__ normals, uint8_t* __restrict__ colors)
		{
			extern __shared__ __align__(16) float2 spill2[];
			const int tilesX = (width + kTileX - 1) / kTileX, tilesY = (height + kTileY - 1) / kTileY;
			const int tile = (int)(blockIdx.x % (unsigned)(tilesX * tilesY)), c = (int)(blockIdx.x / (unsigned)(tilesX * tilesY));
			const int x = (tile % tilesX) * kTileX + (int)(threadIdx.x & 7), y = (tile / tilesX) * kTileY + (int)(threadIdx.x >> 3);
			if (x >= width || y >= height || c >= count) return;
			const int64_t t = ((int64_t)c * height + y) * width + x;
			const CameraBasis& cam = cams[c];
			float2* spill = spill2 + threadIdx.x;
			parts::PointRun run;
			const March m = MarchTapes(prog, lat, tapes, Vec3(cam.Position[0], cam.Position[1], cam.Position[2]), PixelRay(cam, x, y, width, height),
				steps, epsilon, reinterpret_cast<float*>(spill), run);
			depth[t] = m.Travel;
			Vec3 n(0.0f, 0.0f, 0.0f);
			uchar4 col = make_uchar4(0, 0, 0, 0);
			if (m.Hit)
			{
				const PairUnits units = LoadPairUnits();
				float none;
				n = parts::RunGradient<false, 32>(prog, tapes, run, m.Position, units, spill, false, none);
				if (colors) col = parts::RunColor<32>(prog, tapes, run, m.Position, units, spill);
			}
			normals[t * 3] = n.x;
			normals[t * 3 + 1] = n.y;
			normals[t * 3 + 2] = n.z;
			if (colors)
			{
				colors[t * 3] = col.x;
				colors[t * 3 + 1] = col.y;
				colors[t * 3 + 2] = col.z;
			}
		}

		size_t TraceSpillBytes(const DeviceProgram& prog)
		{
			const int depth = prog.MaxStack > 1 ? prog.MaxStack - 1 : 1;
			return (size_t)depth * 2 * kTraceThreads * sizeof(float);
		}
	}

	cudaError_t LaunchRayMarch(const DeviceProgram& prog, const float* origins, const float* dirs, int64_t n, int max_iterations,
		float epsilon, uint8_t* hit, float* travel, float* position, cudaStream_t stream)
	{
		if (n <= 0) return cudaSuccess;
		const size_t smem = TraceSpillBytes(prog);
		if (smem > 48 * 1024) cudaFuncSetAttribute(RayMarchKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
		RayMarchKernel<<<(unsigned)((n + kTraceThreads - 1) / kTraceThreads), kTraceThreads, smem, stream>>>(
			prog, origins, dirs, n, max_iterations, epsilon, hit, travel, position);
		return cudaGetLastError();
	}

	cudaError_t LaunchRayQuery(const DeviceProgram& prog, const RayFrame& frame, const float* origins, const float* dirs, int64_t n,
		int max_iterations, float epsilon, uint8_t* hit, float* travel, float* position, cudaStream_t stream)
	{
		if (n <= 0) return cudaSuccess;
		const size_t smem = TraceSpillBytes(prog);
		if (smem > 48 * 1024)
		{
			cudaError_t e = cudaFuncSetAttribute(RayQueryKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		RayQueryKernel<<<(unsigned)((n + kTraceThreads - 1) / kTraceThreads), kTraceThreads, smem, stream>>>(
			prog, frame, origins, dirs, n, max_iterations, epsilon, hit, travel, position);
		return cudaGetLastError();
	}

	cudaError_t LaunchPointQuery(const DeviceProgram& prog, const float* points, int64_t n, bool gradient, float* out,
		cudaStream_t stream)
	{
		if (n <= 0) return cudaSuccess;
		const size_t pairs = parts::SpillPairs(prog, 1), smem = kQueryThreads / 32 * (64 * sizeof(float4) + pairs * 32 * sizeof(float2));
		auto* kernel = gradient ? PointQueryKernel<true> : PointQueryKernel<false>;
		if (smem > 48 * 1024)
		{
			cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		const int64_t per = kQueryThreads / 32 * (gradient ? 16 : 64);
		kernel<<<(unsigned)((n + per - 1) / per), kQueryThreads, smem, stream>>>(prog, points, n, out, (int)pairs);
		return cudaGetLastError();
	}

	cudaError_t LaunchRender(const DeviceProgram& prog, const CameraBasis* cameras, int count, int width, int height,
		int max_steps, float epsilon, bool exact, float* depth, float* normals, uint8_t* colors, cudaStream_t stream)
	{
		const int64_t total = (int64_t)width * height * count;
		if (total <= 0) return cudaSuccess;
		const size_t smem = TraceSpillBytes(prog);
		if (smem > 48 * 1024) cudaFuncSetAttribute(RenderKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
		RenderKernel<<<(unsigned)((total + kTraceThreads - 1) / kTraceThreads), kTraceThreads, smem, stream>>>(
			prog, cameras, count, width, height, max_steps, epsilon, exact || !prog.Lipschitz, depth, normals, colors);
		return cudaGetLastError();
	}

	// Bricks per axis for the renderer's tapes, 0 for none.  A tape costs a pass of its cell's
	// program by one warp, and building them all 120 us at least; without, a render of any size
	// lasts as long as the ray that grazes the surface longest, some hundred whole programs one
	// after the other.  So what counts are the pixels and what a program has beyond two brushes
	// (ten quads), which a tape mostly leaves; fitted to 240 images of 40 trees.  Measured on a GB300, none against tapes, us an image
	// (quads a point runs in brackets): 1 primitive (5) 1920 x 1080 168 / 238, 2 (10) 256 / 270, 4 (12)
	// 200 x 150 137 / 185, 800 x 500 385 / 260, 8 (18) 64 x 48 152 / 193, 128 x 96 231 / 216, 16 (25)
	// 355 / 280, 32 (61) 64 x 48 356 / 258, 64 (50) 382 / 237, 256 (107) 1757 / 667; the rule's worst,
	// 16 (44) 128 x 96 159 / 224.  Scenes so wide that their cells ask for 64 bricks an axis build
	// eight times the tapes, of space that is mostly empty: 60 strewn primitives 640 x 360 566 / 815,
	// 1920 x 1080 1453 / 1024.
	int RenderBricks(const DeviceProgram& prog, float root_clip, int64_t pixels, double quads)
	{
		if (!prog.Lipschitz || !(prog.Form & kFormPrunable)) return 0;
		const float span = 2.0f * fabsf(root_clip) * 0.57735f;
		// The cells' edge: the cube halved until no more than the octree's target.
		int cells = 1;
		while (cells < 128 && span / (float)cells > 0.25f) cells *= 2;
		const int n = cells < 32 ? 32 : cells;
		const double gain = quads > 10.0 ? (double)pixels * std::sqrt(quads - 10.0) : 0.0;
		return n <= 64 && gain >= (n > 32 ? 2e6 : 1.8e4) ? n : 0;
	}

	cudaError_t LaunchRenderTapes(const DeviceProgram& prog, const float* pivot, float root_clip, int bricks, const BrickTapes& tapes, const BrickTapes& above,
		const CameraBasis* cameras, int count, int width, int height, int max_steps, float epsilon, float* depth, float* normals,
		uint8_t* colors, int sms, cudaStream_t stream)
	{
		RenderLattice lat;
		const float half = fabsf(root_clip) * 0.57735f;
		lat.N = bricks;
		lat.Step = 2.0f * half / (float)(bricks * parts::kBox);
		for (int a = 0; a < 3; ++a) lat.Origin[a] = pivot[a] - half;
		cudaError_t e = cudaSuccess;
		if (above.Bricks)
		{
			RenderBricksOf<1> coarse;
			coarse.N = bricks / 4;
			coarse.Step = 4.0f * lat.Step;
			for (int a = 0; a < 3; ++a) coarse.Origin[a] = lat.Origin[a];
			e = parts::LaunchParts(prog, coarse, nullptr, nullptr, nullptr, above, sms, stream);
			if (e != cudaSuccess) return e;
		}
		e = parts::LaunchParts(prog, lat, nullptr, nullptr, nullptr, tapes, sms, stream, above);
		if (e != cudaSuccess) return e;
		// The colour's walk takes two words a level, the gradient one pair.
		const size_t smem = parts::SpillPairs(prog, 2) * 32 * sizeof(float2);
		if (smem > 48 * 1024)
		{
			e = cudaFuncSetAttribute(RenderTapesKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		const int64_t blocks = (int64_t)((width + kTileX - 1) / kTileX) * ((height + kTileY - 1) / kTileY) * count;
		if (blocks > 0x7FFFFFFF) return cudaErrorInvalidValue;
		RenderTapesKernel<<<(unsigned)blocks, 32, smem, stream>>>(prog, lat, tapes, cameras, count, width, height, max_steps, epsilon,
			depth, normals, colors);
		return cudaGetLastError();
	}
}
