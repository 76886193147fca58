// The whole tree at one point by many threads: exact ray casts and point queries where there
// are too few of them to fill the GPU with a thread each.
//
// A thread takes the tree's surface program record by record, some six hundred cycles a
// record one after the other, and a ray a hundred times over.  A team (a warp, or a whole
// block for the fewest) evaluates all brushes at once, a brush per thread, and then the
// operators level by level: operators of one level have their operands ready and do not wait
// for each other.  The operations and their operands are SDFNode::Eval's, so the values are
// the program's bit for bit, whatever the order they are computed in.
#include <cmath>

#include "tg_device.cuh"
#include "tg_kernels.hpp"
#include "tg_surface.cuh"
#include "tg_tape.cuh"

namespace tg
{
	namespace
	{
		constexpr int kTeamThreads = 256;
		constexpr int kTeamSmem = 200 * 1024;

		// The tree in shared memory: brushes 0 .. Brushes - 1, then the operators sorted by level
		// (operands' slots, opcode and own slot, threshold).
		struct TeamTree
		{
			float4* Head;           // opcode and parameters
			float4* Turn;           // inverse quaternion
			float4* Move;           // translation, scale
			uint4* Ops;             // left slot, right slot, own slot << 8 | opcode, threshold
			uint32_t* Level;        // first operator of each level, and their end
			float* Value;           // the teams' values: (brushes + operators) x points each
			int Brushes, Count, Levels, Root;
		};

		__host__ __device__ inline size_t TeamTreeBytes(int brushes, int ops)
		{
			// Head, Turn, Move; Ops twice (as parsed, and by level); levels; the parse's own tables.
			const size_t n = (size_t)brushes + ops;
			return (size_t)brushes * 48 + (size_t)ops * 32 + ((size_t)ops + 4) * 8 + n * 4 + 64 * sizeof(float4) + (kMaxStack + 4) * 4 + 64;
		}

		// Reads the program at prog.FullSurfaceCode into `shared` by the whole block.
		__device__ __forceinline__ TeamTree LoadTeamTree(const DeviceProgram& prog, uint8_t* shared)
		{
			TeamTree t;
			const int nb = prog.FullBrushes, no = prog.FullOps;
			float4* at = reinterpret_cast<float4*>(shared);
			t.Head = at; at += nb;
			t.Turn = at; at += nb;
			t.Move = at; at += nb;
			t.Ops = reinterpret_cast<uint4*>(at); at += no;
			uint4* parsed = reinterpret_cast<uint4*>(at); at += no;
			float4* window = at; at += 64;
			uint32_t* words = reinterpret_cast<uint32_t*>(at);
			t.Level = words; words += no + 4;
			uint32_t* cursor = words; words += no + 4;
			uint32_t* stack = words; words += kMaxStack + 4;
			uint32_t* slot = words;             // per brush its first quad; per operator its level
			t.Brushes = nb;
			t.Count = no;
			const float4* code = prog.Code + prog.FullSurfaceCode;
			const int tid = (int)threadIdx.x;
			for (int i = tid; i < no + 4; i += (int)blockDim.x) t.Level[i] = cursor[i] = 0;
			__syncthreads();
			if (tid < 32)
			{
				// The operands' slots and levels, by the program's own stack: level << 16 | slot.
				SurfaceSource src;
				src.In.Open(code, prog.CodeQuads - prog.FullSurfaceCode, window);
				int depth = 0, b = 0, o = 0;
				for (int guard = 0; guard < (1 << 24); ++guard)
				{
					const uint32_t head = src.Head();
					const uint32_t op = head & 0xFFu;
					if (op == OpStop || b + o >= nb + no) break;
					if (op >= OpSphere && op <= OpPlane)
					{
						if (tid == 0) { slot[b] = (uint32_t)src.Pc; stack[depth] = (uint32_t)b; }
						++b;
						++depth;
					}
					else
					{
						const bool pair = op >= OpUnion && op <= OpBlendDiff;
						if (tid == 0)
						{
							const uint32_t r = stack[depth - 1], l = pair ? stack[depth - 2] : r;
							const uint32_t level = max(l >> 16, r >> 16) + 1u;
							parsed[o] = make_uint4(l & 0xFFFFu, r & 0xFFFFu, ((uint32_t)(nb + o) << 8) | op, __float_as_uint(src.Operand()));
							slot[nb + o] = level;
							++t.Level[level];
							stack[depth - (pair ? 2 : 1)] = (level << 16) | (uint32_t)(nb + o);
						}
						if (pair) --depth;
						++o;
					}
					src.Advance(head);
				}
				if (tid == 0)
				{
					// Level[i]: first operator of level i + 1; levels start at 1.
					uint32_t sum = 0;
					int levels = 0;
					for (int i = 1; i <= no && t.Level[i]; ++i)
					{
						const uint32_t c = t.Level[i];
						t.Level[i - 1] = cursor[i] = sum;
						sum += c;
						levels = i;
					}
					t.Level[levels] = sum;
					stack[kMaxStack + 1] = stack[0] & 0xFFFFu;
					stack[kMaxStack + 2] = (uint32_t)levels;
				}
			}
			__syncthreads();
			t.Root = (int)stack[kMaxStack + 1];
			t.Levels = (int)stack[kMaxStack + 2];
			for (int i = tid; i < nb; i += (int)blockDim.x)
			{
				const int pc = (int)slot[i];
				t.Head[i] = __ldg(code + pc);
				t.Turn[i] = __ldg(code + pc + 1);
				t.Move[i] = __ldg(code + pc + 2);
			}
			for (int i = tid; i < no; i += (int)blockDim.x)
				t.Ops[atomicAdd(&cursor[slot[nb + i]], 1u)] = parsed[i];
			__syncthreads();
			return t;
		}

		template<int Team>
		__device__ __forceinline__ void TeamSync()
		{
			if (Team == 32) __syncwarp();
			else __syncthreads();
		}

		// SDFNode::Eval at P points by the team; every thread gets the values.  `value`: the team's
		// slots, P floats each.
		template<int P, int Team>
		__device__ __forceinline__ void TeamEval(const TeamTree& t, float* value, int lane, const Vec3 (&p)[P], float (&out)[P])
		{
			for (int k = lane; k < t.Brushes; k += Team)
			{
				const float4 h = t.Head[k], Q = t.Turn[k], T = t.Move[k];
				const Quat qi{ Q.x, Q.y, Q.z, Q.w };
				const uint32_t op = __float_as_uint(h.x) & 0xFFu;
				const bool scaled = T.w != 1.0f;    // x / 1 and x * 1 are x exactly
#pragma unroll
				for (int j = 0; j < P; ++j)
				{
					Vec3 local = Rotate(qi, p[j] - Vec3(T.x, T.y, T.z));
					if (scaled) local = local / T.w;
					const float d = TapeBrush(op, h, local.x, local.y, local.z);
					value[k * P + j] = scaled ? d * T.w : d;
				}
			}
			TeamSync<Team>();
			for (int level = 0; level < t.Levels; ++level)
			{
				const uint32_t end = t.Level[level + 1];
				for (uint32_t i = t.Level[level] + (uint32_t)lane; i < end; i += Team)
				{
					const uint4 o = t.Ops[i];
					const uint32_t op = o.z & 0xFFu, own = o.z >> 8;
					const float k = __uint_as_float(o.w);
#pragma unroll
					for (int j = 0; j < P; ++j)
					{
						const float l = value[o.x * P + j], r = value[o.y * P + j];
						value[own * P + j] = op == OpFlate ? r - k : TapeSet(op, l, r, k);
					}
				}
				TeamSync<Team>();
			}
#pragma unroll
			for (int j = 0; j < P; ++j) out[j] = value[t.Root * P + j];
			TeamSync<Team>();
		}

		template<int Team, int P>
		__device__ __forceinline__ float* TeamValues(const DeviceProgram& prog, uint8_t* shared)
		{
			const size_t n = (size_t)prog.FullBrushes + prog.FullOps;
			uint8_t* base = shared + (TeamTreeBytes(prog.FullBrushes, prog.FullOps) + 15) / 16 * 16;
			return reinterpret_cast<float*>(base) + (Team == 32 ? threadIdx.x / 32 : 0) * n * P;
		}

		// SDFNode::RayMarch (sdf_evaluator.cpp:336-353), a team per ray.
		template<int Team>
		__global__ void __launch_bounds__(kTeamThreads) TeamRayKernel(DeviceProgram prog, RayFrame f, const float* __restrict__ origins,
			const float* __restrict__ dirs, int64_t n, int iterations, float epsilon, uint8_t* __restrict__ hit, float* __restrict__ travel,
			float* __restrict__ position)
		{
			extern __shared__ __align__(16) uint8_t shared[];
			const TeamTree t = LoadTeamTree(prog, shared);
			float* value = TeamValues<Team, 1>(prog, shared);
			const int lane = Team == 32 ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
			const int64_t teams = Team == 32 ? (int64_t)gridDim.x * (kTeamThreads / 32) : gridDim.x;
			for (int64_t r = Team == 32 ? (int64_t)blockIdx.x * (kTeamThreads / 32) + threadIdx.x / 32 : blockIdx.x; r < n; r += teams)
			{
				Vec3 start(origins[r * 3], origins[r * 3 + 1], origins[r * 3 + 2]);
				Vec3 dir(dirs[r * 3], dirs[r * 3 + 1], dirs[r * 3 + 2]);
				FrameRay(f, start, dir);
				dir = Normalize(dir);
				Vec3 pos = start;
				float far = 0.0f;
				bool found = false;
				for (int i = 0; i < iterations && !found; ++i)
				{
					const Vec3 p[1] = { pos };
					float d[1];
					TeamEval<1, Team>(t, value, lane, p, d);
					found = d[0] <= epsilon;
					if (found) break;
					far = far + d[0];
					pos = dir * far + start;
				}
				if (lane == 0)
				{
					hit[r] = found ? 1 : 0;
					travel[r] = found ? far : INFINITY;
					position[r * 3] = pos.x;
					position[r * 3 + 1] = pos.y;
					position[r * 3 + 2] = pos.z;
				}
			}
		}

		// SDFNode::Eval or SDFNode::Gradient (sdf_evaluator.cpp:298-333), a team per point.
		template<int Team, bool Gradient>
		__global__ void __launch_bounds__(kTeamThreads) TeamPointKernel(DeviceProgram prog, const float* __restrict__ points, int64_t n,
			float* __restrict__ out)
		{
			constexpr int P = Gradient ? 4 : 1;
			extern __shared__ __align__(16) uint8_t shared[];
			const TeamTree t = LoadTeamTree(prog, shared);
			float* value = TeamValues<Team, P>(prog, shared);
			const int lane = Team == 32 ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
			const int64_t teams = Team == 32 ? (int64_t)gridDim.x * (kTeamThreads / 32) : gridDim.x;
			for (int64_t r = Team == 32 ? (int64_t)blockIdx.x * (kTeamThreads / 32) + threadIdx.x / 32 : blockIdx.x; r < n; r += teams)
			{
				const Vec3 p(points[r * 3], points[r * 3 + 1], points[r * 3 + 2]);
				float d[P];
				if constexpr (!Gradient)
				{
					const Vec3 q[1] = { p };
					TeamEval<1, Team>(t, value, lane, q, d);
					if (lane == 0) out[r] = d[0];
				}
				else
				{
					const Vec3 q[4] = { TetraPoint(p, 0), TetraPoint(p, 1), TetraPoint(p, 2), TetraPoint(p, 3) };
					TeamEval<4, Team>(t, value, lane, q, d);
					float e[5] = { d[0], d[1], d[2], d[3], 0.0f };
					const float h = 0.0001f;
					const Vec3 xyy(h, -h, -h), yyx(-h, -h, h), yxy(-h, h, -h), xxx(h, h, h);
					Vec3 g = xyy * e[0];
					g = g + yyx * e[1];
					g = g + yxy * e[2];
					g = g + xxx * e[3];
					if ((g.x * g.x + g.y * g.y) + g.z * g.z == 0.0f)
					{
						const Vec3 c[4] = { p, p, p, p };
						float at[4];
						TeamEval<4, Team>(t, value, lane, c, at);
						e[4] = at[0];
					}
					const Vec3 r3 = GradientOf(e);
					if (lane == 0)
					{
						out[r * 3] = r3.x;
						out[r * 3 + 1] = r3.y;
						out[r * 3 + 2] = r3.z;
					}
				}
			}
		}

		// The block's shared memory with `points` values a slot, 0 where the tree does not fit.
		size_t TeamSmem(const DeviceProgram& prog, bool block, int points)
		{
			const size_t n = (size_t)prog.FullBrushes + prog.FullOps;
			if (prog.FullBrushes < 1 || n > 0xFFFF) return 0;
			const size_t bytes = (TeamTreeBytes(prog.FullBrushes, prog.FullOps) + 15) / 16 * 16 + n * points * sizeof(float) * (block ? 1 : kTeamThreads / 32);
			return bytes <= kTeamSmem ? bytes : 0;
		}

		template<typename Kernel>
		cudaError_t TeamGrid(Kernel kernel, size_t smem, bool block, int64_t n, int sms, unsigned& blocks)
		{
			cudaError_t e = cudaSuccess;
			if (smem > 48 * 1024) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			int per = 1;
			if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kTeamThreads, smem);
			if (e != cudaSuccess) return e;
			const int64_t want = block ? n : (n + kTeamThreads / 32 - 1) / (kTeamThreads / 32), most = (int64_t)sms * (per > 0 ? per : 1);
			blocks = (unsigned)(want < most ? want : most);
			return cudaSuccess;
		}
	}

	// A thread per ray (two lanes or half a lane per point, PointQueryKernel) takes about as long
	// for one as for many (the program's records one after the other); a team's time grows with
	// the count.  Measured on a GB300, teams against that, us a call: rays through 8 primitives
	// 3000 220 / 363, 9000 464 / 384; 64 primitives 30 288 / 2414, 16384 1298 / 2547; 128
	// primitives 16384 1584 / 4901; gradients of 16 primitives 1000 31 / 32, 4000 37 / 34; of 64
	// primitives 1000 56 / 60, 8000 76 / 69; of 256 primitives 200 119 / 173, 8000 179 / 189,
	// 16000 239 / 202; values of 64 primitives 1000 47 / 59, 16000 68 / 68; of 256 primitives 1000
	// 117 / 169, 30000 179 / 182.
	int TeamForm(const DeviceProgram& prog, int64_t n, TeamWork work, int sms)
	{
		const int points = work == TeamWork::Gradient ? 4 : 1;
		// One evaluation of a small tree is over before a team has read it.
		if (work == TeamWork::Eval && prog.FullBrushes < 24) return 0;
		if (n <= sms && TeamSmem(prog, true, points)) return 2;
		const double brushes = (double)prog.FullBrushes;
		const double most = work == TeamWork::Ray ? 26.0 * brushes / (0.037 + 0.0004 * brushes)
			: work == TeamWork::Gradient ? 10000.0 * brushes / (brushes + 48.0) : 0.6 * brushes / (0.0017 + 0.000022 * brushes);
		return (double)n <= most && TeamSmem(prog, false, points) ? 1 : 0;
	}

	cudaError_t LaunchTeamRays(const DeviceProgram& prog, const RayFrame& frame, const float* origins, const float* dirs, int64_t n,
		int max_iterations, float epsilon, uint8_t* hit, float* travel, float* position, int form, int sms, cudaStream_t stream)
	{
		const bool block = form == 2;
		const size_t smem = TeamSmem(prog, block, 1);
		if (!smem || n <= 0) return cudaErrorInvalidValue;
		auto* kernel = block ? TeamRayKernel<kTeamThreads> : TeamRayKernel<32>;
		unsigned blocks = 1;
		const cudaError_t e = TeamGrid(kernel, smem, block, n, sms, blocks);
		if (e != cudaSuccess) return e;
		kernel<<<blocks, kTeamThreads, smem, stream>>>(prog, frame, origins, dirs, n, max_iterations, epsilon, hit, travel, position);
		return cudaGetLastError();
	}

	cudaError_t LaunchTeamPoints(const DeviceProgram& prog, const float* points, int64_t n, bool gradient, float* out, int form, int sms,
		cudaStream_t stream)
	{
		const bool block = form == 2;
		const size_t smem = TeamSmem(prog, block, gradient ? 4 : 1);
		if (!smem || n <= 0) return cudaErrorInvalidValue;
		auto* kernel = gradient ? (block ? TeamPointKernel<kTeamThreads, true> : TeamPointKernel<32, true>)
			: (block ? TeamPointKernel<kTeamThreads, false> : TeamPointKernel<32, false>);
		unsigned blocks = 1;
		const cudaError_t e = TeamGrid(kernel, smem, block, n, sms, blocks);
		if (e != cudaSuccess) return e;
		kernel<<<blocks, kTeamThreads, smem, stream>>>(prog, points, n, out);
		return cudaGetLastError();
	}
}
