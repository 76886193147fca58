// Shortened programs ("tapes") for a small box of space.
//
// An octree cell's program covers a cube of up to 0.25 units; a brick of a fine export is a
// few hundredths.  Inside such a box most set operators always take the same operand: every
// brush here (the ellipsoid, and trees with rotations that are not unit quaternions, excepted)
// is 1-Lipschitz and union, intersection, difference, the polynomial blends, flate and uniform
// scale keep that, so when two operands differ at the centre of a ball of radius r by more than
// 2r (and the rounding of both sides), the same one wins at every point of the ball.  The other
// operand's records can then be left out: min, max and the blends (where the operands are at
// least the blend radius apart) return the winning operand's value itself, so the shortened
// program's value at a point is the whole program's, bit for bit.
//
// BuildTape runs one program once per box, a warp at 64 points (two per lane, the centres of
// the box's 4 x 4 x 4 sub-boxes), and votes on every set operator: a side is left out when it
// loses in every sub-box.  A tape is a list of events, one per record that is left, in the
// program's own order; the records themselves stay where they are, shared by all tapes of the
// program.  Each event also names the record's place in the cell's surface program, so the
// same list serves the gradient (SDFNode::Eval's form); a second list keeps what GetMaterial
// needs (the left operand of a difference has the material even where the right one decides
// the distance).
#pragma once

#include "tg_device.cuh"
#include "tg_kernels.hpp"
#include "tg_pair.cuh"

namespace tg
{
	// Event: x = distance record (quad offset in the cell's distance program) << 16 | opcode |
	// record flags; y = quad offset of the record in the cell's surface program.
	constexpr uint32_t kTapeHead = 0xFFu | RecMatrix | RecOffset | RecScale | RecThenSet;
	// Opcodes of events without a record: the operand a difference left alone is negated, and a
	// blend's sum with its zero term turns -0 into +0.
	enum : uint32_t { OpTapeNegate = 40, OpTapeAddZero = 41 };

	constexpr int kTapeCap = 128;               // events of a brick's list while it is built
	constexpr uint32_t kNoTape = 0xFFFFu;       // an event count: run the cell's whole program

	__device__ __forceinline__ uint32_t ProgramHead(float word) { return __float_as_uint(word) & kTapeHead; }

	__device__ __forceinline__ int DistanceRecordQuads(uint32_t head)
	{
		const uint32_t op = head & 0xFFu;
		if (op < OpSphere || op > OpPlane) return 1;
		return 1 + ((head & RecMatrix) ? 3 : (head & RecOffset) ? 1 : 0) + ((head & RecScale) ? 1 : 0);
	}

	// The brushes a modeller uses least, out of line: one copy of their code for all callers.
	static __device__ __noinline__ float RareBrushDistance(uint32_t op, float a, float b, float c, float x, float y, float z)
	{
		const float prm[3] = { a, b, c };
		return BrushDistance(op, prm, Vec3(x, y, z));
	}

	// BrushDistance2 and SetDistance2 (tg_pair.cuh), the same values from less code: the
	// evaluations by tapes are short, and a kernel that holds several interpreters waited for
	// instructions more than for anything else (10 to 12 of 17 stall cycles an issue in the
	// vertex attributes and the point cloud's refinement with the formulas expanded one by one).
	// The common brushes share their squares and roots: a sphere and a box end with the length
	// of a 3-vector, a torus and a cylinder with that of a 2-vector made from one.  Kernels with
	// one interpreter, whose warps run it in step, take the formulas one by one instead
	// (Compact = false: the builds and the brick evaluation 4 to 5 % faster so, the refinement
	// 20 % slower).
	template<bool Compact = true>
	__device__ __forceinline__ float2 TapeBrush2(uint32_t op, const float4& h, float2 x, float2 y, float2 z, const PairUnits& u)
	{
		const bool round = op == OpTorus || op == OpCylinder;
		if (op != OpSphere && op != OpBox && !round)
			return make_float2(RareBrushDistance(op, h.y, h.z, h.w, x.x, y.x, z.x), RareBrushDistance(op, h.y, h.z, h.w, x.y, y.y, z.y));
		if (!Compact)
		{
			if (op == OpSphere) return SdSphere2(x, y, z, h.y, u);
			if (op == OpBox) return SdBox2(x, y, z, h.y, h.z, h.w, u);
			return op == OpTorus ? SdTorus2(x, y, z, h.y, h.z, u) : SdCylinder2(x, y, z, h.y, h.z, u);
		}
		float2 last = Pair(-h.y), zz = z;
		if (op == OpBox)
		{
			x = Sub2(Abs2(x), Pair(h.y), u);
			y = Sub2(Abs2(y), Pair(h.z), u);
			zz = Sub2(Abs2(z), Pair(h.w), u);
			last = make_float2(fminf(fmaxf(fmaxf(x.x, y.x), zz.x), 0.0f), fminf(fmaxf(fmaxf(x.y, y.y), zz.y), 0.0f));
			x = TernaryMax2(x, 0.0f);
			y = TernaryMax2(y, 0.0f);
			zz = TernaryMax2(zz, 0.0f);
		}
		float2 s = Add2(Mul2(x, x, u), Mul2(y, y, u), u);
		if (!round) s = Add2(s, Mul2(zz, zz, u), u);
#pragma unroll 1
		for (int root = 0; ; ++root)
		{
			const float2 length = Sqrt2(s);
			if (!round || root == 1) return Add2(length, last, u);
			// The distance from the axis less the major radius (a cylinder's radius).
			float2 a = Add2(length, Pair(-h.y), u), b = z;
			last = Pair(-h.z);
			if (op == OpCylinder)
			{
				b = Sub2(Abs2(z), Pair(h.z), u);
				last = make_float2(fminf(fmaxf(a.x, b.x), 0.0f), fminf(fmaxf(a.y, b.y), 0.0f));
				a = TernaryMax2(a, 0.0f);
				b = TernaryMax2(b, 0.0f);
			}
			s = Add2(Mul2(a, a, u), Mul2(b, b, u), u);
		}
	}

	// TapeBrush2 for one point; the kinds of brush are told apart by selection, so that lanes on
	// different tapes stay together.
	__device__ __forceinline__ float TapeBrush(uint32_t op, const float4& h, float x, float y, float z)
	{
		const bool box = op == OpBox, cylinder = op == OpCylinder, round = op == OpTorus || cylinder;
		if (!box && !round && op != OpSphere) return RareBrushDistance(op, h.y, h.z, h.w, x, y, z);
		const float ax = box ? fabsf(x) - h.y : x, ay = box ? fabsf(y) - h.z : y, az = box ? fabsf(z) - h.w : z;
		float last = box ? fminf(fmaxf(fmaxf(ax, ay), az), 0.0f) : -h.y;
		const float vx = box ? TernaryMax(ax, 0.0f) : ax, vy = box ? TernaryMax(ay, 0.0f) : ay, vz = box ? TernaryMax(az, 0.0f) : az;
		const float s = vx * vx + vy * vy;
		float length = sqrtf(round ? s : s + vz * vz);
		if (round)
		{
			// The distance from the axis less the major radius (a cylinder's radius).
			const float a = length + -h.y, b = cylinder ? fabsf(z) - h.z : z;
			last = cylinder ? fminf(fmaxf(a, b), 0.0f) : -h.z;
			const float va = cylinder ? TernaryMax(a, 0.0f) : a, vb = cylinder ? TernaryMax(b, 0.0f) : b;
			length = sqrtf(va * va + vb * vb);
		}
		return length + last;
	}

	static __device__ __noinline__ float TapeBlendTerm(float m, float h, float k, bool subtract) { return BlendTerm(m, h, k, subtract); }

	// The blends share one term, out of line where it is not zero: the difference blends as the
	// intersection with its right operand negated (|l + r| is |l - -r|).
	__device__ __forceinline__ float TapeBlend(bool unions, float l, float r, float k)
	{
		const float m = unions ? fminf(l, r) : fmaxf(l, r);
		const float h = fmaxf(k - fabsf(l - r), 0.0f);
		if (h == 0.0f && k > 0.0f) return unions ? m - 0.0f : m + 0.0f;
		return TapeBlendTerm(m, h, k, unions);
	}

	__device__ __forceinline__ float TapeSet(uint32_t op, float l, float r, float k)
	{
		if (op == OpDiff || op == OpBlendDiff) r = -r;
		if (op >= OpBlendUnion) return TapeBlend(op == OpBlendUnion, l, r, k);
		return op == OpUnion ? fminf(l, r) : fmaxf(l, r);
	}

	__device__ __forceinline__ float2 TapeSet2(uint32_t op, float2 l, float2 r, float k)
	{
		if (op == OpDiff || op == OpBlendDiff) r = make_float2(-r.x, -r.y);
		if (op >= OpBlendUnion)
		{
			const bool unions = op == OpBlendUnion;
			return make_float2(TapeBlend(unions, l.x, r.x, k), TapeBlend(unions, l.y, r.y, k));
		}
		if (op == OpUnion) return make_float2(fminf(l.x, r.x), fminf(l.y, r.y));
		return make_float2(fmaxf(l.x, r.x), fmaxf(l.y, r.y));
	}

	// Transform::ApplyInv's division by a brush's scale, out of line: most brushes have none.
	static __device__ __noinline__ float2 DividePair(float2 a, float s) { return make_float2(a.x / s, a.y / s); }

	// A brush's distance (RunDistancePairs' step) from its record at `pc`, whose head is known;
	// q is left at the points in the brush's own frame, h at the record's first quad.
	template<int NP, bool Compact = true, typename Load>
	__device__ __forceinline__ void BrushStep(Load load, int pc, uint32_t head, const float2 (&px)[NP], const float2 (&py)[NP],
		const float2 (&pz)[NP], const PairUnits& u, float2 (&qx)[NP], float2 (&qy)[NP], float2 (&qz)[NP], float4& h, float2 (&d)[NP])
	{
		h = load(pc);
#pragma unroll
		for (int j = 0; j < NP; ++j) { qx[j] = px[j]; qy[j] = py[j]; qz[j] = pz[j]; }
		int at = pc + 1;
		if (head & RecMatrix)
		{
			const float4 X = load(at), Y = load(at + 1), Z = load(at + 2);
			at += 3;
#pragma unroll
			for (int j = 0; j < NP; ++j)
			{
				qx[j] = AffineRow2(X, px[j], py[j], pz[j], u);
				qy[j] = AffineRow2(Y, px[j], py[j], pz[j], u);
				qz[j] = AffineRow2(Z, px[j], py[j], pz[j], u);
			}
		}
		else if (head & RecOffset)
		{
			const float4 O = load(at++);
#pragma unroll
			for (int j = 0; j < NP; ++j)
			{
				qx[j] = Add2(px[j], Pair(O.x), u);
				qy[j] = Add2(py[j], Pair(O.y), u);
				qz[j] = Add2(pz[j], Pair(O.z), u);
			}
		}
#pragma unroll
		for (int j = 0; j < NP; ++j) d[j] = TapeBrush2<Compact>(head & 0xFFu, h, qx[j], qy[j], qz[j], u);
		if (head & RecScale)
		{
			const float4 S = load(at);
#pragma unroll
			for (int j = 0; j < NP; ++j) d[j] = Mul2(d[j], Pair(S.x), u);
		}
	}

	// The distance at NP pairs of points by a tape of `count` (at least one) events over the
	// program at `base`; `event(i)` returns event i (from global or shared memory).  Operands
	// below the top of the stack are at spill[(depth * NP + pair) * stride].  The set
	// operator's code appears once: a brush that is its right operand falls through to it.
	template<int NP, bool Compact = true, typename Load, typename Event>
	__device__ __forceinline__ void RunTapePairs(Load load, int base, Event event, uint32_t count, const float2 (&px)[NP],
		const float2 (&py)[NP], const float2 (&pz)[NP], const PairUnits& u, float2 (&acc)[NP], float2* spill, int stride)
	{
		float2 left[NP];
#pragma unroll
		for (int j = 0; j < NP; ++j) acc[j] = left[j] = make_float2(0.0f, 0.0f);
		int depth = 0;
		uint32_t e = 0, x = event(0u).x;
		for (;;)
		{
			uint32_t op = x & 0xFFu;
			int at = base + (int)(x >> 16);
			if (op >= OpSphere && op <= OpPlane)
			{
				const uint32_t head = x;
				if (++e < count) x = event(e).x;
				if (!(head & RecThenSet))
				{
					if (depth > 0)
					{
#pragma unroll
						for (int j = 0; j < NP; ++j) spill[((depth - 1) * NP + j) * stride] = acc[j];
					}
					++depth;
				}
#pragma unroll
				for (int j = 0; j < NP; ++j) left[j] = acc[j];
				float2 qx[NP], qy[NP], qz[NP];
				float4 h;
				BrushStep<NP, Compact>(load, at, head, px, py, pz, u, qx, qy, qz, h, acc);
				if (e >= count) break;
				if (!(head & RecThenSet)) continue;
				op = x & 0xFFu;
				at = base + (int)(x >> 16);
			}
			else if (op >= OpUnion && op <= OpBlendDiff)
			{
				--depth;
#pragma unroll
				for (int j = 0; j < NP; ++j) left[j] = spill[((depth - 1) * NP + j) * stride];
			}
			if (op >= OpUnion && op <= OpBlendDiff)
			{
				const float k = op >= OpBlendUnion ? load(at).y : 0.0f;
#pragma unroll
				for (int j = 0; j < NP; ++j) acc[j] = TapeSet2(op, left[j], acc[j], k);
			}
			else if (op == OpFlate)
			{
				const float k = load(at).y;
#pragma unroll
				for (int j = 0; j < NP; ++j) acc[j] = Sub2(acc[j], Pair(k), u);
			}
			else
			{
#pragma unroll
				for (int j = 0; j < NP; ++j)
					acc[j] = op == OpTapeNegate ? make_float2(-acc[j].x, -acc[j].y) : make_float2(acc[j].x + 0.0f, acc[j].y + 0.0f);
			}
			if (++e >= count) break;
			x = event(e).x;
		}
	}

	// The distance at one point by a tape (RunTapePairs, one lane) whose first event is x.
	// Operands below the top of the stack are at spill[depth * stride].
	template<typename Load, typename Event>
	__device__ __forceinline__ float RunTapePoint(Load load, int base, uint32_t x, Event event, uint32_t count, float px, float py, float pz,
		float* spill, int stride)
	{
		float acc = 0.0f, left = 0.0f;
		int depth = 0;
		uint32_t e = 0;
		for (;;)
		{
			uint32_t op = x & 0xFFu;
			int at = base + (int)(x >> 16);
			if (op >= OpSphere && op <= OpPlane)
			{
				const uint32_t head = x;
				if (++e < count) x = event(e).x;
				if (!(head & RecThenSet))
				{
					if (depth > 0) spill[(depth - 1) * stride] = acc;
					++depth;
				}
				left = acc;
				const float4 h = load(at++);
				float qx = px, qy = py, qz = pz;
				if (head & RecMatrix)
				{
					const float4 X = load(at), Y = load(at + 1), Z = load(at + 2);
					at += 3;
					qx = (X.x * px + X.y * py) + (X.z * pz + X.w);
					qy = (Y.x * px + Y.y * py) + (Y.z * pz + Y.w);
					qz = (Z.x * px + Z.y * py) + (Z.z * pz + Z.w);
				}
				else if (head & RecOffset)
				{
					const float4 O = load(at++);
					qx = px + O.x; qy = py + O.y; qz = pz + O.z;
				}
				acc = TapeBrush(op, h, qx, qy, qz);
				if (head & RecScale) acc = acc * load(at).x;
				if (e >= count) break;
				if (!(head & RecThenSet)) continue;
				op = x & 0xFFu;
				at = base + (int)(x >> 16);
			}
			else if (op >= OpUnion && op <= OpBlendDiff)
			{
				--depth;
				left = spill[(depth - 1) * stride];
			}
			if (op >= OpUnion && op <= OpBlendDiff) acc = TapeSet(op, left, acc, op >= OpBlendUnion ? load(at).y : 0.0f);
			else if (op == OpFlate) acc = acc - load(at).y;
			else acc = op == OpTapeNegate ? -acc : acc + 0.0f;
			if (++e >= count) break;
			x = event(e).x;
		}
		return acc;
	}

	// The whole distance program at one point.
	static __device__ __noinline__ float RunWholePoint(const float4* __restrict__ code, int pc, float x, float y, float z, float* spill, int stride)
	{
		const float px[1] = { x }, py[1] = { y }, pz[1] = { z };
		float d[1];
		RunDistance<1>(code, pc, px, py, pz, d, spill, stride);
		return d[0];
	}

	// The whole distance program at one pair of points, where there is no tape.  Out of line:
	// rare beside the tapes, and the callers' code stays small.
	static __device__ __noinline__ float2 RunWholePair(const float4* __restrict__ code, int pc, float2 px, float2 py, float2 pz, float2* spill,
		int stride)
	{
		const float2 x[1] = { px }, y[1] = { py }, z[1] = { pz };
		float2 d[1];
		RunDistancePairs<1>([&](int q) { return __ldg(code + q); }, pc, x, y, z, d, spill, stride);
		return d[0];
	}

	// A brush's distance in a surface program (RunSurfacePair's step): T the translation and
	// scale, Q the inverse quaternion as (w, x, y, z).
	template<bool Compact = true>
	__device__ __forceinline__ float2 SurfaceBrushStep(uint32_t op, const float4& h, const float4& Q, const float4& T, float2 px, float2 py,
		float2 pz, const PairUnits& u)
	{
		const float2 vx = Sub2(px, Pair(T.x), u), vy = Sub2(py, Pair(T.y), u), vz = Sub2(pz, Pair(T.z), u);
		float2 ux, uy, uz, wx, wy, wz;
		CrossPair(Q.y, Q.z, Q.w, vx, vy, vz, ux, uy, uz, u);
		CrossPair(Q.y, Q.z, Q.w, ux, uy, uz, wx, wy, wz, u);
		float2 lx = Add2(vx, Mul2(Add2(Mul2(ux, Pair(Q.x), u), wx, u), Pair(2.0f), u), u);
		float2 ly = Add2(vy, Mul2(Add2(Mul2(uy, Pair(Q.x), u), wy, u), Pair(2.0f), u), u);
		float2 lz = Add2(vz, Mul2(Add2(Mul2(uz, Pair(Q.x), u), wz, u), Pair(2.0f), u), u);
		const bool scaled = T.w != 1.0f;    // x / 1 and x * 1 are x exactly
		if (scaled)
		{
			lx = DividePair(lx, T.w);
			ly = DividePair(ly, T.w);
			lz = DividePair(lz, T.w);
		}
		const float2 d = TapeBrush2<Compact>(op, h, lx, ly, lz, u);
		return scaled ? Mul2(d, Pair(T.w), u) : d;
	}

	// SDFNode::Eval at NP pairs of points (RunSurfacePair's steps) by the surface records a
	// tape names, those of the surface program at `base`.
	template<int NP, typename Load, typename Event>
	__device__ __forceinline__ void RunSurfaceTapePairs(Load load, int base, Event event, uint32_t count, const float2 (&px)[NP],
		const float2 (&py)[NP], const float2 (&pz)[NP], const PairUnits& u, float2 (&acc)[NP], float2* spill, int stride)
	{
		float2 left[NP];
#pragma unroll
		for (int j = 0; j < NP; ++j) acc[j] = left[j] = make_float2(0.0f, 0.0f);
		int depth = 0;
		uint32_t e = 0;
		uint2 ev = event(0u);
		for (;;)
		{
			uint32_t op = ev.x & 0xFFu;
			int at = base + (int)ev.y;
			if (op >= OpSphere && op <= OpPlane)
			{
				const uint32_t head = ev.x;
				if (++e < count) ev = event(e);
				if (!(head & RecThenSet))
				{
					if (depth > 0)
					{
#pragma unroll
						for (int j = 0; j < NP; ++j) spill[((depth - 1) * NP + j) * stride] = acc[j];
					}
					++depth;
				}
				const float4 h = load(at), Q = load(at + 1), T = load(at + 2);
#pragma unroll
				for (int j = 0; j < NP; ++j)
				{
					left[j] = acc[j];
					acc[j] = SurfaceBrushStep(op, h, Q, T, px[j], py[j], pz[j], u);
				}
				if (e >= count) break;
				if (!(head & RecThenSet)) continue;
				op = ev.x & 0xFFu;
				at = base + (int)ev.y;
			}
			else if (op >= OpUnion && op <= OpBlendDiff)
			{
				--depth;
#pragma unroll
				for (int j = 0; j < NP; ++j) left[j] = spill[((depth - 1) * NP + j) * stride];
			}
			if (op >= OpUnion && op <= OpBlendDiff)
			{
				const float k = op >= OpBlendUnion ? load(at).y : 0.0f;
#pragma unroll
				for (int j = 0; j < NP; ++j) acc[j] = TapeSet2(op, left[j], acc[j], k);
			}
			else if (op == OpFlate)
			{
				const float k = load(at).y;
#pragma unroll
				for (int j = 0; j < NP; ++j) acc[j] = Sub2(acc[j], Pair(k), u);
			}
			else
			{
#pragma unroll
				for (int j = 0; j < NP; ++j)
					acc[j] = op == OpTapeNegate ? make_float2(-acc[j].x, -acc[j].y) : make_float2(acc[j].x + 0.0f, acc[j].y + 0.0f);
			}
			if (++e >= count) break;
			ev = event(e);
		}
	}

	// RunTapePairs<1> (surface = false) or RunSurfaceTapePairs<1> (surface = true) from one copy
	// of code, for a kernel that runs both.
	template<typename Load, typename Event>
	__device__ __forceinline__ float2 RunEitherTapePair(bool surface, Load load, int base, Event event, uint32_t count, float2 px, float2 py,
		float2 pz, const PairUnits& u, float2* spill, int stride)
	{
		float2 acc = make_float2(0.0f, 0.0f), left = acc;
		int depth = 0;
		uint32_t e = 0;
		uint2 ev = event(0u);
		for (;;)
		{
			uint32_t op = ev.x & 0xFFu;
			int at = base + (surface ? (int)ev.y : (int)(ev.x >> 16));
			if (op >= OpSphere && op <= OpPlane)
			{
				const uint32_t head = ev.x;
				if (++e < count) ev = event(e);
				if (!(head & RecThenSet))
				{
					if (depth > 0) spill[(depth - 1) * stride] = acc;
					++depth;
				}
				left = acc;
				const float4 h = load(at);
				float2 qx = px, qy = py, qz = pz;
				float scale = 1.0f;
				if (surface)
				{
					const float4 Q = load(at + 1), T = load(at + 2);
					const float2 vx = Sub2(px, Pair(T.x), u), vy = Sub2(py, Pair(T.y), u), vz = Sub2(pz, Pair(T.z), u);
					float2 ux, uy, uz, wx, wy, wz;
					CrossPair(Q.y, Q.z, Q.w, vx, vy, vz, ux, uy, uz, u);
					CrossPair(Q.y, Q.z, Q.w, ux, uy, uz, wx, wy, wz, u);
					qx = Add2(vx, Mul2(Add2(Mul2(ux, Pair(Q.x), u), wx, u), Pair(2.0f), u), u);
					qy = Add2(vy, Mul2(Add2(Mul2(uy, Pair(Q.x), u), wy, u), Pair(2.0f), u), u);
					qz = Add2(vz, Mul2(Add2(Mul2(uz, Pair(Q.x), u), wz, u), Pair(2.0f), u), u);
					scale = T.w;
					if (scale != 1.0f)
					{
						qx = DividePair(qx, scale);
						qy = DividePair(qy, scale);
						qz = DividePair(qz, scale);
					}
				}
				else
				{
					++at;
					if (head & RecMatrix)
					{
						const float4 X = load(at), Y = load(at + 1), Z = load(at + 2);
						at += 3;
						qx = AffineRow2(X, px, py, pz, u);
						qy = AffineRow2(Y, px, py, pz, u);
						qz = AffineRow2(Z, px, py, pz, u);
					}
					else if (head & RecOffset)
					{
						const float4 O = load(at++);
						qx = Add2(px, Pair(O.x), u);
						qy = Add2(py, Pair(O.y), u);
						qz = Add2(pz, Pair(O.z), u);
					}
					if (head & RecScale) scale = load(at).x;
				}
				acc = TapeBrush2(op, h, qx, qy, qz, u);
				// x * 1 is x exactly; a scale record of 1 multiplies the same.
				if (scale != 1.0f) acc = Mul2(acc, Pair(scale), u);
				if (e >= count) break;
				if (!(head & RecThenSet)) continue;
				op = ev.x & 0xFFu;
				at = base + (surface ? (int)ev.y : (int)(ev.x >> 16));
			}
			else if (op >= OpUnion && op <= OpBlendDiff)
			{
				--depth;
				left = spill[(depth - 1) * stride];
			}
			if (op >= OpUnion && op <= OpBlendDiff) acc = TapeSet2(op, left, acc, op >= OpBlendUnion ? load(at).y : 0.0f);
			else if (op == OpFlate) acc = Sub2(acc, Pair(load(at).y), u);
			else acc = op == OpTapeNegate ? make_float2(-acc.x, -acc.y) : make_float2(acc.x + 0.0f, acc.y + 0.0f);
			if (++e >= count) break;
			ev = event(e);
		}
		return acc;
	}

	// The whole surface program at one pair of points, and GetMaterial's walk of it at one
	// point: where there is no tape.
	static __device__ __noinline__ float2 RunWholeSurfacePair(const float4* __restrict__ code, int pc, float2 px, float2 py, float2 pz,
		float2* spill, int stride)
	{
		return RunSurfacePair([&](int q) { return __ldg(code + q); }, pc, px, py, pz, spill, stride);
	}

	static __device__ __noinline__ int RunWholeMaterial(const float4* __restrict__ code, int pc, Vec3 p, float* spill, int stride)
	{
		const float px[1] = { p.x }, py[1] = { p.y }, pz[1] = { p.z };
		float d[1];
		int m = -1;
		RunSurfaceBatch<1>(code, pc, px, py, pz, d, 0, &m, spill, stride);
		return m;
	}

	// GetMaterial at one point over a painted tree without stencils (every brush has a
	// material, so intersections and blends choose by distance): the material list of a tape.
	// `spill` as RunSurfaceBatch<1>'s, which other threads of the block may run meanwhile.
	template<typename Load, typename Event>
	__device__ __forceinline__ int RunMaterialTape(Load load, int base, Event event, uint32_t count, Vec3 p, const PairUnits& u, float* spill,
		int stride)
	{
		// One brush left: its material, whatever its distance.
		if (count == 1) return __float_as_int(load(base + (int)event(0u).y + 3).x);
		float acc = 0.0f, left = 0.0f;
		int macc = -1, mleft = -1;
		int depth = 0;
		for (uint32_t e = 0; e < count; )
		{
			uint2 ev = event(e++);
			uint32_t op = ev.x & 0xFFu;
			int at = base + (int)ev.y;
			if (op >= OpSphere && op <= OpPlane)
			{
				const bool thenSet = (ev.x & RecThenSet) != 0;
				left = acc;
				mleft = macc;
				if (!thenSet)
				{
					if (depth > 0)
					{
						spill[(depth - 1) * 2 * stride] = acc;
						spill[((depth - 1) * 2 + 1) * stride] = __int_as_float(macc);
					}
					++depth;
				}
				const float4 h = load(at), Q = load(at + 1), T = load(at + 2), M = load(at + 3);
				acc = SurfaceBrushStep(op, h, Q, T, Pair(p.x), Pair(p.y), Pair(p.z), u).x;
				macc = __float_as_int(M.x);
				if (!thenSet) continue;
				if (e >= count) break;
				ev = event(e++);
				op = ev.x & 0xFFu;
				at = base + (int)ev.y;
			}
			else if (op >= OpUnion && op <= OpBlendDiff)
			{
				--depth;
				left = spill[(depth - 1) * 2 * stride];
				mleft = __float_as_int(spill[((depth - 1) * 2 + 1) * stride]);
			}
			else
			{
				if (op == OpFlate) acc = acc - load(at).y;
				else acc = acc + 0.0f;      // OpTapeAddZero; this list negates nothing
				continue;
			}
			const float k = op >= OpBlendUnion ? load(at).y : 0.0f;
			const float d = TapeSet2(op, Pair(left), Pair(acc), k).x;
			// SetNode::GetMaterial (sdf_evaluator.cpp:957-1012).
			const bool blend = op == OpBlendUnion || op == OpBlendInter;
			const bool takeLeft = (op == OpDiff || op == OpBlendDiff) || (blend ? (fabsf(left - d) <= fabsf(acc - d)) : (d == left));
			if (takeLeft) macc = mleft;
			acc = d;
		}
		return macc;
	}

	// A program read by a whole warp through a window in shared memory, 32 quads at a time,
	// the next 32 in flight: read one by one from memory, every record's first use waited for
	// L2, and a program of some hundred records held its warp longer than all others took
	// together.
	struct WindowReader
	{
		const float4* Code;
		int Quads;
		float4* Window;         // 64 quads: [32 * Chunk, 32 * Chunk + 64)
		int Chunk;
		float4 Ahead;           // this lane's quad of the 32 after those

		__device__ __forceinline__ float4 Fetch(int q) const { return __ldg(Code + min(q, Quads - 1)); }
		__device__ __forceinline__ void Open(const float4* code, int quads, float4* window)
		{
			const int lane = (int)(threadIdx.x & 31);
			Code = code;
			Quads = quads;
			Window = window;
			Chunk = 0;
			Window[lane] = Fetch(lane);
			Window[lane + 32] = Fetch(lane + 32);
			Ahead = Fetch(lane + 64);
			__syncwarp();
		}
		// Makes the record at pc readable: at most 33 quads from pc's chunk on.
		__device__ __forceinline__ void Seek(int pc)
		{
			const int lane = (int)(threadIdx.x & 31);
			while (Chunk < (pc >> 5))
			{
				__syncwarp();
				Window[(Chunk & 1) * 32 + lane] = Ahead;
				++Chunk;
				Ahead = Fetch(32 * Chunk + 64 + lane);
				__syncwarp();
			}
		}
		__device__ __forceinline__ float4 Load(int q) const { return Window[q & 63]; }
	};

	// A distance brush's distance at two points, from its record's quads, and the size its float
	// error goes with (its scale apart: DeviceProgram::Slack).
	template<typename Load>
	__device__ __forceinline__ float2 DistanceBrush(Load load, uint32_t head, float2 px, float2 py, float2 pz, const PairUnits& u, float2& size)
	{
		const float2 x[1] = { px }, y[1] = { py }, z[1] = { pz };
		float2 qx[1], qy[1], qz[1], d[1];
		float4 h;
		BrushStep<1, false>(load, 0, head, x, y, z, u, qx, qy, qz, h, d);
		const float sizes = fabsf(h.y) + fabsf(h.z) + fabsf(h.w);
		size = make_float2(fabsf(qx[0].x) + fabsf(qy[0].x) + fabsf(qz[0].x) + sizes + fabsf(d[0].x),
			fabsf(qx[0].y) + fabsf(qy[0].y) + fabsf(qz[0].y) + sizes + fabsf(d[0].y));
		return d[0];
	}

	// What BuildTape reads: the records of a program in order, each with its event.
	//
	// A cell's distance program; events name the surface records too (the same brushes and
	// operators in the same order, a brush 4 quads and an operator 1).
	struct DistanceSource
	{
		WindowReader In;
		int Pc = 0, Surface = 0;

		__device__ __forceinline__ uint32_t Head()
		{
			In.Seek(Pc);
			return ProgramHead(In.Load(Pc).x);
		}
		__device__ __forceinline__ uint2 Event(uint32_t head) const { return make_uint2(((uint32_t)Pc << 16) | (head & ~RecThenSet), (uint32_t)Surface); }
		__device__ __forceinline__ float Operand() const { return In.Load(Pc).y; }
		__device__ __forceinline__ void Advance(uint32_t head)
		{
			Pc += DistanceRecordQuads(head);
			Surface += (head & 0xFFu) <= OpPlane ? 4 : 1;
		}
		__device__ __forceinline__ float2 Brush(uint32_t head, float2 px, float2 py, float2 pz, const PairUnits& u, float2& size) const
		{
			return DistanceBrush([&](int q) { return In.Load(Pc + q); }, head, px, py, pz, u, size);
		}
	};

	__device__ __forceinline__ float2 SurfaceBrushSize(float4 h, float4 T, float2 px, float2 py, float2 pz, float2 d)
	{
		const float sizes = (fabsf(h.y) + fabsf(h.z) + fabsf(h.w)) * fabsf(T.w) + fabsf(T.x) + fabsf(T.y) + fabsf(T.z);
		return make_float2(fabsf(px.x) + fabsf(py.x) + fabsf(pz.x) + sizes + fabsf(d.x),
			fabsf(px.y) + fabsf(py.y) + fabsf(pz.y) + sizes + fabsf(d.y));
	}

	// A surface program (stencils' masks are passed over: they change no distance).
	struct SurfaceSource
	{
		WindowReader In;
		int Pc = 0;

		__device__ __forceinline__ uint32_t Head()
		{
			for (;;)
			{
				In.Seek(Pc);
				const float4 h = In.Load(Pc);
				const uint32_t head = __float_as_uint(h.x) & (0xFFu | RecThenSet);
				if ((head & 0xFFu) != OpMaskBegin) return head;
				Pc += 1 + (int)__float_as_uint(h.y);
			}
		}
		__device__ __forceinline__ uint2 Event(uint32_t head) const { return make_uint2(head & ~RecThenSet, (uint32_t)Pc); }
		__device__ __forceinline__ float Operand() const { return In.Load(Pc).y; }
		__device__ __forceinline__ void Advance(uint32_t head) { Pc += (head & 0xFFu) <= OpPlane ? 4 : 1; }
		__device__ __forceinline__ float2 Brush(uint32_t head, float2 px, float2 py, float2 pz, const PairUnits& u, float2& size) const
		{
			const float4 h = In.Load(Pc), T = In.Load(Pc + 2);
			const float2 d = SurfaceBrushStep<false>(head & 0xFFu, h, In.Load(Pc + 1), T, px, py, pz, u);
			size = SurfaceBrushSize(h, T, px, py, pz, d);
			return d;
		}
	};

	// The surface records that a tape of a larger box has left: eight events at a time, four
	// quads each, with the next eight in flight.
	struct SurfaceEventSource
	{
		const float4* Code;     // the surface program
		const uint2* Events;
		int Count;
		float4* Window;         // 16 events x 4 quads
		uint2* Heads;           // 16 events
		int At = 0, Chunk = 0;
		float4 Ahead;           // of this lane's event of the chunk after the two in the window,
		uint2 AheadEvent, NextEvent;    // its event, and that of the chunk after it

		__device__ __forceinline__ uint2 FetchEvent(int chunk) const
		{
			const int e = chunk * 8 + (int)((threadIdx.x & 31) >> 2);
			return e < Count ? __ldg(Events + e) : make_uint2(0u, 0u);
		}
		__device__ __forceinline__ float4 FetchQuad(uint2 ev) const
		{
			const int q = (int)(threadIdx.x & 3);
			const uint32_t op = ev.x & 0xFFu;
			const bool brush = op >= OpSphere && op <= OpPlane;
			return brush || (q == 0 && op != 0u && op < OpTapeNegate) ? __ldg(Code + ev.y + q) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
		}
		__device__ __forceinline__ void Put(int half, uint2 ev, float4 quad)
		{
			const int lane = (int)(threadIdx.x & 31);
			Window[half * 32 + lane] = quad;
			if ((lane & 3) == 0) Heads[half * 8 + (lane >> 2)] = ev;
		}
		__device__ __forceinline__ void Open(const float4* code, const uint2* events, int count, float4* window, uint2* heads)
		{
			Code = code;
			Events = events;
			Count = count;
			Window = window;
			Heads = heads;
			const uint2 e0 = FetchEvent(0), e1 = FetchEvent(1);
			AheadEvent = FetchEvent(2);
			NextEvent = FetchEvent(3);
			Put(0, e0, FetchQuad(e0));
			Put(1, e1, FetchQuad(e1));
			Ahead = FetchQuad(AheadEvent);
			__syncwarp();
		}
		__device__ __forceinline__ uint32_t Head()
		{
			while (Chunk < (At >> 3))
			{
				__syncwarp();
				Put(Chunk & 1, AheadEvent, Ahead);
				++Chunk;
				AheadEvent = NextEvent;
				Ahead = FetchQuad(AheadEvent);
				NextEvent = FetchEvent(Chunk + 3);
				__syncwarp();
			}
			return At < Count ? Heads[At & 15].x & 0xFFFFu : OpStop;
		}
		__device__ __forceinline__ float4 Quad(int q) const { return Window[(At & 15) * 4 + q]; }
		__device__ __forceinline__ uint2 Event(uint32_t head) const { return make_uint2(head & ~RecThenSet, Heads[At & 15].y); }
		__device__ __forceinline__ float Operand() const { return Quad(0).y; }
		__device__ __forceinline__ void Advance(uint32_t) { ++At; }
		__device__ __forceinline__ float2 Brush(uint32_t head, float2 px, float2 py, float2 pz, const PairUnits& u, float2& size) const
		{
			const float4 h = Quad(0), T = Quad(2);
			const float2 d = SurfaceBrushStep<false>(head & 0xFFu, h, Quad(1), T, px, py, pz, u);
			size = SurfaceBrushSize(h, T, px, py, pz, d);
			return d;
		}
	};

	// The same for distance records: four events at a time, eight lanes each (a brush takes up to
	// five quads), with the next four in flight.
	struct DistanceEventSource
	{
		const float4* Code;     // the distance program
		const uint2* Events;
		int Count;
		float4* Window;         // 8 events x 8 quads
		uint2* Heads;           // 8 events
		int At = 0, Chunk = 0;
		float4 Ahead;           // of this lane's event of the chunk after the two in the window,
		uint2 AheadEvent, NextEvent;    // its event, and that of the chunk after it

		__device__ __forceinline__ uint2 FetchEvent(int chunk) const
		{
			const int e = chunk * 4 + (int)((threadIdx.x & 31) >> 3);
			return e < Count ? __ldg(Events + e) : make_uint2(0u, 0u);
		}
		__device__ __forceinline__ float4 FetchQuad(uint2 ev) const
		{
			const int q = (int)(threadIdx.x & 7);
			const uint32_t op = ev.x & 0xFFu;
			return op != 0u && op < OpTapeNegate && q < DistanceRecordQuads(ev.x) ? __ldg(Code + (ev.x >> 16) + q) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
		}
		__device__ __forceinline__ void Put(int half, uint2 ev, float4 quad)
		{
			const int lane = (int)(threadIdx.x & 31);
			Window[half * 32 + lane] = quad;
			if ((lane & 7) == 0) Heads[half * 4 + (lane >> 3)] = ev;
		}
		__device__ __forceinline__ void Open(const float4* code, const uint2* events, int count, float4* window, uint2* heads)
		{
			Code = code;
			Events = events;
			Count = count;
			Window = window;
			Heads = heads;
			const uint2 e0 = FetchEvent(0), e1 = FetchEvent(1);
			AheadEvent = FetchEvent(2);
			NextEvent = FetchEvent(3);
			Put(0, e0, FetchQuad(e0));
			Put(1, e1, FetchQuad(e1));
			Ahead = FetchQuad(AheadEvent);
			__syncwarp();
		}
		__device__ __forceinline__ uint32_t Head()
		{
			while (Chunk < (At >> 2))
			{
				__syncwarp();
				Put(Chunk & 1, AheadEvent, Ahead);
				++Chunk;
				AheadEvent = NextEvent;
				Ahead = FetchQuad(AheadEvent);
				NextEvent = FetchEvent(Chunk + 3);
				__syncwarp();
			}
			return At < Count ? Heads[At & 7].x & 0xFFFFu : OpStop;
		}
		__device__ __forceinline__ uint2 Event(uint32_t) const { const uint2 ev = Heads[At & 7]; return make_uint2(ev.x & ~RecThenSet, ev.y); }
		__device__ __forceinline__ float Operand() const { return Window[(At & 7) * 8].y; }
		__device__ __forceinline__ void Advance(uint32_t) { ++At; }
		__device__ __forceinline__ float2 Brush(uint32_t head, float2 px, float2 py, float2 pz, const PairUnits& u, float2& size) const
		{
			return DistanceBrush([&](int q) { return Window[(At & 7) * 8 + q]; }, head, px, py, pz, u, size);
		}
	};

	// The source's program at a pair of points a lane, by all lanes of a warp.
	template<typename Source>
	__device__ __forceinline__ float2 RunSourcePair(Source& src, float2 px, float2 py, float2 pz, const PairUnits& u, float2* spill, int stride)
	{
		float2 acc = make_float2(0.0f, 0.0f), left = acc;
		int depth = 0;
		for (int guard = 0; guard < (1 << 24); ++guard)
		{
			uint32_t head = src.Head();
			uint32_t op = head & 0xFFu;
			if (op >= OpSphere && op <= OpPlane)
			{
				const bool thenSet = (head & RecThenSet) != 0;
				left = acc;
				if (!thenSet)
				{
					if (depth > 0) spill[(depth - 1) * stride] = acc;
					++depth;
				}
				float2 size;
				acc = src.Brush(head, px, py, pz, u, size);
				src.Advance(head);
				if (!thenSet) continue;
				head = src.Head();
				op = head & 0xFFu;
			}
			else if (op >= OpUnion && op <= OpBlendDiff)
			{
				--depth;
				left = spill[(depth - 1) * stride];
			}
			else if (op == OpFlate)
			{
				acc = Sub2(acc, Pair(src.Operand()), u);
				src.Advance(head);
				continue;
			}
			else
			{
				break;   // OpStop
			}
			acc = TapeSet2(op, left, acc, src.Operand());
			src.Advance(head);
		}
		return acc;
	}

	// The lists a warp writes its tape to, in shared memory.
	struct TapeLists
	{
		uint2* Value;           // events of the distance
		uint2* Material;        // events of the material walk (null: not wanted)
		uint2* Start;           // each operand on the stack: its first events (kMaxStack + 1)
		int Cap;                // events a list holds
	};

	struct TapeCounts
	{
		int Value, Material;
		bool Same;              // no difference was decided by its right operand: one list serves both
		float2 Distance;        // the program's values at this lane's two points,
		float2 Error;           // and the part of their rounding that grows with the operands
	};

	// Builds the tape of a program for a box, by all lanes of a warp: lane l's pair of points
	// are centres of two balls, and the balls of all lanes cover the box.  `reach` is how far
	// the difference of two operands can move inside a ball, with the fixed part of the
	// rounding (TapeReach); the part that grows with the operands' own coordinates (brushes
	// far from the box) is added here: each brush's float error is at most a few roundings of
	// its local coordinates and sizes, that of a flate or a blend a few of what goes in and of
	// its own width: `slack` times the largest of the brushes' sizes and of all widths together.
	// (Scales, rotations and widths are the whole tree's, from the host: looked at record by record
	// here they took 2 to 4 % of the building.)  Returns false when a list outgrows its room; with
	// Finish the rest of the program still runs then, for the distances.
	template<bool Materials, bool Finish = false, typename Source>
	__device__ __forceinline__ bool BuildTape(Source& src, float2 px, float2 py, float2 pz, float reach, float slack, float widths, const PairUnits& u,
		float2* spill, int stride, const TapeLists& ts, TapeCounts& out)
	{
		const int lane = (int)(threadIdx.x & 31);
		float2 acc = make_float2(0.0f, 0.0f), left = acc;
		float2 size = make_float2(widths, widths);
		int depth = 0;
		int nv = 0, nm = 0;
		bool same = true, full = false;
		// [from, to) of a list moves down to `down`.
		auto move = [&](uint2* list, int down, int from, int to)
		{
			for (int i = 0; from + i < to; i += 32)
			{
				uint2 ev = make_uint2(0u, 0u);
				if (from + i + lane < to) ev = list[from + i + lane];
				__syncwarp();
				if (from + i + lane < to) list[down + i + lane] = ev;
				__syncwarp();
			}
		};
		for (int guard = 0; guard < (1 << 24); ++guard)
		{
			if (nv + 4 > ts.Cap || (Materials && nm + 4 > ts.Cap))
			{
				if (!Finish) return false;
				full = true;
			}
			// A list that is full: nothing is left out any more, and what is written goes over its start.
			if (Finish && full) nv = nm = 0;
			uint32_t head = src.Head();
			uint32_t op = head & 0xFFu;
			int rv = nv, rm = nm;       // first events of the right operand
			if (op >= OpSphere && op <= OpPlane)
			{
				const bool thenSet = (head & RecThenSet) != 0;
				left = acc;
				if (!thenSet)
				{
					if (depth > 0) spill[(depth - 1) * stride] = acc;
					ts.Start[depth] = make_uint2((uint32_t)nv, (uint32_t)nm);
					++depth;
				}
				const uint2 ev = src.Event(head);
				ts.Value[nv++] = ev;
				if (Materials) ts.Material[nm++] = ev;
				float2 own;
				acc = src.Brush(head, px, py, pz, u, own);
				size = make_float2(fmaxf(size.x, own.x), fmaxf(size.y, own.y));
				src.Advance(head);
				if (!thenSet) continue;
				head = src.Head();
				op = head & 0xFFu;
			}
			else if (op >= OpUnion && op <= OpBlendDiff)
			{
				--depth;
				const uint2 r = ts.Start[depth];
				rv = (int)r.x; rm = (int)r.y;
				left = spill[(depth - 1) * stride];
			}
			else if (op == OpStop)
			{
				break;
			}
			else
			{
				// Flate, or what an earlier tape put in.
				const uint2 ev = src.Event(head);
				ts.Value[nv++] = ev;
				if (Materials) ts.Material[nm++] = ev;
				if (op == OpFlate) acc = Sub2(acc, Pair(src.Operand()), u);
				else acc = op == OpTapeNegate ? make_float2(-acc.x, -acc.y) : make_float2(acc.x + 0.0f, acc.y + 0.0f);
				src.Advance(head);
				continue;
			}
			const float k = src.Operand();
			const bool blend = op >= OpBlendUnion;
			const bool diff = op == OpDiff || op == OpBlendDiff;
			const bool unions = op == OpUnion || op == OpBlendUnion;
			// s > 0 where the left operand wins: by more than the reach everywhere, it always does.
			const float2 s = unions ? make_float2(acc.x - left.x, acc.y - left.y)
				: diff ? make_float2(left.x + acc.x, left.y + acc.y) : make_float2(left.x - acc.x, left.y - acc.y);
			const float2 t = make_float2(reach + slack * size.x + (blend ? k : 0.0f), reach + slack * size.y + (blend ? k : 0.0f));
			const bool decides = (!blend || k > 0.0f) && !full;
			__syncwarp();       // every lane's list writes so far come before any slot is reused
			const bool leftWins = __all_sync(0xFFFFFFFFu, decides && s.x > t.x && s.y > t.y);
			const bool rightWins = __all_sync(0xFFFFFFFFu, decides && s.x < -t.x && s.y < -t.y);
			const uint2 l = ts.Start[depth - 1];
			const uint2 set = src.Event(head);
			const uint2 addZero = make_uint2(OpTapeAddZero, 0u);
			if (leftWins)
			{
				nv = rv;
				nm = rm;
				if (blend && !unions)
				{
					ts.Value[nv++] = addZero;
					if (Materials) ts.Material[nm++] = addZero;
				}
			}
			else
			{
				if (rightWins)
				{
					move(ts.Value, (int)l.x, rv, nv);
					nv -= rv - (int)l.x;
					if (diff) ts.Value[nv++] = make_uint2(OpTapeNegate, 0u);
					if (blend && !unions) ts.Value[nv++] = addZero;
				}
				else
				{
					// A right operand that is now a single brush is combined in its own step.
					if (nv - rv == 1 && (ts.Value[rv].x & 0xFFu) <= OpPlane) ts.Value[rv].x |= RecThenSet;
					ts.Value[nv++] = set;
				}
				if (Materials)
				{
					if (rightWins && !diff)
					{
						move(ts.Material, (int)l.y, rm, nm);
						nm -= rm - (int)l.y;
						if (blend && !unions) ts.Material[nm++] = addZero;
					}
					else
					{
						if (rightWins) same = false;
						if (nm - rm == 1 && (ts.Material[rm].x & 0xFFu) <= OpPlane) ts.Material[rm].x |= RecThenSet;
						ts.Material[nm++] = set;
					}
				}
			}
			acc = TapeSet2(op, left, acc, k);
			src.Advance(head);
		}
		__syncwarp();
		out.Value = nv;
		out.Material = nm;
		out.Same = same;
		out.Distance = acc;
		out.Error = make_float2(slack * size.x, slack * size.y);
		return !full;
	}

	// How far the difference of two operands can move inside a ball of radius r about a point
	// near c, for trees whose rotations are within 1e-3 of unit quaternions, and the rounding
	// of two operands at two points near c (as the brick test's margin, four times).
	__device__ __forceinline__ float TapeReach(float r, float cx, float cy, float cz, float rootClip)
	{
		return 2.0f * 1.01f * r + 2e-4f * (1.0f + fabsf(cx) + fabsf(cy) + fabsf(cz) + fabsf(rootClip));
	}

	// The gradient's evaluation points lie up to this far from the point itself.
	constexpr float kTetraReach = 1.8e-4f;
}
