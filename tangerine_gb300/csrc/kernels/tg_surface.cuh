// Per-cell pieces of naive surface nets shared by the dense and the brick-culled passes
// (third_party/naive-surface-nets/src/surface_nets.cpp:864-1121).
#pragma once

#include "tg_device.cuh"
#include "tg_kernels.hpp"

namespace tg
{
	struct CellGeom
	{
		int64_t sx, sy, sz;     // cells per axis
		int64_t nx, ny;         // lattice points per axis (x, y)
	};

	__device__ __forceinline__ CellGeom Geom(const GridSpec& g)
	{
		return { g.NX - 1, g.NY - 1, g.NZ - 1, g.NX, g.NY };
	}

	__device__ __forceinline__ float Corner(const float* __restrict__ lat, const CellGeom& cg, int64_t i, int64_t j, int64_t k)
	{
		return __ldg(lat + (k * cg.ny + j) * cg.nx + i);
	}

	// Corner order and edge list of the reference (surface_nets.cpp:889-901).
	static __constant__ int8_t kCornerOfs[8][3] = { {0,0,0},{1,0,0},{1,1,0},{0,1,0},{0,0,1},{1,0,1},{1,1,1},{0,1,1} };
	static __constant__ int8_t kEdges[12][2] = { {0,1},{1,2},{2,3},{3,0},{4,5},{5,6},{6,7},{7,4},{0,4},{1,5},{2,6},{3,7} };

	__device__ __forceinline__ void LoadCorners(const float* __restrict__ lat, const CellGeom& cg, int64_t i, int64_t j, int64_t k, float (&v)[8])
	{
		const int64_t base = (k * cg.ny + j) * cg.nx + i;
		const int64_t dy = cg.nx, dz = cg.nx * cg.ny;
		v[0] = __ldg(lat + base);
		v[1] = __ldg(lat + base + 1);
		v[2] = __ldg(lat + base + dy + 1);
		v[3] = __ldg(lat + base + dy);
		v[4] = __ldg(lat + base + dz);
		v[5] = __ldg(lat + base + dz + 1);
		v[6] = __ldg(lat + base + dz + dy + 1);
		v[7] = __ldg(lat + base + dz + dy);
	}

	__device__ __forceinline__ bool IsActive(const uint32_t* __restrict__ words, int64_t cell)
	{
		return (__ldg(words + (cell >> 5)) >> (cell & 31)) & 1u;
	}

	__device__ __forceinline__ uint32_t VertexOf(const uint32_t* __restrict__ words, const uint32_t* __restrict__ base, int64_t cell)
	{
		const uint32_t w = __ldg(words + (cell >> 5));
		return __ldg(base + (cell >> 5)) + __popc(w & ((1u << (cell & 31)) - 1u));
	}


	// Cell c's coordinates, in 32 bits: cell numbers fit, and a 64-bit division is some hundred
	// instructions.
	struct CellIndex { int64_t i, j, k; };

	__device__ __forceinline__ CellIndex CellAt(uint32_t c, const CellGeom& cg)
	{
		const uint32_t sx = (uint32_t)cg.sx, sy = (uint32_t)cg.sy, row = c / sx, k = row / sy;
		return { (int64_t)(c - row * sx), (int64_t)(row - k * sy), (int64_t)k };
	}

	// SecondLoopThunk's triangles (surface_nets.cpp:1016-1115) of the vertex of active cell c,
	// from triangle `out` on; vertex numbers less `first`.
	__device__ __forceinline__ void EmitCellFaces(const float* __restrict__ lat, const CellGeom& cg, const uint32_t* __restrict__ words,
		const uint32_t* __restrict__ base, uint32_t cell, uint32_t self, uint32_t first, uint32_t out, uint32_t* __restrict__ faces)
	{
		const CellIndex at = CellAt(cell, cg);
		const int64_t i = at.i, j = at.j, k = at.k, c = cell;
		if (i == 0 || j == 0 || k == 0) return;
		const int64_t dy = cg.sx, dz = cg.sx * cg.sy;
		const int64_t nb[6] = { c - 1, c - 1 - dy, c - dy, c - dy - dz, c - dz, c - 1 - dz };
		// All the neighbours' words at once, then all the numbers.
		uint32_t w[6];
		bool on[6];
		uint32_t id[6];
#pragma unroll
		for (int q = 0; q < 6; ++q) w[q] = __ldg(words + (nb[q] >> 5));
#pragma unroll
		for (int q = 0; q < 6; ++q)
		{
			on[q] = (w[q] >> (nb[q] & 31)) & 1u;
			id[q] = on[q] ? __ldg(base + (nb[q] >> 5)) + __popc(w[q] & ((1u << (nb[q] & 31)) - 1u)) - first : 0u;
		}
		// Directed edges (0,4), (3,0), (0,1) decide the winding (surface_nets.cpp:1041-1105).
		const float c0 = Corner(lat, cg, i, j, k);
		const float s[3][2] = { { c0, Corner(lat, cg, i, j, k + 1) }, { Corner(lat, cg, i, j + 1, k), c0 }, { c0, Corner(lat, cg, i + 1, j, k) } };
		constexpr int quads[3][3] = { {0, 1, 2}, {0, 5, 4}, {2, 3, 4} };
#pragma unroll
		for (int q = 0; q < 3; ++q)
		{
			if (!(on[quads[q][0]] && on[quads[q][1]] && on[quads[q][2]])) continue;
			const bool rising = s[q][1] > s[q][0];
			const uint32_t a = id[quads[q][0]], v2 = id[quads[q][1]], d = id[quads[q][2]];
			const uint32_t v1 = rising ? a : d, v3 = rising ? d : a;
			uint32_t* f = faces + (int64_t)out * 3;
			f[0] = self; f[1] = v1; f[2] = v2;
			f[3] = self; f[4] = v2; f[5] = v3;
			out += 2;
		}
	}

	// The sum of a cell's edge points whatever its values (infinities, NaN).
	static __device__ __noinline__ void CellSumGeneral(const float (&v)[8], float fi, float fj, float fk, float& sx, float& sy, float& sz)
	{
		sx = sy = sz = 0.0f;
#pragma unroll 1
		for (int e = 0; e < 12; ++e)
		{
			const int a = kEdges[e][0], b = kEdges[e][1];
			const float s1 = v[a], s2 = v[b];
			if ((s1 >= 0.0f) == (s2 >= 0.0f)) continue;
			const float p1x = fi + (float)kCornerOfs[a][0], p1y = fj + (float)kCornerOfs[a][1], p1z = fk + (float)kCornerOfs[a][2];
			const float p2x = fi + (float)kCornerOfs[b][0], p2y = fj + (float)kCornerOfs[b][1], p2z = fk + (float)kCornerOfs[b][2];
			const float t = (0.0f - s1) / (s2 - s1);
			sx = sx + (p1x + t * (p2x - p1x));
			sy = sy + (p1y + t * (p2y - p1y));
			sz = sz + (p1z + t * (p2z - p1z));
		}
	}

	// FirstLoopInnerThunk's vertex (surface_nets.cpp:915-965) for active cell c = (i, j, k)
	// at its rank `vid`, and the number of triangles SecondLoopThunk will emit for it
	// (surface_nets.cpp:1016-1115).
	__device__ __forceinline__ void EmitCellVertex(const float* __restrict__ lat, const GridSpec& g, const CellGeom& cg,
		const uint32_t* __restrict__ words, int64_t c, int64_t i, int64_t j, int64_t k, uint32_t vid,
		float* __restrict__ vertices, uint32_t* __restrict__ cubes, uint32_t* __restrict__ face_counts)
	{
		float v[8];
		LoadCorners(lat, cg, i, j, k, v);
		const float fi = (float)i, fj = (float)j, fk = (float)k;
		float sx = 0.0f, sy = 0.0f, sz = 0.0f;
		int count = 0;
		// An edge's point is its first corner and, along its axis, t or -t more: the other axes'
		// t * 0 changes nothing while t is a number from 0 to 1.  All edges are computed and the
		// bipolar ones counted, without branches.  With the edges looked up and taken one by one
		// the vertex pass took 1370 instructions a warp and was bound by issue (1.2 million vertices
		// 53 us), now 600 and half waits for memory (36).
		constexpr int kFrom[12] = { 0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3 }, kTo[12] = { 1, 2, 3, 0, 5, 6, 7, 4, 4, 5, 6, 7 };
		constexpr int kX[8] = { 0, 1, 1, 0, 0, 1, 1, 0 }, kY[8] = { 0, 0, 1, 1, 0, 0, 1, 1 }, kZ[8] = { 0, 0, 0, 0, 1, 1, 1, 1 };
		const float x[2] = { fi, fi + 1.0f }, y[2] = { fj, fj + 1.0f }, z[2] = { fk, fk + 1.0f };
		bool usual = true;
#pragma unroll
		for (int e = 0; e < 12; ++e)
		{
			const int a = kFrom[e], b = kTo[e];
			const float s1 = v[a], s2 = v[b];
			const bool bipolar = (s1 >= 0.0f) != (s2 >= 0.0f);
			const float t = (0.0f - s1) / (bipolar ? s2 - s1 : 1.0f);
			usual = usual && (!bipolar || (t >= 0.0f && t <= 1.0f));
			const int dx = kX[b] - kX[a], dy = kY[b] - kY[a], dz = kZ[b] - kZ[a];
			const float px = dx > 0 ? x[0] + t : dx < 0 ? x[1] - t : x[kX[a]];
			const float py = dy > 0 ? y[0] + t : dy < 0 ? y[1] - t : y[kY[a]];
			const float pz = dz > 0 ? z[0] + t : dz < 0 ? z[1] - t : z[kZ[a]];
			sx = bipolar ? sx + px : sx;
			sy = bipolar ? sy + py : sy;
			sz = bipolar ? sz + pz : sz;
			count += bipolar ? 1 : 0;
		}
		if (!usual) CellSumGeneral(v, fi, fj, fk, sx, sy, sz);
		const float n = (float)count;
		const float cx = sx / n, cy = sy / n, cz = sz / n;
		const float fsx = (float)cg.sx, fsy = (float)cg.sy, fsz = (float)cg.sz;
		const float maxx = g.X0 + fsx * g.DX, maxy = g.Y0 + fsy * g.DY, maxz = g.Z0 + fsz * g.DZ;
		vertices[(int64_t)vid * 3 + 0] = g.X0 + (maxx - g.X0) * (cx - 0.0f) / (fsx - 0.0f);
		vertices[(int64_t)vid * 3 + 1] = g.Y0 + (maxy - g.Y0) * (cy - 0.0f) / (fsy - 0.0f);
		vertices[(int64_t)vid * 3 + 2] = g.Z0 + (maxz - g.Z0) * (cz - 0.0f) / (fsz - 0.0f);
		cubes[vid] = (uint32_t)c;

		uint32_t faces = 0;
		if (i > 0 && j > 0 && k > 0)
		{
			const int64_t dy = cg.sx, dz = cg.sx * cg.sy;
			// neighbours 0..5: (i-1,j,k) (i-1,j-1,k) (i,j-1,k) (i,j-1,k-1) (i,j,k-1) (i-1,j,k-1)
			const bool n0 = IsActive(words, c - 1), n1 = IsActive(words, c - 1 - dy), n2 = IsActive(words, c - dy);
			const bool n3 = IsActive(words, c - dy - dz), n4 = IsActive(words, c - dz), n5 = IsActive(words, c - 1 - dz);
			if (n0 && n1 && n2) faces += 2;
			if (n0 && n5 && n4) faces += 2;
			if (n2 && n3 && n4) faces += 2;
		}
		face_counts[vid] = faces;
	}

	// SDFNode::Gradient's evaluation points (sdf_evaluator.cpp:298-333): the four
	// tetrahedral offsets for lanes 0..3, the point itself for lane 4.
	__device__ __forceinline__ Vec3 TetraPoint(Vec3 p, int lane)
	{
		const float h = 0.0001f;
		switch (lane)
		{
		case 0: return p + Vec3(h, -h, -h);
		case 1: return p + Vec3(-h, -h, h);
		case 2: return p + Vec3(-h, h, -h);
		case 3: return p + Vec3(h, h, h);
		default: return p;
		}
	}

	// SDFNode::Gradient (sdf_evaluator.cpp:298-333) from the five evaluations.
	__device__ __forceinline__ Vec3 GradientOf(const float* e)
	{
		const float h = 0.0001f;
		const Vec3 xyy(h, -h, -h), yyx(-h, -h, h), yxy(-h, h, -h), xxx(h, h, h);
		Vec3 g = xyy * e[0];
		g = g + yyx * e[1];
		g = g + yxy * e[2];
		g = g + xxx * e[3];
		const float ls = (g.x * g.x + g.y * g.y) + g.z * g.z;
		if (ls == 0.0f)
		{
			const float d = e[4];
			return Normalize(Vec3(e[0] - d, e[2] - d, e[1] - d));
		}
		return g / sqrtf(ls);
	}

	// The app's framed casts: mode 1 is Lua's magnet cast (lua_sdf.cpp:410-417, the direction is
	// normalize(target - origin)); mode 2 is SDFModel::RayMarch (sdf_model.cpp:261-266): origin
	// = Transform::ApplyInv (rotate by the inverse rotation after removing the translation, then
	// divide by the scale), direction rotated by the inverse rotation.  Mode 0: as they are.
	__device__ __forceinline__ void FrameRay(const RayFrame& f, Vec3& o, Vec3& d)
	{
		if (f.Mode == 1)
		{
			d = Normalize(d - o);
		}
		else if (f.Mode == 2)
		{
			const Quat qi = Inverse(Quat{ f.Rotation[0], f.Rotation[1], f.Rotation[2], f.Rotation[3] });
			o = Rotate(qi, o - Vec3(f.Translation[0], f.Translation[1], f.Translation[2])) / f.Scale;
			d = Rotate(qi, d);
		}
	}
}
