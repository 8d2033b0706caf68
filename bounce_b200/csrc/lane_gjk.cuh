// GJK for warps that advance one query per lane in step (toi.cu, the shape
// casts of queries.cu): the same arithmetic as gjk.cuh's gjk_cached, cut into
// the pieces a warp runs together, with the simplex in shared memory where
// rolled loops can index it. The pieces are kept small: written out inline at
// every place they are used, the kernels outgrow the instruction cache.
#pragma once

#include "collide_common.cuh"

// Shared memory of one warp is an array of rows, one word per lane; the odd
// row length keeps both a row and a column free of bank conflicts.
constexpr uint32_t LANE_ROW = 33;

// A proxy (b3GJKProxy): a hull's vertices, or the shape's own, which are the
// first words of its params (sphere, capsule and triangle alike). ROW: the
// distance between words of the params.
template <uint32_t ROW>
struct LaneProxy
{
	const float4* gv; // hull vertices or nullptr
	const float* lv;  // the params
	uint32_t count;

	// b3GJKProxy::Set (gjk.cpp:37-95); returns the radius, which follows the
	// vertices in the params (a hull's is their first word).
	__device__ __forceinline__ float set(const DevScene& S, uint32_t type, uint32_t hull, const float* params)
	{
		static_assert(B3G_SHAPE_SPHERE == 0 && B3G_SHAPE_CAPSULE == 1 && B3G_SHAPE_TRIANGLE == 2, "vertex counts");
		gv = nullptr;
		lv = params;
		if (type <= B3G_SHAPE_TRIANGLE)
		{
			count = type + 1u; // sphere 1, capsule 2, triangle 3
			return lv[3 * count * ROW];
		}
		const HullDesc h = S.hulls[hull];
		gv = S.hverts + h.vOff;
		count = h.vCnt;
		return lv[0];
	}

	__device__ __forceinline__ V3 vertex(uint32_t i) const
	{
		if (gv)
		{
			const float4 w = __ldg(gv + i);
			return V3{w.x, w.y, w.z};
		}
		return V3{lv[3 * i * ROW], lv[(3 * i + 1) * ROW], lv[(3 * i + 2) * ROW]};
	}

	// b3GJKProxy::GetSupportIndex (gjk_proxy.h:72-86): first maximum. A
	// hull's vertices load four at a time. Out of line: one copy for both
	// proxies.
	__device__ __noinline__ uint32_t support(V3 d) const
	{
		uint32_t index = 0;
		if (gv)
		{
			float best = 0.0f;
			for (uint32_t i0 = 0; i0 < count; i0 += 4)
			{
				float4 w[4];
#pragma unroll
				for (uint32_t k = 0; k < 4; ++k)
					w[k] = __ldg(gv + min(i0 + k, count - 1u));
#pragma unroll
				for (uint32_t k = 0; k < 4; ++k)
				{
					const float proj = dot(d, V3{w[k].x, w[k].y, w[k].z});
					// The last vertex repeats past the end: never above itself.
					const bool take = i0 + k == 0u || proj > best;
					best = take ? proj : best;
					index = take ? i0 + k : index;
				}
			}
			return index;
		}
		float best = dot(d, vertex(0));
		for (uint32_t i = 1; i < count; ++i)
		{
			const float proj = dot(d, vertex(i));
			if (proj > best)
			{
				best = proj;
				index = i;
			}
		}
		return index;
	}
};

// The simplex of a lane: per vertex the point (3 words), the weight and the
// two support indices, LANE_ROW words apart.
constexpr uint32_t LANE_SIMPLEX_WORDS = 24;

struct LaneSimplex
{
	float* mine;
	uint32_t count;
	float metric;   // of the last GJK's simplex (b3SimplexCache::metric)
	uint32_t steps; // support iterations of the GJK under way
	uint32_t save1[4], save2[4], saveCount;

	__device__ __forceinline__ float& word(uint32_t v, uint32_t k) const { return mine[(6 * v + k) * LANE_ROW]; }
	__device__ __forceinline__ V3 point(uint32_t v) const { return V3{word(v, 0), word(v, 1), word(v, 2)}; }
	__device__ __forceinline__ uint32_t index1(uint32_t v) const { return __float_as_uint(word(v, 4)); }
	__device__ __forceinline__ uint32_t index2(uint32_t v) const { return __float_as_uint(word(v, 5)); }
	__device__ __forceinline__ void set(uint32_t v, V3 p, float w, uint32_t i1, uint32_t i2) const
	{
		word(v, 0) = p.x, word(v, 1) = p.y, word(v, 2) = p.z;
		word(v, 3) = w;
		word(v, 4) = __uint_as_float(i1), word(v, 5) = __uint_as_float(i2);
	}

	// b3Simplex::GetMetric (gjk.cpp:881-912).
	__device__ __forceinline__ float size() const
	{
		if (count < 2u)
			return 0.0f;
		const V3 A = point(0), E1 = point(1) - A;
		if (count == 2u)
			return len(A - point(1));
		const V3 E2 = point(2) - A;
		if (count == 3u)
			return len(cross(E1, E2));
		const float det = det3(E1, E2, point(3) - A);
		return signf_(det) * det;
	}

	// b3Simplex::ReadCache (gjk.cpp:820-868): the last simplex's support
	// points at these transforms, dropped for the arbitrary first vertex when
	// their metric changed by more than a factor of two or vanished.
	template <uint32_t RA, uint32_t RB>
	__device__ __forceinline__ void start(const LaneProxy<RA>& pA, const LaneProxy<RB>& pB, const XF& xfA, const XF& xfB)
	{
#pragma unroll 1
		for (uint32_t i = 0; i < count; ++i)
		{
			const uint32_t i1 = index1(i), i2 = index2(i);
			set(i, xmul(xfB, pB.vertex(i2)) - xmul(xfA, pA.vertex(i1)), 0.0f, i1, i2);
		}
		if (count > 1u)
		{
			const float now = size();
			if (now < 0.5f * metric || 2.0f * metric < now || now < B3G_EPSILON)
				count = 0;
		}
		if (count == 0u)
		{
			set(0, xmul(xfB, pB.vertex(0)) - xmul(xfA, pA.vertex(0)), 1.0f, 0u, 0u);
			count = 1;
		}
		steps = 0;
	}

	// An iteration of b3GJK's loop (gjk.cpp:683-768) up to the supports: their
	// directions in the proxies' frames; false when the GJK ends here.
	__device__ __forceinline__ bool directions(const XF& xfA, const XF& xfB, V3& dA, V3& dB)
	{
		SimplexRegion r;
		r.keep();
		const V3 A = point(0), B = point(1), C = point(2);
		saveCount = count;
#pragma unroll
		for (uint32_t i = 0; i < 4; ++i)
		{
			save1[i] = index1(i);
			save2[i] = index2(i);
		}
		if (count == 2u)
			r = solve2(A, B);
		else if (count == 3u)
			r = solve3(A, B, C);
		else if (count == 4u)
		{
			float w[4] = {word(0, 3), word(1, 3), word(2, 3), word(3, 3)};
			r = solve4(A, B, C, point(3), w);
			word(0, 3) = w[0], word(1, 3) = w[1], word(2, 3) = w[2], word(3, 3) = w[3];
		}
		if (r.n != 0u)
		{
			const V3 P0 = point(r.c0), P1 = point(r.c1), P2 = point(r.c2);
			const uint32_t i0 = index1(r.c0), i1 = index1(r.c1), i2 = index1(r.c2);
			const uint32_t j0 = index2(r.c0), j1 = index2(r.c1), j2 = index2(r.c2);
			const float s = 1.0f / r.div;
			set(0, P0, r.n == 1u ? 1.0f : s * r.w0, i0, j0);
			set(1, P1, s * r.w1, i1, j1);
			set(2, P2, s * r.w2, i2, j2);
			count = r.n;
		}
		// b3Simplex::GetSearchDirection
		V3 d = V3{0.0f, 0.0f, 0.0f};
		if (count < 4u)
		{
			const V3 X = point(0), E = point(1) - X, O = V3{0.0f, 0.0f, 0.0f} - X;
			d = O;
			if (count == 2u)
				d = cross(cross(E, O), E);
			else if (count == 3u)
			{
				d = cross(E, point(2) - X);
				if (!(dot(d, O) > 0.0f))
					d = -d;
			}
		}
		dA = rotc(xfA.q, -d);
		dB = rotc(xfB.q, d);
		return !(count == 4u || dot(d, d) < B3G_EPSILON * B3G_EPSILON);
	}

	// The rest of the iteration with the supports found; false when the GJK
	// ends with it.
	template <uint32_t RA, uint32_t RB>
	__device__ __forceinline__ bool add(const LaneProxy<RA>& pA, const LaneProxy<RB>& pB, const XF& xfA, const XF& xfB,
		uint32_t ia, uint32_t ib)
	{
		++steps;
		bool duplicate = false;
#pragma unroll
		for (uint32_t i = 0; i < 4; ++i)
			if (i < saveCount && ia == save1[i] && ib == save2[i])
				duplicate = true;
		if (duplicate)
			return false;
		set(count, xmul(xfB, pB.vertex(ib)) - xmul(xfA, pA.vertex(ia)), 0.0f, ia, ib);
		++count;
		return steps != 20u;
	}

	// The witness points (gjk.cpp:770-790) of the ended GJK, and its simplex's
	// metric for the next one.
	template <uint32_t RA, uint32_t RB>
	__device__ __forceinline__ void end(const LaneProxy<RA>& pA, const LaneProxy<RB>& pB, const XF& xfA, const XF& xfB,
		V3& P1, V3& P2)
	{
		P1 = P2 = V3{0.0f, 0.0f, 0.0f};
#pragma unroll 1
		for (uint32_t i = 0; i < count; ++i)
		{
			const float w = word(i, 3);
			const V3 x1 = xmul(xfA, pA.vertex(index1(i))), x2 = xmul(xfB, pB.vertex(index2(i)));
			const V3 q1 = count == 1u ? x1 : w * x1, q2 = count == 1u ? x2 : w * x2;
			P1 = i == 0u ? q1 : P1 + q1;
			P2 = i == 0u ? q2 : P2 + q2;
		}
		if (count == 4u)
			P2 = P1;
		metric = size();
	}
};
