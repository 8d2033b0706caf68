// Time of impact and GJK shape cast as batched device functions, one lane per
// query, with the reference's arithmetic:
//   b3TimeOfImpact(const b3TOIInput&)   time_of_impact.cpp:26-660 (the local
//       separating axis method on two sweeps: b3SeparationFunction, the
//       secant / bisection root finder, b3GJK with its simplex cache)
//   b3TimeOfImpact(aabb1, d1, aabb2, d2) time_of_impact.cpp:782-902
//   b3ShapeCast                          gjk.cpp:938-1102 (GJK ray cast)
// with b3GetFeaturePair (gjk_feature_pair.cpp:21-236) and
// b3Sweep::GetTransform (sweep.h:43-63).
#include <algorithm>

#include "lane_gjk.cuh"

static_assert(sizeof(b3g_toi_input) == 272, "b3g_toi_input: 68 words");
static_assert(sizeof(b3g_gjk_cast_input) == 192, "b3g_gjk_cast_input: 48 words");

namespace {

// b3Sweep::GetTransform (sweep.h:43-63) of the sweep in a lane's column, in
// the b3g_toi_input layout: localCenter, orientation0, worldCenter0, t0,
// orientation, worldCenter (sweep.h:28-41). Out of line: one copy of the code
// for both sweeps.
__device__ __noinline__ XF sweep_at(const float* s, uint32_t row, float t)
{
	auto v3_at = [&](uint32_t w) { return V3{s[w * row], s[(w + 1) * row], s[(w + 2) * row]}; };
	const V3 c = (1.0f - t) * v3_at(7) + t * v3_at(15);
	Q4 q1 = Q4{v3_at(3), s[6 * row]};
	const Q4 q2 = Q4{v3_at(11), s[14 * row]};
	if (qdot(q1, q2) < 0.0f)
		q1 = qneg(q1);
	const float u = 1.0f - t;
	Q4 q = Q4{u * q1.v + t * q2.v, u * q1.s + t * q2.s};
	qnormalize_inplace(q);
	XF xf;
	xf.p = c - rot(q, v3_at(0));
	xf.q = q;
	return xf;
}

// b3UniqueCount (math.h:84-104).
__device__ __forceinline__ uint32_t unique3(const uint32_t* v, uint32_t n)
{
	uint32_t count = 0;
	for (uint32_t i = 0; i < n; ++i)
	{
		uint32_t j = 0;
		while (j < n && v[i] != v[j])
			++j;
		count += i == j ? 1u : 0u;
	}
	return count;
}

struct FeaturePair
{
	uint32_t index1[3], count1, index2[3], count2;
};

// b3GetFeaturePair (gjk_feature_pair.cpp:21-236); counts 0 for the
// combinations the reference asserts never happen.
__device__ FeaturePair feature_pair(const GJKCache& cache)
{
	FeaturePair p;
	p.count1 = p.count2 = 0;
	for (int k = 0; k < 3; ++k)
		p.index1[k] = p.index2[k] = 0;
	const uint32_t n = cache.count;
	if (n == 0 || n > 3)
		return p;
	const uint32_t u1 = unique3(cache.index1, n), u2 = unique3(cache.index2, n);
	auto second = [](const uint32_t* v) { return v[0] == v[1] ? v[2] : v[1]; };
	if (n == 1)
	{
		p.count1 = p.count2 = 1;
		p.index1[0] = cache.index1[0];
		p.index2[0] = cache.index2[0];
		return p;
	}
	if (n == 2)
	{
		if (u1 == 2 && u2 == 2)
		{
			p.count1 = p.count2 = 2;
			p.index1[0] = cache.index1[0];
			p.index1[1] = cache.index1[1];
			p.index2[0] = cache.index2[0];
			p.index2[1] = cache.index2[1];
		}
		else if (u1 == 1)
		{
			p.count1 = 1;
			p.count2 = 2;
			p.index1[0] = cache.index1[0];
			p.index2[0] = cache.index2[0];
			p.index2[1] = cache.index2[1];
		}
		else if (u2 == 1)
		{
			p.count1 = 2;
			p.count2 = 1;
			p.index1[0] = cache.index1[0];
			p.index1[1] = cache.index1[1];
			p.index2[0] = cache.index2[0];
		}
		return p;
	}
	if (u1 == 1 && u2 == 3)
	{
		p.count1 = 1;
		p.count2 = 3;
		p.index1[0] = cache.index1[0];
		for (int k = 0; k < 3; ++k)
			p.index2[k] = cache.index2[k];
	}
	else if (u1 == 3 && u2 == 1)
	{
		p.count1 = 3;
		p.count2 = 1;
		for (int k = 0; k < 3; ++k)
			p.index1[k] = cache.index1[k];
		p.index2[0] = cache.index2[0];
	}
	else if (u1 == 2 && u2 == 2)
	{
		p.count1 = p.count2 = 2;
		p.index1[0] = cache.index1[0];
		p.index1[1] = second(cache.index1);
		p.index2[0] = cache.index2[0];
		p.index2[1] = second(cache.index2);
	}
	else if (u1 == 2 && u2 == 3)
	{
		p.count1 = 2;
		p.count2 = 3;
		p.index1[0] = cache.index1[0];
		p.index1[1] = second(cache.index1);
		for (int k = 0; k < 3; ++k)
			p.index2[k] = cache.index2[k];
	}
	else if (u1 == 3 && u2 == 2)
	{
		p.count1 = 3;
		p.count2 = 2;
		for (int k = 0; k < 3; ++k)
			p.index1[k] = cache.index1[k];
		p.index2[0] = cache.index2[0];
		p.index2[1] = second(cache.index2);
	}
	else if (u1 == 3 && u2 == 3)
	{
		p.count1 = p.count2 = 3;
		for (int k = 0; k < 3; ++k)
		{
			p.index1[k] = cache.index1[k];
			p.index2[k] = cache.index2[k];
		}
	}
	return p;
}

enum : uint32_t
{
	SEP_POINTS = 0,
	SEP_EDGE_A,
	SEP_FACE_A,
	SEP_EDGE_B,
	SEP_FACE_B,
	SEP_EDGES,
	SEP_NONE
};

// b3TOIOutput::State (time_of_impact.h:40-47).
enum : uint32_t
{
	ST_UNKNOWN = 0,
	ST_FAILED,
	ST_OVERLAPPED,
	ST_TOUCHING,
	ST_SEPARATED
};

// One query on a lane: its record stays in the lane's column of its warp's
// shared memory (lane_gjk.cuh).
constexpr uint32_t TOI_WORDS = sizeof(b3g_toi_input) / 4;
constexpr uint32_t TOI_ROW = LANE_ROW;
using ToiProxy = LaneProxy<TOI_ROW>;

// b3SeparationFunction (time_of_impact.cpp:26-461) for the feature pair the
// GJK ended with.
struct Separation
{
	uint32_t type;
	V3 localPoint, axis;
	bool parallel;

	__device__ __forceinline__ void init(const GJKCache& cache, const ToiProxy& pA, const ToiProxy& pB, const XF& xfA,
		const XF& xfB)
	{
		const FeaturePair fp = feature_pair(cache);
		const uint32_t countA = fp.count1, countB = fp.count2;
		parallel = false;
		localPoint = V3{0.0f, 0.0f, 0.0f};
		axis = V3{0.0f, 0.0f, 0.0f};
		type = SEP_NONE;
		if (countA == 0u)
			return;
		if (countA == 1 && countB == 1)
		{
			type = SEP_POINTS;
			const V3 A = xmul(xfA, pA.vertex(fp.index1[0]));
			const V3 B = xmul(xfB, pB.vertex(fp.index2[0]));
			axis = B - A;
			normalize_inplace(axis);
			return;
		}
		if (countA == 2 && countB == 2)
		{
			type = SEP_EDGES;
			const V3 A = pA.vertex(fp.index1[0]);
			const V3 B = pA.vertex(fp.index1[1]);
			const V3 C = xmult(xfA, xmul(xfB, pB.vertex(fp.index2[0])));
			const V3 D = xmult(xfA, xmul(xfB, pB.vertex(fp.index2[1])));
			const V3 E1 = B - A, E2 = D - C;
			const float L1 = len(E1), L2 = len(E2);
			const float kTol = 0.005f;
			const V3 E1_x_E2 = cross(E1, E2);
			const float L = len(E1_x_E2);
			if (L < (kTol * L1) * L2)
			{
				// Parallel edges: the closest points of the segments.
				V3 C1, C2;
				closest_on_segments(C1, C2, A, B, C, D);
				C1 = xmul(xfA, C1);
				C2 = xmul(xfA, C2);
				axis = C2 - C1;
				normalize_inplace(axis);
				parallel = true;
				return;
			}
			const V3 C1 = 0.5f * (A + B);
			const V3 C2 = 0.5f * (C + D);
			V3 N = (1.0f / L) * E1_x_E2;
			if (dot(N, C2 - C1) < 0.0f)
				N = -N;
			axis = N;
			localPoint = C1;
			return;
		}
		// An edge or face of one shape against a point of the other, in the
		// first shape's frame: the two sides run the same code.
		const bool ofA = (countA == 2 && countB == 1) || countA == 3;
		const uint32_t face = ofA ? countA : countB;
		const uint32_t i0 = ofA ? fp.index1[0] : fp.index2[0], i1 = ofA ? fp.index1[1] : fp.index2[1];
		const uint32_t i2 = ofA ? fp.index1[2] : fp.index2[2], io = ofA ? fp.index2[0] : fp.index1[0];
		const ToiProxy pf{ofA ? pA.gv : pB.gv, ofA ? pA.lv : pB.lv, 0u}, po{ofA ? pB.gv : pA.gv, ofA ? pB.lv : pA.lv, 0u};
		const XF xf = ofA ? xfA : xfB, xo = ofA ? xfB : xfA;
		const V3 A = pf.vertex(i0), B = pf.vertex(i1);
		const V3 X = xmult(xf, xmul(xo, po.vertex(io)));
		if (face == 3)
		{
			type = ofA ? SEP_FACE_A : SEP_FACE_B;
			V3 N = -cross(B - A, pf.vertex(i2) - A);
			if (dot(X - A, N) < 0.0f)
				N = -N;
			axis = N;
			localPoint = A;
		}
		else
		{
			type = ofA ? SEP_EDGE_A : SEP_EDGE_B;
			const V3 AB = B - A, AC = X - A;
			axis = rot(xf.q, cross(cross(AB, AC), AB));
		}
		normalize_inplace(axis);
	}

	// Whether a face (or the plane of two edges) of shape A / of shape B is
	// the reference.
	__device__ __forceinline__ bool plane_a() const { return type == SEP_FACE_A || (type == SEP_EDGES && !parallel); }
	__device__ __forceinline__ bool plane_b() const { return type == SEP_FACE_B; }

	// The support directions of FindMinSeparation (zero where it looks for
	// none), in the shapes' frames.
	__device__ __forceinline__ void directions(const XF& xfA, const XF& xfB, V3& dA, V3& dB) const
	{
		V3 N = axis;
		if (plane_a())
			N = rot(xfA.q, axis);
		else if (plane_b())
			N = rot(xfB.q, axis);
		// The point of A is looked for along the axis where the axis leads from A
		// to B, against it otherwise; B's the other way round.
		const bool fromB = type == SEP_EDGE_B || type == SEP_FACE_B;
		const V3 M = -N;
		dA = rotc(xfA.q, fromB ? M : N);
		dB = rotc(xfB.q, fromB ? N : M);
	}

	// FindMinSeparation's and Evaluate's distance of the points indexA,
	// indexB.
	__device__ __forceinline__ float value(const ToiProxy& pA, const ToiProxy& pB, const XF& xfA, const XF& xfB,
		uint32_t indexA, uint32_t indexB) const
	{
		V3 N = axis;
		if (plane_a())
			N = rot(xfA.q, axis);
		else if (plane_b())
			N = rot(xfB.q, axis);
		const V3 A = xmul(xfA, plane_a() ? localPoint : pA.vertex(indexA));
		const V3 B = xmul(xfB, plane_b() ? localPoint : pB.vertex(indexB));
		const bool fromB = type == SEP_EDGE_B || type == SEP_FACE_B;
		return dot(fromB ? A - B : B - A, N);
	}
};

// b3TimeOfImpact(aabb1, d1, aabb2, d2) (time_of_impact.cpp:782-902).
__device__ void toi_aabbs(const float* in, uint32_t& state, float& tOut)
{
	const float aLo[3] = {in[0], in[1], in[2]}, aHi[3] = {in[3], in[4], in[5]};
	const float d1[3] = {in[6], in[7], in[8]};
	const float bLo[3] = {in[9], in[10], in[11]}, bHi[3] = {in[12], in[13], in[14]};
	const float d2[3] = {in[15], in[16], in[17]};
	AABB A, B;
	A.lo = V3{aLo[0], aLo[1], aLo[2]};
	A.hi = V3{aHi[0], aHi[1], aHi[2]};
	B.lo = V3{bLo[0], bLo[1], bLo[2]};
	B.hi = V3{bHi[0], bHi[1], bHi[2]};
	if (aabb_overlap(A, B))
	{
		state = ST_OVERLAPPED;
		tOut = 0.0f;
		return;
	}
	float t1[3] = {0.0f, 0.0f, 0.0f}, t2[3] = {1.0f, 1.0f, 1.0f};
	for (int i = 0; i < 3; ++i)
	{
		const float d = d2[i] - d1[i];
		if (d == 0.0f && (aLo[i] > bHi[i] || aHi[i] < bLo[i]))
		{
			state = ST_SEPARATED;
			tOut = 1.0f;
			return;
		}
		if (d < 0.0f)
		{
			if (bHi[i] < aLo[i])
			{
				state = ST_SEPARATED;
				tOut = 1.0f;
				return;
			}
			t2[i] = (aLo[i] - bHi[i]) / d;
			if (bLo[i] > aHi[i])
			{
				t1[i] = (aHi[i] - bLo[i]) / d;
				if (t1[i] >= 1.0f)
				{
					state = ST_SEPARATED;
					tOut = 1.0f;
					return;
				}
			}
		}
		if (d > 0.0f)
		{
			if (bLo[i] > aHi[i])
			{
				state = ST_SEPARATED;
				tOut = 1.0f;
				return;
			}
			t2[i] = (aHi[i] - bLo[i]) / d;
			if (bHi[i] < aLo[i])
			{
				t1[i] = (aLo[i] - bHi[i]) / d;
				if (t1[i] >= 1.0f)
				{
					state = ST_SEPARATED;
					tOut = 1.0f;
					return;
				}
			}
		}
	}
	const float t1max = fmaxr(t1[0], fmaxr(t1[1], t1[2]));
	const float t2min = fminr(t2[0], fminr(t2[1], t2[2]));
	if (t1max > t2min)
	{
		state = ST_SEPARATED;
		tOut = 0.0f;
		return;
	}
	state = ST_TOUCHING;
	tOut = t1max;
}

// b3ShapeCast (gjk.cpp:938-1102): GJK ray cast of proxy 2 along r against
// proxy 1 (radii included). Returns false when they do not meet within r.
__device__ bool gjk_ray_cast(const XF& xf1, const GProxy& p1, const XF& xf2, const GProxy& p2, V3 r, float& tOut,
	V3& point, V3& normalOut, uint32_t& iterations)
{
	const float r1 = p1.radius, r2 = p2.radius;
	const float radius = r1 + r2;
	float t = 0.0f;
	V3 n = V3{0.0f, 0.0f, 0.0f};
	uint32_t index1 = gp_support(p1, rotc(xf1.q, -r));
	uint32_t index2 = gp_support(p2, rotc(xf2.q, r));
	V3 w1 = xmul(xf1, gp_vertex(p1, index1));
	V3 w2 = xmul(xf2, gp_vertex(p2, index2));
	V3 v = w1 - w2;
	Simplex sx;
	sx.count = 0;
	for (int i = 0; i < 4; ++i)
	{
		sx.v[i].point1 = sx.v[i].point2 = sx.v[i].point = V3{0.0f, 0.0f, 0.0f};
		sx.v[i].weight = 0.0f;
		sx.v[i].index1 = sx.v[i].index2 = 0u;
	}
	uint32_t save1[4], save2[4];
	uint32_t saveCount = 0;
	const uint32_t kMaxIters = 20;
	const float kTolerance = 10.0f * B3G_EPSILON;
	float maxTolerance = 1.0f;
	uint32_t iter = 0;
	while (iter < kMaxIters && fabsr(len2(v) - radius * radius) > kTolerance * maxTolerance)
	{
		index1 = gp_support(p1, rotc(xf1.q, -v));
		index2 = gp_support(p2, rotc(xf2.q, v));
		w1 = xmul(xf1, gp_vertex(p1, index1));
		w2 = xmul(xf2, gp_vertex(p2, index2));
		const V3 p = w1 - w2;
		const float vp = dot(v, p);
		const float vr = dot(v, r);
		if (vp - radius > t * vr)
		{
			if (vr > 0.0f)
			{
				t = (vp - radius) / vr;
				if (t > 1.0f)
				{
					iterations = iter;
					return false;
				}
				n = -v;
				sx.count = 0;
				saveCount = 0;
			}
			else
			{
				iterations = iter;
				return false;
			}
		}
		const V3 s = t * r;
		SVert vx;
		vx.index1 = index1;
		vx.point1 = w1;
		vx.index2 = index2;
		vx.point2 = w2;
		vx.point = p - s;
		vx.weight = 0.0f;
		bool duplicate = false;
		for (uint32_t i = 0; i < 4; ++i)
			if (i < saveCount && vx.index1 == save1[i] && vx.index2 == save2[i])
				duplicate = true;
		if (duplicate)
			break;
		if (sx.count == 0)
			sx.v[0] = vx;
		else if (sx.count == 1)
			sx.v[1] = vx;
		else if (sx.count == 2)
			sx.v[2] = vx;
		else
			sx.v[3] = vx;
		++sx.count;
		maxTolerance = -B3G_EPSILON;
#pragma unroll
		for (int i = 0; i < 4; ++i)
			if ((uint32_t)i < sx.count)
				maxTolerance = fmaxr(maxTolerance, len2(sx.v[i].point));
		saveCount = sx.count;
#pragma unroll
		for (int i = 0; i < 4; ++i)
		{
			save1[i] = sx.v[i].index1;
			save2[i] = sx.v[i].index2;
		}
		sx.solve();
		if (sx.count == 4)
			break;
		v = sx.closest();
		++iter;
	}
	V3 point1, point2;
	sx.closest_points(point1, point2);
	if (len2(v) > B3G_EPSILON * B3G_EPSILON)
		n = -v;
	normalize_inplace(n);
	tOut = t;
	point = point1 + r1 * n;
	normalOut = n;
	iterations = iter;
	return true;
}

__device__ __forceinline__ GProxy input_proxy(const DevScene& S, const float* w, uint32_t type, uint32_t hull)
{
	return convex_proxy(S, type, make_float4(w[0], w[1], w[2], w[3]), make_float4(w[4], w[5], w[6], w[7]),
		make_float4(w[8], w[9], w[10], w[11]), hull);
}

// b3TimeOfImpact(const b3TOIInput&) (time_of_impact.cpp:465-660), a query per
// lane. The reference's nested loops (GJK iterations, separations pushed back,
// root finding, all inside up to 20 rounds) are unrolled into a state per
// lane; the warp takes the step that most of its lanes wait for, for all
// lanes that wait for it, and a lane whose query is done takes the next of its
// warp's share. As nested loops the lanes of a warp sat in different copies of
// this code (5 of 32 active) and the kernel waited on the instruction cache
// for 13 of 17 cycles per instruction; for the same reason the code is kept
// small, with the query and its simplex in shared memory, where rolled loops
// can index them. Bound by issue (a third of the cycles, 9 lanes) and the
// instruction cache. Measured, 262,144 queries of mixed shapes: 10.5 ms
// before, 2.78 ms now (every lane one step of its own at a time: 3.10 ms).
//
// A feature pair the reference asserts never happens ends the query as failed.
enum : uint32_t
{
	TOI_START = 0, // a GJK at t1 from the simplex of the last one
	TOI_GJK,       // its iterations
	TOI_END,       // its distance, and the separation function
	TOI_MIN,       // the points of minimum separation at t2
	TOI_VALUE,     // a separation (one of the three below)
	TOI_STEPS,
	TOI_IDLE = TOI_STEPS
};
enum : uint32_t
{
	VALUE_MIN = 0, // at t2, of the points just found
	VALUE_AT1,     // at t1
	VALUE_ROOT     // at the root finder's time
};
constexpr uint32_t TOI_WARPS = 2;
constexpr uint32_t TOI_BLOCKS = 6; // per SM: 4 took 2.92 ms, 8 (128 registers, spills) 2.94 ms
constexpr uint32_t TOI_REFILL = 4; // lanes without a query before the warp brings new ones: 8 took 3.00 ms

__global__ void __launch_bounds__(TOI_WARPS * 32, TOI_BLOCKS) k_toi_sweeps(DevScene S, const float* in, uint32_t n,
	uint32_t share, uint32_t* out)
{
	__shared__ float record[TOI_WARPS][(TOI_WORDS + LANE_SIMPLEX_WORDS) * TOI_ROW];
	const uint32_t lane = threadIdx.x & 31u;
	float* const W = record[threadIdx.x >> 5];
	float* const mine = W + lane;
	const uint32_t warp = blockIdx.x * TOI_WARPS + (threadIdx.x >> 5);
	uint32_t next = min(warp * share, n);
	const uint32_t end = min(next + share, n);
	const float tolerance = 0.25f * B3G_LINEAR_SLOP;

	uint32_t state = TOI_IDLE, query = 0;
	LaneSimplex sx;
	sx.mine = mine + TOI_WORDS * TOI_ROW;
	sx.count = sx.steps = sx.saveCount = 0;
	sx.metric = 0.0f;
	ToiProxy pA, pB;
	pA.gv = pB.gv = nullptr;
	pA.lv = mine + 4 * TOI_ROW;
	pB.lv = mine + 16 * TOI_ROW;
	pA.count = pB.count = 0;
	float target = 0.0f, tMax = 0.0f, t1 = 0.0f, t2 = 0.0f, a1 = 0.0f, a2 = 0.0f, s1 = 0.0f, s2 = 0.0f;
	float tRoot = 0.0f;
	uint32_t kind = VALUE_MIN;
	uint32_t iteration = 0, pushBack = 0, steps = 0, indexA = 0, indexB = 0; // steps: of the GJK or the root finder
	Separation sep;
	sep.type = SEP_NONE;
	sep.localPoint = sep.axis = V3{0.0f, 0.0f, 0.0f};
	sep.parallel = false;
	XF xfA, xfB;
	xfA.p = xfB.p = V3{0.0f, 0.0f, 0.0f};
	xfA.q = xfB.q = Q4{V3{0.0f, 0.0f, 0.0f}, 1.0f};

	for (;;)
	{
		// Lanes without a query take the warp's next ones; the warp brings each
		// record in together.
		const uint32_t idle = __ballot_sync(0xFFFFFFFFu, state == TOI_IDLE);
		if (idle == 0xFFFFFFFFu && next >= end)
			break;
		if (next < end && ((uint32_t)__popc(idle) >= TOI_REFILL || idle == 0xFFFFFFFFu))
		{
			uint32_t left = idle;
			const uint32_t first = next;
			while (left != 0u && next < end)
			{
				const uint32_t l = __ffs(left) - 1;
				left &= left - 1u;
				const float* r = in + TOI_WORDS * (size_t)next;
				for (uint32_t w = lane; w < TOI_WORDS; w += 32u)
					W[w * TOI_ROW + l] = r[w];
				++next;
			}
			__syncwarp();
			const uint32_t rank = __popc(idle & ((1u << lane) - 1u));
			if (state == TOI_IDLE && first + rank < next)
			{
				query = first + rank;
				const float rA = pA.set(S, __float_as_uint(mine[0]), __float_as_uint(mine[TOI_ROW]), mine + 4 * TOI_ROW);
				const float rB =
					pB.set(S, __float_as_uint(mine[2 * TOI_ROW]), __float_as_uint(mine[3 * TOI_ROW]), mine + 16 * TOI_ROW);
				target = fmaxr(B3G_LINEAR_SLOP, (rA + rB) - 3.0f * B3G_LINEAR_SLOP);
				tMax = mine[64 * TOI_ROW];
				t1 = 0.0f;
				iteration = 0;
				sx.count = 0;
				sx.metric = 0.0f;
				state = TOI_START;
			}
			__syncwarp();
		}
		// The step most lanes wait for (the later one of two: it ends queries).
		uint32_t step = TOI_START, most = 0;
#pragma unroll
		for (uint32_t k = 0; k < TOI_STEPS; ++k)
		{
			const uint32_t waiting = __popc(__ballot_sync(0xFFFFFFFFu, state == k));
			if (waiting >= most)
			{
				step = k;
				most = waiting;
			}
		}
		const bool active = state == step;
		// How the step ends a query: the state and time to write, or nothing.
		uint32_t how = ST_UNKNOWN;
		float tEnd = t1;
		if (step != TOI_GJK && step != TOI_END)
		{
			// The transforms at the lane's time (a GJK's stay for its
			// iterations, a minimum search's for its value).
			float t = t1;
			if (step == TOI_MIN)
				t = t2;
			else if (step == TOI_VALUE && kind == VALUE_ROOT && active)
			{
				t = 0.5f * (a1 + a2);
				if (steps & 1u)
					t = a1 + (target - s1) * (a2 - a1) / (s2 - s1);
				++steps;
				tRoot = t;
			}
			if (active && !(step == TOI_VALUE && kind == VALUE_MIN))
			{
				xfA = sweep_at(mine + 28 * TOI_ROW, TOI_ROW, t);
				xfB = sweep_at(mine + 46 * TOI_ROW, TOI_ROW, t);
			}
			__syncwarp();
		}
		if (step == TOI_START)
		{
			if (active)
			{
				sx.start(pA, pB, xfA, xfB);
				state = TOI_GJK;
			}
		}
		else if (step == TOI_GJK || step == TOI_MIN)
		{
			// One GJK iteration (gjk.cpp:683-768), or the points of minimum
			// separation: both end in support scans.
			V3 dA = V3{0.0f, 0.0f, 0.0f}, dB = dA;
			bool scanA = false, scanB = false;
			if (active && step == TOI_GJK)
			{
				scanA = scanB = sx.directions(xfA, xfB, dA, dB);
				if (!scanA)
					state = TOI_END;
			}
			else if (active)
			{
				sep.directions(xfA, xfB, dA, dB);
				scanA = !sep.plane_a();
				scanB = !sep.plane_b();
			}
			__syncwarp();
			uint32_t ia = B3G_NULL, ib = B3G_NULL;
			if (scanA)
				ia = pA.support(dA);
			__syncwarp();
			if (scanB)
				ib = pB.support(dB);
			__syncwarp();
			if (active && step == TOI_MIN)
			{
				indexA = ia;
				indexB = ib;
				kind = VALUE_MIN;
				state = TOI_VALUE;
			}
			else if (active && scanA && !sx.add(pA, pB, xfA, xfB, ia, ib))
				state = TOI_END;
		}
		else if (step == TOI_VALUE)
		{
			if (active)
			{
				const float s = sep.value(pA, pB, xfA, xfB, indexA, indexB);
				bool round = false; // the round ends: the next starts at t1
				if (kind == VALUE_MIN)
				{
					s2 = s;
					if (s2 > target + tolerance)
					{
						how = ST_SEPARATED;
						tEnd = tMax;
					}
					else if (s2 > target - tolerance)
					{
						t1 = t2;
						round = true;
					}
					else
						kind = VALUE_AT1;
				}
				else if (kind == VALUE_AT1)
				{
					s1 = s;
					if (s1 < target - tolerance)
						how = ST_FAILED;
					else if (s1 <= target + tolerance)
						how = ST_TOUCHING;
					else
					{
						steps = 0;
						a1 = t1;
						a2 = t2;
						kind = VALUE_ROOT;
					}
				}
				else
				{
					const bool found = fabsr(s - target) < tolerance;
					if (found)
						t2 = tRoot;
					else if (s > target)
					{
						a1 = tRoot;
						s1 = s;
					}
					else
					{
						a2 = tRoot;
						s2 = s;
					}
					if (found || steps == 50u)
					{
						state = TOI_MIN;
						round = ++pushBack == 64u;
					}
				}
				if (round || how != ST_UNKNOWN)
					++iteration;
				if (round)
				{
					state = TOI_START;
					if (iteration == 20u)
					{
						how = ST_FAILED;
						tEnd = t1;
					}
				}
			}
		}
		else if (active)
		{
			V3 P1, P2;
			sx.end(pA, pB, xfA, xfB, P1, P2);
			const float distance = len(P1 - P2);
			if (distance == 0.0f)
			{
				how = ST_OVERLAPPED;
				tEnd = 0.0f;
			}
			else if (distance < target + tolerance)
				how = ST_TOUCHING;
			else
			{
				GJKCache cache;
				cache.count = sx.count;
#pragma unroll
				for (uint32_t i = 0; i < 4; ++i)
				{
					cache.index1[i] = sx.index1(i);
					cache.index2[i] = sx.index2(i);
				}
				sep.init(cache, pA, pB, xfA, xfB);
				if (sep.type == SEP_NONE)
					how = ST_FAILED;
				t2 = tMax;
				pushBack = 0;
				state = TOI_MIN;
			}
		}
		if (how != ST_UNKNOWN)
		{
			uint32_t* o = out + 4 * (size_t)query;
			o[0] = how;
			o[1] = __float_as_uint(tEnd);
			o[2] = iteration;
			o[3] = 0;
			state = TOI_IDLE;
		}
		__syncwarp();
	}
}

// As many warps as the GPU holds, each with an equal share of the queries.
void launch_toi_sweeps(const DevScene& S, const float* in, uint32_t n, uint32_t* out, cudaStream_t s)
{
	const uint32_t warps = std::min(n, 148u * TOI_BLOCKS * TOI_WARPS);
	const uint32_t share = (n + warps - 1u) / warps;
	k_toi_sweeps<<<(warps + TOI_WARPS - 1u) / TOI_WARPS, TOI_WARPS * 32, 0, s>>>(S, in, n, share, out);
}

__global__ void k_toi_aabbs(const float* in, uint32_t n, uint32_t* out)
{
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	uint32_t state;
	float t;
	toi_aabbs(in + 18 * (size_t)i, state, t);
	out[4 * (size_t)i] = state;
	out[4 * (size_t)i + 1] = __float_as_uint(t);
	out[4 * (size_t)i + 2] = 0;
	out[4 * (size_t)i + 3] = 0;
}

__global__ void k_gjk_ray_cast(DevScene S, const float* in, uint32_t n, float* out)
{
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	const float* r = in + 48 * (size_t)i;
	const uint32_t typeA = __float_as_uint(r[0]), hullA = __float_as_uint(r[1]);
	const uint32_t typeB = __float_as_uint(r[2]), hullB = __float_as_uint(r[3]);
	const GProxy pA = input_proxy(S, r + 4, typeA, hullA);
	const GProxy pB = input_proxy(S, r + 16, typeB, hullB);
	XF xfA, xfB;
	xfA.p = V3{r[28], r[29], r[30]};
	xfA.q = Q4{V3{r[31], r[32], r[33]}, r[34]};
	xfB.p = V3{r[35], r[36], r[37]};
	xfB.q = Q4{V3{r[38], r[39], r[40]}, r[41]};
	const V3 tr = V3{r[42], r[43], r[44]};
	float t = 0.0f;
	V3 point = V3{0.0f, 0.0f, 0.0f}, normal = V3{0.0f, 0.0f, 0.0f};
	uint32_t iterations = 0;
	const bool hit = gjk_ray_cast(xfA, pA, xfB, pB, tr, t, point, normal, iterations);
	float* o = out + 9 * (size_t)i;
	o[0] = __uint_as_float(hit ? 1u : 0u);
	o[1] = hit ? t : 0.0f;
	o[2] = hit ? point.x : 0.0f;
	o[3] = hit ? point.y : 0.0f;
	o[4] = hit ? point.z : 0.0f;
	o[5] = hit ? normal.x : 0.0f;
	o[6] = hit ? normal.y : 0.0f;
	o[7] = hit ? normal.z : 0.0f;
	o[8] = __uint_as_float(iterations);
}

int tfail(b3g_ctx* c, int code, const char* msg)
{
	c->err = msg;
	return code;
}

// Copies n records of `bytes` each in, runs the launch, copies `outBytes`
// per record out (synchronous, on the context's stream). The device copies
// live in the context's scratch, grown on demand.
template <class Launch>
int run_batch(b3g_ctx* c, uint32_t n, const void* in, size_t bytes, void* out, size_t outBytes, Launch&& launch)
{
	if (n == 0)
		return 0;
	if (cudaSetDevice(c->device) != cudaSuccess)
		return tfail(c, B3G_E_CUDA, "time of impact: device");
	const size_t inBytes = (bytes * n + 255) & ~(size_t)255;
	const size_t need = inBytes + outBytes * n;
	if (c->toiScratchBytes < need)
	{
		if (c->toiScratch && cudaFree(c->toiScratch) != cudaSuccess)
			return tfail(c, B3G_E_CUDA, "time of impact: device free failed");
		c->toiScratch = nullptr;
		c->toiScratchBytes = 0;
		if (cudaMalloc(&c->toiScratch, need) != cudaSuccess)
			return tfail(c, B3G_E_CUDA, "time of impact: device allocation failed");
		c->toiScratchBytes = need;
	}
	void* dIn = c->toiScratch;
	void* dOut = (char*)c->toiScratch + inBytes;
	if (cudaMemcpyAsync(dIn, in, bytes * n, cudaMemcpyHostToDevice, c->stream) != cudaSuccess)
		return tfail(c, B3G_E_CUDA, "time of impact: copy");
	launch((const float*)dIn, dOut, c->stream);
	if (cudaGetLastError() != cudaSuccess ||
		cudaMemcpyAsync(out, dOut, outBytes * n, cudaMemcpyDeviceToHost, c->stream) != cudaSuccess ||
		cudaStreamSynchronize(c->stream) != cudaSuccess)
		return tfail(c, B3G_E_CUDA, "time of impact: kernel or copy failed");
	return (int)n;
}

// Shape types and hulls of a query's two proxies: convex types only.
bool proxies_ok(const b3g_ctx* c, uint32_t typeA, uint32_t hullA, uint32_t typeB, uint32_t hullB)
{
	auto ok = [&](uint32_t t, uint32_t h) { return t < B3G_SHAPE_MESH && (t != B3G_SHAPE_HULL || h < c->nHulls); };
	return ok(typeA, hullA) && ok(typeB, hullB);
}

} // namespace

extern "C" int b3g_time_of_impact(b3g_ctx* c, uint32_t n, const b3g_toi_input* in, uint32_t* out)
{
	if (!c || (n && (!in || !out)))
		return c ? tfail(c, B3G_E_INVALID, "b3g_time_of_impact: null argument") : B3G_E_INVALID;
	for (uint32_t i = 0; i < n; ++i)
		if (!proxies_ok(c, in[i].type_a, in[i].hull_a, in[i].type_b, in[i].hull_b))
			return tfail(c, B3G_E_INVALID, "b3g_time_of_impact: shape type or hull out of range");
	const DevScene S = c->scene;
	return run_batch(c, n, in, sizeof(b3g_toi_input), out, 16, [&](const float* dIn, void* dOut, cudaStream_t s) {
		launch_toi_sweeps(S, dIn, n, (uint32_t*)dOut, s);
	});
}

extern "C" int b3g_time_of_impact_device(b3g_ctx* c, uint32_t n, const b3g_toi_input* in, uint32_t* out,
	void* stream)
{
	if (!c || (n && (!in || !out)))
		return c ? tfail(c, B3G_E_INVALID, "b3g_time_of_impact_device: null argument") : B3G_E_INVALID;
	if (n == 0)
		return B3G_OK;
	if (cudaSetDevice(c->device) != cudaSuccess)
		return tfail(c, B3G_E_CUDA, "time of impact: device");
	cudaStream_t s = stream ? (cudaStream_t)stream : c->stream;
	launch_toi_sweeps(c->scene, (const float*)in, n, out, s);
	if (cudaGetLastError() != cudaSuccess)
		return tfail(c, B3G_E_CUDA, "b3g_time_of_impact_device: launch");
	return B3G_OK;
}

extern "C" int b3g_time_of_impact_aabb(b3g_ctx* c, uint32_t n, const float* in, uint32_t* out)
{
	if (!c || (n && (!in || !out)))
		return c ? tfail(c, B3G_E_INVALID, "b3g_time_of_impact_aabb: null argument") : B3G_E_INVALID;
	return run_batch(c, n, in, 18 * sizeof(float), out, 16, [&](const float* dIn, void* dOut, cudaStream_t s) {
		k_toi_aabbs<<<(n + 127) / 128, 128, 0, s>>>(dIn, n, (uint32_t*)dOut);
	});
}

extern "C" int b3g_gjk_shape_cast(b3g_ctx* c, uint32_t n, const b3g_gjk_cast_input* in, float* out)
{
	if (!c || (n && (!in || !out)))
		return c ? tfail(c, B3G_E_INVALID, "b3g_gjk_shape_cast: null argument") : B3G_E_INVALID;
	for (uint32_t i = 0; i < n; ++i)
		if (!proxies_ok(c, in[i].type_a, in[i].hull_a, in[i].type_b, in[i].hull_b))
			return tfail(c, B3G_E_INVALID, "b3g_gjk_shape_cast: shape type or hull out of range");
	const DevScene S = c->scene;
	return run_batch(c, n, in, sizeof(b3g_gjk_cast_input), out, 36, [&](const float* dIn, void* dOut, cudaStream_t s) {
		k_gjk_ray_cast<<<(n + 127) / 128, 128, 0, s>>>(S, dIn, n, (float*)dOut);
	});
}
