// Resident solvers: whole Krylov solves in one cooperative launch, with the
// fields of a right-hand side kept on chip (sm_100a).
//
// A grid of up to 148 x 16384 points (CG) or 148 x 6144 (pipelined CG and
// BiCGStab) has Krylov vectors that fit the registers and shared memory of the
// GPU's 148 SMs, with some own-point fields in L2.  A group of G blocks (one per
// SM; two in one box shape, for many small solves) then solves one right-hand
// side (FP64) or two (FP32, a float2 per point): each block owns a box of rows x
// planes, all n1 points wide, with the stencil input in shared memory (one ghost
// layer around it) and the residual in registers.  An iteration moves no Krylov
// vector through HBM; x, which no stencil reads, goes through L2.  CG's two
// reductions per iteration are the group's only two synchronisations: the one
// that ends an iteration also publishes the boundary rows of the new residual,
// from which every block forms its ghost points of the next direction itself.
// With more right-hand sides than one group needs blocks for, groups run side by
// side and take them in turn.
//
// Elementwise values round as the sweeps of the other forms: FP64 operator by
// operator as the reference (Cg.hpp:107-207), FP32 with the products fused
// into the following sum, so only the dot products' summation order differs.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

#include "resident.cuh"
#include "resident_room.h"
#include "sedi_internal.h"

namespace sedi {

// What a launch works on (device pointers; right-hand side k of every field
// at offset k * npts, or pair k / 2 for float2 fields).
struct ResArgs {
	int n1, n2, n3;
	long long npts;
	double a, b, c, iM;
	int lanes;            // right-hand sides
	int G, groups;        // blocks of a group, groups
	int s2, RG, nd;       // splits of a group along i2, row groups of a block, planes of a block
	const double *rhs;    // right-hand sides
	double *x;            // FP64: x (in: first guess); FP32: x_hi
	float2 *xlo;          // FP32: correction since the last reliable update
	void *edge;           // boundary rows: [fields][groups][G][2 nd + 2 RG*C][n1] of Face
	Word2 *words;         // [groups][res_words(G)]: the groups' reductions
	unsigned long long stamp;  // stamps of this launch lie above it
	double *scratch[4];   // own-point fields that do not fit shared memory: q, s, p, z (pipelined CG)
	int nsm;              // own-point fields that do
	double tol, tol_in;   // stop targets (tol_in = theta * tol for FP32)
	int maxiter, period;
	double *o_err, *o_bb, *o_rr;  // per right-hand side
	int *o_exit, *o_reason, *o_done;
	double *o_snorm, *o_omega, *o_rho;  // BiCGStab, else null
	double *hist;         // err after each iteration of right-hand side 0, or null
	int *err;             // a wait ran out
};

namespace {

template <class V>
struct Lanes;
template <>
struct Lanes<double> {
	typedef double S;
	static constexpr int N = 1;
};
template <>
struct Lanes<float2> {
	typedef float S;
	static constexpr int N = 2;
};
__device__ __forceinline__ double lane_get(double v, int) { return v; }
__device__ __forceinline__ void lane_set(double &v, int, double s) { v = s; }
__device__ __forceinline__ float lane_get(const float2 &v, int l) { return l ? v.y : v.x; }
__device__ __forceinline__ void lane_set(float2 &v, int l, float s) {
	if (l) v.y = s;
	else v.x = s;
}
template <class V>
__device__ __forceinline__ V lane_zero();
template <>
__device__ __forceinline__ double lane_zero<double>() {
	return 0.0;
}
template <>
__device__ __forceinline__ float2 lane_zero<float2>() {
	return make_float2(0.f, 0.f);
}

__device__ __forceinline__ unsigned long long bits(double v) { return __double_as_longlong(v); }
__device__ __forceinline__ unsigned long long bits(const float2 &v) {
	return (unsigned long long)__float_as_uint(v.y) << 32 | __float_as_uint(v.x);
}
template <class V>
__device__ __forceinline__ V value(unsigned long long b);
template <>
__device__ __forceinline__ double value<double>(unsigned long long b) {
	return __longlong_as_double(b);
}
template <>
__device__ __forceinline__ float2 value<float2>(unsigned long long b) {
	return make_float2(__uint_as_float((unsigned)b), __uint_as_float((unsigned)(b >> 32)));
}

// A point of a block's faces.  Plain (S false): written through L1 and made
// visible by a fenced group sum.  Stamped (S true): value and stamp of its
// publication in one atomic exchange, so the sum needs no fence (800-900 cycles
// for the stores, 300 for the reader) and a reader that comes too early waits
// for the stamp.  Exchanges are slower per point, so boxes with few planes
// take them.
template <class V, bool S>
struct Face;
template <class V>
struct Face<V, false> {
	V v;
	__device__ __forceinline__ void put(const V &x, unsigned long long) { stl2(&v, x); }
	typedef V Got;
	__device__ __forceinline__ Got load() const { return ldl2(&v); }
	__device__ __forceinline__ V get(const Got &g, unsigned long long, ResGroup *) const { return g; }
};
template <class V>
struct Face<V, true> {
	Word2 w;
	__device__ __forceinline__ void put(const V &x, unsigned long long stamp) { swap2(&w, bits(x), stamp); }
	typedef Word2 Got;
	__device__ __forceinline__ Got load() const { return load2(&w); }
	__device__ __forceinline__ V get(const Got &g, unsigned long long stamp, ResGroup *gr) const {
		return value<V>(g.b == stamp ? g.a : wait2(&w, stamp, gr).a);
	}
};

// r iM + beta p, and x + a y: FP64 rounds each operator, FP32 fuses.
__device__ __forceinline__ double comb(double r, double im, double beta, double p) {
	return add(mul(r, im), mul(beta, p));
}
__device__ __forceinline__ float comb(float r, float im, float beta, float p) {
	return __fmaf_rn(r, im, __fmul_rn(beta, p));
}
__device__ __forceinline__ double mul_s(double a, double b) { return mul(a, b); }
__device__ __forceinline__ float mul_s(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double axpy(double x, double a, double y) { return add(x, mul(a, y)); }
__device__ __forceinline__ float axpy(float x, float a, float y) { return __fmaf_rn(a, y, x); }

// Hides a value's origin, so that the addresses an unrolled loop derives from
// it are formed there by running increments instead of being kept in (or
// spilled from) registers across the whole solve.
__device__ __forceinline__ int opaque(int v) {
	asm volatile("" : "+r"(v));
	return v;
}

// The x an iteration updates: x itself (FP64) or the pair's correction (FP32).
template <class V>
__device__ __forceinline__ V *step_x(double *x, float2 *xlo);
template <>
__device__ __forceinline__ double *step_x<double>(double *x, float2 *) {
	return x;
}
template <>
__device__ __forceinline__ float2 *step_x<float2>(double *, float2 *xlo) {
	return xlo;
}

// Stencil.hpp:43-50 term order; UNIT: b = c = 1 (exact products left out).
template <bool UNIT>
__device__ __forceinline__ double st7r(double a, double b, double c, double xc, double xm1, double xm2, double xm3,
                                       double xp1, double xp2, double xp3) {
	double y = mul(a, xc);
	y = sub(y, UNIT ? xm1 : mul(c, xm1));
	y = sub(y, UNIT ? xm2 : mul(c, xm2));
	y = sub(y, UNIT ? xm3 : mul(c, xm3));
	y = sub(y, UNIT ? xp1 : mul(b, xp1));
	y = sub(y, UNIT ? xp2 : mul(b, xp2));
	y = sub(y, UNIT ? xp3 : mul(b, xp3));
	return y;
}
template <bool UNIT>
__device__ __forceinline__ float st7r(float a, float b, float c, float xc, float xm1, float xm2, float xm3, float xp1,
                                      float xp2, float xp3) {
	float y = __fmaf_rn(a, xc, -__fmul_rn(c, xm1));
	y = __fmaf_rn(-c, xm2, y);
	y = __fmaf_rn(-c, xm3, y);
	y = __fmaf_rn(-b, xp1, y);
	y = __fmaf_rn(-b, xp2, y);
	y = __fmaf_rn(-b, xp3, y);
	return y;
}

// Where a block's ghost rows are: {shared offset of the row's first point, its
// place in the neighbour's faces relative to the block's own}, built once, so
// that an iteration spends no index arithmetic on them (dealt out and decoded
// in place they cost 50 instructions a row and thread, a fifth of all).
// `nbr`: neighbours, bit 0 i2 low, 1 i2 high, 2 i3 low, 3 i3 high.
__device__ __forceinline__ void ghost_table(const ResArgs &A, int2 *tab, int *count, int B2, int nd, int nr, unsigned nbr,
                                            int pitch, int pp, int face_rows) {
	const int t = threadIdx.x, n1 = A.n1;
	int n = 0;
	if (nbr & 1u) {  // row -1, from the high i2 face of the block below
		for (int j = t; j < nd; j += blockDim.x) tab[n + j] = make_int2((j + 1) * pp + 1, (A.nd + j - face_rows) * n1);
		n += nd;
	}
	if (nbr & 2u) {
		for (int j = t; j < nd; j += blockDim.x)
			tab[n + j] = make_int2((j + 1) * pp + (nr + 1) * pitch + 1, (face_rows + j) * n1);
		n += nd;
	}
	if (nbr & 4u) {  // plane -1, from the high i3 face
		for (int j = t; j < nr; j += blockDim.x)
			tab[n + j] = make_int2((j + 1) * pitch + 1, (2 * A.nd + B2 + j - A.s2 * face_rows) * n1);
		n += nr;
	}
	if (nbr & 8u) {
		for (int j = t; j < nr; j += blockDim.x)
			tab[n + j] = make_int2((nd + 1) * pp + (j + 1) * pitch + 1, (2 * A.nd + j + A.s2 * face_rows) * n1);
		n += nr;
	}
	if (t == 0) *count = n;
}
// Bytes of shared memory before the table: `ghosted` fields with ghosts and
// `own` fields of the block's own points.
__host__ __device__ __forceinline__ size_t ghost_table_offset(const ResArgs &A, size_t elem, int ghosted, int own, int B2, int T) {
	const size_t e = (size_t)(A.n1 + 1) * (B2 + 2) * (A.nd + 2) + 1;
	return ((e * ghosted + (size_t)own * A.nd * T) * elem + 7) / 8 * 8;
}
__host__ __device__ __forceinline__ size_t ghost_table_bytes(int B2, int nd) { return 8 + 8 * (size_t)(2 * nd + 2 * B2); }

// CG's boxes of one row a thread have stamped faces (32^3: 5.6 -> 5.4 us an
// iteration, 48^3 6.2 -> 5.9); larger ones publish too many points, and
// pipelined CG and BiCGStab gained nothing (64^3: 5.1 -> 5.4, 11.2 -> 12.2 us).
__host__ __device__ constexpr bool stamped(int ks, int C) { return ks == SEDI_CG && C == 1; }

// Uniform state of the solve a block runs, in shared memory: written by warp 0
// at the end of a group sum, read by every thread after it.  Registers are
// left to the Krylov fields.
template <int NL>
struct CgState {
	const double *rhs[NL];
	double *x[NL];
	double bb[NL], rr[NL], ru[NL], alpha[NL], beta[NL], err[NL];
	double xa[NL];    // step of x still to take, along the p in shared memory
	int done[NL], reason[NL], ex[NL];
	int upd[NL];      // FP32: the lane takes part in this iteration's reliable update
	int restart[NL];  // FP32: p = u after the update
	int live, any;    // some lane still iterates / is updated
};

// ---------------------------------------------------------------------------
// CG.  Block m of a group owns rows [row0, row0 + RG*C) and planes
// [z0, z0 + nd) of the grid; thread t column i1 = t % n1 of the C consecutive
// rows of row group t / n1 on every plane, so the stencil marches along i3
// with the column in registers and takes one i2 neighbour of each of its rows
// from the row beside it.  Shared memory holds p with its ghosts, rows padded
// by one zero column that serves both neighbours of the row ends.
//
// Per iteration: A: p = u + beta p on the box (where x takes the step along
// the p that leaves) and, from the published rows of r, on the ghosts; <A p,
// p>; group sum; B: r -= alpha A p, boundary rows published; <r,u>, <r,r>;
// group sum.
//
// 128^3 FP64: 144 blocks of 128 x 8 x 15 points (176 KB of shared memory, 64
// registers of r per thread).
// ---------------------------------------------------------------------------
template <class V, int C, int D, int TMAX, int BLOCKS, bool UNIT>
__global__ void __launch_bounds__(TMAX, BLOCKS) k_res_cg(const __grid_constant__ ResArgs A) {
	typedef typename Lanes<V>::S S;
	constexpr int NL = Lanes<V>::N;
	constexpr bool MIXED = NL == 2;
	constexpr bool KEEP = C * D <= 16;  // A p stays in registers between its two uses
	constexpr bool STAMP = stamped(SEDI_CG, C);
	typedef Face<V, STAMP> FaceT;
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ ResGroup gsh;
	__shared__ CgState<NL> st;
	ResGroup *const g = &gsh;
	const int t = threadIdx.x, n1 = A.n1;
	const int B2 = A.RG * C, pitch = n1 + 1, pp = pitch * (B2 + 2);  // box rows, shared row and plane pitches
	const int i1 = t % n1, rg = t / n1;
	V *const sp = reinterpret_cast<V *>(smem);
	const int group = blockIdx.x / A.G;
	const int s3 = n1 * A.n2;  // the grid has far fewer than 2^31 points
	int nd, rows, so, go, own3, hi_c, hi_d;
	bool lo_c, lo_d;
	unsigned nbr;  // neighbours: bit 0 i2 low, 1 i2 high, 2 i3 low, 3 i3 high; box rows above
	{
		const int m = blockIdx.x % A.G;
		const int row0 = (m % A.s2) * B2, z0 = (m / A.s2) * A.nd, nr = min(B2, A.n2 - row0);
		nd = min(A.nd, A.n3 - z0);  // valid planes of the box, nr rows
		rows = rg < A.RG ? max(0, min(C, nr - rg * C)) : 0;  // valid rows of the thread
		so = pp + (rg * C + 1) * pitch + 1 + i1;              // own point (c, d) = (0, 0): shared offset
		go = z0 * s3 + (row0 + rg * C) * n1 + i1;             // and place in the grid
		own3 = (2 * A.nd + rg * C) * n1 + i1;                 // and in the low i3 face
		const bool lo2 = row0 > 0, hi2 = row0 + nr < A.n2, lo3 = z0 > 0, hi3 = z0 + nd < A.n3;
		nbr = (lo2 ? 1u : 0u) | (hi2 ? 2u : 0u) | (lo3 ? 4u : 0u) | (hi3 ? 8u : 0u) | (unsigned)nr << 4;
		lo_c = lo2 && rg == 0;  // published rows and planes: the first, and which of the last
		hi_c = hi2 ? nr - 1 - rg * C : -1;
		lo_d = lo3;
		hi_d = hi3 ? nd - 1 : -1;
		if (t == 0) {
			g->G = A.G;
			g->m = m;
			g->words = A.words + (size_t)group * res_words(A.G);
			g->err = A.err;
			g->base = A.stamp;
			g->fail = 0;
		}
	}
	const int face_rows = 2 * A.nd + 2 * B2;  // face rows of a block: i2 low, high, i3 low, high
	unsigned round = 0;                       // group sums so far
	unsigned pub = 0;                         // publications of face rows
	FaceT *const faces = static_cast<FaceT *>(A.edge) + (size_t)blockIdx.x * face_rows * n1;  // this block's
	int *const ghost_count = reinterpret_cast<int *>(smem + ghost_table_offset(A, sizeof(V), 1, 0, B2, blockDim.x));
	int2 *const ghost_rows = reinterpret_cast<int2 *>(ghost_count + 2);
	ghost_table(A, ghost_rows, ghost_count, B2, nd, (int)(nbr >> 4), nbr, pitch, pp, face_rows);
	const S im = (S)A.iM;

	const int units = (A.lanes + NL - 1) / NL;
	for (int unit = group; unit < units; unit += A.groups) {
		const int lane0 = unit * NL;
		if (t == 0)
			for (int l = 0; l < NL; l++) {
				const int k = lane0 + l < A.lanes ? lane0 + l : lane0;  // an odd last pair has one right-hand side
				st.rhs[l] = A.rhs + (size_t)k * A.npts;
				st.x[l] = A.x + (size_t)k * A.npts;
			}
		for (int e = t; e < pp * (A.nd + 2) + 1; e += blockDim.x) sp[e] = lane_zero<V>();
		__syncthreads();
		V r[C][D];
		// The x an iteration updates: x itself (FP64) or the pair's correction.
		auto step_ptr = [&]() { return step_x<V>(st.x[0], MIXED ? A.xlo + (size_t)unit * A.npts : nullptr); };
		// r = b - A x from x in global memory (ghost layer zero): the setup and
		// the FP64 residual of a reliable update.  part: per lane <b,b>, <r,r>,
		// <r, r iM>; a lane outside the update keeps its r.
		auto residual = [&](double (&part)[3 * NL], bool setup) {
#pragma unroll
			for (int l = 0; l < NL; l++) {
				part[3 * l] = part[3 * l + 1] = part[3 * l + 2] = 0.0;
				if (!setup && !st.upd[l]) continue;
				const double *x = st.x[l], *b = st.rhs[l];
				const bool live = lane0 + l < A.lanes;
				const int z0 = go / s3, i2 = (go - z0 * s3) / n1;
#pragma unroll
				for (int c = 0; c < C; c++) {
					int i = opaque(go) + c * n1;
					const bool ok = c < rows;
					double prev = (ok && z0 > 0) ? ldl2(x + i - s3) : 0.0, cur = ok ? ldl2(x + i) : 0.0;
#pragma unroll
					for (int d = 0; d < D; d++) {
						if (d < nd && ok) {
							const double next = z0 + d + 1 < A.n3 ? ldl2(x + i + s3) : 0.0;
							const double xm1 = i1 > 0 ? ldl2(x + i - 1) : 0.0, xp1 = i1 < n1 - 1 ? ldl2(x + i + 1) : 0.0;
							const double xm2 = i2 + c > 0 ? ldl2(x + i - n1) : 0.0, xp2 = i2 + c < A.n2 - 1 ? ldl2(x + i + n1) : 0.0;
							const double ax = st7r<UNIT>(A.a, A.b, A.c, cur, xm1, xm2, prev, xp1, xp2, next);
							const double bi = live ? b[i] : 0.0;
							const double ri = live ? add(bi, -ax) : 0.0;  // combine2(1.0, b, -1.0, A x) (Cg.hpp:123)
							const S rt = (S)ri;
							lane_set(r[c][d], l, rt);
							part[3 * l] = fma(bi, bi, part[3 * l]);
							part[3 * l + 1] = fma(ri, ri, part[3 * l + 1]);
							if (setup) part[3 * l + 2] = fma((double)rt, (double)mul_s(rt, im), part[3 * l + 2]);
							else part[3 * l + 2] = fma(ri, mul(ri, A.iM), part[3 * l + 2]);
							prev = cur;
							cur = next;
							i += s3;
							asm volatile("" ::: "memory");  // one point's loads at a time: registers hold r
						} else if (setup) {
							lane_set(r[c][d], l, (S)0);
						}
					}
				}
			}
		};
		// Publishes a point of the box's faces (f2, f3: the thread's place in the
		// i2 and i3 faces) for the neighbours to read after the next fenced sum.
		auto publish = [&](int c, int d, int f2, int f3, const V &v) {
			const unsigned long long stamp = A.stamp + pub;
			if (c == 0 && lo_c) faces[f2].put(v, stamp);
			if (c == hi_c) faces[f2 + A.nd * n1].put(v, stamp);
			if (d == 0 && lo_d) faces[f3 + c * n1].put(v, stamp);
			if (d == hi_d) faces[f3 + (B2 + c) * n1].put(v, stamp);
		};
		auto publish_all = [&]() {
			pub++;
			int f2 = opaque(i1);
			const int f3 = opaque(own3);
#pragma unroll
			for (int d = 0; d < D; d++, f2 += n1)
#pragma unroll
				for (int c = 0; c < C; c++)
					if (c < rows && d < nd) publish(c, d, f2, f3, r[c][d]);
		};

		{
			double part[3 * NL];
			residual(part, true);
			publish_all();
			if (!group_sum<3 * NL, !STAMP>(g, round, part, Nothing(), [&](int lane, const double (&v)[3 * NL]) {
				    if (lane == 0) {
					    int live = 0;
#pragma unroll
					    for (int l = 0; l < NL; l++) {
						    const double bb = v[3 * l] == 0.0 ? 1.0 : v[3 * l];  // Cg.hpp:112-115
						    const double err = sqrt(__ddiv_rn(v[3 * l + 1], bb));
						    int done = 0, reason = STOP_NONE, ex = 0;
						    if (lane0 + l >= A.lanes) {
							    done = 1;
						    } else if (err < A.tol) {  // :130-134
							    done = 1;
							    reason = STOP_EARLY;
						    } else if (A.maxiter < 1) {
							    done = 1;
							    reason = STOP_MAXITER;
							    ex = 1;
						    }
						    st.bb[l] = bb;
						    st.rr[l] = v[3 * l + 1];
						    st.ru[l] = v[3 * l + 2];
						    st.err[l] = err;
						    st.beta[l] = st.xa[l] = 0.0;
						    st.done[l] = done;
						    st.reason[l] = reason;
						    st.ex[l] = ex;
						    st.upd[l] = st.restart[l] = 0;
						    live |= !done;
					    }
					    st.live = live;
					    if (A.hist && unit == 0 && blockIdx.x % A.G == 0) A.hist[0] = st.err[0];
				    }
			    }))
				return;
		}
		if (MIXED) {
			V *xs = step_ptr() + go;
			for (int d = 0; d < nd; d++, xs += s3)
#pragma unroll
				for (int c = 0; c < C; c++)
					if (c < rows) stl2(xs + c * n1, lane_zero<V>());
		}

		for (int it = 1; st.live; it++) {
			// ---- A: p = u + beta p (Cg.hpp:188) on the ghosts, from the neighbours' r, and on the box.
			if (rg < A.RG) {
				S be[NL];
#pragma unroll
				for (int l = 0; l < NL; l++) be[l] = (S)st.beta[l];
				const int ghosts = *ghost_count;
				constexpr int HB = 6;
				for (int h0 = rg; h0 < ghosts; h0 += HB * A.RG) {  // dealt to the row groups
					typename FaceT::Got got[HB];
					int off[HB], from[HB];
#pragma unroll
					for (int k = 0; k < HB; k++) {
						off[k] = -1;
						if (h0 + k * A.RG >= ghosts) continue;
						const int2 e = ghost_rows[h0 + k * A.RG];
						off[k] = e.x + i1;
						from[k] = e.y + i1;
						got[k] = faces[from[k]].load();
					}
#pragma unroll
					for (int k = 0; k < HB; k++) {
						if (off[k] < 0) continue;
						const V rh = faces[from[k]].get(got[k], A.stamp + pub, g);
						V p = sp[off[k]];
#pragma unroll
						for (int l = 0; l < NL; l++) lane_set(p, l, comb(lane_get(rh, l), im, be[l], lane_get(p, l)));
						sp[off[k]] = p;
					}
				}
				// x takes the step of the iteration before here, where its p is read
				// anyway; x of the next plane is on its way, and the stores drain
				// during the stencil.
				S ax[NL];
				bool step = false;
#pragma unroll
				for (int l = 0; l < NL; l++) {
					ax[l] = (S)st.xa[l];
					step |= st.xa[l] != 0.0;
				}
				V *xp = step_ptr() + opaque(go);
				V *q = sp + opaque(so);
				V xn[C];
				auto load_x = [&](int d) {
					if (step && d < nd)
#pragma unroll
						for (int c = 0; c < C; c++)
							if (c < rows) xn[c] = ldl2(xp + c * n1);
				};
				load_x(0);
#pragma unroll
				for (int d = 0; d < D; d++, q += pp) {
					if (d >= nd) break;
					V x[C];
#pragma unroll
					for (int c = 0; c < C; c++) x[c] = xn[c];
					xp += s3;
					load_x(d + 1);
#pragma unroll
					for (int c = 0; c < C; c++) {
						if (c >= rows) continue;
						V p = q[c * pitch];
						if (step) {
#pragma unroll
							for (int l = 0; l < NL; l++)
								if (NL == 1 || ax[l] != (S)0) lane_set(x[c], l, axpy(lane_get(x[c], l), ax[l], lane_get(p, l)));
							stl2(xp - s3 + c * n1, x[c]);
						}
#pragma unroll
						for (int l = 0; l < NL; l++)
							lane_set(p, l, comb(lane_get(r[c][d], l), im, be[l], lane_get(p, l)));
						q[c * pitch] = p;
					}
				}
			}
			__syncthreads();
			// Stencil march over the thread's rows: f(c, d, p, A p) of its points.
			auto march_rows = [&](auto f) {
				const S ka = (S)A.a, kb = (S)A.b, kc = (S)A.c;
				const V *q = sp + opaque(so);
				V prev[C], cur[C];
#pragma unroll
				for (int c = 0; c < C; c++) {
					prev[c] = q[c * pitch - pp];
					cur[c] = q[c * pitch];
				}
#pragma unroll
				for (int d = 0; d < D; d++) {
					if (d >= nd) break;
					V next[C];
#pragma unroll
					for (int c = 0; c < C; c++) next[c] = q[pp + c * pitch];
					const V up = q[-pitch], dn = q[C * pitch];
#pragma unroll
					for (int c = 0; c < C; c++) {
						const V xm1 = q[c * pitch - 1], xp1 = q[c * pitch + 1];
						const V &xm2 = c > 0 ? cur[c > 0 ? c - 1 : 0] : up;
						const V &xp2 = c + 1 < C ? cur[c + 1 < C ? c + 1 : c] : dn;
						V y;
#pragma unroll
						for (int l = 0; l < NL; l++)
							lane_set(y, l, st7r<UNIT>(ka, kb, kc, lane_get(cur[c], l), lane_get(xm1, l), lane_get(xm2, l),
							                          lane_get(prev[c], l), lane_get(xp1, l), lane_get(xp2, l),
							                          lane_get(next[c], l)));
						f(c, d, cur[c], y);
					}
#pragma unroll
					for (int c = 0; c < C; c++) {
						prev[c] = cur[c];
						cur[c] = next[c];
					}
					q += pp;
				}
			};
			V ap[C][KEEP ? D : 1];
			{
				double v[NL];
#pragma unroll
				for (int l = 0; l < NL; l++) v[l] = 0.0;
				if (rows > 0)
					march_rows([&](int c, int d, const V &p, const V &s) {
						if (KEEP) ap[c][KEEP ? d : 0] = s;
						if (c < rows)
#pragma unroll
							for (int l = 0; l < NL; l++) v[l] = fma((double)lane_get(s, l), (double)lane_get(p, l), v[l]);
					});
				if (!group_sum<NL>(g, round, v, Nothing(), [&](int lane, const double (&tot)[NL]) {
#pragma unroll
					    for (int l = 0; l < NL; l++)
						    if (lane == l) {
							    double a = __ddiv_rn(st.ru[l], tot[l]);  // :166
							    st.upd[l] = 0;
							    if (st.done[l]) {
								    a = 0.0;
							    } else if (MIXED && !(tot[l] > 0.0 && isfinite(a))) {
								    // FP32 breakdown (p = 0 once the recurrence residual is exactly
								    // zero, or overflow): no step, then a restart from the true residual.
								    a = 0.0;
								    st.upd[l] = st.restart[l] = 1;
							    }
							    st.alpha[l] = st.xa[l] = a;
						    }
				    }))
					return;
			}
			const bool periodic = MIXED && A.period > 0 && it % A.period == 0;
			// ---- B: r -= alpha s, u = r iM (:172-175); the boundary rows of r go out.
			{
				double v[2 * NL];
#pragma unroll
				for (int d = 0; d < 2 * NL; d++) v[d] = 0.0;
				pub++;
				if (rows > 0) {
					S al[NL];
#pragma unroll
					for (int l = 0; l < NL; l++) al[l] = -(S)st.alpha[l];
					int f2 = opaque(i1);
					const int f3 = opaque(own3);
					auto update = [&](int c, int d, const V &, const V &s) {
						if (c < rows) {
							V rv = r[c][d];
#pragma unroll
							for (int l = 0; l < NL; l++) {
								const S q = axpy(lane_get(rv, l), al[l], lane_get(s, l));
								lane_set(rv, l, q);
								v[2 * l] = fma((double)q, (double)mul_s(q, im), v[2 * l]);
								v[2 * l + 1] = fma((double)q, (double)q, v[2 * l + 1]);
							}
							r[c][d] = rv;
							publish(c, d, f2, f3, rv);
						}
						if (c == C - 1) f2 += n1;
					};
					if (KEEP) {
#pragma unroll
						for (int d = 0; d < D; d++) {
							if (d >= nd) break;
#pragma unroll
							for (int c = 0; c < C; c++) update(c, d, ap[c][KEEP ? d : 0], ap[c][KEEP ? d : 0]);
						}
					} else {
						march_rows(update);
					}
				}
				if (!group_sum<2 * NL, !STAMP>(g, round, v, Nothing(), [&](int lane, const double (&tot)[2 * NL]) {
#pragma unroll
					    for (int l = 0; l < NL; l++) {
						    // Lane 2l: beta; lane 2l + 1: the error and the stop test.
						    if (lane / 2 != l || st.done[l]) continue;
						    const bool e = lane & 1;
						    const double q = __ddiv_rn(e ? tot[2 * l + 1] : tot[2 * l], e ? st.bb[l] : st.ru[l]);
						    if (!e) {
							    st.beta[l] = q;  // :185
							    continue;
						    }
						    const double err = sqrt(q);  // :191
						    st.rr[l] = tot[2 * l + 1];
						    st.err[l] = err;
						    if (A.hist && unit == 0 && l == 0 && blockIdx.x % A.G == 0) A.hist[it] = err;
						    if (MIXED) {
							    // The FP32 recurrence only proposes; the FP64 true residual decides.
							    if (!(err == err)) st.restart[l] = 1;
							    if (err <= A.tol_in || it >= A.maxiter || !(err == err) || periodic) st.upd[l] = 1;
						    } else if (err <= A.tol_in) {  // :193
							    st.done[l] = 1;
							    st.ex[l] = it;
							    st.reason[l] = STOP_CONVERGED;
						    } else if (it >= A.maxiter) {
							    st.done[l] = 1;
							    st.ex[l] = A.maxiter + 1;
							    st.reason[l] = STOP_MAXITER;
						    }
					    }
					    __syncwarp();
					    if (lane == 0) {
						    st.live = st.any = 0;
#pragma unroll
						    for (int l = 0; l < NL; l++) {
							    st.live |= !st.done[l];
							    st.any |= !st.done[l] && st.upd[l];
							    if (st.done[l]) st.beta[l] = 0.0;
							    // An update forms its beta over the old <r,u> first.
							    if (!MIXED || !st.upd[l]) st.ru[l] = tot[2 * l];
						    }
					    }
				    }))
					return;
			}
			if (MIXED && st.any) {
				// Reliable update: x_hi += x_lo and the pending step (in FP32 through
				// x_lo after an even iteration, in FP64 after an odd one and then only
				// for lanes in the update), then r = b - A x_hi in FP64.  Both lanes of
				// a pair fold their x_lo; only lanes in the update take a new r.
				const bool odd = it & 1;
				{
					V *xp = step_ptr() + go;
					int i = go;
					const V *q = sp + so;
					for (int d = 0; d < nd; d++, i += s3, xp += s3, q += pp)
#pragma unroll
						for (int c = 0; c < C; c++) {
							if (c >= rows) continue;
							const V p = q[c * pitch], x = ldl2(xp + c * n1);
#pragma unroll
							for (int l = 0; l < NL; l++) {
								if (lane0 + l >= A.lanes) continue;
								double *const xh = st.x[l] + i + c * n1;
								S lo = lane_get(x, l);
								if (!odd && st.xa[l] != 0.0) lo = axpy(lo, (S)st.xa[l], lane_get(p, l));
								double hi = ldl2(xh) + (double)lo;
								if (odd && st.upd[l] && !st.done[l]) hi = fma(st.xa[l], (double)lane_get(p, l), hi);
								stl2(xh, hi);
							}
							stl2(xp + c * n1, lane_zero<V>());
						}
				}
				double part[3 * NL];
				part[0] = 0.0;
				double none[1] = {0.0};
				if (!group_sum<1, true>(g, round, none, Nothing(), [&](int lane, const double (&)[1]) {
					    if (lane < NL && (!odd || (st.upd[lane] && !st.done[lane]))) st.xa[lane] = 0.0;
				    }))
					return;  // x_hi complete
				residual(part, false);
				publish_all();
				if (!group_sum<3 * NL, !STAMP>(g, round, part, Nothing(), [&](int lane, const double (&tot)[3 * NL]) {
					    if (lane != 0) return;
					    st.live = 0;
#pragma unroll
					    for (int l = 0; l < NL; l++) {
						    if (!st.done[l] && st.upd[l]) {
							    const double rr = tot[3 * l + 1], ru = tot[3 * l + 2];
							    // A recurrence residual far below the true one (squared norms 1e-6
							    // apart) no longer describes it: restart from the replaced one.
							    const bool lost = !(st.rr[l] >= 1e-6 * rr);
							    const double err = sqrt(rr / st.bb[l]);
							    st.rr[l] = rr;
							    st.err[l] = err;
							    if (err <= A.tol_in) {
								    st.done[l] = 1;
								    st.ex[l] = it;
								    st.reason[l] = STOP_CONVERGED;
							    } else if (it >= A.maxiter) {
								    st.done[l] = 1;
								    st.ex[l] = A.maxiter + 1;
								    st.reason[l] = STOP_MAXITER;
							    } else {
								    double be = ru / st.ru[l];
								    if (lost || st.restart[l] || !(be >= 0.0 && isfinite(be))) be = 0.0;  // p = u
								    st.beta[l] = be;
								    st.ru[l] = ru;
								    st.restart[l] = 0;
							    }
							    if (st.done[l]) st.beta[l] = 0.0;
						    }
						    st.live |= !st.done[l];
					    }
				    }))
					return;
			}
		}
		if (!MIXED && st.xa[0] != 0.0) {  // the last iteration's step (FP32: x_hi is complete)
			V *xp = step_ptr() + go;
			const V *q = sp + so;
			for (int d = 0; d < nd; d++, xp += s3, q += pp)
#pragma unroll
				for (int c = 0; c < C; c++) {
					if (c >= rows) continue;
					V x = ldl2(xp + c * n1);
					lane_set(x, 0, axpy(lane_get(x, 0), (S)st.xa[0], lane_get(q[c * pitch], 0)));
					stl2(xp + c * n1, x);
				}
		}
		if (blockIdx.x % A.G == 0 && t == 0)
			for (int l = 0; l < NL; l++) {
				const int k = lane0 + l;
				if (k >= A.lanes) continue;
				A.o_err[k] = st.err[l];
				A.o_bb[k] = st.bb[l];
				A.o_rr[k] = st.rr[l];
				A.o_exit[k] = st.ex[l];
				A.o_reason[k] = st.reason[l];
				A.o_done[k] = 1;
			}
		__syncthreads();  // shared memory is reused by the next right-hand side
	}
}

// ---------------------------------------------------------------------------
// A block's box and a thread's column in it, for solvers whose stencil input
// is in shared memory with its ghosts (one row per thread and plane).
// ---------------------------------------------------------------------------
struct ResBox {
	int i1, rg, pitch, pp;    // column, row group (= box row); shared row and plane pitches
	int nd, nr;               // valid planes and rows of the box
	int so, go, s3;           // own point of plane 0: shared offset, place in the grid; plane stride
	int z0, row0, face_rows;
	bool own, lo2, hi2, lo3, hi3;
	__device__ ResBox(const ResArgs &A) {
		const int m = blockIdx.x % A.G, n1 = A.n1;
		i1 = threadIdx.x % n1;
		rg = threadIdx.x / n1;
		pitch = n1 + 1;
		pp = pitch * (A.RG + 2);
		row0 = (m % A.s2) * A.RG;
		z0 = (m / A.s2) * A.nd;
		nr = min(A.RG, A.n2 - row0);
		nd = min(A.nd, A.n3 - z0);
		own = rg < nr;
		s3 = n1 * A.n2;
		so = pp + (rg + 1) * pitch + 1 + i1;
		go = z0 * s3 + (row0 + rg) * n1 + i1;
		face_rows = 2 * A.nd + 2 * A.RG;
		lo2 = row0 > 0;
		hi2 = row0 + nr < A.n2;
		lo3 = z0 > 0;
		hi3 = z0 + nd < A.n3;
	}
	// A block's faces of a field in global memory: rows i2 low [nd], i2 high
	// [nd], i3 low [RG], i3 high [RG].
	__device__ void publish(const ResArgs &A, double *faces, int d, double v) const {
		if (rg == 0 && lo2) stl2(faces + d * A.n1 + i1, v);
		if (rg == nr - 1 && hi2) stl2(faces + (A.nd + d) * A.n1 + i1, v);
		if (d == 0 && lo3) stl2(faces + (2 * A.nd + rg) * A.n1 + i1, v);
		if (d == nd - 1 && hi3) stl2(faces + (2 * A.nd + A.RG + rg) * A.n1 + i1, v);
	}
	// Ghost points of the box, HB rows of a thread at a time: load(k, from) of
	// the neighbour's face point, then use(k, shared offset).
	template <int HB, class Load, class Use>
	__device__ __forceinline__ void ghosts(const ResArgs &A, const int2 *tab, int count, Load load, Use use) const {
		if (rg >= A.RG) return;
		for (int h0 = rg; h0 < count; h0 += HB * A.RG) {
			int off[HB];
#pragma unroll
			for (int k = 0; k < HB; k++) {
				off[k] = -1;
				if (h0 + k * A.RG >= count) continue;
				const int2 e = tab[h0 + k * A.RG];
				off[k] = e.x + i1;
				load(k, e.y + i1);
			}
#pragma unroll
			for (int k = 0; k < HB; k++)
				if (off[k] >= 0) use(k, off[k]);
		}
	}
	__device__ void table(const ResArgs &A, int2 *tab, int *count) const {
		ghost_table(A, tab, count, A.RG, nd, nr, (lo2 ? 1u : 0u) | (hi2 ? 2u : 0u) | (lo3 ? 4u : 0u) | (hi3 ? 8u : 0u), pitch, pp,
		            face_rows);
	}
	// f(d, centre, A (scale .* field)) of the thread's points; SCALED as the
	// reference stores the stencil input (each value read times scale).
	template <int D, bool UNIT, bool SCALED, class F>
	__device__ __forceinline__ void march(const ResArgs &A, const double *field, double scale, F f) const {
		if (!own) return;
		auto in = [&](double v) { return SCALED ? mul(v, scale) : v; };
		const double *q = field + opaque(so);
		double prev = in(q[-pp]), raw = q[0], cur = in(raw);
#pragma unroll
		for (int d = 0; d < D; d++) {
			if (d >= nd) break;
			const double rnext = q[pp], next = in(rnext);
			f(d, raw, st7r<UNIT>(A.a, A.b, A.c, cur, in(q[-1]), in(q[-pitch]), prev, in(q[1]), in(q[pitch]), next));
			prev = cur;
			raw = rnext;
			cur = next;
			q += pp;
		}
	}
	// f(d, grid index, b - A x) of the thread's points, x in global memory.
	template <int D, bool UNIT, class F>
	__device__ __forceinline__ void residual(const ResArgs &A, const double *x, const double *b, F f) const {
		if (!own) return;
		const int n1 = A.n1, i2 = row0 + rg;
		int i = opaque(go);
		double prev = z0 > 0 ? ldl2(x + i - s3) : 0.0, cur = ldl2(x + i);
#pragma unroll
		for (int d = 0; d < D; d++) {
			if (d >= nd) break;
			const double next = z0 + d + 1 < A.n3 ? ldl2(x + i + s3) : 0.0;
			const double xm1 = i1 > 0 ? ldl2(x + i - 1) : 0.0, xp1 = i1 < n1 - 1 ? ldl2(x + i + 1) : 0.0;
			const double xm2 = i2 > 0 ? ldl2(x + i - n1) : 0.0, xp2 = i2 < A.n2 - 1 ? ldl2(x + i + n1) : 0.0;
			const double bi = b[i];
			f(d, cur, bi, add(bi, -st7r<UNIT>(A.a, A.b, A.c, cur, xm1, xm2, prev, xp1, xp2, next)));
			prev = cur;
			cur = next;
			i += s3;
		}
	}
};

__device__ __forceinline__ void group_init(ResGroup *g, const ResArgs &A) {
	g->G = A.G;
	g->m = blockIdx.x % A.G;
	g->words = A.words + (size_t)(blockIdx.x / A.G) * res_words(A.G);
	g->err = A.err;
	g->base = A.stamp;
	g->fail = 0;
}

// Uniform state of a pipelined CG or BiCGStab solve, in shared memory: warp 0
// writes it at the end of a group sum.
struct KrylovState {
	double bb, rr, err, alpha, beta;
	double gamma, gamma_old, delta;              // pipelined CG
	double rho, rho_prev, omega, bo, s_norm2;    // BiCGStab
	int done, reason, ex, s_exit;
};

__device__ __forceinline__ void stop(KrylovState &st, int reason, int ex) {
	st.done = 1;
	st.reason = reason;
	st.ex = ex;
}

// <b,b>, <r,r>: the initial error and test (Cg.hpp:112-134 and its twins).
__device__ __forceinline__ void initial_state(KrylovState &st, const ResArgs &A, double bb, double rr, bool hist) {
	st.bb = bb == 0.0 ? 1.0 : bb;
	st.rr = rr;
	st.err = sqrt(__ddiv_rn(rr, st.bb));
	st.done = st.s_exit = 0;
	st.reason = STOP_NONE;
	st.ex = 0;
	st.s_norm2 = st.rho_prev = 0.0;
	st.omega = 1.0;  // BiCgStab.hpp:147-150
	st.alpha = st.beta = 0.0;
	if (hist) A.hist[0] = st.err;
	if (st.err < A.tol) stop(st, STOP_EARLY, 0);
	else if (A.maxiter < 1) stop(st, STOP_MAXITER, 1);
}

__device__ __forceinline__ void write_state(const KrylovState &st, const ResArgs &A, int k) {
	A.o_err[k] = st.err;
	A.o_bb[k] = st.bb;
	A.o_rr[k] = st.rr;
	A.o_exit[k] = st.ex;
	A.o_reason[k] = st.reason;
	A.o_done[k] = 1;
	if (A.o_snorm) {
		A.o_snorm[k] = st.s_norm2;
		A.o_omega[k] = st.omega;
		A.o_rho[k] = st.rho;
	}
}

// ---------------------------------------------------------------------------
// Pipelined CG (PipelinedCg.hpp:136-230), FP64.  Shared memory holds m = w .*
// iM with its ghosts and the thread's own points of q, s, p, z and x; r, u and
// w are in registers.  An iteration is one stencil pass with the eight updates
// and one group reduction, which also publishes the boundary rows of m.  Boxes
// of more than 8 planes keep in shared memory what fits (A.nsm fields) and the
// other own points in global memory, that is in L2.
// ---------------------------------------------------------------------------
template <int D, int TMAX, bool UNIT>
__global__ void __launch_bounds__(TMAX, 1) k_res_pcg(const __grid_constant__ ResArgs A) {
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ ResGroup gsh;
	__shared__ KrylovState st;
	ResGroup *const g = &gsh;
	const ResBox B(A);
	const int t = threadIdx.x, T = blockDim.x;
	const int elems = B.pp * (A.nd + 2) + 1;
	double *const sm = reinterpret_cast<double *>(smem);
	constexpr bool GLOBAL = D > 8;
	// The faces of two rounds: a block publishes new rows while a neighbour may
	// still read the old ones.
	double *const faces = static_cast<double *>(A.edge) + (size_t)blockIdx.x * B.face_rows * A.n1;
	const size_t other = (size_t)gridDim.x * B.face_rows * A.n1;
	if (t == 0) group_init(g, A);
	int *const ghost_count = reinterpret_cast<int *>(smem + ghost_table_offset(A, sizeof(double), 1, A.nsm, A.RG, T));
	int2 *const ghost_rows = reinterpret_cast<int2 *>(ghost_count + 2);
	B.table(A, ghost_rows, ghost_count);
	unsigned round = 0;
	const double im = A.iM;
	for (int unit = blockIdx.x / A.G; unit < A.lanes; unit += A.groups) {
		double *const x = A.x + (size_t)unit * A.npts;
		const bool hist = A.hist && unit == 0 && blockIdx.x % A.G == 0;
		const double *in = faces;     // read
		double *out = faces + other;  // published next
		// Own point of plane d of field k (q, s, p, z, x).
		double *own[5];
		int step[5];
#pragma unroll
		for (int k = 0; k < 5; k++) {
			own[k] = sm + elems + t + k * A.nd * T;
			step[k] = T;
			if (GLOBAL && k >= A.nsm) {
				own[k] = (k < 4 ? A.scratch[k] + (size_t)unit * A.npts : x) + B.go;
				step[k] = B.s3;
			}
		}
		auto at = [&](int k, int d) -> double & { return own[k][d * step[k]]; };
		for (int e = t; e < elems; e += T) sm[e] = 0.0;
		__syncthreads();
		double r[D], u[D], w[D];
		{
			double v[2] = {0.0, 0.0};
			B.residual<D, UNIT>(A, x, A.rhs + (size_t)unit * A.npts, [&](int d, double xi, double bi, double ri) {
				r[d] = ri;
				u[d] = mul(ri, im);  // :138
				at(4, d) = xi;
				at(0, d) = at(1, d) = at(2, d) = at(3, d) = 0.0;  // :146-149
				sm[B.so + d * B.pp] = u[d];
				B.publish(A, faces, d, u[d]);
				v[0] = fma(bi, bi, v[0]);
				v[1] = fma(ri, ri, v[1]);
			});
			if (!group_sum<2, true>(g, round, v, Nothing(), [&](int lane, const double (&tot)[2]) {
				    if (lane == 0) initial_state(st, A, tot[0], tot[1], hist);
			    }))
				return;
		}
		constexpr int HB = 6;
		double hv[HB];
		auto load = [&](int k, int from) { hv[k] = ldl2(in + from); };
		auto put = [&](int k, int off) { sm[off] = hv[k]; };
		// fin of a sum of <r,u>, <w,u>, <r,r>: the scalars of the next iteration (:175-181).
		auto next_scalars = [&](const double (&tot)[3], bool first) {
			st.gamma_old = st.gamma;
			st.gamma = tot[0];
			st.delta = tot[1];
			st.rr = tot[2];
			if (first) {
				st.beta = 0.0;
				st.alpha = __ddiv_rn(tot[0], tot[1]);
			} else {
				st.beta = __ddiv_rn(tot[0], st.gamma_old);
				st.alpha = __ddiv_rn(1.0, __dsub_rn(__ddiv_rn(tot[1], tot[0]), __ddiv_rn(st.beta, st.alpha)));
			}
		};
		if (!st.done) {
			B.ghosts<HB>(A, ghost_rows, *ghost_count, load, put);
			__syncthreads();
			double v[3] = {0.0, 0.0, 0.0};
			B.march<D, UNIT, false>(A, sm, 1.0, [&](int d, double, double wi) {  // w = A u (:141-143)
				w[d] = wi;
				v[0] = fma(r[d], u[d], v[0]);
				v[1] = fma(wi, u[d], v[1]);
				v[2] = fma(r[d], r[d], v[2]);
				B.publish(A, out, d, mul(wi, im));
			});
			auto new_m = [&]() {  // m = w .* iM (:158): every thread has left the stencil pass
				if (B.own)
#pragma unroll
					for (int d = 0; d < D; d++)
						if (d < B.nd) sm[B.so + d * B.pp] = mul(w[d], im);
			};
			if (!group_sum<3, true>(g, round, v, new_m, [&](int lane, const double (&tot)[3]) {
				    if (lane == 0) next_scalars(tot, true);
			    }))
				return;
			for (int it = 1; !st.done; it++) {
				in = faces + (it & 1) * other;
				out = faces + (~it & 1) * other;
				B.ghosts<HB>(A, ghost_rows, *ghost_count, load, put);
				__syncthreads();
				const double alpha = st.alpha, beta = st.beta;
				v[0] = v[1] = v[2] = 0.0;
				B.march<D, UNIT, false>(A, sm, 1.0, [&](int d, double mi, double ni) {  // n = A m (:161-184)
					const double qi = add(mi, mul(beta, at(0, d)));       // :200
					const double si = add(w[d], mul(beta, at(1, d)));     // :203
					const double pi = add(u[d], mul(beta, at(2, d)));     // :206
					const double zi = add(ni, mul(beta, at(3, d)));       // :209
					const double xi = add(at(4, d), mul(alpha, pi));      // :215
					at(0, d) = qi;
					at(1, d) = si;
					at(2, d) = pi;
					at(3, d) = zi;
					at(4, d) = xi;
					r[d] = add(r[d], mul(-alpha, si));                    // :212
					u[d] = add(u[d], mul(-alpha, qi));                    // :218
					w[d] = add(w[d], mul(-alpha, zi));                    // :221
					B.publish(A, out, d, mul(w[d], im));
					v[0] = fma(r[d], u[d], v[0]);
					v[1] = fma(w[d], u[d], v[1]);
					v[2] = fma(r[d], r[d], v[2]);
				});
				if (!group_sum<3, true>(g, round, v, new_m, [&](int lane, const double (&tot)[3]) {
					    if (lane != 0) return;
					    // The stop test uses <r,r> from the top of this iteration (:173, :227).
					    const double rr = st.rr;
					    st.err = sqrt(__ddiv_rn(rr, st.bb));
					    if (hist) A.hist[it] = st.err;
					    if (st.err <= A.tol_in) stop(st, STOP_CONVERGED, it);
					    else if (it >= A.maxiter) stop(st, STOP_MAXITER, A.maxiter + 1);
					    if (st.done) st.rr = rr;
					    else next_scalars(tot, false);
				    }))
					return;
			}
			if (B.own && (!GLOBAL || A.nsm > 4))
				for (int d = 0; d < B.nd; d++) stl2(x + B.go + d * B.s3, at(4, d));
		}
		if (blockIdx.x % A.G == 0 && t == 0) write_state(st, A, unit);
		__syncthreads();  // shared memory is reused by the next right-hand side
	}
}

// ---------------------------------------------------------------------------
// BiCGStab (BiCgStab.hpp:157-232), FP64.  Shared memory holds p and s with
// their ghosts and the thread's own points of x and r_hat; r, v and t are in
// registers.  Three group reductions an iteration; the first publishes the
// boundary rows of v, the third those of r, and every block forms its ghosts
// of p and s from them (times iM at each read, as the reference rounds p_hat
// and s_hat).  Boxes of more than 8 planes leave x in global memory (A.nsm 1).
// ---------------------------------------------------------------------------
template <int D, int TMAX, bool UNIT>
__global__ void __launch_bounds__(TMAX, 1) k_res_bicg(const __grid_constant__ ResArgs A) {
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ ResGroup gsh;
	__shared__ KrylovState st;
	ResGroup *const g = &gsh;
	const ResBox B(A);
	const int t = threadIdx.x, T = blockDim.x;
	const int elems = B.pp * (A.nd + 2) + 1;
	double *const sp = reinterpret_cast<double *>(smem), *const ss = sp + elems;
	constexpr bool GLOBAL = D > 8;
	double *const fh = ss + elems + t;  // own r_hat of plane d at [d * T]
	double *const rfaces = static_cast<double *>(A.edge) + (size_t)blockIdx.x * B.face_rows * A.n1;
	// v's faces of two iterations: a block publishes new rows while a neighbour
	// may still form its p from the old ones.
	const size_t other = (size_t)gridDim.x * B.face_rows * A.n1;
	const double *vin = nullptr;
	if (t == 0) group_init(g, A);
	int *const ghost_count = reinterpret_cast<int *>(smem + ghost_table_offset(A, sizeof(double), 2, A.nsm, A.RG, T));
	int2 *const ghost_rows = reinterpret_cast<int2 *>(ghost_count + 2);
	B.table(A, ghost_rows, ghost_count);
	unsigned round = 0;
	const double im = A.iM;
	constexpr int HB = 4;
	double hr[HB], hw[HB];
	auto load_r = [&](int k, int from) { hr[k] = ldl2(rfaces + from); };
	auto load_rv = [&](int k, int from) {
		hr[k] = ldl2(rfaces + from);
		hw[k] = ldl2(vin + from);
	};
	for (int unit = blockIdx.x / A.G; unit < A.lanes; unit += A.groups) {
		double *const x = A.x + (size_t)unit * A.npts;
		const bool hist = A.hist && unit == 0 && blockIdx.x % A.G == 0;
		const bool xg = GLOBAL && A.nsm < 2;
		double *const fx = xg ? x + B.go : fh + A.nd * T;  // own x of plane d at [d * xstep]
		const int xstep = xg ? B.s3 : T;
		for (int e = t; e < 2 * elems; e += T) sp[e] = 0.0;
		__syncthreads();
		double r[D], vv[D], tt[D];
		{
			double v[2] = {0.0, 0.0};
			B.residual<D, UNIT>(A, x, A.rhs + (size_t)unit * A.npts, [&](int d, double xi, double bi, double ri) {
				r[d] = ri;
				fx[d * xstep] = xi;
				fh[d * T] = ri;  // r_hat = r (:153)
				B.publish(A, rfaces, d, ri);
				v[0] = fma(bi, bi, v[0]);
				v[1] = fma(ri, ri, v[1]);
			});
			if (!group_sum<2, true>(g, round, v, Nothing(), [&](int lane, const double (&tot)[2]) {
				    if (lane != 0) return;
				    initial_state(st, A, tot[0], tot[1], hist);
				    st.rho = tot[1];  // <r, r_hat> with r_hat == r (:159-160)
				    if (!st.done && st.rho == 0.0) stop(st, STOP_RHO, 1);
			    }))
				return;
		}
		for (int it = 1; !st.done; it++) {
			// ---- 1: p = r + beta p - beta omega v (p = r first), v = A p_hat, <v, r_hat>.
			double *const vnew = rfaces + (1 + (it & 1)) * other;
			vin = rfaces + (1 + (~it & 1)) * other;
			{
				const bool first = it == 1;
				const double beta = st.beta, bo = st.bo;
				auto new_p = [&](double ri, double pi, double vi) {
					return first ? ri : add(add(ri, mul(beta, pi)), mul(bo, vi));  // :168, :171
				};
				if (first) B.ghosts<HB>(A, ghost_rows, *ghost_count, load_r, [&](int k, int off) { sp[off] = hr[k]; });
				else B.ghosts<HB>(A, ghost_rows, *ghost_count, load_rv, [&](int k, int off) { sp[off] = new_p(hr[k], sp[off], hw[k]); });
				if (B.own)
#pragma unroll
					for (int d = 0; d < D; d++)
						if (d < B.nd) {
							double *const p = sp + B.so + d * B.pp;
							*p = new_p(r[d], *p, first ? 0.0 : vv[d]);
						}
				__syncthreads();
				double v[1] = {0.0};
				B.march<D, UNIT, true>(A, sp, im, [&](int d, double, double vi) {  // :178-180
					vv[d] = vi;
					v[0] = fma(vi, fh[d * T], v[0]);
					B.publish(A, vnew, d, vi);
				});
				if (!group_sum<1, true>(g, round, v, Nothing(), [&](int lane, const double (&tot)[1]) {
					    if (lane == 0) st.alpha = __ddiv_rn(st.rho, tot[0]);  // :186
				    }))
					return;
			}
			// ---- 2: s = r - alpha v, t = A s_hat; <s,s>, <t,s>, <t,t>.
			const double alpha = st.alpha;
			vin = vnew;
			{
				B.ghosts<HB>(A, ghost_rows, *ghost_count, load_rv, [&](int k, int off) { ss[off] = add(hr[k], mul(-alpha, hw[k])); });  // :189
				if (B.own)
#pragma unroll
					for (int d = 0; d < D; d++)
						if (d < B.nd) ss[B.so + d * B.pp] = add(r[d], mul(-alpha, vv[d]));
				__syncthreads();
				double v[3] = {0.0, 0.0, 0.0};
				B.march<D, UNIT, true>(A, ss, im, [&](int d, double si, double ti) {  // :204-206
					tt[d] = ti;
					v[0] = fma(si, si, v[0]);
					v[1] = fma(ti, si, v[1]);
					v[2] = fma(ti, ti, v[2]);
				});
				if (!group_sum<3>(g, round, v, Nothing(), [&](int lane, const double (&tot)[3]) {
					    if (lane != 0) return;
					    st.s_norm2 = tot[0];  // :192-193
					    st.s_exit = tot[0] < __dmul_rn(A.tol_in, A.tol_in);  // :194
					    if (!st.s_exit) st.omega = __ddiv_rn(tot[1], tot[2]);  // :212
				    }))
					return;
			}
			// ---- 3: x += alpha p_hat (+ omega s_hat), r = s - omega t; <r,r>, <r, r_hat>.
			const double omega = st.omega;
			const bool s_exit = st.s_exit != 0;
			double v[2] = {0.0, 0.0};
			if (B.own)
#pragma unroll
				for (int d = 0; d < D; d++) {
					if (d >= B.nd) break;
					const double ph = mul(sp[B.so + d * B.pp], im), si = ss[B.so + d * B.pp];
					const double x1 = add(fx[d * xstep], mul(alpha, ph));
					if (s_exit) {
						fx[d * xstep] = x1;  // :196
						continue;
					}
					fx[d * xstep] = add(x1, mul(omega, mul(si, im)));  // :216
					r[d] = add(si, mul(-omega, tt[d]));            // :219
					B.publish(A, rfaces, d, r[d]);
					v[0] = fma(r[d], r[d], v[0]);
					v[1] = fma(r[d], fh[d * T], v[1]);
				}
			if (!group_sum<2, true>(g, round, v, Nothing(), [&](int lane, const double (&tot)[2]) {
				    if (lane != 0) return;
				    if (s_exit) {
					    stop(st, STOP_SNORM, it);
					    return;
				    }
				    st.rr = tot[0];
				    st.err = sqrt(__ddiv_rn(tot[0], st.bb));  // :226
				    if (hist) A.hist[it] = st.err;
				    if (st.err <= A.tol_in) {                   // :228
					    stop(st, STOP_CONVERGED, it);
				    } else if (omega == 0.0) {                  // :229
					    stop(st, STOP_OMEGA, it);
				    } else {
					    st.rho_prev = st.rho;                    // :231
					    if (it >= A.maxiter) {
						    stop(st, STOP_MAXITER, A.maxiter + 1);
					    } else {
						    st.rho = tot[1];                     // next iteration :159-160
						    if (tot[1] == 0.0) stop(st, STOP_RHO, it + 1);  // :162
						    st.beta = __dmul_rn(__ddiv_rn(st.rho, st.rho_prev), __ddiv_rn(st.alpha, st.omega));  // :166
						    st.bo = __dmul_rn(-st.beta, st.omega);
					    }
				    }
			    }))
				return;
		}
		if (st.reason != STOP_EARLY && B.own && !xg)
			for (int d = 0; d < B.nd; d++) stl2(x + B.go + d * B.s3, fx[d * xstep]);
		if (blockIdx.x % A.G == 0 && t == 0) write_state(st, A, unit);
		__syncthreads();  // shared memory is reused by the next right-hand side
	}
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
namespace {

typedef void (*ResKernel)(const ResArgs);

// Box shapes: C rows x at most D planes per thread, at most T threads, so many
// blocks per SM.  The last ones, one row per thread, are those of pipelined CG
// and BiCGStab.
constexpr int kShapes = 10, kCgShapes = 6;
constexpr int kShapeC[kShapes] = {1, 1, 2, 2, 3, 2, 1, 1, 1, 1}, kShapeD[kShapes] = {2, 8, 8, 16, 16, 16, 2, 4, 8, 16},
              kShapeT[kShapes] = {512, 512, 512, 512, 384, 256, 512, 512, 512, 384},
              kShapeB[kShapes] = {1, 1, 1, 1, 1, 2, 1, 1, 1, 1};
// Fields of a solver in shared memory with ghosts, and own points only (of
// which the last shape may leave some in global memory); fields whose faces
// it publishes.
constexpr int kGhosted[4] = {0, 2, 1, 1}, kOwn[4] = {0, 2, 0, 5}, kFaces[4] = {0, 3, 1, 2};  // by solver id

template <class V, bool UNIT>
ResKernel cg_kernel(int shape) {
	switch (shape) {
	case 0: return k_res_cg<V, 1, 2, 512, 1, UNIT>;
	case 1: return k_res_cg<V, 1, 8, 512, 1, UNIT>;
	case 2: return k_res_cg<V, 2, 8, 512, 1, UNIT>;
	case 3: return k_res_cg<V, 2, 16, 512, 1, UNIT>;
	case 4: return k_res_cg<V, 3, 16, 384, 1, UNIT>;
	default: return k_res_cg<V, 2, 16, 256, 2, UNIT>;
	}
}

template <bool UNIT>
ResKernel krylov_kernel(int ks, int shape) {
	switch (shape) {
	case 6: return ks == SEDI_BICGSTAB ? (ResKernel)k_res_bicg<2, 512, UNIT> : (ResKernel)k_res_pcg<2, 512, UNIT>;
	case 7: return ks == SEDI_BICGSTAB ? (ResKernel)k_res_bicg<4, 512, UNIT> : (ResKernel)k_res_pcg<4, 512, UNIT>;
	case 8: return ks == SEDI_BICGSTAB ? (ResKernel)k_res_bicg<8, 512, UNIT> : (ResKernel)k_res_pcg<8, 512, UNIT>;
	default: return ks == SEDI_BICGSTAB ? (ResKernel)k_res_bicg<16, 384, UNIT> : (ResKernel)k_res_pcg<16, 384, UNIT>;
	}
}

ResKernel kernel_for(int ks, bool fp32, bool unit, int shape) {
	if (ks != SEDI_CG) return unit ? krylov_kernel<true>(ks, shape) : krylov_kernel<false>(ks, shape);
	if (fp32) return cg_kernel<float2, false>(shape);  // FP32 folds b, c into its multiply-adds
	return unit ? cg_kernel<double, true>(shape) : cg_kernel<double, false>(shape);
}

struct Plan {
	int shape = -1, G = 0, groups = 0, RG = 0, T = 0, s2 = 0, nd = 0, nsm = 0;
	size_t smem = 0;
};

// Device memory of a launch: the groups' reduction words, then the boxes' faces.
size_t word_bytes(int G, int groups) { return sizeof(Word2) * res_words(G) * groups; }
size_t buffer_bytes(int ks, int shape, int G, int groups, int nd, int RG, int n1) {
	return word_bytes(G, groups) +
	       (stamped(ks, kShapeC[shape]) ? 16 : 8) * (size_t)kFaces[ks] * groups * G * (2 * nd + 2 * RG * kShapeC[shape]) * n1;
}

// Plan with the smallest estimated time of an iteration of `units` solves, and
// that time in cycles; *most grows to the buffer of any plan for at most `units`
// solves.  Measured on B200 (FP64, 1.95 GHz) before the ghost rows came from a
// table, which took 1500-6000 cycles off every CG shape alike (16384 points now
// 32000; the rule against the streaming sweeps is that much on their side): the
// two reductions, ghost rows and launch of each phase take 9000-11000 cycles
// between blocks; a point adds 1.3 where A p stays in registers (2048 points a block 13600, 8192
// 20100), 1.65 with two stencil passes (16384: 38000), 1.8 at three rows a
// thread (12672: 32500), and 3.2 with two blocks on an SM (2 x 8192: 37400).
// Pipelined CG: 256 points a block 7700, 2048 10400, 4096 14000; BiCGStab: 512
// points 19000, 2048 24000, 4096 29000, 6144 (x in L2) 52000; pipelined CG's
// 6144 points (two or three fields in L2) 27700.
Plan plan_for(int ks, const Geo &g, int units, int sms, size_t smem_max, double *cycles, size_t *most = nullptr) {
	constexpr double kPoint[kCgShapes] = {1.3, 1.3, 1.3, 1.65, 1.8, 3.2};
	constexpr double kSync[4] = {0.0, 16000.0, 9000.0, 6000.0}, kPointOf[4] = {0.0, 2.9, 0.0, 1.6};  // by solver id
	Plan best;
	for (int sh = ks == SEDI_CG ? 0 : kCgShapes; sh < (ks == SEDI_CG ? kCgShapes : kShapes); sh++) {
		const int C = kShapeC[sh], slots = sms * kShapeB[sh];  // blocks at once
		for (int RG = kShapeT[sh] / g.n1; RG >= 1; RG--) {
			if (RG > 1 && (RG - 1) * C >= g.n2) continue;  // a row group with nothing to do
			const int T = (RG * g.n1 + 31) / 32 * 32, B2 = RG * C, s2 = (g.n2 + B2 - 1) / B2;
			for (int nd = 1; nd <= kShapeD[sh] && nd <= g.n3; nd++) {
				const long long G = (long long)s2 * ((g.n3 + nd - 1) / nd);
				const size_t ghosted = ((size_t)(g.n1 + 1) * (B2 + 2) * (nd + 2) + 1) * kGhosted[ks] * 8 + ghost_table_bytes(B2, nd),
				             own = (size_t)nd * T * 8;
				int nsm = kOwn[ks];
				if (sh == kShapes - 1)
					while (nsm > (ks == SEDI_BICGSTAB ? 1 : 0) && ghosted + nsm * own > smem_max) nsm--;
				const size_t smem = ghosted + nsm * own;
				if (G > slots || smem * kShapeB[sh] > smem_max) continue;
				const int groups = units < slots / (int)G ? units : slots / (int)G;
				if (most) {
					const size_t bytes = buffer_bytes(ks, sh, (int)G, groups, nd, RG, g.n1);
					if (bytes > *most) *most = bytes;
				}
				const double point = ks == SEDI_CG ? kPoint[sh < kCgShapes ? sh : 0] : kPointOf[ks] * (ks == SEDI_BICGSTAB && nd > 8 ? 1.7 : 1.0);
				const double deep = ks != SEDI_CG && nd > 4 ? 1500.0 : 0.0;  // the deeper kernels' start-up
				const double cost = ((G > 1 ? kSync[ks] + 15.0 * G : kSync[ks] / 3.0) + deep +
				                     (point + 0.75 * (kOwn[ks] - nsm)) * T * C * nd) *
				                    ((units + groups - 1) / groups);
				if (best.shape >= 0 && cost >= *cycles) continue;
				*cycles = cost;
				best.shape = sh;
				best.G = (int)G;
				best.groups = groups;
				best.RG = RG;
				best.T = T;
				best.s2 = s2;
				best.nd = nd;
				best.nsm = nsm;
				best.smem = smem;
			}
		}
	}
	return best;
}

// Estimated time of an iteration of the streaming sweeps on a batch, in cycles
// of the same clock: launches and latency, then HBM (words per point and lane;
// BiCGStab's 15 at five sixths of CG's rate), more where the tiles overhang
// the grid.  Measured (us): pipelined CG 32^3 x 64 60, 64^3 x 64 374; BiCGStab
// 82, 457; CG FP64
// 32^3 x 16 27, 64^3 x 64 188, 96^3 x 64 578, 128^3 x 64 1418; FP32 64^3 x 64
// 122, 96^3 x 64 320, 128^3 x 64 798.
double stream_cycles(int ks, const Geo &g, int lanes, bool fp32) {
	const double over = (double)((g.n1 + 31) / 32 * 32) * ((g.n2 + 31) / 32 * 32) / ((double)g.n1 * g.n2);
	constexpr double kLaunch[4] = {0.0, 42.0, 26.0, 18.0}, kWords[4] = {0.0, 18.0, 7.5, 16.0};  // by solver id
	return 1950.0 * (kLaunch[ks] + kWords[ks] * (fp32 ? 4.0 : 8.0) * (double)g.n * lanes * std::sqrt(over) / 5.9e6);
}

}  // namespace

struct Resident {
	struct {
		Plan plan;
		int units = 0;      // solves the plan is for
	} plans[2];             // a last batch may be smaller than the others
	int now = 0;            // the one whose launch the buffer is laid out for
	int ks = 0;
	bool fp32 = false, unit = false;
	size_t shared = 0;      // shared memory of a block, at most
	bool ready[kShapes] = {};
	void *buf = nullptr;    // the owner's memory, enough for every plan
	size_t buf_bytes = 0;
	unsigned long long launch = 0;
	int device = 0, sms = 0;
	cudaEvent_t done = nullptr;  // after the latest launch
	RoomUse use;                 // of that launch while it may run
};

// Launches that may be running, oldest first (resident_room.h says which of
// them a new one waits for).  One entry per context, taken out when the context
// goes.
static std::mutex g_running_mu;
static std::vector<Resident *> g_running;

static void running_remove(Resident *R) {
	for (size_t i = 0; i < g_running.size(); i++)
		if (g_running[i] == R) {
			g_running.erase(g_running.begin() + (long)i);
			return;
		}
}

// Makes plan p's kernel ready; false where it cannot run.
static bool kernel_ready(Resident *R, const Plan &p) {
	if (R->ready[p.shape]) return true;
	const void *const k = (const void *)kernel_for(R->ks, R->fp32, R->unit, p.shape);
	int per_sm = 0;
	// (The attribute is the kernel's, whoever launches it: its largest use.)
	if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(R->shared / kShapeB[p.shape])) !=
	        cudaSuccess ||
	    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kShapeT[p.shape], R->shared / kShapeB[p.shape]) !=
	        cudaSuccess ||
	    per_sm < kShapeB[p.shape]) {
		cudaGetLastError();
		return false;
	}
	return R->ready[p.shape] = true;
}

// Plan for `units` solves, chosen by their number and the grid alone (so a
// result does not depend on the context's room for more): 10 FP64 solves of
// 58^3 on a plan for 16 ran as 9 groups and one more round.  The one in use
// stays where the kernel of a better one cannot run.  Two are kept, and the
// buffer holds any, so that no call allocates and batches whose size alternates
// do not search again (1-110 us).
static int use_plan(Ctx *c, Resident *R, int units) {
	if (units == R->plans[R->now].units) return 0;
	const int other = R->now ^ 1;
	if (units != R->plans[other].units) {
		double cycles = 0.0;
		const Plan p = plan_for(R->ks, c->g, units, R->sms, R->shared, &cycles);
		if (p.shape < 0 || !kernel_ready(R, p)) return 0;
		R->plans[other].plan = p;
		R->plans[other].units = units;
	}
	// No word may carry a stamp of a launch to come, whatever another plan left in its place.
	const Plan &p = R->plans[other].plan;
	const cudaError_t e =
	    cudaMemsetAsync(R->buf, 0, buffer_bytes(R->ks, p.shape, p.G, p.groups, p.nd, p.RG, c->g.n1), c->stream);
	if (e != cudaSuccess) return set_cuda_error(c, e, "resident solver");
	R->now = other;
	return 0;
}

// What a block may use and the blocks at once, of the current device; of a B200
// where there is none.
static bool resident_limits(int device, int *sms, size_t *shared) {
	int coop = 1, smem_max = 232448;
	*sms = 148;
	if (device >= 0 && (cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
	                    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess ||
	                    cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess)) {
		cudaGetLastError();
		return false;
	}
	// Beside the static arrays and what the system keeps, for up to two blocks of an SM.
	*shared = (size_t)smem_max - 2 * (sizeof(ResGroup) + sizeof(CgState<2>) + 1024);
	if (*sms > kResMaxBlocks / 2) *sms = kResMaxBlocks / 2;
	return coop != 0;
}

// Whether `lanes` right-hand sides of a grid are solved on chip; then *most is
// the buffer that any number of them up to that needs.
static bool resident_takes(int ks, bool fp32, int lanes, const Geo &g, int sms, size_t shared, size_t *most) {
	*most = 0;
	if (ks != SEDI_CG && fp32) return false;
	if (g.n1 > 512 || g.n > (1 << 22)) return false;  // no box shape takes them
	double cycles = 0.0;
	const Plan p = plan_for(ks, g, fp32 ? (lanes + 1) / 2 : lanes, sms, shared, &cycles, most);
	if (p.shape < 0) return false;
	if (lanes == 1) *most = buffer_bytes(ks, p.shape, p.G, p.groups, p.nd, p.RG, g.n1);  // (one plan)
	// A pair of FP32 lanes takes 1.45-1.7 times what the estimate says of an FP64
	// lane (conversions for its FP64 sums, less since the ghost table); at 1.6 no
	// measured batch goes on chip that is slower there (us an iteration, on chip and
	// streaming: 80^3 x 32 110 / 133; 96^3 x 16 105 / 99, 96^3 x 32 208 / 168,
	// 128^3 x 16 230 / 201); two that would gain 7% stream (64^3 x 64, 107 / 115,
	// and 80^3 x 64, 221 / 240).  One right-hand side has no streaming form at
	// these sizes (its march kernels take 11.7 us an iteration at 32^3, 47 at
	// 128^3; this 5.5 and 16.4), a batch does.
	if (fp32) cycles *= 1.6;
	return lanes <= 1 || cycles <= stream_cycles(ks, g, lanes, fp32);
}

// Buffer of a resident solver (see resident_alloc), 0 where there is none.
size_t resident_bytes(int ks, bool fp32, int lanes, const Geo &g) {
	int device = -1, count = 0, sms = 0;
	size_t shared = 0, most = 0;
	if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0 || cudaGetDevice(&device) != cudaSuccess) {
		cudaGetLastError();
		device = -1;
	}
	return resident_limits(device, &sms, &shared) && resident_takes(ks, fp32, lanes, g, sms, shared, &most) ? most : 0;
}

// A resident solver for up to `lanes` right-hand sides of the context's grid,
// planned for `batch` of them; *out stays null where the grid or the device does
// not take one (the streaming and march kernels serve those).  The caller gives
// it *bytes of device memory, 16-byte aligned, with resident_bind: behind its
// vectors, since an allocation of its own took 0.2-0.4 ms of a context's creation.
int resident_alloc(Ctx *c, int ks, bool fp32, int lanes, int batch, Resident **out, size_t *bytes) {
	*out = nullptr;
	*bytes = 0;
	int sms = 0;
	size_t shared = 0, most = 0;
	if (!resident_limits(c->device, &sms, &shared) || !resident_takes(ks, fp32, lanes, c->g, sms, shared, &most)) return 0;
	Resident *R = new (std::nothrow) Resident();
	if (!R) return SEDI_ERR_NOMEM;
	R->ks = ks;
	R->fp32 = fp32;
	R->unit = c->k.b == 1.0 && c->k.c == 1.0;
	R->shared = shared;
	R->device = c->device;
	R->sms = sms;
	R->buf_bytes = most;
	const int units = fp32 ? (batch + 1) / 2 : batch;
	double cycles = 0.0;
	R->plans[0].plan = plan_for(ks, c->g, units, sms, shared, &cycles);
	R->plans[0].units = units;
	if (R->plans[0].plan.shape < 0 || !kernel_ready(R, R->plans[0].plan) ||
	    cudaEventCreateWithFlags(&R->done, cudaEventDisableTiming) != cudaSuccess) {
		cudaGetLastError();
		resident_free(R);
		return 0;
	}
	*out = R;
	*bytes = most;
	return 0;
}

// The owner's memory for R; zeroed on the context's stream, for which the caller waits.
int resident_bind(Ctx *c, Resident *R, void *buf) {
	R->buf = buf;
	const cudaError_t e = cudaMemsetAsync(buf, 0, R->buf_bytes, c->stream);
	return e == cudaSuccess ? 0 : set_cuda_error(c, e, "resident solver");
}

void resident_free(Resident *R) {
	if (!R) return;
	{
		std::lock_guard<std::mutex> lk(g_running_mu);
		running_remove(R);
	}
	if (R->done) cudaEventDestroy(R->done);
	delete R;
}

// Solves io.lanes right-hand sides on the context's stream.
int resident_launch(Ctx *c, Resident *R, const ResIO &io) {
	const int units = R->fp32 ? (io.lanes + 1) / 2 : io.lanes;
	if (units < 1) return 0;
	const int rc = use_plan(c, R, units);
	if (rc) return rc;
	const Plan &p = R->plans[R->now].plan;
	const int groups = units < p.groups ? units : p.groups;
	ResArgs a;
	a.n1 = c->g.n1;
	a.n2 = c->g.n2;
	a.n3 = c->g.n3;
	a.npts = c->g.n;
	a.a = c->k.a;
	a.b = c->k.b;
	a.c = c->k.c;
	a.iM = 1.0 / c->k.a;  // stochastic-estimator.cc:103
	a.lanes = io.lanes;
	a.G = p.G;
	a.groups = groups;
	a.s2 = p.s2;
	a.RG = p.RG;
	a.nd = p.nd;
	a.nsm = p.nsm;
	for (int k = 0; k < 4; k++) a.scratch[k] = io.scratch[k];
	a.rhs = io.rhs;
	a.x = io.x;
	a.xlo = (float2 *)io.xlo;
	a.words = (Word2 *)R->buf;
	a.edge = (char *)R->buf + word_bytes(p.G, p.groups);
	a.stamp = ++R->launch << 36;
	a.tol = io.tol;
	a.tol_in = io.tol_in;
	a.maxiter = io.maxiter;
	a.period = io.period;
	a.o_err = io.o_err;
	a.o_bb = io.o_bb;
	a.o_rr = io.o_rr;
	a.o_exit = io.o_exit;
	a.o_reason = io.o_reason;
	a.o_done = io.o_done;
	a.o_snorm = io.o_snorm;
	a.o_omega = io.o_omega;
	a.o_rho = io.o_rho;
	a.hist = io.hist;
	a.err = io.err;
	void *args[] = {&a};
	const int blocks = groups * p.G;
	const RoomUse use = room_use(blocks, p.G, R->sms);
	std::lock_guard<std::mutex> lk(g_running_mu);
	// A context's launch has ended when its next one comes: a call waits for its
	// stream, an estimate's next step for its event.
	running_remove(R);
	std::vector<Resident *> others;
	std::vector<RoomUse> uses;
	for (size_t i = 0; i < g_running.size();) {
		Resident *const o = g_running[i];
		if (o->device == R->device) {
			if (cudaEventQuery(o->done) == cudaSuccess) {
				g_running.erase(g_running.begin() + (long)i);
				continue;
			}
			others.push_back(o);
			uses.push_back(o->use);
		}
		i++;
	}
	const std::vector<char> wait = room_waits(uses, use, R->sms);
	for (size_t i = 0; i < others.size(); i++) {
		if (!wait[i]) continue;
		const cudaError_t w = cudaStreamWaitEvent(c->stream, others[i]->done, 0);
		if (w != cudaSuccess) return set_cuda_error(c, w, "resident solver launch");
	}
	cudaError_t e = cudaLaunchCooperativeKernel((const void *)kernel_for(R->ks, R->fp32, R->unit, p.shape), dim3((unsigned)blocks),
	                                            dim3((unsigned)p.T), args, p.smem, c->stream);
	if (e == cudaSuccess) {
		e = cudaEventRecord(R->done, c->stream);
		R->use = use;
		g_running.push_back(R);
	}
	if (e != cudaSuccess) return set_cuda_error(c, e, "resident solver launch");
	c->launches++;
	return 0;
}

}  // namespace sedi
