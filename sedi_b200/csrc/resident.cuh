// Device helpers of the resident solvers (resident.cu): one cooperative
// launch runs whole solves, each by a group of blocks (one per SM) that keeps
// the Krylov fields of its right-hand side on chip.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "sedi_common.cuh"

namespace sedi {

constexpr int kResMaxDots = 6;                           // doubles of one group reduction
constexpr int kResMaxWarps = 16;                         // warps of a block
constexpr long long kResWaitClocks = 4000000000ll;        // bound of every wait: 2 s at 2 GHz

// 16 bytes written and read as one access.
struct __align__(16) Word2 {
	unsigned long long a, b;
};

__device__ __forceinline__ void swap2(Word2 *p, unsigned long long a, unsigned long long b) {
	asm volatile(
	    "{\n\t.reg .b128 t, old;\n\tmov.b128 t, {%1, %2};\n\tatom.relaxed.gpu.global.exch.b128 old, [%0], t;\n\t}" ::"l"(p),
	    "l"(a), "l"(b)
	    : "memory");
}
__device__ __forceinline__ Word2 load2(const Word2 *p) {
	Word2 r;
	asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
	             : "=l"(r.a), "=l"(r.b)
	             : "l"(p)
	             : "memory");
	return r;
}
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
// A group's exchange of reduction results, in global memory: [2 parities of
// rounds][kResCopies][kResMaxDots][G] words stamped with their round.
constexpr int kResMaxBlocks = 320;  // G
constexpr int kResCopies = 2;
__host__ __device__ constexpr size_t res_words(int G) { return (size_t)2 * kResCopies * kResMaxDots * G; }

struct ResGroup {
	double red[kResMaxDots][kResMaxWarps];           // warp sums of the block
	double part[kResMaxDots][kResMaxBlocks / 32];    // sums of 32 blocks
	Word2 *words;             // global
	int *err;                 // device flag the host reads: a wait ran out
	unsigned long long base;  // stamps of this launch lie above it
	int G, m;                 // blocks of the group, this block's index in it
	int fail;                 // a wait of this block ran out
};

// Waits (bounded) until the word at p is stamped `stamp` and returns it.
__device__ __forceinline__ Word2 wait2(const Word2 *p, unsigned long long stamp, ResGroup *g) {
	Word2 w;
	const long long t0 = clock64();
	do {
		w = load2(p);
		if (w.b != stamp && clock64() - t0 > kResWaitClocks) {
			g->fail = 1;
			*(volatile int *)g->err = 1;  // (host memory for a single vector)
			break;
		}
	} while (w.b != stamp);
	return w;
}

// Sums of ND doubles over every thread of the group, in an order fixed by the
// launch shape; also the group's barrier.  between() runs in every thread
// after the block's sums are on their way and before the others' are waited
// for: work that hides the exchange.  Warp 0 calls fin(lane, totals) before the
// block goes on: what it leaves in shared memory every thread of the block
// sees.  False when a wait ran out (in every thread of the block).
//
// Every block publishes its sums and reads everybody's.  A word carries its
// value and the stamp of its round in one 16-byte access, so no flag and no
// fence stand between writer and reader; a block can be one round ahead of a
// block that still reads, hence two parities.  Words are written with atomic
// exchanges: on B200 a plain store may sit in the SM for 5000-6000 cycles
// before other SMs see it (a fence behind it takes 800-900 cycles), an exchange
// is performed in L2 at once.  A round of 128 blocks takes 2200 cycles (1.1
// us), of 2 blocks 1400; with plain stores 128 blocks took 9000, through an
// adding block 4300 and through clusters and distributed shared memory 10000
// (the hop between clusters again a plain store).
//
// FENCE: what any thread of the group wrote to global memory before the call
// is visible (through L2) to every thread after it.
template <int ND, bool FENCE = false, class Between, class Fin>
__device__ __forceinline__ bool group_sum(ResGroup *g, unsigned &round, double (&v)[ND], Between between, Fin fin) {
	static_assert(ND * kResCopies <= 32 && ND <= kResMaxDots, "dots");
	const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = blockDim.x >> 5;
	round++;
	warp_sum<ND>(v);
	if (lane == 0)
#pragma unroll
		for (int d = 0; d < ND; d++) g->red[d][warp] = v[d];
	__syncthreads();
	const int G = g->G, segs = (G + 31) / 32;
	const unsigned long long stamp = g->base + round;
	Word2 *const words = g->words + (round & 1) * kResCopies * kResMaxDots * G;
	if (warp == 0) {
#pragma unroll
		for (int d = 0; d < ND; d++) v[d] = lane < nw ? g->red[d][lane] : 0.0;
		warp_sum<ND>(v);
		if (G > 1) {
			if (FENCE) fence_gpu();
#pragma unroll
			for (int d = 0; d < ND; d++)
				if (lane / kResCopies == d)
					swap2(words + ((lane % kResCopies) * kResMaxDots + d) * G + g->m, __double_as_longlong(v[d]), stamp);
		}
	}
	between();
	if (G > 1) {
		for (int u = warp; u < ND * segs; u += nw) {  // a warp per 32 blocks of a sum
			const int d = u / segs, b = (u - d * segs) * 32 + lane;
			const Word2 *const word = words + ((g->m % kResCopies) * kResMaxDots + d) * G + b;
			double q[1] = {0.0};
			if (b < G) {
				Word2 w = load2(word);
				if (w.b != stamp) w = wait2(word, stamp, g);
				q[0] = __longlong_as_double(w.a);
				if (FENCE) fence_gpu();
			}
			warp_sum<1>(q);
			if (lane == 0) g->part[d][u - d * segs] = q[0];
		}
		__syncthreads();
	}
	if (warp == 0) {
		if (G > 1)
#pragma unroll
			for (int d = 0; d < ND; d++) {
				v[d] = 0.0;
				for (int k = 0; k < segs; k++) v[d] += g->part[d][k];
			}
		fin(lane, v);
	}
	__syncthreads();
	return !g->fail;
}

struct Nothing {
	__device__ void operator()() const {}
};

// Streamed accesses of fields only their owner block touches, and reads of
// what other blocks wrote before a fenced group_sum (both bypass L1).
__device__ __forceinline__ double ldl2(const double *p) { return __ldcg(p); }
__device__ __forceinline__ float2 ldl2(const float2 *p) { return __ldcg(p); }
__device__ __forceinline__ void stl2(double *p, double v) { __stcg(p, v); }
__device__ __forceinline__ void stl2(float2 *p, float2 v) { __stcg(p, v); }

}  // namespace sedi
