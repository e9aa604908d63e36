// SpMM on B200 (sm_100a): Y = diag(s_out) * A * diag(s_in) * X.
//
// Replaces FlashMatrix's CPU SpMM tasks (row_part_func / coo_func /
// block_spmm_task_impl::run_on_block, matrix/sparse_matrix.h:219-375, driven
// by block_compute_task::run, matrix/sparse_matrix.cpp:251-314).
//
// Layout in HBM (built once per matrix from the decoded 2D image, resident):
//   col      uint32[]           one entry stream.  Bit 31 is set on the last
//                               entry of a row; with bit 30 set, bits 0-29 hold
//                               a hot slot, else the column id.  First every
//                               row in ascending order: a row of 1..kExactMax
//                               entries as its entries in the order the
//                               reference visits them (ascending block column,
//                               then column); an empty or longer row as one
//                               entry naming the pack's zero row.  Then the
//                               entries of the longer rows (> kExactMax).
//   val      entry[]            only for weighted images, same order
//   hot_col  int32[H]           the H <= kHotMax columns of highest in-degree;
//                               entry slot s + 1 names hot_col[s], slot 0 the
//                               pack's zero row
//   ranges   range_t[]          work units, sorted by entry count (largest
//                               first): a run of consecutive rows of up to ~kRange
//                               entries, or one of the equal chunks (<= kChunk
//                               entries) of a longer row.  Each starts at a
//                               multiple of 8 entries and is padded to one
//                               with zero-row entries (after the last row end
//                               of a run they are never stored; in a chunk
//                               they add zeros), so steps need no bounds.
//   heavy    heavy_row[]        longer rows: spmm_fixup_kernel overwrites their
//                               Y rows with their chunk partials added in
//                               chunk order
// Scratch (allocated with the matrix):
//   xhot     (H+1) x 128 bytes  per call, the hot columns' X rows of the
//                               current panel, packed back to back (times s_in
//                               when given) after row 0, which stays zero
//   partial  AccT[chunks][kPartialStride]  chunk sums of longer rows
//
// Why the hot pack: the X gathers of an R-MAT graph are random 64-byte reads
// that mostly miss the L2, and a hot row shares its 128-byte line with a cold
// one.  Packing the highest in-degree rows (about 87% of the gathers at scale
// 24) two to a line keeps them in a range the L2 can hold.
//
// Execution: persistent grids whose lane groups take ranges round-robin and
// walk them as a stream of entries in aligned steps; when an entry closes a
// row, the group stores that row (the range's first row plus the rows closed
// before it).  Every row of up to kExactMax entries is summed by one group in
// the reference's order (bit-identical results).  No atomics: every output
// row is written exactly once.  Two row kernels share that scheme:
//   spmm_lane_kernel  every panel: a lane owns 2 to 32 bytes of each gathered
//                     row, the gathers of 8, 16 or 32 entries in flight per lane
//   spmv_kernel       k = 1 of small matrices and PageRank: a warp per range,
//                     gathers staged in shared memory
// Each call first packs the hot rows: pack_hot_vec_kernel in 16-byte units,
// pack_hot_kernel one element per thread (k = 1 and rows of odd widths).
#include "fmx_internal.h"

#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>

#include "part.h"

namespace fmx {

// ---------------------------------------------------------------------------
// Device helpers
// ---------------------------------------------------------------------------

// Arithmetic without contraction: dest = dest + src * w, rounded per step,
// like the reference's dest_row[j] += src_row[j] * data (no FMA).
__device__ __forceinline__ float acc_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float acc_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double acc_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double acc_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ int32_t acc_add(int32_t a, int32_t b) { return int32_t(uint32_t(a) + uint32_t(b)); }
__device__ __forceinline__ int32_t acc_mul(int32_t a, int32_t b) { return int32_t(uint32_t(a) * uint32_t(b)); }
__device__ __forceinline__ int64_t acc_add(int64_t a, int64_t b) { return int64_t(uint64_t(a) + uint64_t(b)); }
__device__ __forceinline__ int64_t acc_mul(int64_t a, int64_t b) { return int64_t(uint64_t(a) * uint64_t(b)); }

template <class A> __device__ __forceinline__ A to_acc(float v) { return A(v); }
template <class A> __device__ __forceinline__ A to_acc(double v) { return A(v); }
template <class A> __device__ __forceinline__ A to_acc(int32_t v) { return A(v); }
template <class A> __device__ __forceinline__ A to_acc(int64_t v) { return A(v); }
template <class A> __device__ __forceinline__ A to_acc(__nv_bfloat16 v) { return A(__bfloat162float(v)); }

template <class Y, class A> __device__ __forceinline__ Y from_acc(A v) { return Y(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_acc<__nv_bfloat16, float>(float v) { return __float2bfloat16_rn(v); }

// Packed FP32 pairs (sm_100 add.rn.f32x2): two IEEE round-to-nearest adds
// per instruction, the same results as two scalar adds.
__device__ __forceinline__ uint64_t pack2(float a, float b)
{
	uint64_t r;
	asm("mov.b64 %0, {%1,%2};" : "=l"(r) : "f"(a), "f"(b));
	return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &a, float &b)
{
	asm("mov.b64 {%0,%1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
	uint64_t r;
	asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}

// VEC elements of T: one 16-byte vector, or a scalar (VEC == 1).
template <class T, int VEC>
struct xvec {
	T v[VEC];
};

// Streaming stores (evict-first), so that the gathered rows keep the caches.
template <class T, int VEC>
__device__ __forceinline__ void st_y(T *p, const T (&v)[VEC])
{
	if constexpr (VEC * sizeof(T) == 16) {
		uint4 u;
		memcpy(&u, v, 16);
		__stcs(reinterpret_cast<uint4 *>(p), u);
	} else if constexpr (VEC * sizeof(T) == 32) {
		uint4 u[2];
		memcpy(u, v, 32);
		__stcs(reinterpret_cast<uint4 *>(p), u[0]);
		__stcs(reinterpret_cast<uint4 *>(p) + 1, u[1]);
	} else if constexpr (VEC * sizeof(T) == 8) {
		uint2 u;
		memcpy(&u, v, 8);
		__stcs(reinterpret_cast<uint2 *>(p), u);
	} else {
#pragma unroll
		for (int i = 0; i < VEC; i++) p[i] = v[i];
	}
}

// One whole sector (32-byte aligned).
template <class T, int VEC>
__device__ __forceinline__ void st_sector(T *p, const T (&v)[VEC])
{
	static_assert(VEC * sizeof(T) == 32, "32 bytes");
	uint32_t u[8];
	memcpy(u, v, 32);
	asm volatile("st.global.cs.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
			:: "l"(p), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]) : "memory");
}

// Programmatic dependent launch.  A call's kernels are launched with the
// attribute, so that the next one's blocks come in while the last one's drain;
// dep_wait() holds them until the kernel before has completed.  Every kernel of
// such a chain waits, and lets its successor in only then: when one starts,
// everything before its predecessor is complete, and the read-only loads see no
// line from before it.  fmx_spmm's first kernel, the pack, carries no attribute
// and follows all earlier work of the stream as usual.  Where a product starts
// with a dependent launch (spmm_packed; a PageRank iteration), the kernel before
// it is a plain one that never lets its successor in early (the solver's filter
// step, init_kernel), or one that itself waited first (the iteration before), or
// a copy.  What a kernel of the chain
// writes is read by plain loads only: ld.global.nc asks for data that nobody
// writes while the kernel is resident, and the compiler may move an __ldg, or
// a load through a const __restrict__ pointer, above the wait.
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... K, class... Args>
static cudaError_t launch_dep(void (*kern)(K...), unsigned grid, unsigned block, cudaStream_t st, Args... args)
{
	cudaLaunchAttribute at[1];
	at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at[0].val.programmaticStreamSerializationAllowed = 1;
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(grid);
	cfg.blockDim = dim3(block);
	cfg.stream = st;
	cfg.attrs = at;
	cfg.numAttrs = 1;
	return cudaLaunchKernelEx(&cfg, kern, K(args)...);
}

struct spmm_args {
	const uint32_t *col;
	const void *val;
	const range_t *ranges;
	const void *X;
	const void *xhot;    // packed hot rows of this panel, row stride hot_ld
	void *Y;
	const void *s_in;
	const void *s_out;
	void *partial;
	int64_t ldx, ldy;
	int hot_ld;      // elements per packed hot row
	int k;           // columns in this panel
	int G;           // lanes per row group
	int R;           // row groups per warp
	uint32_t n_ranges;
	const unsigned long long *state;     // PageRank's loop state (pr_epi), read by the forms of its loop
};

// The running sums of one lane: NV vectors of VEC elements.  FP32 with
// VEC == 4 or 8 is kept as packed pairs.
template <class A, int VEC, int NV>
struct accum {
	static constexpr bool kPacked = std::is_same<A, float>::value && (VEC % 2 == 0) && NV == 1;
	A s[NV][VEC];
	uint64_t p[VEC / 2 > 0 ? VEC / 2 : 1];

	__device__ __forceinline__ void zero()
	{
		if constexpr (kPacked) {
#pragma unroll
			for (int i = 0; i < VEC / 2; i++) p[i] = 0;
		} else {
#pragma unroll
			for (int v = 0; v < NV; v++)
#pragma unroll
				for (int i = 0; i < VEC; i++) s[v][i] = A(0);
		}
	}
	// s[v] += x (* m1) (* m2), each operation rounded (no contraction)
	template <class XT, int NMUL>
	__device__ __forceinline__ void add(int v, const xvec<XT, VEC> &x, A m1, A m2)
	{
		if constexpr (kPacked) {
			// products stay scalar __fmul_rn (never fused into the add);
			// only the adds are packed
#pragma unroll
			for (int i = 0; i < VEC / 2; i++) {
				float t0 = to_acc<float>(x.v[2 * i]), t1 = to_acc<float>(x.v[2 * i + 1]);
				if constexpr (NMUL >= 1) { t0 = __fmul_rn(t0, m1); t1 = __fmul_rn(t1, m1); }
				if constexpr (NMUL >= 2) { t0 = __fmul_rn(t0, m2); t1 = __fmul_rn(t1, m2); }
				p[i] = add2(p[i], pack2(t0, t1));
			}
		} else {
#pragma unroll
			for (int i = 0; i < VEC; i++) {
				A t = to_acc<A>(x.v[i]);
				if constexpr (NMUL >= 1) t = acc_mul(t, m1);
				if constexpr (NMUL >= 2) t = acc_mul(t, m2);
				s[v][i] = acc_add(s[v][i], t);
			}
		}
	}
	// s[0] += t
	__device__ __forceinline__ void add_terms(const A (&t)[VEC])
	{
		if constexpr (kPacked) {
#pragma unroll
			for (int i = 0; i < VEC / 2; i++) p[i] = add2(p[i], pack2(t[2 * i], t[2 * i + 1]));
		} else {
#pragma unroll
			for (int i = 0; i < VEC; i++) s[0][i] = acc_add(s[0][i], t[i]);
		}
	}
	__device__ __forceinline__ A get(int v, int i) const
	{
		if constexpr (kPacked) {
			float a, b;
			unpack2(p[i / 2], a, b);
			return (i & 1) ? b : a;
		} else {
			return s[v][i];
		}
	}
};

// The PageRank update at a row close (EPI): rows of the fixup's heavy list
// are left to the fixup.
struct pr_row {
	float pr1, deg;
	uint32_t slot;
};
__device__ __forceinline__ pr_row pr_load(const pr_epi &e, int64_t row)
{
	return {e.pr1[row], e.deg[row], __ldg(e.slot + row)};
}
__device__ __forceinline__ void pr_update(const pr_epi &e, int64_t row, const pr_row &o, float out, unsigned &cnt)
{
	const float p2 = __fadd_rn(__fmul_rn(out, e.damping), e.teleport);
	const float diff = fabsf(__fsub_rn(o.pr1, p2));
	cnt += diff < e.eps;
	e.pr[row] = p2;
	const float x = __fdiv_rn(p2, o.deg);
	e.in_next[row] = x;
	if (o.slot) e.xhot_next[o.slot] = x;
	e.pr1[row] = __fmul_rn(x, o.deg);
}

// The loop test (PageRank.cpp:96,124-129) by the last block of an iteration's
// last kernel, every thread of which comes here.
__device__ __forceinline__ void pr_finish(const pr_epi &e)
{
	__syncthreads();
	if (threadIdx.x != 0) return;
	__threadfence();
	if (atomicAdd(e.state + 3, 1ull) != gridDim.x - 1) return;
	__threadfence();
	e.state[3] = 0;
	const unsigned long long it = ++e.state[2], converged = atomicExch(e.state, 0ull);
	if (converged >= e.n || it >= e.max_iters) e.state[1] = 1;
}

// ---------------------------------------------------------------------------
// The row kernel: lane groups walk ranges.
//
// A lane owns VN elements of every X row it gathers, so a panel of k columns
// takes G = k / VN lanes and a warp runs 32 / G groups.  Groups take ranges
// round-robin and walk them U entries a step: all of a step's gathers, and
// the next step's column ids, are in flight before its adds.  Any width runs
// in whole lanes: VN is the widest unit that divides the rows (lane_width).
//
// What bounds it: the L1 data pipe (a gathered row costs about one data-pipe
// cycle to return and half a cycle of tag output, whatever lanes ask for it)
// and instruction issue.  Measured by ncu at R-MAT scale 22, k = 16 FP32: the
// former 32-byte lanes with 4 gathers in flight kept the pipe 82 % busy at
// 458 us with 106M wavefronts; 16-byte lanes with 8 in flight need 81M.  The
// row close is a branch: predicated stores cost every entry the conversion.
// Times of the former kernels -> this one (whole fmx_spmm, B200):
//   FP32 k = 16, R-MAT scale 16 / 20 / 22 / 24   41 / 177 / 512 / 1855 ->
//                                               21 / 119 / 411 / 1785 us
//   FP64 k = 8, scale 22                         593 -> 430 us
//   FP32 k = 10 / 33, scale 20                   427 / 1111 -> 156 / 684 us
//   int64 k = 4 weighted, scale 20               177 -> 149 us
//   D^-1/2 A D^-1/2, k = 16, symmetric scale 21  FP32 567 -> 471 us,
//                                                BF16 531 -> 393 us
// ---------------------------------------------------------------------------
__device__ __forceinline__ void ld32_nc(const void *p, uint32_t (&r)[8])
{
	asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
			: "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
			: "l"(p));
}

// VN elements of T in one load (2 to 32 bytes).  Volatile: a step's loads
// stay where they are written, all before the adds.  Not .nc: the kernel
// before may have written the rows while this one was already resident.
template <class T, int VN>
__device__ __forceinline__ xvec<T, VN> ld_n(const char *p)
{
	xvec<T, VN> r;
	if constexpr (VN * sizeof(T) == 32) {
		uint32_t v[8];
		asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
				: "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
				: "l"(p));
		memcpy(&r, v, 32);
	} else if constexpr (VN * sizeof(T) == 16) {
		uint32_t v[4];
		asm volatile("ld.global.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "l"(p));
		memcpy(&r, v, 16);
	} else if constexpr (VN * sizeof(T) == 8) {
		uint32_t v[2];
		asm volatile("ld.global.v2.b32 {%0,%1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "l"(p));
		memcpy(&r, v, 8);
	} else if constexpr (VN * sizeof(T) == 4) {
		uint32_t v;
		asm volatile("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p));
		memcpy(&r, &v, 4);
	} else {
		static_assert(VN == 1 && sizeof(T) == 2, "one 2-byte element");
		unsigned short v;
		asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p));
		memcpy(&r, &v, 2);
	}
	return r;
}

// The same for elements `stride` bytes apart, the first `live` of them (zeros
// behind).
template <class T, int VN>
__device__ __forceinline__ xvec<T, VN> ld_apart(const char *p, uint32_t stride, int live)
{
	static_assert(sizeof(T) == 2, "2-byte elements");
	xvec<T, VN> r;
#pragma unroll
	for (int i = 0; i < VN; i++) {
		unsigned short v;
		asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.u16 %0, 0;\n\t@q ld.global.u16 %0, [%1];\n\t}"
				: "=h"(v) : "l"(p + i * stride), "r"(uint32_t(i < live)));
		memcpy(&r.v[i], &v, 2);
	}
	return r;
}

// v = *p when `pred` holds (predicated, no branch)
__device__ __forceinline__ void ld_if(float &v, const float *p, bool pred)
{
	asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.global.nc.f32 %0, [%1];\n\t}"
			: "+f"(v) : "l"(p), "r"(uint32_t(pred)));
}
__device__ __forceinline__ void ld_if(double &v, const double *p, bool pred)
{
	asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.global.nc.f64 %0, [%1];\n\t}"
			: "+d"(v) : "l"(p), "r"(uint32_t(pred)));
}
template <class A>
__device__ __forceinline__ void ld_if(A &, const A *, bool) {}       // integers take no scales

// U weights of consecutive entries
template <class WT, class A, int U>
__device__ __forceinline__ void ld_wn(const void *val, uint32_t e0, A (&w)[U])
{
	constexpr int per = int(16 / sizeof(WT));
	const uint4 *p = reinterpret_cast<const uint4 *>(static_cast<const WT *>(val) + e0);
#pragma unroll
	for (int q = 0; q < U / per; q++) {
		const uint4 a = __ldg(p + q);
		WT t[per];
		memcpy(t, &a, 16);
#pragma unroll
		for (int i = 0; i < per; i++) w[q * per + i] = A(t[i]);
	}
}

// A chunk's sum in the row kernel at k = 1 without row scales: binary trees over
// blocks of 16 places, block b added to running sum b % 4, and a tree over
// those.  Its error is that of the warp-per-range kernel's 32 strided sums and a
// tree over them (8000 chunks of 129 to 256 FP32 numbers, RMS against FP64:
// 7.6e-8 of normal ones against 7.8e-8, 4.0e-8 of uniform ones in both; a single
// running sum of the blocks has 8.9e-8 and 5.9e-8; a whole binary tree 7.6e-8
// and 4.3e-8, for more registers).  The order does not depend on the step.
static_assert(kChunk == 256, "chunk_sum and warp_chunk add 256 places");
template <class A, int U>
struct chunk_sum {
	static_assert(U == 8 || U == 16, "half blocks or blocks");
	A s0, s1, s2, s3, half;
	bool odd;                                        // `half` waits for its right neighbour

	__device__ __forceinline__ void zero()
	{
		s0 = s1 = s2 = s3 = half = A(0);
		odd = false;
	}
	__device__ __forceinline__ void turn(A t)
	{
		s0 = s1; s1 = s2; s2 = s3; s3 = t;
	}
	// the sum of the next U entries
	__device__ __forceinline__ void add(A t)
	{
		if (U == 16) {
			turn(acc_add(s0, t));
			return;
		}
		if (odd) turn(acc_add(s0, acc_add(half, t)));
		else half = t;
		odd = !odd;
	}
	// the sum of a chunk of `len` (padded) entries
	__device__ __forceinline__ A sum(uint32_t len)
	{
		if (U == 8 && odd) turn(acc_add(s0, half));
		for (uint32_t b = (len + 15) / 16; b & 3u; b++) turn(s0);      // running sum 0 first
		return acc_add(acc_add(s0, s1), acc_add(s2, s3));
	}
};

// The same sum by a warp whose lane l holds the terms 32 j + l in t[j], j < 8
// (zeros beyond the chunk): the warp-per-range kernel's, in a streamed part whose
// resident form takes the row kernel, so that the products are equal.
template <class A>
__device__ __forceinline__ A warp_chunk(const A *t, int lane)
{
	A v[8];
#pragma unroll
	for (int j = 0; j < 8; j++) v[j] = t[j];
	// bits 0 to 2 of the place; each exchange halves the lane's values of j
#pragma unroll
	for (int b = 0; b < 3; b++) {
		const bool hi = (lane >> b) & 1;
#pragma unroll
		for (int q = 0; q < (4 >> b); q++) {
			const A give = hi ? v[2 * q] : v[2 * q + 1], keep = hi ? v[2 * q + 1] : v[2 * q];
			v[q] = acc_add(keep, __shfl_xor_sync(0xffffffffu, give, 1 << b));
		}
	}
	// bit 3: lane l has block 2 (l % 8) + l / 16
	const A blk = acc_add(v[0], __shfl_xor_sync(0xffffffffu, v[0], 8));
	A r = __shfl_sync(0xffffffffu, blk, lane & 25);
#pragma unroll
	for (int q = 1; q < 4; q++) r = acc_add(r, __shfl_sync(0xffffffffu, blk, (lane & 25) | (2 * q)));
	r = acc_add(r, __shfl_xor_sync(0xffffffffu, r, 16));
	return acc_add(r, __shfl_xor_sync(0xffffffffu, r, 1));
}

// One range, U entries per step: the gathers (and scales, weights and the
// next step's column ids) of a step are all issued before its adds.  Entries
// of chunks carry no end flag, so only row runs store.
// K1: k = 1 without row scales (chunks by chunk_sum, in the loop that row runs
// take: a warp's lanes differ, and a loop of its own took R-MAT scale 18 from
// 23 to 27 us); else a chunk is one running sum, of whole steps in one-element
// lanes.  APART: a lane's columns are colbase + i * G instead of neighbours.
// BRANCH: a lane's 32 result bytes go out as one sector or as two halves, by
// Y's alignment, which makes the row close a branch (branch_close).
template <class XT, class YT, class A, class WT, int VN, int U, bool SI, bool SO, bool K1, bool APART, bool BRANCH>
__device__ __forceinline__ void run_range(const spmm_args &a, const range_t rg, int colbase)
{
	constexpr bool kBinary = std::is_void<WT>::value;
	static_assert(U % kStep == 0, "whole id loads");
	const int apart = APART ? a.G : 1;
	const int live = APART ? (a.k - colbase + a.G - 1) / a.G : VN;     // columns below k
	const char *Xb = static_cast<const char *>(a.X) + size_t(colbase) * sizeof(XT);
	const char *Hb = static_cast<const char *>(a.xhot) + size_t(colbase) * sizeof(XT);
	// 32-bit row strides (one wide multiply-add per address); one-element
	// lanes also take the strides beyond 4 GB
	typedef typename std::conditional<VN == 1, uint64_t, uint32_t>::type stride_t;
	const stride_t xs = stride_t(a.ldx) * stride_t(sizeof(XT)), hs = stride_t(a.hot_ld) * stride_t(sizeof(XT));
	YT *yp = static_cast<YT *>(a.Y) + int64_t(rg.row0) * a.ldy + colbase;
	const A *sop = SO ? static_cast<const A *>(a.s_out) + rg.row0 : nullptr;
	accum<A, VN, 1> acc;
	acc.zero();
	chunk_sum<A, U == 8 ? 8 : 16> chunk;
	if constexpr (K1) chunk.zero();
	uint32_t e = rg.e0;
	const uint32_t e_end = e + rg.len;
	auto ids = [&](uint32_t at, uint32_t (&r)[U]) {
#pragma unroll
		for (int q = 0; q < U / kStep; q++) {
			// past the end: entries of the zero row
			uint32_t t[8] = {kHot, kHot, kHot, kHot, kHot, kHot, kHot, kHot};
			if (at + kStep * q < e_end) ld32_nc(a.col + at + kStep * q, t);
#pragma unroll
			for (int i = 0; i < kStep; i++) r[kStep * q + i] = t[i];
		}
	};
	uint32_t raw[U];
	ids(e, raw);
	while (true) {
		xvec<XT, VN> x[U];
		A sc[SI ? U : 1], w[kBinary ? 1 : U], so[SO ? U : 1];
#pragma unroll
		for (int u = 0; u < U; u++) {
			const uint32_t c = raw[u] & kIdxMask;
			const bool hot = raw[u] & kHot;
			const char *xp = (hot ? Hb : Xb) + uint64_t(c) * (hot ? hs : xs);
			if constexpr (APART) x[u] = ld_apart<XT, VN>(xp, uint32_t(apart) * uint32_t(sizeof(XT)), live);
			else x[u] = ld_n<XT, VN>(xp);
		}
		// the scales that this step needs, loaded with its rows: s_in of cold
		// entries (the pack's rows carry theirs) and s_out of the rows that
		// close in it
		uint32_t all = raw[0], any = raw[0];
#pragma unroll
		for (int u = 1; u < U; u++) {
			all &= raw[u];
			any |= raw[u];
		}
		// steps without a cold entry skip the scales (4-byte types: the second
		// copy of the sums spills in the others, BF16 695 against 393 us at
		// scale 21).  The lanes that are together here decide together: with each
		// group its own way a warp mostly ran both (input scales, FP32 k = 32, R-MAT
		// scale 18 / 21 / 23 75 / 440 / 2090 against 70 / 394 / 1700 us); an entry of
		// the pack takes a scale of 1.  Nothing branches between the mask and the
		// vote, so every lane of the mask arrives.  One-element lanes, whose second
		// copy costs one add an entry, decide by group (k = 17 at scale 21 2160
		// against 2219 us with the vote).
		bool cold = SI && (sizeof(XT) != 4 || !(all & kHot));
		if constexpr (SI && sizeof(XT) == 4 && VN > 1) cold = __any_sync(__activemask(), cold);
		if constexpr (SI)
			if (cold) {
#pragma unroll
				for (int u = 0; u < U; u++) {
					sc[u] = A(1);
					ld_if(sc[u], static_cast<const A *>(a.s_in) + (raw[u] & kIdxMask), !(raw[u] & kHot));
				}
			}
		if constexpr (SO)
			if (int32_t(any) < 0) {
#pragma unroll
				for (int u = 0; u < U; u++) {
					ld_if(so[u], sop, raw[u] >> 31);
					sop += raw[u] >> 31;
				}
			}
		if constexpr (!kBinary) {
#pragma unroll
			for (int q = 0; q < U / kStep; q++) {
				A t[kStep] = {};
				if (e + kStep * q < e_end) ld_wn<WT, A, kStep>(a.val, e + kStep * q, t);
#pragma unroll
				for (int i = 0; i < kStep; i++) w[kStep * q + i] = t[i];
			}
		}
		e += U;
		uint32_t nraw[U];
		ids(e, nraw);
		auto sums = [&](auto scaled) {
			constexpr bool kSc = decltype(scaled)::value;
#pragma unroll
			for (int u = 0; u < U; u++) {
				// (x * s_in) * w, rounded per step like scale_rows then SpMM
				if constexpr (kSc && !kBinary) acc.template add<XT, 2>(0, x[u], sc[u], w[u]);
				else if constexpr (kSc) acc.template add<XT, 1>(0, x[u], sc[u], A(1));
				else if constexpr (!kBinary) acc.template add<XT, 1>(0, x[u], w[u], A(1));
				else acc.template add<XT, 0>(0, x[u], A(1), A(1));
				if (int32_t(raw[u]) < 0) {
					YT out[VN];
#pragma unroll
					for (int i = 0; i < VN; i++) {
						A v = acc.get(0, i);
						if constexpr (SO) v = acc_mul(v, so[u]);
						out[i] = from_acc<YT, A>(v);
					}
					if constexpr (APART) {
#pragma unroll
						for (int i = 0; i < VN; i++)
							if (i < live) yp[i * apart] = out[i];
					} else if constexpr (BRANCH) {
						if ((reinterpret_cast<uintptr_t>(yp) & 31) == 0) st_sector<YT, VN>(yp, out);
						else st_y<YT, VN>(yp, out);
					} else {
						st_y<YT, VN>(yp, out);
					}
					yp += a.ldy;
					acc.zero();
				}
			}
		};
		bool done = false;
		if constexpr (VN == 1 || APART) {
			if (rg.slot != kNoSlot) {
				// the step's terms of a column by a tree
				A r[VN];
#pragma unroll
				for (int i = 0; i < VN; i++) {
					A t[U];
#pragma unroll
					for (int u = 0; u < U; u++) {
						t[u] = to_acc<A>(x[u].v[i]);
						if constexpr (SI) { if (cold) t[u] = acc_mul(t[u], sc[u]); }
						if constexpr (!kBinary) t[u] = acc_mul(t[u], w[u]);
					}
#pragma unroll
					for (int d = 1; d < U; d *= 2)
#pragma unroll
						for (int u = 0; u + d < U; u += 2 * d) t[u] = acc_add(t[u], t[u + d]);
					r[i] = t[0];
				}
				if constexpr (K1) chunk.add(r[0]);
				else acc.add_terms(r);
				done = true;
			}
		}
		if (done) {
		} else if constexpr (SI && sizeof(XT) != 4) {
			sums(std::true_type{});
		} else if constexpr (SI) {
			if (cold) sums(std::true_type{});
			else sums(std::false_type{});
		} else {
			sums(std::false_type{});
		}
		if (e >= e_end) break;
#pragma unroll
		for (int u = 0; u < U; u++) raw[u] = nraw[u];
	}
	if (rg.slot != kNoSlot) {
		A *p = static_cast<A *>(a.partial) + int64_t(rg.slot) * kPartialStride + colbase;
		if constexpr (K1) {
			p[0] = chunk.sum(rg.len);
		} else {
#pragma unroll
			for (int i = 0; i < VN; i++)
				if (!APART || i < live) p[i * apart] = acc.get(0, i);
		}
	}
}

// Threads and resident blocks per SM: at most 24 warps (FP32 rows in 16-byte
// lanes: 24 warps 411 us, 20 warps 429 us at scale 22), fewer where the loads
// in flight and the sums need the registers (spills cost more than the warps:
// BF16 with 24 warps 801 us against 446 us with 20).
constexpr int kLaneThreads = 128;
constexpr int lane_blocks(int bytes, bool scaled, int esize, int step, bool k1)
{
	if (k1 && esize == 8 && step == 16) return 5;        // FP64 chunk_sum (6: 204 bytes spilled, scale 22 279 -> 319 us)
	if (step == 32) return 2;                            // small matrices: the longest chain decides
	if (step == 16 && bytes == 16) return 3;
	if (bytes == 32) return scaled ? 4 : 3;              // 8 x 32 bytes a lane; unscaled 3 or 4 within 2 %
	if (scaled && esize == 8) return 4;
	return scaled || esize == 2 ? 5 : 6;                 // BF16's sums are FP32, twice its rows
}
// Entries per step (launch_lanes takes more for small matrices): 16 in lanes of
// at most 8 bytes of an unweighted, unscaled product (small or odd panels: R-MAT
// scale 18, k = 5, 39 against 43 us with 8), else 8.
constexpr int lane_step(int bytes, int esize, bool plain) { return bytes <= 8 && esize >= 4 && plain ? 16 : 8; }

// FORM: kAny, kOne (k = 1 without row scales) or kLoop (the same in a PageRank
// loop: it returns at once when the loop has ended) or kApart (VN columns per
// lane, G apart, in rows that are no whole units: lanes_apart) or kBranch
// (branch_close).
enum { kAny, kOne, kLoop, kApart, kBranch };
template <class XT, class YT, class A, class WT, int VN, int U, bool SI, bool SO, int FORM>
__global__ void __launch_bounds__(kLaneThreads, lane_blocks(VN * int(sizeof(XT)), SI || SO, int(sizeof(XT)), U, FORM == kOne || FORM == kLoop))
spmm_lane_kernel(const spmm_args a)
{
	dep_wait();
	dep_launch();
	if constexpr (FORM == kLoop) {
		if (a.state[1]) return;
	}
	constexpr bool K1 = FORM == kOne || FORM == kLoop, kSplit = FORM == kApart, kBr = FORM == kBranch;
	const int lane = threadIdx.x & 31;
	const int G = a.G, R = a.R;
	const int grp = lane / G;
	if (grp >= R) return;
	const int colbase = (lane - grp * G) * (kSplit ? 1 : VN);
	constexpr uint32_t wpb = kLaneThreads / 32;
	const uint32_t wib = threadIdx.x >> 5;
	const uint32_t ng = gridDim.x * wpb * uint32_t(R);
	// full rounds give a block neighbouring ranges; the last, partial one is
	// dealt out over the blocks (a round of neighbours left some SMs idle
	// through the tail: 528 -> 488 us for the BF16 operator at scale 21)
	const uint32_t g0 = (blockIdx.x * wpb + wib) * uint32_t(R) + uint32_t(grp);
	const uint32_t g1 = (wib * gridDim.x + blockIdx.x) * uint32_t(R) + uint32_t(grp);
	uint32_t base = 0;
	for (; base + ng <= a.n_ranges; base += ng)
		run_range<XT, YT, A, WT, VN, U, SI, SO, K1, kSplit, kBr>(a, a.ranges[base + g0], colbase);
	if (base + g1 < a.n_ranges)
		run_range<XT, YT, A, WT, VN, U, SI, SO, K1, kSplit, kBr>(a, a.ranges[base + g1], colbase);
}

// k = 1 (SpMV): a warp per range.  The 32 lanes load the range's column ids
// (coalesced) and gather its X values into shared memory, one entry each;
// then each lane sums whole rows of the range from shared memory in entry
// order, with one running sum per row and every add rounded, which is the
// lane-group kernel's arithmetic: rows of up to 256 entries come out
// identical.  A chunk of a longer row is added up by the whole warp into its
// partial slot: each lane its own entries, then a fixed xor tree, or, with
// BLOCKS, in the row kernel's order (warp_chunk).
// (spmv_by_warps says which matrices come here.)
constexpr int kSpmvMax = 512;            // most entries of one range
static_assert(((kRange - 1 + kExactMax + kStep - 1) / kStep) * kStep <= uint32_t(kSpmvMax) &&
		kChunk <= uint32_t(kSpmvMax), "a range fits the SpMV kernel's staging");
// ... and so does a run of kRangeMin with its fine runs padded one by one
static_assert(kRangeMin - 1 + kExactMax + ((kRangeMin - 1 + kExactMax) / kRangeFine + 2) * (kStep - 1) <= uint32_t(kSpmvMax),
		"a run of fine runs fits the SpMV kernel's staging");

// A chunk of a PageRank row: the warp whose chunk arrives last adds the row's
// partials, in spmm_fixup_kernel's order at k = 1 (the same parts, the same
// tree), and updates the row, which saves the iteration a kernel.  Partials
// are read past the L1.
__device__ __forceinline__ void pr_chunk(const pr_epi &e, float *partial, uint32_t slot, float acc, int lane, unsigned &cnt)
{
	uint32_t h = 0, old = 0;
	if (lane == 0) {
		__stcg(partial + int64_t(slot) * kPartialStride, acc);
		__threadfence();
		h = e.chunk_heavy[slot];
		old = atomicAdd(e.arrived + h, 1u);
	}
	h = __shfl_sync(0xffffffffu, h, 0);
	old = __shfl_sync(0xffffffffu, old, 0);
	const heavy_row hr = static_cast<const heavy_row *>(e.heavy)[h];
	if (old != hr.count - 1) return;
	__threadfence();
	const float *pc = partial + int64_t(hr.first) * kPartialStride;
	auto sums = [&](uint32_t part, uint32_t P) {
		float s0 = 0.f, s1 = 0.f;
		uint32_t c = part;
		for (; c + P < hr.count; c += 2u * P) {
			s0 = acc_add(s0, __ldcg(pc + int64_t(c) * kPartialStride));
			s1 = acc_add(s1, __ldcg(pc + int64_t(c + P) * kPartialStride));
		}
		if (c < hr.count) s0 = acc_add(s0, __ldcg(pc + int64_t(c) * kPartialStride));
		return acc_add(s0, s1);
	};
	auto tree = [&](float v, int lanes) {
		for (int o = 1; o < lanes; o <<= 1) v = acc_add(v, __shfl_xor_sync(0xffffffffu, v, o));
		return v;
	};
	float v;
	if (hr.count > kBlockChunks) {
		v = tree(sums(uint32_t(lane), 256), 32);
		for (uint32_t w = 1; w < 8; w++) v = acc_add(v, tree(sums(w * 32 + uint32_t(lane), 256), 32));
	} else if (hr.count > kLongChunks) {
		v = tree(sums(uint32_t(lane), 32), 32);
	} else {
		v = tree(sums(uint32_t(lane & 1), 2), 2);
	}
	if (lane == 0) {
		e.arrived[h] = 0;
		pr_update(e, hr.row, pr_load(e, hr.row), v, cnt);
	}
}

template <class T, class WT, bool EPI, bool BLOCKS>
__global__ void __launch_bounds__(kThreads) spmv_kernel(const spmm_args a, const pr_epi e)
{
	constexpr int kWarps = kThreads / 32;
	constexpr int J = kSpmvMax / 32;
	constexpr bool kBinary = std::is_void<WT>::value;
	__shared__ T sval[kWarps][kSpmvMax];
	__shared__ uint16_t send[kWarps][kSpmvMax];
	const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
	const uint32_t gw = (blockIdx.x * kThreads + threadIdx.x) >> 5;
	const uint32_t nw = (gridDim.x * kThreads) >> 5;
	const T *X = static_cast<const T *>(a.X);
	const T *H = static_cast<const T *>(a.xhot);
	unsigned cnt = 0;
	// the matrix does not change: the first range's ids load while the kernel
	// before this one still runs
	bool waited = false, done = false;
	auto wait = [&]() {
		if (waited) return;
		dep_wait();
		dep_launch();
		waited = true;
		if constexpr (EPI) done = e.state[1] != 0;    // converged in an earlier iteration
	};
	for (uint32_t r = gw; r < a.n_ranges; r += nw) {
		const range_t rg = a.ranges[r];
		const bool runs = rg.slot == kNoSlot;
		uint32_t raw[J];
#pragma unroll
		for (int j = 0; j < J; j++) {
			const uint32_t i = uint32_t(j * 32 + lane);
			raw[j] = i < rg.len ? __ldcs(a.col + rg.e0 + i) : 0u;
		}
		wait();
		if constexpr (EPI) {
			if (done) break;
		}
		T t[J];
#pragma unroll
		for (int j = 0; j < J; j++) {
			const uint32_t i = uint32_t(j * 32 + lane);
			t[j] = T(0);
			if (i < rg.len) {
				const uint32_t c = raw[j] & kIdxMask;
				const bool hot = raw[j] & kHot;
				// a plain load (the wait's memory clobber keeps it behind): as volatile
				// asm the 16 guarded FP64 gathers came one after the other, 7.2 us
				// for a launch of 500 ranges instead of 4.5
				t[j] = (hot ? H : X)[int64_t(c) * (hot ? int64_t(1) : a.ldx)];
			}
		}
		if constexpr (!kBinary) {
#pragma unroll
			for (int j = 0; j < J; j++) {
				const uint32_t i = uint32_t(j * 32 + lane);
				if (i < rg.len) t[j] = acc_mul(t[j], T(__ldcs(static_cast<const WT *>(a.val) + rg.e0 + i)));
			}
		}
		// stage the products and the row ends (entry index of each row's last entry)
		int nrow = 0;
#pragma unroll
		for (int j = 0; j < J; j++) {
			const uint32_t i = uint32_t(j * 32 + lane);
			const bool is_end = runs && i < rg.len && (raw[j] >> 31);
			const uint32_t b = __ballot_sync(0xffffffffu, is_end);
			if (is_end) send[wib][nrow + __popc(b & ((1u << lane) - 1u))] = uint16_t(i);
			nrow += __popc(b);
			sval[wib][i] = t[j];
		}
		__syncwarp();
		if (runs) {
			for (int q = lane; q < nrow; q += 32) {
				const int b0 = q ? int(send[wib][q - 1]) + 1 : 0, b1 = send[wib][q] + 1;
				const uint32_t row = rg.row0 + uint32_t(q);
				// the row's old values load while it is summed
				pr_row old{};
				uint32_t heavy = 0;
				if constexpr (EPI) {
					old = pr_load(e, int64_t(row));
					heavy = (__ldg(e.heavy_mask + (row >> 5)) >> (row & 31)) & 1u;
				}
				T acc = T(0);
				int i = b0;
				for (; i + 8 <= b1; i += 8) {         // 8 shared-memory reads in flight
					T v[8];
#pragma unroll
					for (int z = 0; z < 8; z++) v[z] = sval[wib][i + z];
#pragma unroll
					for (int z = 0; z < 8; z++) acc = acc_add(acc, v[z]);
				}
				for (; i < b1; i++) acc = acc_add(acc, sval[wib][i]);
				if constexpr (EPI) {
					if (!heavy) pr_update(e, int64_t(row), old, acc, cnt);
				} else {
					static_cast<T *>(a.Y)[int64_t(row) * a.ldy] = acc;
				}
			}
		} else {
			// a chunk: each lane adds its entries (j order), then a fixed xor tree
			T acc = T(0);
			if constexpr (BLOCKS) {
				acc = warp_chunk(t, lane);
			} else {
#pragma unroll
				for (int j = 0; j < J; j++) acc = acc_add(acc, t[j]);
#pragma unroll
				for (int o = 16; o > 0; o >>= 1) acc = acc_add(acc, __shfl_xor_sync(0xffffffffu, acc, o));
			}
			if constexpr (EPI) pr_chunk(e, static_cast<float *>(a.partial), rg.slot, acc, lane, cnt);
			else if (lane == 0) static_cast<T *>(a.partial)[int64_t(rg.slot) * kPartialStride] = acc;
		}
		__syncwarp();
	}
	wait();
	if constexpr (EPI) {
		if (done) return;
		cnt = __reduce_add_sync(0xffffffffu, cnt);
		if (lane == 0 && cnt) atomicAdd(e.state, (unsigned long long)cnt);
		if (e.finish) pr_finish(e);
	}
}

// The update of one PageRank iteration over `out` = A^T in.
__global__ void __launch_bounds__(kThreads) pr_apply_kernel(const float *out, int64_t n, const pr_epi e)
{
	dep_wait();
	dep_launch();
	if (e.state[1]) return;
	unsigned cnt = 0;
	for (int64_t i = int64_t(blockIdx.x) * kThreads + threadIdx.x; i < n; i += int64_t(gridDim.x) * kThreads)
		pr_update(e, i, pr_load(e, i), out[i], cnt);
	cnt = __reduce_add_sync(0xffffffffu, cnt);
	if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(e.state, (unsigned long long)cnt);
	pr_finish(e);
}

// Pack the hot columns' X rows of this panel behind a zero row:
// xhot[0][j] = 0 and xhot[s+1][j] = X[hot_col[s]][c0 + j] (times
// s_in[hot_col[s]], rounded, when SCALE_IN), j < kp.  The zero row is
// rewritten every call because a narrower earlier panel packs over it.
template <class XT, class A, bool SCALE_IN>
__global__ void pack_hot_kernel(const int32_t *hot_col, uint32_t n_hot, const XT *X, int64_t ldx, int kp,
		XT *xhot, int hot_ld, const A *s_in)
{
	dep_launch();
	const uint64_t total = uint64_t(n_hot + 1) * kp;
	for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < total; t += uint64_t(gridDim.x) * blockDim.x) {
		const uint32_t s = uint32_t(t / kp);
		const int j = int(t - uint64_t(s) * kp);
		XT v = XT(0);
		if (s > 0) {
			const int32_t c = __ldg(hot_col + s - 1);
			v = X[int64_t(c) * ldx + j];
			if constexpr (SCALE_IN) v = from_acc<XT, A>(acc_mul(to_acc<A>(v), s_in[c]));
		}
		xhot[int64_t(s) * hot_ld + j] = v;
	}
}

// The same in 16-byte units (rows of whole units, 16-byte aligned), with 4
// units in flight per thread: the copy is a gather of random rows of X, and
// one 4-byte element per thread left it at a third of the bandwidth its
// bytes allow.
template <class XT, class A, bool SCALE_IN>
__global__ void pack_hot_vec_kernel(const int32_t *hot_col, uint32_t n_hot, const XT *X, int64_t ldx, int units,
		XT *xhot, int hot_ld, const A *s_in)
{
	dep_launch();
	constexpr int E = int(16 / sizeof(XT));
	constexpr int D = 4;
	const uint64_t total = uint64_t(n_hot + 1) * units;
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t t0 = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t0 < total; t0 += D * stride) {
		uint4 v[D];
		int32_t c[D];
#pragma unroll
		for (int q = 0; q < D; q++) {
			const uint64_t t = t0 + q * stride;
			v[q] = make_uint4(0, 0, 0, 0);
			c[q] = -1;
			if (t < total) {
				const uint32_t sl = uint32_t(t / units);
				const int u = int(t - uint64_t(sl) * units);
				if (sl > 0) {
					c[q] = __ldg(hot_col + sl - 1);
					v[q] = __ldg(reinterpret_cast<const uint4 *>(X + int64_t(c[q]) * ldx) + u);
				}
			}
		}
#pragma unroll
		for (int q = 0; q < D; q++) {
			const uint64_t t = t0 + q * stride;
			if (t >= total) continue;
			const uint32_t sl = uint32_t(t / units);
			const int u = int(t - uint64_t(sl) * units);
			if constexpr (SCALE_IN) {
				if (c[q] >= 0) {
					XT e[E];
					memcpy(e, &v[q], 16);
					const A sc = s_in[c[q]];
#pragma unroll
					for (int i = 0; i < E; i++) e[i] = from_acc<XT, A>(acc_mul(to_acc<A>(e[i]), sc));
					memcpy(&v[q], e, 16);
				}
			}
			*reinterpret_cast<uint4 *>(xhot + int64_t(sl) * hot_ld + int64_t(u) * E) = v[q];
		}
	}
}

// The hot pack of one panel: 16-byte units when the rows allow it.
template <class XT, class A>
static int launch_pack(const gpu_part &p, const XT *X, int64_t ldx, int kp, XT *xhot, int hot_ld, const A *s_in,
		cudaStream_t st)
{
	const bool vec = (kp * sizeof(XT)) % 16 == 0 && (ldx * sizeof(XT)) % 16 == 0 && (hot_ld * sizeof(XT)) % 16 == 0 &&
			(reinterpret_cast<uintptr_t>(X) & 15) == 0 && (reinterpret_cast<uintptr_t>(xhot) & 15) == 0;
	if (vec) {
		const int units = int(kp * sizeof(XT) / 16);
		const uint64_t total = uint64_t(p.n_hot + 1) * units;
		const unsigned pb = unsigned(std::max<uint64_t>(1, std::min<uint64_t>((total + 1023) / 1024, 148ull * 8)));
		if (s_in) pack_hot_vec_kernel<XT, A, true><<<pb, 256, 0, st>>>(p.hot_col, p.n_hot, X, ldx, units, xhot, hot_ld, s_in);
		else pack_hot_vec_kernel<XT, A, false><<<pb, 256, 0, st>>>(p.hot_col, p.n_hot, X, ldx, units, xhot, hot_ld, nullptr);
	} else {
		const uint64_t total = uint64_t(p.n_hot + 1) * kp;
		const unsigned pb = unsigned(std::min<uint64_t>((total + 255) / 256, 148ull * 16));
		if (s_in) pack_hot_kernel<XT, A, true><<<pb, 256, 0, st>>>(p.hot_col, p.n_hot, X, ldx, kp, xhot, hot_ld, s_in);
		else pack_hot_kernel<XT, A, false><<<pb, 256, 0, st>>>(p.hot_col, p.n_hot, X, ldx, kp, xhot, hot_ld, nullptr);
	}
	CUDA_TRY(cudaGetLastError());
	return FMX_OK;
}

// Part `part` of P adds chunks part, part + P, ... of one column unit (a
// float4 when vec, else one element) into two running sums (even and odd
// steps).
template <class A>
__device__ __forceinline__ void chunk_sums(const A *pc, uint32_t part, uint32_t P, uint32_t count, bool vec,
		A (&s0)[4], A (&s1)[4])
{
	constexpr bool kVec4 = std::is_same<A, float>::value;
	uint32_t c = part;
	for (; c + P < count; c += 2u * P) {
		if constexpr (kVec4) {
			if (vec) {
				const float4 a = *reinterpret_cast<const float4 *>(pc + int64_t(c) * kPartialStride);
				const float4 b = *reinterpret_cast<const float4 *>(pc + int64_t(c + P) * kPartialStride);
				s0[0] = acc_add(s0[0], a.x); s0[1] = acc_add(s0[1], a.y);
				s0[2] = acc_add(s0[2], a.z); s0[3] = acc_add(s0[3], a.w);
				s1[0] = acc_add(s1[0], b.x); s1[1] = acc_add(s1[1], b.y);
				s1[2] = acc_add(s1[2], b.z); s1[3] = acc_add(s1[3], b.w);
				continue;
			}
		}
		s0[0] = acc_add(s0[0], pc[int64_t(c) * kPartialStride]);
		s1[0] = acc_add(s1[0], pc[int64_t(c + P) * kPartialStride]);
	}
	if (c < count) {
		if constexpr (kVec4) {
			if (vec) {
				const float4 a = *reinterpret_cast<const float4 *>(pc + int64_t(c) * kPartialStride);
				s0[0] = acc_add(s0[0], a.x); s0[1] = acc_add(s0[1], a.y);
				s0[2] = acc_add(s0[2], a.z); s0[3] = acc_add(s0[3], a.w);
				return;
			}
		}
		s0[0] = acc_add(s0[0], pc[int64_t(c) * kPartialStride]);
	}
}

// Heavy rows: add the chunk partials, scale, convert, store.  A row's
// columns are covered by L lanes (L = k / 4 float4 lanes for FP32 panels of
// k % 4 == 0, else one lane per column, rounded up to a power of two, at most
// 32) and its chunks by P parts: part q adds chunks q, q + P, ... into two
// running sums, and the parts are combined by a fixed xor tree.  The heavy
// rows come longest first.  The first n_block of them (more than kBlockChunks
// chunks) get a block of 8 warps each, P = 8 * 32 / L, the warps' sums added in
// warp order: the chain of one part is then at most count / P chunks long,
// where a single warp's bounded the whole fixup by its longest row.  Of the
// others, each of the first n_long (more than kLongChunks chunks) gets a warp
// with P = 32 / L; the rest go 32 / (2 L) rows to a warp with P = 2 (one row
// and P = 1 when L = 32).  Deterministic, with many loads in flight.
template <class YT, class A, bool SCALE_OUT>
__device__ __forceinline__ void fix_store(const heavy_row &h, const A (&v)[4], int nv, YT *Y, int64_t ldy, int col,
		const A *s_out)
{
	A so = A(1);
	if constexpr (SCALE_OUT) so = s_out[h.row];
	YT *y = Y + int64_t(h.row) * ldy + col;
	for (int i = 0; i < nv; i++) {
		A x = v[i];
		if constexpr (SCALE_OUT) x = acc_mul(x, so);
		y[i] = from_acc<YT, A>(x);
	}
}

template <class YT, class A, bool SCALE_OUT, bool STOP>
__global__ void __launch_bounds__(256) spmm_fixup_kernel(const heavy_row *heavy, uint32_t n_heavy, uint32_t n_block,
		uint32_t n_long, const A *partial, YT *Y, int64_t ldy, int k, const A *s_out, int L,
		const unsigned long long *state)
{
	__shared__ A red[8][32][4];
	dep_wait();
	dep_launch();
	if constexpr (STOP) {
		if (state[1]) return;
	}
	constexpr bool kVec4 = std::is_same<A, float>::value;
	const bool vec = kVec4 && (k % 4) == 0;
	const int units = vec ? k / 4 : k, nv = vec ? 4 : 1;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const bool block_row = blockIdx.x < n_block;
	const uint64_t w = uint64_t(blockIdx.x - n_block) * 8 + warp;
	const bool long_row = w < n_long;
	const int per_warp = 32 / L;
	const int P = block_row ? 8 * per_warp : long_row ? per_warp : (L < 32 ? 2 : 1);
	const int lanes = block_row ? 32 : L * P;         // of a warp, per row
	const uint64_t r = block_row ? blockIdx.x
			: n_block + (long_row ? w : uint64_t(n_long) + (w - n_long) * uint64_t(32 / lanes) + uint64_t(lane / lanes));
	const int sub = lane % lanes, cl = sub % L;
	const int part = block_row ? warp * per_warp + lane / L : sub / L;
	const bool live = r < n_heavy;
	heavy_row h{0, 0, 0};
	if (live) h = heavy[r];
	for (int u0 = 0; u0 < units; u0 += L) {           // the same trip count on every thread
		const int u = u0 + cl;
		const bool mine = live && u < units;
		A s0[4] = {A(0), A(0), A(0), A(0)}, s1[4] = {A(0), A(0), A(0), A(0)};
		if (mine) chunk_sums<A>(partial + int64_t(h.first) * kPartialStride + (vec ? 4 * u : u), uint32_t(part),
				uint32_t(P), h.count, vec, s0, s1);
		A t[4];
#pragma unroll
		for (int i = 0; i < 4; i++) t[i] = acc_add(s0[i], s1[i]);
		for (int o = L; o < lanes; o <<= 1)
#pragma unroll
			for (int i = 0; i < 4; i++) t[i] = acc_add(t[i], __shfl_xor_sync(0xffffffffu, t[i], o));
		if (block_row) {
			if (lane < L)
#pragma unroll
				for (int i = 0; i < 4; i++) red[warp][lane][i] = t[i];
			__syncthreads();
			if (warp == 0 && lane < L && mine) {
				A v[4];
#pragma unroll
				for (int i = 0; i < 4; i++) {
					v[i] = red[0][lane][i];
					for (int q = 1; q < 8; q++) v[i] = acc_add(v[i], red[q][lane][i]);
				}
				fix_store<YT, A, SCALE_OUT>(h, v, nv, Y, ldy, vec ? 4 * u : u, s_out);
			}
			__syncthreads();
		} else if (mine && part == 0) {
			fix_store<YT, A, SCALE_OUT>(h, t, nv, Y, ldy, vec ? 4 * u : u, s_out);
		}
	}
}

template <class YT, class A, bool SCALE_OUT, bool STOP = false>
static int launch_fixup(const gpu_part &p, const A *partial, YT *Y, int64_t ldy, int k, const A *s_out, cudaStream_t st,
		const unsigned long long *state = nullptr)
{
	if (!p.n_heavy) return FMX_OK;
	const bool vec = std::is_same<A, float>::value && (k % 4) == 0;
	const int units = vec ? k / 4 : k;
	int L = 1;
	while (L < units && L < 32) L <<= 1;
	const uint32_t nb = p.n_block_heavy;
	const uint64_t n_long = p.n_long_heavy - nb;
	const uint64_t n_short = p.n_heavy - p.n_long_heavy;
	const uint64_t per_warp = uint64_t(32 / (L * (L < 32 ? 2 : 1)));    // short rows per warp
	const uint64_t warps = n_long + (n_short + per_warp - 1) / per_warp;
	const unsigned grid = nb + unsigned((warps + 7) / 8);
	auto kern = spmm_fixup_kernel<YT, A, SCALE_OUT, STOP>;
	if (p.streamed)
		kern<<<grid, 256, 0, st>>>(p.heavy, p.n_heavy, nb, uint32_t(n_long), partial, Y, ldy, k, s_out, L, state);
	else
		CUDA_TRY(launch_dep(kern, grid, 256, st, p.heavy, p.n_heavy, nb, uint32_t(n_long), partial, Y, ldy, k, s_out, L, state));
	CUDA_TRY(cudaGetLastError());
	return FMX_OK;
}

// ---------------------------------------------------------------------------
// Host: building the resident layout
// ---------------------------------------------------------------------------

template <class T>
static int upload(T **dst, const T *src, size_t n, uint64_t &bytes, size_t alloc_n = 0)
{
	*dst = nullptr;
	alloc_n = std::max(alloc_n, n);
	if (!alloc_n) return FMX_OK;
	cudaError_t e = cudaMalloc(reinterpret_cast<void **>(dst), alloc_n * sizeof(T));
	if (e != cudaSuccess)
		return set_error(e == cudaErrorMemoryAllocation ? FMX_ERR_OOM : FMX_ERR_CUDA,
				"cudaMalloc of %zu bytes failed: %s", alloc_n * sizeof(T), cudaGetErrorString(e));
	bytes += alloc_n * sizeof(T);
	if (n) CUDA_TRY(cudaMemcpy(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice));
	if (alloc_n > n) CUDA_TRY(cudaMemset(reinterpret_cast<char *>(*dst) + n * sizeof(T), 0, (alloc_n - n) * sizeof(T)));
	return FMX_OK;
}

template <class F>
static void par_for(uint64_t n, F fn)
{
	int nt = std::max(1, std::min<int>(default_threads(), int((n + 65535) / 65536)));
	std::vector<std::thread> th;
	uint64_t per = (n + nt - 1) / nt;
	for (int t = 0; t < nt; t++)
		th.emplace_back([&, t]() {
			uint64_t b = uint64_t(t) * per, e = std::min(n, b + per);
			if (b < e) fn(b, e);
		});
	for (auto &x : th) x.join();
}

// A streamed part's pinned host copy of the entry stream, its two device
// slots (the largest slice plus kStep entries, zeroed) and its copy stream
// and events.  Called with the part's device current.
static int stream_buffers(gpu_part &p, const std::vector<uint32_t> &col, const std::vector<char> &val, size_t es)
{
	uint64_t cap = 0;
	for (const auto &sl : p.slices) cap = std::max<uint64_t>(cap, sl.e1 - sl.e0);
	cap += kStep;
	auto host = [&](void **h, const void *src, size_t n) -> int {
		cudaError_t e = cudaHostAlloc(h, std::max<size_t>(n, 16), cudaHostAllocDefault);
		if (e != cudaSuccess) return set_error(FMX_ERR_OOM, "pinned host stream of %zu bytes: %s", n, cudaGetErrorString(e));
		if (n) memcpy(*h, src, n);
		p.host_bytes += n;
		return FMX_OK;
	};
	if (int rc = host(reinterpret_cast<void **>(&p.h_col), col.data(), col.size() * sizeof(uint32_t))) return rc;
	if (es)
		if (int rc = host(&p.h_val, val.data(), val.size())) return rc;
	for (int b = 0; b < 2; b++) {
		CUDA_TRY(cudaMalloc(&p.slot_col[b], cap * sizeof(uint32_t)));
		CUDA_TRY(cudaMemset(p.slot_col[b], 0, cap * sizeof(uint32_t)));
		p.bytes += cap * sizeof(uint32_t);
		if (es) {
			CUDA_TRY(cudaMalloc(&p.slot_val[b], cap * es));
			CUDA_TRY(cudaMemset(p.slot_val[b], 0, cap * es));
			p.bytes += cap * es;
		}
		CUDA_TRY(cudaEventCreateWithFlags(&p.ev_copied[b], cudaEventDisableTiming));
		CUDA_TRY(cudaEventCreateWithFlags(&p.ev_free[b], cudaEventDisableTiming));
	}
	CUDA_TRY(cudaEventCreateWithFlags(&p.ev_start, cudaEventDisableTiming));
	CUDA_TRY(cudaStreamCreateWithFlags(&p.copy_st, cudaStreamNonBlocking));
	return FMX_OK;
}

constexpr uint64_t kWholeRunSlice = 1 << 18;     // entries of a slice from which it holds whole runs
// slice_entries > 0: a streamed part whose slices hold about that many entries.
static int make_part(const host_csr &csr, int device, std::shared_ptr<gpu_part> &out, uint64_t slice_entries = 0)
{
	if (csr.ncols > (1ull << 30))
		return set_error(FMX_ERR_UNSUPPORTED, "%llu columns: the entry stream holds 30-bit column ids",
				(unsigned long long)csr.ncols);
	auto p = std::make_shared<gpu_part>();
	p->device = device;
	p->nrows = csr.nrows; p->ncols = csr.ncols; p->nnz = csr.nnz;
	p->prim = csr.prim; p->esize = csr.esize;
	const uint64_t n = csr.nrows;
	const size_t es = csr.esize;

	// hot columns: the highest in-degrees (at least 2), up to kHotMax
	std::vector<std::atomic<uint32_t>> indeg(csr.ncols);
	par_for(csr.ncols, [&](uint64_t b, uint64_t e) { for (uint64_t i = b; i < e; i++) indeg[i].store(0, std::memory_order_relaxed); });
	par_for(csr.nnz, [&](uint64_t b, uint64_t e) {
		for (uint64_t i = b; i < e; i++) indeg[csr.col[i]].fetch_add(1, std::memory_order_relaxed);
	});
	std::vector<int32_t> hot_col;
	std::vector<uint32_t> slot_of(csr.ncols, 0);
	{
		// counting sort of the columns by in-degree, descending, capped
		const uint32_t cap = 1u << 16;
		std::vector<uint64_t> cnt(cap + 2, 0);
		for (uint64_t c = 0; c < csr.ncols; c++) {
			uint32_t d = std::min(indeg[c].load(std::memory_order_relaxed), cap);
			if (d >= 2) cnt[cap - d + 1]++;
		}
		for (size_t i = 1; i < cnt.size(); i++) cnt[i] += cnt[i - 1];
		const uint64_t nhot = std::min<uint64_t>(kHotMax, cnt.back());
		std::vector<int32_t> order(cnt.back());
		for (uint64_t c = 0; c < csr.ncols; c++) {
			uint32_t d = std::min(indeg[c].load(std::memory_order_relaxed), cap);
			if (d >= 2) order[cnt[cap - d]++] = int32_t(c);
		}
		hot_col.assign(order.begin(), order.begin() + nhot);
		// slot 0 is the zero row; hot columns take slots 1..nhot
		for (uint64_t s = 0; s < nhot; s++) slot_of[hot_col[s]] = uint32_t(s + 1);
	}

	// Work segments: runs of consecutive rows (every row in order; an exact
	// row with its entries, an empty or longer row as one zero-row entry),
	// then the equal chunks of the longer rows (the rule of seg_row_len in
	// part.h, which make_part_device follows too).  Each segment starts at a
	// multiple of kStep in the stream and is padded to one.
	const uint32_t zero_entry = 0u | kHot;          // slot 0: the zero row
	struct seg_t { uint64_t row0, row1; uint32_t b, e; uint32_t slot; uint64_t at; uint32_t len; uint64_t run; };
	std::vector<seg_t> segs;
	std::vector<heavy_row> heavy;
	uint32_t n_exact = 0;
	bool has_fine = false;
	{
		uint64_t total = 0;
		for (uint64_t r = 0; r < n; r++) total += seg_row_len(csr.row_ptr[r + 1] - csr.row_ptr[r]);
		// Slices of a streamed part that are copied for longer than their kernels
		// run take whole runs: fine ones are padded to kStep each, 4 % more to copy
		// (R-MAT scale 18, slices of 512k entries, k = 1 / 16 372 / 419 against 357 /
		// 400 us; slices of 64k 711 / 1291 against 708 / 1425).
		const uint32_t coarse = range_entries(total), run = slice_entries >= kWholeRunSlice ? coarse : fine_entries(total);
		has_fine = run != coarse;
		uint64_t L = 0, bucket = ~0ull;           // lens of the rows before r
		for (uint64_t r = 0; r < n; r++) {
			const uint32_t d = csr.row_ptr[r + 1] - csr.row_ptr[r];
			const uint32_t len = seg_row_len(d);
			n_exact += (d >= 1 && d <= kExactMax);
			if (L / run != bucket) {
				segs.push_back({r, r + 1, 0, 0, kNoSlot, 0, 0, L / coarse});
				bucket = L / run;
			} else {
				segs.back().row1 = r + 1;
			}
			L += len;
			segs.back().len += len;
		}
	}
	uint32_t slots = 0;
	for (uint64_t r = 0; r < n; r++) {
		const uint32_t d = csr.row_ptr[r + 1] - csr.row_ptr[r];
		if (d <= kExactMax) continue;
		const uint32_t cnt = (d + kChunk - 1) / kChunk;   // equal chunks of <= kChunk entries
		heavy.push_back({int32_t(r), slots, cnt});
		for (uint32_t c = 0; c < cnt; c++) {
			const uint32_t b = uint32_t(uint64_t(d) * c / cnt), e = uint32_t(uint64_t(d) * (c + 1) / cnt);
			segs.push_back({r, r + 1, b, e, slots + c, 0, e - b, 0});
		}
		slots += cnt;
	}
	uint64_t total = 0;
	for (auto &g : segs) {
		g.at = total;
		g.len = (g.len + kStep - 1) / kStep * kStep;
		total += g.len;
	}
	if (total >= (1ull << 32) - 64)
		return set_error(FMX_ERR_UNSUPPORTED, "%llu stream entries: offsets are 32-bit", (unsigned long long)total);
	// the segments as ranges, and the list of whole runs (equal to them without
	// a fine list); starts[i]: the first segment of the i-th whole run
	std::vector<range_t> fine(segs.size()), ranges;
	std::vector<size_t> starts;
	for (size_t i = 0; i < segs.size(); i++) {
		const seg_t &g = segs[i];
		fine[i] = {uint32_t(g.at), g.len, uint32_t(g.row0), g.slot};
		if (i && has_fine && g.slot == kNoSlot && segs[i - 1].run == g.run) {
			ranges.back().len += g.len;
		} else {
			ranges.push_back(fine[i]);
			starts.push_back(i);
		}
	}
	starts.push_back(segs.size());
	// largest ranges first, so that round-robin assignment balances the groups
	// (within each slice of a streamed part: a slice is whole runs in stream
	// order, at least slice_entries entries but the last)
	auto by_len = [](const range_t &x, const range_t &y) { return x.len > y.len; };
	if (slice_entries) {
		p->streamed = true;
		uint64_t e0 = 0;
		size_t i0 = 0;
		for (size_t i = 0; i < ranges.size(); i++) {
			const uint64_t e1 = uint64_t(ranges[i].e0) + ranges[i].len;
			if (e1 - e0 >= slice_entries || i + 1 == ranges.size()) {
				const size_t f0 = starts[i0], f1 = starts[i + 1];
				p->slices.push_back({e0, e1, uint32_t(i0), uint32_t(i + 1 - i0), uint32_t(f0), uint32_t(f1 - f0)});
				std::stable_sort(fine.begin() + f0, fine.begin() + f1, by_len);
				e0 = e1;
				i0 = i + 1;
			}
		}
		for (const auto &sl : p->slices)
			std::stable_sort(ranges.begin() + sl.r0, ranges.begin() + sl.r0 + sl.nr, by_len);
	} else {
		std::stable_sort(fine.begin(), fine.end(), by_len);
		std::stable_sort(ranges.begin(), ranges.end(), by_len);
	}
	if (!has_fine) fine.clear();

	// the entry stream (plus kStep entries so that index prefetches stay in bounds)
	const size_t padded = total + kStep;
	std::vector<uint32_t> col(total, zero_entry);
	std::vector<char> val(total * es, 0);
	std::atomic<uint64_t> hot_entries{0};
	auto put = [&](uint64_t r, uint32_t b, uint32_t e, uint64_t at) {
		const uint32_t rb = csr.row_ptr[r];
		uint64_t h = 0;
		for (uint32_t i = b; i < e; i++) {
			const uint32_t c = uint32_t(csr.col[rb + i]);
			const uint32_t sl = slot_of[c];
			col[at + (i - b)] = sl ? (sl | kHot) : c;
			h += sl != 0;
		}
		if (es) memcpy(&val[at * es], &csr.val[size_t(rb + b) * es], size_t(e - b) * es);
		return h;
	};
	par_for(segs.size(), [&](uint64_t sb, uint64_t se) {
		uint64_t h = 0;
		for (uint64_t i = sb; i < se; i++) {
			const seg_t &g = segs[i];
			if (g.slot != kNoSlot) { h += put(g.row0, g.b, g.e, g.at); continue; }
			uint64_t at = g.at;
			for (uint64_t r = g.row0; r < g.row1; r++) {
				const uint32_t d = csr.row_ptr[r + 1] - csr.row_ptr[r];
				if (d >= 1 && d <= kExactMax) {
					h += put(r, 0, d, at);
					at += d;
				} else {
					at += 1;                 // the zero-row entry already there
				}
				col[at - 1] |= kEnd;
			}
		}
		hot_entries += h;
	});
	p->hot_entries = hot_entries.load();

	int cur = 0;
	cudaGetDevice(&cur);
	CUDA_TRY(cudaSetDevice(device));
	int rc = FMX_OK;
	uint64_t &bytes = p->bytes;
	if (p->streamed) {
		rc = stream_buffers(*p, col, val, es);
	} else {
		rc = upload(&p->col, col.data(), col.size(), bytes, padded);
		if (!rc && es) {
			char *v = nullptr;
			rc = upload(&v, val.data(), val.size(), bytes, padded * es);
			p->val = v;
		}
	}
	if (!rc) rc = upload(&p->hot_col, hot_col.data(), hot_col.size(), bytes);
	if (!rc) rc = upload(&p->slot, slot_of.data(), slot_of.size(), bytes);
	if (!rc) rc = upload(&p->ranges, ranges.data(), ranges.size(), bytes);
	if (!rc) rc = upload(&p->fine, fine.data(), fine.size(), bytes);
	// longest first (the fixup gives each long row a warp and packs the short
	// ones several to a warp); ties keep row order
	std::stable_sort(heavy.begin(), heavy.end(), [](const heavy_row &x, const heavy_row &y) { return x.count > y.count; });
	p->n_long_heavy = uint32_t(std::count_if(heavy.begin(), heavy.end(),
			[](const heavy_row &h) { return h.count > kLongChunks; }));
	p->n_block_heavy = uint32_t(std::count_if(heavy.begin(), heavy.end(),
			[](const heavy_row &h) { return h.count > kBlockChunks; }));
	if (!rc) rc = upload(&p->heavy, heavy.data(), heavy.size(), bytes);
	p->n_hot = uint32_t(hot_col.size());
	p->n_exact = n_exact;
	p->n_ranges = uint32_t(ranges.size());
	p->n_fine = uint32_t(fine.size());
	p->n_heavy = uint32_t(heavy.size());
	p->n_partials = slots;
	auto scratch = [&](void **ptr, size_t sz, const char *what) {
		if (rc || !sz) return;
		cudaError_t e = cudaMalloc(ptr, sz);
		if (e != cudaSuccess)
			rc = set_error(FMX_ERR_OOM, "cudaMalloc of %zu %s bytes failed: %s", sz, what, cudaGetErrorString(e));
		else bytes += sz;
	};
	scratch(&p->partial, size_t(slots) * kPartialStride * 8, "partial-sum");
	scratch(&p->xhot, size_t(p->n_hot + 1) * kPanelBytes, "hot-pack");
	if (!rc && cudaMemset(p->xhot, 0, size_t(p->n_hot + 1) * kPanelBytes) != cudaSuccess)
		rc = set_error(FMX_ERR_CUDA, "clearing the hot pack failed");
	cudaSetDevice(cur);
	if (rc) return rc;
	out = p;
	return FMX_OK;
}

// ---------------------------------------------------------------------------
// Host: launching
// ---------------------------------------------------------------------------

template <class K>
static unsigned persistent_blocks(K kernel, int device, int threads)
{
	int sms = 0, per = 0;
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
	cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, 0);
	return unsigned(std::max(1, sms) * std::max(1, per));
}

// The persistent grid of `kernel` on `device`, kept in `slot` (one array of
// slots per kernel instantiation, indexed by device; racing first calls
// compute the same value).
template <class K>
static unsigned cached_blocks(std::atomic<unsigned> &slot, K kernel, int device, int threads)
{
	unsigned b = slot.load(std::memory_order_relaxed);
	if (!b) {
		b = persistent_blocks(kernel, device, threads);
		slot.store(b, std::memory_order_relaxed);
	}
	return b;
}

// Run launch(args) over the part's ranges: once for a resident entry stream;
// slice by slice for a streamed part.  Each slice is copied from pinned host
// memory into one of two device slots on the part's copy stream; the kernel
// of slice i (on st) waits for its copy, and the copy of slice i + 2 waits
// for that kernel, so copies overlap the kernels.  The slot pointer is
// rebased by the slice's first entry, so the ranges keep their absolute
// entry offsets.  The slots are the part's scratch: calls on one part must
// not overlap on the GPU (as for the hot pack and the partial sums).
template <class F>
static int over_slices(const gpu_part &p, spmm_args a, cudaStream_t st, F &&launch)
{
	if (!p.streamed) return launch(a);
	gpu_part &q = const_cast<gpu_part &>(p);
	const bool fine = p.fine && a.ranges == p.fine;
	CUDA_TRY(cudaEventRecord(q.ev_start, st));
	CUDA_TRY(cudaStreamWaitEvent(q.copy_st, q.ev_start, 0));
	for (size_t i = 0; i < p.slices.size(); i++) {
		const gpu_part::slice_t &sl = p.slices[i];
		const int b = int(i & 1);
		if (i >= 2) CUDA_TRY(cudaStreamWaitEvent(q.copy_st, q.ev_free[b], 0));
		const uint64_t ne = sl.e1 - sl.e0;
		CUDA_TRY(cudaMemcpyAsync(q.slot_col[b], p.h_col + sl.e0, ne * sizeof(uint32_t), cudaMemcpyHostToDevice,
				q.copy_st));
		if (p.esize)
			CUDA_TRY(cudaMemcpyAsync(q.slot_val[b], static_cast<const char *>(p.h_val) + sl.e0 * p.esize,
					ne * p.esize, cudaMemcpyHostToDevice, q.copy_st));
		CUDA_TRY(cudaEventRecord(q.ev_copied[b], q.copy_st));
		CUDA_TRY(cudaStreamWaitEvent(st, q.ev_copied[b], 0));
		a.col = q.slot_col[b] - sl.e0;
		a.val = p.esize ? static_cast<const void *>(static_cast<const char *>(q.slot_val[b]) - sl.e0 * p.esize)
				: nullptr;
		a.ranges = fine ? p.fine + sl.f0 : p.ranges + sl.r0;
		a.n_ranges = fine ? sl.nf : sl.nr;
		if (int rc = launch(a)) return rc;
		CUDA_TRY(cudaEventRecord(q.ev_free[b], st));
	}
	return FMX_OK;
}

// SMs of a device, asked once.
static unsigned device_sms(int device)
{
	static std::atomic<unsigned> sms[64];
	unsigned n = sms[device & 63].load(std::memory_order_relaxed);
	if (!n) {
		int v = 0;
		cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device);
		sms[device & 63].store(n = unsigned(std::max(v, 1)), std::memory_order_relaxed);
	}
	return n;
}

template <class XT, class YT, class A, class WT, int VN, int U, bool SI, bool SO, int FORM = kAny>
static int launch_step(const gpu_part &p, const spmm_args &a, cudaStream_t st)
{
	auto kern = spmm_lane_kernel<XT, YT, A, WT, VN, U, SI, SO, FORM>;
	static std::atomic<unsigned> blocks[64];
	const unsigned b = cached_blocks(blocks[p.device & 63], kern, p.device, kLaneThreads);
	// A dependent launch hides the launch of a short kernel (R-MAT scale 16,
	// k = 16: 26.8 -> 23.3 us with the fixup's).  Its blocks land where the pack's
	// drain first instead of in SM order, which cost the BF16 operator at scale
	// 21 2.6 %, so kernels of more than two rounds launch plainly (launch_lanes
	// takes longer steps only for fewer); so do those of a streamed part,
	// which follow their slice's copy.
	const uint64_t groups = uint64_t(b) * (kLaneThreads / 32) * unsigned(a.R);
	constexpr bool kFew = U > lane_step(VN * int(sizeof(XT)), int(sizeof(XT)), std::is_void<WT>::value && !SI && !SO);
	if (p.streamed || (!kFew && a.n_ranges > 2 * groups)) kern<<<b, kLaneThreads, 0, st>>>(a);
	else CUDA_TRY(launch_dep(kern, b, kLaneThreads, st, a));
	CUDA_TRY(cudaGetLastError());
	return FMX_OK;
}

template <class XT, class YT, class A, class WT, int VN, bool SI, bool SO, int FORM>
static int launch_lanes(const gpu_part &p, const spmm_args &a, cudaStream_t st)
{
	constexpr int U = lane_step(VN * int(sizeof(XT)), int(sizeof(XT)), std::is_void<WT>::value && !SI && !SO);
	// A small matrix leaves the machine to its longest ranges, rows of up to 256
	// entries whose steps each wait for their gathers: more entries a step then
	// beat more warps.  Lines in entries per group at 24 warps per SM.  Steps of
	// 8, 16, 32 at 2 / 8 / 17 entries (FP32 k = 16, R-MAT scale 12 / 14 / 15):
	// 20.6, 17.6, 17.2 / 22.6, 20.0, 16.6 / 22.7, 20.6, 17.8 us; at 33 (k = 8 at
	// scale 17; int64 weighted k = 4) 24.8, 22.7, 24.7 and 30.8, 28.8, 32.4; at 45
	// (int64, n = 300k) 36.2, 37.1, 41.1 us.
	if constexpr (FORM == kAny && VN > 1 && (VN * sizeof(XT) == 16 || VN * sizeof(XT) == 8) && sizeof(XT) >= 4 && !SI && !SO) {
		const uint64_t groups = uint64_t(device_sms(p.device)) * 24 * unsigned(a.R);
		if (p.nnz <= 24 * groups) return launch_step<XT, YT, A, WT, VN, 32, SI, SO>(p, a, st);
		if (U < 16 && p.nnz <= 40 * groups) return launch_step<XT, YT, A, WT, VN, 16, SI, SO>(p, a, st);
	}
	return launch_step<XT, YT, A, WT, VN, U, SI, SO, FORM>(p, a, st);
}

template <class XT, class YT, class A, class WT, int VN, int FORM = kAny>
static int launch_lanes_scaled(const gpu_part &p, const spmm_args &a, cudaStream_t st)
{
	if constexpr (std::is_floating_point<A>::value && (sizeof(XT) <= 4 || VN * sizeof(XT) <= 16)) {
		if constexpr (FORM != kBranch) {
			if (a.s_in && a.s_out) return launch_lanes<XT, YT, A, WT, VN, true, true, FORM>(p, a, st);
			if (a.s_out) return launch_lanes<XT, YT, A, WT, VN, false, true, FORM>(p, a, st);
		}
		if (a.s_in) return launch_lanes<XT, YT, A, WT, VN, true, false, FORM>(p, a, st);
	} else if (a.s_in || a.s_out) {
		return set_error(FMX_ERR_UNSUPPORTED, "no scaled kernel for lanes of %d elements", VN);
	}
	return launch_lanes<XT, YT, A, WT, VN, false, false, FORM>(p, a, st);
}

static bool aligned_to(const void *p, size_t n) { return (reinterpret_cast<uintptr_t>(p) % n) == 0; }

// BF16 lanes of 32 bytes exist for unweighted products into BF16.
template <class XT, class YT, class WT>
constexpr bool kWideBf16 = sizeof(XT) == 2 && sizeof(YT) == 2 && std::is_void<WT>::value;

// Elements per lane for a call: the widest unit of at most 16 bytes that
// every X and Y row is made of and starts on (stores go in units of up to 16
// bytes), or 32 bytes where that measured faster: FP32 with row scales (471
// against 528 us at R-MAT scale 21, k = 16: the scales cost instructions per
// entry, which wider lanes halve), and unscaled rows of 96 bytes or more
// (FP32 k = 32 weighted 786 against 882 us, FP64 k = 16 701 against 784 us at
// scale 22), but not shorter ones (k = 16 FP32 507 against 412 us).  Of BF16 rows
// those of 96 bytes or more into BF16, unweighted, on matrices with entries
// enough (input scales, k = 64, R-MAT scale 21 644 against 557 us, in the lanes
// before this kernel's 603; scale 16 39 against 43; weighted within 3 %).  FP32
// rows of less than a line with row scales, in operands of 2 GB or more, stay with
// 16 bytes: there the gathers miss most of the time, and twice the lanes hide
// more of it (symmetric scale 25, k = 16 / 24 / 32 14.3 / 19.4 / 19.9 ms against
// 14.9 / 20.2 / 17.4, the kernel before this one 14.2 / 19.5 / 19.5; scale 24 5.3 /
// 8.3 / 9.0 against 4.8 / 7.3 / 7.2).
template <class XT, class YT, class WT>
static int lane_width(const gpu_part &p, const void *X, int64_t ldx, const void *Y, int64_t ldy, int64_t k, bool scaled)
{
	if (uint64_t(ldx) * sizeof(XT) >= (1ull << 32)) return 1;
	auto fits = [&](int vn) {
		return k % vn == 0 && ldx % vn == 0 && aligned_to(X, vn * sizeof(XT)) && (ldy * sizeof(YT)) % std::min<size_t>(16, vn * sizeof(YT)) == 0 &&
				aligned_to(Y, std::min<size_t>(16, vn * sizeof(YT)));
	};
	constexpr int V32 = int(32 / sizeof(XT)), V16 = V32 / 2;
	const bool f32 = std::is_same<XT, float>::value;
	const int64_t row = std::min<int64_t>(k * int64_t(sizeof(XT)), kPanelBytes);
	const bool huge = p.ncols * uint64_t(ldx) * sizeof(XT) >= (2ull << 30);
	const bool wide = sizeof(XT) == 2 ? kWideBf16<XT, YT, WT> && row >= 96 && p.nnz >= (8u << 20) : scaled ? f32 && (row >= 128 || !huge) : row >= 96;
	if (wide && fits(V32)) return V32;
	int vn = V16;
	while (vn > 1 && !fits(vn)) vn /= 2;
	return vn;
}

// BF16 rows that are no whole units of two or more elements (odd widths, odd
// strides or starts): lanes of four elements, G apart, instead of one-element
// lanes, where those hold at most two rows a warp and an entry's decoding
// weighs more than its loads (R-MAT scale 21, k = 15 / 31 / 63: unscaled 544 ->
// 456, 1056 -> 727, 2146 -> 1372 us; D^-1/2 A D^-1/2 1374 -> 861, 2652 -> 1510,
// 5324 -> 2900 us; before the row kernel 500, 907, 1722 and 985, 1826, 3497 us),
// and, where cold entries load scales, for 7 to 10 columns of large matrices (7
// columns at scale 21 722 -> 641 us, unscaled 284 -> 339).  Fewer entries than 300
// per warp leave the grid to the longest chains, which one-element lanes walk
// faster (scale 14, k = 15 18.6 against 27 us; scale 16, k = 15 27 against 33 us,
// k = 17, one row a warp, 45 against 36 us).
constexpr int kApartUnit = 4;
template <class XT>
static bool lanes_apart(const gpu_part &p, int vn, int64_t ldx, int64_t k, bool scales_in)
{
	if (sizeof(XT) != 2 || vn != 1 || k < 7 || uint64_t(ldx) * sizeof(XT) >= (1ull << 32)) return false;
	const uint64_t warps = uint64_t(device_sms(p.device)) * 20 * uint64_t(32 / std::min<int64_t>(k, 32));
	return k >= 11 ? p.nnz >= 300 * warps : scales_in && p.nnz >= 1500 * warps;
}

// BF16 rows into FP32, eight columns a lane.  With one way to store them the
// compiler predicates the row close, so that every entry pays for its stores
// and resets; with two it branches around them.  The branch pays from three
// lanes a row on, where few rows share a warp (R-MAT scale 20 / 22, input scales,
// k = 32 222 / 784 -> 196 / 714 us, k = 48 341 / 1228 -> 292 / 1088, unscaled k = 64
// 343 / 1222 -> 298 / 1131; the kernel before this one 218 / 748, 324 / 1160 and
// 356 / 1265), not below (k = 8 96 us either way), where the matrix has entries
// enough (scale 18, k = 40 66 -> 74 us; scale 14, k = 24 25 -> 27), and without output
// scales, whose loads the branch holds up (scale 21, k = 48 839 -> 868).  Stores of
// whole sectors in a predicated close gained 1 to 5 %; FP32 lanes of 32 bytes
// measured within 4 % either way, FP64 ones 15 % slower.
static bool branch_close(const gpu_part &p, int vn, int64_t k, bool scales_out)
{
	return vn == 8 && k >= 24 && !scales_out && p.nnz >= (8u << 20);
}

// k = 1: the warp-per-range kernel while its grid (64 warps per SM) takes the
// ranges in one round, where its short chain wins (R-MAT scale 16: 18.9
// against 20.6 us); beyond that a lane per range in the row kernel, which
// issues a third of the instructions per entry (scale 18 / 20 / 22 / 24: 38 /
// 111 / 325 / 1400 against 29 / 66 / 251 / 1150 us).  A streamed part is
// launched slice by slice, so its largest slice decides (R-MAT scale 18 in
// slices of 64k entries 700 against 975 us), while the order of its sums is the
// resident form's (row_kernel_order).
static bool row_kernel_order(const gpu_part &p) { return p.n_ranges > device_sms(p.device) * 64; }
static bool spmv_by_warps(const gpu_part &p)
{
	uint32_t most = p.streamed ? 0 : p.n_ranges;
	for (const auto &sl : p.slices) most = std::max(most, sl.nr);
	return most <= device_sms(p.device) * 64;
}

// k = 1 without row scales: pack, the warp-per-range SpMV, fixup.
// `xhot` and `partial` default to the part's own scratch.
template <class T, class WT, bool EPI>
static int run_spmv(const gpu_part &p, const T *X, int64_t ldx, T *Y, int64_t ldy, cudaStream_t st,
		const pr_epi &e = pr_epi{}, void *xhot = nullptr, void *partial = nullptr, bool packed = false)
{
	if (!xhot) xhot = p.xhot;
	if (!partial) partial = p.partial;
	spmm_args a{};
	a.col = p.col; a.val = p.val; a.ranges = p.ranges;
	a.X = X; a.xhot = xhot; a.hot_ld = 1;
	a.Y = Y;
	a.partial = partial;
	a.ldx = ldx; a.ldy = ldy; a.k = 1;
	a.G = 1; a.R = 32;
	a.n_ranges = p.n_ranges;
	if (!packed) {
		const unsigned pb = unsigned(std::min<uint64_t>((uint64_t(p.n_hot) + 256) / 256, 148ull * 16));
		pack_hot_kernel<T, T, false><<<pb, 256, 0, st>>>(p.hot_col, p.n_hot, X, ldx, 1, static_cast<T *>(xhot), 1,
				nullptr);
		CUDA_TRY(cudaGetLastError());
	}
	const bool in_blocks = row_kernel_order(p);
	auto kern = in_blocks ? spmv_kernel<T, WT, EPI, true> : spmv_kernel<T, WT, EPI, false>;
	static std::atomic<unsigned> blocks[2][64];
	const unsigned b = cached_blocks(blocks[in_blocks][p.device & 63], kern, p.device, kThreads);
	if (int rc = over_slices(p, a, st, [&](const spmm_args &sa) -> int {
			if (p.streamed) kern<<<b, kThreads, 0, st>>>(sa, e);
			else CUDA_TRY(launch_dep(kern, b, kThreads, st, sa, e));
			CUDA_TRY(cudaGetLastError());
			return FMX_OK;
		}))
		return rc;
	if constexpr (EPI) return FMX_OK;          // the kernel's last warp of a heavy row finished it
	return launch_fixup<T, T, false>(p, static_cast<const T *>(partial), Y, ldy, 1, nullptr, st);
}

// One orientation over all column panels (kPanelBytes of X row each).
template <class XT, class YT, class A, class WT>
static int run_typed(const gpu_part &p, const void *X, int64_t ldx, void *Y, int64_t ldy, int64_t k,
		const void *sin, const void *sout, cudaStream_t st, void *xhot = nullptr, void *partial = nullptr,
		bool packed = false)
{
	if (!xhot) xhot = p.xhot;
	if (!partial) partial = p.partial;
	if constexpr (std::is_same<XT, A>::value && std::is_same<YT, A>::value && std::is_floating_point<A>::value) {
		if (k == 1 && !sin && !sout && spmv_by_warps(p))
			return run_spmv<A, WT, false>(p, static_cast<const A *>(X), ldx, static_cast<A *>(Y), ldy, st, pr_epi{}, xhot,
					partial);
	}
	const int vn = lane_width<XT, YT, WT>(p, X, ldx, Y, ldy, k, sin || sout);
	constexpr int V32 = int(32 / sizeof(XT));
	// column panels of at most kPanelBytes of X row, and 32 lanes
	const bool apart = lanes_apart<XT>(p, vn, ldx, k, sin != nullptr);
	const int unit = apart ? kApartUnit : vn;
	const int panel = std::min(kPanelBytes / int(sizeof(XT)), 32 * unit);
	// the pack that a producer left holds whole rows: one panel
	if (packed && k > panel) return set_error(FMX_ERR_INVAL, "a packed product of %lld columns takes several panels", (long long)k);
	for (int64_t c0 = 0; c0 < k; c0 += panel) {
		const int kp = int(std::min<int64_t>(panel, k - c0));
		spmm_args a{};
		a.col = p.col; a.val = p.val; a.ranges = p.fine ? p.fine : p.ranges;
		a.X = static_cast<const XT *>(X) + c0;
		a.xhot = xhot;
		a.hot_ld = kp;                // packed rows back to back (two 64-byte rows per line)
		a.Y = static_cast<YT *>(Y) + c0;
		a.s_in = sin; a.s_out = sout; a.partial = partial;
		a.ldx = ldx; a.ldy = ldy; a.k = kp;
		a.n_ranges = p.fine ? p.n_fine : p.n_ranges;
		a.G = (kp + unit - 1) / unit;
		a.R = 32 / a.G;
		if (!packed)
			if (int rc = launch_pack<XT, A>(p, static_cast<const XT *>(a.X), ldx, kp, static_cast<XT *>(xhot), kp,
					static_cast<const A *>(sin), st))
				return rc;
		if (int rc = over_slices(p, a, st, [&](const spmm_args &sa) -> int {
				if constexpr (std::is_same<XT, A>::value && std::is_same<YT, A>::value && std::is_floating_point<A>::value)
					if (k == 1 && !sin && !sout)
						return launch_step<A, A, A, WT, 1, lane_step(int(sizeof(A)), int(sizeof(A)), std::is_void<WT>::value), false,
								false, kOne>(p, sa, st);
				if constexpr (sizeof(XT) == 2)
					if (apart) return launch_lanes_scaled<XT, YT, A, WT, kApartUnit, kApart>(p, sa, st);
				if constexpr (sizeof(XT) == 2 && sizeof(YT) == 4)
					if (branch_close(p, vn, k, sout != nullptr)) return launch_lanes_scaled<XT, YT, A, WT, 8, kBranch>(p, sa, st);
				switch (vn) {
				case 1: return launch_lanes_scaled<XT, YT, A, WT, 1>(p, sa, st);
				case 2: return launch_lanes_scaled<XT, YT, A, WT, 2>(p, sa, st);
				case 4: return launch_lanes_scaled<XT, YT, A, WT, 4>(p, sa, st);
				}
				if constexpr (kWideBf16<XT, YT, WT>)
					if (vn == 16) return launch_lanes_scaled<XT, YT, A, WT, 16>(p, sa, st);
				if constexpr (V32 >= 8) return launch_lanes_scaled<XT, YT, A, WT, 8>(p, sa, st);
				return set_error(FMX_ERR_UNSUPPORTED, "no kernel for lanes of %d elements", vn);
			}))
			return rc;
		const A *so = static_cast<const A *>(sout);
		if (int rc = sout ? launch_fixup<YT, A, true>(p, static_cast<const A *>(partial), static_cast<YT *>(a.Y), ldy, kp, so, st)
				: launch_fixup<YT, A, false>(p, static_cast<const A *>(partial), static_cast<YT *>(a.Y), ldy, kp, nullptr, st))
			return rc;
	}
	return FMX_OK;
}

template <class XT, class YT, class A>
static int run_w(const gpu_part &p, const void *X, int64_t ldx, void *Y, int64_t ldy, int64_t k,
		const void *sin, const void *sout, cudaStream_t st, bool packed)
{
	switch (p.prim) {
	case FMX_P_BOOL: return run_typed<XT, YT, A, void>(p, X, ldx, Y, ldy, k, sin, sout, st, nullptr, nullptr, packed);
	case FMX_P_FLOAT:
		if constexpr (std::is_floating_point<A>::value) return run_typed<XT, YT, A, float>(p, X, ldx, Y, ldy, k, sin, sout, st, nullptr, nullptr, packed);
		break;
	case FMX_P_DOUBLE:
		if constexpr (std::is_same<A, double>::value) return run_typed<XT, YT, A, double>(p, X, ldx, Y, ldy, k, sin, sout, st, nullptr, nullptr, packed);
		break;
	case FMX_P_INTEGER:
		if constexpr (std::is_integral<A>::value) return run_typed<XT, YT, A, int32_t>(p, X, ldx, Y, ldy, k, sin, sout, st, nullptr, nullptr, packed);
		break;
	case FMX_P_LONG:
		if constexpr (std::is_same<A, int64_t>::value) return run_typed<XT, YT, A, int64_t>(p, X, ldx, Y, ldy, k, sin, sout, st, nullptr, nullptr, packed);
		break;
	}
	return set_error(FMX_ERR_TYPE, "matrix entry type %d does not match the dense type "
			"(sparse_matrix.cpp:759-766 allows a binary matrix or equal types; float entries "
			"with FP64 operands as spmm_creator<double,float>)", p.prim);
}

int spmm_part(const gpu_part &p, int xt, const void *X, int64_t ldx, int yt, void *Y, int64_t ldy,
		int64_t k, const void *sin, const void *sout, cudaStream_t st, bool packed = false)
{
	if (k <= 0) return set_error(FMX_ERR_DIM, "k must be positive (got %lld)", (long long)k);
	if (!X || !Y) return set_error(FMX_ERR_INVAL, "null X or Y");
	if (ldx < k || ldy < k) return set_error(FMX_ERR_DIM, "leading dimensions (%lld, %lld) smaller than k=%lld",
			(long long)ldx, (long long)ldy, (long long)k);
	int cur = 0;
	cudaGetDevice(&cur);
	if (cur != p.device) CUDA_TRY(cudaSetDevice(p.device));
	int rc;
	if (xt == FMX_F32 && yt == FMX_F32) rc = run_w<float, float, float>(p, X, ldx, Y, ldy, k, sin, sout, st, packed);
	else if (xt == FMX_F64 && yt == FMX_F64) rc = run_w<double, double, double>(p, X, ldx, Y, ldy, k, sin, sout, st, packed);
	else if (xt == FMX_BF16 && yt == FMX_F32) rc = run_w<__nv_bfloat16, float, float>(p, X, ldx, Y, ldy, k, sin, sout, st, packed);
	else if (xt == FMX_BF16 && yt == FMX_BF16) rc = run_w<__nv_bfloat16, __nv_bfloat16, float>(p, X, ldx, Y, ldy, k, sin, sout, st, packed);
	else if (xt == FMX_I32 && yt == FMX_I32) {
		rc = (sin || sout) ? set_error(FMX_ERR_UNSUPPORTED, "row scales need a floating-point type")
				: run_w<int32_t, int32_t, int32_t>(p, X, ldx, Y, ldy, k, nullptr, nullptr, st, packed);
	} else if (xt == FMX_I64 && yt == FMX_I64) {
		rc = (sin || sout) ? set_error(FMX_ERR_UNSUPPORTED, "row scales need a floating-point type")
				: run_w<int64_t, int64_t, int64_t>(p, X, ldx, Y, ldy, k, nullptr, nullptr, st, packed);
	} else rc = set_error(FMX_ERR_TYPE, "unsupported type pair x=%d y=%d "
			"(input and output matrices need the same type, sparse_matrix.cpp:754-758)", xt, yt);
	if (cur != p.device) cudaSetDevice(cur);
	return rc;
}

hot_pack_target pack_target(const fmx_matrix *m)
{
	return {m->a->slot, m->a->xhot, kPanelBytes};
}

int spmm_packed(const fmx_matrix *m, int xt, const void *X, int64_t ldx, int yt, void *Y, int64_t ldy, int64_t k,
		const void *sin, const void *sout, cudaStream_t st)
{
	return spmm_part(*m->a, xt, X, ldx, yt, Y, ldy, k, sin, sout, st, true);
}

// ---------------------------------------------------------------------------
// Fused PageRank iteration (SpMV on A^T with the update at each row close)
// ---------------------------------------------------------------------------

// The same loop test as a kernel, for streamed parts (several SpMV launches).
__global__ void pr_finish_kernel(unsigned long long *state, unsigned long long n, unsigned long long max_iters)
{
	if (threadIdx.x == 0 && !state[1]) {
		const unsigned long long it = ++state[2];
		if (state[0] >= n || it >= max_iters) state[1] = 1;
		state[0] = 0;
	}
}

__global__ void chunk_heavy_kernel(const heavy_row *heavy, uint32_t n_heavy, uint32_t *chunk_heavy)
{
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_heavy; i += gridDim.x * blockDim.x)
		for (uint32_t c = 0; c < heavy[i].count; c++) chunk_heavy[heavy[i].first + c] = i;
}

__global__ void heavy_mask_kernel(const heavy_row *heavy, uint32_t n_heavy, uint32_t *mask)
{
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_heavy; i += gridDim.x * blockDim.x) {
		const uint32_t r = uint32_t(heavy[i].row);
		atomicOr(mask + (r >> 5), 1u << (r & 31));
	}
}

int pagerank_maps(const fmx_matrix *mt, uint32_t *mask, uint32_t *chunk_heavy, const uint32_t **slot, const void **heavy,
		cudaStream_t st)
{
	const gpu_part &p = *mt->a;
	*heavy = p.heavy;
	*slot = p.slot;
	auto grid = [](uint32_t n) { return unsigned(std::min<uint32_t>((n + 255) / 256, 1024)); };
	if (p.n_heavy) heavy_mask_kernel<<<grid(p.n_heavy), 256, 0, st>>>(p.heavy, p.n_heavy, mask);
	CUDA_TRY(cudaGetLastError());
	if (p.n_heavy) chunk_heavy_kernel<<<grid(p.n_heavy), 256, 0, st>>>(p.heavy, p.n_heavy, chunk_heavy);
	CUDA_TRY(cudaGetLastError());
	return FMX_OK;
}

void pagerank_sizes(const fmx_matrix *mt, uint64_t *hot, uint64_t *heavy, uint64_t *chunks)
{
	*hot = mt->a->n_hot;
	*heavy = mt->a->n_heavy;
	*chunks = mt->a->n_partials;
}
bool pagerank_streamed(const fmx_matrix *mt) { return mt->a->streamed; }
bool pagerank_needs_out(const fmx_matrix *mt) { return !spmv_by_warps(*mt->a); }

template <class WT>
static int pr_iteration_typed(const gpu_part &p, const float *in, float *xhot, float *out, pr_epi e, cudaStream_t st)
{
	if (spmv_by_warps(p)) {
		// the update writes pr, pr1, the next input and its hot pack instead of Y
		e.finish = !p.streamed;
		if (int rc = run_spmv<float, WT, true>(p, in, 1, nullptr, 1, st, e, xhot, nullptr, true)) return rc;
		if (p.streamed) {
			pr_finish_kernel<<<1, 32, 0, st>>>(e.state, e.n, e.max_iters);
			CUDA_TRY(cudaGetLastError());
		}
		return FMX_OK;
	}
	// the row kernel of fmx_spmm at k = 1, then the update over all rows: a row
	// close there would wait on its own loads of deg and pr1
	spmm_args a{};
	a.col = p.col; a.val = p.val; a.ranges = p.fine ? p.fine : p.ranges;
	a.X = in; a.xhot = xhot; a.hot_ld = 1;
	a.Y = out; a.partial = p.partial;
	a.ldx = a.ldy = 1; a.k = 1; a.G = 1; a.R = 32;
	a.n_ranges = p.fine ? p.n_fine : p.n_ranges;
	a.state = e.state;
	constexpr int U = lane_step(int(sizeof(float)), int(sizeof(float)), std::is_void<WT>::value);
	if (int rc = over_slices(p, a, st, [&](const spmm_args &sa) -> int {
			return launch_step<float, float, float, WT, 1, U, false, false, kLoop>(p, sa, st);
		}))
		return rc;
	if (int rc = launch_fixup<float, float, false, true>(p, static_cast<const float *>(p.partial), out, 1, 1, nullptr, st, e.state))
		return rc;
	const unsigned g = unsigned(std::max<uint64_t>(1, std::min<uint64_t>((p.nrows + kThreads - 1) / kThreads, 148ull * 8)));
	CUDA_TRY(launch_dep(pr_apply_kernel, g, kThreads, st, out, int64_t(p.nrows), e));
	return FMX_OK;
}

int pagerank_iteration(const fmx_matrix *mt, const float *in, float *xhot, float *out, const pr_epi &e, cudaStream_t st)
{
	const gpu_part &p = *mt->a;
	if (p.prim == FMX_P_BOOL) return pr_iteration_typed<void>(p, in, xhot, out, e, st);
	if (p.prim == FMX_P_FLOAT) return pr_iteration_typed<float>(p, in, xhot, out, e, st);
	return set_error(FMX_ERR_TYPE, "PageRank: binary or float-weighted matrices");
}

// ---------------------------------------------------------------------------
// R-MAT (counter-based; identical streams on host and device)
// ---------------------------------------------------------------------------

struct rmat_params {
	uint64_t seed_key;
	uint32_t t_a, t_ab, t_abc;      // cumulative quadrant thresholds * 2^32
	int scale;
	int permute;
	uint64_t pm[4];                 // odd multipliers of the relabelling
	uint64_t pa[4];                 // addends
};

__host__ __device__ __forceinline__ uint64_t mix64(uint64_t z)
{
	// splitmix64 finaliser (Steele, Lea, Flood 2014)
	z += 0x9E3779B97F4A7C15ULL;
	z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
	z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
	return z ^ (z >> 31);
}

// A seeded bijection on [0, 2^scale): odd multiplies, adds and xor-shifts,
// each invertible modulo 2^scale.
__host__ __device__ __forceinline__ uint32_t relabel(const rmat_params &p, uint32_t v)
{
	const uint64_t mask = (p.scale >= 64) ? ~0ULL : ((1ULL << p.scale) - 1);
	uint64_t x = v;
	const int sh = p.scale / 2 + 1;
	for (int r = 0; r < 4; r++) {
		x = (x * p.pm[r] + p.pa[r]) & mask;
		x ^= x >> sh;
	}
	return uint32_t(x);
}

__host__ __device__ __forceinline__ void rmat_edge(const rmat_params &p, uint64_t e, uint32_t &src, uint32_t &dst)
{
	uint64_t h0 = mix64(p.seed_key ^ (e * 0xD6E8FEB86659FD93ULL));
	uint32_t r = 0, c = 0;
	uint64_t h = 0;
	for (int l = 0; l < p.scale; l++) {
		if ((l & 1) == 0) h = mix64(h0 + uint64_t(l) * 0x9E3779B97F4A7C15ULL);
		uint32_t u = (l & 1) ? uint32_t(h >> 32) : uint32_t(h);
		uint32_t rb = u >= p.t_ab;                 // quadrants c, d: row bit set
		uint32_t cb = (u >= p.t_a && u < p.t_ab) || u >= p.t_abc;  // b, d: col bit set
		r = (r << 1) | rb;
		c = (c << 1) | cb;
	}
	if (p.permute) { r = relabel(p, r); c = relabel(p, c); }
	src = r; dst = c;
}

static int rmat_setup(int scale, double a, double b, double c, uint64_t seed, int permute, rmat_params &p)
{
	if (scale < 1 || scale > 31) return set_error(FMX_ERR_INVAL, "R-MAT scale %d outside 1..31", scale);
	if (!(a >= 0 && b >= 0 && c >= 0 && a + b + c <= 1.0))
		return set_error(FMX_ERR_INVAL, "R-MAT probabilities a=%g b=%g c=%g invalid", a, b, c);
	auto th = [](double x) -> uint32_t {
		double v = x * 4294967296.0;
		return v >= 4294967295.0 ? 0xFFFFFFFFu : uint32_t(v);
	};
	p.seed_key = mix64(seed ^ 0x5851F42D4C957F2DULL);
	p.t_a = th(a); p.t_ab = th(a + b); p.t_abc = th(a + b + c);
	p.scale = scale;
	p.permute = permute;
	uint64_t s = mix64(seed + 0x1234567ULL);
	for (int r = 0; r < 4; r++) {
		s = mix64(s);
		p.pm[r] = s | 1ULL;
		s = mix64(s);
		p.pa[r] = s;
	}
	return FMX_OK;
}

__global__ void rmat_kernel(rmat_params p, uint64_t n, uint32_t *src, uint32_t *dst)
{
	for (uint64_t e = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < n; e += uint64_t(gridDim.x) * blockDim.x) {
		uint32_t s, d;
		rmat_edge(p, e, s, d);
		src[e] = s;
		dst[e] = d;
	}
}

int matrix_device(const fmx_matrix *m) { return m && m->a ? m->a->device : 0; }

int matrix_from_csr(const host_csr &a, const host_csr *at, int device, fmx_matrix **out)
{
	*out = nullptr;
	int ndev = 0;
	if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
		return set_error(FMX_ERR_CUDA, "no CUDA device is available");
	if (device < 0 || device >= ndev) return set_error(FMX_ERR_INVAL, "device %d out of range (%d devices)", device, ndev);
	std::unique_ptr<fmx_matrix> m(new (std::nothrow) fmx_matrix);
	if (!m) return set_error(FMX_ERR_OOM, "out of host memory");
	if (int rc = make_part(a, device, m->a)) return rc;
	if (at)
		if (int rc = make_part(*at, device, m->at)) return rc;
	m->symmetric = at == nullptr;
	*out = m.release();
	return FMX_OK;
}

} // namespace fmx

using namespace fmx;

extern "C" {

int fmx_matrix_create(const fmx_image *img, const fmx_image *t_img, int device, fmx_matrix **out)
{
	if (!img || !out) return set_error(FMX_ERR_INVAL, "null argument");
	*out = nullptr;
	int ndev = 0;
	if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
		return set_error(FMX_ERR_CUDA, "no CUDA device is available");
	if (device < 0 || device >= ndev) return set_error(FMX_ERR_INVAL, "device %d out of range (%d devices)", device, ndev);
	if (t_img && (t_img->im.h.nrows != img->im.h.ncols || t_img->im.h.ncols != img->im.h.nrows))
		return set_error(FMX_ERR_DIM, "transpose image is %llux%llu, expected %llux%llu",
				(unsigned long long)t_img->im.h.nrows, (unsigned long long)t_img->im.h.ncols,
				(unsigned long long)img->im.h.ncols, (unsigned long long)img->im.h.nrows);
	std::unique_ptr<fmx_matrix> m(new (std::nothrow) fmx_matrix);
	if (!m) return set_error(FMX_ERR_OOM, "out of host memory");
	const fmx_image *parts[2] = {img, t_img};
	for (int i = 0; i < 2; i++) {
		if (!parts[i]) continue;
		host_csr csr;
		int rc;
		try {
			rc = decode_to_csr(parts[i]->im, csr, default_threads());
		} catch (const std::bad_alloc &) {
			rc = set_error(FMX_ERR_OOM, "host allocation failed while decoding the image");
		}
		if (rc) return rc;
		rc = make_part(csr, device, i == 0 ? m->a : m->at);
		if (rc) return rc;
	}
	m->symmetric = (t_img == nullptr);
	*out = m.release();
	return FMX_OK;
}

int fmx_matrix_create_streamed(const fmx_image *img, const fmx_image *t_img, int device, uint64_t slice_entries,
		fmx_matrix **out)
{
	if (!img || !out) return set_error(FMX_ERR_INVAL, "null argument");
	*out = nullptr;
	if (!slice_entries) slice_entries = uint64_t(1) << 26;
	int ndev = 0;
	if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
		return set_error(FMX_ERR_CUDA, "no CUDA device is available");
	if (device < 0 || device >= ndev) return set_error(FMX_ERR_INVAL, "device %d out of range (%d devices)", device, ndev);
	if (t_img && (t_img->im.h.nrows != img->im.h.ncols || t_img->im.h.ncols != img->im.h.nrows))
		return set_error(FMX_ERR_DIM, "transpose image is %llux%llu, expected %llux%llu",
				(unsigned long long)t_img->im.h.nrows, (unsigned long long)t_img->im.h.ncols,
				(unsigned long long)img->im.h.ncols, (unsigned long long)img->im.h.nrows);
	std::unique_ptr<fmx_matrix> m(new (std::nothrow) fmx_matrix);
	if (!m) return set_error(FMX_ERR_OOM, "out of host memory");
	const fmx_image *parts[2] = {img, t_img};
	for (int i = 0; i < 2; i++) {
		if (!parts[i]) continue;
		host_csr csr;
		int rc;
		try {
			rc = decode_to_csr(parts[i]->im, csr, default_threads());
			if (!rc) rc = make_part(csr, device, i == 0 ? m->a : m->at, slice_entries);
		} catch (const std::bad_alloc &) {
			rc = set_error(FMX_ERR_OOM, "host allocation failed while decoding the image");
		}
		if (rc) return rc;
	}
	m->symmetric = (t_img == nullptr);
	*out = m.release();
	return FMX_OK;
}

int fmx_matrix_stream_info(const fmx_matrix *m, uint64_t *slices, uint64_t *host_bytes)
{
	if (!m || !m->a) return set_error(FMX_ERR_INVAL, "null matrix");
	if (slices) *slices = m->a->streamed ? m->a->slices.size() : 0;
	if (host_bytes) *host_bytes = m->a->host_bytes;
	return FMX_OK;
}

int fmx_matrix_build_device(const uint32_t *src, const uint32_t *dst, const void *vals, int val_type,
		uint64_t nedges, uint64_t nrows, uint64_t ncols, int flags, int device, void *stream, fmx_matrix **out)
{
	if (!out || (nedges && (!src || !dst)) || (val_type != FMX_P_BOOL && nedges && !vals))
		return set_error(FMX_ERR_INVAL, "null argument");
	*out = nullptr;
	if (flags & ~(FMX_BUILD_DEDUP | FMX_BUILD_KEEP_SELF_LOOPS | FMX_BUILD_TRANSPOSE))
		return set_error(FMX_ERR_INVAL, "flags 0x%x: the device builder takes DEDUP, KEEP_SELF_LOOPS and TRANSPOSE",
				flags);
	int ndev = 0;
	if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return set_error(FMX_ERR_CUDA, "no CUDA device is available");
	if (device < 0 || device >= ndev) return set_error(FMX_ERR_INVAL, "device %d out of range (%d devices)", device, ndev);
	int cur = 0;
	cudaGetDevice(&cur);
	CUDA_TRY(cudaSetDevice(device));
	std::unique_ptr<fmx_matrix> m(new (std::nothrow) fmx_matrix);
	int rc = m ? FMX_OK : set_error(FMX_ERR_OOM, "out of host memory");
	cudaStream_t st = static_cast<cudaStream_t>(stream);
	try {
		uint64_t nr = nrows, nc = ncols;
		{
			dev_csr csr;
			if (!rc) rc = edges_to_dev_csr(src, dst, vals, val_type, nedges, nrows, ncols, flags, st, csr);
			if (!rc) rc = make_part_device(csr, device, st, m->a);
			nr = csr.nrows;
			nc = csr.ncols;
		}
		if (!rc && (flags & FMX_BUILD_TRANSPOSE)) {
			dev_csr t;
			rc = edges_to_dev_csr(dst, src, vals, val_type, nedges, nc, nr, flags, st, t);
			if (!rc) rc = make_part_device(t, device, st, m->at);
		}
		if (!rc && cudaStreamSynchronize(st) != cudaSuccess) rc = set_error(FMX_ERR_CUDA, "device builder failed");
	} catch (const std::bad_alloc &) {
		rc = set_error(FMX_ERR_OOM, "host allocation failed in the device builder");
	}
	cudaSetDevice(cur);
	if (rc) return rc;
	m->symmetric = !(flags & FMX_BUILD_TRANSPOSE);
	*out = m.release();
	return FMX_OK;
}

int fmx_matrix_load(const char *mat_idx_path, const char *mat_path, const char *t_mat_idx_path,
		const char *t_mat_path, int device, fmx_matrix **out)
{
	fmx_image *a = nullptr, *t = nullptr;
	int rc = fmx_image_load(mat_idx_path, mat_path, &a);
	if (!rc && t_mat_idx_path && t_mat_path) rc = fmx_image_load(t_mat_idx_path, t_mat_path, &t);
	if (!rc) rc = fmx_matrix_create(a, t, device, out);
	fmx_image_free(a);
	fmx_image_free(t);
	return rc;
}

int fmx_matrix_info(const fmx_matrix *m, uint64_t *nrows, uint64_t *ncols, uint64_t *nnz, int *prim_type, int *symmetric)
{
	if (!m || !m->a) return set_error(FMX_ERR_INVAL, "null matrix");
	if (nrows) *nrows = m->a->nrows;
	if (ncols) *ncols = m->a->ncols;
	if (nnz) *nnz = m->a->nnz;
	if (prim_type) *prim_type = m->a->prim;
	if (symmetric) *symmetric = m->symmetric ? 1 : 0;
	return FMX_OK;
}

int fmx_matrix_device_bytes(const fmx_matrix *m, uint64_t *bytes)
{
	if (!m || !m->a || !bytes) return set_error(FMX_ERR_INVAL, "null argument");
	*bytes = m->a->bytes + (m->at ? m->at->bytes : 0);
	return FMX_OK;
}

int fmx_matrix_transpose(const fmx_matrix *m, fmx_matrix **out)
{
	if (!m || !out) return set_error(FMX_ERR_INVAL, "null argument");
	std::unique_ptr<fmx_matrix> t(new (std::nothrow) fmx_matrix);
	if (!t) return set_error(FMX_ERR_OOM, "out of host memory");
	t->symmetric = m->symmetric;
	if (m->symmetric) t->a = m->a;
	else { t->a = m->at; t->at = m->a; }
	*out = t.release();
	return FMX_OK;
}

int fmx_matrix_free(fmx_matrix *m)
{
	delete m;
	return FMX_OK;
}

int fmx_spmm(const fmx_matrix *m, int x_type, const void *X, int64_t ldx, int y_type, void *Y,
		int64_t ldy, int64_t k, const void *row_scale_in, const void *row_scale_out, void *stream)
{
	if (!m || !m->a) return set_error(FMX_ERR_INVAL, "null matrix");
	return spmm_part(*m->a, x_type, X, ldx, y_type, Y, ldy, k, row_scale_in, row_scale_out,
			static_cast<cudaStream_t>(stream));
}

static size_t dtype_size(int t)
{
	switch (t) {
	case FMX_F32: case FMX_I32: return 4;
	case FMX_F64: case FMX_I64: return 8;
	case FMX_BF16: return 2;
	}
	return 0;
}

int fmx_spmm_host(const fmx_matrix *m, int x_type, const void *X_host, int64_t ldx, int y_type,
		void *Y_host, int64_t ldy, int64_t k)
{
	if (!m || !m->a || !X_host || !Y_host) return set_error(FMX_ERR_INVAL, "null argument");
	size_t xs = dtype_size(x_type), ys = dtype_size(y_type);
	if (!xs || !ys) return set_error(FMX_ERR_TYPE, "unknown dtype");
	if (k <= 0 || ldx < k || ldy < k) return set_error(FMX_ERR_DIM, "bad k / leading dimensions");
	gpu_part &p = *m->a;
	std::lock_guard<std::mutex> guard(p.stage_mu);
	int cur = 0;
	cudaGetDevice(&cur);
	CUDA_TRY(cudaSetDevice(p.device));
	size_t xb = size_t(p.ncols) * k * xs, yb = size_t(p.nrows) * k * ys;
	int rc = FMX_OK;
	auto grow = [&](void *&buf, size_t &have, size_t need) -> int {
		if (have >= need) return FMX_OK;
		if (buf) cudaFree(buf);
		buf = nullptr; have = 0;
		if (cudaMalloc(&buf, need) != cudaSuccess) return set_error(FMX_ERR_OOM, "cudaMalloc of %zu staging bytes failed", need);
		have = need;
		return FMX_OK;
	};
	rc = grow(p.stage_x, p.stage_xb, xb);
	if (!rc) rc = grow(p.stage_y, p.stage_yb, yb);
	if (!rc && !p.stage_st && cudaStreamCreateWithFlags(&p.stage_st, cudaStreamNonBlocking) != cudaSuccess)
		rc = set_error(FMX_ERR_CUDA, "stream creation failed");
	if (!rc) {
		cudaStream_t st = p.stage_st;
		try {
			rc = run_host_copies(p.device, st, {p.stage_x, const_cast<void *>(X_host), k * xs, ldx * xs, p.ncols},
					{p.stage_y, Y_host, k * ys, ldy * ys, p.nrows}, [&] {
						return spmm_part(p, x_type, p.stage_x, k, y_type, p.stage_y, k, k, nullptr, nullptr, st);
					});
		} catch (const std::exception &e) {
			rc = set_error(FMX_ERR_OOM, "host copies: %s", e.what());
		}
		cudaError_t e = cudaStreamSynchronize(st);
		if (!rc && e != cudaSuccess) rc = set_error(FMX_ERR_CUDA, "SpMM failed: %s", cudaGetErrorString(e));
	}
	cudaSetDevice(cur);
	return rc;
}

int fmx_spmm_host_async(const fmx_matrix *m, int x_type, const void *X_host, int64_t ldx, int y_type,
		void *Y_host, int64_t ldy, int64_t k, void *stream)
{
	if (!m || !m->a || !X_host || !Y_host) return set_error(FMX_ERR_INVAL, "null argument");
	size_t xs = dtype_size(x_type), ys = dtype_size(y_type);
	if (!xs || !ys) return set_error(FMX_ERR_TYPE, "unknown dtype");
	if (k <= 0 || ldx < k || ldy < k) return set_error(FMX_ERR_DIM, "bad k / leading dimensions");
	gpu_part &p = *m->a;
	cudaStream_t st = static_cast<cudaStream_t>(stream);
	std::lock_guard<std::mutex> guard(p.stage_mu);
	int cur = 0;
	cudaGetDevice(&cur);
	CUDA_TRY(cudaSetDevice(p.device));
	const size_t xb = size_t(p.ncols) * k * xs, yb = size_t(p.nrows) * k * ys;
	int rc = FMX_OK;
	auto ev = [&](cudaEvent_t &e) {
		if (!rc && !e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess)
			rc = set_error(FMX_ERR_CUDA, "event creation failed");
	};
	auto stm = [&](cudaStream_t &s) {
		if (!rc && !s && cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess)
			rc = set_error(FMX_ERR_CUDA, "stream creation failed");
	};
	stm(p.h2d_st);
	stm(p.d2h_st);
	ev(p.ev_scratch);
	gpu_part::async_slot &sl = p.aslot[p.anext & 1];
	ev(sl.x_ready);
	ev(sl.spmm_done);
	ev(sl.y_out);
	if (!rc && (sl.xb < xb || sl.yb < yb)) {
		// growing: the slot's earlier call must be through first
		cudaEventSynchronize(sl.spmm_done);
		cudaEventSynchronize(sl.y_out);
		auto grow = [&](void *&buf, size_t &have, size_t need) -> int {
			if (have >= need) return FMX_OK;
			if (buf) cudaFree(buf);
			buf = nullptr; have = 0;
			if (cudaMalloc(&buf, need) != cudaSuccess)
				return set_error(FMX_ERR_OOM, "cudaMalloc of %zu staging bytes failed", need);
			have = need;
			return FMX_OK;
		};
		rc = grow(sl.x, sl.xb, xb);
		if (!rc) rc = grow(sl.y, sl.yb, yb);
	}
	auto copy = [&](void *dst, size_t dpitch, const void *src, size_t spitch, size_t width, size_t rows,
			cudaMemcpyKind kind, cudaStream_t s) {
		if (dpitch == width && spitch == width) return cudaMemcpyAsync(dst, src, width * rows, kind, s);
		return cudaMemcpy2DAsync(dst, dpitch, src, spitch, width, rows, kind, s);
	};
	auto wait = [&](cudaStream_t s, cudaEvent_t e) {
		if (!rc && cudaStreamWaitEvent(s, e, 0) != cudaSuccess) rc = set_error(FMX_ERR_CUDA, "stream wait failed");
	};
	auto record = [&](cudaEvent_t e, cudaStream_t s) {
		if (!rc && cudaEventRecord(e, s) != cudaSuccess) rc = set_error(FMX_ERR_CUDA, "event record failed");
	};
	// X in, on the copy-in stream, once the slot's last SpMM has read its X
	wait(p.h2d_st, sl.spmm_done);
	if (!rc && copy(sl.x, k * xs, X_host, ldx * xs, k * xs, p.ncols, cudaMemcpyHostToDevice, p.h2d_st) != cudaSuccess)
		rc = set_error(FMX_ERR_CUDA, "copy of X to the device failed");
	record(sl.x_ready, p.h2d_st);
	// the SpMM on the caller's stream: X arrived, the slot's last Y copied
	// out, and the SpMM issued before this one done (shared scratch)
	wait(st, sl.x_ready);
	wait(st, sl.y_out);
	wait(st, p.ev_scratch);
	if (!rc) rc = spmm_part(p, x_type, sl.x, k, y_type, sl.y, k, k, nullptr, nullptr, st);
	record(sl.spmm_done, st);
	record(p.ev_scratch, st);
	// Y out, on the copy-out stream; the call ends on the caller's stream
	// when Y has arrived
	wait(p.d2h_st, sl.spmm_done);
	if (!rc && copy(Y_host, ldy * ys, sl.y, k * ys, k * ys, p.nrows, cudaMemcpyDeviceToHost, p.d2h_st) != cudaSuccess)
		rc = set_error(FMX_ERR_CUDA, "copy of Y to the host failed");
	record(sl.y_out, p.d2h_st);
	wait(st, sl.y_out);
	p.anext++;
	cudaSetDevice(cur);
	return rc;
}

int fmx_matrix_hot(const fmx_matrix *m, uint64_t *n_hot_cols, uint64_t *hot_entries, uint64_t *scratch_bytes)
{
	if (!m || !m->a) return set_error(FMX_ERR_INVAL, "null matrix");
	const gpu_part &p = *m->a;
	if (n_hot_cols) *n_hot_cols = p.n_hot;
	if (hot_entries) *hot_entries = p.hot_entries;
	if (scratch_bytes) *scratch_bytes = uint64_t(p.n_hot + 1) * kPanelBytes + uint64_t(p.n_partials) * kPartialStride * 8;
	return FMX_OK;
}

int fmx_matrix_layout_digest(const fmx_matrix *m, int transpose, uint64_t *digest)
{
	if (!m || !m->a || !digest) return set_error(FMX_ERR_INVAL, "null argument");
	const gpu_part *pp = transpose && !m->symmetric ? m->at.get() : m->a.get();
	if (!pp) return set_error(FMX_ERR_INVAL, "the matrix has no transpose part");
	const gpu_part &p = *pp;
	if (p.streamed) return set_error(FMX_ERR_UNSUPPORTED, "a streamed matrix keeps its entry stream in host memory");
	device_guard on_device(p.device);
	if (!on_device.ok()) return set_error(FMX_ERR_CUDA, "cannot make device %d current", p.device);
	uint64_t h = 0xcbf29ce484222325ull;          // FNV-1a, 64 bits
	auto mix_host = [&](const void *q, size_t bytes) {
		const unsigned char *c = static_cast<const unsigned char *>(q);
		for (size_t i = 0; i < bytes; i++) { h ^= c[i]; h *= 0x100000001b3ull; }
	};
	std::vector<unsigned char> buf;
	auto mix = [&](const void *dev, size_t bytes) -> int {
		mix_host(&bytes, sizeof(bytes));
		buf.resize(bytes);
		if (bytes) CUDA_TRY(cudaMemcpy(buf.data(), dev, bytes, cudaMemcpyDeviceToHost));
		mix_host(buf.data(), bytes);
		return FMX_OK;
	};
	std::vector<range_t> rg(p.n_ranges);
	if (p.n_ranges) CUDA_TRY(cudaMemcpy(rg.data(), p.ranges, rg.size() * sizeof(range_t), cudaMemcpyDeviceToHost));
	uint64_t total = 0;
	for (const range_t &r : rg) total = std::max<uint64_t>(total, uint64_t(r.e0) + r.len);
	const size_t padded = size_t(total) + kStep;
	const uint64_t counts[] = {p.nrows, p.ncols, p.nnz, p.n_hot, p.n_exact, p.n_ranges, p.n_heavy, p.n_long_heavy,
			p.n_block_heavy, p.n_partials, p.hot_entries, p.n_fine};
	mix_host(counts, sizeof(counts));
	for (int rc : {mix(p.ranges, rg.size() * sizeof(range_t)), mix(p.fine, size_t(p.n_fine) * sizeof(range_t)), mix(p.col, padded * sizeof(uint32_t)),
			mix(p.val, p.esize ? padded * p.esize : 0), mix(p.heavy, size_t(p.n_heavy) * sizeof(heavy_row)),
			mix(p.hot_col, size_t(p.n_hot) * sizeof(int32_t)), mix(p.slot, size_t(p.ncols) * sizeof(uint32_t))})
		if (rc) return rc;
	*digest = h;
	return FMX_OK;
}

int fmx_matrix_schedule(const fmx_matrix *m, uint64_t *n_light_rows, uint64_t *n_split_tasks,
		uint64_t *n_heavy_rows, uint64_t *kernels_per_spmm)
{
	if (!m || !m->a) return set_error(FMX_ERR_INVAL, "null matrix");
	const gpu_part &p = *m->a;
	if (n_light_rows) *n_light_rows = p.n_exact;
	if (n_split_tasks) *n_split_tasks = p.fine ? p.n_fine : p.n_ranges;
	if (n_heavy_rows) *n_heavy_rows = p.n_heavy;
	if (kernels_per_spmm)
		*kernels_per_spmm = 2 + (p.n_heavy ? 1 : 0);
	return FMX_OK;
}

int fmx_rmat_edges_host(int scale, uint64_t nedges, double a, double b, double c, uint64_t seed,
		int permute, uint32_t *src, uint32_t *dst, int nthreads)
{
	rmat_params p;
	int rc = rmat_setup(scale, a, b, c, seed, permute, p);
	if (rc) return rc;
	if (nedges && (!src || !dst)) return set_error(FMX_ERR_INVAL, "null output arrays");
	if (nthreads <= 0) nthreads = default_threads();
	std::vector<std::thread> th;
	uint64_t per = (nedges + nthreads - 1) / nthreads;
	for (int t = 0; t < nthreads; t++)
		th.emplace_back([&, t]() {
			uint64_t b0 = uint64_t(t) * per, b1 = std::min(nedges, b0 + per);
			for (uint64_t e = b0; e < b1; e++) rmat_edge(p, e, src[e], dst[e]);
		});
	for (auto &x : th) x.join();
	return FMX_OK;
}

int fmx_rmat_edges_device(int scale, uint64_t nedges, double a, double b, double c, uint64_t seed,
		int permute, uint32_t *src_dev, uint32_t *dst_dev, void *stream)
{
	rmat_params p;
	int rc = rmat_setup(scale, a, b, c, seed, permute, p);
	if (rc) return rc;
	if (!nedges) return FMX_OK;
	if (!src_dev || !dst_dev) return set_error(FMX_ERR_INVAL, "null output arrays");
	unsigned blocks = unsigned(std::min<uint64_t>((nedges + 255) / 256, 148ULL * 64));
	rmat_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(p, nedges, src_dev, dst_dev);
	CUDA_TRY(cudaGetLastError());
	return FMX_OK;
}

} // extern "C"

// ---------------------------------------------------------------------------
// SpMM that allocates nothing
//
// For callers that cannot allocate device memory while they run: code inside
// a memory pool or arena that owns all of the device's memory, code running
// where the allocator is off limits (a custom allocator's own callbacks, a
// signal-driven or real-time path), or hosts that forbid device allocation
// after start-up.  fmx_spmm itself allocates nothing per call either, but its
// scratch is allocated with the matrix; this entry point instead uses a fixed
// scratch array compiled into the library, so its scratch exists on every
// GPU that loads libfmx from load until process exit.
// ---------------------------------------------------------------------------
namespace fmx {

constexpr size_t kNoAllocScratchBytes = size_t(32) << 20;     // 32 MiB per device
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

static std::mutex g_noalloc_mu;
static void *g_noalloc_ptr[64];

// The device address of the scratch array on `device` (the current device).
// Host code cannot use g_noalloc_scratch directly: there it is only a host
// stand-in for the symbol, not a device address.
static int noalloc_scratch(int device, void **ptr)
{
	if (device < 0 || device >= 64) return set_error(FMX_ERR_UNSUPPORTED, "device %d out of range for the fixed scratch", device);
	std::lock_guard<std::mutex> g(g_noalloc_mu);
	if (!g_noalloc_ptr[device]) {
		void *p = nullptr;
		cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
		if (e != cudaSuccess || !p)
			return set_error(FMX_ERR_CUDA, "cudaGetSymbolAddress of the fixed scratch failed: %s", cudaGetErrorString(e));
		g_noalloc_ptr[device] = p;
	}
	*ptr = g_noalloc_ptr[device];
	return FMX_OK;
}

} // namespace fmx

extern "C" int fmx_spmm_noalloc(const fmx_matrix *m, const float *X, int64_t ldx, float *Y, int64_t ldy,
		int64_t k, void *stream)
{
	using namespace fmx;
	if (!m || !m->a || !X || !Y) return set_error(FMX_ERR_INVAL, "null argument");
	const gpu_part &p = *m->a;
	if (k <= 0 || ldx < k || ldy < k) return set_error(FMX_ERR_DIM, "bad k (%lld) or leading dimensions", (long long)k);
	if (p.prim != FMX_P_BOOL && p.prim != FMX_P_FLOAT)
		return set_error(FMX_ERR_TYPE, "fmx_spmm_noalloc takes binary or float-weighted matrices");
	if (p.streamed) return set_error(FMX_ERR_UNSUPPORTED, "fmx_spmm_noalloc takes matrices resident in HBM");
	// scratch layout: the hot pack (widest panel), then the long-row partial sums
	const size_t hot_bytes = (size_t(p.n_hot + 1) * kPanelBytes + 255) / 256 * 256;
	const size_t need = hot_bytes + size_t(p.n_partials) * kPartialStride * sizeof(float);
	if (need > kNoAllocScratchBytes)
		return set_error(FMX_ERR_UNSUPPORTED, "this matrix needs %zu bytes of SpMM scratch; the fixed scratch of "
				"fmx_spmm_noalloc holds %zu bytes (use fmx_spmm)", need, kNoAllocScratchBytes);
	int cur = 0;
	cudaGetDevice(&cur);
	if (cur != p.device && cudaSetDevice(p.device) != cudaSuccess)
		return set_error(FMX_ERR_CUDA, "cannot select device %d", p.device);
	void *base = nullptr;
	int rc = noalloc_scratch(p.device, &base);
	if (!rc) {
		void *xhot = base;
		void *partial = static_cast<char *>(base) + hot_bytes;
		cudaStream_t st = static_cast<cudaStream_t>(stream);
		// the kernels fmx_spmm runs for the same call, on the fixed scratch
		rc = (p.prim == FMX_P_BOOL)
				? run_typed<float, float, float, void>(p, X, ldx, Y, ldy, k, nullptr, nullptr, st, xhot, partial)
				: run_typed<float, float, float, float>(p, X, ldx, Y, ldy, k, nullptr, nullptr, st, xhot, partial);
	}
	if (cur != p.device) cudaSetDevice(cur);
	return rc;
}
