// gwf_blocks.cuh — the distance kernel of the batch forms: block wavefronts with exact pruning.
//
// Same scores as the sorted wavefront of gwf_kernels.cuh, another data structure. The diagonals of
// a read live in blocks of 8 neighbouring diagonals of one vertex, one 128-byte line each, found
// through a hash table of block ids and linked to their neighbours. A score step
//   1. walks the list of live blocks: each diagonal's successor is max(k[d-1], k[d] + 1,
//      k[d+1] + 1, arc-side candidate), dropped where the diagonal has passed the vertex end,
//      extended and written to the row of the step's parity (gwf-ed.cu:902-1016);
//   2. sends the vertex-end states over their arcs in waves (gwf-ed.cu:1106-1255): an arrival is
//      a bit of the target diagonal's cell, a candidate a max into it, so that no arrival set, no
//      sort, no merge and no interval list remain.
//
// Exact pruning. A lag-pruned run of the same loop first gives an upper bound U of the read's
// distance (an alignment of U edits exists). Then a state at score s and query position i is
// dropped when s + h(i + 1) >= U, where h counts edits that the rest of the query cannot avoid
// (bw_seeds). Dropped states cannot lead to a distance below U, and the states of a shorter
// alignment all survive, so the distance is the one of the unpruned run: U where that run finds
// none below it. States per read, against the unpruned loop: configuration 3 39,200 -> 5,700,
// configuration 4 962,000 -> 107,000, and 10,700 with windows from every base; the lag run needs
// 600 and 2,300.
//
// What bounds it: instruction fetch and issue (ncu, 20,000 mixed reads of at most 4 kbp: 0.37
// instructions issued per cycle and scheduler at 32 warps per SM, 9.2 of a warp's 20.4 cycles per
// instruction waiting for its next instruction, 4.6 for loads, 2.8 for fixed latencies; DRAM 0.76 GB
// in 7.6 ms), and the latency of one read's chain of steps where a batch has few or unequal reads.
// Resident reads, graph replay, kernel_ms against the sorted form: 100,000 x 1 kbp 26.1 -> 12.6 ms,
// 50,000 mixed 137 -> 27 ms, 4,000 x 10 kbp on the dense graph 600 -> 30 ms, one 20 kbp read at 10%
// 374 -> 67 ms (243 with one warp, 16 here). With several warps per read barriers bound it: 100 reads
// of 10 kbp at 5% with 16 warps each, 38 of a warp's 48 cycles per instruction, 2.3 for loads: most of
// a read's steps have work for a warp or two.
#pragma once
#include "gwf_kernels.cuh"

namespace gwfb {

constexpr int32_t BW_NONE = -(1 << 29);
constexpr int32_t BW_ENDED = 1 << 29; // arc-side candidate that ends its diagonal
constexpr int32_t BW_INF = 0x3fffffff;

// One block, 128 bytes. rows[s & 1] holds the extended k of score step s.
struct __align__(128) BwBlock {
	uint32_t gb;       // first base of the vertex in the concatenated sequence
	uint32_t arcs;     // its arcs (DevGraph::varcs)
	uint32_t v;
	int32_t db;        // diagonal of cell 0 (a multiple of 8)
	int32_t vl;
	int32_t left, right; // neighbouring blocks, -1 = none yet
	uint32_t flags;    // BwBits
	int32_t row[2][8];
	int32_t c[8];      // arc-side candidate of the next step: k << 1 | arrived with one warp, k with several
};
static_assert(sizeof(BwBlock) == 128, "one line per block");

// Bits of a block's flags: diagonals past the vertex end (0 to 7), an arc-side candidate is there, in
// the live list of even / odd steps. With one warp per read the lists and the candidate flag have a
// byte each, which lanes store without a read; with several warps (MW) they are bits set by
// atomicOr, and bits 8 to 15 are the cells that an arc has reached, so that one atomicOr takes an
// arrival, flags its candidate and lists the block.
template <bool MW>
struct BwBits {
	static constexpr uint32_t has_c = MW ? 1u << 18 : 0x100u, clear_c = MW ? 1u << 18 : 0xff00u;
	static __device__ __forceinline__ uint32_t inl(int par) { return 0x10000u << (MW ? par : 8 * par); }
	static __device__ __forceinline__ uint32_t drop(int par) { return clear_c | (MW ? 0x10000u << par : 0xff0000u << (8 * par)); }
	static constexpr int32_t none = MW ? BW_NONE : 2 * BW_NONE;
	static __device__ __forceinline__ int32_t k(int32_t c) { return MW ? c : c >> 1; }
	static __device__ __forceinline__ int32_t taken(int32_t c) { return MW ? BW_NONE : 2 * BW_NONE | (c & 1); }
};

// Word of a string in the graph's filter, and its bits there: two in each half of the word. The
// multipliers, here and in bw_tag, are those of published 32-bit mixers: 2^32 / golden ratio (xxHash's
// first prime), MurmurHash3's finaliser, and a pair found by the hash-prospector search.
__host__ __device__ inline uint32_t bloom_word(uint32_t x, uint32_t mask)
{
	x *= 0x9E3779B1u;
	x ^= x >> 15;
	x *= 0x2C1B3C6Du;
	return (x ^ x >> 13) & mask;
}
__host__ __device__ inline uint2 bloom_bits(uint32_t x)
{
	const uint32_t y = (x ^ x >> 16) * 0x85EBCA6Bu;
	return make_uint2(1u << (y >> 27) | 1u << (y >> 22 & 31), 1u << (y >> 17 & 31) | 1u << (y >> 12 & 31));
}

#ifndef GWF_KERNELS_DECL_ONLY
// Lag of the run that gives an upper bound. A larger one costs more states (24: 2,000 x 10 kbp at 10%
// 97.6 -> 102.0 ms), a smaller one loses the read's path sooner, and the bound with it (6: 4,000 x
// 10 kbp at 5% on the dense graph 29.7 -> 238 ms, 8: 29.7).
constexpr int32_t kPruneLag = 10;

// The filter's build: every string of K = bloom_k bases that a walk of the graph spells, from
// every position, one start per thread (its vertex by binary search, so that a long vertex is as
// many threads as it has bases); walks branch through a stack (fewer than K levels, as each vertex
// gives at least one base). A walk that dead-ends after K - 1 bases enters all four extensions, so
// that a string of K - 1 bases may be looked up by extending it. A start with more than kBloomLeaves
// walks sets *many, the graph gets no filter, and threads that start later have nothing to do.
constexpr int32_t kBloomLeaves = 1024;
__device__ __forceinline__ void bloom_put(unsigned long long *bloom, uint32_t mask, uint32_t x)
{
	const uint2 b = bloom_bits(x);
	atomicOr(bloom + bloom_word(x, mask), (unsigned long long)b.y << 32 | b.x);
}
__global__ void __launch_bounds__(256) k_bloom(const __grid_constant__ DevGraph g, unsigned long long *bloom,
                                               int32_t *many)
{
	const uint64_t p0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (p0 >= g.total_len || *(volatile const int32_t *)many) return;
	const int32_t K = g.bloom_k;
	const uint32_t mask = g.bloom_mask;
	uint32_t v = 0; // the last vertex that begins at or before p0
	for (uint32_t hi = g.n_vtx; hi - v > 1;) {
		const uint32_t mid = v + (hi - v) / 2;
		if (__ldg(g.base + mid) <= p0) v = mid;
		else hi = mid;
	}
	uint32_t st_x[17], st_a[17], st_e[17];
	int32_t st_n[17];
	int32_t depth = 0, n = 0, leaves = 0;
	uint32_t o = (uint32_t)(p0 - __ldg(g.base + v)), x = 0;
	for (int64_t guard = 0; guard < 64LL * kBloomLeaves; ++guard) {
		const uint32_t vl = __ldg(g.len + v);
		const uint64_t gb = __ldg(g.base + v);
		for (; o < vl && n < K; ++o, ++n) {
			const uint64_t p = gb + o;
			x |= (uint32_t)(__ldg(g.pk + (p >> 5)) >> (2 * (p & 31)) & 3) << (2 * n);
		}
		bool up = false;
		if (n == K) {
			bloom_put(bloom, mask, x);
			up = true;
		} else {
			const uint32_t a = __ldg(g.arc_off + v), e = __ldg(g.arc_off + v + 1);
			if (a == e) {
				if (n == K - 1)
					for (uint32_t y = 0; y < 4; ++y) bloom_put(bloom, mask, x | y << (2 * K - 2));
				up = true;
			} else
				st_x[depth] = x, st_n[depth] = n, st_a[depth] = a, st_e[depth] = e, ++depth;
		}
		if (up && ++leaves > kBloomLeaves) break;
		while (depth > 0 && st_a[depth - 1] == st_e[depth - 1]) --depth;
		if (depth == 0) break;
		const uint2 arc = __ldg(g.arc + st_a[depth - 1]++);
		v = arc.x, o = arc.y, x = st_x[depth - 1], n = st_n[depth - 1];
	}
	if (leaves > kBloomLeaves || depth > 0) *many = 1;
}

// State of a read's run, in the CTA's shared memory (a CTA aligns one read at a time, with one warp
// or, MW, with several). The parts of the kernel that are not run at every step are functions of
// their own that work on it: with everything inlined the kernel had 87 KB of code, its 32 warps per
// SM stood in different parts of it, and waits for instructions took 11 of 21 cycles per issue
// (100,000 x 1 kbp 18.8 ms, 14.3 as functions). bw_ext stays inlined: 12.7 ms, 13.4 out of line.
constexpr int kBwQueue = 31 + 16 * 8;
struct BwShm {
	BwBlock *blk;
	uint2 *hash;               // (tag, id) per slot, all ones = empty
	uint32_t *slot;            // slot of each block
	int32_t *nxt;              // live list of the next step
	uint32_t *e, *f, *n;       // vertex-end states of a wave and of the next, entered states: id << 3 | cell
	int32_t *nk;               // offsets of the entered states
	uint16_t *h;               // edits that the last rem bases cannot avoid
	const uint64_t *qpk;
	const uint8_t *qraw;
	const uint32_t *gpk;
	const uint8_t *graw;
	const uint4 *arcx;
	const uint32_t *varcs, *arc_off;
	const uint64_t *bloom;
	uint32_t bloom_mask;
	int32_t K;
	uint32_t hmask;
	int32_t nb;                // blocks in the pool
	int32_t ql, packed, quirk;
	int32_t n_blk;             // blocks in use
	int32_t ovf;               // a buffer is full
	// of a step
	int32_t s, imin;           // score; query position behind which a lag run drops states
	int32_t lag;               // the caller's max_lag, 0 = none
	int32_t far_c;             // with it: the furthest query position of a candidate
	int32_t n_nxt, n_e;        // lengths of nxt and e
	int32_t next;              // next entry of the live list to be taken
	int32_t any, found, far;   // a state lives, one reached the query's end, furthest query position
	int32_t n_n[2], n_f[2];    // of a wave, by its parity
	int32_t claim;             // MW: queue position of the group's read
	int32_t pad;
};
__device__ __forceinline__ BwShm &bw_sh()
{
	extern __shared__ __align__(16) unsigned char bw_smem[];
	return *(BwShm *)bw_smem;
}
// Diagonals on their way to the extension: id << 4 | side << 3 | cell, k; one queue per warp
__device__ __forceinline__ uint2 *bw_queue()
{
	return (uint2 *)(&bw_sh() + 1) + (threadIdx.x >> 5) * (kBwQueue + 1);
}
constexpr size_t bw_shm_bytes(int warps) { return sizeof(BwShm) + (size_t)warps * (kBwQueue + 1) * sizeof(uint2); }
static_assert(sizeof(BwShm) % 16 == 0, "the queues follow");

template <bool MW>
__device__ __forceinline__ void bw_bar()
{
	if constexpr (MW) __syncthreads();
	else __syncwarp();
}
// n entries appended behind the counter c (a warp's; the lanes of mask m, in lane order): this
// lane's place
template <bool MW>
__device__ __forceinline__ int32_t bw_append(int32_t *c, uint32_t m)
{
	int32_t at;
	if constexpr (MW) {
		at = 0;
		if ((threadIdx.x & 31) == 0 && m) at = atomicAdd(c, __popc(m));
		at = __shfl_sync(FULL, at, 0);
	} else {
		at = *c;
		__syncwarp();
		*c = at + __popc(m);
		__syncwarp();
	}
	return at + __popc(m & lanemask_lt());
}

__device__ __forceinline__ bool bloom_has(const BwShm &sh, uint32_t x)
{
	const uint2 b = bloom_bits(x), w = __ldg((const uint2 *)sh.bloom + bloom_word(x, sh.bloom_mask));
	return ((b.x & ~w.x) | (b.y & ~w.y)) == 0;
}

// Does the graph (as its filter says) spell the K-base string y with one edit at base a? Kind 0: the
// base xor t; 1: the base t inserted before a (K + 1 bases: the first K and the last K); 2: the base
// taken out and t appended.
template <int KIND>
__device__ __forceinline__ bool bw_edit(const BwShm &sh, uint32_t y, int a, uint32_t t)
{
	const int K = sh.K, a2 = 2 * a;
	if (KIND == 0) return bloom_has(sh, y ^ t << a2);
	const uint32_t lo = y & ((1u << a2) - 1), hi = y >> a2;
	if (KIND == 2) return bloom_has(sh, hi >> 2 << a2 | lo | t << (2 * K - 2));
	const uint64_t z = (uint64_t)(hi << 2 | t) << a2 | lo;
	bool ok = bloom_has(sh, (uint32_t)z & ~0u >> (32 - 2 * K));
	if (ok) ok = bloom_has(sh, (uint32_t)(z >> 2));
	return ok;
}

// Edits that the last rem bases of the query cannot avoid, rem = 0 .. ql, into h[rem]; returns
// h[ql]. A window of K bases costs 0, 1 or 2 edits when the graph spells a string within 0, 1 or
// more edits of it; windows that do not overlap add up, so h[rem] = max(h[rem - 1], h[rem - K] +
// cost of the window that starts rem bases before the end). Windows start every `stride` bases: K
// (side by side, first) or 1 (after that, on the same read).
// Lanes test 32 windows for exact presence. An absent one is looked up with one edit by the whole
// warp (3 K substitutions, 4 (K - 1) insertions, 4 K deletions with any appended base); an edit
// that is found is then tried on the other absent windows of the 32 that hold its position. A
// window with a byte other than A/C/G/T costs 1 (the graph has none). With stride 1 every other
// absent window counts 1 without the one-edit lookups: half of them, for a bound 0.5% lower.
template <bool MW>
static __device__ __noinline__ int32_t bw_seeds(int32_t stride)
{
	const BwShm &sh = bw_sh();
	const int lane = threadIdx.x & 31;
	const int32_t K = sh.K, ql = sh.ql;
	uint16_t *const h = sh.h;
	const int32_t wid = MW ? threadIdx.x >> 5 : 0, nw = MW ? blockDim.x >> 5 : 1;
	bw_bar<MW>();
#pragma unroll 1
	for (int32_t base = K + 32 * stride * wid; base <= ql; base += 32 * stride * nw) {
		const int32_t rem = base + lane * stride, p = ql - rem;
		uint32_t x = 0, nb = 0; // the window and the base after it
		int32_t cost = 0;
		if (rem <= ql) {
			uint32_t lo, hi;
			window32<false>((const uint32_t *)sh.qpk, p, lo, hi);
			x = lo & ~0u >> (32 - 2 * K);
			nb = (K == 16 ? hi : lo >> (2 * K)) & 3;
			bool odd = false;
			if (!sh.packed)
#pragma unroll 1
				for (int t = 0; t < K; ++t) {
					const uint8_t ch = sh.qraw[p + t];
					odd |= !(ch == 'A' || ch == 'C' || ch == 'G' || ch == 'T');
				}
			cost = odd ? 1 : bloom_has(sh, x) ? 0 : stride == 1 && (rem & 1) ? 1 : 2;
		}
		uint32_t todo = __ballot_sync(FULL, cost == 2);
#pragma unroll 1
		while (todo) {
			const int src = __ffs(todo) - 1;
			todo &= todo - 1;
			const uint32_t y = __shfl_sync(FULL, x, src);
			const int32_t sp = __shfl_sync(FULL, p, src);
			uint32_t hit = 0;
			int kind = 0, code = 0; // a << 2 | t of the lane's last try
#pragma unroll 1
			for (int t = lane; t < 3 * K + lane && !hit; t += 32) {
				code = (t / 3) << 2 | (t % 3 + 1);
				hit = __ballot_sync(FULL, t < 3 * K && bw_edit<0>(sh, y, code >> 2, code & 3));
			}
			if (!hit) kind = 1;
#pragma unroll 1
			for (int t = 4 + lane; t < 4 * K + lane && !hit; t += 32) {
				code = t;
				hit = __ballot_sync(FULL, t < 4 * K && bw_edit<1>(sh, y, code >> 2, code & 3));
			}
			if (!hit) kind = 2;
#pragma unroll 1
			for (int t = lane; t < 4 * K + lane && !hit; t += 32) {
				code = t;
				hit = __ballot_sync(FULL, t < 4 * K && bw_edit<2>(sh, y, code >> 2, code & 3));
			}
			if (!hit) continue;
			if (lane == src) cost = 1;
			if (todo && stride == 1) { // the same edit in this lane's window
				const int c = __shfl_sync(FULL, code, __ffs(hit) - 1), a = sp + (c >> 2) - p;
				bool same = (todo >> lane & 1) && a >= (kind == 1) && a < K;
				if (same)
					same = kind == 0 ? bw_edit<0>(sh, x, a, c & 3) : kind == 1 ? bw_edit<1>(sh, x, a, c & 3)
					                                               : bw_edit<2>(sh, x, a, nb);
				if (same) cost = 1;
				todo &= __ballot_sync(FULL, cost == 2);
			}
		}
		if (rem <= ql) h[rem] = (uint16_t)cost;
	}
	bw_bar<MW>();
	if (stride == K) {
		// windows side by side: h[rem] is the sum over the rem / K last of them
		int32_t sum = 0;
#pragma unroll 1
		for (int32_t base = K; base <= ql && wid == 0; base += 32 * K) {
			const int32_t rem = base + lane * K;
			int32_t tot;
			const int32_t c = rem <= ql ? (int32_t)h[rem] : 0, pre = sum + warp_excl_scan(c, &tot);
			if (rem < ql + K)
#pragma unroll 1
				for (int32_t j = rem - K; j < rem && j <= ql; ++j) h[j] = (uint16_t)min(pre, 65535);
			sum += tot;
			__syncwarp();
			if (rem <= ql && rem + K > ql)
#pragma unroll 1
				for (int32_t j = rem; j <= ql; ++j) h[j] = (uint16_t)min(pre + c, 65535);
			__syncwarp();
		}
		bw_bar<MW>();
		return (int32_t)h[ql];
	}
	// the maximum over disjoint windows, K entries at a time: lane l's entry takes its window after
	// h[rem - K] of the pass before
	int32_t prev = 0; // lane l < K: h[b - K + l]
	int32_t last = 0; // h[b - 1]
#pragma unroll 1
	for (int32_t b = K; b <= ql && wid == 0; b += K) {
		const int32_t rem = b + lane;
		const bool on = lane < K && rem <= ql;
		int32_t v = on ? prev + (int32_t)h[rem] : 0;
		v = max(v, last);
#pragma unroll
		for (int o = 1; o < 16; o <<= 1) {
			const int32_t u = __shfl_up_sync(FULL, v, o);
			if (lane >= o) v = max(v, u);
		}
		if (on) h[rem] = (uint16_t)min(v, 65535);
		prev = v;
		last = __shfl_sync(FULL, v, K - 1);
	}
	bw_bar<MW>();
	return (int32_t)h[ql];
}

// gwf_extend1 (see ext) with the vertex's first base gb at hand. The whole warp calls it; on: this
// lane extends. Every compare covers 32 bases and may run past either end (padding words).
static __device__ __noinline__ int32_t bw_ext_raw(uint32_t gb, int32_t d, int32_t k, int32_t m)
{
	const BwShm &sh = bw_sh();
#pragma unroll 1
	for (int guard = 0; k < m && guard < (1 << 28); ++guard) {
		const uint64_t x = window8<true>(sh.graw, (int64_t)gb + k + 1) ^ window8<false>(sh.qraw, (int64_t)d + k + 1);
		if (x == 0) {
			k += 8;
			continue;
		}
		k += __ffsll((long long)x) - 1 >> 3;
		break;
	}
	return k;
}
__device__ __forceinline__ int32_t bw_ext(const BwShm &sh, uint32_t gb, int32_t d, int32_t k, int32_t vl, bool on)
{
	const int32_t m = min(sh.ql - d, vl) - 1;
	bool more = on && k < m && !(k < 0 && m < 31 && sh.quirk);
	if (sh.packed) {
		const uint32_t *const gp = sh.gpk, *const qp = (const uint32_t *)sh.qpk;
#pragma unroll 1
		while (__any_sync(FULL, more)) {
			if (more) {
				const uint32_t gx = gb + k + 1, qx = d + k + 1;
				const uint32_t *const gw = gp + (gx >> 4), *const qw = qp + (qx >> 4);
				const uint32_t g0 = __ldg(gw), g1 = __ldg(gw + 1), g2 = __ldg(gw + 2), q0 = qw[0], q1 = qw[1], q2 = qw[2];
				const uint32_t gs = 2 * gx, qs = 2 * qx;
				const uint32_t lo = __funnelshift_r(g0, g1, gs & 30) ^ __funnelshift_r(q0, q1, qs & 30);
				const uint32_t hi = __funnelshift_r(g1, g2, gs & 30) ^ __funnelshift_r(q1, q2, qs & 30);
				const int32_t a = __clz(__brev(lo)) >> 1, b = __clz(__brev(hi)) >> 1; // 16 where all are equal
				const int32_t n = a < 16 ? a : 16 + b;
				k += n;
				more = n == 32 && k < m;
			}
		}
	} else if (more)
		k = bw_ext_raw(gb, d, k, m);
	return min(k, m); // lanes that are on
}

// Hash table of the blocks: linear probing over slots of (tag, id).
__device__ __forceinline__ uint32_t bw_tag(uint32_t v, int32_t bi)
{
	uint32_t x = v * 0x9E3779B1u + (uint32_t)bi * 0x85EBCA6Bu;
	x ^= x >> 15;
	return x * 0x2C1B3C6Du;
}

__device__ __forceinline__ uint2 bw_slot_load(const uint2 *p)
{
	unsigned long long v;
	asm volatile("ld.relaxed.cta.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
	return make_uint2((uint32_t)v, (uint32_t)(v >> 32));
}
constexpr uint32_t BW_BUSY = 0xfffffffeu; // MW: a slot whose block is being made

// Block bi (diagonals 8 bi .. 8 bi + 7) of vertex v, made where it is missing (the whole warp calls
// it; on: this lane asks). Of a warp's lanes that want one empty slot the first makes its block; MW:
// it claims the slot by compare-and-swap, and lanes of other warps that want the same tag look again
// until it is published (the maker never waits in between; the tries are bounded). Sets ovf when the
// pool is full. gb, vl: the vertex's first base and length.
template <bool MW>
static __device__ __noinline__ int32_t bw_get(bool on, uint32_t v, int32_t bi, uint32_t gb, int32_t vl)
{
	BwShm &sh = bw_sh();
	const int lane = threadIdx.x & 31;
	BwBlock *const blk = sh.blk;
	uint2 *const hash = sh.hash;
	const uint32_t hmask = sh.hmask;
	int32_t id = on ? -1 : 0;
	bool made = false;
	uint32_t tag = bw_tag(v, bi), sl = (tag ^ tag >> 16) & hmask;
	int32_t n_blk = MW ? 0 : sh.n_blk;
#pragma unroll 1
	for (uint32_t guard = 0; guard <= hmask + (1u << 16); ++guard) {
		bool want = false;
		if (id < 0) {
			const uint2 e = MW ? bw_slot_load(hash + sl) : hash[sl];
			want = e.y == 0xffffffffu;
			if (!want) {
				const bool busy = MW && e.y == BW_BUSY;
				if (!busy && e.x == tag && blk[e.y].v == v && blk[e.y].db == 8 * bi) id = (int32_t)e.y;
				else if (!busy || e.x != tag) sl = sl + 1 & hmask;
			}
		}
		if (__any_sync(FULL, want)) {
			const uint32_t same = __match_any_sync(FULL, want ? (int32_t)sl : -1 - lane);
			bool won = want && (same & lanemask_lt()) == 0;
			int32_t at = 0;
			if constexpr (MW) {
				if (won)
					won = atomicCAS((unsigned long long *)(hash + sl), ~0ULL,
					                (unsigned long long)BW_BUSY << 32 | tag) == ~0ULL;
				if (won) at = atomicAdd(&sh.n_blk, 1);
				if (won && at >= sh.nb) { // full: the claimed slot goes back
					atomicExch((unsigned long long *)(hash + sl), ~0ULL);
					won = false;
					sh.ovf = 1;
				}
				if (__any_sync(FULL, sh.ovf != 0)) {
					if (won) sh.slot[at] = sl, atomicExch((unsigned long long *)(hash + sl), (unsigned long long)at << 32 | tag);
					sh.ovf = 1;
					break;
				}
			} else {
				const uint32_t m = __ballot_sync(FULL, won);
				if (n_blk + __popc(m) > sh.nb) {
					sh.ovf = 1;
					break;
				}
				at = n_blk + __popc(m & lanemask_lt());
				n_blk += __popc(m);
			}
			if (won) {
				id = at;
				int4 *q = (int4 *)(blk + id);
				q[1] = make_int4(vl, -1, -1, 0);
				const int4 none = make_int4(BW_NONE, BW_NONE, BW_NONE, BW_NONE);
				const int4 nonec = make_int4(BwBits<MW>::none, BwBits<MW>::none, BwBits<MW>::none, BwBits<MW>::none);
				q[2] = none, q[3] = none, q[4] = none, q[5] = none, q[6] = nonec, q[7] = nonec;
				q[0] = make_int4((int)gb, (int)__ldg(sh.varcs + v), (int)v, 8 * bi);
				sh.slot[id] = sl;
				made = true;
				if constexpr (MW) {
					__threadfence_block(); // the block before its id
					atomicExch((unsigned long long *)(hash + sl), (unsigned long long)(uint32_t)id << 32 | tag);
				} else
					hash[sl] = make_uint2(tag, (uint32_t)id);
			}
			__syncwarp();
		}
		if (!__any_sync(FULL, id < 0)) break;
		if (MW && guard == hmask + (1u << 16)) sh.ovf = 1; // not reached: a maker publishes at once
	}
	if constexpr (!MW) sh.n_blk = n_blk;
	if (__any_sync(FULL, made)) {
		// links to the neighbours that exist (MW: of two neighbours made at once, the one that is
		// published last finds the other)
		if constexpr (MW) __threadfence_block();
#pragma unroll 1
		for (int side = -1; made && side <= 1; side += 2) {
			tag = bw_tag(v, bi + side), sl = (tag ^ tag >> 16) & hmask;
#pragma unroll 1
			for (uint32_t guard = 0; guard <= hmask; ++guard) {
				const uint2 e = MW ? bw_slot_load(hash + sl) : hash[sl];
				if (e.y == 0xffffffffu) break;
				if (!(MW && e.y == BW_BUSY)) {
					BwBlock *const B = blk + e.y;
					if (e.x == tag && B->v == v && B->db == 8 * (bi + side)) {
						*(side < 0 ? &blk[id].left : &blk[id].right) = (int32_t)e.y;
						*(side < 0 ? &B->right : &B->left) = id;
						break;
					}
				}
				sl = sl + 1 & hmask;
			}
		}
	}
	__syncwarp();
	return max(id, 0);
}

// Puts block id into the next live list, once (several lanes may name one block), and flags its
// candidates where they have some (has_c). np: the parity of the next step.
template <bool MW>
static __device__ __noinline__ void bw_push(bool on, int32_t id, int np, bool has_c)
{
	BwShm &sh = bw_sh();
	uint32_t *const f = &sh.blk[id].flags;
	bool app;
	if constexpr (MW) {
		const uint32_t bit = BwBits<MW>::inl(np);
		app = on && !(atomicOr(f, bit | (has_c ? BwBits<MW>::has_c : 0u)) & bit);
	} else {
		if (on && has_c) ((uint8_t *)f)[1] = 1;
		const uint32_t same = __match_any_sync(FULL, on ? id : -1 - (int)(threadIdx.x & 31));
		uint8_t *const in = (uint8_t *)f + 2 + np;
		app = on && (same & lanemask_lt()) == 0 && !*in;
		if (app) *in = 1;
	}
	const uint32_t m = __ballot_sync(FULL, app);
	if (m) {
		const int32_t at = bw_append<MW>(&sh.n_nxt, m);
		if (app) sh.nxt[at] = id;
	}
	__syncwarp();
}

// Arc-side candidate k for a cell (lanes of a warp that meet on one cell bring the same k)
template <bool MW>
__device__ __forceinline__ void bw_raise(int32_t *c, int32_t k)
{
	if constexpr (MW) atomicMax(c, k);
	else {
		const int32_t c0 = *c;
		if (c0 >> 1 < k) *c = k << 1 | (c0 & 1);
	}
}

// Arc-side candidate k for diagonal d of vertex v at the next step
template <bool MW>
static __device__ __noinline__ void bw_cand(bool on, uint32_t v, int32_t d, uint32_t gb, int32_t vl, int32_t k, int np)
{
	BwShm &sh = bw_sh();
	const int32_t id = bw_get<MW>(on, v, d >> 3, gb, vl);
	if (__any_sync(FULL, sh.ovf != 0)) return;
	if (on) bw_raise<MW>(sh.blk[id].c + (d & 7), k);
	bw_push<MW>(on, id, np, true);
}

// A live edge diagonal (act: block id, cell l) gives the neighbouring block a candidate at the next
// step: lists the neighbour, made where it is missing.
template <bool MW>
static __device__ __noinline__ void bw_side(bool act, int32_t id, int32_t l, int np)
{
	BwShm &sh = bw_sh();
	__syncwarp();
	const BwBlock *const B = sh.blk + id;
	const int32_t t = l == 0 ? B->left : B->right;
	const bool miss = act && t < 0;
	int32_t u = t;
	if (__any_sync(FULL, miss)) {
		const int32_t w = bw_get<MW>(miss, B->v, (B->db >> 3) + (l == 0 ? -1 : 1), B->gb, B->vl);
		if (__any_sync(FULL, sh.ovf != 0)) return;
		if (miss) u = w;
	}
	bw_push<MW>(act, act ? u : 0, np, false);
}

// Successors of the live blocks of the list cur (n_cur entries), two lanes per block and four
// diagonals per lane, until the warp's queue (n_q entries) holds 32 diagonals that may live or the
// list is empty. Blocks that stay go to the next list. kmin: the least offset of a candidate.
// Returns (1 = the list may hold more, n_q).
template <bool MW>
static __device__ __noinline__ int2 bw_fill(const int32_t *cur, int32_t n_cur, int32_t n_q, int par, int32_t kmin)
{
	BwShm &sh = bw_sh();
	uint2 *const queue = bw_queue();
	const int lane = threadIdx.x & 31, np = par ^ 1, hf = lane & 1;
#pragma unroll 1
	while (n_q < 32) {
		int32_t base;
		if constexpr (MW) {
			base = 0;
			if (lane == 0) base = atomicAdd(&sh.next, 16);
			base = __shfl_sync(FULL, base, 0);
		} else {
			base = sh.next;
			__syncwarp();
			sh.next = base + 16;
		}
		if (base >= n_cur) return make_int2(0, n_q);
		const bool in = base + (lane >> 1) < n_cur;
		const int32_t bid = cur[in ? base + (lane >> 1) : base];
		BwBlock *const B = sh.blk + bid;
		const int4 h1 = *((const int4 *)B + 1);
		const int32_t nid = hf ? h1.z : h1.y; // the neighbour at this lane's side
		const uint32_t fl = (uint32_t)h1.w;   // ended, has_c, inl[0], inl[1]
		const int4 kk = *((const int4 *)B->row[np] + hf);
		int32_t ek = BW_NONE;
		if (nid >= 0) ek = sh.blk[nid].row[np][hf ? 0 : 7];
		const int32_t ok = __shfl_xor_sync(FULL, hf ? kk.x : kk.w, 1);
		const int32_t lf = hf ? ok : ek, rt = hf ? ek : ok;
		int32_t kq[4] = {max(lf, max(kk.x, kk.y) + 1), max(kk.x, max(kk.y, kk.z) + 1),
		                 max(kk.y, max(kk.z, kk.w) + 1), max(kk.z, max(kk.w, rt) + 1)};
		if (__any_sync(FULL, (fl & BwBits<MW>::clear_c) != 0)) {
			int4 *const cp = (int4 *)B->c + hf;
			const int4 c = *cp;
			__syncwarp();
			typedef BwBits<MW> X;
			kq[0] = max(kq[0], X::k(c.x)), kq[1] = max(kq[1], X::k(c.y));
			kq[2] = max(kq[2], X::k(c.z)), kq[3] = max(kq[3], X::k(c.w));
			if (in) *cp = make_int4(X::taken(c.x), X::taken(c.y), X::taken(c.z), X::taken(c.w));
		}
		uint32_t en = 0, up = 0;
#pragma unroll
		for (int q = 0; q < 4; ++q) {
			en |= (uint32_t)(kq[q] >= h1.x) << q;
			up |= (uint32_t)(kq[q] >= kmin) << q;
		}
		up &= in ? ~(en | fl >> (4 * hf)) & 15u : 0u;
		// the block stays listed while it has, or just lost, live diagonals (a block that leaves has
		// both rows empty)
		const bool stays = up != 0 || (in && max(max(kk.x, kk.y), max(kk.z, kk.w)) > BW_NONE);
		const uint32_t w = en << (4 * hf) | (stays ? 0x100u : 0u);
		const uint32_t w2 = w | __shfl_xor_sync(FULL, w, 1);
		const uint32_t inb = BwBits<MW>::inl(np);
		const bool first = hf == 0 && in;
		bool app = first && (w2 & 0x100) && !(fl & inb);
		if (in) *((int4 *)B->row[par] + hf) = make_int4(BW_NONE, BW_NONE, BW_NONE, BW_NONE);
		if constexpr (MW) { // other warps may list the block meanwhile
			if (first) atomicAnd(&B->flags, ~BwBits<MW>::drop(par));
			if (first && (app || (w2 & 0xff & ~fl))) app = !(atomicOr(&B->flags, (w2 & 0xff) | (app ? inb : 0)) & inb) && app;
		} else if (first)
			B->flags = (fl & ~BwBits<MW>::drop(par)) | (w2 & 0xff) | (app ? inb : 0);
		const uint32_t mp = __ballot_sync(FULL, app);
		const int32_t at = bw_append<MW>(&sh.n_nxt, mp);
		if (app) sh.nxt[at] = bid;
		// side: an edge diagonal whose neighbour has no live diagonal beside it
		const uint32_t tag = (uint32_t)bid << 4 | (uint32_t)hf << 2, sq = ek > BW_NONE ? 0u : hf ? 8u : 1u;
#pragma unroll
		for (int q = 0; q < 4; ++q) {
			const bool on = up >> q & 1;
			const uint32_t m = __ballot_sync(FULL, on);
			if (on) queue[n_q + __popc(m & lanemask_lt())] = make_uint2(tag | q | ((sq >> q & 1) << 3), (uint32_t)kq[q]);
			n_q += __popc(m);
		}
		__syncwarp();
	}
	return make_int2(1, n_q);
}

// Step 1 for up to four blocks, by one warp: one lane per diagonal, and step after step in registers
// until one reaches its vertex's end or the query's, none lives, or a live edge diagonal has its
// neighbour outside the four blocks (unlisted blocks have no live diagonals).
template <bool MW>
__device__ __forceinline__ void bw_narrow(const int32_t *cur, int32_t n_cur, int32_t *list0, int32_t *list1, int32_t T,
                                              bool lag, int32_t max_steps)
{
	BwShm &sh = bw_sh();
	const int lane = threadIdx.x & 31, gr = lane >> 3, l = lane & 7;
	const int32_t ql = sh.ql, kmin1 = sh.quirk ? 0 : -1;
	const int32_t user = sh.lag;
	int32_t s = sh.s, imin = sh.imin;
	const bool has = gr < n_cur;
	const int32_t id = cur[has ? gr : 0];
	BwBlock *const B = sh.blk + id;
	const int4 b0 = *(const int4 *)B, h1 = *((const int4 *)B + 1); // gb, arcs, v, db; vl, left, right, flags
	int32_t k = has ? B->row[~s & 1][l] : BW_NONE;
	const uint32_t fl = (uint32_t)h1.w; // ended, has_c, inl[0], inl[1]
	const bool edge = (0x81 >> l & 1) != 0;
	const int32_t nid = l == 0 ? h1.y : h1.z, vl = h1.x, d = b0.w + l;
	int src = -1; // edge lanes: the lane of the diagonal across
#pragma unroll
	for (int j = 0; j < 4; ++j)
		if (__shfl_sync(FULL, id, 8 * j) == nid && j < n_cur && edge) src = 8 * j + 7 - l;
	const bool out = edge && src < 0, nu = l == 0 && out, nd = l == 7 && out;
	const int su = l == 0 ? max(src, 0) : lane - 1, sd = l == 7 ? max(src, 0) : lane + 1;
	bool dead = !has || (fl >> l & 1); // absent, or past the vertex end
	int32_t c = BW_NONE;               // the first step's arc-side candidates
	if (__any_sync(FULL, has && (fl & BwBits<MW>::clear_c))) {
		const int32_t cw = B->c[l];
		__syncwarp();
		if (has) c = BwBits<MW>::k(cw), B->c[l] = BwBits<MW>::taken(cw);
	}
	int32_t i;
	bool live, qend, vend;
	auto successor = [&]() {
		const int32_t up = __shfl_sync(FULL, k, su), dn = __shfl_sync(FULL, k, sd);
		return max(nu ? BW_NONE : up, max(k, nd ? BW_NONE : dn) + 1);
	};
	k = max(successor(), c);
	dead |= k >= vl; // later steps follow no vertex end
	live = !dead && k >= (s == 0 ? -1 : kmin1);
#pragma unroll 1
	for (;;) {
		if (user) imin = max(__reduce_max_sync(FULL, live ? d + k : INT32_MIN), INT32_MIN / 2) - user;
		const int32_t hv = sh.h[live ? ql - 1 - d - k : 0]; // any value below BW_INF while T is BW_INF
		live = live && s + hv < T && d + k >= imin;
		k = bw_ext(sh, (uint32_t)b0.x, d, k, vl, live);
		if (!live) k = BW_NONE;
		i = live ? d + k : INT32_MIN;
		qend = i == ql - 1, vend = live && k == vl - 1 && !qend;
		const bool stop = qend || vend || (live && out) || s + 1 >= max_steps;
		if (__any_sync(FULL, stop) || !__any_sync(FULL, live)) break;
		if (lag) imin = __reduce_max_sync(FULL, i) - kPruneLag;
		++s;
		k = successor();
		live = !dead && k >= kmin1;
	}
	const int par = s & 1, np = par ^ 1;
	// back to the blocks: both rows, the ended diagonals, the next list
	const uint32_t em = (__ballot_sync(FULL, has && dead) >> (8 * gr)) & 0xff;
	const uint32_t ml = __ballot_sync(FULL, live);
	if (has) B->row[par][l] = k, B->row[np][l] = BW_NONE;
	const bool first = l == 0 && has, app = first && (ml >> (8 * gr) & 0xff) != 0;
	if (first) B->flags = (MW ? fl & 0xff00u : 0u) | em | (app ? BwBits<MW>::inl(np) : 0u); // MW: the cells reached stay
	const uint32_t mp = __ballot_sync(FULL, app);
	int32_t *const nxt = par ? list0 : list1; // the list at hand is in registers
	if (app) nxt[__popc(mp & lanemask_lt())] = id;
	const uint32_t me = __ballot_sync(FULL, vend);
	if (vend) sh.e[__popc(me & lanemask_lt())] = (uint32_t)id << 3 | l;
	const int32_t far = __reduce_max_sync(FULL, i);
	const bool any_q = __any_sync(FULL, qend);
	__syncwarp();
	sh.s = s, sh.imin = imin, sh.nxt = nxt, sh.n_nxt = __popc(mp), sh.n_e = __popc(me), sh.far = far;
	sh.found = any_q, sh.any = ml != 0;
	__syncwarp();
	// a live edge diagonal gives the neighbouring block a candidate at the next step
	const bool act = live && edge && (src < 0 || (ml >> (src & 24) & 0xff) == 0);
	if (__any_sync(FULL, act)) bw_side<MW>(act, id, l, np);
}

// The furthest query position of a candidate of this step (the caller's lag pruning,
// gwf-ed.cu:1286-1287, drops what lags it by more than max_lag), as bw_fill forms them, into far_c.
template <bool MW>
static __device__ __noinline__ void bw_far(const int32_t *cur, int32_t n_cur, int par, int32_t kmin)
{
	BwShm &sh = bw_sh();
	const int lane = threadIdx.x & 31, np = par ^ 1, l = lane & 7;
	const int32_t wid = MW ? threadIdx.x >> 5 : 0, nw = MW ? blockDim.x >> 5 : 1;
	int32_t far = INT32_MIN / 2;
#pragma unroll 1
	for (int32_t base = 4 * wid; base < n_cur; base += 4 * nw) { // a lane per diagonal
		const bool in = base + (lane >> 3) < n_cur;
		const BwBlock *const B = sh.blk + cur[in ? base + (lane >> 3) : base];
		const int32_t nid = l == 0 ? B->left : B->right, kk = B->row[np][l];
		int32_t up = __shfl_up_sync(FULL, kk, 1), dn = __shfl_down_sync(FULL, kk, 1), ek = BW_NONE;
		if ((l == 0 || l == 7) && nid >= 0) ek = sh.blk[nid].row[np][7 - l];
		if (l == 0) up = ek;
		if (l == 7) dn = ek;
		const int32_t k = max(max(up, max(kk, dn) + 1), BwBits<MW>::k(B->c[l]));
		if (in && k >= kmin && k < B->vl && !(B->flags >> l & 1)) far = max(far, B->db + l + k);
	}
	far = __reduce_max_sync(FULL, far);
	if constexpr (MW) {
		if (lane == 0) atomicMax(&sh.far_c, far);
		__syncthreads();
	} else
		sh.far_c = far;
	__syncwarp();
}

// Step 1 for more blocks: bw_fill's diagonals through the warp's queue, so that the extension runs on
// full warps (of a dense graph's diagonals in live blocks one in four lives).
template <bool MW>
__device__ __forceinline__ void bw_wide(const int32_t *cur, int32_t n_cur, int32_t T)
{
	BwShm &sh = bw_sh();
	const uint2 *const queue = bw_queue();
	const int lane = threadIdx.x & 31;
	const int32_t ql = sh.ql, s = sh.s, ne = sh.nb;
	const int par = s & 1;
	int32_t imin = sh.imin;
	if (sh.lag) {
		bw_far<MW>(cur, n_cur, par, s == 0 || !sh.quirk ? -1 : 0);
		imin = sh.far_c - sh.lag;
	}
	bool found = false, any = false;
	int32_t far = INT32_MIN;
	int2 at = make_int2(1, 0); // more blocks, queued diagonals
#pragma unroll 1
	do {
		if (at.x && at.y < 32) at = bw_fill<MW>(cur, n_cur, at.y, par, s == 0 || !sh.quirk ? -1 : 0);
		const int32_t take = min(at.y, 32); // from the queue's end
		at.y -= take;
		const bool alive = lane < take;
		const uint2 e = queue[at.y + (alive ? lane : 0)];
		const int32_t id = alive ? (int32_t)(e.x >> 4) : 0, l = (int32_t)(e.x & 7);
		int32_t k = (int32_t)e.y;
		BwBlock *const B = sh.blk + id;
		const int4 b0 = *(const int4 *)B;
		const int32_t vl = B->vl, d = b0.w + l;
		const int32_t hv = sh.h[alive ? ql - 1 - d - k : 0];
		const bool live = alive && s + hv < T && d + k >= imin;
		k = bw_ext(sh, (uint32_t)b0.x, d, k, vl, live);
		if (live) B->row[par][l] = k;
		const int32_t i = live ? d + k : INT32_MIN;
		far = max(far, i);
		const bool qend = i == ql - 1, vend = live && k == vl - 1 && !qend;
		found |= qend;
		any |= live;
		const uint32_t me = __ballot_sync(FULL, vend);
		if (me) {
			const int32_t pos = bw_append<MW>(&sh.n_e, me);
			if (vend && pos < ne) sh.e[pos] = (uint32_t)id << 3 | l;
		}
		// a neighbour whose diagonal beside it was live stays listed by itself
		const bool act = live && (e.x & 8);
		if (__any_sync(FULL, act)) {
			bw_side<MW>(act, id, l, par ^ 1);
			if (__any_sync(FULL, sh.ovf != 0)) break;
		}
	} while (at.x || at.y > 0);
	found = __any_sync(FULL, found), any = __any_sync(FULL, any);
	far = __reduce_max_sync(FULL, far);
	if (lane == 0) {
		if (found) sh.found = 1;
		if (any) sh.any = 1;
		if constexpr (MW) atomicMax(&sh.far, far);
		else sh.far = far;
	}
	__syncwarp();
}

// Inlined into the one-warp kernel (100,000 x 1 kbp: 14.3 -> 13.4 ms when this was taken); out of line
// with several warps, whose time is that of one read (20 kbp at 10%: 84.7 against 88.7 ms inlined)
static __device__ __noinline__ void bw_narrow_mw(const int32_t *cur, int32_t n_cur, int32_t *list0, int32_t *list1,
                                                 int32_t T, bool lag, int32_t max_steps)
{
	bw_narrow<true>(cur, n_cur, list0, list1, T, lag, max_steps);
}
static __device__ __noinline__ void bw_wide_mw(const int32_t *cur, int32_t n_cur, int32_t T)
{
	bw_wide<true>(cur, n_cur, T);
}

// Step 2: the vertex-end states of e over their arcs, in waves, until no state is entered with a
// free match (gwf-ed.cu:1106-1255). Four lanes per state, one arc each. Begins and ends at a
// barrier.
template <bool MW>
static __device__ __noinline__ void bw_waves(int32_t T)
{
	BwShm &sh = bw_sh();
	const int lane = threadIdx.x & 31;
	const int32_t wid = MW ? threadIdx.x >> 5 : 0, nw = MW ? blockDim.x >> 5 : 1;
	const int32_t ql = sh.ql, ne = sh.nb, s = sh.s;
	const int np = ~s & 1;
	BwBlock *const blk = sh.blk;
	int32_t far = INT32_MIN, n_e = sh.n_e;
	bw_bar<MW>(); // every warp has read the flags of step 1 before one is set here
#pragma unroll 1
	for (int32_t wave = 0; n_e > 0; ++wave) {
		const uint32_t *const E = wave & 1 ? sh.f : sh.e;
		uint32_t *const F = wave & 1 ? sh.e : sh.f;
#pragma unroll 1
		for (int32_t base = 8 * wid; base < n_e; base += 8 * nw) {
			const bool act = base + (lane >> 2) < n_e;
			const uint32_t e = E[act ? base + (lane >> 2) : 0];
			const int32_t id = (int32_t)(e >> 3), cl = (int32_t)(e & 7);
			const int4 b0 = *(const int4 *)(blk + id); // gb, arcs, v, db
			const int32_t vl = blk[id].vl, i = b0.w + cl + vl - 1;
			const uint32_t aoff = (uint32_t)b0.y & kVArcsMask;
			uint32_t deg = (uint32_t)b0.y >> kVArcsBits, n_ext = 0;
			if (deg == kVArcsMany) deg = __ldg(sh.arc_off + b0.z + 1) - aoff;
			if (!act) deg = 0;
			const uint32_t qc = (uint32_t)(sh.qpk[(i + 1) >> 5] >> (2 * ((i + 1) & 31))) & 3;
			// least scores of a path through the deletion into an arc's target and the mismatch
			const int32_t ha = s + 1 + (int32_t)sh.h[ql - 1 - i], hb = s + 1 + (int32_t)sh.h[ql - 2 - i];
			const uint32_t max_deg = __reduce_max_sync(FULL, deg);
			bool full = false;
#pragma unroll 1
			for (uint32_t t0 = lane & 3; t0 < max_deg + (lane & 3); t0 += 4) {
				const bool has = t0 < deg;
				uint4 a = make_uint4(0, 0, 0, 0);
				if (has) a = __ldg(sh.arcx + aoff + t0);
				const uint32_t w = a.x;
				const int32_t ol = (int32_t)(a.y & 0x3fffffff), dd = i + 1 - ol;
				const bool eq = has && (sh.packed ? a.y >> 30 == qc : __ldg(sh.graw + a.z + ol) == sh.qraw[i + 1]);
				n_ext += __popc(__ballot_sync(FULL, eq) >> (lane & 28) & 15);
				// arrival key 0 is never new (gwf-ed.cu:1022-1026); a state that the bound drops leaves
				// no mark: later arrivals are dropped too
				const bool on = has && !(w == 0 && i == -1) && (eq ? hb - 1 : hb) < T;
				if (!__any_sync(FULL, on)) continue;
				const int32_t id2 = bw_get<MW>(on, w, dd >> 3, a.z, (int32_t)a.w);
				if ((full = __any_sync(FULL, sh.ovf != 0))) break;
				BwBlock *const B = blk + id2;
				const int cell = dd & 7;
				bool neu, enter, two;
				if constexpr (MW) { // of several lanes one sets the cell's bit; a mismatch lists the block
					const uint32_t inb = BwBits<MW>::inl(np);
					uint32_t was = inb;
					if (on) was = atomicOr(&B->flags, 0x100u << cell | (eq ? 0u : inb | BwBits<MW>::has_c));
					neu = on && !(was >> (8 + cell) & 1);
					enter = neu && eq, two = neu && !eq;
					if (two) atomicMax(B->c + cell, ol);
					const bool app = on && !eq && !(was & inb);
					const uint32_t ma = __ballot_sync(FULL, app);
					if (ma) {
						const int32_t at = bw_append<MW>(&sh.n_nxt, ma);
						if (app) sh.nxt[at] = id2;
					}
				} else {
					int32_t *const cp = B->c + cell;
					const int32_t cw = *cp;
					neu = on && !(cw & 1);
					const uint32_t same = __match_any_sync(FULL, neu ? (id2 << 3 | cell) : -1 - lane);
					neu = neu && (same & lanemask_lt()) == 0;
					enter = neu && eq, two = neu && !eq;
					if (neu) *cp = (two ? max(cw >> 1, ol) : cw >> 1) << 1 | 1;
				}
				const uint32_t mn = __ballot_sync(FULL, enter);
				if (mn) {
					const int32_t pn = bw_append<MW>(&sh.n_n[wave & 1], mn);
					if (enter && pn < ne) sh.n[pn] = (uint32_t)id2 << 3 | cell, sh.nk[pn] = ol;
				}
				__syncwarp();
				if (__any_sync(FULL, two)) {
					// the deletion: one diagonal below, most often in the same block
					const bool del = two && ha < T, lo = del && cell == 0;
					if (del && !lo) bw_raise<MW>(B->c + cell - 1, ol);
					if constexpr (!MW) bw_push<MW>(two, id2, np, true);
					if (__any_sync(FULL, lo)) {
						bw_cand<MW>(lo, w, dd - 1, a.z, (int32_t)a.w, ol, np);
						if ((full = __any_sync(FULL, sh.ovf != 0))) break;
					}
				}
			}
			// entered states that reached the vertex end: the diagonal has ended (gwf-ed.cu:1177-1183),
			// and the insertion at the vertex end stays where an arc did not match
			// (gwf-ed.cu:1225-1226). For the states of step 1 the successor rule does both.
			if (wave > 0 && !full) {
				const bool one = act && (lane & 3) == 0, ins = one && (n_ext != deg || deg == 0), hi = ins && cl == 7;
				if (one) {
					if constexpr (MW) atomicMax(blk[id].c + cl, BW_ENDED);
					else blk[id].c[cl] = BW_ENDED << 1 | 1;
				}
				__syncwarp();
				if (ins && !hi) bw_raise<MW>(blk[id].c + cl + 1, vl - 1);
				bw_push<MW>(one, id, np, true);
				if (__any_sync(FULL, hi))
					bw_cand<MW>(hi, (uint32_t)b0.z, i - vl + 2, (uint32_t)b0.x, vl, vl - 1, np);
			}
			if (__any_sync(FULL, sh.ovf != 0)) break;
		}
		bw_bar<MW>();
		const int32_t n_n = sh.n_n[wave & 1];
		if (threadIdx.x == 0) { // the other parity's counters: read before the barrier above
			sh.n_n[~wave & 1] = 0, sh.n_f[~wave & 1] = 0;
			if (n_n > ne || wave > ql + 2) sh.ovf = 1;
		}
		// extension of the entered states (gwf-ed.cu:1132-1160): one that stays inside its vertex
		// joins the step's row, whose successors are its three candidates
#pragma unroll 1
		for (int32_t base = 32 * wid; base < n_n && n_n <= ne; base += 32 * nw) {
			const bool act = base + lane < n_n;
			const int32_t j = act ? base + lane : 0;
			const uint32_t e = sh.n[j];
			const int32_t id = (int32_t)(e >> 3), cl = (int32_t)(e & 7);
			BwBlock *const B = blk + id;
			const int32_t vl = B->vl, d = B->db + cl;
			const int32_t k = bw_ext(sh, B->gb, d, sh.nk[j], vl, act);
			const int32_t i = act ? d + k : INT32_MIN;
			far = max(far, i);
			const bool qend = i == ql - 1, in = act && !qend && k + 1 < vl, toF = act && !qend && !in;
			if (qend) sh.found = 1;
			if (in && B->row[np ^ 1][cl] < k) B->row[np ^ 1][cl] = k;
			const uint32_t mf = __ballot_sync(FULL, toF);
			if (mf) {
				const int32_t pf = bw_append<MW>(&sh.n_f[wave & 1], mf); // n_f <= n_n <= ne
				if (toF) F[pf] = (uint32_t)id << 3 | cl;
			}
			if (__any_sync(FULL, in)) {
				bw_push<MW>(in, id, np, false);
				const bool eb = in && (cl == 0 || cl == 7);
				if (__any_sync(FULL, eb)) bw_side<MW>(eb, id, cl, np);
			}
		}
		bw_bar<MW>();
		n_e = sh.n_f[wave & 1];
		const bool stop = sh.found || sh.ovf;
		bw_bar<MW>(); // every warp has read them before the next wave sets them
		if (stop) break;
	}
	far = __reduce_max_sync(FULL, far);
	if (lane == 0) {
		if constexpr (MW) atomicMax(&sh.far, far);
		else sh.far = max(sh.far, far);
	}
	bw_bar<MW>();
}

// Aligns read r with the CTA in the arena wsb laid out by p.bw; the hash table is empty on entry and
// on return. All control flow is uniform over the CTA between barriers.
template <bool MW>
__device__ __forceinline__ void align_read_blocks(const KParams &p, int32_t r, uint8_t *wsb)
{
	BwShm &sh = bw_sh();
	const int lane = threadIdx.x & 31;
	const bool lead = threadIdx.x == 0, warp0 = !MW || threadIdx.x < 32;
	const DevGraph &g = p.g;
	const int32_t ql = p.r.ql[r], v0 = p.r.v0[r];
	if (ql <= 0 || v0 < 0 || (uint32_t)v0 >= g.n_vtx) {
		if (lead) p.dist[r] = -1, p.status[r] = ST_BAD_INPUT;
		return;
	}
	int32_t *const list0 = (int32_t *)(wsb + p.bw.list0), *const list1 = (int32_t *)(wsb + p.bw.list1);
	if (lead) {
		sh.qpk = p.r.pk + p.r.pk_off[r], sh.qraw = p.r.raw + p.r.raw_off[r];
		sh.ql = ql, sh.packed = g.pure && p.r.pure[r], sh.quirk = !(p.flags & 1), sh.lag = p.max_lag;
	}
	bw_bar<MW>();
	const int32_t max_steps = (ql < 64 ? 64 : ql) * 4 + 1024;

	int32_t dist = -1, st = ST_OK, steps = 0;
	int32_t T = BW_INF;    // states with s + h >= T are dropped
	bool attained = false; // an alignment of T edits exists
	bool lag = false;      // the run that looks for such a T
	int32_t h0 = 0;
	if (g.bloom && ql >= kPruneMinQl && p.max_lag == 0) {
		h0 = bw_seeds<MW>(g.bloom_k);
		// nearly all windows at their largest cost: the read is unlike the graph, and no bound helps
		lag = (float)h0 < 1.7f * (float)(ql / g.bloom_k);
		if (!lag && p.defer) { // such a read makes thousands of states per step: left to a group of warps
			if (lead) {
				p.dist[r] = -1, p.status[r] = p.retry_list ? ST_CAPACITY : ST_UNLIKE;
				if (p.retry_list) p.retry_list[atomicAdd(p.retry_n, 1)] = ~r;
			}
			return;
		}
	}
#pragma unroll 1
	for (;;) { // runs of the score loop
		if (lead) sh.n_blk = 0, sh.ovf = 0, sh.s = 0, sh.imin = INT32_MIN;
		__syncwarp();
		if (warp0) {
			bw_get<MW>(lane == 0, (uint32_t)v0, 0, (uint32_t)__ldg(g.base + v0), (int32_t)__ldg(g.len + v0));
			// the start state (v0, 0), k = -1, as an arc-side candidate (gwf-ed.cu:1303-1308)
			if (lane == 0) {
				sh.blk[0].c[0] = MW ? -1 : -2;
				sh.blk[0].flags = BwBits<MW>::has_c | BwBits<MW>::inl(0);
				list0[0] = 0;
			}
		}
		const int32_t *cur = list0;
		int32_t n_cur = 1, s = 0;
		int32_t sc = -1; // the run's score
		bool ovf = false;
#pragma unroll 1
		for (;;) {
			if (lead) {
				sh.nxt = s & 1 ? list0 : list1;
				sh.n_nxt = 0, sh.n_e = 0, sh.next = 0, sh.any = 0, sh.found = 0, sh.far = INT32_MIN;
				sh.n_n[0] = 0, sh.n_f[0] = 0, sh.far_c = INT32_MIN / 2;
			}
			bw_bar<MW>();
			if (s >= max_steps) {
				ovf = true;
				break;
			}
			// ---- 1. successors and extension of the live blocks (may go on to a later step)
			if constexpr (MW) {
				if (n_cur > 4) bw_wide_mw(cur, n_cur, T);
				else if (warp0) bw_narrow_mw(cur, n_cur, list0, list1, T, lag, max_steps);
			} else if (n_cur > 4)
				bw_wide<MW>(cur, n_cur, T);
			else
				bw_narrow<MW>(cur, n_cur, list0, list1, T, lag, max_steps);
			bw_bar<MW>();
			s = sh.s;
			if (sh.found) {
				sc = s;
				break;
			}
			if (!sh.any) break; // no state is left
			// ---- 2. vertex-end states over arcs
			ovf = sh.ovf || sh.n_e > sh.nb;
			if (ovf) break;
			if (sh.n_e > 0) {
				bw_waves<MW>(T);
				if (sh.found) {
					sc = s;
					break;
				}
				ovf = sh.ovf != 0;
				if (ovf) break;
			}
			n_cur = sh.n_nxt;
			cur = s & 1 ? list0 : list1;
			++s;
			const int32_t far = sh.far;
			bw_bar<MW>();
			if (lead) {
				sh.s = s;
				if (lag) sh.imin = far - kPruneLag;
			}
			__syncwarp();
		}
		// the hash table back to empty
		bw_bar<MW>();
		const int32_t n_blk = min(sh.n_blk, sh.nb);
#pragma unroll 1
		for (int32_t j = threadIdx.x; j < n_blk; j += MW ? blockDim.x : 32)
			sh.hash[sh.slot[j]] = make_uint2(0xffffffffu, 0xffffffffu);
		bw_bar<MW>();
		if (lag) { // its score, where it found one, is the bound
			lag = false;
			if (sc >= 0) {
				attained = true, T = sc;
				// The exact run makes about beta / 4 slack^2 iterations of step 1 more than one per
				// score (slack = T - h; beta 1.2 measured on the sparse benchmark graph, 4 to 14 on the
				// dense one, 5 and 49 vertices per 1000 bases, nothing between measured: the line
				// decides time only); windows from every base cost the time of ~0.2 per base and make the
				// slack 2.2 times smaller.
				const float slack = (float)(T - h0);
				if ((p.dens_milli >= 20 ? 8.0f : 1.2f) * slack * slack > (float)ql) bw_seeds<MW>(1);
			}
			continue;
		}
		if (ovf && sc < 0) {
			st = ST_CAPACITY, steps = s + 1;
			break;
		}
		dist = sc >= 0 ? sc : attained ? T : -1;
		steps = dist >= 0 ? dist + 1 : s;
		break;
	}
	if (lead) {
		p.dist[r] = st == ST_OK ? dist : -1;
		p.status[r] = st;
		if (st == ST_CAPACITY && p.retry_list) {
			const int32_t q = atomicAdd(p.retry_n, 1);
			p.retry_list[q] = r;
		}
		if (p.steps_out) p.steps_out[r] = steps;
	}
}

// Points the CTA's shared state at its arena and empties the hash table.
__device__ __forceinline__ void bw_init(const DevGraph &g, const BwLay &bw, uint8_t *wsb)
{
	BwShm &sh = bw_sh();
	if (threadIdx.x == 0) {
		sh.blk = (BwBlock *)wsb, sh.hash = (uint2 *)(wsb + bw.hash), sh.slot = (uint32_t *)(wsb + bw.slot);
		sh.e = (uint32_t *)(wsb + bw.e), sh.f = (uint32_t *)(wsb + bw.f), sh.n = (uint32_t *)(wsb + bw.n);
		sh.nk = (int32_t *)(wsb + bw.nk), sh.h = (uint16_t *)(wsb + bw.h);
		sh.gpk = (const uint32_t *)g.pk, sh.graw = g.raw, sh.arcx = g.arcx, sh.varcs = g.varcs;
		sh.arc_off = g.arc_off, sh.bloom = g.bloom, sh.bloom_mask = g.bloom_mask, sh.K = g.bloom_k;
		sh.hmask = (uint32_t)bw.hs - 1, sh.nb = bw.nb;
	}
	int4 *const h4 = (int4 *)(wsb + bw.hash);
#pragma unroll 1
	for (int32_t j = threadIdx.x; j < bw.hs / 2; j += blockDim.x) h4[j] = make_int4(-1, -1, -1, -1);
	__syncthreads();
}

// Persistent form: each one-warp CTA owns one arena (p.bw, sized for the longest read of the
// launch) and pulls reads from the cost-ordered queue. 32 warps per SM at 64 registers; 24 or 28
// lose more on 1 kbp reads (2% and up) than they gain elsewhere.
__global__ void __launch_bounds__(32, 32) k_align_blocks(const __grid_constant__ KParams p)
{
	uint8_t *const wsb = p.ws + (int64_t)blockIdx.x * p.bw.total;
	bw_init(p.g, p.bw, wsb);
#pragma unroll 1
	for (int32_t guard = 0; guard < p.n_order + 1; ++guard) {
		int32_t qi = 0;
		if (threadIdx.x == 0) qi = atomicAdd(p.head, 1);
		qi = __shfl_sync(FULL, qi, 0);
		if (qi >= p.n_order) break;
		align_read_blocks<false>(p, p.order[qi], wsb);
	}
}

// The same with all warps of a CTA on one read: one read of 20 kbp at 10% takes 259 ms with one warp,
// 178 with 2, 111 with 4, 81 with 8, 69 with 16 and 67 with 32; 100 reads of 10 kbp at 5% on the dense
// graph 21.1, 18.0, 15.1, 14.5, 14.3 and 14.5 ms. So 16 is the most a read gets.
__global__ void __launch_bounds__(512, 2) k_align_blocks_mw(const __grid_constant__ KParams p)
{
	BwShm &sh = bw_sh();
	uint8_t *const wsb = p.ws + (int64_t)blockIdx.x * p.bw.total;
	bw_init(p.g, p.bw, wsb);
#pragma unroll 1
	for (int32_t guard = 0; guard < p.n_order + 1; ++guard) {
		if (threadIdx.x == 0) sh.claim = atomicAdd(p.head, 1);
		__syncthreads();
		const int32_t qi = sh.claim;
		__syncthreads(); // every thread has the claim before the next one is written
		if (qi >= p.n_order) break;
		align_read_blocks<true>(p, p.order[qi], wsb);
		__syncthreads();
	}
}
#endif

} // namespace gwfb
