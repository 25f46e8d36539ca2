/*
 * The factored sweep (kernel in dk_kernels.cu, batches in dk_batch.cu; programs
 * from dk_plan_fx.c, layout in dk_internal.h).
 *
 * A tile of 2^m amplitudes (12 bits: 64 or 32 KiB) comes into shared memory by
 * cp.async and goes through the passes of the program; thread t holds 16
 * amplitudes of a pass in registers, applies the pass's operations to them and
 * puts them back, and the last pass writes to the register from there.  16
 * registers rather than 8: 4 passes per sweep of the 30-qubit job instead of 5.3
 * and a third less shared-memory traffic, for 128 registers a thread (complex128,
 * two CTAs per SM) or 80 (complex64, three).
 *
 * What bounds it: FP64 (FP32) arithmetic and shared-memory wavefronts, about
 * half each of a sweep's time beside the streaming; they overlap little, since
 * the groups of warps that one register file holds are few.  A sweep of the
 * 28-qubit brickwork circuit takes 3.24 ms in complex128 (4.13 with 8x8 complex
 * products on FP64 MMAs) and 1.65 ms in complex64 (3.02 with TF32-split
 * products in tensor memory; 2.01 at the same number of sweeps); the streaming
 * alone takes 1.75 and 0.89.  Tried and slower, at 3.57 ms before the kernel made
 * the register's scalars itself: a ring of three tile buffers for
 * two groups of one CTA, the next tile in flight throughout (4.15 ms), 11-bit
 * tiles (3.85), every stage with its four rotations whether it has them or not
 * (3.90).  Coefficients read one by one at their use instead of in batches: 3.62.
 */
#ifndef DK_SWEEP_FX_CUH_
#define DK_SWEEP_FX_CUH_

#ifndef DK_IN_BOUNDS /* translation units without index checks */
#define DK_IN_BOUNDS(i, lim, site) true
#endif

/* Rotation of the 8 register pairs (p, p ^ V): a[p] += x a[q], a[q] += y a[p]
 * with the pair's real coefficients.  complex64 takes each pair's two
 * components in one packed multiply-add. */
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
	unsigned long long r;
	asm("fma.rn.f32x2 %0, %1, %2, %3;"
	    : "=l"(r)
	    : "l"(*reinterpret_cast<unsigned long long *>(&a)),
	      "l"(*reinterpret_cast<unsigned long long *>(&b)),
	      "l"(*reinterpret_cast<unsigned long long *>(&c)));
	return *reinterpret_cast<float2 *>(&r);
}

__device__ __forceinline__ void fx_pair(double2 &p, double2 &q, const double2 &w)
{
	const double2 x = p, y = q;
	p = make_double2(fma(w.x, y.x, x.x), fma(w.x, y.y, x.y));
	q = make_double2(fma(w.y, x.x, y.x), fma(w.y, x.y, y.y));
}
__device__ __forceinline__ void fx_pair(float2 &p, float2 &q, const float4 &w)
{
	const float2 x = p, y = q;
	p = fma2(make_float2(w.x, w.y), y, x);
	q = fma2(make_float2(w.z, w.w), x, y);
}

template <typename C2> struct FxCoef;
template <> struct FxCoef<double2> {
	typedef double2 T;
};
template <> struct FxCoef<float2> {
	typedef float4 T;
};

/* Rotation along V with one pair of reals, or with a pair for each of the 8
 * register pairs. */
template <int V, typename C2, typename W>
__device__ __forceinline__ void fx_rot1(C2 (&a)[DK_FX_REGS], const W w)
{
	constexpr int low = V & -V;
#pragma unroll
	for (int p = 0; p < DK_FX_REGS; ++p)
		if (!(p & low))
			fx_pair(a[p], a[p ^ V], w);
}

template <int V, typename C2>
__device__ __forceinline__ void fx_rot(C2 (&a)[DK_FX_REGS], const uint4 *co)
{
	constexpr int low = V & -V;
	const typename FxCoef<C2>::T *c = reinterpret_cast<const typename FxCoef<C2>::T *>(co);
	int i = 0;
#pragma unroll
	for (int p = 0; p < DK_FX_REGS; ++p)
		if (!(p & low))
			fx_pair(a[p], a[p ^ V], c[i++]);
}

template <int V, typename C2>
__device__ __forceinline__ void fx_swap(C2 (&a)[DK_FX_REGS], uint32_t mask)
{
	constexpr int low = V & -V;
	int i = 0;
#pragma unroll
	for (int p = 0; p < DK_FX_REGS; ++p) {
		if (p & low)
			continue;
		if ((mask >> i++) & 1u) {
			const C2 x = a[p];
			a[p] = a[p ^ V];
			a[p ^ V] = x;
		}
	}
}

/* 16 bytes of coefficients.  Volatile, so that a batch of them is requested
 * before the arithmetic that the caller writes behind it.  `at` is an address in
 * shared memory, or (GLOBAL) a pointer. */
__device__ __forceinline__ void fx_load(double2 &v, uint32_t at)
{
	asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(at));
}
__device__ __forceinline__ void fx_load(float4 &v, uint32_t at)
{
	asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
		     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
		     : "r"(at));
}
__device__ __forceinline__ void fx_load(double2 &v, const unsigned char *at)
{
	asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(at));
}
__device__ __forceinline__ void fx_load(float4 &v, const unsigned char *at)
{
	asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
		     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
		     : "l"(at));
}
template <bool GLOBAL> struct FxAddr;
template <> struct FxAddr<false> {
	static __device__ __forceinline__ uint32_t of(const uint4 *p)
	{
		return (uint32_t)__cvta_generic_to_shared(p);
	}
};
template <> struct FxAddr<true> {
	static __device__ __forceinline__ const unsigned char *of(const uint4 *p)
	{
		return reinterpret_cast<const unsigned char *>(p);
	}
};

/* a[4 b .. 4 b + 3] *= the diagonal's values, a batch of four ahead */
template <typename A>
__device__ __forceinline__ void fx_diag(double2 (&a)[DK_FX_REGS], A at)
{
	double2 c[2][4];
#pragma unroll
	for (int i = 0; i < 4; ++i)
		fx_load(c[0][i], at + 16 * i);
#pragma unroll
	for (int b = 0; b < 4; ++b) {
		if (b < 3)
#pragma unroll
			for (int i = 0; i < 4; ++i)
				fx_load(c[(b + 1) & 1][i], at + 64 * (b + 1) + 16 * i);
#pragma unroll
		for (int i = 0; i < 4; ++i)
			a[4 * b + i] = cmul(c[b & 1][i], a[4 * b + i]);
	}
}
template <typename A>
__device__ __forceinline__ void fx_diag(float2 (&a)[DK_FX_REGS], A at)
{
	float4 c[2][2];
#pragma unroll
	for (int i = 0; i < 2; ++i)
		fx_load(c[0][i], at + 16 * i);
#pragma unroll
	for (int b = 0; b < 4; ++b) {
		if (b < 3)
#pragma unroll
			for (int i = 0; i < 2; ++i)
				fx_load(c[(b + 1) & 1][i], at + 32 * (b + 1) + 16 * i);
#pragma unroll
		for (int i = 0; i < 2; ++i) {
			const float4 w = c[b & 1][i];
			a[4 * b + 2 * i] = cmul(make_float2(w.x, w.y), a[4 * b + 2 * i]);
			a[4 * b + 2 * i + 1] = cmul(make_float2(w.z, w.w), a[4 * b + 2 * i + 1]);
		}
	}
}

template <bool GLOBAL, typename C2>
__device__ __forceinline__ void fx_op(C2 (&a)[DK_FX_REGS], uint32_t code, uint32_t mask,
				      const uint4 *co)
{
	typedef typename FxCoef<C2>::T W;
	const C2 *c = reinterpret_cast<const C2 *>(co);
	if (code == DK_FX_STAGE) {
		const auto at = FxAddr<GLOBAL>::of(co);
		W w[4];
#pragma unroll
		for (int i = 0; i < 4; ++i)
			fx_load(w[i], at + 16 * i);
		if (mask & 16u)
			fx_diag(a, at + 64);
		if ((mask & 15u) == 15u) {
			/* the four in a row: no branch between them */
			fx_rot1<1>(a, w[0]);
			fx_rot1<2>(a, w[1]);
			fx_rot1<4>(a, w[2]);
			fx_rot1<8>(a, w[3]);
		} else {
			if (mask & 1u)
				fx_rot1<1>(a, w[0]);
			if (mask & 2u)
				fx_rot1<2>(a, w[1]);
			if (mask & 4u)
				fx_rot1<4>(a, w[2]);
			if (mask & 8u)
				fx_rot1<8>(a, w[3]);
		}
		return;
	}
	switch (code) {
	case DK_FX_PHASE: {
		const C2 u = c[0];
#pragma unroll
		for (int p = 0; p < DK_FX_REGS; ++p)
			if ((mask >> p) & 1u)
				a[p] = cmul(u, a[p]);
		break;
	}
	case DK_FX_NEG:
#pragma unroll
		for (int p = 0; p < DK_FX_REGS; ++p)
			if ((mask >> p) & 1u)
				a[p] = mk(-a[p].x, -a[p].y);
		break;
#define DK_FX_V(V)                                      \
	case DK_FX_ROT + V: fx_rot<V>(a, co); break;    \
	case DK_FX_SWAP + V: fx_swap<V>(a, mask); break;
	DK_FX_V(1) DK_FX_V(2) DK_FX_V(3) DK_FX_V(4) DK_FX_V(5)
	DK_FX_V(6) DK_FX_V(7) DK_FX_V(8) DK_FX_V(9) DK_FX_V(10)
	DK_FX_V(11) DK_FX_V(12) DK_FX_V(13) DK_FX_V(14) DK_FX_V(15)
#undef DK_FX_V
	default: break;
	}
}

/* One sweep: the tiles first, first + step, ... of the register.  `sm` holds a
 * tile and the program.  Sums of |amp|^2 of the tiles read (where tiles are
 * skipped) and written go to insq and outsq. */
template <typename R, bool NARROW>
__device__ __forceinline__ void fx_sweep(const typename CT<R>::T *__restrict__ in,
					 typename CT<R>::T *out,
					 const unsigned char *__restrict__ prog, unsigned char *sm,
					 uint64_t first, uint64_t step, int sums, double &insq,
					 double &outsq)
{
	typedef typename CT<R>::T C2;
	__shared__ uint64_t sdep[DK_DEP_NIBBLES][16];
	/* byte offsets in the register: of stream bit j, of the last pass's bit j */
	__shared__ uint64_t soff[DK_FX_BITS], poff[DK_FX_BITS];
	__shared__ uint32_t sro[DK_FX_BITS]; /* byte offset of stream bit j in the tile */
	const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
	const dk_sweep_hdr *gh = reinterpret_cast<const dk_sweep_hdr *>(prog);
	const int m = gh->m;
	const int lanes = m - DK_FX_BITS;
	/* NARROW: a tile below 9 bits does not fill a warp; its other threads
	 * follow along on the slots of the first ones and write nothing */
	const bool writes = !NARROW || tid < (1u << lanes);
	[[maybe_unused]] const uint32_t tile_bytes = (uint32_t)sizeof(C2) << m;
	unsigned char *const sp = sm + (sizeof(C2) << m);
	{
		const uint32_t units = gh->bytes >> 4;
		for (uint32_t i = tid; i < units; i += blockDim.x)
			cp_async16(sp + 16 * i, prog + 16 * i);
		cp_async_commit();
		cp_async_wait_all();
	}
	__syncthreads();
	const dk_sweep_hdr *h = reinterpret_cast<const dk_sweep_hdr *>(sp);
	const int npass = h->npass, ncond = (int)h->ncond;
	const dk_fx_pass *passes = reinterpret_cast<const dk_fx_pass *>(sp + sizeof(dk_sweep_hdr));
	const uint4 *lists = reinterpret_cast<const uint4 *>(passes + npass);
	const uint4 *ops = reinterpret_cast<const uint4 *>(sp + h->gate_off);
	const dk_gate_cond *conds = reinterpret_cast<const dk_gate_cond *>(sp + h->cond_off);
	const uint4 *table = reinterpret_cast<const uint4 *>(sp + h->mat_off);
	const dk_fx_pass *const last = passes + npass - 1;
	/* a last pass that stores to the register */
	const bool store = last->flags & DK_FX_STORE;
	if (tid < DK_FX_BITS) {
		soff[tid] = (uint64_t)sizeof(C2) << h->qpos[lanes + tid];
		sro[tid] = (uint32_t)sizeof(C2) * swz_map(1u << (lanes + tid), h->bankv);
		poff[tid] = (uint64_t)sizeof(C2) << h->qpos[__ffs(last->pm[tid]) - 1];
	}
	const int ndep = (h->n - m + 3) >> 2;
	for (int e = tid; e < ndep * 16; e += blockDim.x) {
		uint64_t v = (uint64_t)(e & 15) << (4 * (e >> 4));
		for (int j = 0; j < m; ++j) {
			const int q = h->qpos[j];
			v = ((v >> q) << (q + 1)) | (v & ((1ull << q) - 1ull));
		}
		sdep[e >> 4][e & 15] = v;
	}
	/* streaming: thread t carries tile indices t + (r << lanes); off_t and
	 * off_out: byte offset of this thread's share of a tile as it is read and
	 * as it is written */
	uint64_t off_t = 0, off_out = 0;
	{
		const uint32_t raw = last->rlo[lane] | last->rhi[warp];
		for (int j = 0; j < m; ++j) {
			const uint64_t bit = (uint64_t)sizeof(C2) << h->qpos[j];
			if (j < lanes && ((tid >> j) & 1u))
				off_t |= bit;
			if ((raw >> j) & 1u)
				off_out |= bit;
		}
		if (!store)
			off_out = off_t;
	}
	const uint32_t stid = (uint32_t)sizeof(C2) * swz_map(tid & ((1u << lanes) - 1u), h->bankv);
	__syncthreads();
	const uint64_t ntiles = h->ntiles;
	const bool skip_idle = (in == out) && !h->all_touched;

	auto tile_base = [&](uint64_t t) -> uint64_t {
		uint64_t base = 0;
#pragma unroll
		for (int k = 0; k < DK_DEP_NIBBLES; ++k)
			if (k < ndep)
				base |= sdep[k][(t >> (4 * k)) & 15u];
		return base;
	};
	/* bit c: condition c holds on the tile (lane c looks at it) */
	auto cond_mask = [&](uint64_t base) -> uint32_t {
		bool on = false;
		if ((int)lane < ncond) {
			const uint64_t gc = conds[lane].gc, ga = conds[lane].ga;
			on = ((base & gc) == gc) && !(base & ga);
		}
		return __ballot_sync(0xffffffffu, on);
	};
	/* the first tile t, t + step, ... that some gate acts on; its
	 * base and conditions */
	uint64_t base = 0;
	uint32_t cmask = 0;
	auto find_tile = [&](uint64_t t) -> uint64_t {
		for (; t < ntiles; t += step) {
			base = tile_base(t);
			cmask = cond_mask(base);
			if (!skip_idle || cmask)
				break;
		}
		return t;
	};
	[[maybe_unused]] const uint64_t nglob = (uint64_t)sizeof(C2) << h->n;
	auto bits4 = [&](int r, uint32_t s0, uint32_t s1, uint32_t s2, uint32_t s3) -> uint32_t {
		return ((r & 1) ? s0 : 0u) ^ ((r & 2) ? s1 : 0u) ^ ((r & 4) ? s2 : 0u) ^
		       ((r & 8) ? s3 : 0u);
	};
	auto off4 = [&](int r, uint64_t s0, uint64_t s1, uint64_t s2, uint64_t s3) -> uint64_t {
		return ((r & 1) ? s0 : 0ull) ^ ((r & 2) ? s1 : 0ull) ^ ((r & 4) ? s2 : 0ull) ^
		       ((r & 8) ? s3 : 0ull);
	};
	auto prefetch = [&]() {
		const uint64_t at = (base * sizeof(C2)) | off_t;
		const uint64_t o0 = soff[0], o1 = soff[1], o2 = soff[2], o3 = soff[3];
		const uint32_t s0 = sro[0], s1 = sro[1], s2 = sro[2], s3 = sro[3];
#pragma unroll
		for (int r = 0; r < DK_FX_REGS; ++r) {
			const uint32_t so = stid ^ bits4(r, s0, s1, s2, s3);
			const uint64_t gi = at ^ off4(r, o0, o1, o2, o3);
			if (!writes || !DK_IN_BOUNDS(so, tile_bytes, CHK_LOAD_SMEM) ||
			    !DK_IN_BOUNDS(gi, nglob, CHK_LOAD_GLOBAL))
				continue;
			if (sizeof(C2) == 16)
				cp_async16(sm + so, reinterpret_cast<const unsigned char *>(in) + gi);
			else
				cp_async8(sm + so, reinterpret_cast<const unsigned char *>(in) + gi);
		}
		cp_async_commit();
	};
	C2 a[DK_FX_REGS];
	auto read16 = [&](uint32_t sl, uint32_t s0, uint32_t s1, uint32_t s2, uint32_t s3) {
#pragma unroll
		for (int r = 0; r < DK_FX_REGS; ++r) {
			const uint32_t x = sl ^ bits4(r, s0, s1, s2, s3);
			a[r] = DK_IN_BOUNDS(x, tile_bytes, CHK_GATHER)
				       ? *reinterpret_cast<const C2 *>(sm + x)
				       : C2{};
		}
	};

	uint64_t t = find_tile(first);
	if (t < ntiles)
		prefetch();
	while (t < ntiles) {
		const uint64_t cbase = base;
		const uint32_t cm = cmask;
		cp_async_wait_all();
		__syncthreads();
		if (skip_idle && sums) {
			/* only touched tiles reach here: their old |amp|^2 leaves csq */
			read16(stid, sro[0], sro[1], sro[2], sro[3]);
			if (writes)
#pragma unroll
				for (int r = 0; r < DK_FX_REGS; ++r)
					insq += sqabs(a[r]);
			__syncthreads();
		}
		uint64_t g0 = 0, g1 = 0, g2 = 0, g3 = 0, at = cbase * sizeof(C2) ^ off_out;
		for (int p = 0; p < npass; ++p) {
			const dk_fx_pass *pd = passes + p;
			const uint4 ph = *reinterpret_cast<const uint4 *>(pd);
			const bool out_now = ph.x & DK_FX_STORE;
			uint32_t li = ph.y;
			if (ph.z >> 15) {
				const uint32_t nc = ph.z >> 15;
				li += (cm >> (ph.z & 31u)) & 1u;
				if (nc > 1)
					li += 2u * ((cm >> ((ph.z >> 5) & 31u)) & 1u);
				if (nc > 2)
					li += 4u * ((cm >> ((ph.z >> 10) & 31u)) & 1u);
			}
			const uint4 l1 = lists[2 * li + 1];
			if (!l1.w || out_now) {
				const uint4 l0 = lists[2 * li];
				const uint32_t sg = pd->slo[lane] ^ pd->shi[warp];
				read16(sg, l0.x & 0xffffu, l0.x >> 16, l0.y & 0xffffu,
				       l0.y >> 16);
				if (out_now) {
					/* the results of this pass go to the register: once every
					 * thread has gathered, the next tile's copy can start */
					__syncthreads();
					t = find_tile(t + step);
					if (t < ntiles)
						prefetch();
				}
				const uint32_t raw = (ph.x & DK_PASS_CTL) ? (pd->rlo[lane] | pd->rhi[warp])
									  : 0u;
				const uint4 *o = ops + (l1.y & 0xffffu), *const o1 = ops + (l1.y >> 16);
				for (; o < o1; ++o) {
					const uint4 d = *o;
					if ((d.z | d.w) && !ctl_ok(raw, d.z, d.w))
						continue;
					fx_op<false>(a, d.x & 0xffffu, d.x >> 16, table + d.y);
				}
				if (out_now) {
					const uint64_t p0 = poff[0], p1 = poff[1], p2 = poff[2],
						       p3 = poff[3];
					const uint32_t lm = l1.z;
					auto pass_off = [&](uint32_t x) -> uint64_t {
						return ((x & 1u) ? p0 : 0ull) ^ ((x & 2u) ? p1 : 0ull) ^
						       ((x & 4u) ? p2 : 0ull) ^ ((x & 8u) ? p3 : 0ull);
					};
					g0 = pass_off(lm);
					g1 = pass_off(lm >> 4);
					g2 = pass_off(lm >> 8);
					g3 = pass_off(lm >> 12);
					at ^= pass_off(lm >> 16);
					break;
				}
				/* every thread writes the slots that it read itself */
				const uint32_t sc = sg ^ (l1.x >> 16);
				const uint32_t u0 = l0.z & 0xffffu, u1 = l0.z >> 16, u2 = l0.w & 0xffffu,
					       u3 = l0.w >> 16;
#pragma unroll
				for (int r = 0; r < DK_FX_REGS; ++r) {
					const uint32_t x = sc ^ bits4(r, u0, u1, u2, u3);
					if (writes && DK_IN_BOUNDS(x, tile_bytes, CHK_SCATTER))
						*reinterpret_cast<C2 *>(sm + x) = a[r];
				}
			}
			/* the flag is uniform over the block */
			if (ph.x & DK_PASS_WARP)
				__syncwarp();
			else
				__syncthreads();
		}
		if (!store) {
			read16(stid, sro[0], sro[1], sro[2], sro[3]);
			__syncthreads(); /* the buffer is free: start the next tile's copy */
			t = find_tile(t + step);
			if (t < ntiles)
				prefetch();
			g0 = soff[0];
			g1 = soff[1];
			g2 = soff[2];
			g3 = soff[3];
		}
		if (sums && writes) {
#pragma unroll
			for (int r = 0; r < DK_FX_REGS; ++r)
				outsq += sqabs(a[r]);
		}
#pragma unroll
		for (int r = 0; r < DK_FX_REGS; ++r) {
			const uint64_t gi = at ^ off4(r, g0, g1, g2, g3);
			if (writes && DK_IN_BOUNDS(gi, nglob, CHK_STORE))
				__stcs(reinterpret_cast<C2 *>(reinterpret_cast<unsigned char *>(out) + gi),
				       a[r]);
		}
	}
	cp_async_wait_all();
}

#endif
