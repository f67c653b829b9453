// FP64 SU(3) molecular-dynamics step from stored link products.
//
// The force on link (x, mu) needs, for every nu, W_mu,nu(x) = U_mu(x) U_nu(x+mu)
// and W_nu,mu(x) for the plaquette, and W_mu,nu(x-nu) for the lower staple
// W^+ U_nu(x-nu). Each of the Nd(Nd-1) products a site enters the forces of
// three links, so they are computed once and stored:
//   k_md_products: W of both orders and A = proj(W_mu,nu W_nu,mu^+) of every
//                  plane, one warp per plane for 32 sites;
//   k_md_force:    P_mu -= coef (sum_nu +-A + proj(U_mu sum_nu W^+ U_nu)), and
//                  with FUSE the link update after it, one warp per direction
//                  for 32 sites.
// No unitarity is used: the forces are those of the staples for any matrices.
// FP64 instructions a site with the link update (four dimensions): 6 x 322 +
// 4 x 754 = 4950, against 7000 for a thread per link (thirteen products a link
// and their sums); GB300 takes a warp's FP64 instruction every 16 cycles per SM,
// and that is all that bounds this path: the products' traffic (2112 bytes a
// site written and read once, mostly through L2) is under a tenth of the time.
// A warp per plane or direction fills the chip on small lattices too (8^4: 128
// tiles of 32 sites), where a thread per link left 88 of 152 SMs without a block.
// SU(3) FP64 on a GB300, one step with the link update: 8^4 195 us as a thread
// per link and a separate update, 52 here (products 19.4, forces 32.1: one tile
// on 128 of 152 SMs, the pipe 79 to 86% busy there); 32^4 16.3 -> 9.55 ms.
//
// Scratch: the products of the whole lattice when they fit kMdScratchCap, else
// a ring of R slices of dimension 0 (a slice's forces read the products of its
// own and of the preceding slice), walked in slabs of R - 1 slices: two slices
// at least, where they fit kMdScratchMax or a quarter of the links. A lattice
// with larger slices steps without scratch, by the kernels of kernels.cuh.
#pragma once

namespace meshgb {

constexpr size_t kMdScratchCap = size_t(256) << 20;
constexpr size_t kMdScratchMax = size_t(512) << 20;

// Slices of dimension 0 whose products are held, S sites each
struct MdRing
{
	int R;     // slices held
	int whole; // R == L0: slice x0 in slot x0; else slice x0 in slot (x0 + 1) mod R
	int64_t S; // sites of a slice
	int64_t V; // R S: sites held
};

// slot of the products of the site `lex` in slice x0 (t: x0 + 1, or 0 for the
// last slice seen as the one before slice 0)
__device__ __forceinline__ int64_t ring_index(MdRing const &r, int32_t lex, int x0, int t, int par)
{
	int slot = r.whole ? x0 : t % r.R;
	int64_t l = int64_t(slot) * r.S + (lex - int64_t(x0) * r.S);
	return int64_t(par) * (r.V / 2) + (l >> 1);
}

// products of the slices [x0, x0 + n) into the ring, slice x0 at t = t0
template <class T, int ND>
__global__ void __launch_bounds__(32 * kPlanes<ND>)
    k_md_products(Geom g, MdRing ring, int x0, int n, int t0, T const *__restrict__ U, T *__restrict__ W, T *__restrict__ A)
{
	using Gp = Group<SU3, T>;
	using E = typename Gp::E;
	LinkLoad<SU3, T, ND> ld{U, g.V};
	int q = threadIdx.x >> 5, mu = plane_mu<ND>(q), nu = plane_nu<ND>(q);
	int ntiles = slab_tiles(ring.S, n);
	for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
	{
		int64_t s;
		if (!slab_site(g, ring.S, x0, n, tile, s))
			continue;
		Site<ND> st = site_from_eo<ND>(g, s);
		int64_t k = ring_index(ring, st.lex, st.x(0), t0 + st.x(0) - x0, st.par);
		E ab = Gp::mul(ld(mu, s), ld(nu, eo_shift1<ND>(g, st, mu, +1)));
		comp<T, Gp::NR>(W, ring.V, 2 * q).store(k, ab.v);
		E dc = Gp::mul(ld(nu, s), ld(mu, eo_shift1<ND>(g, st, nu, +1)));
		comp<T, Gp::NR>(W, ring.V, 2 * q + 1).store(k, dc.v);
		T a[Gp::NA];
		Gp::proj(Gp::mul_nd(ab, dc), a);
		comp<T, Gp::NA>(A, ring.V, q).store(k, a);
	}
}

// plane index of mu < nu
template <int ND> __device__ __forceinline__ int plane_of(int mu, int nu) { return mu * ND - mu * (mu + 1) / 2 + nu - mu - 1; }

// momentum step (and with FUSE the link update) of the slices [x0, x0 + n)
template <class T, int ND, bool FUSE>
__global__ void __launch_bounds__(32 * ND)
    k_md_force(Geom g, MdRing ring, int x0, int n, T const *__restrict__ U, T const *__restrict__ W,
               T const *__restrict__ A, T *__restrict__ P, T coef, RedSlot kin, T *__restrict__ Uout, T tu, int reunit)
{
	using Gp = Group<SU3, T>;
	using E = typename Gp::E;
	LinkLoad<SU3, T, ND> ld{U, g.V};
	int mu = threadIdx.x >> 5;
	int ntiles = slab_tiles(ring.S, n);
	double acc = 0.0;
	for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
	{
		int64_t s;
		if (!slab_site(g, ring.S, x0, n, tile, s))
			continue;
		Site<ND> st = site_from_eo<ND>(g, s);
		int64_t k = ring_index(ring, st.lex, st.x(0), st.x(0) + 1, st.par);
		T f[Gp::NA];
#pragma unroll
		for (int a = 0; a < Gp::NA; ++a)
			f[a] = T(0);
		E S = Gp::zero();
		// unrolled: the loads of all planes are in flight before the first product
#pragma unroll
		for (int j = 0; j < ND - 1; ++j)
		{
			int nu = j < mu ? j : j + 1;
			int q = mu < nu ? plane_of<ND>(mu, nu) : plane_of<ND>(nu, mu);
			T a[Gp::NA];
			comp<T, Gp::NA>(const_cast<T *>(A), ring.V, q).load(k, a);
			T sg = mu < nu ? T(1) : T(-1);
#pragma unroll
			for (int r = 0; r < Gp::NA; ++r)
				f[r] = fma(sg, a[r], f[r]);
			int32_t ly = lex_step(g, st.px, st.lex, nu, -1);
			int xy = nu == 0 ? (st.x(0) == 0 ? g.L[0] - 1 : st.x(0) - 1) : st.x(0);
			E w;
			comp<T, Gp::NR>(const_cast<T *>(W), ring.V, 2 * q + (mu < nu ? 0 : 1))
			    .load(ring_index(ring, ly, xy, st.x(0) + (nu != 0), st.par ^ 1), w.v);
			Gp::add_dn(S, w, ld(nu, int64_t(st.par ^ 1) * g.Vh + (ly >> 1)));
		}
		E u = ld(mu, s);
		{
			T a[Gp::NA];
			Gp::proj(Gp::mul(u, S), a);
#pragma unroll
			for (int j = 0; j < Gp::NA; ++j)
				f[j] += a[j];
		}
		auto Pv = comp<T, Gp::NA>(P, g.V, mu);
		T p[Gp::NA];
		Pv.template load<CACHE_STREAM>(s, p);
#pragma unroll
		for (int j = 0; j < Gp::NA; ++j)
			p[j] = fma(-coef, f[j], p[j]);
		Pv.template store<CACHE_STREAM>(s, p);
		if (kin.result)
			acc += double(Gp::kin(p));
		if constexpr (FUSE)
		{
			E r = Gp::mul(Gp::exp_alg(p, tu), u);
			if (reunit)
				r = Gp::reunit_fast(r);
			comp<T, Gp::NR>(Uout, g.V, mu).store(s, r.v);
		}
	}
	if (kin.result) // uniform over the grid
		grid_sum<32 * ND>(acc, kin);
}

// the ring of a lattice (site_bytes held for a site, link_bytes of links) and its
// bytes; none (R = 0) where two slices are too large
inline MdRing md_ring(Geom const &g, size_t site_bytes, size_t link_bytes, size_t *bytes)
{
	MdRing r{};
	r.S = g.V / g.L[0];
	size_t slice = size_t(r.S) * site_bytes;
	int64_t fit = int64_t(kMdScratchCap / slice);
	if (fit < 2)
		fit = 2 * slice <= kMdScratchMax || 2 * slice <= link_bytes / 4 ? 2 : 0;
	r.R = int(fit < g.L[0] ? fit : g.L[0]);
	r.whole = r.R == g.L[0];
	r.V = r.R * r.S;
	*bytes = slice * size_t(r.R);
	return r;
}

} // namespace meshgb
