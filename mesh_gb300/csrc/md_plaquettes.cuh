// FP32 SU(3) molecular-dynamics step of the trajectory from stored plaquettes.
//
// With special unitary links all four forces of a plaquette follow from one
// algebra element A = proj(P), P = U_mu(y) U_nu(y+mu) U_mu(y+nu)^+ U_nu(y)^+
// (mu < nu): the links (y, mu) and (y, nu) get +A and -A, and for h = U_nu(y) the
// loop of link (y + nu, mu) that starts with it is h^+ P^+ h, whose projection is
// -h^+ A h; likewise +h^+ A h with h = U_mu(y) for link (y + mu, nu).
//   k_md_plaquettes: A of every plane, one warp per plane for 32 sites;
//   k_md_transport:  P_mu -= coef sum_nu +-(A(x) - h^+ A(x-nu) h) and the link
//                    update, one warp per direction for 32 sites.
// 2811 and 4014 instructions a site, about what the thread-per-site kernel takes
// (6584), whose lower staples take two products each; but a sixth of the chain of
// dependent loads a thread, twice the warps, and any extents, no tiles. The price is
// A (192 bytes a site written, read by the site and its neighbours): 1.2 GB of DRAM
// traffic for a step of 32^4 where the thread-per-site kernel has 0.74. The
// plaquettes are bound by issue (68% of the slots), the transport by load latency at
// 24 warps per SM (61% of the slots, 4.9 TB/s of DRAM).
// One step with the link update, SU(3) FP32 on a GB300, before and after:
// 12x20x14x30 59.5 -> 32.9 us, 24^4 115 -> 98, 32^4 328 -> 286 (117 + 173), 8^4
// 13.1 -> 9.0. Measured and not kept: packed FP32x2 products (the same time),
// five or six blocks per SM for the plaquettes (133 us), a rolled loop over the
// planes of the transport (172 us at seven blocks), five blocks (183).
#pragma once

namespace meshgb {

// rows 0, 1 of a b and of a b^+ from rows 0, 1 of a, as chains of fused
// multiply-adds (72; 36 packed ones and about 50 moves)
__device__ __forceinline__ Group<SU3, float>::E su3_rows01(Group<SU3, float>::E const &a, Group<SU3, float>::E const &b)
{
	Group<SU3, float>::E r;
	Group<SU3, float>::chain<2, false>(r, [&](int i, int k) { return a.at(i, k); }, [&](int k, int j) { return b.at(k, j); });
	return r;
}
__device__ __forceinline__ Group<SU3, float>::E su3_rows01_nd(Group<SU3, float>::E const &a, Group<SU3, float>::E const &b)
{
	Group<SU3, float>::E r;
	Group<SU3, float>::chain<2, false>(r, [&](int i, int k) { return a.at(i, k); },
	                                   [&](int k, int j) { return cconj(b.at(j, k)); });
	return r;
}

// h^+ A h for special unitary h and A = from_alg(a), packed. B = A h is needed in
// columns 1 and 2 only: they give the entries (0,1), (0,2), (1,2) and the
// imaginary parts of (1,1) and (2,2), and the trace is zero. 108 fused
// multiply-adds; packed FP32x2 operations take 66, but 90 moves to pair their
// operands.
__device__ __forceinline__ void conj_alg(Group<SU3, float>::E const &h, float const *a, float *o)
{
	float a2 = -(a[0] + a[1]);
	float br[3][3], bi[3][3];
#pragma unroll
	for (int j = 1; j < 3; ++j)
	{
		float h0r = h.v[2 * j], h0i = h.v[2 * j + 1], h1r = h.v[6 + 2 * j], h1i = h.v[7 + 2 * j];
		float h2r = h.v[12 + 2 * j], h2i = h.v[13 + 2 * j];
		// rows of A: (i a0, b01, b02), (-b01^*, i a1, b12), (-b02^*, -b12^*, i a2)
		br[0][j] = fmaf(-a[0], h0i, fmaf(a[2], h1r, fmaf(-a[3], h1i, fmaf(a[4], h2r, -a[5] * h2i))));
		bi[0][j] = fmaf(a[0], h0r, fmaf(a[2], h1i, fmaf(a[3], h1r, fmaf(a[4], h2i, a[5] * h2r))));
		br[1][j] = fmaf(-a[1], h1i, fmaf(-a[2], h0r, fmaf(-a[3], h0i, fmaf(a[6], h2r, -a[7] * h2i))));
		bi[1][j] = fmaf(a[1], h1r, fmaf(-a[2], h0i, fmaf(a[3], h0r, fmaf(a[6], h2i, a[7] * h2r))));
		br[2][j] = fmaf(-a2, h2i, fmaf(-a[4], h0r, fmaf(-a[5], h0i, fmaf(-a[6], h1r, -a[7] * h1i))));
		bi[2][j] = fmaf(a2, h2r, fmaf(-a[4], h0i, fmaf(a[5], h0r, fmaf(-a[6], h1i, a[7] * h1r))));
	}
	// sum_k conj(h_ki) B_kj
	auto re = [&](int i, int j) {
		float t = h.v[2 * i] * br[0][j];
		t = fmaf(h.v[2 * i + 1], bi[0][j], t);
		t = fmaf(h.v[6 + 2 * i], br[1][j], fmaf(h.v[7 + 2 * i], bi[1][j], t));
		return fmaf(h.v[12 + 2 * i], br[2][j], fmaf(h.v[13 + 2 * i], bi[2][j], t));
	};
	auto im = [&](int i, int j) {
		float t = h.v[2 * i] * bi[0][j];
		t = fmaf(-h.v[2 * i + 1], br[0][j], t);
		t = fmaf(h.v[6 + 2 * i], bi[1][j], fmaf(-h.v[7 + 2 * i], br[1][j], t));
		return fmaf(h.v[12 + 2 * i], bi[2][j], fmaf(-h.v[13 + 2 * i], br[2][j], t));
	};
	float r11 = im(1, 1), r22 = im(2, 2);
	o[0] = -(r11 + r22);
	o[1] = r11;
	o[2] = re(0, 1), o[3] = im(0, 1);
	o[4] = re(0, 2), o[5] = im(0, 2);
	o[6] = re(1, 2), o[7] = im(1, 2);
}

// rows 0, 1 brought back to orthonormal to first order: R - (R R^+ - 1) R / 2,
// R R^+ - 1 accumulated from -1. Between its first and last step a trajectory's
// links drift from unitary by rounding (row norms by 4.6e-7 after 40 steps of
// 16^4), and h^+ A h feels that more than staples do: the force was 4.9e-7 off at
// the end, against 3.0e-7 from staples. 60 operations a link.
__device__ __forceinline__ void unitary_rows01(Group<SU3, float>::E &r)
{
	float e00 = -1.f, e11 = -1.f, er = 0.f, ei = 0.f;
#pragma unroll
	for (int k = 0; k < 3; ++k)
	{
		float xr = r.v[2 * k], xi = r.v[2 * k + 1], yr = r.v[6 + 2 * k], yi = r.v[7 + 2 * k];
		e00 = fmaf(xr, xr, fmaf(xi, xi, e00));
		e11 = fmaf(yr, yr, fmaf(yi, yi, e11));
		er = fmaf(xr, yr, fmaf(xi, yi, er));
		ei = fmaf(xi, yr, fmaf(-xr, yi, ei));
	}
	e00 *= -0.5f, e11 *= -0.5f, er *= -0.5f, ei *= -0.5f;
#pragma unroll
	for (int k = 0; k < 3; ++k)
	{
		float xr = r.v[2 * k], xi = r.v[2 * k + 1], yr = r.v[6 + 2 * k], yi = r.v[7 + 2 * k];
		r.v[2 * k] = xr + fmaf(e00, xr, fmaf(er, yr, -ei * yi));
		r.v[2 * k + 1] = xi + fmaf(e00, xi, fmaf(er, yi, ei * yr));
		r.v[6 + 2 * k] = yr + fmaf(e11, yr, fmaf(er, xr, ei * xi));
		r.v[7 + 2 * k] = yi + fmaf(e11, yi, fmaf(er, xi, -ei * xr));
	}
}

// packed algebra elements with 32-bit float4 offsets
struct AlgR32
{
	float4 *A4;
	uint32_t V;
	__device__ __forceinline__ void load(int q, uint32_t k, float *a) const
	{
		uint32_t o = uint32_t(2 * q) * V + k;
		float4 x = A4[o], y = A4[o + V];
		a[0] = x.x, a[1] = x.y, a[2] = x.z, a[3] = x.w;
		a[4] = y.x, a[5] = y.y, a[6] = y.z, a[7] = y.w;
	}
	__device__ __forceinline__ void store(int q, uint32_t k, float const *a) const
	{
		uint32_t o = uint32_t(2 * q) * V + k;
		A4[o] = make_float4(a[0], a[1], a[2], a[3]);
		A4[o + V] = make_float4(a[4], a[5], a[6], a[7]);
	}
};

// A of every plane of the slices [x0, x0 + n) into the ring, slice x0 at t = t0
template <int ND, bool WHOLE>
__global__ void __launch_bounds__(32 * kPlanes<ND>, ND == 4 ? 4 : 8)
    k_md_plaquettes(Geom g, MdRing ring, int x0, int n, int t0, LinkLoadSU3R32 ld, AlgR32 A)
{
	using Gp = Group<SU3, float>;
	using E = typename Gp::E;
	int q = threadIdx.x >> 5, mu = plane_mu<ND>(q), nu = plane_nu<ND>(q);
	int ntiles = slab_tiles(ring.S, n);
	for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
	{
		int64_t s;
		if (!slab_site(g, ring.S, x0, n, tile, s))
			continue;
		Site<ND> st = site_from_eo<ND>(g, s);
		// the plaquette is special unitary: rows 0 and 1 of a b and of it suffice
		E b = ld.rows(nu, eo_shift1<ND>(g, st, mu, +1)), a = ld.rows(mu, s);
		E c = ld.rows(mu, eo_shift1<ND>(g, st, nu, +1)), d = ld.rows(nu, s);
		Gp::complete_row2(b);
		Gp::complete_row2(c);
		E ab = su3_rows01(a, b), dc = su3_rows01(d, c);
		Gp::complete_row2(dc);
		float o[8];
		Gp::proj_rows01(su3_rows01_nd(ab, dc), o);
		uint32_t k = WHOLE ? uint32_t(s) : uint32_t(ring_index(ring, st.lex, st.x(0), t0 + st.x(0) - x0, st.par));
		A.store(q, k, o);
	}
}

// momentum step and link update of the slices [x0, x0 + n);
// row2: the new links' third rows are written (the trajectory reads rows 0 and 1
// of the links between its first and last step)
template <int ND, bool WHOLE>
__global__ void __launch_bounds__(32 * ND, ND == 4 ? 6 : 8)
    k_md_transport(Geom g, MdRing ring, int x0, int n, LinkLoadSU3R32 ld, AlgR32 A, float *__restrict__ P, float coef,
                   RedSlot kin, float *__restrict__ Uout, float tu, int reunit, int row2)
{
	using Gp = Group<SU3, float>;
	using E = typename Gp::E;
	int mu = threadIdx.x >> 5;
	int ntiles = slab_tiles(ring.S, n);
	double acc = 0.0;
	for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
	{
		int64_t s;
		if (!slab_site(g, ring.S, x0, n, tile, s))
			continue;
		Site<ND> st = site_from_eo<ND>(g, s);
		uint32_t k = WHOLE ? uint32_t(s) : uint32_t(ring_index(ring, st.lex, st.x(0), st.x(0) + 1, st.par));
		float f[8];
#pragma unroll
		for (int r = 0; r < 8; ++r)
			f[r] = 0.f;
#pragma unroll
		for (int j = 0; j < ND - 1; ++j)
		{
			int nu = j < mu ? j : j + 1;
			int q = mu < nu ? plane_of<ND>(mu, nu) : plane_of<ND>(nu, mu);
			int32_t ly = lex_step(g, st.px, st.lex, nu, -1);
			uint32_t sy = uint32_t(st.par ^ 1) * uint32_t(g.Vh) + uint32_t(ly >> 1), ky = sy;
			if constexpr (!WHOLE)
			{
				int xy = nu == 0 ? (st.x(0) == 0 ? g.L[0] - 1 : st.x(0) - 1) : st.x(0);
				ky = uint32_t(ring_index(ring, ly, xy, st.x(0) + (nu != 0), st.par ^ 1));
			}
			float a[8], w[8], v[8];
			E h = ld.rows(nu, sy);
			A.load(q, ky, w);
			A.load(q, k, a);
			Gp::complete_row2(h);
			conj_alg(h, w, v);
			float sg = mu < nu ? 1.f : -1.f;
#pragma unroll
			for (int r = 0; r < 8; ++r)
				f[r] = fmaf(sg, a[r] - v[r], f[r]);
		}
		auto Pv = comp<float, 8>(P, g.V, mu);
		float p[8];
		Pv.template load<CACHE_STREAM>(s, p);
#pragma unroll
		for (int r = 0; r < 8; ++r)
			p[r] = fmaf(-coef, f[r], p[r]);
		Pv.template store<CACHE_STREAM>(s, p);
		if (kin.result)
			acc += double(Gp::kin(p));
		E u = ld.rows(mu, s);
		Gp::complete_row2(u);
		E r = su3_rows01(Gp::exp_packed_rows01(p, tu), u);
		if (row2)
		{
			Gp::complete_row2(r);
			if (reunit)
				r = Gp::reunit_fast(r);
			comp<float, Gp::NR>(Uout, g.V, mu).store(s, r.v);
		}
		else
		{
			unitary_rows01(r);
			float4 *U4 = reinterpret_cast<float4 *>(Uout) + (uint32_t(mu) * ld.Vmu + uint32_t(s));
#pragma unroll
			for (int c = 0; c < 3; ++c)
				U4[uint32_t(c) * ld.V] = make_float4(r.v[4 * c], r.v[4 * c + 1], r.v[4 * c + 2], r.v[4 * c + 3]);
		}
	}
	if (kin.result) // uniform over the grid
		grid_sum<32 * ND>(acc, kin);
}

} // namespace meshgb
