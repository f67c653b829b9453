"""FP64 SU(3) arithmetic of the device code, compiled for the host (it is
__host__ __device__) and compared with long double: the products as chains of
fused multiply-adds, their accumulating forms, and the exponential on both
sides of the norm where the closed form takes over from the series. No GPU
needed."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "csrc/group.cuh"
#include <cmath>
#include <complex>
#include <cstdio>
#include <random>
using namespace meshgb;
using D = Group<SU3, double>;
using Z = std::complex<long double>;
struct M { Z a[3][3]; };
static M wide(D::E const &e)
{
	M m;
	for (int i = 0; i < 3; ++i)
		for (int j = 0; j < 3; ++j)
			m.a[i][j] = Z(e.at(i, j).re, e.at(i, j).im);
	return m;
}
static M mul(M const &x, M const &y)
{
	M r;
	for (int i = 0; i < 3; ++i)
		for (int j = 0; j < 3; ++j)
		{
			r.a[i][j] = 0;
			for (int k = 0; k < 3; ++k)
				r.a[i][j] += x.a[i][k] * y.a[k][j];
		}
	return r;
}
static M adj(M const &x)
{
	M r;
	for (int i = 0; i < 3; ++i)
		for (int j = 0; j < 3; ++j)
			r.a[i][j] = std::conj(x.a[j][i]);
	return r;
}
static M add(M const &x, M const &y)
{
	M r;
	for (int i = 0; i < 3; ++i)
		for (int j = 0; j < 3; ++j)
			r.a[i][j] = x.a[i][j] + y.a[i][j];
	return r;
}
static double off(D::E const &e, M const &m)
{
	long double d = 0;
	for (int i = 0; i < 3; ++i)
		for (int j = 0; j < 3; ++j)
			d = std::fmax(d, std::abs(Z(e.at(i, j).re, e.at(i, j).im) - m.a[i][j]));
	return double(d);
}
// Taylor series of exp in long double
static M expm(M const &x)
{
	M r{}, t{};
	for (int i = 0; i < 3; ++i)
		r.a[i][i] = t.a[i][i] = 1;
	for (int k = 1; k < 60; ++k)
	{
		t = mul(t, x);
		for (auto &row : t.a)
			for (auto &z : row)
				z /= k;
		r = add(r, t);
	}
	return r;
}
int main()
{
	std::mt19937_64 rng(5);
	std::normal_distribution<double> nd;
	double e_prod = 0, e_exp = 0;
	for (int t = 0; t < 2000; ++t)
	{
		D::E a, b, s;
		for (int k = 0; k < 18; ++k)
			a.v[k] = 0.5 * nd(rng), b.v[k] = 0.5 * nd(rng), s.v[k] = 0.5 * nd(rng);
		M A = wide(a), B = wide(b), S = wide(s);
		e_prod = std::fmax(e_prod, off(D::mul(a, b), mul(A, B)));
		e_prod = std::fmax(e_prod, off(D::mul_nd(a, b), mul(A, adj(B))));
		e_prod = std::fmax(e_prod, off(D::mul_dn(a, b), mul(adj(A), B)));
		D::E r = s;
		D::add_nd(r, a, b);
		e_prod = std::fmax(e_prod, off(r, add(S, mul(A, adj(B)))));
		r = s;
		D::add_dn(r, a, b);
		e_prod = std::fmax(e_prod, off(r, add(S, mul(adj(A), B))));
		r = s;
		D::add_mul_adj(r, a, b);
		e_prod = std::fmax(e_prod, off(r, add(S, adj(mul(A, B)))));
	}
	// |X| from zero past the bound of the series (1)
	double const norms[] = {0, 1e-9, 1e-3, 0.05, 0.1999, 0.2001, 0.4999, 0.5, 0.5001, 0.9999, 1.0001, 2.0};
	for (double n : norms)
		for (int t = 0; t < 200; ++t)
		{
			double o[8];
			for (double &x : o)
				x = nd(rng);
			double f = n / std::sqrt(D::kin(o));
			for (double &x : o)
				x *= f;
			e_exp = std::fmax(e_exp, off(D::exp_alg(o, 1.0), expm(wide(D::from_alg(o)))));
		}
	std::printf("%.3e %.3e\n", e_prod, e_exp);
	return 0;
}
"""


def test_su3_fp64_products_and_exponential(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    src = tmp_path / "su3_fp64.cu"
    src.write_text(SRC)
    exe = tmp_path / "su3_fp64"
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++20", "-O2", "-I",
                        os.path.join(ROOT, "mesh_gb300"), str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    e_prod, e_exp = (float(v) for v in out.stdout.split())
    # a chain of seven terms of entries up to about 4: 7 * 2^-53 * 7 * 16
    assert e_prod < 9e-14
    # Horner's rule on three bounded coefficients and six products: some tens
    # of roundings at |exp| <= 1; the closed form loses more near |X| = 1
    assert e_exp < 2e-14
