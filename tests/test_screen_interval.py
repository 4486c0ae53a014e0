"""The yield screen's material terms against the FP64 properties, on the CPU.

screen_terms (csrc/des_common.cuh) gives FP32 values of plastic_props' anphi,
amc and ten_max that lie within its own 2^-17 of the FP64 ones, whichever end
of the softening interval or place in it the plastic strain has.  The header
itself is compiled for the host, with the device intrinsics restated, so that
its branches are the ones under test: plastic strains at, around and beyond
both ends, intervals that start above zero, empty and inverted intervals (an
immediate drop to the saturated values), a zero friction angle and per-element
cohesions.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <math.h>
#define __device__
#define __forceinline__ inline
#define __noinline__
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
struct double2 { double x, y; };
struct double4 { double x, y, z, w; };
template <class T, class S> static T bits_of(S s) { T t; memcpy(&t, &s, sizeof t); return t; }
static int __double2hiint(double x) { return (int)(bits_of<uint64_t>(x) >> 32); }
static int __double2loint(double x) { return (int)(uint32_t)bits_of<uint64_t>(x); }
static double __hiloint2double(int h, int l) { return bits_of<double>((uint64_t)(uint32_t)h << 32 | (uint32_t)l); }
static long long __double_as_longlong(double x) { return bits_of<long long>(x); }
static double __longlong_as_double(long long x) { return bits_of<double>(x); }
static unsigned __float_as_uint(float x) { return bits_of<unsigned>(x); }
static float __uint_as_float(unsigned x) { return bits_of<float>(x); }
static void atomicOr(unsigned *p, unsigned b) { *p |= b; }
#include "des_common.cuh"

// row: pls0, pls1, cohesion0, cohesion1, friction0, friction1, tension_max
extern "C" void terms(const double *row, int own_cohesion, int n, const double *pls, double *exact, float *screen)
{
    using namespace des;
    KP p;
    memset((void *)&p, 0, sizeof p);
    MatC &m = p.mat;
    p.ne = 1;
    m.nmat = 1;
    m.pls0[0] = row[0], m.pls1[0] = row[1];
    // a per-element cohesion stands in for the material's, which is then another
    m.cohesion0[0] = own_cohesion ? 7 * row[2] : row[2], m.cohesion1[0] = own_cohesion ? 7 * row[3] : row[3];
    if (own_cohesion) p.ef[DES_EF_COHESION0] = row + 2, p.ef[DES_EF_COHESION1] = row + 3;
    m.friction_angle0[0] = row[4], m.friction_angle1[0] = row[5];
    m.tension_max = row[6];
    m.pt_n = 2;
    for (int k = 0; k < 2; ++k) {   // as the context's creation fills the table
        m.pt_phi[k] = row[4 + k];
        plastic_angles(m.pt_phi[k], 0, m.pt_anphi[k], m.pt_anpsi[k], m.pt_sqrt_anphi[k], m.pt_tanphi[k]);
        m.pt_coh_over_tan[k] = (k ? m.cohesion1 : m.cohesion0)[0] / m.pt_tanphi[k];
        m.pt_anphi_f[k] = (float)m.pt_anphi[k];
        m.pt_sqrt_anphi_f[k] = (float)m.pt_sqrt_anphi[k];
        m.pt_tanphi_f[k] = m.pt_phi[k] == 0 ? 0.0f : (float)m.pt_tanphi[k];
    }
    m.tension_max_f = (float)m.tension_max;
    m.softens = m.pls0[0] < m.pls1[0];
    m.hardening[0] = (m.cohesion1[0] - m.cohesion0[0]) / (m.pls1[0] - m.pls0[0]);
    for (int i = 0; i < n; ++i) {
        double anpsi, hardn;
        m_plastic_props(p, 0, pls[i], exact[3 * i + 1], exact[3 * i], anpsi, hardn, exact[3 * i + 2]);
        const ScreenTerms t = screen_terms(p, 0, pls[i]);
        screen[4 * i] = t.af, screen[4 * i + 1] = t.cf, screen[4 * i + 2] = t.tf, screen[4 * i + 3] = t.err;
    }
}
"""


@pytest.fixture(scope="module")
def terms(tmp_path_factory):
    d = tmp_path_factory.mktemp("screen")
    src, lib = str(d / "h.cpp"), str(d / "h.so")
    with open(src, "w") as f:
        f.write(HARNESS)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-w", "-shared", "-fPIC",
                           "-I", os.path.join(ROOT, "dynearthsol_gb300", "csrc"), src, "-o", lib])
    fn = C.CDLL(lib).terms
    dp, fp = C.POINTER(C.c_double), C.POINTER(C.c_float)
    fn.argtypes = [dp, C.c_int, C.c_int, dp, dp, fp]

    def call(row, own, pls):
        row, pls = np.array(row, np.float64), np.array(pls, np.float64)
        exact, screen = np.zeros((pls.size, 3)), np.zeros((pls.size, 4), np.float32)
        fn(row.ctypes.data_as(dp), own, pls.size, pls.ctypes.data_as(dp), exact.ctypes.data_as(dp),
           screen.ctypes.data_as(fp))
        return exact, screen
    return call


@pytest.mark.parametrize("own", [0, 1])
@pytest.mark.parametrize("phi", [(30.0, 15.0), (10.0, 40.0), (0.0, 0.0), (0.0, 20.0)])
@pytest.mark.parametrize("l0,l1", [(0.0, 0.1), (0.05, 0.1), (0.0, 0.0), (0.05, 0.05), (0.1, 0.05), (-0.0, 0.0)])
def test_terms_lie_within_their_allowance_of_the_fp64_properties(terms, l0, l1, phi, own):
    ends = [e for l in (l0, l1) for e in (np.nextafter(l, -1), l, np.nextafter(l, 1))]
    pls = ends + [-0.0, 0.0, 1e-300, 0.5 * (l0 + l1), 0.07, 0.2, 5.0]
    for c0, c1 in [(4e7, 4e6), (1e6, 3e6)]:
        exact, screen = terms((l0, l1, c0, c1, *phi, 1e9), own, pls)
        want = exact.astype(np.float32).astype(np.float64)
        err = screen[:, 3:].astype(np.float64)
        assert np.all(err <= 2.0 ** -17)
        # 2^-22: f32_of rounds halves away from zero where NumPy rounds to even
        assert np.all(np.abs(screen[:, :3] - want) <= (err + 2.0 ** -22) * np.abs(want))
