"""The FP64 Boys function of the FP64 kernels (csrc/fp64_boys.cuh), compiled for
the host: whatever the argument, it reads inside its table, which lies between
two pages that cannot be read; non-finite and huge arguments give what the
asymptotic form gives (a NaN stays one, F_n(inf) = 0).  Against F_n in extended
precision elsewhere: the downward and upward recursions and the rounded table
leave a few units of 2^-53, bounded here by 2^-49 of F_n."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), 'pyscf_wb97mv_fast_gb300', 'csrc')

SOURCE = r'''
#include "boys_host.hpp"
#include "fp64_boys.cuh"
#include <cstdio>
#include <cstdlib>
#include <sys/mman.h>
#include <unistd.h>
#include <vector>

typedef long double real;
// F_0 .. F_m at T: the ascending series at m, downward from it
static void boys_ref(int m, real T, real* F) {
    real t = 1 / (2 * (real)m + 1), s = t;
    for (int k = 1; k < 4000 && t > s * 1e-22L; ++k) { t *= 2 * T / (2 * m + 2 * k + 1); s += t; }
    F[m] = s * expl(-T);
    for (int n = m - 1; n >= 0; --n) F[n] = (2 * T * F[n + 1] + expl(-T)) / (2 * n + 1);
}

// the table with its last byte at the end of a page (upper) or its first at the
// start of one, between pages without access
static double* guarded(size_t bytes, bool upper) {
    const size_t pg = (size_t)sysconf(_SC_PAGESIZE), n = (bytes + pg - 1) / pg * pg;
    char* p = (char*)mmap(nullptr, n + 2 * pg, PROT_READ | PROT_WRITE,
                          MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (p == MAP_FAILED || mprotect(p, pg, PROT_NONE) || mprotect(p + pg + n, pg, PROT_NONE))
        exit(3);
    return (double*)(upper ? p + pg + n - bytes : p + pg);
}

template<int L> static int run(const std::vector<double>& fine, bool upper) {
    using namespace wb::f64;
    double* tab = guarded(BoysTable<L>::kBytes, upper);
    load_boys<L>(fine.data(), tab);
    double F[L + 1];
    auto at = [&](uint64_t bits) { boys_fast<L>(bits_as<double>(bits), tab, F); };
    for (uint64_t b : {0x7ff8000000000000ull, 0xfff8000000000000ull, 0x7fffffffffffffffull,
                       0xffffffffffffffffull, 0xfff0000000000001ull}) {
        at(b);
        for (int n = 0; n <= L; ++n) if (F[n] == F[n]) return 10;
    }
    at(0x7ff0000000000000ull);
    for (int n = 0; n <= L; ++n) if (F[n] != 0.0) return 11;
    // huge: from 2^126 to the largest double, powers of two and just below
    for (int e = 1149; e <= 2046; ++e)
        for (int d = 0; d < 2; ++d) {
            const uint64_t b = ((uint64_t)e << 52) - d;
            at(b);
            const double T = bits_as<double>(b), f0 = std::sqrt(M_PI / 4 / T);
            if (!(std::fabs(F[0] - f0) <= 4e-16 * f0)) return 12;
            for (int n = 0; n < L; ++n)
                if (!(std::fabs(F[n + 1] - (n + 0.5) * F[n] / T) <= 1e-15 * F[n + 1] + 1e-307))
                    return 13;
        }
    double worst = 0.0;
    srand(7);
    for (int k = 0; k < 40000; ++k) {
        double T = k < 1153 ? k / 32.0 : 120.0 * rand() / RAND_MAX;
        if (k >= 20000) T = std::exp(std::log(1e-12) + 32.0 * rand() / RAND_MAX);
        if (k == 39999) T = std::nextafter(36.0, 0.0);
        if (k == 39998) T = 36.0;
        real R[L + 41];
        boys_fast<L>(T, tab, F);
        if (T < 200) boys_ref(L + 40, T, R);
        else {
            R[0] = sqrtl(acosl(-1.0L) / 4 / (real)T);
            for (int n = 0; n < L; ++n) R[n + 1] = (2 * n + 1) * R[n] / (2 * (real)T);
        }
        for (int n = 0; n <= L; ++n)
            worst = std::fmax(worst, (double)fabsl((F[n] - R[n]) / R[n]));
    }
    return worst <= 0x1p-49 ? 0 : 14;
}

int main() {
    std::vector<double> fine;
    for (int k = 0; k < wb::kBoysFineNodes; ++k) {
        real R[wb::kBoysFineCols + 40];
        boys_ref(wb::kBoysFineCols + 39, k / 32.0L, R);
        for (int n = 0; n < wb::kBoysFineCols; ++n) fine.push_back((double)R[n]);
    }
    for (int j = 0; j < 64; ++j)
        fine.push_back(bits_as<double>((unsigned long long)ldexpl(exp2l(-j / 64.0L), 63)));
    for (bool upper : {false, true}) {
        int r[8] = {run<0>(fine, upper), run<1>(fine, upper), run<2>(fine, upper),
                    run<3>(fine, upper), run<4>(fine, upper), run<5>(fine, upper),
                    run<6>(fine, upper), run<7>(fine, upper)};
        for (int l = 0; l < 8; ++l)
            if (r[l]) { printf("L = %d: check %d\n", l, r[l]); return r[l]; }
    }
    return 0;
}
'''


def test_boys_reads_inside_its_table(tmp_path):
    src = tmp_path / 'boys.cpp'
    src.write_text(SOURCE)
    exe = tmp_path / 'boys'
    cuda = os.environ.get('CUDA_HOME', '/usr/local/cuda')
    subprocess.run(['g++', '-O1', '-std=c++17', '-w', '-ffp-contract=off', '-I', HERE,
                    '-I', CSRC, '-I', os.path.join(cuda, 'include'), str(src), '-o', str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout)


@pytest.mark.gpu
@pytest.mark.parametrize('value', [float('nan'), -float('nan'), float('inf'), -float('inf')])
def test_points_off_the_map_stay_alone(value):
    """AO values and the FP64 Hartree potential on a grid with one coordinate
    that is no number or infinite: AO values of zero there, no finite potential
    (a NaN) from the classes above (s,s), every other point as without it."""
    import numpy as np
    import torch

    from helpers import density, dimer
    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine
    mol = dimer('synthetic-tzvp')
    eng = CosxEngine(mol)
    rng = np.random.default_rng(4)
    pts = eng.relative(mol.atom_coords()[rng.integers(mol.natm, size=70)]
                       + rng.normal(size=(70, 3)))
    bad = pts.clone()
    bad[37, 1] = torch.tensor(np.copysign(abs(value), value), dtype=torch.float64)
    keep = [i for i in range(70) if i != 37]
    for f in (eng.ao_eval, eng.ao_eval_deriv1):
        a, b = f(pts), f(bad)
        assert torch.equal(a[..., keep], b[..., keep])
        assert not bool(b[..., 37].any())
    dm = torch.as_tensor(density(mol.nao, 10, 3), device=eng.device)
    v, vb = (eng.hartree(p, dm, fp64=True, tol=0.0) for p in (pts, bad))
    assert torch.equal(v[keep], vb[keep])
    assert bool(torch.isnan(vb[37]))
