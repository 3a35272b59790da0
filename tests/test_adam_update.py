"""The Adam update of the training kernels (adam_update of tc_train.cuh) against the same update
with the language's divisions and square root, bit for bit, over all the moments that training can
hold: it forms quotients and root from approximations and one residual correction each.

Compiled here from the kernels' own header.  With betas of 1 an update keeps the moments it is
given, and from a weight of 0 it returns minus the step."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "tc_train.cuh"
using epi::tc::AdamHyper;
__global__ void both(const float* m, const float* v, const float* c1, const float* c2, unsigned n, float lr, float eps,
                     float* mine, float* plain) {
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float p = 0.f, mi = m[i], vi = v[i];
        const float4 c = make_float4(c1[i], c2[i], __frcp_rn(c1[i]), __frcp_rn(c2[i]));
        const AdamHyper hp{lr, 1.f, 1.f, eps};
        epi::tc::adam_update(p, mi, vi, 0.f, epi::tc::adam_corrections(c, hp), hp);
        if (epi::tc::either_nan(p, p)) p = epi::tc::adam_exact(0.f, mi, vi, c, lr, eps);
        mine[i] = p;
        const float step = __fdiv_rn(__fmul_rn(lr, __fdiv_rn(m[i], c1[i])),
                                     __fadd_rn(__fsqrt_rn(__fdiv_rn(v[i], c2[i])), eps));
        plain[i] = __fadd_rn(0.f, -step);
    }
}
extern "C" int run(const float* h, unsigned n, float lr, float eps, float* mine, float* plain) {
    float* d = nullptr;
    const size_t b = n * sizeof(float);
    if (cudaMalloc(&d, 6 * b)) return 1;
    int rc = cudaMemcpy(d, h, 4 * b, cudaMemcpyHostToDevice);
    if (!rc) {
        both<<<1024, 256>>>(d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n, n, lr, eps, d + 4 * (size_t)n, d + 5 * (size_t)n);
        rc = cudaGetLastError();
    }
    if (!rc) rc = cudaMemcpy(mine, d + 4 * (size_t)n, b, cudaMemcpyDeviceToHost);
    if (!rc) rc = cudaMemcpy(plain, d + 5 * (size_t)n, b, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return rc;
}
"""

MIN, MAX = np.float32(2.0 ** -126), np.finfo(np.float32).max


@pytest.fixture(scope="module")
def updates(gpu, tmp_path_factory):
    from epirust_gb300 import build

    d = tmp_path_factory.mktemp("adam")
    src, so = str(d / "adam.cu"), str(d / "adam.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "-I", os.path.join(ROOT, "epirust_gb300", "csrc"), "-o", so, src], check=True, capture_output=True)
    run = C.CDLL(so).run
    run.argtypes = [C.c_void_p, C.c_uint, C.c_float, C.c_float, C.c_void_p, C.c_void_p]

    def call(m, v, t, eps, lr=1e-3):
        """Steps of the two forms for moments m, v after t steps (betas 0.9 and 0.999)."""
        t = np.asarray(t, dtype=np.float64)
        h = np.ascontiguousarray(np.stack(np.broadcast_arrays(m, v, 1 - 0.9 ** t, 1 - 0.999 ** t)).astype(np.float32))
        mine, plain = np.empty(h.shape[1], np.float32), np.empty(h.shape[1], np.float32)
        assert run(h.ctypes.data, h.shape[1], lr, eps, mine.ctypes.data, plain.ctypes.data) == 0
        return mine, plain, h
    return call


def _moments(rng, n, lo, hi):
    """v over the powers of two from lo to hi; |m| up to 7 sqrt(v), the most that one sequence of
    gradients gives both."""
    v = np.exp2(rng.uniform(lo, hi, n)).clip(max=float(MAX)).astype(np.float32)
    m = np.sqrt(v.astype(np.float64)) * np.exp2(rng.uniform(-10, 2.8, n)) * rng.choice([-1, 1], n)
    return m.astype(np.float32), v, np.floor(np.exp2(rng.uniform(0, 15, n)))


@pytest.mark.parametrize("eps", [1e-8, 1e-30, 0.0])
@pytest.mark.parametrize("lo,hi", [(-126, -93), (-93, 0), (0, 93), (93, 128)])
def test_every_normal_moment(updates, lo, hi, eps):
    m, v, t = _moments(np.random.default_rng(lo + 200), 1 << 22, lo, hi)
    mine, plain, _ = updates(m, v, t, eps)
    assert (mine.view(np.uint32) == plain.view(np.uint32)).all()


@pytest.mark.parametrize("eps", [1e-8, 0.0])
def test_subnormal_second_moments(updates, eps):
    """Below the normal numbers v / c2 is rounded to few digits; the update keeps more of them: its
    step is no further from the exact one than the plain form's (two ulps for the roundings)."""
    m, v, t = _moments(np.random.default_rng(3), 1 << 20, -149, -126)
    mine, plain, h = updates(m, v, t, eps)
    m, v, c1, c2 = h.astype(np.float64)
    exact = -(np.float64(np.float32(1e-3)) * (m / c1)) / (np.sqrt(v / c2) + np.float64(np.float32(eps)))
    assert (np.abs(mine - exact) <= np.abs(plain - exact) + 2.0 ** -22 * np.abs(exact)).all()


def test_ends_of_the_range(updates):
    """Zeros, the largest numbers and infinities; an overflowed second moment gives no step."""
    inf = np.float32(np.inf)
    cases = [(m, v, t) for m in (0.0, 1e-30, 1.0, -1e19, 1e38, -float(MAX), inf) for t in (1, 7, 30000)
             for v in (0.0, float(MIN), 1e-20, 1.0, 2.9e38, 3.1e38, float(MAX), inf)]
    m, v, t = (np.array(c) for c in zip(*cases))
    mine, plain, h = updates(m, v, t, 1e-8)
    nan = np.isnan(plain)
    assert (np.isnan(mine) == nan).all()
    finite = np.isfinite(plain)
    assert (mine[finite] == plain[finite]).all()
    with np.errstate(over="ignore"):
        gone = np.isinf(h[1]) & np.isfinite(h[0] / h[2])
    assert gone.any() and (mine[gone] == 0).all()


def _order(seed, n):
    """The rows of member `seed`'s first minibatch: Fisher-Yates from splitmix64."""
    mask, perm = (1 << 64) - 1, list(range(n))
    for i in range(n - 1, 0, -1):
        seed = (seed + 0x9E3779B97F4A7C15) & mask
        z = ((seed ^ (seed >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        j = (z ^ (z >> 31)) % (i + 1)
        perm[i], perm[j] = perm[j], perm[i]
    return perm


@pytest.mark.parametrize("eps", [1e-8, 1e-30])
@pytest.mark.parametrize("members", [1, 5, 16])
@pytest.mark.parametrize("scale", [1e6, 1e3, 1.0, 1e-6, 1e-12, 1e-16, 1e-25])
def test_first_step_of_large_and_small_gradients(gpu, scale, members, eps):
    """A first step from the handle's own gradients, by NumPy's correctly rounded operators, bit for
    bit: with output weights of `scale` the hidden layers' second moments go from 1e13 down to 1e-50,
    at the top beyond what the kernels' epilogues take directly."""
    from epirust_gb300.surrogate import Surrogate

    f, lr, eps = np.float32, np.float32(1e-3), np.float32(eps)
    rng = np.random.default_rng(4)
    net = Surrogate(in_dim=8, out_dim=120, hidden=256, hidden_layers=2, batch=128, lr=float(lr), eps=float(eps), seed=6,
                    members=members)
    p = np.atleast_2d(net.get_params()).copy()
    p[:, 8 * 256 + 256 + 256 * 256 + 256:] *= f(scale)
    net.set_params(p)
    x, t = rng.random((128, 8)).astype(f), (rng.random((128, 120)) * 0.5).astype(f)
    orders = [_order(m, 128) for m in range(members)]
    g = np.stack([np.atleast_2d(net.gradients(x[o], t[o])[1])[m] for m, o in enumerate(orders)])
    net.set_dataset(x, t)
    net.train(1, seed=0)
    one, b1, b2 = f(1), f(0.9), f(0.999)
    with np.errstate(under="ignore", invalid="ignore", divide="ignore"):
        m, v = (one - b1) * g, (one - b2) * g * g
        want = p - lr * (m / (one - b1)) / (np.sqrt(v / (one - b2)) + eps)
    got = np.atleast_2d(net.get_params())
    assert (got.view(np.uint32) == want.view(np.uint32)).all()
    net.close()
