"""Solution files cut into chunks of values (csrc/cs_text.cu): sections that
start, end or are empty at a chunk's edge (1024 values), files of two nodes and
of many chunks, problems without algebraic variables or parameters, and numbers
in and out of the fast digit range.  Reference: the host writer's text."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu

SIG = "const double* __restrict__ y, const double* __restrict__ z, const double* __restrict__ p, const double* __restrict__ th"
BC = SIG.replace("y, const double* __restrict__ z", "y0, const double* __restrict__ y1")


def _problem(cs, ny, nz, npar):
    """y' = -y, z = 0: only its sizes matter."""
    f = " ".join("f[%d] = -y[%d];" % (i, i) for i in range(ny))
    g = " ".join("g[%d] = z[%d];" % (i, i) for i in range(nz))
    nc = ny + nz + npar
    zero = "for (int i = 0; i < %d; ++i) %s[i] = 0.0; "
    Df = zero % (ny * nc, "D") + " ".join("D[%d] = -1.0;" % (i * nc + i) for i in range(ny))
    Dg = (zero % (nz * nc, "D") if nz else "") + " ".join("D[%d] = 1.0;" % (i * nc + ny + i) for i in range(nz))
    n, w = ny + npar, 2 * ny + npar
    r = " ".join("r[%d] = %s;" % (i, "y0[%d]" % i if i < ny else "p[%d]" % (i - ny)) for i in range(n))
    Dr = zero % (n * w, "D") + " ".join("D[%d] = 1.0;" % (i * w + (i if i < ny else ny + i)) for i in range(n))
    A = "__device__ __forceinline__ void "
    src = "\n".join([A + "cs_f(%s, double* f) { %s }" % (SIG, f), A + "cs_g(%s, const double a, double* g) { %s }" % (SIG, g),
                     A + "cs_Df(%s, double* D) { %s }" % (SIG, Df), A + "cs_Dg(%s, const double a, double* D) { %s }" % (SIG, Dg),
                     A + "cs_r(%s, double* r) { %s }" % (BC, r), A + "cs_Dr(%s, double* D) { %s }" % (BC, Dr)]) + "\n"
    return cs.GeneratedProblem(src, ny, nz, npar, 0, 0)


def _file(cs, t, y, z, p):
    f = lambda a: "".join(cs.io._fmt(v) + " " for v in a)  # noqa: E731
    rows = lambda a: "".join(f(r) + "\n" for r in a)  # noqa: E731
    return ("nt:\n%d\nt:\n" % len(t) + f(t) + "\nny:\n%d\ny:\n" % y.shape[1] + rows(y) + "nz:\n%d\nz:\n" % z.shape[1] + rows(z) +
            "np:\n%d\np:\n" % len(p) + f(p)).encode()


@pytest.mark.parametrize("ny,nz,npar", [(1, 0, 0), (1, 1, 2), (2, 0, 1), (3, 2, 0)])
def test_files_at_chunk_edges(ny, nz, npar):
    cs = pkg()
    N = np.array([2, 3, 255, 256, 511, 512, 1023, 1024, 1025, 2048, 3001], np.int32)
    rng = np.random.default_rng(ny * 10 + nz)
    T = int(N.sum())
    val = lambda *s: rng.standard_normal(s) * 10.0 ** rng.integers(-60, 25, s)  # noqa: E731
    t, y, z, p = val(T), val(T, ny), val(T, nz), val(len(N), npar)
    y.flat[:6] = [0.0, -0.0, 1e22, 5e-324, 2.0 ** 53, 2.0 ** -143]
    bt = cs.Batch(cs.CompiledProblem(_problem(cs, ny, nz, npar), 3), len(N))
    bt.set_guess_packed(N, t, y, z if nz else None, p if npar else None)
    text, off = bt.solution_text()
    _, ts, ys, zs, ps, _ = bt.solution_packed()  # z at the nodes, as the files hold it
    o = 0
    for b, n in enumerate(N):
        ref = _file(cs, ts[o:o + n], ys[o:o + n], zs[o:o + n], ps[b])
        assert bytes(text[off[b]:off[b + 1]]) == ref, "instance %d" % b
        o += n
