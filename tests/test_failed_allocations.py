"""Workspaces after a failed allocation -- no GPU.

A child process runs the library's host side on a runtime without a device (tests/cpp/fake_cudart.cpp) and
lets every device allocation of a call fail in turn.  The call has to report it, and the same call again
has to succeed with the same buffers as one that never failed: a workspace left half allocated would send
null pointers to the kernels.
"""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CALLS = ["batch", "batch_grows", "batch_mixed", "solve", "solve_mixed", "solve_restart", "solve_flexible", "solve_batch",
         "solve_batch_flexible", "solve_batch_mixed", "group", "group_flexible"]


def _child(call):
    sys.path.insert(0, ROOT)
    import ifgf2d_gb300 as G
    G.load_library()
    fake = ctypes.CDLL(None)
    fake.fake_fail_at.argtypes = [ctypes.c_longlong]
    fake.fake_allocs.restype = fake.fake_live.restype = ctypes.c_longlong
    fake.fake_live.argtypes = [ctypes.c_longlong, ctypes.c_void_p]

    def live():
        v = np.zeros(4096, np.int64)
        n = fake.fake_live(v.size, v.ctypes.data)
        return v[:n].tolist()

    def prepared():
        """what the call needs before, the call, and its end"""
        def make():
            return G.ForwardMap(0.02, [G.Kite()], (), 1.0, 20.0, Np=10, patches_per_curve=64, formulation="combined")
        fm = make()
        if call.startswith("group"):
            other = make()
            for f in (fm, other):
                f.prepare(20.0, 0)
            g = G.Group([fm, other])
            b = np.ones(2 * fm.total_num_unknowns_, complex)
            return (lambda: g.solve(b, mixed=False, precond="spectral" if "flexible" in call else None)), [g, fm, other]
        fm.precomps_and_setup(20.0, 0)
        X = np.ones((fm.total_num_unknowns_, 24), complex)
        b = X[:, 0].copy()
        if call == "batch_grows":
            fm.apply_batch(X[:, :12])
        if call == "solve_restart":
            fm.gmres(b, restart=20)
        return {"batch": lambda: fm.apply_batch(X[:, :12]), "batch_grows": lambda: fm.apply_batch(X),
                "batch_mixed": lambda: fm.apply_batch(X, mixed=True), "solve": lambda: fm.gmres(b), "solve_mixed": lambda: fm.gmres(b, mixed=True),
                "solve_restart": lambda: fm.gmres(b, restart=30), "solve_flexible": lambda: fm.solve_flexible(b),
                "solve_batch": lambda: fm.gmres_batch(X[:, :4]), "solve_batch_flexible": lambda: fm.gmres_batch(X[:, :4], precond="spectral"),
                "solve_batch_mixed": lambda: fm.gmres_batch(X[:, :4], mixed=True)}[call], [fm]

    def end(owners):
        for o in owners:
            o.close()

    f, owners = prepared()
    fake.fake_fail_at(0)
    f()
    count, want = fake.fake_allocs(), live()
    assert count > 0
    f()
    assert live() == want
    end(owners)
    for i in range(1, count + 1):
        f, owners = prepared()
        fake.fake_fail_at(i)
        with pytest.raises(G.IFGF2DError):
            f()
        fake.fake_fail_at(0)
        if call == "solve_restart" and i % 2:      # the size that was there before
            owners[0].gmres(np.ones(owners[0].total_num_unknowns_, complex), restart=20)
        f()
        assert live() == want, (i, count)
        end(owners)


@pytest.fixture(scope="module")
def fake_runtime(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", os.path.join(HERE, "cpp", "fake_cudart.cpp"), "-o", so], check=True)
    return so


@pytest.mark.parametrize("call", CALLS)
def test_failed_allocation_leaves_no_half_workspace(lib, fake_runtime, call):
    r = subprocess.run([sys.executable, os.path.abspath(__file__), call], env=dict(os.environ, LD_PRELOAD=fake_runtime), capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]


if __name__ == "__main__":
    _child(sys.argv[1])
