"""The library's host code on the CPU, against a stand-in for the CUDA runtime
(fake_cudart.c, preloaded into a child process): how much scratch a call
takes, which calls allocate at all, and what a launch needs to have been set
on its device.  No kernel runs, and none needs a GPU."""
import ctypes as C
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
F64, F32 = 0, 1   # HFB_F64, HFB_F32


# ------------------------------------------------------------- scenarios ----
# each runs in a child process with the stand-in preloaded; its return value
# is printed
class _Lib:
    def __init__(self):
        sys.path.insert(0, os.path.join(os.path.dirname(HERE), "jax-hfbfft_b200", "hfb"))
        import types
        sys.modules.setdefault("torch", types.ModuleType("torch"))   # only the prototypes are needed
        import _lib
        self.hfb, self.fake = _lib.load(), C.CDLL(None)
        self.fake.fake_bytes.restype = C.c_ulonglong
        self.fake.fake_widest_cluster.restype = self.fake.fake_allocs.restype = C.c_long
        self.fake.fake_launches.restype = C.c_long
        assert self.fake.fake_launches() == 0
        self.mem = C.create_string_buffer(1 << 16)
        self.p = (C.addressof(self.mem) + 255) & ~255   # any device address: nothing is read

    def ctx(self, n):
        h = C.c_void_p()
        assert self.hfb.hfb_ctx_create(n, n, n, 1.0, 1.0, 1.0, 0, 0, C.byref(h)) == 0
        return h

    def add_density(self, ctx, prec, nst, nneut):
        p = self.p
        return self.hfb.hfb_add_density(ctx, prec, nst, nneut, p, p, p, p, p, 1.0, p, p, p, p, p, p, None, None, None)

    def pair_density(self, ctx, prec, nst, nneut):
        return self.hfb.hfb_pair_density(ctx, prec, nst, nneut, *[self.p] * 10, None)


def density_scratch():
    lib = _Lib()
    ctx = lib.ctx(16)
    b0 = lib.fake.fake_bytes()
    rc = [lib.add_density(ctx, F64, 601, 1)]
    taken, a0 = lib.fake.fake_bytes() - b0, lib.fake.fake_allocs()
    for prec in (F64, F32):
        for nst, nneut in ((20, 10), (300, 299), (900, 450)):
            rc += [lib.add_density(ctx, prec, nst, nneut), lib.pair_density(ctx, prec, nst, nneut)]
    return rc, taken, lib.fake.fake_allocs() - a0


def nyquist_scratch():
    lib = _Lib()
    ctx, p = lib.ctx(16), lib.p
    a0 = lib.fake.fake_allocs()
    rc = [lib.hfb.hfb_nyquist_apply(ctx, prec, 40, 20, p, p, p, p + 256, None) for prec in (F64, F32)]
    applied = lib.fake.fake_allocs() - a0
    rc += [lib.hfb.hfb_nyquist_pair(ctx, F64, 5, 3, p, p, p, p, None)]
    a0 = lib.fake.fake_allocs()
    rc += [lib.hfb.hfb_nyquist_pair(ctx, prec, 400, 3, p, p, p, p, None) for prec in (F64, F32)]
    return rc, applied, lib.fake.fake_allocs() - a0


def hpsi_f64_scratch():
    lib = _Lib()
    ctx, p = lib.ctx(48), lib.p
    a0 = lib.fake.fake_allocs()
    rc = [lib.hfb.hfb_hpsi(ctx, F64, p, nst, 1, p, p, p, p, p, p, None) for nst in (1, 60, 236)]
    return rc, lib.fake.fake_allocs() - a0


def clusters():
    lib = _Lib()
    p, out = lib.p, []
    eigh = lambda ctx, n: lib.hfb.hfb_eigh_near_diagonal(ctx, 2, n, n, p, p, p, None)  # noqa: E731
    for device in (0, 1):
        lib.fake.fake_set_device(device)
        ctx = lib.ctx(8)
        out += [(eigh(ctx, 80), lib.fake.fake_widest_cluster()), (eigh(ctx, 100), lib.fake.fake_widest_cluster())]
    lib.fake.fake_cluster_places(0)          # no place for a cluster of 16
    out.append((eigh(lib.ctx(8), 100), lib.fake.fake_widest_cluster()))
    lib.fake.fake_attribute_fails(1)         # the opt-in is refused
    out.append((eigh(lib.ctx(8), 100), lib.fake.fake_widest_cluster()))
    return out


def hpsi_alignment():
    lib = _Lib()
    p, out = lib.p, []
    from _lib import GrstepArgs
    ctx = lib.ctx(24)

    def hpsi(kind, prec, psi, pout, mf):
        lib.hfb.hfb_set_hpsi_kernel(ctx, kind)
        n0 = lib.fake.fake_launches()
        r = lib.hfb.hfb_hpsi(ctx, prec, p, 2, 1, psi, None, None, pout, mf, None, None)
        return r, lib.fake.fake_launches() - n0 > 0

    for kind in (0, 1, 2):
        out.append([hpsi(kind, F32, p, p + 8, p), hpsi(kind, F32, p + 8, p, p), hpsi(kind, F32, p, p + 8, None),
                    hpsi(kind, F32, p, p, p + 8)])
    out.append([hpsi(0, F64, p, p, p), hpsi(0, F64, p + 8, p, p)])
    steps = []
    for off in ("psi", "hampsi", "hmfpsi", None):
        a = GrstepArgs()
        for f, t in a._fields_:
            if t is C.c_void_p:
                setattr(a, f, p + 8 * (f == off))
        a.nst, a.nneut, a.e0dmp = 2, 1, 100.0
        n0 = lib.fake.fake_launches()
        steps.append((lib.hfb.hfb_grstep(ctx, F32, C.byref(a), None), lib.fake.fake_launches() - n0 > 0))
    return out, steps


# ----------------------------------------------------------------- tests ----
@pytest.fixture(scope="module")
def child(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-I", "/usr/local/cuda/include",
                    os.path.join(HERE, "fake_cudart.c"), "-o", so], check=True)
    sys.path.insert(0, os.path.join(os.path.dirname(HERE), "jax-hfbfft_b200"))
    import build
    if not os.path.exists(build.OUT):
        build.build()

    def run(name):
        env = {k: v for k, v in os.environ.items() if not k.startswith("HFB_")}
        env["LD_PRELOAD"] = so
        r = subprocess.run([sys.executable, os.path.abspath(__file__), name], env=env, capture_output=True, text=True,
                           timeout=120)
        assert r.returncode == 0, r.stderr
        import ast
        return ast.literal_eval(r.stdout.strip().splitlines()[-1])
    return run


def test_density_scratch_does_not_grow_with_the_states(child):
    """At most one partial tile per CTA (four an SM) and one per (axis,
    isospin, tile), whatever the state counts: at 16^3, with tiles of 16 lines
    and 7 fields, (4 * 148 + 6 * 16) * 7 * 16 * 16 * 8 bytes and the arena's
    eighth on top, 11.1 MB.  A later call with other counts, in the other
    precision or for pairs finds the buffer large enough."""
    rc, taken, later = child("density_scratch")
    assert set(rc) == {0}
    assert taken <= 12e6
    assert later == 0


def test_nyquist_calls_do_not_allocate_with_the_states(child):
    """hfb_nyquist_apply takes no scratch, so it may be a context's first call
    inside a capture; hfb_nyquist_pair's has one size."""
    rc, applied, later = child("nyquist_scratch")
    assert set(rc) == {0}
    assert applied == 0
    assert later == 0


def test_hpsi_f64_takes_no_scratch(child):
    """With few planes a CTA and with many (the table of line means): what a
    capture holds is not moved by a later single-precision call."""
    rc, allocs = child("hpsi_f64_scratch")
    assert set(rc) == {0}
    assert allocs == 0


def test_refinement_cluster_on_every_device(child):
    """The opt-in to 16 CTAs (from 81 states on) holds for one device; where it
    is refused or such a cluster has no place, 8 do."""
    assert child("clusters") == [(0, 8), (0, 16)] * 2 + [(0, 8), (0, 8)]


def test_misaligned_states_are_refused_before_any_launch(child):
    """16 bytes for psi and for the array that takes h psi; any address of a
    float2 for the other outputs and for the kernel on CUDA cores."""
    ok, bad = (0, True), (1, False)
    out, steps = child("hpsi_alignment")
    assert out[0] == out[1] == [ok, bad, bad, bad]
    assert out[2] == [ok, ok, ok, ok]
    assert out[3] == [ok, bad]
    assert steps == [bad, bad, bad, ok]


if __name__ == "__main__":
    print(repr(globals()[sys.argv[1]]()))
