"""Allocations that fail, on the library with a stand-in for the CUDA runtime (no GPU): a build whose buffers could not be
regrown leaves a context that refuses its queries, launches nothing without buffers, and builds again once there is memory."""
import ctypes
import os
import subprocess
import sys

import pytest

from sesdf_gb300 import _build

HERE = os.path.dirname(os.path.abspath(__file__))
SECTORS, SEGMENTS = 1, 7  # words of the build's counter record


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    _build.build_cuda()
    so = str(tmp_path_factory.mktemp("fake") / "libfakecudart.so")
    subprocess.run(["gcc", "-O1", "-w", "-fno-builtin", "-shared", "-fPIC", "-o", so, os.path.join(HERE, "fake_cudart.c")], check=True)
    return so


def child(shim, body):
    head = "import ctypes, sys\nsys.path[:0] = [%r, %r]\nimport test_alloc_failure as t\n" % (os.path.dirname(HERE), HERE)
    r = subprocess.run([sys.executable, "-c", head + "t.%s(ctypes.CDLL(%r))\nprint('done')" % (body, shim)],
                       env={**os.environ, "LD_PRELOAD": shim}, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("done"), r.stdout + r.stderr


def regrow_fails(fake):
    import numpy as np
    from sesdf_gb300 import SesBuild, SesgbError
    atoms = np.random.default_rng(1).uniform(1, 40, (300, 4)).astype(np.float32)
    for word, use, graph in ((SECTORS, "build", False), (SEGMENTS, "async", False), (SECTORS, "build", True)):
        g = SesBuild(atoms, 1.4, "full", graph=graph)
        g.build()
        before = fake.fake_launches()
        fake.fake_poke(word, 10_000_000, 1)
        fake.fake_fail(2)  # the regrown buffers, and those of the next build
        try:
            g.build()
            raise AssertionError("built without memory")
        except SesgbError as e:
            assert "out of memory" in str(e)
        assert fake.fake_launches() > before  # the build that overflowed
        after = fake.fake_launches()
        for call in (g.counts, g.data, lambda: g.sdf(64, 1, 64), lambda: g.ses_area(), lambda: g.cavities(0.5), g.finish):
            try:
                call()
                raise AssertionError("a query of no build")
            except SesgbError:
                pass
        try:
            g.build() if use == "build" else g.build_async()
            raise AssertionError("built without memory")
        except SesgbError as e:
            assert "out of memory" in str(e)
        assert fake.fake_launches() == after, "kernels were launched without buffers"
        if use == "build":
            g.build()  # the memory is back
        else:
            g.build_async()
            g.finish()
        assert fake.fake_launches() > after
        g.counts()
        g.close()
    assert fake.fake_live() == 0


def query_buffers_fail(fake):
    import numpy as np
    from sesdf_gb300 import SesBuild, SesgbError
    atoms = np.random.default_rng(1).uniform(1, 40, (300, 4)).astype(np.float32)
    q = (ctypes.c_float * 3)()
    for call in (lambda g: g.sdf(ctypes.addressof(q), 1, 64), lambda g: g.sdf_backward(ctypes.addressof(q), 1, 64, 64), lambda g: g.ses_area(),
                 lambda g: g.ses_area_backward(64)):
        g = SesBuild(atoms, 1.4, "full")
        g.build()
        fake.fake_fail(1)
        try:
            call(g)
            raise AssertionError("ran without memory")
        except SesgbError as e:
            assert "out of memory" in str(e)
        call(g)
        g.close()
    assert fake.fake_live() == 0


def cavity_buffers_fail(fake):
    import numpy as np
    from sesdf_gb300 import SesBuild, SesgbError
    atoms = np.random.default_rng(1).uniform(1, 10, (50, 4)).astype(np.float32)
    box = np.array([0, 0, 0, 20, 20, 20], np.float64)
    keys = box.view(np.uint64) | np.uint64(1 << 63)  # as the bounds' kernel leaves them
    fake.fake_fill(ctypes.c_void_p(keys.ctypes.data), 48)
    g = SesBuild(atoms, 1.4, "full")
    g.build()
    first = g.cavities(1.0)
    assert len(g.cavity_labels()) == np.prod(first["dims"])
    fake.fake_fail(1)
    for call, error in ((lambda: g.cavities(0.25), "out of memory"), (g.cavity_labels, "not built"), (lambda: g.cavity_components(0), "not built")):
        try:
            call()
            raise AssertionError("labels without memory")
        except SesgbError as e:
            assert error in str(e)
    second = g.cavities(0.25)
    assert len(g.cavity_labels()) == np.prod(second["dims"])
    g.close()
    assert fake.fake_live() == 0


def mask_bytes(fake):
    # the masks of slots 64 to 127 have room for the atoms that such lists occur with: few at the usual probe radius
    import numpy as np
    from sesdf_gb300 import SesBuild
    fake.fake_bytes.restype = ctypes.c_ulonglong
    n, used = 100_000, []
    atoms = np.random.default_rng(1).uniform(1, 100, (n, 4)).astype(np.float32)
    for radius in (1.4, 2.4):
        before = fake.fake_bytes()
        SesBuild(atoms, radius, "full").close()
        used.append(fake.fake_bytes() - before)
    assert used[1] - used[0] >= 300 * n


@pytest.mark.parametrize("body", ["mask_bytes", "regrow_fails", "query_buffers_fail", "cavity_buffers_fail"])
def test_allocation_failure(shim, body):
    child(shim, body)
