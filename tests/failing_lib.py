"""A build of the library in which chosen CUDA calls of one source can be made to
fail or to finish late (failing_calls.cuh), for tests of what follows then."""
import os
import subprocess
import sys
import textwrap

from ptwalker_gb300 import _build

HERE = os.path.dirname(os.path.abspath(__file__))
NO_POOL, NO_CLUSTERS, LATE_COPIES = 0, 1, 2


def build(source, out_dir):
    """The library with `source` compiled behind failing_calls.cuh; the other
    objects are the library's own."""
    _build.build()
    obj = os.path.join(str(out_dir), source.replace(".cu", ".o"))
    so = os.path.join(str(out_dir), "libptw_failing.so")
    objs = [obj if s == source else os.path.join(_build.OUT, "obj", s.replace(".cu", ".o")) for s in _build.SOURCES]
    for cmd in ([_build._nvcc(), *_build.ARCH, *_build.NVCC_FLAGS, "-include", os.path.join(HERE, "failing_calls.cuh"),
                 "-c", os.path.join(_build.CSRC, source), "-o", obj],
                [_build._nvcc(), *_build.ARCH, "-shared", "-o", so, *objs, "-Xcompiler", "-fPIC"]):
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
    return so


def run(so, code, timeout=300):
    """Runs `code` in a child process on library `so` (the normal one if None):
    `ptw` is the package, `fake(what, on)` the switch.  Returns its output."""
    head = textwrap.dedent("""
        import sys
        sys.path.insert(0, %r)
        import numpy as np
        from ptwalker_gb300 import _build, _capi
        so = %r
        if so:
            _build.SO, _build.up_to_date = so, lambda: True
        import ptwalker_gb300 as ptw
        fake = (lambda what, on: ptw.load_library().ptw_test_fake(what, int(on))) if so else (lambda what, on: None)
    """) % (os.path.dirname(HERE), so)
    r = subprocess.run([sys.executable, "-c", head + textwrap.dedent(code)], capture_output=True, text=True,
                       timeout=timeout)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
