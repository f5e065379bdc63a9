"""Admission when no memory is left for the list of tables to clear: the server's
results are those of a server that had it."""
import pytest

import failing_lib

pytestmark = pytest.mark.gpu

SERVE = """
    import hashlib
    h = hashlib.sha256()
    with ptw.Graph.rmat(12, 16, 0.57, 0.19, 0.19, seed=1, clean=True) as G, \\
            ptw.Server(G, sp=0.2, seed=3, tick_walkers=1 << 14, table_bytes=1 << 19) as srv:
        for k in range(8):
            srv.submit(k, 4000, k)
        got = srv.drain()  # every table of the arena has been used
        for k in range(8):
            srv.submit(100 + k, 4000, 100 + k)
        fake(%d, True)
        try:
            got += srv.step()
        except ptw.PTWError as e:
            print("step:", e, file=sys.stderr)
        fake(%d, False)
        got += srv.drain()
        assert sorted(r["query_id"] for r in got) == list(range(8)) + list(range(100, 108))
        for r in sorted(got, key=lambda r: r["query_id"]):
            h.update(r["names"].tobytes() + r["counts"].tobytes())
    print(h.hexdigest())
""" % (failing_lib.NO_POOL, failing_lib.NO_POOL)


def test_step_without_pool_memory(gpu, tmp_path):
    want = failing_lib.run(None, SERVE)
    got = failing_lib.run(failing_lib.build("capi.cu", tmp_path), SERVE)
    assert got == want
