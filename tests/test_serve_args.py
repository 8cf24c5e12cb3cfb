"""What a server adds to its requests' arguments."""
import types

import pytest

from equelle_b200 import serve


@pytest.mark.parametrize("slots,given,want", [(1, [], []), (2, [], ["linsolver_pdl=0"]), (32, [], ["linsolver_pdl=0"]),
                                              (32, ["linsolver_pdl=1"], ["linsolver_pdl=1"])])
def test_early_start_is_off_for_requests_that_share_the_gpu(monkeypatch, slots, given, want):
    """Unless the request says otherwise, kernels wait for each other's end
    where other requests can use the SMs."""
    seen = []

    def run(program, args, allow_failure=False):
        seen.append(list(args))
        return types.SimpleNamespace(error=b"", stats=types.SimpleNamespace(device_bytes_peak=0))

    monkeypatch.setattr(serve.simrun, "run", run)
    reqs = [serve.Request(k, "heateq", 8, 8, 1, 0, args=["nx=8", *given]) for k in range(3)]
    serve.Server(slots=slots).run(reqs, realtime=False)
    assert len(seen) == 3
    for args in seen:
        assert [a for a in args if a.startswith("linsolver_pdl=")] == want and args[0] == "nx=8"
    assert all(r.args == ["nx=8", *given] for r in reqs)
