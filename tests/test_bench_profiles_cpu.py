"""bench.py's DRAM traffic comes from a committed counter summary of the kernel
that ran: there is one for every engine candidate, with the line it reads."""
import importlib.util
import pathlib

import pytest

from comcot_b200 import _lib

ROOT = pathlib.Path(__file__).resolve().parents[1]


def _bench():
    spec = importlib.util.spec_from_file_location("bench_under_test", ROOT / "bench.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.mark.parametrize("kind,key", [("linear", "traffic_bytes_per_launch"),
                                      ("ensemble", "traffic_bytes_per_member_launch")])
def test_every_candidate_has_a_summary(kind, key):
    bench = _bench()
    for v in range(_lib.load().gc_engine_num_candidates()):
        name = bench.profile_name(kind, v)
        traffic = bench.profiled_traffic(name, key)
        assert traffic is not None and traffic > 0, (v, name)
