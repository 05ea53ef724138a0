"""The autotuner times the library's own launch shape first, keeps it where it is the
fastest, and does not return results cached for other kernels (no GPU)."""
import json

from rapt_gb300 import autotune as A
from tests.test_autotune_cpu import FakeEnsemble


class OwnShapeBest(FakeEnsemble):
    def advance(self, kind, delta):
        super().advance(kind, delta)
        c = self.config
        return {"kernel_ms": 1.0 if c["threads_per_block"] == c["blocks_per_sm"] == 0 else 2.0, "kernel_launches": 1}


def test_own_shape_is_a_candidate(tmp_path):
    assert A.candidates()[0] == dict(threads_per_block=0, blocks_per_sm=0, use_graph=0)
    best, table = A.tune(OwnShapeBest(), "gc", 1.0, key="k", path=str(tmp_path / "t.json"))
    assert best == {"threads_per_block": 0, "blocks_per_sm": 0, "use_graph": 0}
    assert table[0]["ms"] == 1.0


def test_results_of_other_kernels_are_timed_again(tmp_path):
    path = tmp_path / "t.json"
    old = {"threads_per_block": 128, "blocks_per_sm": 8, "use_graph": 0}
    for entry in ({"best": old, "table": []}, {"best": old, "table": [], "version": A.VERSION - 1}):
        path.write_text(json.dumps({"k": entry}))
        ens = OwnShapeBest()
        best, _ = A.tune(ens, "gc", 1.0, key="k", path=str(path))
        assert ens.advances == len(A.candidates()) and best["threads_per_block"] == 0
        assert A.load_cache(str(path))["k"]["version"] == A.VERSION
