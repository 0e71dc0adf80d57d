"""The tuner's cache answers only for the kernels, the kinds of block and the candidates it timed."""
import numpy as np
import torch

from wmles_jax_b200 import Block, KEP, Mesh
from wmles_jax_b200 import autotune as A


def _case(twist):
    x, y, z = np.meshgrid(*(np.linspace(0.0, 1.0, m) for m in (5, 6, 7)), indexing="ij")
    return Mesh([Block("b", np.stack([x + twist * z, y, z]))]), None, dict(scheme=KEP(4), sgs="wale"), None


def test_key_knows_library_and_kind_of_block(tmp_path, monkeypatch):
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda *a: "B200")
    lib = tmp_path / "lib.so"
    lib.write_bytes(b"one")
    monkeypatch.setattr("wmles_jax_b200._native.LIB_PATH", str(lib))
    first = A.key_for([_case(0.0)], "mixed")
    assert first == A.key_for([_case(0.0)], "mixed")
    assert first != A.key_for([_case(0.1)], "mixed")                  # the same extents by other kernels
    lib.write_bytes(b"two")
    assert first != A.key_for([_case(0.0)], "mixed")
    # of several blocks, which is of which kind counts
    dims = [(4, 4, 4), (8, 8, 8)]
    keys = {A.workload_key(dims, "fp64", "KEP4", "wale", "B200", e, "v") for e in ((0, 0), (0, 1), (1, 0), (1, 1))}
    assert len(keys) == 4
    assert A.workload_key(dims, "fp64", "KEP4", "wale", "B200", (0, 1)) == \
        A.workload_key(dims[::-1], "fp64", "KEP4", "wale", "B200", (1, 0))


def test_entry_without_a_candidate_is_no_answer(tmp_path):
    path = str(tmp_path / "tiles.json")
    A.store("k", {"tile": 3, "ms_per_step": {"0": 2.0, "1": 3.0, "2": 4.0, "3": 1.0}}, path)     # before -1 was one
    assert A.lookup("k", "mixed", path=path) is None
    assert A.lookup("k", "mixed", (0, 3), path) == (3, {0: 2.0, 1: 3.0, 2: 4.0, 3: 1.0})
    A.store("k", {"tile": -1, "ms_per_step": {"-1": 0.5, "0": 2.0, "1": 3.0, "2": 4.0, "3": 1.0}}, path)
    assert A.lookup("k", "mixed", path=path)[0] == -1
    assert A.lookup("j", "mixed", path=path) is None
