"""The predictor's structs as a C and a C++ caller lay them out, against their
mirror in stonefish_gb300/abi.py (no GPU)."""
import ctypes as C

import pytest

from stonefish_gb300 import abi
from tests import test_header_compile as base


@pytest.mark.parametrize("compiler,std,suffix", [("gcc", "c11", ".c"), ("g++", "c++17", ".cpp")])
def test_predictor_structs(built_library, tmp_path, monkeypatch, compiler, std, suffix):
    structs = {"hydro_nn_predict_net": abi.NnPredictNet, "hydro_nn_predictor": abi.NnPredictor}
    monkeypatch.setattr(base, "STRUCTS", structs)
    got = base.compile_and_run(tmp_path, compiler, std, base.layout_program(), suffix)
    for cname, st in structs.items():
        assert int(got[cname]) == C.sizeof(st), cname
        for f, _ in st._fields_:
            assert int(got[f"{cname}.{f}"]) == getattr(st, f).offset, (cname, f)
