"""Finding and building the native call module: installed copies, other versions of torch, machines without a compiler."""
import subprocess
import sysconfig

import pytest
import torch

from zorse_b200.ops import build
from zorse_b200.ops import sm100 as k


def test_an_installed_copy_loads_the_module_it_came_with(monkeypatch, tmp_path):
    have = build.build_fast()
    monkeypatch.setattr(build, "FAST_SRC", tmp_path / "csrc" / "host" / "fastops.cpp")
    assert build.build_fast() == have and build.build_fast(force=True) == have


def test_the_module_is_named_for_its_torch_and_its_interpreter(monkeypatch):
    have = build.build_fast()
    assert torch.__version__ in have.name and have.name.endswith(sysconfig.get_config_var("EXT_SUFFIX"))
    built = []

    def run(cmd, **kw):
        built.append(cmd)
        return subprocess.CompletedProcess(cmd, 1, "", "not now")

    monkeypatch.setattr(build.subprocess, "run", run)
    assert build.build_fast() == have and not built
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    with pytest.raises(RuntimeError, match="does not build"):
        build.build_fast()
    assert len(built) == 1


@pytest.mark.parametrize("missing", ["source", "compiler"])
def test_without_a_module_the_wrappers_take_every_call(monkeypatch, tmp_path, missing):
    from zorse_b200.ops.api import Sm100Ops

    calls = []

    class Lib:
        def __getattr__(self, name):
            return lambda *a: calls.append(name) or 0

    monkeypatch.setattr(torch, "__version__", "9.9.9")
    if missing == "source":
        monkeypatch.setattr(build, "FAST_SRC", tmp_path / "fastops.cpp")
    else:
        monkeypatch.setattr(build.shutil, "which", lambda name: None)
        monkeypatch.delenv("CXX", raising=False)
    monkeypatch.setattr(k, "_lib", Lib())
    monkeypatch.setattr(k, "_fast", None)
    monkeypatch.setattr(k, "_bf16", lambda t, name: None)
    monkeypatch.setattr(k, "status_word", lambda device=None: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(k, "_stream", lambda: None)
    with pytest.warns(RuntimeWarning, match="no native call module"):
        k._load_fast()
    assert k._fast is None
    ops = Sm100Ops()
    x, w, g = (torch.zeros(s, dtype=torch.bfloat16) for s in ((64, 128), (256, 128), (64, 256)))
    later = ops.collect()
    assert ops.act_linear_fwd(x, w, None, "relu", True)[0].shape == (64, 256)
    ops.linear_wgrad(g, x, torch.zeros(256, 128), torch.zeros(256), later=later)
    ops.finish(later)
    assert calls == ["zb_gemm_bf16", "zb_act_fwd", "zb_gemm_bf16", "zb_colsum"] and k.launch_count() >= 4
