"""Arguments on their way from Python into a C entry (csrc/launcher.cpp): order, widths and what is refused."""
import ctypes
import itertools
import os
import subprocess
import sys

import numpy
import pytest
import torch

from fms_b200.kernels import build
from fms_b200.kernels.ops import _SIGNATURES, KernelError

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
C_TYPES = {"p": "void*", "i": "int", "l": "long", "f": "float"}


def entry(tmp_path, kinds):
    """An entry of these parameters that writes each, as a double, to the address in its first, and that address."""
    source = tmp_path / "echo.c"
    names = ", ".join(f"{C_TYPES[k]} a{i}" for i, k in enumerate(kinds))
    body = "".join(f"  out[{i}] = (double){'(long)' if k == 'p' else ''}a{i};\n" for i, k in enumerate(kinds) if i)
    source.write_text(f"int echo({names}) {{\n  double* out = (double*)a0;\n{body}  return 7;\n}}\n")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "echo.so"), str(source)], check=True)
    lib = ctypes.CDLL(str(tmp_path / "echo.so"))
    address = ctypes.cast(lib.echo, ctypes.c_void_p).value
    return build.load_launcher().entry(address, kinds.replace("l", "i"), KernelError), (ctypes.c_double * len(kinds))(), lib


@pytest.mark.parametrize("kinds", ["p", "pi", "pf", "pifl", "piiiii", "piiiiii", "pfffffffi", "p" + "if" * 8, "pilfp" * 6 + "lliipp",
                                   "p" + "i" * 45])
def test_arguments_arrive_in_order(tmp_path, kinds):
    f, out, lib = entry(tmp_path, kinds)
    given = {"i": itertools.cycle((3, -5, 2 ** 31 - 1, True)), "l": itertools.cycle((-2 ** 40, 2 ** 45)),
             "p": itertools.cycle((None, 4096)), "f": itertools.cycle((0.25, -3, 1e30))}
    args = [ctypes.addressof(out)] + [next(given[k]) for k in kinds[1:]]
    assert f(*args) == 7
    single = lambda x: ctypes.c_float(x).value  # noqa: E731
    assert list(out)[1:] == [single(a) if k == "f" else float(a or 0) for k, a in zip(kinds[1:], args[1:])]


class Indexed:
    def __index__(self):
        return -9


def test_whole_numbers_that_are_no_python_int(tmp_path):
    """Whatever has an ``__index__`` is a whole number, as for ctypes; an address is an int, a tensor or None."""
    f, out, lib = entry(tmp_path, "pilf")
    at = ctypes.addressof(out)
    for a, b in ((numpy.int64(-3), numpy.int64(2 ** 40)), (numpy.uint8(5), numpy.int32(-1)), (Indexed(), torch.tensor(7)), (True, Indexed())):
        assert f(at, a, b, numpy.float32(0.5)) == 7
        assert list(out)[1:] == [float(a.__index__()), float(b.__index__()), 0.5]
    for bad in (numpy.float32(1.0), numpy.bool_(True), torch.zeros(1), torch.zeros(2, dtype=torch.int32)):
        with pytest.raises(TypeError):
            f(at, bad, 1, 1.0)
    for bad in (numpy.int64(at), Indexed()):
        with pytest.raises(TypeError):
            f(bad, 1, 1, 1.0)


def test_what_an_entry_refuses(tmp_path):
    f, out, lib = entry(tmp_path, "pif")
    at = ctypes.addressof(out)
    for args in ((at, 1), (at, 1, 1.0, 1), (at, 1.0, 1.0), (at, None, 1.0), (at, 1, None), (at, 1, "1"), (at, torch.zeros(1), 1.0)):
        with pytest.raises(TypeError):
            f(*args)
    with pytest.raises(KernelError, match="on the CPU"):
        f(torch.zeros(4), 1, 1.0)
    for kinds in ("px", "p" * 47, "p" + "f" * 9):
        with pytest.raises(ValueError):
            build.load_launcher().entry(1, kinds, KernelError)


def test_every_entry_fits():
    for name, kinds in _SIGNATURES.items():
        assert build.load_launcher().entry(1, "".join(kinds), KernelError), name


def test_a_machine_without_a_compiler_takes_what_is_built(monkeypatch):
    build.load_launcher()
    built = build.find_built(build.LAUNCHER)
    monkeypatch.delenv("CXX", raising=False)
    monkeypatch.setattr(build.shutil, "which", lambda *_: None)
    assert built is not None and build.find_built(build.LAUNCHER) == built
    with pytest.raises(build.KernelBuildError, match="no C"):
        build.compile_library(build.LAUNCHER)


@pytest.mark.parametrize("decay", ["head", "channel"])
def test_an_engine_compiles_what_its_first_prompt_will_launch(monkeypatch, decay):
    """The launcher, and the runs' kernels where a layer's prompts may go run by run: not in the middle of a request."""
    import types

    import fms_b200.parts.state_space  # noqa: F401
    from fms_b200.config.specs import MixerSpec
    from fms_b200.engine.step import Engine
    from fms_b200.parts.registry import build_mixer

    asked = []
    monkeypatch.setattr(build, "compile_many", lambda names, *_: asked.extend(names))
    options = (("vdim", 128), ("conv", 4), ("eps", 1e-5), ("decay", decay), ("decay_rank", 8), ("gate_rank", 8))
    part = build_mixer(MixerSpec("gated_delta_rule", dim=64, nheads=2, kvheads=1, head_dim=128, options=options))
    decoder = types.SimpleNamespace(kernel_libraries=part.kernel_libraries, dtype=torch.bfloat16)
    Engine._compile_what_this_model_needs(types.SimpleNamespace(decoder=decoder), True)
    assert {build.LAUNCHER, "state_scan", "sampling"} <= set(asked)
    assert ("chunk_scan" in asked) == (decay == "head")


@pytest.mark.parametrize("switch,expanded", [({}, True), ({"FMS_B200_LATENT_MMA": "0"}, False), ({"FMS_B200_ATTN_TC": "0"}, False)])
def test_the_switches_of_the_tensor_core_kernels_reach_latent_prompts(switch, expanded):
    """Each, in a process of its own: a prompt's latent attention does not take the form that the switched-off kernel makes."""
    code = ("import torch; from fms_b200.kernels import ops; from fms_b200.engine.batch import Batch; "
            "b = Batch.from_lists([0], [0], [[0] * 500], [[]], 'cpu'); "
            "print(*(bool(ops.latent_expanded_members(b, 0, 32, h, 512, 32)) for h in (128, 48)))")
    env = {**os.environ, **switch}
    out = subprocess.run([sys.executable, "-c", code], env=env, cwd=ROOT, capture_output=True, text=True, check=True)
    assert out.stdout.split() == [str(expanded), "False"]


def test_the_form_of_a_sequences_latent_attention_does_not_depend_on_what_the_others_bring():
    """Heads of 128 over a latent of 512: in steps of up to eight sequences every one is made keys and values, in larger ones those of
    23 tokens or more, whatever is cached and whatever the others bring."""
    from fms_b200.engine.batch import Batch
    from fms_b200.kernels import ops

    def members(new, before=0, heads=32):
        return ops.latent_expanded_members(Batch.from_lists(list(range(len(new))), [before] * len(new), [[0] * n for n in new], [[]] * len(new), "cpu"),
                                           0, heads, 128, 512, 32)

    assert members([2] * 8, 8000) == members([1, 2, 500, 1, 1, 1, 1, 1]) == list(range(8))
    for others in (2, 22, 500):
        assert [i for i in members([others] * 9 + [23, 22, 1, 600], 1000) if i > 8] == [9, 12]
    assert members([2, 40] * 4, heads=64) == [1, 3, 5, 7]  # eight sequences of 64 heads would not be made sooner than one is walked
    assert members([40], before=200000) == [] and members([1] * 4) == []
