"""The host path around the kernels, without a GPU: what happens after a failed native call, and how a replaced parameter is noticed."""
import pytest
import torch

from matmulfreellm_b200 import _build, _lib, kernels


@pytest.fixture(scope="module", autouse=True)
def built():
    _build.build_library()
    _build.build_native()


def test_failed_native_call_clears_the_workspaces(monkeypatch):
    """A failed launch may leave partial sums in the split-K workspaces, which the kernels expect zeroed: they are cleared before
    the error is raised, on the native path as on the ctypes one; refused arguments (nothing was launched) clear nothing."""
    from matmulfreellm_b200.engine import FusedRunner

    class Failing:
        code = -4

        def bitlinear(self, *args):
            raise _lib.MMFreeError("mmf_bitlinear", self.code, "launch failed")

        chain_forward = bitlinear

    cleared = []
    monkeypatch.setattr(kernels, "_rezero_workspaces", lambda: cleared.append(1))
    monkeypatch.setattr(_lib, "native", Failing)
    pw = kernels.PackedWeight(torch.zeros(1), torch.zeros(1), 1, 64)
    with pytest.raises(_lib.MMFreeError, match="launch failed"):
        kernels.bitlinear_forward(torch.zeros(1, 64), None, pw, 1e-6)
    assert len(cleared) == 1
    runner = object.__new__(FusedRunner)
    runner._native, runner.chain, runner.device = Failing(), None, torch.device("cpu")
    with pytest.raises(_lib.MMFreeError, match="launch failed"):
        runner.forward(None, None, [], False)
    assert len(cleared) == 2
    monkeypatch.setattr(Failing, "code", -3)
    with pytest.raises(_lib.MMFreeError):
        kernels.bitlinear_forward(torch.zeros(1, 64), None, pw, 1e-6)
    with pytest.raises(_lib.MMFreeError):
        runner.forward(None, None, [], False)
    assert len(cleared) == 2


@pytest.mark.parametrize("n", [16, 300, 5000])
def test_replaced_parameter_is_noticed_where_memory_is_reused(n):
    """A parameter that is dropped and replaced changes the watch even where the allocator hands out the same addresses again, by
    assignment of the parameter and of its .data; what is not touched does not."""
    native = _lib.native()
    for _ in range(200):
        slots = {"w": torch.nn.Parameter(torch.zeros(n))}
        watch = native.watch([(slots, "w")])
        assert native.unchanged(watch)
        del slots["w"]
        slots["w"] = torch.nn.Parameter(torch.ones(n))
        assert not native.unchanged(watch)
        watch = native.watch([(slots, "w")])
        slots["w"].data = torch.empty(0)
        slots["w"].data = torch.full((n,), 2.0)
        assert not native.unchanged(watch)
        watch = native.watch([(slots, "w"), (slots, "absent")])
        assert native.unchanged(watch)
        with torch.no_grad():
            slots["w"].add_(1)
        assert not native.unchanged(watch)


def test_watch_does_not_keep_a_dropped_parameter():
    import weakref
    slots = {"w": torch.nn.Parameter(torch.zeros(8))}
    watch = _lib.native().watch([(slots, "w")])
    gone = weakref.ref(slots.pop("w"))
    assert gone() is None and not _lib.native().unchanged(watch)


def test_replaced_norm_weight_is_noticed_where_memory_is_reused():
    from matmulfreellm_b200.ops.fusedbitnet import BitLinear
    lin = BitLinear(64, 128).bfloat16()
    for i in range(200):
        lin.norm.weight = None
        lin.norm.weight = torch.nn.Parameter(torch.full((64,), float(i % 7), dtype=torch.bfloat16))
        assert torch.equal(lin.norm_weight_f32(), torch.full((64,), float(i % 7)))
    with torch.no_grad():
        lin.norm.weight.add_(1)
    assert torch.equal(lin.norm_weight_f32(), lin.norm.weight.float())
    assert lin.norm_weight_f32() is lin.norm_weight_f32()


def test_a_step_that_gave_up_clears_the_workspaces(monkeypatch):
    """The report that a step gave up waiting clears its status word, wherever it is raised; no step has given up here, so the real look at
    the words raises nothing."""
    from matmulfreellm_b200.engine import FusedRunner
    for index in (0, 63, 64, -1):
        _lib.native().check_gave_up(index)
    _lib.native().take_gave_up()

    class GaveUp:
        def check_gave_up(self, *args):
            raise _lib.MMFreeError("mmf_decode_step", _lib.ERR_TIMEOUT, "gave up")

        chain_forward = check_gave_up

        def take_gave_up(self):
            pass

    cleared = []
    monkeypatch.setattr(kernels, "_rezero_workspaces", lambda: cleared.append(1))
    monkeypatch.setattr(_lib, "native", GaveUp)
    with pytest.raises(_lib.MMFreeError, match="MMF_ERR_TIMEOUT"):
        kernels.raise_if_gave_up(torch.device("cuda", 0))
    assert len(cleared) == 1
    runner = object.__new__(FusedRunner)
    runner._native, runner.chain, runner.device = GaveUp(), None, torch.device("cpu")
    with pytest.raises(_lib.MMFreeError, match="MMF_ERR_TIMEOUT"):
        runner.forward(None, None, [], False)
    assert len(cleared) == 2
