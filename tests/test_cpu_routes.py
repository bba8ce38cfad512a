"""The checks that decide whether a fused kernel may stand in for modules or torch operations."""
import pytest
import torch
from torch import nn
from torch.autograd import forward_ad
from torch.utils._python_dispatch import TorchDispatchMode

from mojodiffusion_b200.models.layers import RMSNorm, globally_hooked, own_parameters, runs_as_defined
from mojodiffusion_b200.ops import functional, native


def _norm():
    return RMSNorm(16, 1e-6, torch.float32)


def test_plain_module_runs_as_defined():
    m = _norm()
    assert runs_as_defined(m, RMSNorm) and own_parameters(m, RMSNorm)["weight"] is m.weight
    h = m.register_forward_hook(lambda *a: None)
    h.remove()
    assert runs_as_defined(m, RMSNorm)


@pytest.mark.parametrize("change", ["hook", "pre-hook", "subclass", "other class", "forward", "parametrised"])
def test_changed_module_does_not(change):
    m = _norm()
    if change == "hook":
        m.register_forward_hook(lambda *a: None)
    elif change == "pre-hook":
        m.register_forward_pre_hook(lambda *a: None)
    elif change == "subclass":
        m = type("Scaled", (RMSNorm,), {})(16, 1e-6, torch.float32)
    elif change == "other class":
        m = nn.Identity()
    elif change == "forward":
        m.forward = lambda x: x
    else:
        nn.utils.parametrize.register_parametrization(m, "weight", nn.Identity())
    assert own_parameters(m, RMSNorm) is None and not runs_as_defined(m, RMSNorm)


def test_global_hooks_count():
    for register in (nn.modules.module.register_module_forward_hook, nn.modules.module.register_module_forward_pre_hook):
        h = register(lambda *a: None)
        try:
            assert globally_hooked() and not runs_as_defined(_norm(), RMSNorm)
        finally:
            h.remove()
        assert not globally_hooked()


def test_direct_sees_transforms_modes_and_subclasses():
    t = torch.ones(3, 2)
    assert native.direct(t, nn.Parameter(t))
    seen = []
    torch.func.vmap(lambda r: (seen.append(native.direct(r)), r)[1])(t)
    torch.func.jvp(lambda r: (seen.append(native.direct(r)), r)[1], (t,), (t,))
    torch.func.grad(lambda r: (seen.append(native.direct(r)), r.sum())[1])(t)
    with forward_ad.dual_level():
        seen.append(native.direct(t))
    with TorchDispatchMode():
        seen.append(native.direct(t))
    seen.append(native.direct(t, t.as_subclass(type("Sub", (torch.Tensor,), {}))))
    torch.jit.trace(lambda r: (seen.append(native.direct(r)), r + 1)[1], t, check_trace=False)
    assert seen == [False] * 7 and native.direct(t)


def test_wide_attention_rule():
    pays = functional._wide_pays
    assert pays(1, 16384, 16384, 512) and pays(3, 5429, 5429, 512) and pays(1, 33, 9000, 512)
    # widths that the library has a tiled kernel for; many small samples; a handful of keys
    assert not any((pays(1, 16384, 16384, 256), pays(64, 64, 64, 512), pays(16, 256, 256, 512), pays(1, 4096, 77, 512), pays(1, 16384, 256, 512)))


@pytest.mark.parametrize("known", [True, False])
def test_forced_reference_follows_the_environment(monkeypatch, known):
    """Set, removed, or in another mapping put in the place of os.environ; also where the standard mapping is not of the known kind."""
    import os
    assert native._Environ is type(os.environ)
    if not known:
        monkeypatch.setattr(native, "_Environ", None)

    class OnGpu:
        is_cuda = True
    monkeypatch.setattr(native, "_loaded", True)
    monkeypatch.delenv("MDB200_FORCE_REFERENCE", raising=False)
    assert native.use_native(OnGpu())
    monkeypatch.setenv("MDB200_FORCE_REFERENCE", "1")
    assert not native.use_native(OnGpu())
    monkeypatch.setenv("MDB200_FORCE_REFERENCE", "0")
    assert native.use_native(OnGpu())
    monkeypatch.setattr(os, "environ", {})
    assert native.use_native(OnGpu())
    monkeypatch.setattr(os, "environ", {"MDB200_FORCE_REFERENCE": "1"})
    assert not native.use_native(OnGpu())
