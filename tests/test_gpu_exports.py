"""Tensors passed to the extension functions as they are against the same
tensors exported as DLPack capsules: same images, same refusals."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _forms():
    g = torch.Generator(device="cuda").manual_seed(5)
    w, h = 37, 23
    xyd = torch.rand(300, 3, generator=g, device="cuda") * torch.tensor([w + 4.0, h + 4.0, 2.0], device="cuda") - 1.0
    rgb = torch.rand(300, 3, generator=g, device="cuda")
    return {
        "plain": (xyd, rgb), "offset": (xyd[1:], rgb[1:]), "one": (xyd[7:8], rgb[7:8]), "none": (xyd[:0], rgb[:0]),
        "one_strided": (xyd[7:8].as_strided((1, 3), (1000, 1)), rgb[7:8]),
        "parameter": (torch.nn.Parameter(xyd, requires_grad=False), rgb),
        "negated": (torch._neg_view(torch._neg_view(xyd).clone()), rgb),
        "other_type": (xyd.double(), rgb), "rows": (xyd[::2], rgb[::2]),
        "grad": (xyd.clone().requires_grad_(True), rgb), "cpu": (xyd.cpu(), rgb.cpu()),
    }, w, h


def _outcome(fn):
    try:
        return fn()
    except Exception as e:  # noqa: BLE001 - the kind of refusal is the result
        return type(e)


@pytest.mark.parametrize("stream", ["default", "own"])
@pytest.mark.parametrize("form", ["plain", "offset", "one", "none", "one_strided", "parameter", "negated", "other_type",
                                  "rows", "grad", "cpu"])
def test_exports(form, stream, monkeypatch):
    from del_splat_dlpack import util_torch
    from del_splat_dlpack.SplatPoint import torch as P

    forms, w, h = _forms()
    xyd, rgb = forms[form]
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.default_stream() if stream == "default" else torch.cuda.Stream()):
        got = _outcome(lambda: P.rasterize_pix_zbuffer(xyd, rgb, (w, h)))
        got_pix = _outcome(lambda: P.rasterize_pix(xyd, rgb, (w, h)))
        with monkeypatch.context() as m:
            m.setattr(util_torch, "to_kernel", util_torch.to_dlpack_safe)
            want = _outcome(lambda: P.rasterize_pix_zbuffer(xyd, rgb, (w, h)))
            want_pix = _outcome(lambda: P.rasterize_pix(xyd, rgb, (w, h)))
        torch.cuda.synchronize()
    for a, b in ((got, want), (got_pix, want_pix)):
        if isinstance(b, torch.Tensor):
            assert isinstance(a, torch.Tensor) and torch.equal(a, b)
        else:
            assert a is b
