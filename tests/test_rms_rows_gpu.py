"""RMSNorm with a row in registers (widths up to 4096) and above: the widths' first, odd and last, rows around a CTA's four."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [128, 384, 1024, 2048, 2176, 4096, 4224])
@pytest.mark.parametrize("rows", [1, 3, 5, 601])
def test_rms_norm_rows(built_lib, rows, channels):
    from pratchya_b200._nnx_impl._glue import rms_norm
    g = torch.Generator(device="cuda").manual_seed(rows + channels)
    x = torch.randn(rows, channels, generator=g, device="cuda")
    scale = torch.randn(channels, generator=g, device="cuda")
    got = rms_norm(x, scale, 1e-6)
    want = x.double() * torch.rsqrt((x.double() ** 2).mean(-1, keepdim=True) + 1e-6) * scale.double()
    # a lane adds 3 + channels / 128 positive terms and five levels of lanes follow; half of that on the root, and eight more roundings
    bound = (0.5 * (8 + channels / 128) + 8) * 2.0 ** -24
    assert ((got.double() - want).abs() <= bound * want.abs()).all()


@pytest.mark.parametrize("channels", [128 * q for q in range(1, 33)])
def test_both_forms_give_the_same_bits(built_lib, diag_lib, monkeypatch, channels):
    """The diagnostics build's switch gives every width to the kernel that loops over a row."""
    rows = 37
    g = torch.Generator(device="cuda").manual_seed(channels)
    x = torch.randn(rows, channels, generator=g, device="cuda") * torch.randn(rows, 1, generator=g, device="cuda").exp()
    scale = torch.randn(channels, generator=g, device="cuda")

    def run(lib):
        y, inv = torch.empty_like(x), torch.empty(rows, device="cuda")
        assert lib.pb_rms_norm(x.data_ptr(), scale.data_ptr(), rows, channels, 1e-6, y.data_ptr(), inv.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        return y, inv

    want = run(built_lib)
    assert all(torch.equal(a, b) for a, b in zip(run(diag_lib), want))
    monkeypatch.setenv("PB_RMS_LOOP", "1")
    assert all(torch.equal(a, b) for a, b in zip(run(diag_lib), want))
