"""Stores of the GEMM kernels: nothing outside the result is written, whatever its width, stride and alignment."""
import pytest
import torch

from multimesh_jax_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


# widths that end inside a 16-byte vector, on one, inside a 32- / 64-column step and inside a 256-column tile
@pytest.mark.parametrize("N", [8, 10, 40, 72, 250, 264, 516])
@pytest.mark.parametrize("M", [40, 333])
@pytest.mark.parametrize("dtype,accumulate", [(torch.bfloat16, False), (torch.float32, False), (torch.float32, True),
                                              (torch.bfloat16, True)])
@pytest.mark.parametrize("pair", [None, True, False])
def test_store_stays_inside_the_result(M, N, dtype, accumulate, pair):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(M, 200, device="cuda", generator=g).bfloat16()
    b = torch.randn(N, 200, device="cuda", generator=g).bfloat16()
    for pitch, shift in ((-(-N // 8) * 8, 0), (-(-N // 8) * 8 + 8, 0), (N + 3, 1)):     # aligned, strided, misaligned
        flat = torch.full((M * pitch + 8 + shift,), 3.0, device="cuda", dtype=dtype)
        out = flat[shift:shift + M * pitch].view(M, pitch)[:, :N]
        want = a.float() @ b.float().t() + (3.0 if accumulate else 0.0)
        K.gemm(a, b, out=out, accumulate=accumulate, pair=pair)
        assert K.read_status() == 0
        # fp32 sums of 200 products in another order: 200 * 2^-24 of the sum of magnitudes; bf16 adds 2^-9 of the value
        scale = (a.float().abs() @ b.float().abs().t()).max().item()
        tol = 200 * 2.0 ** -24 * scale + (2.0 ** -8 * want.abs().max().item() if dtype == torch.bfloat16 else 0.0)
        assert (out.float() - want).abs().max().item() <= tol
        rest = flat.clone()
        rest[shift:shift + M * pitch].view(M, pitch)[:, :N] = 3.0
        assert (rest == 3.0).all()


def test_a_thread_that_never_touched_the_device_can_launch():
    import threading
    a, b = torch.randn(64, 128, device="cuda").bfloat16(), torch.randn(256, 128, device="cuda").bfloat16()
    out, seen = torch.empty(64, 256, device="cuda", dtype=torch.bfloat16), []
    torch.cuda.synchronize()

    def work():
        try:
            K.gemm(a, b, out=out, pair=False)
        except Exception as e:  # noqa: BLE001 - reported below, in the test's own thread
            seen.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert not seen, seen
    # 128 products: 2^-8 of a value for its rounding to bf16
    err = ((out.float() - a.float() @ b.float().t()).norm() / out.float().norm()).item()
    assert err <= 2.0 ** -8
