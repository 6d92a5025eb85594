"""The tiles' packed absorbed fractions against the scalar forms whose bits they
must give, for every optical width of their ranges.  The table generator checks
the scalar restatements on the host; the device runs pairs with turned signs."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fn,top", [(7, 0x3B800000), (8, 0x3D800000), (9, 0x3E800000)])
def test_packed_forms_exhaustive(mcg, fn, top):
    """Strict: equal to 1 - expf(-u), the host library's expf (fn 1, itself checked
    for every argument), or left to the full step; the latter for at most 2 % of
    the widths from 2^-24 on (the thin form's bound takes away 0.1 % of half a grid
    unit, the mid form's 0.2 %, and the exceptions are fewer).  Fast: equal to the
    scalar form of the full step (fn 5), for every width below the line."""
    import torch
    with mcg.Context(mode="strict") as ctx:
        bad = left = 0
        for a in range(0, top, 1 << 26):
            # an odd number of arguments pairs every argument with one of the
            # other parity or itself
            u = torch.arange(a, min(a + (1 << 26), top), dtype=torch.int32, device="cuda")[:-1].view(torch.float32)
            last = torch.arange(min(a + (1 << 26), top) - 3, min(a + (1 << 26), top), dtype=torch.int32,
                                device="cuda").view(torch.float32)
            for x in (u, last):
                got, ref = torch.empty_like(x), torch.empty_like(x)
                ctx.libm_eval_device(fn, x.data_ptr(), got.data_ptr(), x.numel())
                arg = x if fn == 9 else -x
                torch.cuda.synchronize()
                ctx.libm_eval_device(5 if fn == 9 else 1, arg.data_ptr(), ref.data_ptr(), x.numel())
                if fn != 9:
                    ref = 1 - ref
                nan = torch.isnan(got)
                bad += int((~nan & (got.view(torch.int32) != ref.view(torch.int32)) & ((got != 0) | (ref != 0))).sum())
                left += int((nan & (x >= 2.0 ** -24)).sum())
        assert bad == 0
        assert left <= (0 if fn == 9 else 0.02 * (top - 0x33800000))
