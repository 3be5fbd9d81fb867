"""The FFT entry point over every line length it accepts (2 to 8192 points: 32 to 4096 in registers,
the others one line per CTA), one to three axes, both directions and precisions, against torch.fft in
FP64.  A transform of N points rounds each value log2(N) times, so the relative error of the whole
array stays below 4 eps log2(N), eps half an ulp of the precision."""
import ctypes as C
import math

import pytest

from zinq_b200 import _abi

pytestmark = pytest.mark.gpu

SHAPES = ([(1, 1 << k) for k in range(1, 14)] + [(2, 1 << k) for k in range(1, 13)] + [(3, 1 << k) for k in range(1, 9)])


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("sign", [-1, 1])
@pytest.mark.parametrize("d,n", SHAPES)
def test_fft_matches_torch(d, n, sign, precision):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(31 * n + d)
    x = torch.view_as_complex(torch.randn([n] * d + [2], generator=g, device="cuda", dtype=torch.float64))
    if precision == "fp32":
        x = x.to(torch.complex64).to(torch.complex128)
    y = x.to(torch.complex64 if precision == "fp32" else torch.complex128).contiguous()
    if y.data_ptr() == x.data_ptr():
        y = y.clone()
    lib, plan = _abi.load(), C.c_void_p()
    _abi.check(lib.zqd_fft_plan_create(d, (C.c_int * d)(*[n] * d), sign, _abi.PRECISION[precision], C.byref(plan)))
    _abi.check(lib.zqd_fft_execute(plan, C.c_void_p(y.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    lib.zqd_fft_destroy(plan)
    ref = torch.fft.fftn(x) if sign < 0 else torch.fft.ifftn(x)
    err = float((y.to(torch.complex128) - ref).norm() / ref.norm())
    eps = 2.0 ** -53 if precision == "fp64" else 2.0 ** -24
    assert err <= 4 * eps * max(1.0, math.log2(float(n) ** d)), err
