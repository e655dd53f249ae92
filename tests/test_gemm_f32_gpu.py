"""gemm_f32 on the GPU against the same product in 64 bits, where its tiles of 16, 32 and 64 rows, its shares of the depth and its
splits over clusters begin and end. A sum of K fp32 products in any order is off by at most K 2^-24 sum |x w|; what the epilogues add
(row factor, stream) rounds a few times more."""

import ctypes

import pytest
import torch

from nanochat_b200.native import MAX_STREAMS, GemmRs, check, cuda_library, stream

pytestmark = pytest.mark.gpu
STORE, F32, GEGLU, STREAM, STREAMS, SWIGLU = 0, 3, 5, 6, 7, 8
CASES = [(rows, 192, 320) for rows in (1, 15, 16, 17, 31, 32, 33, 64, 65, 100)] + \
        [(1, 64, 64), (64, 64, 64), (300, 64, 64), (3, 4160, 128), (17, 64, 1984), (300, 768, 1920), (300, 3840, 768), (129, 2752, 576), (1000, 128, 512)]


@pytest.mark.parametrize("rows, N, K", CASES)
@pytest.mark.parametrize("epilogue", [STORE, F32, GEGLU, STREAM, STREAMS, SWIGLU])
def test_product_and_epilogue(rows, N, K, epilogue):
    gen = torch.Generator(device="cuda").manual_seed(rows * 7919 + N * 31 + K + epilogue)

    def rand(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    x, w, parts = rand(rows, K), rand(N, K) * K ** -0.5, 5
    ss, gain, status = rand(rows, parts).abs(), rand(N), torch.zeros(1, dtype=torch.int32, device="cuda")
    a = GemmRs(x=x.data_ptr(), w=w.data_ptr(), rows=rows, N=N, K=K, n_store=N - 3, epilogue=epilogue, scale=0.5, eps=1e-5, norm_count=K, mult=0.25,
               ss=ss.data_ptr(), ss_parts=parts, status=status.data_ptr())
    columns = N // 2 if epilogue in (GEGLU, SWIGLU) else N
    y = torch.full((rows, columns + 3), 7.0, device="cuda")  # an odd stride
    a.y, a.ldy = y.data_ptr(), columns + 3
    streams = 3 if epilogue == STREAMS else 1
    h = rand(rows, streams, N)
    old, x_next, ss_next = h.double(), torch.zeros(rows, N, device="cuda"), torch.zeros(rows, N // 64, device="cuda")
    if epilogue in (STREAM, STREAMS):
        a.h, a.gain, a.x_next, a.ss_next = h.data_ptr(), gain.data_ptr(), x_next.data_ptr(), ss_next.data_ptr()
        a.streams = streams
        for s in range(streams):
            a.in_[s], a.out[s] = 0.3 + s, 1.0 - 0.4 * s
            for t in range(streams):
                a.mix[s * MAX_STREAMS + t] = 0.5 * (s == t) + 0.1 * s - 0.2 * t
    check(cuda_library("gemm_f32").gemm_f32_rs(ctypes.byref(a), stream()), "gemm_f32_rs")
    factor = 0.5 / (ss.double().sum(1) / K + 1e-5).sqrt()
    v = x.double() @ w.double().t() * factor[:, None]
    off = (x.double().abs() @ w.double().abs().t() * factor[:, None]) * ((K + 8) * 2.0 ** -24)  # bound of v's error
    if epilogue in (STORE, F32):
        assert bool(((y[:, :N - 3] - v[:, :N - 3]).abs() <= off[:, :N - 3]).all()) and bool((y[:, N - 3:] == 7.0).all())
    elif epilogue in (GEGLU, SWIGLU):
        gate, up = v[:, ::2], v[:, 1::2]
        act = gate * torch.sigmoid(gate) if epilogue == SWIGLU else torch.nn.functional.gelu(gate, approximate="tanh")
        bound = 1.13 * off[:, ::2] * up.abs() + act.abs() * off[:, 1::2] + 2.0 ** -19 * (gate * up).abs() + 1e-12  # |act'| <= 1.13; tanhf and expf: a few ulps of the gate
        assert bool(((y[:, :columns] - act * up).abs() <= bound).all()) and bool((y[:, columns:] == 7.0).all())
    else:
        if epilogue == STREAM:
            new, bound = old + 0.25 * v[:, None], 0.25 * off + 2.0 ** -22 * (old[:, 0].abs() + v.abs())
            u = new[:, 0]
        else:
            mix = torch.tensor([[a.mix[s * MAX_STREAMS + t] for t in range(3)] for s in range(3)], dtype=torch.float64, device="cuda")
            write, read = (torch.tensor(list(c)[:3], dtype=torch.float64, device="cuda") for c in (a.out, a.in_))
            new = torch.einsum("rsn,st->rtn", old, mix) + write[:, None] * v[:, None]
            size = torch.einsum("rsn,st->rtn", old.abs(), mix.abs()) + write.abs()[:, None] * v.abs()[:, None]
            u = (new * read[:, None]).sum(1)
            bound = (write * read).abs().sum() * off + 2.0 ** -21 * (size * read.abs()[:, None]).sum(1)
            assert bool(((h - new).abs() <= write.abs()[:, None] * off[:, None] + 2.0 ** -21 * size).all())
        if epilogue == STREAM:
            assert bool(((h - new).abs() <= bound[:, None]).all())
        assert bool(((x_next - u * gain).abs() <= 2 * bound * gain.abs() + 1e-12).all())
        sums = (u * u).view(rows, N // 64, 64).sum(-1)
        assert bool(((ss_next - sums).abs() <= (2 * u.abs() * 2 * bound + 64 * 2.0 ** -24 * u * u).view(rows, N // 64, 64).sum(-1) + 1e-12).all())
    assert int(status.item()) == 0
