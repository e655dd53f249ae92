"""The bf16 GEMMs on the residual stream where their forms begin and end: stream_gemm beyond 64 rows (streamed), tile_gemm's 128 x 128
tiles up to one round of the SMs and its block pairs beyond, both widths. Against the same product in 64 bits: products of bf16 values
are exact, so a sum of K of them is off by at most K 2^-24 sum |x w| in any order; what the epilogues add rounds a few times more, a bf16
output once (2^-9)."""

import ctypes

import pytest
import torch

from nanochat_b200.hybrid import HybridDecoder, streamed
from nanochat_b200.native import MAX_STREAMS, GemmRs, check, cuda_library, stream

pytestmark = pytest.mark.gpu
STORE, F32, GEGLU, STREAM, STREAMS, SWIGLU = 0, 3, 5, 6, 7, 8
STREAMED = [(rows, 384, 2048) for rows in (65, 100, 128, 129, 255, 256)] + [(200, 1280, 3072), (65, 4096, 2048), (128, 4096, 2112)]
PAIRS = [(2100, 1280, 384), (2433, 1024, 64), (1281, 1920, 192), (2048 + 1, 1280, 1024)]  # 128 x 128 tiles: 170, 160, 165, 170
TILES = [(257, 384, 2048), (257, 1280, 3072), (129, 2048, 2048), (1100, 1280, 320), (640, 3584, 256)]


@pytest.mark.parametrize("rows, N, K", STREAMED + PAIRS + TILES)
@pytest.mark.parametrize("epilogue", [STORE, F32, GEGLU, STREAM, STREAMS, SWIGLU])
def test_product_and_epilogue(rows, N, K, epilogue):
    dec = HybridDecoder.__new__(HybridDecoder)
    dec.f32 = False
    kind = dec.gemm_kernel(rows, N, K)
    tiles = -(-rows // 128) * (N // 128)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert (kind == "stream") == streamed(rows, N, K) == ((rows, N, K) in STREAMED) and (tiles > sms) == ((rows, N, K) in PAIRS)
    lib, entry, part = HybridDecoder.ENTRY[kind]
    gen = torch.Generator(device="cuda").manual_seed(rows * 7919 + N * 31 + K + epilogue)

    def rand(*shape, dtype=torch.float32, scale=1.0):
        return (torch.randn(*shape, generator=gen, device="cuda") * scale).to(dtype)

    x, w, parts, stored = rand(rows, K, dtype=torch.bfloat16), rand(N, K, dtype=torch.bfloat16, scale=K ** -0.5), 5, N - 40
    ss, gain, status = rand(rows, parts).abs(), rand(N), torch.zeros(1, dtype=torch.int32, device="cuda")
    a = GemmRs(x=x.data_ptr(), w=w.data_ptr(), rows=rows, N=N, K=K, n_store=stored, epilogue=epilogue, scale=0.5, eps=1e-5, norm_count=K, mult=0.25,
               ss=ss.data_ptr(), ss_parts=parts, status=status.data_ptr())
    columns = N // 2 if epilogue in (GEGLU, SWIGLU) else N
    y = torch.full((rows, columns + 8), 7.0, dtype=torch.float32 if epilogue == F32 else torch.bfloat16, device="cuda")
    streams = 3 if epilogue == STREAMS else 1
    h = rand(rows, streams, N)
    old, x_next = h.double(), torch.zeros(rows, N, dtype=torch.bfloat16, device="cuda")
    ss_next = torch.zeros(rows, N // part, device="cuda")
    if epilogue in (STREAM, STREAMS):
        a.h, a.gain, a.x_next, a.ss_next = h.data_ptr(), gain.data_ptr(), x_next.data_ptr(), ss_next.data_ptr()
        a.streams = streams
        for s in range(streams):
            a.in_[s], a.out[s] = 0.3 + s, 1.0 - 0.4 * s
            for t in range(streams):
                a.mix[s * MAX_STREAMS + t] = 0.5 * (s == t) + 0.1 * s - 0.2 * t
    else:
        a.y, a.ldy = y.data_ptr(), columns + 8
    check(getattr(cuda_library(lib), entry)(ctypes.byref(a), stream()), entry)
    factor = 0.5 / (ss.double().sum(1) / K + 1e-5).sqrt()
    v = x.double() @ w.double().t() * factor[:, None]
    off = (x.double().abs() @ w.double().abs().t() * factor[:, None]) * ((K + 8) * 2.0 ** -24)  # bound of v's error

    def within(got, want, bound, rounds=0.0):
        err = (got.double() - want).abs() - (bound + rounds * (want.abs() + bound))
        assert float(err.max()) <= 1e-12, float(err.max())

    if epilogue in (STORE, F32):
        within(y[:, :stored], v[:, :stored], off[:, :stored], 2.0 ** -8 if epilogue == STORE else 0.0)
        assert bool((y[:, stored:] == 7.0).all())
    elif epilogue in (GEGLU, SWIGLU):
        gate, up = v[:, ::2], v[:, 1::2]
        act = gate * torch.sigmoid(gate) if epilogue == SWIGLU else torch.nn.functional.gelu(gate, approximate="tanh")
        # |act'| <= 1.13; tanhf and expf: a few ulps of the gate
        within(y[:, :columns], act * up, 1.13 * off[:, ::2] * up.abs() + act.abs() * off[:, 1::2] + 2.0 ** -19 * (gate * up).abs(), 2.0 ** -8)
        assert bool((y[:, columns:] == 7.0).all())
    else:
        if epilogue == STREAM:
            new, bound = old + 0.25 * v[:, None], 0.25 * off + 2.0 ** -22 * (old[:, 0].abs() + v.abs())
            u = new[:, 0]
            within(h, new, bound[:, None])
        else:
            mix = torch.tensor([[a.mix[s * MAX_STREAMS + t] for t in range(3)] for s in range(3)], dtype=torch.float64, device="cuda")
            write, read = (torch.tensor(list(c)[:3], dtype=torch.float64, device="cuda") for c in (a.out, a.in_))
            new = torch.einsum("rsn,st->rtn", old, mix) + write[:, None] * v[:, None]
            size = torch.einsum("rsn,st->rtn", old.abs(), mix.abs()) + write.abs()[:, None] * v.abs()[:, None]
            u = (new * read[:, None]).sum(1)
            bound = (write * read).abs().sum() * off + 2.0 ** -21 * (size * read.abs()[:, None]).sum(1)
            within(h, new, write.abs()[:, None] * off[:, None] + 2.0 ** -21 * size)
        within(x_next, u * gain, 2 * bound * gain.abs(), 2.0 ** -8)
        sums = (u * u).view(rows, N // part, part).sum(-1)
        within(ss_next, sums, (2 * u.abs() * 2 * bound + (part + 8) * 2.0 ** -24 * u * u).view(rows, N // part, part).sum(-1))
    assert int(status.item()) == 0
