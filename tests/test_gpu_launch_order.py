"""Launches that overlap give the bits of the same launches one at a time: many layers of routed experts, the recurrence and
the split-K product, each behind the kernel that writes its inputs, in scratch that the layers and their parts share."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,requests", [(1, 1), (2, 2), (16, 16), (24, 3)])
def test_overlapping_launches_give_the_bits_of_single_ones(rows, requests):
    from kvcm.kernels import library as K
    D, E, top, F, G, H, d, taps, layers = 128, 16, 4, 64, 2, 4, 32, 4, 24
    C = (2 * G + H) * d
    g = torch.Generator(device="cuda").manual_seed(rows)

    def weights(*shape, scale=None, dtype=torch.bfloat16):
        return (torch.randn(*shape, generator=g, device="cuda") * (shape[-1] ** -0.5 if scale is None else scale)).to(dtype)

    f32 = torch.float32
    W = [dict(qkv=weights(C, D), ba=weights(2 * H, D), gate=weights(H * d, D), o=weights(D, H * d), conv=weights(C, taps, dtype=f32),
              a_log=weights(H, dtype=f32), dt=weights(H, dtype=f32), head=1 + weights(d, scale=0.1, dtype=f32),
              n1=1 + weights(D, scale=0.1, dtype=f32), n2=1 + weights(D, scale=0.1, dtype=f32), router=weights(E + 1, D, scale=0.3),
              gu=weights(E, 2 * F, D), down=weights(E, D, F), table=weights(64, D)) for _ in range(layers)]
    i32 = dict(dtype=torch.int32, device="cuda")
    per = rows // requests
    ctx = types.SimpleNamespace(seqs=requests, row_seq=torch.arange(rows, **i32) // per, seq_q_start=torch.arange(0, rows, per, **i32),
                                seq_q_len=torch.full((requests,), per, **i32), seq_state_slot=torch.arange(requests, **i32))
    ids = torch.randint(0, 64, (rows,), generator=g, **i32)

    def empty(*shape, dtype=f32):
        return torch.empty(shape, dtype=dtype, device="cuda")

    x, h, ba, wt, gates = empty(rows, D), empty(rows, D, dtype=torch.bfloat16), empty(rows, 2 * H), empty(rows, top), empty(rows)
    gate, y16, mixed = (empty(rows, n, dtype=torch.bfloat16) for n in (H * d, D, H * d))
    proj, qkv, out, y = empty(rows, C), empty(rows, C), empty(rows, D), empty(rows * top, D)
    o = empty(rows, H * d)
    idx = o.view(torch.int32).flatten()[:rows * top].view(rows, top)          # the recurrence's floats lie where the choices go
    work = torch.empty(K.moe_work_ints(rows, top, E), **i32)
    act, xs = empty(rows * top, F, dtype=torch.bfloat16), empty(rows * top, D, dtype=torch.bfloat16)
    state = empty(requests, H * d * d + (taps - 1) * C)

    def run(one_at_a_time):
        state.zero_()
        o.fill_(1.0)
        torch.cuda.synchronize()

        def launch(f, *args, **kw):
            f(*args, **kw)
            if one_at_a_time:
                torch.cuda.synchronize()

        launch(K.embed, ids, W[0]["table"], x)
        launch(K.cast_rows, x, h)
        for w in W:
            launch(K.gemm_tcgen05_splitk, h, w["qkv"], proj, weights_ready=True)
            launch(K.gemm_tcgen05_splitk, h, w["ba"], ba, weights_ready=True)
            launch(K.gemm_tcgen05_splitk, h, w["gate"], gate, weights_ready=True)
            launch(K.delta_conv, proj, w["conv"], state, H * d * d, ctx, qkv)
            launch(K.delta_prepare, qkv, ba, w["a_log"], w["dt"], H, G, d)
            launch(K.delta_scan, qkv, ba, state, ctx, o, H, G, d, d)
            launch(K.gated_rms, o, gate, w["head"], mixed, H, d, 1e-5)
            launch(K.gemm_tcgen05_splitk, mixed, w["o"], y16, weights_ready=True)
            launch(K.rms_scale_add, x, y16, w["n1"], h, 1e-5, 0.7)
            launch(K.moe_route, h, w["router"], E, 4, 2, top, 1.5, idx, wt, gates, weights_ready=True)
            if K.moe_few_supported(h, top, E, F):
                launch(K.moe_experts_few, h, w["gu"], w["down"], idx, work, act, y)
            else:
                launch(K.moe_experts, h, w["gu"], w["down"], idx, work, act, y, xs)
            launch(K.moe_combine, y, work, wt, E, x, gates, out)
            launch(K.rms_scale_add, x, out, w["n2"], h, 1e-5, 0.7)
        torch.cuda.synchronize()
        K.check_errors()
        return x.clone(), state.clone()

    want = run(True)
    assert all(bool(torch.isfinite(t).all()) for t in want)
    for _ in range(25):
        assert all(torch.equal(a, b) for a, b in zip(run(False), want))
