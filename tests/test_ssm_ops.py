"""Recurrent ops: the CUDA scans agree with the step-by-step PyTorch recurrences, including carried state."""

import pytest
import torch

from easydel_b200.ops import ssm


def _close(a, b, tol=3e-2):
    return (a.float() - b.float()).abs().max() <= tol * b.float().abs().max().clamp_min(1.0)


def test_references_carry_state_across_calls():
    torch.manual_seed(0)
    T, D, N = 12, 6, 4
    u, delta = torch.randn(T, D), torch.randn(T, D)
    A = -torch.rand(D, N)
    B, C = torch.randn(T, N), torch.randn(T, N)
    full = ssm.selective_scan_reference(u, delta, A, B, C)
    st = torch.zeros(1, D, N)
    a = ssm.selective_scan_reference(u[:7], delta[:7], A, B[:7], C[:7], state=st)
    b = ssm.selective_scan_reference(u[7:], delta[7:], A, B[7:], C[7:], state=st)
    assert torch.allclose(torch.cat([a, b]), full, atol=1e-5)
    q, k, v = torch.randn(T, 2, 8), torch.randn(T, 2, 8), torch.randn(T, 2, 5)
    g, beta = -torch.rand(T, 2), torch.rand(T, 2)
    full = ssm.delta_rule_reference(q, k, v, g, beta)
    st = torch.zeros(1, 2, 8, 5)
    parts = torch.cat([ssm.delta_rule_reference(q[:5], k[:5], v[:5], g[:5], beta[:5], state=st),
                       ssm.delta_rule_reference(q[5:], k[5:], v[5:], g[5:], beta[5:], state=st)])
    assert torch.allclose(parts, full, atol=1e-5)


@pytest.mark.gpu
def test_selective_scan_cuda():
    torch.manual_seed(1)
    dev, T, D, N = "cuda", 70, 192, 16
    cu = torch.tensor([0, 30, 70], dtype=torch.int32, device=dev)
    bf = lambda *s: torch.randn(*s, device=dev).to(torch.bfloat16)  # noqa: E731
    u, delta, z, B, C = bf(T, D), bf(T, D), bf(T, D), bf(T, N), bf(T, N)
    A, Dv, bias = -torch.rand(D, N, device=dev), torch.randn(D, device=dev), torch.randn(D, device=dev)
    s1, s2 = torch.zeros(2, D, N, device=dev), torch.zeros(2, D, N, device=dev)
    with torch.no_grad():
        got = ssm.selective_scan(u, delta, A, B, C, Dv, z, bias, True, cu, s1)
        ref = ssm.selective_scan_reference(u, delta, A, B, C, Dv, z, bias, True, cu, s2)
    assert _close(got, ref) and _close(s1, s2)


@pytest.mark.gpu
def test_ssd_scan_cuda():
    torch.manual_seed(2)
    dev, T, H, P, G, N = "cuda", 40, 4, 64, 2, 128
    cu = torch.tensor([0, 17, 40], dtype=torch.int32, device=dev)
    bf = lambda *s: torch.randn(*s, device=dev).to(torch.bfloat16)  # noqa: E731
    x, dt, B, C = bf(T, H, P), bf(T, H), bf(T, G, N) * 0.3, bf(T, G, N) * 0.3
    A, Dv = -torch.rand(H, device=dev), torch.randn(H, device=dev)
    s1, s2 = torch.zeros(2, H, P, N, device=dev), torch.zeros(2, H, P, N, device=dev)
    with torch.no_grad():
        got = ssm.ssd_scan(x, dt, A, B, C, Dv, None, True, cu, s1)
        ref = ssm.ssd_scan_reference(x, dt, A, B, C, Dv, None, True, cu, s2)
    assert _close(got, ref) and _close(s1, s2)


@pytest.mark.gpu
@pytest.mark.parametrize("DK,DV,kda", [(128, 128, False), (64, 96, False), (128, 128, True), (128, 256, False)])
def test_delta_rule_cuda(DK, DV, kda):
    torch.manual_seed(3)
    dev, T, H = "cuda", 33, 3
    cu = torch.tensor([0, 13, 33], dtype=torch.int32, device=dev)
    q = torch.nn.functional.normalize(torch.randn(T, H, DK, device=dev), dim=-1).to(torch.bfloat16)
    k = torch.nn.functional.normalize(torch.randn(T, H, DK, device=dev), dim=-1).to(torch.bfloat16)
    v = torch.randn(T, H, DV, device=dev).to(torch.bfloat16)
    g = -torch.rand(T, H, DK, device=dev) if kda else -torch.rand(T, H, device=dev)
    beta = torch.rand(T, H, device=dev).to(torch.bfloat16)
    s1, s2 = torch.zeros(2, H, DK, DV, device=dev), torch.zeros(2, H, DK, DV, device=dev)
    with torch.no_grad():
        got = ssm.gated_delta_rule(q, k, v, g, beta, None, cu, s1)
        ref = ssm.delta_rule_reference(q, k, v, g, beta, None, cu, s2)
    assert _close(got, ref) and _close(s1, s2)


@pytest.mark.gpu
@pytest.mark.parametrize("what", [float("inf"), -float("inf"), float("nan"), 3.3895e38])
@pytest.mark.parametrize("at", [0, 7, 18, 31, 40])
def test_scans_keep_what_is_not_finite_from_earlier_tokens(what, at):
    """A value that is not finite (or is once it has been multiplied) reaches its head's column from its token on and nothing
    else: not the tokens before it, that share products of sixteen with it, nor other columns, heads or sequences. A key that
    is not finite does so for all columns of its head."""
    torch.manual_seed(5)
    dev, T, H, D = "cuda", 90, 2, 64
    cu = torch.tensor([0, 45, 90], dtype=torch.int32, device=dev)
    rnd = lambda *s: torch.randn(*s, device=dev)
    q, k = (torch.nn.functional.normalize(rnd(T, H, D), dim=-1).to(torch.bfloat16) for _ in range(2))
    v, g, beta = rnd(T, H, D).to(torch.bfloat16), -torch.rand(T, H, device=dev), torch.rand(T, H, device=dev).to(torch.bfloat16)
    B, C = rnd(T, 1, D).to(torch.bfloat16), rnd(T, 1, D).to(torch.bfloat16)
    dt, A, Dv = rnd(T, H).to(torch.bfloat16), -torch.rand(H, device=dev) - 0.5, torch.randn(H, device=dev)
    ops = [(lambda v, k: ssm.gated_delta_rule(q, k, v, g, beta, None, cu), k), (lambda v, k: ssm.gated_delta_rule(
               q, k, v, g[..., None].expand(T, H, D), beta, None, cu), k), (lambda v, B: ssm.ssd_scan(v, dt, A, B, C, Dv, None, True, cu), B)]
    for op, key in ops:
        clean = op(v, key).float()
        v2, k2 = v.clone(), key.clone()
        v2[at, 1, 5] = what
        k2[at, -1] = float("nan")
        for got, hit in ((op(v2, key), (slice(at, 45), 1, 5)), (op(v, k2), (slice(at, 45), slice(1 if key is k else 0, 2)))):
            off = torch.zeros(T, H, D, dtype=torch.bool, device=dev)
            off[hit] = True
            assert _close(got.float()[~off], clean[~off])
            if what != 3.3895e38:
                assert not got[hit][1:].isfinite().any()


@pytest.mark.gpu
@pytest.mark.parametrize("with_state", [True, False])
@pytest.mark.parametrize("cu", [[0, 5000], [0, 700, 1024, 1025, 1025, 3500, 5000], [0, 1024, 2048, 5000], [3, 40, 4990]])
def test_scans_in_windows_give_what_one_pass_gives(cu, with_state, monkeypatch):
    """Inputs longer than the workspace holds records of: sequences cut by windows of 1024 tokens once, several times or at a
    window's end, with the caller's states and with their own; segments inside windows (the state space with few heads)."""
    torch.manual_seed(len(cu))
    dev, T, H, D, n = "cuda", 5000, 2, 64, len(cu) - 1
    cu = torch.tensor(cu, dtype=torch.int32, device=dev)
    rnd = lambda *s: torch.randn(*s, device=dev)
    q, k = (torch.nn.functional.normalize(rnd(T, H, D), dim=-1).to(torch.bfloat16) for _ in range(2))
    v, g, beta = rnd(T, H, D).to(torch.bfloat16), -0.1 * torch.rand(T, H, device=dev), torch.rand(T, H, device=dev).to(torch.bfloat16)
    B, C, dt = rnd(T, 1, D).to(torch.bfloat16), rnd(T, 1, D).to(torch.bfloat16), (rnd(T, H) - 3).to(torch.bfloat16)
    A, Dv = -torch.rand(H, device=dev) - 0.5, rnd(H)
    got = []
    for limit in (ssm.SCAN_WORKSPACE, 1 << 14):
        monkeypatch.setattr(ssm, "SCAN_WORKSPACE", limit)
        states = [torch.ones(n, H, D, D, device=dev) if with_state else None for _ in range(2)]
        o = ssm.gated_delta_rule(q, k, v, g, beta, None, cu, states[0])
        y = ssm.ssd_scan(v, dt, A, B, C, Dv, None, True, cu, states[1])
        got.append([t[int(cu[0]):int(cu[-1])].float() for t in (o, y)] + [s for s in states if s is not None])
    assert ssm._scan_window(H, 1680) == 1024
    for i, (a, b) in enumerate(zip(*got)):      # outputs are rounded to bf16 once, states are fp32 sums in another order
        assert (a - b).abs().max() <= (2.0 ** -7 if i < 2 else 1e-5) * b.abs().max(), i


@pytest.mark.gpu
def test_ragged_conv1d_cuda():
    torch.manual_seed(4)
    dev, T, Cn, W = "cuda", 50, 96, 4
    cu = torch.tensor([0, 3, 20, 50], dtype=torch.int32, device=dev)
    x = torch.randn(T, Cn, device=dev).to(torch.bfloat16)
    w = torch.randn(Cn, W, device=dev).to(torch.bfloat16)
    b = torch.randn(Cn, device=dev).to(torch.bfloat16)
    c1 = torch.randn(3, W - 1, Cn, device=dev).to(torch.bfloat16)
    c2 = c1.clone()
    with torch.no_grad():
        got = ssm.ragged_conv1d(x, w, b, cu, "silu", c1)
        ref = ssm.ragged_conv1d_reference(x, w, b, cu, "silu", c2)
    assert _close(got, ref) and torch.equal(c1, c2)


@pytest.mark.gpu
def test_wkv4_kernel_matches_reference_with_state():
    from easydel_b200.ops import ssm

    torch.manual_seed(0)
    C = 200
    cu = torch.tensor([0, 37, 100], dtype=torch.int32, device="cuda")
    k = torch.randn(100, C, device="cuda").to(torch.bfloat16)
    v = torch.randn(100, C, device="cuda").to(torch.bfloat16)
    decay, first = torch.randn(C, device="cuda") * 0.5 - 1.0, torch.randn(C, device="cuda") * 0.5
    st = torch.zeros(2, 3, C, device="cuda")
    st[:, 2] = -1e38
    st_ref = st.clone()
    out = ssm.wkv4(decay, first, k, v, cu, st)
    ref = ssm.wkv4_reference(decay, first, k.float(), v.float(), cu, st_ref)
    assert (out.float() - ref).abs().max() < 2e-2
    assert (st[:, :2] - st_ref[:, :2]).abs().max() < 1e-3 * max(1.0, float(st_ref[:, :2].abs().max()))
    # a second call continues from the state
    out2 = ssm.wkv4(decay, first, k, v, cu, st)
    ref2 = ssm.wkv4_reference(decay, first, k.float(), v.float(), cu, st_ref)
    assert (out2.float() - ref2).abs().max() < 2e-2


def test_chunked_selective_scan_and_ssd_match_the_sequential_references_with_gradients():
    """The forms training runs (parallel scan per chunk / chunked matrix form) against the one-token-at-a-time
    references: outputs, final states and every input gradient, on two packed sequences with initial states."""
    import torch

    from easydel_b200.ops import ssm

    torch.manual_seed(0)

    def mk(*s):
        return (torch.randn(*s) * 0.5).requires_grad_(True)

    cu = torch.tensor([0, 70, 150], dtype=torch.int32)
    T, Dm, N = 150, 12, 8
    u, delta, B, C, z = mk(T, Dm), mk(T, Dm), mk(T, N), mk(T, N), mk(T, Dm)
    A = (-torch.rand(Dm, N) - 0.1).requires_grad_(True)
    D, dtb = mk(Dm), mk(Dm)
    ins = [u, delta, A, B, C, D, z, dtb]
    s1 = torch.randn(2, Dm, N)
    s2 = s1.clone()
    y1 = ssm.selective_scan_reference(u, delta, A, B, C, D, z, dtb, True, cu, s1)
    y2 = ssm.selective_scan_chunked(u, delta, A, B, C, D, z, dtb, True, cu, s2, chunk=32)
    g1 = torch.autograd.grad(y1.square().sum(), ins)
    g2 = torch.autograd.grad(y2.square().sum(), ins)
    assert torch.allclose(y1, y2, atol=1e-5) and torch.allclose(s1, s2, atol=1e-5)
    assert all(torch.allclose(a, b, atol=2e-4, rtol=1e-4) for a, b in zip(g1, g2))

    T, H, P, G, N = 150, 4, 6, 2, 8
    x, dt, B, C = mk(T, H, P), mk(T, H), mk(T, G, N), mk(T, G, N)
    A = (-torch.rand(H) - 0.1).requires_grad_(True)
    D, dtb = mk(H), mk(H)
    ins = [x, dt, A, B, C, D, dtb]
    s1 = torch.randn(2, H, P, N)
    s2 = s1.clone()
    y1 = ssm.ssd_scan_reference(x, dt, A, B, C, D, dtb, True, cu, s1)
    y2 = ssm.ssd_scan_chunked(x, dt, A, B, C, D, dtb, True, cu, s2, chunk=32)
    g1 = torch.autograd.grad(y1.square().sum(), ins)
    g2 = torch.autograd.grad(y2.square().sum(), ins)
    assert torch.allclose(y1, y2, atol=2e-5) and torch.allclose(s1, s2, atol=2e-5)
    assert all(torch.allclose(a, b, atol=5e-4, rtol=1e-3) for a, b in zip(g1, g2))


@pytest.mark.gpu
def test_chunked_scans_on_the_gpu_match_the_recurrent_kernels():
    """Training's chunked forms (autograd on, CUDA tensors) against the inference kernels on the same inputs."""
    import torch

    from easydel_b200.ops import ssm

    torch.manual_seed(0)
    dev = "cuda"
    T, Dm, N = 700, 256, 16
    bf = lambda *s: (torch.randn(*s, device=dev) * 0.5).to(torch.bfloat16)   # noqa: E731
    u, delta, B, C, z = bf(T, Dm), bf(T, Dm), bf(T, N), bf(T, N), bf(T, Dm)
    A = -torch.rand(Dm, N, device=dev) - 0.1
    D, dtb = torch.randn(Dm, device=dev), torch.randn(Dm, device=dev) * 0.1
    cu = torch.tensor([0, 300, 700], dtype=torch.int32, device=dev)
    with torch.no_grad():
        want = ssm.selective_scan(u, delta, A, B, C, D, z, dtb, True, cu)
    ug = u.clone().requires_grad_(True)
    got = ssm.selective_scan(ug, delta, A, B, C, D, z, dtb, True, cu)          # gradients wanted: chunked form
    got.float().square().sum().backward()
    assert ug.grad is not None and torch.isfinite(ug.grad).all()
    assert (got.float() - want.float()).abs().max() < 0.06 * want.float().abs().max() + 0.02

    H, P, G, N = 8, 64, 2, 32
    x, dt, Bm, Cm = bf(T, H, P), bf(T, H), bf(T, G, N), bf(T, G, N)
    A2 = -torch.rand(H, device=dev) - 0.1
    D2, dtb2 = torch.randn(H, device=dev), torch.randn(H, device=dev) * 0.1
    with torch.no_grad():
        want = ssm.ssd_scan(x, dt, A2, Bm, Cm, D2, dtb2, True, cu)
    xg = x.clone().requires_grad_(True)
    got = ssm.ssd_scan(xg, dt, A2, Bm, Cm, D2, dtb2, True, cu)
    got.float().square().sum().backward()
    assert xg.grad is not None and torch.isfinite(xg.grad).all()
    assert (got.float() - want.float()).abs().max() < 0.06 * want.float().abs().max() + 0.02

    Cn = 256
    k, v = bf(T, Cn), bf(T, Cn)
    decay, first = torch.randn(Cn, device=dev) * 0.5 - 1.0, torch.randn(Cn, device=dev) * 0.5
    with torch.no_grad():
        want = ssm.wkv4(decay, first, k, v, cu)                                  # the recurrent kernel
    kg = k.clone().requires_grad_(True)
    got = ssm.wkv4(decay, first, kg, v, cu)                                      # gradients wanted: chunked form
    got.float().square().sum().backward()
    assert kg.grad is not None and torch.isfinite(kg.grad).all()
    assert (got.float() - want.float()).abs().max() < 0.03


def test_chunked_wkv4_matches_the_sequential_reference_with_gradients():
    """RWKV-4's chunked matrix form against the per-token recurrence: outputs, the carried (num, den, max) triple
    and the gradients of decay, bonus, keys and values, on two packed sequences that start from a state."""
    import torch

    from easydel_b200.ops import ssm

    torch.manual_seed(0)
    T, C = 150, 24
    cu = torch.tensor([0, 70, 150], dtype=torch.int32)
    k = (torch.randn(T, C) * 2.0).requires_grad_(True)              # wide keys exercise the running maximum
    v = torch.randn(T, C).requires_grad_(True)
    decay = (torch.randn(C) * 0.5 - 1.0).requires_grad_(True)
    first = (torch.randn(C) * 0.5).requires_grad_(True)
    ins = [decay, first, k, v]
    s1 = torch.zeros(2, 3, C)
    s1[:, 2] = -1e38
    with torch.no_grad():                                           # a state that has already seen tokens
        ssm.wkv4_reference(decay, first, torch.randn(40, C), torch.randn(40, C), torch.tensor([0, 15, 40]), s1)
    s2 = s1.clone()
    y1 = ssm.wkv4_reference(decay, first, k, v, cu, s1)
    y2 = ssm.wkv4_chunked(decay, first, k, v, cu, s2, chunk=32)
    g1 = torch.autograd.grad(y1.square().sum(), ins)
    g2 = torch.autograd.grad(y2.square().sum(), ins)
    assert torch.allclose(y1, y2, atol=1e-5)
    assert torch.allclose(s1[:, 2], s2[:, 2], atol=1e-5)                                   # same maximum
    assert torch.allclose(s1[:, :2], s2[:, :2], atol=1e-5, rtol=1e-5)
    assert all(torch.allclose(a, b, atol=2e-4, rtol=1e-4) for a, b in zip(g1, g2))
    # the dispatcher agrees with the reference, and a fresh state and a ragged last chunk work too
    with torch.no_grad():
        assert torch.allclose(ssm.wkv4(decay, first, k, v, cu), ssm.wkv4_reference(decay, first, k, v, cu), atol=1e-5)
        assert torch.allclose(ssm.wkv4_chunked(decay, first, k[:7], v[:7], chunk=4),
                              ssm.wkv4_reference(decay, first, k[:7], v[:7]), atol=1e-5)


def _tokens_of(lens):
    return torch.tensor([0] + lens, device="cuda").cumsum(0).to(torch.int32), sum(lens)


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [[8], [1, 7, 8, 9, 0, 16], [130, 3, 257], [5, 1]])
@pytest.mark.parametrize("DK,DV,H", [(128, 128, 3), (128, 200, 2), (64, 72, 5), (32, 33, 1), (128, 128, 40)])
@pytest.mark.parametrize("gate", ["head", "channel", "none"])
def test_delta_rule_many_tokens_at_a_time_matches_the_tokens_one_by_one(lens, DK, DV, H, gate):
    """Chunks of sixteen and blocks of eight tokens (remainders, empty sequences, column tiles that are not full, plain resets by a gate of minus
    infinity) against the one-token recurrence in fp32, from a state that is not empty."""
    torch.manual_seed(5)
    cu, T = _tokens_of(lens)
    unit = lambda: torch.nn.functional.normalize(torch.randn(T, H, DK, device="cuda"), dim=-1).to(torch.bfloat16)  # noqa: E731
    q, k, v = unit(), unit(), torch.randn(T, H, DV, device="cuda").to(torch.bfloat16)
    g = None if gate == "none" else -3 * torch.rand(*((T, H, DK) if gate == "channel" else (T, H)), device="cuda")
    if g is not None:
        g[T // 2] = -float("inf")
    beta = None if gate == "none" else torch.rand(T, H, device="cuda").to(torch.bfloat16)
    s1 = torch.randn(len(lens), H, DK, DV, device="cuda")
    s2 = s1.clone()
    with torch.no_grad():
        got = ssm.gated_delta_rule(q, k, v, g, beta, None, cu, s1)
        want = ssm.delta_rule_reference(q.float(), k.float(), v.float(), g, beta, None, cu, s2)
    # fp32 sums in another order: a few 2^-24 per token; the output is rounded to bf16 (2^-9 of a value)
    assert (s1 - s2).abs().max() < 1e-5 * s2.abs().max()
    assert ((got.float() - want).abs() <= 2 ** -8 * want.abs() + 1e-5 * want.abs().max()).all()


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [[8], [1, 7, 8, 9, 0, 16], [130, 3, 257]])
@pytest.mark.parametrize("H,P,G,N", [(4, 64, 2, 128), (3, 50, 1, 16), (6, 128, 3, 64), (8, 33, 8, 32), (64, 64, 1, 128)])
def test_ssd_scan_many_tokens_at_a_time_matches_the_tokens_one_by_one(lens, H, P, G, N):
    torch.manual_seed(6)
    cu, T = _tokens_of(lens)
    bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)  # noqa: E731
    x, dt, B, C = bf(T, H, P), bf(T, H), bf(T, G, N), bf(T, G, N)
    A, D, bias = -4 * torch.rand(H, device="cuda"), torch.randn(H, device="cuda"), torch.randn(H, device="cuda")
    s1 = torch.randn(len(lens), H, P, N, device="cuda")
    s2 = s1.clone()
    with torch.no_grad():
        got = ssm.ssd_scan(x, dt, A, B, C, D, bias, True, cu, s1)
        want = ssm.ssd_scan_reference(x.float(), dt, A, B, C, D, bias, True, cu, s2)
    assert (s1 - s2).abs().max() < 1e-5 * s2.abs().max()
    assert ((got.float() - want).abs() <= 2 ** -8 * want.abs() + 1e-5 * want.abs().max()).all()


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [[300], [1, 47, 48, 49, 0, 16, 0, 97], [130, 0, 3, 257], [0, 161]])
@pytest.mark.parametrize("H,P,G,N", [(4, 64, 2, 128), (3, 50, 1, 16), (6, 128, 3, 64)])
@pytest.mark.parametrize("seg", [16, 48, 160])
@pytest.mark.parametrize("with_state", [True, False])
def test_ssd_segments_match_the_tokens_one_by_one(lens, H, P, G, N, seg, with_state, monkeypatch):
    """Sequences cut into segments that run side by side: ends of segments and sequences together and apart, empty sequences,
    with and without a state to start from."""
    monkeypatch.setattr(ssm, "_scan_segment", lambda *a: seg)
    torch.manual_seed(7)
    cu, T = _tokens_of(lens)
    bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)  # noqa: E731
    x, dt, B, C = bf(T, H, P), bf(T, H), bf(T, G, N), bf(T, G, N)
    A, D, bias = -4 * torch.rand(H, device="cuda"), torch.randn(H, device="cuda"), torch.randn(H, device="cuda")
    s1 = torch.randn(len(lens), H, P, N, device="cuda") if with_state else None
    s2 = s1.clone() if with_state else None
    with torch.no_grad():
        got = ssm.ssd_scan(x, dt, A, B, C, D, bias, True, cu, s1)
        want = ssm.ssd_scan_reference(x.float(), dt, A, B, C, D, bias, True, cu, s2)
    # fp32 sums in another order: a few 2^-24 per token; the output is rounded to bf16 (2^-9 of a value)
    if with_state:
        assert (s1 - s2).abs().max() < 1e-5 * s2.abs().max()
    assert ((got.float() - want).abs() <= 2 ** -8 * want.abs() + 1e-5 * want.abs().max()).all()


def test_layers_of_a_packed_pass_share_its_segment_plan(monkeypatch):
    """The bounds of packed documents make the host wait for the device: the first layer that asks finds them, the others (and
    recomputations) take what it found, and a pass whose layers do not ask finds none. Without a plan, as before, each its own."""
    from easydel_b200.layers.lightning_attention import LightningAttention
    from easydel_b200.layers.linear_attention import GatedDeltaNet, KimiDeltaAttention
    from easydel_b200.layers.ssm_branch import SSDMixer
    from easydel_b200.ops import attention

    torch.manual_seed(7)
    found = []
    real = attention.segment_ids_to_cu_seqlens
    monkeypatch.setattr(attention, "segment_ids_to_cu_seqlens", lambda ids: found.append(1) or real(ids))
    layers = [LightningAttention(32, 2, 16, 2), GatedDeltaNet(32, 2, 2, 16, 16), KimiDeltaAttention(32, 2, 16, 16, gate_low_rank_dim=8),
              SSDMixer(32, 32, 2, 16, 1, 16)]
    x = torch.randn(2, 12, 32)
    ids = torch.tensor([[1] * 5 + [2] * 7, [1] * 12])
    with torch.no_grad():
        want = [l(x, segment_ids=ids) for l in layers]
        assert len(found) == len(layers)
        found.clear()
        own = attention.with_segment_plan(ids)
        assert not found
        got = [l(x, segment_ids=own) for l in layers] + [layers[0](x, segment_ids=own)]
    assert len(found) == 1
    for a, b in zip(got, want + want[:1]):
        assert torch.equal(a, b)
