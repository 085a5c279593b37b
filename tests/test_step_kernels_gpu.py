"""Launches that a rule on sizes chooses, each against what it stands in for or against 64 bits, at the sizes where the rule
or a remainder changes."""

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


def rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


@pytest.mark.parametrize("T, E, top, K, groups, keep, rows, score, bias, real", [
    (1, 16, 2, 2048, 4, 2, 16, "sigmoid", False, 16), (4, 16, 2, 2048, 1, 1, 16, "softmax", False, 16),
    (8, 64, 6, 1024, 8, 4, 16, "softmax", True, 64),          # a token a CTA, the most of them
    (7, 7, 3, 264, 1, 1, 16, "sigmoid", False, 7), (8, 1024, 16, 64, 1, 1, 16, "softmax_top", False, 1024),
    (3, 40, 4, 4104, 1, 1, 64, "sigmoid", False, 36),         # experts without tiles; a row of more than the threads hold
    (6, 16, 2, 2048, 4, 2, 16, "sigmoid", True, 16), (8, 513, 9, 520, 1, 1, 16, "sigmoid", False, 513), (5, 3, 1, 8, 1, 1, 16, "softmax", False, 3)])
def test_router_that_sorts_and_gathers(T, E, top, K, groups, keep, rows, score, bias, real):
    """The same choices and weights as the router alone, and the order, tiles and rows that follow from them, exactly."""
    from llmoxide_b200 import kernels
    torch.manual_seed(T * E)
    x, w = torch.randn(T, K, device=DEV).bfloat16(), torch.randn(E, K, device=DEV) * 0.05
    b = torch.randn(E, device=DEV) * 0.1 if bias else None
    args = (groups, keep, 2, score, True, 1e-9, 1.5)
    ids, wts = torch.empty(T, top, dtype=torch.int32, device=DEV), torch.empty(T, top, device=DEV)
    kernels.moe_router(x, w, ids, wts, *args, bias=b)
    ids2, wts2, P = torch.empty_like(ids), torch.empty_like(wts), T * top
    perm, dest = (torch.full((P,), -7, dtype=torch.int32, device=DEV) for _ in range(2))
    sorted_w, xs = torch.empty(P, device=DEV), torch.empty(P, K, dtype=torch.bfloat16, device=DEV)
    tiles = torch.full((kernels.moe_max_tiles(P, E, rows), 3), -9, dtype=torch.int32, device=DEV)
    kernels.moe_router(x, w, ids2, wts2, *args, bias=b, places=(perm, dest, sorted_w, tiles, rows, real, xs))
    assert torch.equal(ids, ids2) and torch.equal(wts, wts2)
    pairs = ids.reshape(-1).long()
    order = torch.sort(pairs, stable=True)[1]
    assert torch.equal(perm.long(), order) and torch.equal(dest.long(), (order % top) * T + order // top)
    assert torch.equal(sorted_w, wts.reshape(-1)[order]) and torch.equal(xs, x[order // top])
    want, at = [], 0
    for e in range(E):
        n = int((pairs == e).sum())
        want += [[e, at + k, min(rows, n - k)] for k in range(0, n, rows)] if e < real else []
        at += n
    got = tiles.tolist()
    assert got[: len(want)] == want and all(t[0] == -1 for t in got[len(want):])


@pytest.mark.parametrize("T", [1, 8, 9])
def test_experts_whose_router_starts_between_vectors(T):
    """A float32 router that lies at no vector's start (a view of a larger buffer) chooses as the same numbers elsewhere do."""
    from types import SimpleNamespace
    from llmoxide_b200.config.spec import PartSpec, TensorSpec
    from llmoxide_b200.parts import Runtime
    from llmoxide_b200.parts.experts import RoutedExperts
    torch.manual_seed(T)
    E, d, ff = 4, 64, 32
    x, numbers = torch.randn(T, d, device=DEV).bfloat16(), torch.randn(E * d + 1, device=DEV)
    sizes = dict(gate=(ff, d), up=(ff, d), down=(d, ff))
    tensors = dict(router=TensorSpec("router", (E, d)), **{f"{k}{e}": TensorSpec(f"{k}{e}", n) for k, n in sizes.items() for e in range(E)})
    w = {f"{k}{e}": (torch.randn(n, device=DEV) * 0.1).bfloat16() for k, n in sizes.items() for e in range(E)}
    made = []
    for router in (numbers[1:].view(E, d), numbers[1:].view(E, d).clone()):
        part = RoutedExperts(PartSpec("routed_experts", dict(hidden_size=d, intermediate_size=ff, n_experts=E, top=2), tensors),
                             dict(w, router=router), Runtime(dtype="bfloat16", device=torch.device(DEV), max_positions=64))
        made.append(part.forward(x, SimpleNamespace(probe=None)))
    assert torch.equal(*made)


@pytest.mark.parametrize("T", [63, 64, 65, 16 * 148, 2500])
@pytest.mark.parametrize("E, n_extra", [(16, 0), (33, 1)])
def test_router_of_few_and_many_tokens(T, E, n_extra):
    """1, 4 and 16 tokens a CTA add up in the same order: a token's choices and weights have the same bits in every step."""
    from llmoxide_b200 import kernels
    torch.manual_seed(T + E)
    x, w = torch.randn(T, 520, device=DEV).bfloat16(), torch.randn(E + n_extra, 520, device=DEV) * 0.05

    def run(x):
        ids, wts = torch.empty(len(x), 3, dtype=torch.int32, device=DEV), torch.empty(len(x), 3, device=DEV)
        extra = torch.empty(len(x), n_extra, device=DEV) if n_extra else None
        kernels.moe_router(x, w, ids, wts, 1, 1, 1, "sigmoid", True, 0.0, 1.0, extra_out=extra)
        return ids, wts, extra

    all_of = run(x)
    for part in (x[:1], x[-20:], x[: T // 2]):
        at = 0 if part.data_ptr() == x.data_ptr() else T - 20
        for a, b in zip(run(part), all_of):
            assert a is None or torch.equal(a, b[at : at + len(part)])


@pytest.mark.parametrize("E", [8, 9, 15, 16, 17])
@pytest.mark.parametrize("K", [520, 517])
def test_router_of_float32_rows(E, K):
    """Rows of few experts are shared out to the warps in several ways: the same bits as in a prompt, which has one."""
    from llmoxide_b200 import kernels
    torch.manual_seed(E + K)
    x, w, made = torch.randn(70, K, device=DEV), torch.randn(E, K, device=DEV) * 0.05, []
    for part in (x, x[:64], x[:1]):
        ids, weights = torch.empty(len(part), 3, dtype=torch.int32, device=DEV), torch.empty(len(part), 3, device=DEV)
        kernels.moe_router(part, w, ids, weights, 1, 1, 1, "softmax", True, 0.0, 1.0)
        made.append((ids, weights))
    for ids, weights in made[1:]:
        assert torch.equal(ids, made[0][0][: len(ids)]) and torch.equal(weights, made[0][1][: len(ids)])


@pytest.mark.parametrize("M, N, K, pad", [(17, 64, 513, 3), (65, 130, 1028, 0), (33, 65, 2048, 0), (70, 66, 2049, 1),
                                          (34, 130, 3072, 0), (129, 65, 3500, 0), (200, 129, 4096, 4)])
def test_float32_tiles_that_share_k(M, N, K, pad):
    """The same bits as the launches that do not share (2 to 8 segments of K); more or fewer segments are refused."""
    from ctypes import c_int, c_longlong, c_void_p
    from llmoxide_b200 import kernels
    torch.manual_seed(M + K)
    x, w = torch.randn(M, K + pad, device=DEV)[:, :K], torch.randn(N, K + pad, device=DEV)[:, :K]
    f = kernels._fn("gemm_fma", "llmx_gemm_f32_form", [c_int] + [c_void_p] * 3 + [c_int] * 3 + [c_longlong] * 3 + [c_void_p])

    def run(form, k=K):
        y = torch.full((M, N + 1), 7.0, device=DEV)
        status = f(form, x.data_ptr(), w.data_ptr(), y.data_ptr(), M, N, k, x.stride(0), w.stride(0), N + 1,
                   torch.cuda.current_stream().cuda_stream)
        assert (y[:, N] == 7.0).all()
        return status, y[:, :N]

    want = run(4)[1]
    assert rel(want, x.double() @ w.double().T) < 1e-6
    for form in (6, 7):
        status, y = run(form)
        assert status == 0 and torch.equal(y, want)
        assert run(form, 512)[0] < 0


@pytest.mark.parametrize("D, n_rot, H, G, T, n_split", [(64, 64, 3, 1, 5, 3), (64, 0, 16, 8, 1, 5), (64, 64, 5, 2, 70, 1),
                                                        (128, 0, 16, 4, 70, 1), (128, 0, 3, 2, 4, 4), (64, 0, 2, 1, 9, 2)])
@pytest.mark.parametrize("gains", [False, True])
def test_heads_of_64_and_unrotated_heads(D, n_rot, H, G, T, n_split, gains):
    """Against 64 bits; q, k and v are rounded to bfloat16 once (2^-9 of a value, 2^-8 after a rotation's sum)."""
    from llmoxide_b200 import kernels
    torch.manual_seed(D + T)
    x = torch.randn(n_split, T, (H + 2 * G) * D, device=DEV)
    x = x[0].bfloat16() if n_split == 1 else x
    row = (x.double() if n_split == 1 else x.double().sum(0)).view(T, H + 2 * G, D)
    pos = torch.arange(30, 30 + T, dtype=torch.int32, device=DEV)
    angle = torch.rand(200, max(n_rot // 2, 1), device=DEV) * 6.28
    gq, gk = (1 + 0.1 * torch.randn(2, D, device=DEV)) if gains else (None, None)
    table = torch.tensor([[2, 0, 1]], dtype=torch.int32, device=DEV)
    kc, vc = (torch.zeros(3, G, 64, D, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    q = torch.empty(T, H * D, dtype=torch.bfloat16, device=DEV)
    kernels.qk_norm_rope_cache(x, q, kc, vc, table, torch.zeros(T, dtype=torch.int32, device=DEV), pos, gq, gk, 1e-6,
                               angle.cos() if n_rot else None, angle.sin() if n_rot else None, n_rot, H, G, D, True)

    def made(y, gain):
        if gains:
            y = y / (y.pow(2).mean(-1, keepdim=True) + 1e-6).sqrt() * gain.double()
        if n_rot:
            c, s = (f(angle.double())[pos.long()][:, None] for f in (torch.cos, torch.sin))
            a, b = y[..., : D // 2], y[..., D // 2 :]
            y = torch.cat([a * c - b * s, b * c + a * s], -1)
        return y

    where = [(int(table[0, int(p) // 64]), int(p) % 64) for p in pos]
    assert rel(q.view(T, H, D), made(row[:, :H], gq)) < 2 ** -8
    assert rel(torch.stack([kc[a, :, r] for a, r in where]), made(row[:, H : H + G], gk)) < 2 ** -8
    assert torch.equal(torch.stack([vc[a, :, r] for a, r in where]), row[:, H + G :].float().bfloat16())


@pytest.mark.parametrize("D, n_rot, T, n_split", [(64, 64, 3, 1), (64, 64, 5, 3), (64, 0, 70, 1), (64, 64, 70, 2), (128, 0, 4, 4),
                                                  (128, 0, 5, 1), (128, 0, 64, 1), (128, 0, 70, 1)])
@pytest.mark.parametrize("act", [torch.float32, torch.bfloat16])
def test_heads_by_vectors_add_squares_as_an_element_a_lane_does(D, n_rot, T, n_split, act):
    """q and k have the same bits whether the heads go by vectors or, for values of another size, an element a lane."""
    from llmoxide_b200 import kernels
    torch.manual_seed(D + T)
    H, G = 5, 2
    qk, v = torch.randn(n_split, T, (H + G) * D, device=DEV), torch.randn(n_split, T, G * D, device=DEV)
    gq, gk = 1 + 0.1 * torch.randn(2, D, device=DEV)
    pos, seq = torch.arange(30, 30 + T, dtype=torch.int32, device=DEV), torch.zeros(T, dtype=torch.int32, device=DEV)
    angle = torch.rand(200, max(n_rot // 2, 1), device=DEV) * 6.28
    cos, sin = (angle.cos(), angle.sin()) if n_rot else (None, None)
    table, made = torch.tensor([[2, 0, 1]], dtype=torch.int32, device=DEV), []
    for Dv in (D, D - 4):
        x = torch.cat([qk, v[:, :, : G * Dv]], 2)
        x = x[0].to(act) if n_split == 1 else x
        k_cache, v_cache = (torch.zeros(3, G, 64, n, dtype=act, device=DEV) for n in (D, Dv))
        q = torch.empty(T, H * D, dtype=act, device=DEV)
        kernels.qk_norm_rope_cache(x, q, k_cache, v_cache, table, seq, pos, gq, gk, 1e-6, cos, sin, n_rot, H, G, D, True, Dv)
        made.append((q, k_cache))
    assert torch.equal(made[0][0], made[1][0]) and torch.equal(made[0][1], made[1][1])


@pytest.mark.parametrize("T", [64, 65, 70])
@pytest.mark.parametrize("which", ["q", "k"])
def test_gains_that_start_between_vectors(T, which):
    """Unrotated heads whose gains lie at no vector's start (a view of a larger tensor): the bits of the same gains elsewhere."""
    from llmoxide_b200 import kernels
    torch.manual_seed(T)
    H, G, D = 3, 2, 128
    x, numbers = torch.randn(T, (H + 2 * G) * D, device=DEV).bfloat16(), 1 + 0.1 * torch.randn(2, D + 1, device=DEV)
    pos, seq = torch.arange(T, dtype=torch.int32, device=DEV), torch.zeros(T, dtype=torch.int32, device=DEV)
    table, made = torch.tensor([[1, 0]], dtype=torch.int32, device=DEV), []
    for aligned in (True, False):
        gains = dict(q=numbers[0, :D].clone(), k=numbers[0, :D].clone())
        gains[which] = numbers.flatten()[1 : D + 1].clone() if aligned else numbers.flatten()[1 : D + 1]
        k_cache, v_cache = (torch.zeros(2, G, 64, D, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        q = torch.empty(T, H * D, dtype=torch.bfloat16, device=DEV)
        kernels.qk_norm_rope_cache(x, q, k_cache, v_cache, table, seq, pos, gains["q"], gains["k"], 1e-6, None, None, 0, H, G, D, True, D)
        made.append((q, k_cache, v_cache))
    assert all(torch.equal(a, b) for a, b in zip(*made))


@pytest.mark.parametrize("dtype, n_split", [(torch.bfloat16, 1), (torch.float32, 3)])
@pytest.mark.parametrize("per_head, H, Dv", [(True, 3, 128), (True, 5, 20), (True, 2, 96), (False, 4, 128), (False, 3, 700),
                                             (False, 16, 128), (False, 17, 300), (False, 1, 8192), (False, 3, 4)])
def test_gated_norm_by_vectors_adds_squares_as_by_elements(dtype, n_split, per_head, H, Dv):
    """The same bits by vectors and, from a column that is no vector's first, by elements."""
    from llmoxide_b200 import kernels
    torch.manual_seed(H * Dv)
    T, n = 5, H * Dv
    o, gain = torch.randn(T, n, device=DEV), 1 + 0.1 * torch.randn(n, device=DEV)
    z, made = torch.randn(n_split, T, n, device=DEV).to(dtype), []
    for g_off in (8, 9):
        proj = torch.zeros(n_split, T, n + 12, dtype=dtype, device=DEV)
        proj[:, :, g_off : g_off + n] = z
        y = torch.empty(T, n, device=DEV)
        kernels.gated_norm(o, proj[0] if n_split == 1 else proj, g_off, gain, 1e-5, "silu", per_head, y, H, Dv)
        made.append(y)
    assert torch.equal(*made)


@pytest.mark.parametrize("d", [4, 60, 2048, 2052, 4096, 8192])
@pytest.mark.parametrize("T, n_a, n_b", [(1, 1, 3), (3, 9, 5), (64, 2, 2), (65, 1, 1), (90, 3, 8)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_two_results_joined_as_one_after_the_other(d, T, n_a, n_b, dtype):
    """A stream that gets two results and is normed in one kernel has the bits of one that gets them one by one."""
    from llmoxide_b200 import kernels
    torch.manual_seed(d + T)
    a, b = (torch.randn(n, T, d, device=DEV) for n in (n_a, n_b))
    a, b = a.to(dtype) if n_a == 1 else a, b.to(dtype) if n_b == 1 else b
    gain, h, rows = 1 + 0.1 * torch.randn(d, device=DEV), torch.randn(T, d, device=DEV), torch.tensor([T - 1, 0], dtype=torch.int32, device=DEV)
    for at in (None, rows):
        one, two = h.clone(), h.clone()
        out, joined = (torch.empty(T if at is None else 2, d, dtype=dtype, device=DEV) for _ in range(2))
        kernels.add_rms_norm(one, a, gain, 1e-6, None)
        kernels.add_rms_norm(one, b, gain, 1e-6, out, rows=at, write_h=at is None)
        kernels.dual_norm(two, [a, b], None, gain, 1e-6, joined, rows=at, write_h=at is None)
        assert torch.equal(out, joined) and (at is not None or torch.equal(one, two))


def test_routing_ahead_of_the_wait_reports_nothing():
    """A correction leaves the first group one expert that can be chosen; the scores keep the second group, and the run of the
    routing on zeros ahead of them, which would keep the first, is nobody's failure.  Where the scores keep the first, it is."""
    from llmoxide_b200 import kernels
    from llmoxide_b200.errors import KernelError
    kernels.check_status()
    x = torch.ones(2, 8, device=DEV).bfloat16()
    correction = torch.tensor([0.0] + [-float("inf")] * 3 + [-0.2] * 4, device=DEV)
    for scores, fails in ((5.0, False), (-5.0, True)):
        w = torch.zeros(8, 8, device=DEV)
        w[4:, 0] = scores * torch.tensor([1.0, 0.9, 0.8, 0.7], device=DEV)
        ids, weights = torch.empty(2, 2, dtype=torch.int32, device=DEV), torch.empty(2, 2, device=DEV)
        kernels.moe_router(x, w, ids, weights, 2, 1, 1, "sigmoid", True, 0.0, 1.0, bias=correction)
        torch.cuda.synchronize()
        if fails:
            with pytest.raises(KernelError):
                kernels.check_status()
        else:
            assert ids.tolist() == [[4, 5]] * 2
            kernels.check_status()


@pytest.mark.parametrize("dtype, n_split", [(torch.bfloat16, 1), (torch.float32, 1), (torch.float32, 9)])
@pytest.mark.parametrize("per_head, H, Dv", [(True, 3, 128), (True, 5, 20), (False, 4, 128), (False, 3, 700), (False, 17, 300),
                                             (True, 2, 132), (False, 1, 8196)])
def test_gated_norm_by_vectors(dtype, n_split, per_head, H, Dv):
    """A row or head of whole vectors, and the first size beyond, against 64 bits; float32 throughout: sums of up to 8196
    squares in chains of at most 33 and trees, 1e-6."""
    from llmoxide_b200 import kernels
    torch.manual_seed(H * Dv)
    T, n = 7, H * Dv
    o, gain = torch.randn(T, n, device=DEV), 1 + 0.1 * torch.randn(n, device=DEV)
    proj = torch.randn(n_split, T, n + 8, device=DEV).to(dtype)
    z = proj.double().sum(0)[:, 8:]
    y = torch.empty(T, n, device=DEV)
    kernels.gated_norm(o, proj[0] if n_split == 1 else proj, 8, gain, 1e-5, "silu", per_head, y, H, Dv)
    v = o.double().view(T, H, Dv) if per_head else o.double().view(T, 1, n)
    v = (v / (v.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt()).view(T, n)
    assert rel(y, v * gain.double() * z * torch.sigmoid(z)) < 1e-6


@pytest.mark.parametrize("design, name", [("tifapel", "C"), ("tifapel", "A"), ("gebasun", "C"), ("gebasun", "D")])
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("batch", [1, 9, 64, 65])
def test_captured_decode_steps_in_two_branches(tmp_path, design, name, dtype, batch):
    """Steps replayed as graphs, whose mixers and feed-forwards are branches up to 64 tokens, give the bits of steps launched
    one after another; several steps, so that what the branches allocate is used again from layer to layer and step to step."""
    import gebasun_configs
    import tifapel_configs
    from llmoxide_b200 import Engine, LoadOptions
    folder = dict(gebasun=gebasun_configs, tifapel=tifapel_configs)[design].make_folder(tmp_path, name, dtype)
    rng = torch.Generator().manual_seed(batch)
    prompts = [torch.randint(0, 200, (1 + 3 * (b % 7),), generator=rng).tolist() for b in range(batch)]
    steps = [[torch.randint(0, 200, (1,), generator=rng).tolist() for _ in range(batch)] for _ in range(4)]
    runs = []
    for graphs in (True, False):
        engine = Engine.load(folder, LoadOptions(dtype=dtype, max_tokens=64 * batch, max_batch=batch, cuda_graphs=graphs))
        slots = [engine.acquire() for _ in prompts]
        engine.step(list(zip(slots, prompts)))
        runs.append([engine.step(list(zip(slots, tokens))).clone() for tokens in steps])
        assert engine.options.cuda_graphs == graphs
    for a, b in zip(*runs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("batch, branched", [(1, True), (64, True), (65, False)])
def test_steps_that_are_captured_in_branches(tmp_path, monkeypatch, batch, branched):
    """Decode steps are cut up where they are captured and have up to 64 tokens, and nowhere else."""
    import tifapel_configs
    from llmoxide_b200 import Engine, LoadOptions
    from llmoxide_b200.parts import branches
    folder, forked, fork = tifapel_configs.make_folder(tmp_path, "C", "bfloat16"), [], branches.fork
    monkeypatch.setattr(branches, "fork", lambda rt, name, work: forked.append(name) or fork(rt, name, work))
    for graphs in (True, False):
        engine = Engine.load(folder, LoadOptions(dtype="bfloat16", max_tokens=64 * batch, max_batch=batch, cuda_graphs=graphs))
        slots = [engine.acquire() for _ in range(batch)]
        for _ in range(4):
            engine.step([(slot, [5]) for slot in slots])
        assert bool(forked) == (graphs and branched)
        forked.clear()
