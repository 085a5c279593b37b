"""The float32 kernels at the sizes where they can go wrong: every launch of the product gives the same bits, and the
tiled attention gives a position the same bits however the tokens are cut.

Tolerances: a product's element has chains of at most 256 multiply-adds and at most a few segment sums, so its error is
below 300 * 2^-24 of the sum of the products' magnitudes; for normal entries, whose rounding errors are independent, the
2-norm of the error stays below 1e-6 of the result's.  Attention adds an exponential of 2 ulp and sums of 64: 2e-6."""

import math
from ctypes import c_int, c_longlong, c_void_p

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


def rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


@pytest.mark.parametrize("M, N, K, pad", [(1, 1, 1, 0), (2, 15, 3, 0), (3, 17, 512, 0), (16, 16, 513, 0), (17, 65, 516, 4),
                                          (33, 64, 2048, 0), (65, 130, 1028, 8), (70, 33, 2560, 3), (5, 129, 4608, 1)])
def test_gemm_f32_forms_agree(M, N, K, pad):
    from llmoxide_b200 import kernels
    torch.manual_seed(M * N + K)
    x, w = torch.randn(M, K + pad, device=DEV)[:, :K], torch.randn(N, K + pad, device=DEV)[:, :K]
    out = torch.full((M, N + 1), 7.0, device=DEV)
    kernels.gemm_fma(x, w, out[:, :N])
    assert (out[:, N] == 7.0).all()
    assert rel(out[:, :N], x.double() @ w.double().T) < 1e-6
    f = kernels._fn("gemm_fma", "llmx_gemm_f32_form", [c_int] + [c_void_p] * 3 + [c_int] * 3 + [c_longlong] * 3 + [c_void_p])
    for form in range(6):
        y = torch.empty(M, N, device=DEV)
        assert f(form, x.data_ptr(), w.data_ptr(), y.data_ptr(), M, N, K, x.stride(0), w.stride(0), N,
                 torch.cuda.current_stream().cuda_stream) == 0
        assert torch.equal(y, out[:, :N]), form


@pytest.mark.parametrize("M, N, K, pad", [(20, 40, 33, 0), (9, 100, 64, 0), (40, 70, 96, 1), (6, 50, 480, 0), (3, 20, 2049, 3),
                                          (18, 33, 2080, 0), (2, 16, 4097, 0)])
def test_gemm_f32_ends_where_a_single_last_segment_does(M, N, K, pad):
    test_gemm_f32_forms_agree(M, N, K, pad)


def test_gemm_f32_keeps_infinities_and_nan_in_their_rows():
    from llmoxide_b200 import kernels
    x, w = torch.randn(20, 70, device=DEV), torch.randn(40, 70, device=DEV)
    x[3, 69], x[5, 0], w[7, 1] = math.inf, math.nan, -math.inf
    out = torch.empty(20, 40, device=DEV)
    kernels.gemm_fma(x, w, out)
    bad = torch.zeros(20, 40, dtype=torch.bool, device=DEV)
    bad[3], bad[5], bad[:, 7] = True, True, True
    assert torch.equal(~torch.isfinite(out), bad)


def test_gemm_f32_takes_a_matrix_that_the_kernel_before_writes():
    """The product of a prompt becomes the matrix of a product of few tokens, launched right behind it."""
    from llmoxide_b200 import kernels
    torch.manual_seed(11)
    a, b, x = torch.randn(700, 2048, device=DEV), torch.randn(2048, 2048, device=DEV) / 45, torch.randn(3, 2048, device=DEV)
    want = x.double() @ (a.double() @ b.double().T).T
    for M in (1, 3):
        w, out = torch.full((700, 2048), 7.0, device=DEV), torch.empty(M, 700, device=DEV)
        for _ in range(3):
            w.fill_(7.0)
            kernels.gemm_fma(a, b, w)
            kernels.gemm_fma(x[:M], w, out)
            assert rel(out, want[:M]) < 2e-6


CASES = [   # H, G, D, Dv, lengths, window, keep_first, chunk, sink, softcap, sinks, bias entries, gate
    (6, 3, 48, 48, [1, 64, 130], None, 0, 0, 0.0, 0.0, False, 0, False),
    (16, 4, 128, 128, [300, 65], 70, 0, 0, 0.0, 0.0, False, 0, False),
    (40, 2, 256, 256, [130, 64], 50, 70, 0, 1.0, 0.0, False, 0, False),
    (4, 4, 96, 128, [200, 77], None, 0, 0, 0.0, 0.0, True, 0, True),
    (12, 1, 64, 192, [260], 90, 5, 0, 0.0, 8.0, True, 0, False),
    (8, 2, 16, 20, [200, 128, 1, 1, 1], None, 0, 48, 0.0, 0.0, False, 0, False),
    (8, 8, 64, 64, [700], 600, 4, 0, 0.0, 0.0, True, 333, False),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_attention_f32_however_cut(case):
    from llmoxide_b200 import kernels
    H, G, D, Dv, lens, window, keep, chunk, sink, softcap, sinks, bias, gate = CASES[case]
    torch.manual_seed(case)
    T, need = sum(lens), sum(-(-L // 64) for L in lens)
    order = torch.randperm(need + 2).tolist()
    # rows that no token wrote hold NaN: nothing of them may be seen
    k, v = torch.full((need + 2, G, 64, D), math.nan, device=DEV), torch.full((need + 2, G, 64, Dv), math.nan, device=DEV)
    table = torch.zeros((len(lens), max(-(-L // 64) for L in lens)), dtype=torch.int32)
    ks, vs = [torch.randn(L, G, D, device=DEV) for L in lens], [torch.randn(L, G, Dv, device=DEV) for L in lens]
    for b, L in enumerate(lens):
        for i in range(-(-L // 64)):
            page, n = order.pop(), min(64, L - 64 * i)
            table[b, i] = page
            k[page, :, :n], v[page, :, :n] = (z[b][64 * i : 64 * i + n].transpose(0, 1) for z in (ks, vs))
    table = table.to(DEV)
    q = torch.randn(T, H * D, device=DEV)
    seq = torch.cat([torch.full((L,), b, dtype=torch.int32) for b, L in enumerate(lens)]).to(DEV)
    pos = torch.cat([torch.arange(L, dtype=torch.int32) for L in lens]).to(DEV)
    sk = torch.randn(H, device=DEV) if sinks else None
    bt = torch.randn(H, bias, device=DEV) if bias else None
    gt = torch.randn(T, H + 3, device=DEV) if gate else None

    def run(rows, single=False):
        out = torch.empty(len(rows), H * Dv, device=DEV)
        kernels.attention_paged(q[rows], out, k, v, table, seq[rows], pos[rows], H, G, D, window, D ** -0.5, v_head_dim=Dv,
                                keep_first=keep, sink=sink, chunk=chunk, gate=gt[rows] if gate else None, softcap=softcap,
                                sinks=sk, score_bias=bt, single_tokens=single)
        return out

    everything, mixed = torch.arange(T, device=DEV), torch.randperm(T, device=DEV)
    out = run(everything)
    assert torch.equal(out, run(everything, single=True))            # a cluster per token
    assert torch.equal(out[mixed], run(mixed))                       # rows of many sequences in one tile of rows
    few = mixed[:7]
    assert torch.equal(out[few], run(few))

    want, t0 = [], 0
    for b, L in enumerate(lens):
        i, j = torch.arange(L, device=DEV)[:, None], torch.arange(L, device=DEV)[None, :]
        hidden = j > i
        if window:
            hidden = hidden | ((i - j >= window) & (j >= keep))
        if chunk:
            hidden = hidden | (i // chunk != j // chunk)
        for h in range(H):
            s = (q[t0 : t0 + L].double().view(L, H, D)[:, h] @ ks[b][:, h * G // H].double().T) * D ** -0.5
            s = softcap * torch.tanh(s / softcap) if softcap else s
            s = s + bt[h].double()[(i - j).clamp(0, bias - 1)] if bias else s
            w = torch.exp(s.masked_fill(hidden, -math.inf))
            total = w.sum(1, keepdim=True) + sink + (torch.exp(sk[h].double()) if sinks else 0.0)
            o = (w @ vs[b][:, h * G // H].double()) / total
            want.append(o * torch.sigmoid(gt[t0 : t0 + L, h, None].double()) if gate else o)
        t0 += L
    want = torch.cat([torch.stack(want[b * H : (b + 1) * H], 1).reshape(L, H * Dv) for b, L in enumerate(lens)])
    assert rel(out, want) < 2e-6


def test_attention_f32_leaves_out_what_a_row_does_not_see():
    """A later token's infinite key and value change nothing for the tokens before it, in one tile of rows or alone."""
    from llmoxide_b200 import kernels
    H, G, D, L = 4, 2, 64, 100
    k, v = torch.randn(2, G, 64, D, device=DEV), torch.randn(2, G, 64, D, device=DEV)
    table, q = torch.tensor([[1, 0]], dtype=torch.int32, device=DEV), torch.randn(L, H * D, device=DEV)
    seq, pos = torch.zeros(L, dtype=torch.int32, device=DEV), torch.arange(L, dtype=torch.int32, device=DEV)
    outs = []
    for poison in (False, True):
        if poison:
            k[0, :, 26], v[0, :, 26] = math.inf, math.nan          # position 90
        out = torch.empty(L, H * D, device=DEV)
        kernels.attention_paged(q, out, k, v, table, seq, pos, H, G, D, None, 0.125)
        outs.append(out)
    assert torch.equal(outs[0][:90], outs[1][:90]) and torch.isnan(outs[1][90:]).all()


def test_attention_f32_tiles_whose_scores_are_all_minus_infinity():
    """A bias of -inf at short distances: the newest tiles of a row hold no finite score, the older ones do."""
    from llmoxide_b200 import kernels
    H, G, D, L, near = 4, 2, 64, 300, 90
    torch.manual_seed(3)
    k, v = torch.randn(5, G, 64, D, device=DEV), torch.randn(5, G, 64, D, device=DEV)
    table, q = torch.arange(5, dtype=torch.int32, device=DEV)[None], torch.randn(L, H * D, device=DEV)
    seq, pos = torch.zeros(L, dtype=torch.int32, device=DEV), torch.arange(L, dtype=torch.int32, device=DEV)
    bias = torch.randn(H, 128, device=DEV)
    bias[:, :near] = -math.inf
    K, V = (z.transpose(1, 2).reshape(-1, G, D)[:L].double() for z in (k, v))
    i, j = torch.arange(L, device=DEV)[:, None], torch.arange(L, device=DEV)[None]
    want = []
    for h in range(H):
        s = q.view(L, H, D)[:, h].double() @ K[:, h * G // H].T * 0.125 + bias[h].double()[(i - j).clamp(0, 127)]
        want.append(torch.softmax(s.masked_fill(j > i, -math.inf), 1) @ V[:, h * G // H])
    want = torch.stack(want, 1).reshape(L, H * D)
    for single in (False, True):
        out = torch.empty(L, H * D, device=DEV)
        kernels.attention_paged(q, out, k, v, table, seq, pos, H, G, D, None, 0.125, score_bias=bias, single_tokens=single)
        assert torch.isnan(out[:near]).all()                  # no finite score at all
        assert rel(out[near:], want[near:]) < 2e-6


@pytest.mark.parametrize("H, G, D, Dv, window, keep, steps", [
    # (tokens held, tokens brought) per sequence
    (4, 4, 64, 64, None, 0, [(200, 1)] * 35 + [(0, 70)] + [(3, 1)]),       # 32 rows hold runs of 32 sequences
    (8, 2, 128, 128, 100, 5, [(600, 1), (0, 1), (63, 2), (64, 9), (0, 130), (500, 3)]),
    (12, 1, 48, 80, None, 0, [(70, 5), (10, 1), (0, 1), (129, 66)]),        # more heads a kv head than 8 rows
    (3, 3, 256, 256, 70, 0, [(300, 7), (0, 20)]),
    (5, 1, 20, 16, None, 0, [(1, 1), (0, 33)]),
])
def test_attention_f32_launches_agree(H, G, D, Dv, window, keep, steps):
    """Every launch, told where the sequences start or not, gives the same bits, and rows of q that are no whole 16-byte
    pieces too; against 64 bits as above."""
    from llmoxide_b200 import kernels
    torch.manual_seed(H * D)
    lens, new = [a + b for a, b in steps], [b for _, b in steps]
    width = max(-(-L // 64) for L in lens)
    pages = torch.randperm(width * len(lens), dtype=torch.int32).view(len(lens), width)
    k, v = (torch.full((pages.numel(), G, 64, n), math.nan, device=DEV) for n in (D, Dv))
    ks, vs = [torch.randn(L, G, D, device=DEV) for L in lens], [torch.randn(L, G, Dv, device=DEV) for L in lens]
    for b, L in enumerate(lens):
        for i in range(-(-L // 64)):
            n = min(64, L - 64 * i)
            k[pages[b, i], :, :n], v[pages[b, i], :, :n] = (z[b][64 * i : 64 * i + n].transpose(0, 1) for z in (ks, vs))
    T = sum(new)
    wide = torch.randn(T, H * D + 3, device=DEV)
    q = wide[:, : H * D].contiguous()
    seq = torch.cat([torch.full((n,), b, dtype=torch.int32) for b, n in enumerate(new)]).to(DEV)
    pos = torch.cat([torch.arange(a, a + n, dtype=torch.int32) for a, n in steps]).to(DEV)
    starts = torch.tensor([sum(new[:b]) for b in range(len(new) + 1)], dtype=torch.int32, device=DEV)

    def run(q, **hints):
        out = torch.full((T, H * Dv), 7.0, device=DEV)
        kernels.attention_paged(q, out, k, v, pages.to(DEV), seq, pos, H, G, D, window, D ** -0.5, v_head_dim=Dv,
                                keep_first=keep, **hints)
        return out

    out = run(q)
    for launch in (-1, 0, 1, 2):
        for start in (None, starts):
            assert torch.equal(run(q, launch=launch, seq_start=start), out), (launch, start is None)
        assert torch.equal(run(q, launch=launch, single_tokens=True), out), launch      # (a token by itself)
        assert torch.equal(run(wide[:, : H * D], launch=launch, seq_start=starts), out), launch
    want, t0 = [], 0
    for b, (past, n) in enumerate(steps):
        i, j = torch.arange(past, past + n, device=DEV)[:, None], torch.arange(past + n, device=DEV)[None]
        hidden = j > i
        if window:
            hidden = hidden | ((i - j >= window) & (j >= keep))
        qs = q[t0 : t0 + n].double().view(n, H, D)
        want.append(torch.stack([torch.softmax((qs[:, h] @ ks[b][:, h * G // H].double().T * D ** -0.5)
                                               .masked_fill(hidden, -math.inf), 1) @ vs[b][:, h * G // H].double()
                                 for h in range(H)], 1).reshape(n, H * Dv))
        t0 += n
    assert rel(out, torch.cat(want)) < 2e-6
