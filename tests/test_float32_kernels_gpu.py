"""The float32 engine's product and attention: every form of a kernel makes the same chain of sums, so forms are
compared bit for bit, and one of them with float64."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _ops():
    from pulsarlm_b200.kernels import ops

    ops.require_device()
    return ops


# Rows of A around every form's edges, K with and without a last piece of its own, N off the tiles and below one.
@pytest.mark.parametrize("m", [1, 4, 5, 8, 9, 16, 17, 32, 33, 65, 129, 300])
@pytest.mark.parametrize("n,k", [(24, 4), (7, 132), (2500, 260), (8200, 64), (33000, 20)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_every_form_of_the_product_gives_the_same_bits(m, n, k, accumulate):
    ops = _ops()
    gen = torch.Generator(device=DEV).manual_seed(m + n + k)
    a = torch.randn((m, k), generator=gen, device=DEV)
    w = torch.randn((n, k), generator=gen, device=DEV)
    off = torch.zeros((m, k + 1), device=DEV)
    off[:, 1:] = a                                       # (rows that start on no 16 bytes take the general form)
    got = torch.full((m, n), 0.5, device=DEV)
    want = got.clone()
    ops.gemm_f32(a, w, got, accumulate=accumulate)
    ops.gemm_f32(off[:, 1:], w, want, accumulate=accumulate)
    assert torch.equal(got, want)
    exact = a.double() @ w.double().t() + (0.5 if accumulate else 0.0)
    # k roundings of partial sums no larger than sum |a| |w|
    bound = (k + 2) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t() + 1.0)
    assert bool(((got.double() - exact).abs() <= bound).all())


# One size and more for every line of the forms' table, with CTAs alone on their SMs and with several: k over twice around the longest ring
# (eight pieces of 128) and off the pieces; k of one piece through registers.
@pytest.mark.parametrize("m,n,k", [
    (2, 100, 2180), (2, 2500, 2180), (1, 8200, 2180), (2, 8200, 2180), (3, 2000, 2180), (3, 12300, 2180), (8, 100, 2180), (8, 2500, 2180),
    (7, 8200, 2180), (16, 100, 2180), (16, 2500, 2180), (15, 2000, 2180), (9, 4100, 2180), (16, 12300, 2180), (9, 16400, 2180),
    (31, 100, 2180), (17, 2000, 2180), (17, 2500, 2180), (31, 12300, 2180), (17, 6000, 2180), (31, 16400, 2180), (40, 12300, 2180),
    (130, 6000, 2180), (300, 8200, 2180), (65, 33000, 132), (40, 5000, 16), (65, 6000, 4), (130, 100, 13 * 4)])
def test_every_tile_gives_the_bits_of_the_general_form(m, n, k):
    ops = _ops()
    gen = torch.Generator(device=DEV).manual_seed(m + n + k)
    a, w = torch.randn((m, k), generator=gen, device=DEV), torch.randn((n, k), generator=gen, device=DEV)
    off = torch.zeros((m, k + 1), device=DEV)
    off[:, 1:] = a
    got, want = torch.empty((m + 1, n), device=DEV).fill_(7.0), torch.empty((m, n), device=DEV)
    ops.gemm_f32(a, w, got[:m])
    ops.gemm_f32(off[:, 1:], w, want)
    assert torch.equal(got[:m], want) and bool((got[m] == 7.0).all())


@pytest.mark.parametrize("heads,kv,dim", [(8, 2, 64), (3, 3, 20), (16, 1, 128), (5, 1, 36), (4, 4, 128)])
@pytest.mark.parametrize("portions", [[1] * 3 + [5], [1] * 40 + [90, 1], [150], [1] * 70, [3] * 30, [70, 45, 2], [40]])
@pytest.mark.parametrize("options", [{}, {"window": 37}, {"window": 37, "keep_first": 5},
                                     {"softcap": 3.0, "sinks": True, "gate": True, "bias": True, "slopes": True}])
def test_staged_attention_gives_the_bits_of_the_plain_walk(heads, kv, dim, portions, options):
    """The plain walk is reached by asking for attention mass. Requests of several lengths, single tokens beside
    portions, a page that holds NaN in the values of tokens no query may see."""
    ops = _ops()
    gen = torch.Generator().manual_seed(heads * dim + len(portions))
    page = 16
    before = [int(torch.randint(0, 100, (1,), generator=gen)) for _ in portions]
    widths = [-(-(b + n + 3) // page) for b, n in zip(before, portions)]
    n_pages = sum(widths) + 1
    order = torch.randperm(n_pages, generator=gen).tolist()
    table = torch.full((len(portions), max(widths)), -1, dtype=torch.int32)
    for e, w in enumerate(widths):
        table[e, :w] = torch.tensor([order.pop() for _ in range(w)], dtype=torch.int32)
    pools = torch.randn((2, n_pages, kv, page, dim), generator=gen)
    for e, (b, n) in enumerate(zip(before, portions)):  # (places past the last token are not written yet)
        for j in range(b + n, widths[e] * page):
            pools[:, table[e, j // page], :, j % page] = float("nan")
    pools = pools.to(DEV)
    tokens = sum(portions)
    pos = torch.tensor([b + i for b, n in zip(before, portions) for i in range(n)], dtype=torch.int32, device=DEV)
    entry = torch.tensor([e for e, n in enumerate(portions) for _ in range(n)], dtype=torch.int32, device=DEV)
    q = torch.randn((tokens, heads, dim), generator=gen).to(DEV)
    more = {}
    if options.get("sinks"):
        more["sinks"] = torch.randn(heads, generator=gen).to(DEV)
        more["gate"] = torch.randn((tokens, heads), generator=gen).to(DEV)
        more["distance_bias"] = torch.randn((heads, 50), generator=gen).to(DEV)
        more["distance_slopes"] = torch.rand(heads, generator=gen).to(DEV) * 0.1
    args = (pools[0], pools[1], table.to(DEV), pos, entry)
    scale = dim ** -0.5
    common = dict(softcap=options.get("softcap", 0.0), keep_first=options.get("keep_first", 0), **more)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    got, want = torch.empty_like(q), torch.empty_like(q)
    ops.attention_simt(q, *args, got, page, options.get("window"), scale, status, **common)
    mass, weight = torch.zeros((n_pages, heads), device=DEV), torch.zeros(n_pages, device=DEV)
    ops.attention_simt(q, *args, want, page, options.get("window"), scale, status, mass, weight, **common)
    assert int(status.item()) == 0 and bool(torch.isfinite(want).all())
    assert torch.equal(got, want)
    one = torch.empty_like(q[-1:])   # (a token alone takes another form than among many)
    if "gate" in common:
        common["gate"] = common["gate"][-1:]
    ops.attention_simt(q[-1:], *args[:3], pos[-1:], entry[-1:], one, page, options.get("window"), scale, status, **common)
    assert torch.equal(one, want[-1:])


def test_more_columns_than_the_tiles_grid_holds():
    """65,535 tiles of 64 columns are one grid's; what is wider goes by the forms whose columns are its first coordinate."""
    ops = _ops()
    n, k, m = 65535 * 64 + 5, 4, 33
    a, w = torch.randn((m, k), device=DEV), torch.randn((n, k), device=DEV)
    out = torch.empty((m, n), device=DEV)
    ops.gemm_f32(a, w, out)
    for columns in (slice(0, 70), slice(n - 70, n)):
        want = a.double() @ w[columns].double().t()
        bound = (k + 2) * 2.0 ** -24 * (a.double().abs() @ w[columns].double().abs().t())
        assert bool(((out[:, columns].double() - want).abs() <= bound).all())


def test_calls_of_several_threads_keep_their_shared_memory():
    """A kernel's limit of shared memory is every thread's: products and attention that ask for different amounts of it, side by
    side."""
    import threading

    ops = _ops()
    failed = []

    def work(n, dim, kv):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                a, w, out = torch.ones((32, 128), device=DEV), torch.ones((n, 128), device=DEV), torch.empty((32, n), device=DEV)
                pools = torch.ones((2, 2, kv, 16, dim), device=DEV)
                q = torch.ones((4, 4, dim), device=DEV)
                table, entry = torch.zeros((1, 1), dtype=torch.int32, device=DEV), torch.zeros(4, dtype=torch.int32, device=DEV)
                pos, result = torch.arange(4, dtype=torch.int32, device=DEV), torch.empty_like(q)
                for _ in range(1500):
                    ops.gemm_f32(a, w, out)
                    ops.attention_simt(q, pools[0], pools[1], table, pos, entry, result, 16, None, 0.1)
                torch.cuda.current_stream().synchronize()
                assert bool((out == 128.0).all()) and bool((result == 1.0).all())
        except Exception as error:  # noqa: BLE001 - reported below
            failed.append(error)

    threads = [threading.Thread(target=work, args=a) for a in ((64, 100, 4), (8192, 128, 1), (64, 68, 2), (8192, 96, 1))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


def test_a_page_outside_the_pool_is_flagged_and_its_keys_are_left_out():
    ops = _ops()
    pools = torch.randn((2, 4, 1, 16, 64), device=DEV)
    q = torch.randn((70, 2, 64), device=DEV)
    pos = torch.arange(70, dtype=torch.int32, device=DEV) % 48
    entry = torch.zeros(70, dtype=torch.int32, device=DEV)
    table = torch.tensor([[0, 9, 2]], dtype=torch.int32, device=DEV)
    for rows in (slice(0, 70), slice(20, 24)):
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        got, want = torch.empty_like(q[rows]), torch.empty_like(q[rows])
        ops.attention_simt(q[rows], pools[0], pools[1], table, pos[rows], entry[rows], got, 16, None, 0.125, status)
        assert int(status.item()) == 4
        mass, weight = torch.zeros((4, 2), device=DEV), torch.zeros(4, device=DEV)
        ops.attention_simt(q[rows], pools[0], pools[1], table, pos[rows], entry[rows], want, 16, None, 0.125, None, mass, weight)
        assert torch.equal(got, want)


@pytest.mark.parametrize("heads,kv,dim", [(8, 2, 64), (3, 3, 20), (16, 1, 128), (6, 1, 36), (4, 4, 128), (2, 1, 64)])
@pytest.mark.parametrize("options", [{}, {"softcap": 3.0, "sinks": True, "gate": True, "bias": True, "slopes": True}])
def test_few_tokens_of_many_keys_give_the_bits_of_the_plain_walk(heads, kv, dim, options):
    """Single tokens whose keys end around a chunk's 32, a step's 64 and 128 and several steps on, a page that is missing in the middle
    of one request and at the start of another (the plain walk is reached by asking for attention mass)."""
    ops = _ops()
    gen = torch.Generator().manual_seed(heads * dim)
    page, ends = 16, [0, 30, 31, 32, 63, 64, 127, 128, 129, 255, 256, 500, 777]
    width = ends[-1] // page + 1
    pools = torch.randn((2, len(ends) * width, kv, page, dim), generator=gen).to(DEV)
    table = torch.randperm(len(ends) * width, generator=gen).int().view(len(ends), width)
    table[10, 5], table[11, 0], table[12, :9] = -1, -1, -1
    more = {}
    if options:
        more = {"sinks": torch.randn(heads, generator=gen).to(DEV), "distance_bias": torch.randn((heads, 50), generator=gen).to(DEV),
                "distance_slopes": torch.rand(heads, generator=gen).to(DEV) * 0.1, "softcap": 3.0}
    for chosen in ([i] for i in range(len(ends))) if heads > 8 else (list(range(len(ends))), [9], [12]):
        n = len(chosen)
        q = torch.randn((n, heads, dim), generator=gen).to(DEV)
        pos = torch.tensor([ends[i] for i in chosen], dtype=torch.int32, device=DEV)
        entry = torch.arange(n, dtype=torch.int32, device=DEV)
        gate = {"gate": torch.randn((n, heads), generator=gen).to(DEV)} if options else {}
        args = (pools[0], pools[1], table[chosen].contiguous().to(DEV), pos, entry)
        got, want = torch.empty_like(q), torch.empty_like(q)
        mass, weight = torch.zeros((pools.shape[1], heads), device=DEV), torch.zeros(pools.shape[1], device=DEV)
        status, plain_status = torch.zeros(1, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        ops.attention_simt(q, *args, got, page, None, dim ** -0.5, status, **more, **gate)
        ops.attention_simt(q, *args, want, page, None, dim ** -0.5, plain_status, mass, weight, **more, **gate)
        assert torch.equal(got, want) and int(status.item()) == int(plain_status.item())


# Steps whose CTAs of two heads outnumber the SMs take four heads each, of one and of two columns a thread.
@pytest.mark.parametrize("heads,kv,dim,tokens", [(32, 8, 64, 13), (8, 2, 128, 39), (8, 2, 100, 39), (16, 1, 128, 26), (16, 4, 36, 26)])
@pytest.mark.parametrize("options", [{}, {"softcap": 3.0}])
def test_four_heads_a_cta_give_the_bits_of_the_plain_walk(heads, kv, dim, tokens, options):
    ops = _ops()
    gen = torch.Generator().manual_seed(heads * dim + tokens)
    page, ends = 16, [0, 30, 31, 32, 63, 64, 127, 128, 129, 255, 256, 500, 777]
    width = ends[-1] // page + 1
    pools = torch.randn((2, tokens * width, kv, page, dim), generator=gen)
    table = torch.randperm(tokens * width, generator=gen).int().view(tokens, width)
    pos = [ends[i % len(ends)] for i in range(tokens)]
    for e in range(tokens):  # (keys past a request's last are not written yet)
        pools[:, table[e, pos[e] // page].item(), :, pos[e] % page + 1:] = float("nan")
    table[10, 5], table[12, :9] = -1, -1
    pools, table, pos = pools.to(DEV), table.to(DEV), torch.tensor(pos, dtype=torch.int32, device=DEV)
    entry = torch.arange(tokens, dtype=torch.int32, device=DEV)
    q = torch.randn((tokens, heads, dim), generator=gen).to(DEV)
    more = {"gate": torch.randn((tokens, heads), generator=gen).to(DEV), "sinks": torch.randn(heads, generator=gen).to(DEV)} if options else {}
    got, want = torch.empty_like(q), torch.empty_like(q)
    mass, weight = torch.zeros((pools.shape[1], heads), device=DEV), torch.zeros(pools.shape[1], device=DEV)
    status, plain_status = torch.zeros(1, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.attention_simt(q, pools[0], pools[1], table, pos, entry, got, page, None, dim ** -0.5, status, **options, **more)
    ops.attention_simt(q, pools[0], pools[1], table, pos, entry, want, page, None, dim ** -0.5, plain_status, mass, weight, **options, **more)
    assert bool(torch.isfinite(want).all()) and torch.equal(got, want) and int(status.item()) == int(plain_status.item())
