"""Edges of the size- and alignment-dependent paths of the kernels, against the CPU codecs or 64-bit restatements."""
import pytest
import torch

from hipress_b200 import ops

pytestmark = pytest.mark.gpu


def gauss(n, std=0.01, seed=0):
    return torch.randn(n, generator=torch.Generator().manual_seed(seed)) * std


def sparse_payload(idx, val):
    k = idx.numel()
    head = torch.tensor([4 + 8 * k], dtype=torch.int32)
    return torch.cat([head.view(torch.uint8), idx.to(torch.int32).view(torch.uint8), val.view(torch.uint8)])


def random_payload(n, k, seed, order="ascending"):
    g = torch.Generator().manual_seed(seed)
    idx = torch.randperm(n, generator=g)[:k]
    if order == "ascending":
        idx = idx.sort().values
    return sparse_payload(idx, torch.randn(k, generator=g))


# ----------------------------------------------------------------------------- sparse decode in tiles
@pytest.mark.parametrize("n,k", [(1, 1), (5, 0), (1023, 7), (1024, 1024), (1025, 33), (8192 * 3, 1), (700001, 32),
                                 (700001, 1025), (5000000, 1300000)])
@pytest.mark.parametrize("world", [1, 2, 3, 8])
@pytest.mark.parametrize("offset", [0, 1])
def test_sparse_decode_tiles(n, k, world, offset):
    payloads = [random_payload(n, min(n, k + 3 * s), s) for s in range(world)]
    ref = torch.empty(n)
    ops.sparse_decompress(payloads, ref, post_scale=1.0 / world)
    out = torch.full((n + offset,), 7.0, device="cuda")[offset:]
    ops.sparse_decompress([p.cuda() for p in payloads], out, post_scale=1.0 / world)
    assert torch.equal(out.cpu(), ref)
    assert ops.read_status(out) == 0


@pytest.mark.parametrize("n,k", [(300007, 40), (5000011, 5000), (5000011, 60000)])
@pytest.mark.parametrize("spread", ["even", "one_tile", "ends"])
@pytest.mark.parametrize("room", [0, 1, 3])
def test_sparse_decode_windows(n, k, spread, room):
    """Where the first probes of the search miss: entries crowded into a few tiles, slots with room for more entries
    than they hold.  Then a single descent, which only the tile that compares these two neighbours can see."""
    g = torch.Generator().manual_seed(k)
    payloads = []
    for r in range(3):
        if spread == "even":
            idx = torch.randperm(n, generator=g)[:k]
        else:
            near = torch.randperm(n // 3, generator=g)[:k] if k > 8000 else 8192 + torch.randperm(8192, generator=g)[:k]
            idx = near if spread == "one_tile" else torch.cat([near[:k // 2] % 8192, n - 1 - near[:k // 2] % 8192]).unique()
        p = sparse_payload(idx.sort().values, torch.randn(idx.numel(), generator=g))
        payloads.append(torch.cat([p, torch.full((8 * k * room,), 0x01, dtype=torch.uint8)]))
    for swap in (None, 0, k // 3):
        if swap is not None and spread != "ends":
            idx = payloads[1][4:4 + 4 * k].view(torch.int32)
            idx[swap], idx[swap + 1] = int(idx[swap + 1]), int(idx[swap])
        ref = torch.empty(n)
        ops.sparse_decompress(payloads, ref, post_scale=0.25)
        out = torch.full((n,), 7.0, device="cuda")
        ops.sparse_decompress([p.cuda() for p in payloads], out, post_scale=0.25)
        assert torch.equal(out.cpu(), ref), swap
    assert ops.read_status(out) == 0


@pytest.mark.parametrize("world", [1, 3])
def test_sparse_decode_of_unordered_payloads(world):
    """Order is a property of this library's compressor, not of the format: any order decodes, and the calls after
    it are not affected."""
    n, k = 300000, 9000
    for order in ("random", "ascending", "random", "random", "ascending"):
        payloads = [random_payload(n, k, 5 + s, order if s == world - 1 else "ascending") for s in range(world)]
        ref = torch.empty(n)
        ops.sparse_decompress(payloads, ref, post_scale=0.5)
        out = torch.full((n,), 7.0, device="cuda")
        ops.sparse_decompress([p.cuda() for p in payloads], out, post_scale=0.5)
        assert torch.equal(out.cpu(), ref), order


def test_sparse_decode_reports_indices_past_the_end():
    n = 50000
    idx = torch.arange(0, 60000, 100)           # the last hundred lie past the tensor
    val = torch.ones(idx.numel())
    out = torch.empty(n, device="cuda")
    ops.sparse_decompress(sparse_payload(idx, val).cuda(), out)
    assert ops.read_status(out) == 2
    ref = torch.zeros(n)
    ref[idx[idx < n]] = 1.0
    assert torch.equal(out.cpu(), ref)


@pytest.mark.parametrize("order", ["ascending", "random"])
@pytest.mark.parametrize("world", [1, 3])
@pytest.mark.parametrize("at", [0, 1234, 4999])
@pytest.mark.parametrize("bad", [400000, 0xffffffff])
def test_sparse_decode_reports_one_index_past_the_end(order, world, at, bad):
    """Wherever it stands in the payload; the other entries are decoded all the same."""
    n, k = 400000, 5000
    payloads = [random_payload(n, k, s, order) for s in range(world)]
    idx = payloads[-1][4:4 + 4 * k].view(torch.int32).long()
    val = payloads[-1][4 + 4 * k:].view(torch.float32)
    others = torch.arange(k) != at
    ref = torch.empty(n)
    ops.sparse_decompress(payloads[:-1] + [sparse_payload(idx[others], val[others])], ref)
    idx[at] = bad
    out = torch.full((n,), 7.0, device="cuda")
    ops.sparse_decompress([p.cuda() for p in payloads[:-1] + [sparse_payload(idx, val)]], out)
    assert ops.read_status(out) == 2
    assert torch.equal(out.cpu(), ref)


def test_sparse_decode_under_capture():
    n = 100000
    p = [random_payload(n, 500, s).cuda() for s in range(2)]
    out = torch.empty(n, device="cuda")
    ops.sparse_decompress(p, out)
    want = out.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.sparse_decompress(p, out)
    out.fill_(3.0)
    graph.replay()
    assert torch.equal(out, want)


# ----------------------------------------------------------------------------- quantisers: decode
def at_offset(payload, offset):
    """The payload `offset` bytes past an allocation's start (16-byte aligned): 6 puts data behind a 10-byte header on
    a 16-byte boundary, as in the exchange's receive slots."""
    buf = torch.zeros(payload.numel() + offset, dtype=torch.uint8, device="cuda")
    buf[offset:] = payload.cuda()
    return buf[offset:]


@pytest.mark.parametrize("bw", [1, 2, 4, 8])
@pytest.mark.parametrize("world", range(1, 9))
@pytest.mark.parametrize("offset", [0, 1, 6])
def test_terngrad_decode_tables(bw, world, offset):
    chunk = 1024 // bw
    for n in (1, chunk - 1, chunk, 9 * chunk + 5):
        payloads = [ops.terngrad_compress(gauss(n, seed=s), bw, True, seed=s) for s in range(world)]
        for add in (False, True):
            ref = gauss(n, 1.0, seed=99)
            out = ref.cuda()
            ops.terngrad_decompress(payloads, ref, add=add, post_scale=1.0 / world, bitwidth=bw)
            ops.terngrad_decompress([at_offset(p, offset) for p in payloads], out, add=add, post_scale=1.0 / world,
                                    bitwidth=bw)
            assert torch.equal(out.cpu(), ref), (n, add)
    assert ops.read_status(out) == 0


@pytest.mark.parametrize("world", range(1, 9))
@pytest.mark.parametrize("offset", [0, 2, 3])
def test_tbq_decode_tables(world, offset):
    for n in (1, 511, 512, 4613):
        payloads = [ops.tbq_compress(gauss(n, 0.03, seed=s), torch.zeros(n), 0.02) for s in range(world)]
        for add in (False, True):
            ref = gauss(n, 1.0, seed=99)
            out = ref.cuda()
            ops.tbq_decompress(payloads, ref, 0.02, add=add, post_scale=1.0 / world)
            ops.tbq_decompress([at_offset(p, offset) for p in payloads], out, 0.02, add=add, post_scale=1.0 / world)
            assert torch.equal(out.cpu(), ref), (n, add)


@pytest.mark.parametrize("bw", [2, 4, 8])
@pytest.mark.parametrize("world", range(1, 9))
def test_ecq_decode_tables(bw, world):
    chunk = 1024 // bw
    for n in (1, chunk, 9 * chunk + 5):
        payloads = [ops.ecq_compress(gauss(n, seed=s), torch.zeros(n), 1.0, 0.9, bw, seed=s) for s in range(world)]
        for add in (False, True):
            ref = gauss(n, 1.0, seed=99)
            ops_ref = ref.clone()
            ops.ecq_decompress(payloads, ops_ref, add=add, post_scale=0.5)
            for offset, shift in ((0, 0), (6, 0), (0, 1)):
                out = torch.empty(n + shift, device="cuda")[shift:]
                out.copy_(ref)
                ops.ecq_decompress([at_offset(p, offset) for p in payloads], out, add=add, post_scale=0.5)
                assert torch.equal(out.cpu(), ops_ref), (n, add, offset, shift)


# ----------------------------------------------------------------------------- quantisers: compress
@pytest.mark.parametrize("bw", [1, 2, 4, 8])
@pytest.mark.parametrize("feedback", [False, True])
@pytest.mark.parametrize("offset", [0, 1, 2, 6])
def test_terngrad_compress_paths(bw, feedback, offset):
    """Both sides of the one-launch limit (131,072 elements) and of the chunked path (296 chunks of 512 bytes)."""
    chunked = 296 * 512 * 8 // bw
    for n in (131072, 131073, chunked - 1, chunked + 777):
        g, r = gauss(n, seed=n), gauss(n, 0.004, seed=n + 1)
        rc = r.clone() if feedback else None
        rg = r.cuda() if feedback else None
        ref = ops.terngrad_compress(g, bw, True, seed=7, residual=rc)
        out = torch.zeros(ref.numel() + offset + 64, dtype=torch.uint8, device="cuda")
        ops.terngrad_compress(g.cuda(), bw, True, seed=7, residual=rg, out=out[offset:offset + ref.numel()])
        assert torch.equal(out[offset:offset + ref.numel()].cpu(), ref), n
        assert int(out[:offset].sum()) == 0 and int(out[offset + ref.numel():].sum()) == 0, n
        if feedback:
            assert torch.equal(rg.cpu(), rc), n


@pytest.mark.parametrize("n", [1, 3, 33, 4096 * 3 + 1])
def test_terngrad_small_unaligned(n):
    g, r = gauss(n + 1, seed=1), gauss(n + 1, 0.004, seed=2)
    rc, rg = r[1:].clone(), r.cuda()
    ref = ops.terngrad_compress(g[1:].clone(), 2, True, seed=3, residual=rc)
    out = ops.terngrad_compress(g.cuda()[1:], 2, True, seed=3, residual=rg[1:])
    assert torch.equal(out.cpu(), ref) and torch.equal(rg[1:].cpu(), rc)


@pytest.mark.parametrize("bw", [2, 4, 8])
@pytest.mark.parametrize("offset", [0, 1, 6])
def test_ecq_compress_paths(bw, offset):
    chunked = 296 * 512 * 8 // bw
    for n in (chunked - 1, chunked + 777):
        g, h = gauss(n, seed=n), gauss(n, 0.002, seed=n + 1)
        hc, hg = h.clone(), h.cuda()
        ref = ops.ecq_compress(g, hc, 1.0, 0.9, bw, seed=4)
        out = torch.zeros(ref.numel() + offset + 64, dtype=torch.uint8, device="cuda")
        ops.ecq_compress(g.cuda(), hg, 1.0, 0.9, bw, seed=4, out=out[offset:offset + ref.numel()])
        assert torch.equal(out[offset:offset + ref.numel()].cpu(), ref), n
        assert torch.equal(hg.cpu(), hc), n


# ----------------------------------------------------------------------------- sparse compress
def compare_sparse(r, rate, keep, seed):
    rc, rg = r.clone(), r.cuda()
    ref = ops.dgc_compress(rc, rate, keep, seed)
    out = ops.dgc_compress(rg, rate, keep, seed)
    total = int(ref[:4].view(torch.int32))
    assert torch.equal(out[:total].cpu(), ref[:total]), (rate, keep, seed)
    assert torch.equal(rg.cpu(), rc), (rate, keep, seed)


@pytest.mark.parametrize("n", [4097, 700001, (1 << 22) + 3])
@pytest.mark.parametrize("keep,rate", [(0.02, 0.01), (0.0625, 0.01), (0.25, 0.01), (0.25, 0.05), (0.9, 0.0)])
def test_sparse_scan_form(n, keep, rate):
    r = gauss(n, seed=n)
    for seed in range(1, 5):     # both sides of the over-selection branch
        compare_sparse(r, rate, keep, seed)


@pytest.mark.parametrize("n", [131072, 6000001])
@pytest.mark.parametrize("keep", [0.001, 0.0099])
def test_sparse_list_form_one_and_eight_ctas(n, keep):
    """The cut over the candidates: one CTA, and (59,400 wanted) a cluster of eight."""
    r = gauss(n, seed=n)
    for seed in range(1, 5):
        compare_sparse(r, 0.01, keep, seed)


@pytest.mark.parametrize("n", [1, 511, 513, 4095, 4097, 8191, 12289, (1 << 21) + 4099])
@pytest.mark.parametrize("few_magnitudes", [False, True])
def test_sparse_write_chunks(n, few_magnitudes):
    """Edges of a warp's 512 elements and a CTA's 4,096, and more chunks than one step of the look-back; with few
    magnitudes most of what lies at the cut is left behind, lane by lane."""
    r = gauss(n, seed=n)
    if few_magnitudes:
        r = torch.sign(r) * torch.tensor([1.0, 0.5, 0.5, 0.25])[torch.randint(4, (n,), generator=torch.Generator().manual_seed(n))]
    for keep in (0.03, 0.6):
        for rate in (0.0, 0.02):
            compare_sparse(r, rate, keep, 3)


@pytest.mark.parametrize("n", [(2 << 20) - 1, 2 << 20, (2 << 20) + 1])
@pytest.mark.parametrize("keep", [0.005, 0.0051, 0.01, 0.0102])
def test_sparse_where_lists_end(n, keep):
    """Both sides of the line between the forms, which must not show."""
    for seed in (1, 2):
        compare_sparse(gauss(n, seed=9), 0.01, keep, seed)


@pytest.mark.parametrize("octaves", [0, 30])
def test_sparse_cut_by_a_cluster(octaves):
    """45,000 wanted: eight CTAs share the candidates.  Over 30 octaves the cut lies in the last of the bins counted by
    distance, and is found by the keys' digits."""
    n = 9000001
    g = torch.Generator().manual_seed(8)
    r = torch.randn(n, generator=g) * torch.exp2(-octaves * torch.rand(n, generator=g))
    for seed in range(1, 5):
        compare_sparse(r, 0.00002 if octaves else 0.01, 0.005, seed)


def test_sparse_lists_longer_than_a_warp():
    """A warp of the collect pass holds the keys of its first 32 candidates; here some have hundreds, others none."""
    n = 3000001
    r = gauss(n, 1e-3, seed=5)
    r[700000:706000] = gauss(6000, 1.0, seed=6)
    for keep in (0.001, 0.004):
        for seed in (1, 2, 3):
            compare_sparse(r, 0.01, keep, seed)


@pytest.mark.parametrize("keep", [0.004, 0.05])
def test_sparse_magnitudes_over_many_octaves(keep):
    """Few samples and magnitudes over 30 octaves: the cut may lie far above the sampled threshold."""
    n = 300000
    g = torch.Generator().manual_seed(3)
    r = torch.randn(n, generator=g) * torch.exp2(-30 * torch.rand(n, generator=g))
    for seed in range(1, 9):
        compare_sparse(r, 0.0002, keep, seed)


@pytest.mark.parametrize("keep", [0.005, 0.05, 0.3])
@pytest.mark.parametrize("rate", [0.0, 0.01])
def test_sparse_many_equal_magnitudes(keep, rate):
    """Ties by the hundred thousand, at and above the cut, kept from the lower index on."""
    n = 400000
    g = torch.Generator().manual_seed(5)
    level = torch.tensor([0.0, 0.25, 0.5, 1.0])[torch.randint(0, 4, (n,), generator=g)]
    r = level * torch.where(torch.rand(n, generator=g) < 0.5, -1.0, 1.0)
    r[torch.rand(n, generator=g) < 0.4] = 0.0
    for seed in (1, 2, 3):
        compare_sparse(r, rate, keep, seed)


@pytest.mark.parametrize("keep", [0.001, 0.25])
@pytest.mark.parametrize("few_magnitudes", [False, True])
def test_sparse_samples_of_several_steps(keep, few_magnitudes):
    """From 15.2 M elements on, a CTA of the selection takes more than 256 sampled keys, in steps: a quarter kept puts
    up to 30 of each 256 into the threshold's bin, few magnitudes all of them."""
    n = (1 << 24) + 3
    r = gauss(n, seed=11)
    if few_magnitudes:
        i = torch.arange(n)
        r = torch.sign(r) * torch.where(i % 2000 == 0, 1.0, torch.tensor([0.5, 0.5, 0.25, 0.25, 0.25] + 5 * [0.0])[i % 10])
    for seed in (1, 2, 3):
        compare_sparse(r, 0.01, keep, seed)


# ----------------------------------------------------------------------------- PowerSGD
@pytest.mark.parametrize("n,r", [(1, 1), (16384, 1), (16385, 1), (16385, 2), (8192, 4), (8193, 3), (4096, 8), (4097, 8),
                                 (2048, 16), (2049, 11), (33, 16)])
def test_gram_schmidt_forms(n, r):
    """In registers and in memory: columns of unit length, pairwise orthogonal, and the column order of the definition."""
    P = gauss(n, 1.0, seed=n + r).view(n, 1).repeat(1, r) * 0.5 + gauss(n * r, 1.0, seed=r).view(n, r)
    want = P.double().clone()
    for j in range(min(r, n)):
        want[:, j] /= want[:, j].norm() + 1e-8
        for c in range(j + 1, r):
            want[:, c] -= (want[:, j] @ want[:, c]) * want[:, j]
    got = ops.gram_schmidt(P.cuda().contiguous())
    cols = min(r, n)
    # a column keeps about sqrt(1 - overlap^2) >= 0.3 of its length here, so 32-bit rounding shows as a few 1e-6
    assert (got[:, :cols].double().cpu() - want[:, :cols]).norm() <= 2e-5 * want[:, :cols].norm()


@pytest.mark.parametrize("n,r", [(3, 4), (4096, 4), (4097, 4), (1025, 8), (2048, 16)])
def test_gram_schmidt_of_rows_off_a_word(n, r):
    """Rows that are whole 16-byte words, at an address that is none: value by value, with the same result."""
    P = gauss(n * r, 1.0, seed=n).view(n, r)
    buf = torch.zeros(n * r + 1, device="cuda")
    buf[1:] = P.view(-1).cuda()
    off = ops.gram_schmidt(buf[1:].view(n, r))
    assert torch.equal(off, ops.gram_schmidt(P.cuda())) and float(buf[0]) == 0.0


@pytest.mark.parametrize("n,m,r", [(1, 4, 1), (7, 1028, 1), (33, 1024, 2), (64, 25088, 4), (9, 4096, 4), (1000, 2052, 4),
                                   (13, 300, 8), (4096, 512, 8)])
@pytest.mark.parametrize("short", [0, 3])
def test_powersgd_encode1_one_pass(n, m, r, short):
    """short: the gradient ends before the matrix does; what lies behind keeps its value and counts in P."""
    N = n * m - min(short, n * m - 1)
    grad, res = gauss(N, 1.0, seed=1), gauss(N, 0.5, seed=2)
    Q, M0 = gauss(m * r, 1.0, seed=3).view(m, r), gauss(n * m, 1.0, seed=4)
    want = M0.clone()
    want[:N] = grad + res
    M, P = M0.clone().view(n, m).cuda(), torch.full((n, r), 7.0, device="cuda")
    ops.powersgd_encode1(grad.cuda(), res.cuda(), Q.cuda(), M, P)
    assert torch.equal(M.cpu().view(-1), want)
    ref = want.view(n, m).double() @ Q.double()
    # fp32 products and sums of m terms: sqrt(m) roundings of 2^-24 each, and a wide margin
    assert (P.cpu().double() - ref).norm() <= 4 * m ** 0.5 * 2 ** -24 * (want.norm() * Q.norm()).double()


# ----------------------------------------------------------------------------- one launch, inputs read once
@pytest.mark.parametrize("bw", [1, 2, 4, 8])
@pytest.mark.parametrize("feedback", [False, True])
@pytest.mark.parametrize("offset", [0, 6])
def test_terngrad_resident_form(bw, feedback, offset):
    """Ragged last parts (148 parts of a multiple of 512 elements), the largest part and one element beyond it."""
    largest = 148 * 208 * 256
    for n in (131073, 148 * 1024 - 1, 148 * 1024 + 1, 2359807) + ((largest, largest + 1) if bw == 2 else ()):
        g, r = gauss(n, seed=n), gauss(n, 0.004, seed=n + 1)
        rc = r.clone() if feedback else None
        rg = r.cuda() if feedback else None
        ref = ops.terngrad_compress(g, bw, True, seed=7, residual=rc)
        out = torch.zeros(ref.numel() + offset + 64, dtype=torch.uint8, device="cuda")
        dev_g = g.cuda()
        for _ in range(2):      # back to back: the shared state is left ready
            if feedback:
                rg.copy_(r)
            ops.terngrad_compress(dev_g, bw, True, seed=7, residual=rg, out=out[offset:offset + ref.numel()])
        assert torch.equal(out[offset:offset + ref.numel()].cpu(), ref), n
        assert int(out[offset + ref.numel():].sum()) == 0, n
        if feedback:
            assert torch.equal(rg.cpu(), rc), n


@pytest.mark.parametrize("bw", [2, 4, 8])
@pytest.mark.parametrize("offset", [0, 6])
def test_ecq_resident_form(bw, offset):
    """One element, ragged last parts, the largest part and one element beyond it; a tensor of zeros."""
    largest = 148 * 208 * 256
    for n in (1, 511, 513, 148 * 1024 - 1, 148 * 1024 + 1, 2359807) + ((largest, largest + 1) if bw == 2 else ()):
        for std in (0.01, 0.0):
            g, h = gauss(n, std, seed=n), gauss(n, 0.4 * std, seed=n + 1)
            hc, hg = h.clone(), h.cuda()
            ref = ops.ecq_compress(g, hc, 1.0, 0.9, bw, 7)
            out = torch.zeros(ref.numel() + offset + 64, dtype=torch.uint8, device="cuda")
            dev_g = g.cuda()
            for _ in range(2):      # back to back: the shared state is left ready
                hg.copy_(h)
                ops.ecq_compress(dev_g, hg, 1.0, 0.9, bw, 7, out=out[offset:offset + ref.numel()])
            assert torch.equal(out[offset:offset + ref.numel()].cpu(), ref), n
            assert int(out[offset + ref.numel():].sum()) == 0, n
            assert torch.equal(hg.cpu(), hc), n


@pytest.mark.parametrize("n", [65537, 148 * 512, 148 * 512 + 1, 300007, 2359807])
def test_resident_forms_find_the_extremes_of_every_part(n):
    """In the first part, the last one and a partial word behind it; zeros of either sign, one sign only."""
    base = gauss(n, seed=n)
    inputs = [torch.zeros(n), torch.full((n,), -0.0), torch.full((n,), -3.0), base.abs() + 1, -base.abs() - 1]
    for at in (0, n // 2, n - 1):
        for value in (9.0, -9.0):
            x = base.clone()
            x[at] = value
            inputs.append(x)
    h = gauss(n, 0.4, seed=n + 1)
    for i, x in enumerate(inputs):
        want = ops.terngrad_compress(x, 2, True, seed=3)
        assert torch.equal(ops.terngrad_compress(x.cuda(), 2, True, seed=3).cpu(), want), i
        hc, hg = h.clone(), h.cuda()
        want = ops.ecq_compress(x, hc, 1.0, 0.9, 4, 7)
        assert torch.equal(ops.ecq_compress(x.cuda(), hg, 1.0, 0.9, 4, 7).cpu(), want), i
        assert torch.equal(hg.cpu(), hc), i


def test_terngrad_resident_form_when_its_wait_runs_out():
    """A counter that starts one short: no CTA ever sees all others arrive.  The wait ends, the status word says so, and
    the next call finds its state ready."""
    from hipress_b200 import _C
    n = 300007
    g = gauss(n, seed=1).cuda()
    want = ops.terngrad_compress(g, 2, False)
    scratch = torch.zeros(1 << 14, dtype=torch.uint8, device="cuda")
    scratch[:4] = 255
    out = torch.full_like(want, 7)
    assert _C._terngrad_resident_wait(g, out, scratch, 20000) == 4
    assert int((out != 7).sum()) == 0
    assert int(scratch[:8].sum()) == 0
    assert _C._terngrad_resident_wait(g, out, scratch, 2000000) == 0
    assert torch.equal(out, want)


@pytest.mark.parametrize("n", [4096, 300007])
def test_terngrad_one_launch_forms_under_capture(n):
    g = gauss(n, seed=1).cuda()
    want = ops.terngrad_compress(g, 2, True, seed=5)
    out = torch.zeros_like(want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.terngrad_compress(g, 2, True, seed=5, out=out)
    for _ in range(3):
        out.zero_()
        graph.replay()
        assert torch.equal(out, want)


def test_terngrad_resident_form_on_two_streams():
    n = 3000001
    g = [gauss(n, seed=s).cuda() for s in range(2)]
    want = [ops.terngrad_compress(x, 2, True, seed=5) for x in g]
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [[torch.zeros_like(w) for _ in range(20)] for w in want]
    torch.cuda.synchronize()
    for i in range(20):
        for s in range(2):
            with torch.cuda.stream(streams[s]):
                ops.terngrad_compress(g[s], 2, True, seed=5, out=outs[s][i])
    torch.cuda.synchronize()
    for s in range(2):
        for o in outs[s]:
            assert torch.equal(o, want[s])


# ----------------------------------------------------------------------------- batch norm
@pytest.mark.parametrize("n,c,h", [(2, 64, 9), (3, 8, 1), (4, 256, 14), (16, 2048, 7), (1, 512, 33)])
def test_bn_statistics_against_64_bits(n, c, h):
    from hipress_b200 import _C
    torch.manual_seed(c)
    x = (torch.randn(n, c, h, h, device="cuda") * 2 + 0.5).bfloat16().contiguous(memory_format=torch.channels_last)
    _, stats = _C.bn_forward(x, None, None, None, None, None, None, 0.1, 1e-5, True)
    xd = x.double().permute(0, 2, 3, 1).reshape(-1, c)
    # a few roundings of 2^-24, on values of order one
    assert (stats[0].double() - xd.mean(0)).abs().max() <= 4e-6
    if xd.shape[0] > 1:
        var = xd.var(0, unbiased=False)
        assert ((stats[1].double() - (var + 1e-5).rsqrt()) * (var + 1e-5).sqrt()).abs().max() <= 4e-6


# ----------------------------------------------------------------------------- sparse decode and update in one pass
@pytest.mark.parametrize("opt", ["sgd", "adamw"])
@pytest.mark.parametrize("world,n", [(1, 70001), (3, 8192 * 2), (8, 100003)])
@pytest.mark.parametrize("device_epoch", [0, 1])
def test_sparse_update_pass_equals_scatter_and_dense_update(opt, world, n, device_epoch):
    """clear_grad=1 (nobody keeps the gradient) decodes straight into the update; clear_grad=0 scatters first."""
    import hipress_b200 as hp
    from hipress_b200.parallel import SymmetricMemory
    results = []
    for clear in (0, 1):
        kw = dict(device_epoch=1, num_workers=0) if device_epoch else {}
        engines = [hp._C.DdpEngine(dict(rank=r, world=world, device=0, codec="graddrop", seed=3, flag_timeout_s=2.0,
                                        defer_recv=1, keep_fraction=0.01, sample_rate=0.05, clear_grad=clear, **kw),
                                   [(0, n, 1)], [0]) for r in range(world)]
        mems = SymmetricMemory.emulate(engines[0].symmetric_bytes, world)
        state = []
        for r, (e, m) in enumerate(zip(engines, mems)):
            bufs = [gauss(n, seed=10 + r).cuda(), torch.zeros(n, device="cuda"), gauss(n, 1.0, seed=5).cuda(),
                    torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")]
            e.set_buffers(bufs[0], bufs[1], bufs[2], bufs[3], None, bufs[4])
            e.set_symmetric(m.buf)
            if opt == "adamw":
                e.set_adamw(0.1, 0.9, 0.999, 1e-8, 0.01)
            else:
                e.set_sgd(0.1, 0.9, 0.01, True)
            state.append(bufs)
        for step in range(3):
            for e in engines:
                e.begin_step()
            for e in engines:
                e.bucket_ready(0, 0)
            for e in engines:
                e.drain()
            torch.cuda.synchronize()
            for e in engines:
                e.finish_step(0)
            torch.cuda.synchronize()
            for r, e in enumerate(engines):
                assert e.check_status() == 0
                if clear:
                    assert float(state[r][0].abs().max()) == 0.0
                state[r][0].copy_(gauss(n, seed=100 * (step + 1) + r))
        results.append([t.cpu() for bufs in state for t in bufs[1:]])
    for a, b in zip(*results):
        assert torch.equal(a, b)


def test_sparse_decode_from_two_threads_on_one_stream():
    """Decodes of ordered and unordered payloads queued by two threads on the default stream do not disturb each other."""
    import threading
    n, k = 200000, 3000
    jobs = []
    for t, order in enumerate(("ascending", "random")):
        p = random_payload(n, k, 40 + t, order)
        ref = torch.empty(n)
        ops.sparse_decompress(p, ref)
        jobs.append((p.cuda(), ref, [torch.empty(n, device="cuda") for _ in range(100)]))

    def work(p, outs):
        for o in outs:
            ops.sparse_decompress(p, o)

    threads = [threading.Thread(target=work, args=(p, outs)) for p, _, outs in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for _, ref, outs in jobs:
        for o in outs:
            assert torch.equal(o.cpu(), ref)


# ----------------------------------------------------------------------------- launch counts
def kernels_of(call):
    """Kernels that a call launches: the kernel nodes of its captured graph."""
    runtime = pytest.importorskip("cuda.bindings.runtime")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        call()               # the stream's scratch exists from here on
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        call()
    raw = runtime.cudaGraph_t(init_value=graph.raw_cuda_graph())
    _, _, count = runtime.cudaGraphGetNodes(raw)
    _, nodes, count = runtime.cudaGraphGetNodes(raw, count)
    return sum(runtime.cudaGraphNodeGetType(x)[1] == runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel for x in nodes[:count])


@pytest.mark.parametrize("codec,n,kw", [
    ("terngrad", 65536, {}), ("terngrad", 300000, {}), ("graddrop", 400000, dict(keep_fraction=0.001, sample_rate=0.01)),
    ("graddrop", 400000, dict(keep_fraction=0.02, sample_rate=0.01)),
    ("graddrop", 400000, dict(keep_fraction=0.02, sample_rate=0.05)),
    ("graddrop", 400000, dict(keep_fraction=0.02, sample_rate=0.0)),
    ("graddrop", 400000, dict(keep_fraction=0.02, sample_rate=0.01, momentum_correction=1, dgc_clip=1.0))])
def test_engine_counts_the_kernels_it_launches(codec, n, kw):
    """Push half of one rank's bucket, against the kernels of the same compression captured on its own."""
    import hipress_b200 as hp
    from hipress_b200.parallel import SymmetricMemory
    grad, res, aux = (gauss(n, seed=s).cuda() for s in range(3))

    def push_launches(codec, **kw):
        e = hp._C.DdpEngine(dict(rank=0, world=1, device=0, codec=codec, seed=3, flag_timeout_s=2.0, defer_recv=1, **kw),
                            [(0, n, 1)], [0])
        m = SymmetricMemory.emulate(e.symmetric_bytes, 1)[0]
        e.set_buffers(grad, res, None, None, aux)
        e.set_symmetric(m.buf)
        e.set_sgd(0.0, 0.0, 0.0, False)
        e.begin_step()
        before = e.launches
        e.bucket_ready(0, 0)
        e.drain()
        count = e.launches - before
        torch.cuda.synchronize()
        e.finish_step(0)
        torch.cuda.synchronize()
        assert e.check_status() == 0
        return count

    if codec == "terngrad":
        want = 2     # one launch is for callers that have the GPU to themselves
    elif kw.get("momentum_correction"):
        out = torch.zeros(ops.sparse_payload_bytes(n, kw["keep_fraction"]), dtype=torch.uint8, device="cuda")
        want = kernels_of(lambda: ops.dgc_momentum_compress(grad, aux, res, kw["sample_rate"], kw["keep_fraction"], 3,
                                                            momentum=0.9, clip=1.0, out=out))
    else:
        out = torch.zeros(ops.sparse_payload_bytes(n, 1 - (1 - kw["keep_fraction"])), dtype=torch.uint8, device="cuda")
        want = kernels_of(lambda: ops.graddrop_compress(grad, res, kw["sample_rate"], 1 - kw["keep_fraction"], 3, out=out))
    assert push_launches(codec, **kw) == want


# ----------------------------------------------------------------------------- calls that overlap the kernel before them
@pytest.mark.parametrize("n", [4096, 200000, 3000001])
@pytest.mark.parametrize("codec", ["tbq", "terngrad", "ecq", "graddrop"])
def test_calls_behind_one_another_and_behind_other_kernels(codec, n):
    """A pass is three kernels of PyTorch's and two calls, ten passes without a wait between them; every input is
    written just before it is read, over what the pass before read."""
    world = 2
    grads = [gauss(n, seed=s) for s in range(10)]
    dev = [g.cuda() for g in grads]
    grad, state, dense = torch.empty(n, device="cuda"), torch.zeros(n, device="cuda"), torch.empty(n, device="cuda")
    other = torch.zeros(n)

    def call(grad, state, dense, payloads):
        if codec == "tbq":
            ops.tbq_compress(grad, state, 0.01, out=payloads[0])
            ops.tbq_decompress(payloads, dense, 0.01, post_scale=0.5)
        elif codec == "terngrad":
            ops.terngrad_compress(grad, 2, True, 3, state, out=payloads[0])
            ops.terngrad_decompress(payloads, dense, post_scale=0.5, bitwidth=2)
        elif codec == "ecq":
            ops.ecq_compress(grad, state, 1.0, 0.9, 4, 3, out=payloads[0])
            ops.ecq_decompress(payloads, dense, post_scale=0.5)
        else:
            ops.graddrop_compress(grad, state, 0.05, 0.99, 3, out=payloads[0])
            ops.sparse_decompress(payloads, dense, post_scale=0.5)

    size = {"tbq": ops.tbq_payload_bytes(n), "terngrad": ops.terngrad_payload_bytes(n, 2),
            "ecq": ops.ecq_payload_bytes(n, 4), "graddrop": ops.sparse_payload_bytes(n, 1.0 - 0.99)}[codec]
    host = [torch.zeros(size, dtype=torch.uint8) for _ in range(world)]
    call(gauss(n, seed=77), other, torch.empty(n), [host[1], host[1]])
    payloads = [torch.zeros(size, dtype=torch.uint8, device="cuda"), host[1].cuda()]
    results = []
    torch.cuda.synchronize()
    for g in dev:
        grad.copy_(g)
        grad.mul_(2.0)
        call(grad, state, dense, payloads)
        results.append(dense.clone())
    state_host, dense_host = torch.zeros(n), torch.empty(n)
    for g, got in zip(grads, results):
        call(g * 2.0, state_host, dense_host, host)
        assert torch.equal(got.cpu(), dense_host)
    assert torch.equal(state.cpu(), state_host)
