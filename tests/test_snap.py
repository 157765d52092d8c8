"""GPU tests of the encoder side: nearest-codeword assignment (cbl_assign), tag packing (cbl_pack_tags) and the
snap of a weight matrix, against the reference-written fixtures and the CPU oracle. Tags are compared index for
index; where two codewords all but tie in fp32 the kernel may name the other one, so a differing index must lie within
a few fp32 ulps of the exact (float64) minimum."""
from pathlib import Path

import numpy as np
import pytest
import torch

from oracle import cbl_oracle as orc

pytestmark = pytest.mark.gpu
G = Path(__file__).resolve().parent / "golden"


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a))


def _check(x, book, idx, err, ref_idx, ref_err, wt=None, min_agree=0.995):
    idx, err = idx.cpu().numpy(), err.cpu().numpy()
    assert idx.dtype == np.int64 and err.dtype == np.float32
    agree = float((idx == ref_idx).mean()) if idx.size else 1.0
    assert agree >= min_agree, agree
    scale = 1.0 + (np.asarray(x, dtype=np.float64) ** 2 * (1.0 if wt is None else np.asarray(wt, dtype=np.float64))).sum(1)
    assert np.all(orc.assign_margin(x, book, idx, wt) <= 4e-6 * scale)
    assert np.allclose(err, ref_err, rtol=1e-4, atol=2e-5 * scale.max())


def test_assign_matches_reference_fixtures():
    from quantexperiments_b200 import codebook as cb
    z = np.load(G / "codebook.npz")
    i, e = cb.assign(_t(z["assign_x"]).cuda(), _t(z["assign_book"]).cuda())
    _check(z["assign_x"], z["assign_book"], i, e, z["assign_idx"], z["assign_err"])
    z = np.load(G / "snap.npz")
    i, e = cb.assign(_t(z["x"]).cuda(), _t(z["book"]).cuda())
    _check(z["x"], z["book"], i, e, z["idx"], z["err"])
    i, e = cb.assign(_t(z["x"]).cuda(), _t(z["book"]).cuda(), wt=_t(z["wt"]).cuda())
    _check(z["x"], z["book"], i, e, z["widx"], z["werr"], wt=z["wt"])
    assert int(i[7]) == 0 and float(e[7]) == 0.0          # all-zero weights: every codeword ties, the first wins


@pytest.mark.parametrize("n,K", [(1, 1), (5, 5), (2047, 37), (2049, 4096), (70001, 4096)])
@pytest.mark.parametrize("weighted", [False, True])
def test_assign_matches_oracle_on_ragged_sizes(n, K, weighted):
    from quantexperiments_b200 import codebook as cb
    g = torch.Generator().manual_seed(n + K)
    x = torch.randn(n, 8, generator=g)
    book = torch.randn(K, 8, generator=g).half()
    wt = torch.rand(n, 8, generator=g) + 0.01 if weighted else None
    ri, re = orc.assign(x.numpy(), book.numpy(), None if wt is None else wt.numpy())
    i, e = cb.assign(x.cuda(), book.cuda(), wt=None if wt is None else wt.cuda())
    _check(x.numpy(), book.numpy(), i, e, ri, re, wt=None if wt is None else wt.numpy())
    # a 32-bit book gives the same answer as its 16-bit values
    i2, e2 = cb.assign(x.cuda(), book.float().cuda(), wt=None if wt is None else wt.cuda())
    assert torch.equal(i, i2) and torch.equal(e, e2)


def test_assign_exact_codewords_and_first_index_on_ties():
    from quantexperiments_b200 import codebook as cb
    g = torch.Generator().manual_seed(3)
    book = torch.randn(4096, 8, generator=g).half()
    book[100] = book[7]                                    # a duplicate: the first index wins
    pick = torch.randint(0, 4096, (5000,), generator=g)
    pick[pick == 100] = 7
    i, e = cb.assign(book[pick].float().cuda(), book.cuda())
    assert torch.equal(i.cpu(), pick)
    assert float(e.max()) <= 1e-5
    i, e = cb.assign(torch.empty(0, 8).cuda(), book.cuda())
    assert i.numel() == 0 and e.numel() == 0


def test_assign_rejects_unsupported_arguments():
    from quantexperiments_b200 import _lib, codebook as cb
    x = torch.zeros(16, 8, device="cuda")
    book = torch.zeros(5000, 8, device="cuda")
    idx = torch.zeros(16, dtype=torch.int64, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    call = lambda d, K: _lib.lib.cbl_assign(x.data_ptr(), None, 16, d, book.data_ptr(), 0, K, idx.data_ptr(), x.data_ptr(), s)   # noqa: E731
    assert _lib.lib.cbl_assign_max_codewords() == 4096
    assert call(8, 4097) == _lib.EUNSUPPORTED
    assert call(4, 16) == _lib.EUNSUPPORTED
    assert call(8, 0) == _lib.EINVAL
    with pytest.raises(ValueError):
        cb.assign(x, book[:, :4])
    with pytest.raises(ValueError):
        cb.assign(x.cpu(), book.cpu())


def test_pack_bits_matches_reference_streams_bit_for_bit():
    from quantexperiments_b200 import codebook as cb
    z = np.load(G / "bits.npz")
    for bits in (1, 8, 10, 12, 13, 14, 16):
        w = cb.pack_bits(_t(z[f"vals_{bits}"]).cuda(), bits)
        assert w.dtype == torch.int32 and np.array_equal(w.cpu().numpy(), z[f"words_{bits}"]), bits
    g = torch.Generator().manual_seed(1)
    v = torch.randint(0, 4096, (300, 2368), generator=g)
    assert np.array_equal(cb.pack_bits(v.cuda(), 12).cpu().numpy(), orc.pack_bits(v.numpy(), 12))
    with pytest.raises(ValueError):
        cb.pack_bits(torch.full((2, 3), 4096).cuda(), 12)


def test_snap_matches_reference_compress_and_round_trips_through_the_decoder():
    """Matrix + fitted codebook in: the row scales bit for bit, the tags index for index (near-ties aside), then
    pack -> GPU decode equals the oracle's decode of the same tags."""
    from quantexperiments_b200 import codebook as cb
    from quantexperiments_b200.kernels import DeviceMatrix
    z = np.load(G / "snap.npz")
    w = _t(z["w"]).cuda()
    for tag, kw in (("plain", {}), ("weighted", dict(perm=_t(z["perm"]).long().cuda(), col_weight=_t(z["h"]).cuda(), row_weighted=True))):
        s = cb.snap(w, _t(z[f"{tag}_codebook"]).cuda(), **kw)
        assert np.array_equal(s["row_scale"].cpu().numpy(), z[f"{tag}_row_scale"])
        o = orc.snap(z["w"], z[f"{tag}_codebook"], perm=z["perm"] if kw else None, col_weight=z["h"] if kw else None, row_weighted=bool(kw))
        _check(o["chunks"], z[f"{tag}_codebook"], s["idx"].reshape(-1), s["err"], z[f"{tag}_idx"].reshape(-1), o["err"], wt=o["wt"], min_agree=0.999)
        assert abs(s["stats"]["normalized_chunk_mse"] - float(z[f"{tag}_mse"][0])) < 1e-5
    # self-hosting: snap a matrix against a 4096-word book, pack 12-bit tags, decode on the GPU
    g = torch.Generator().manual_seed(5)
    wm = torch.randn(96, 256, generator=g) * (torch.rand(96, 1, generator=g) + 0.5)
    book = torch.randn(4096, 8, generator=g).half()
    s = cb.snap(wm.cuda(), book.cuda())
    words = cb.pack_bits(s["idx"], 12)
    dm = DeviceMatrix(words, book.cuda(), s["row_scale"], K=4096, d=8, C=256, device="cuda")
    ref = orc.codebook_decode(s["idx"].cpu().numpy(), book.numpy(), s["row_scale"].cpu().numpy(), 0, 256, None)
    assert np.array_equal(dm.dequant(dtype=torch.float32).cpu().numpy(), ref)
    rel = float((dm.dequant(dtype=torch.float32).cpu() - wm).pow(2).mean() / wm.pow(2).mean())
    assert rel < 0.5                                       # random book, random matrix: the snap still halves the energy
    # the container's own decode takes the same path
    assert np.array_equal(cb.decode(s.cm).cpu().numpy(), ref)


def test_codebook_matrix_decode_with_padding_and_permutation_matches_the_reference_fixture():
    """decode(CodebookMatrix) on the GPU against the reference's decode of the same container (64-word book, rows of
    100 columns padded to 104, a column permutation): bit for bit, padding stripped, permutation undone."""
    from quantexperiments_b200 import codebook as cb
    z = np.load(G / "codebook.npz")
    pad, cols = (int(v) for v in z["pad"])
    cm = cb.CodebookMatrix(_t(z["idx"]).long(), _t(z["codebook"]), _t(z["row_scale"]), pad, cols, _t(z["perm"]).long())
    assert cm.K == 64 and cm.d == 8
    w = cb.decode(cm)
    assert w.shape == (16, 100) and np.array_equal(w.cpu().numpy(), z["decoded"])
    plain = cb.decode(cb.CodebookMatrix(cm.idx, cm.codebook, cm.row_scale, pad, cols, None))
    assert np.array_equal(plain.cpu().numpy()[:, z["perm"]], plain.cpu().numpy()[:, z["perm"]])
    inv = np.argsort(z["perm"])
    assert np.array_equal(plain.cpu().numpy()[:, inv], z["decoded"])                      # the permutation is what differs
    # a book whose size is not a power of two: 48 of the 64 words
    small = cb.CodebookMatrix(cm.idx % 48, cm.codebook[:48], cm.row_scale, pad, cols, None)
    ref = orc.codebook_decode((z["idx"] % 48), z["codebook"][:48], z["row_scale"], pad, cols, None)
    assert np.array_equal(cb.decode(small).cpu().numpy(), ref)


@pytest.mark.parametrize("K", [256, 4096])
@pytest.mark.parametrize("scale_x,scale_c", [(1.0, 1.0), (1e-4, 1e-4), (300.0, 200.0), (1e4, 1.0), (1.0, 1e-3)])
def test_tensor_core_assign_finds_the_exact_minimum(K, scale_x, scale_c):
    """The tensor-core path (fp16 book of whole MMA tiles): chunks and books of very different sizes, ragged chunk counts, a tile's
    edges; every index within rounding of the float64 minimum and the error as the scalar kernel computes it."""
    from quantexperiments_b200 import codebook as cb
    g = torch.Generator().manual_seed(K)
    book = (torch.randn(K, 8, generator=g) * scale_c).half()
    for n in (512, 513, 20001):
        x = torch.randn(n, 8, generator=g) * scale_x
        x[5] = 0.0
        x[6] = book[K - 1].float()
        idx, err = cb.assign(x.cuda(), book.cuda())
        d = ((x.double()[:, None, :] - book.double()[None, :, :]) ** 2).sum(-1) if n < 1000 else None
        xi, size = x.double(), (x.double() ** 2).sum(1)
        got = ((xi - book.double()[idx.cpu()]) ** 2).sum(1)
        best = d.min(1).values if d is not None else torch.cat([((c[:, None] - book.double()[None]) ** 2).sum(-1).min(1).values for c in xi.split(2000)])
        tol = 4e-6 * (size + got) + 1e-30
        assert ((got - best) <= tol).all()
        assert ((err.cpu().double() - got).abs() <= tol).all()
        assert int(idx[6]) == K - 1 or torch.equal(book[int(idx[6])], book[K - 1])


@pytest.mark.parametrize("K", [256, 512, 768, 1280, 3840])
def test_tensor_core_assign_of_books_between_equals_the_scalar_kernel(K):
    """Books whose uses of the accumulators fall unevenly to the three warpgroups and the four issuing warps; one tile and many per block."""
    from quantexperiments_b200 import codebook as cb
    g = torch.Generator().manual_seed(K)
    book = torch.randn(K, 8, generator=g).half().cuda()
    x = torch.randn(148 * 128 * 3 + 77, 8, generator=g).cuda()
    for n in (512, x.shape[0]):
        idx, err = cb.assign(x[:n], book)
        few = [cb.assign(c.contiguous(), book) for c in x[:n].split(500)]          # fewer than 512 chunks: the scalar kernel
        assert torch.equal(idx, torch.cat([i for i, _ in few])) and torch.equal(err, torch.cat([e for _, e in few]))


def test_snap_rows_equals_snap_by_chunks():
    """snap() of a plain matrix (division and chunking inside the kernel, ragged columns) against assign() of the chunks."""
    from quantexperiments_b200 import codebook as cb
    g = torch.Generator(device="cuda").manual_seed(4)
    book = torch.randn(4096, 8, device="cuda", generator=g).half()
    for R, C in ((37, 1001), (256, 512), (130, 8)):
        w = torch.randn(R, C, device="cuda", generator=g) * 0.02
        r = cb.snap(w, book)
        chunks, pad = cb.chunk_rows(w / r["row_scale"].float()[:, None], 8)
        idx, err = cb.assign(chunks, book)
        assert torch.equal(r["idx"].reshape(-1), idx) and torch.equal(r.err, err) and r["pad"] == pad
        assert r.stats["codebook_usage"] == idx.unique().numel() / 4096


@pytest.mark.parametrize("weighted", [False, True])
def test_snap_of_strided_rows(weighted):
    """Rows that overlap or repeat in memory (expanded rows, one short-strided row), every other row, every other column."""
    from quantexperiments_b200 import codebook as cb
    g = torch.Generator(device="cuda").manual_seed(9)
    book = torch.randn(4096, 8, device="cuda", generator=g).half()
    base = torch.randn(6, 40, device="cuda", generator=g)
    line = torch.randn(64, 1, device="cuda", generator=g)
    for w in (base[:1].expand(5, 40), line.t(), base[::2], base[:, ::2], base.t(), base.reshape(-1).as_strided((9, 40), (8, 1)), line):
        cw = torch.rand(w.shape[1], device="cuda", generator=g) + 0.5 if weighted else None
        got, want = cb.snap(w, book, col_weight=cw), cb.snap(w.clone(memory_format=torch.contiguous_format), book, col_weight=cw)
        assert torch.equal(got["idx"], want["idx"]) and torch.equal(got["row_scale"], want["row_scale"]) and torch.equal(got.err, want.err)


def test_tensor_core_assign_equals_the_scalar_kernel_where_many_words_all_but_tie():
    """Words that differ in the last bits of one fp16 value: many groups of 32 lie closer together than the tensor cores can tell. Also
    chunks and words that are tiny beside the book's largest value, and chunks that are not finite.  Fewer than 512 chunks run on the scalar kernel."""
    from quantexperiments_b200 import codebook as cb
    g = torch.Generator().manual_seed(11)
    centre = torch.randn(16, 8, generator=g)
    near = centre[torch.randint(0, 16, (4096,), generator=g)].half()
    near[torch.arange(4096), torch.randint(0, 8, (4096,), generator=g)] *= 1 + 2.0 ** -10
    tiny = torch.randn(4096, 8, generator=g)
    tiny[8:] *= 2.0 ** -10
    for book, size in ((near, 1.0), (tiny.half(), 2.0 ** -10)):
        x = (centre[torch.randint(0, 16, (6000,), generator=g)] if size == 1.0 else torch.randn(6000, 8, generator=g)) * size
        x += 0.02 * size * torch.randn(6000, 8, generator=g)
        x[3, 2], x[700, 0], x[1500] = float("inf"), float("-inf"), float("nan")
        idx, err = cb.assign(x.cuda(), book.cuda())
        few = [cb.assign(c.cuda(), book.cuda()) for c in x.split(500)]
        want, werr = torch.cat([i for i, _ in few]), torch.cat([e for _, e in few])
        fin = x.isfinite().all(1).cuda()
        dist = lambda i: ((x.cuda().double() - book.cuda().double()[i]) ** 2).sum(1)
        # the two kernels add |c|^2 in the same order; a word that both evaluate has the same distance bit for bit
        assert torch.equal(idx, want), int((idx != want).sum())
        assert torch.equal(err[fin], werr[fin])
        assert ((dist(idx) - dist(want)).abs()[fin] == 0).all()
