"""GPU numerics: every CUDA kernel against a plain PyTorch fp32 reference (or, for the lossless
codec, against the scalar C++ codec byte for byte)."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

from fsdp_comm_opt_b200 import _lib
from fsdp_comm_opt_b200.ops import adamw, attention, codec, gpt2_ops, loss, norm, quant, rope, swiglu
from zipccl import hopper_fastzip2 as hz

DEV = "cuda"


def bits(t):
    return t.view(torch.int16)


def gauss(n, std=0.02, seed=0, device=DEV):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(n, generator=g) * std).to(torch.bfloat16).to(device)


def rand_bits(n, seed=0, device=DEV):
    g = torch.Generator().manual_seed(seed)
    return torch.randint(0, 65536, (n,), generator=g, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).to(device)


def test_native_library_is_loaded():
    assert _lib.cuda_lib_path().exists()
    assert _lib.cuda().zc_v2_encode is not None


# ------------------------------------------------------------------ codec
@pytest.mark.parametrize("n", [1, 1000, 1024, 4097, 1 << 20, (1 << 20) + 77])
@pytest.mark.parametrize("maker", [gauss, rand_bits])
def test_v2_gpu_matches_cpu_bytes_and_roundtrips(n, maker):
    x = maker(n, seed=3)
    rec, hdr = codec.v2_encode(x)
    rec_c, hdr_c = codec.v2_encode(x.cpu())
    assert torch.equal(hdr.cpu(), hdr_c)
    sizes = codec.v2_record_bytes(hdr_c)
    r = rec.cpu().view(-1, 2048)
    rc = rec_c.view(-1, 2048)
    mask = torch.arange(2048)[None, :] < sizes[:, None]
    assert torch.equal(r[mask], rc[mask])
    out = codec.v2_decode(rec, hdr, n)
    assert torch.equal(bits(out), bits(x))
    # GPU decodes CPU streams too
    out2 = codec.v2_decode(rec_c.to(DEV), hdr_c.to(DEV), n)
    assert torch.equal(bits(out2), bits(x))


@pytest.mark.parametrize("n", [1000, 4097, 1 << 20, (1 << 20) + 77])
@pytest.mark.parametrize("maker", [gauss, rand_bits])
def test_v2_nibble_mode_gpu_matches_cpu_bytes_and_roundtrips(n, maker):
    x = maker(n, seed=4)
    if maker is gauss:
        x[::700] = 2.0                                   # escapes below the window
    rec, hdr = codec.v2_encode(x, nibble=True)
    rec_c, hdr_c = codec.v2_encode(x.cpu(), nibble=True)
    assert torch.equal(hdr.cpu(), hdr_c)
    sizes = codec.v2_record_bytes(hdr_c)
    mask = torch.arange(2048)[None, :] < sizes[:, None]
    assert torch.equal(rec.cpu().view(-1, 2048)[mask], rec_c.view(-1, 2048)[mask])
    assert torch.equal(bits(codec.v2_decode(rec, hdr, n, nibble=True)), bits(x))
    assert torch.equal(bits(codec.v2_decode(rec_c.to(DEV), hdr_c.to(DEV), n, nibble=True)), bits(x))
    assert torch.equal(bits(codec.v2_decode(rec.cpu(), hdr.cpu(), n, nibble=True)), bits(x.cpu()))


def test_v2_unaligned_output_and_input():
    x = gauss(5000 + 3, seed=5)[3:]          # 6-byte offset: not 16-byte aligned
    rec, hdr = codec.v2_encode(x.contiguous() if False else x)
    buf = torch.zeros(5000 + 1, dtype=torch.bfloat16, device=DEV)
    out = codec.v2_decode(rec, hdr, 5000, buf[1:])
    assert torch.equal(bits(out), bits(x))


def _split_encode(x, base, n_works=1):
    n = x.numel()
    per = codec.pad_to_block((n + n_works - 1) // n_works)
    dev = x.device
    n_8 = torch.full((n_works,), per, dtype=torch.int32, device=dev)
    bases = torch.full((256,), base, dtype=torch.int32, device=dev)
    det = torch.zeros(n_works * codec.v1_det_bytes(per), dtype=torch.uint8, device=dev)
    scratch = torch.zeros(n_works * per, dtype=torch.uint8, device=dev)
    esc = torch.zeros(n_works * codec.align128(per), dtype=torch.uint8, device=dev)
    gc = torch.zeros(n_works, dtype=torch.int32, device=dev)
    hz.compress_split_store(x, n_8, bases, det, scratch, esc, gc, n_works)
    return n_8, det, esc, gc


@pytest.mark.parametrize("n,n_works", [(4096, 1), (10000, 1), (3 * 8192, 3), (1 << 20, 1), (8 * 12288, 8)])
@pytest.mark.parametrize("base", [116, 0, 252])
def test_v1_split_gpu_matches_cpu_bytes(n, n_works, base):
    x = torch.cat([gauss(n - 64, seed=n_works), rand_bits(64, seed=1)])
    n_8, det, esc, gc = _split_encode(x, base, n_works)
    n_8c, detc, escc, gcc = _split_encode(x.cpu(), base, n_works)
    assert torch.equal(gc.cpu(), gcc)
    assert torch.equal(det.cpu(), detc)
    off = 0
    for w in range(n_works):
        c = int(gcc[w])
        assert torch.equal(esc.cpu()[off:off + c], escc[off:off + c])
        off += codec.align128(c)
    per = int(n_8[0])
    out = torch.zeros(n_works * per, dtype=torch.bfloat16, device=DEV)
    hz.decompress_split_store(det, esc, n_8, gc, out, n_works)
    xp = torch.zeros(n_works * per, dtype=torch.bfloat16, device=DEV)
    xp[:n] = x
    assert torch.equal(bits(out), bits(xp))


def test_v1_gather_protocol_unpad_and_unpad_v():
    world, orig = 4, 5000 + 3
    per = codec.pad_to_block(orig)
    xs = [gauss(orig, seed=r) for r in range(world)]
    dets, escs, gcs = [], [], []
    for x in xs:
        _, det, esc, gc = _split_encode(x, 116)
        dets.append(det), escs.append(esc), gcs.append(int(gc[0]))
    stride = codec.align128(max(gcs))
    det_all = torch.cat(dets)
    esc_all = torch.cat([e[:stride] for e in escs])
    n_8 = torch.full((world,), per, dtype=torch.int32, device=DEV)
    nbytes = torch.full((world,), stride, dtype=torch.int32, device=DEV)
    out = torch.zeros(world * orig, dtype=torch.bfloat16, device=DEV)
    hz.decompress_split_store_unpad(det_all, esc_all, n_8, nbytes, out, orig, world)   # odd offsets: scalar stores
    assert torch.equal(bits(out), bits(torch.cat(xs)))
    out_off = torch.tensor([(world - 1 - r) * orig for r in range(world)], dtype=torch.int32, device=DEV)
    orig_n = torch.full((world,), orig, dtype=torch.int32, device=DEV)
    out2 = torch.zeros(world * orig, dtype=torch.bfloat16, device=DEV)
    hz.decompress_split_store_unpad_v(det_all, esc_all, n_8, nbytes, out_off, orig_n, out2, world * per, world)
    assert torch.equal(bits(out2), bits(torch.cat(xs[::-1])))


@pytest.mark.parametrize("orig,works,off,base", [(4095, 3, 0, 116), (4097, 9, 1, 116), (33000, 5, 3, 130), (20001, 2, 7, 252),
                                                (5_000_003, 3, 5, 116), (9_000_001, 1, 8, 118)])
def test_v1_packed_works_at_any_alignment(orig, works, off, base):
    """Works packed back to back at odd element offsets (loads and stores cut out of 16-byte pieces), several
    chunks per warp, outliers from none to all: bytes equal to the scalar codec's, round trip into a buffer that
    starts ``off`` elements in."""
    torch.manual_seed(orig)
    x = torch.cat([torch.zeros(off, dtype=torch.bfloat16, device=DEV)] + [
        torch.cat([gauss(orig - orig // 4, seed=w), rand_bits(orig // 4, seed=w)]) for w in range(works)])[off:]
    per = codec.pad_to_block(orig)

    def encode(v):
        dev = v.device
        n_8 = torch.full((works,), per, dtype=torch.int32, device=dev)
        on = torch.full((works,), orig, dtype=torch.int32, device=dev)
        bases = torch.full((256,), base, dtype=torch.int32, device=dev)
        det = torch.zeros(works * codec.v1_det_bytes(per), dtype=torch.uint8, device=dev)
        esc = torch.zeros(works * codec.align128(per), dtype=torch.uint8, device=dev)
        gc = torch.zeros(works, dtype=torch.int32, device=dev)
        hz.compress_split_store_pad(v, n_8, on, bases, det, torch.zeros(works * per, dtype=torch.uint8, device=dev), esc,
                                    gc, works * per, works)
        return n_8, det, esc, gc

    n_8, det, esc, gc = encode(x)
    _, detc, escc, gcc = encode(x.cpu())
    assert torch.equal(gc.cpu(), gcc) and torch.equal(det.cpu(), detc)
    at = 0
    for c in gcc.tolist():
        assert torch.equal(esc[at:at + c].cpu(), escc[at:at + c])
        at += codec.align128(c)
    out = torch.full((off + works * orig + 16,), 3.0, dtype=torch.bfloat16, device=DEV)
    out_off = torch.tensor([off + w * orig for w in range(works)], dtype=torch.int32, device=DEV)
    on = torch.full((works,), orig, dtype=torch.int32, device=DEV)
    hz.decompress_split_store_unpad_v(det, esc, n_8, gc, out_off, on, out, works * per, works)
    assert torch.equal(bits(out[off:off + works * orig]), bits(x))
    assert bool((out[:off] == 3.0).all()) and bool((out[off + works * orig:] == 3.0).all())


@pytest.mark.parametrize("step", [1, 7, 15, 16, 17, 31, 33, 1000])
def test_v1_outliers_that_leave_an_unfinished_piece(step):
    """Chunks of 0, step, 2 step, ... outliers, at random lanes: the unfinished 16-byte piece that a warp carries into its
    next chunk has every length, and the next chunk's outliers start behind it.  Enough chunks for dozens per warp."""
    n = 16 << 20
    g = torch.Generator(device=DEV).manual_seed(step)
    c = torch.arange(n // 1024, device=DEV)
    per = (c * step) % 1025
    order = torch.rand(n // 1024, 1024, generator=g, device=DEV).argsort(1)
    exponent = torch.where(order < per[:, None], torch.randint(1, 116, (n // 1024, 1024), generator=g, device=DEV), 118)
    x = (exponent << 7).to(torch.int16).view(torch.bfloat16).reshape(-1).contiguous()

    def encode(v):
        dev = v.device
        n_8, bases = torch.full((1,), n, dtype=torch.int32, device=dev), torch.full((256,), 116, dtype=torch.int32, device=dev)
        det, esc = (torch.zeros(m, dtype=torch.uint8, device=dev) for m in (codec.v1_det_bytes(n), n))
        gc = torch.zeros(1, dtype=torch.int32, device=dev)
        hz.compress_split_store(v, n_8, bases, det, torch.zeros(n, dtype=torch.uint8, device=dev), esc, gc, 1)
        return det.cpu(), esc.cpu(), int(gc)

    det, esc, count = encode(x)
    detc, escc, countc = encode(x.cpu())
    assert count == countc == int(per.sum()) and torch.equal(det, detc) and torch.equal(esc[:count], escc[:count])


def test_v1_works_that_end_inside_a_block_are_coded_up_to_their_last_whole_block():
    """Sizes that are not a multiple of 4096: the stream has offsets for whole blocks, and the base stands behind the last."""
    sizes = [6144, 4096, 2048, 10240]
    x = torch.cat([gauss(s, seed=i) for i, s in enumerate(sizes)])
    n_8 = torch.tensor(sizes, dtype=torch.int32, device=DEV)
    bases = torch.full((256,), 118, dtype=torch.int32, device=DEV)
    at = [0]
    for s in sizes:
        at.append(at[-1] + codec.align128(s + s // 8 * 3 + s // 4096 * 4 + 4))
    det = torch.zeros(at[-1], dtype=torch.uint8, device=DEV)
    scratch, esc = (torch.zeros(1 << 15, dtype=torch.uint8, device=DEV) for _ in range(2))
    gc = torch.full((4,), -1, dtype=torch.int32, device=DEV)
    hz.compress_split_store(x, n_8, bases, det, scratch, esc, gc, 4)
    start = 0
    for w, s in enumerate(sizes):
        whole = s // 4096 * 4096
        e = (bits(x[start:start + whole]).int() >> 7) & 255
        out = (e < 118) | (e > 124)
        assert int(gc[w]) == int(out.sum())
        offsets = det[at[w] + s + s // 8 * 3:][:s // 4096 * 4 + 4].clone().view(torch.int32).tolist()
        if whole:
            assert offsets == [int(out[:4096 * b].sum()) for b in range(s // 4096)] + [118]
        start += s


@pytest.mark.parametrize("n", [1, 7, 4095, 4096, 100_001, 3_000_003])
def test_v1_base_statistic_sizes(n):
    for scale in (0.02, 3.0):
        x = gauss(n, seed=n) * (scale / 0.02)
        got = torch.zeros(1, dtype=torch.int32, device=DEV)
        codec.v1_base_from_std(x, got)
        std = x.double().std().item() if n > 1 else 0.0
        want = math.floor(math.log2(max(std, 1e-30)) - 5.35 + 127.0)
        assert int(got) == min(max(want, 0), 255)


def test_v1_pad_variant_and_fused_layout():
    origs = [100, 4096, 7168, 1]
    xs = [rand_bits(o, seed=i) for i, o in enumerate(origs)]
    dense = torch.cat(xs)
    n_8 = torch.tensor([codec.pad_to_block(o) for o in origs], dtype=torch.int32, device=DEV)
    orig_n = torch.tensor(origs, dtype=torch.int32, device=DEV)
    total_pad = int(n_8.sum())
    bases = torch.full((256,), 120, dtype=torch.int32, device=DEV)
    det = torch.zeros(sum(codec.v1_det_bytes(int(p)) for p in n_8), dtype=torch.uint8, device=DEV)
    scratch = torch.zeros(total_pad, dtype=torch.uint8, device=DEV)
    esc = torch.zeros(total_pad + 128 * 4, dtype=torch.uint8, device=DEV)
    gc = torch.zeros(4, dtype=torch.int32, device=DEV)
    hz.compress_split_store_pad(dense, n_8, orig_n, bases, det, scratch, esc, gc, total_pad, 4)
    detc = torch.zeros_like(det, device="cpu"); escc = torch.zeros_like(esc, device="cpu"); gcc = torch.zeros(4, dtype=torch.int32)
    hz.compress_split_store_pad(dense.cpu(), n_8.cpu(), orig_n.cpu(), bases.cpu(), detc, scratch.cpu(), escc, gcc, total_pad, 4)
    assert torch.equal(det.cpu(), detc) and torch.equal(gc.cpu(), gcc)
    # fused layout, 3 works, GPU encode -> CPU decode and GPU decode
    per = 8192
    x = torch.cat([gauss(per, std=10.0 ** (-w), seed=w) for w in range(3)])
    n8 = torch.full((3,), per, dtype=torch.int32, device=DEV)
    nbytes = torch.zeros(3, dtype=torch.int32, device=DEV)
    sc = torch.zeros(4 * x.numel(), dtype=torch.uint8, device=DEV)
    fin = torch.zeros(4 * x.numel(), dtype=torch.uint8, device=DEV)
    g3 = torch.zeros(3, dtype=torch.int32, device=DEV)
    hz.compress_8(x, n8, nbytes, bases, sc, fin, g3, 3)
    out = torch.zeros_like(x)
    hz.decompress_8(fin, n8, nbytes, out, 3)
    assert torch.equal(bits(out), bits(x))
    outc = torch.zeros_like(x, device="cpu")
    hz.decompress_8(fin.cpu(), n8.cpu(), nbytes.cpu(), outc, 3)
    assert torch.equal(bits(outc), bits(x.cpu()))
    buf = hz.compress_8_padded(x[:9999], bases, 1)
    back = hz.decompress_8_padded(buf, 9999, torch.zeros(1, dtype=torch.int32, device=DEV), 1)
    assert torch.equal(bits(back), bits(x[:9999]))
    out2 = torch.zeros(3 * 5000, dtype=torch.bfloat16, device=DEV)
    hz.decompress_8_unpad(fin, n8, nbytes, out2, 5000, 3)
    for w in range(3):
        assert torch.equal(bits(out2[w * 5000:(w + 1) * 5000]), bits(x[w * per:w * per + 5000]))


def test_v1_base_statistic_kernel():
    x = gauss(1 << 20, 0.02, seed=1)
    bases = torch.zeros(256, dtype=torch.int32, device=DEV)
    codec.v1_base_from_std(x, bases)
    codec.v1_base_from_std(x * 0 + x, bases)   # second call reuses the zeroed accumulator
    assert int(bases[0]) == 116


@pytest.mark.parametrize("trips,more", [(4, 0), (7, 0), (7, 8), (8, -8), (8, 0), (8, 24), (11, 8), (12, 5)])
def test_v1_base_statistic_adds_every_element_once(trips, more):
    """One value among zeros, at the ends of the CTAs' trips and in between, around the last trip that is loaded without checks (of 148 SMs).
    Its logarithm lies three quarters of the way between two bases: without the value the base is another, with it twice the next."""
    nt = 8 * 148 * 1024
    n = nt * trips + more
    want = 60
    value = 2.0 ** (want - 127 + 5.35 + 0.75) * n ** 0.5
    x = torch.zeros(n, device=DEV, dtype=torch.bfloat16)
    got = torch.zeros(64, dtype=torch.int32, device=DEV)
    places = sorted({0, 7, n // 3, n - 1, n - 8, n - 9, n - n % 8 - 1, *(min(k * nt + d, n - 1) for k in range(trips + 1) for d in (-1, 0))} - {-1})
    for i, at in enumerate(places):
        x[at] = value
        codec.v1_base_from_std(x, got[i:])
        x[at] = 0
    assert got[:len(places)].tolist() == [want] * len(places)


def test_v1_base_statistic_on_several_streams_and_replayed():
    """Launches of different streams, and those of a recorded graph replayed beside them, have workspaces of their own."""
    xs = [gauss(1 << 22, std=0.02 * 4 ** i, seed=i) for i in range(4)]
    want = [math.floor(math.log2(x.double().std().item()) - 5.35 + 127.0) for x in xs]
    outs = [torch.zeros(300, dtype=torch.int32, device=DEV) for _ in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    recorded = torch.zeros(1, dtype=torch.int32, device=DEV)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        codec.v1_base_from_std(xs[3], recorded)
    torch.cuda.synchronize()
    replays = []
    for k in range(300):
        for x, out, st in zip(xs[:3], outs, streams):
            with torch.cuda.stream(st):
                codec.v1_base_from_std(x, out[k:])
        with torch.cuda.stream(streams[3]):
            recorded.zero_()
            graph.replay()
            replays.append(recorded.clone())
    torch.cuda.synchronize()
    for out, w in zip(outs[:3] + [torch.cat(replays)], want):
        assert bool((out == w).all())


# ------------------------------------------------------------------ elementwise
def test_rmsnorm_fwd_bwd():
    torch.manual_seed(0)
    for rows, cols in [(64, 4096), (33, 256), (8, 8192)]:
        x = torch.randn(rows, cols, device=DEV).bfloat16().requires_grad_()
        r = torch.randn(rows, cols, device=DEV).bfloat16().requires_grad_()
        w = (1 + 0.1 * torch.randn(cols, device=DEV)).bfloat16().requires_grad_()
        y, h = norm.add_rms_norm(x, r, w, 1e-5)
        g = torch.randn_like(y)
        (y.float() * g.float()).sum().backward()
        xf, rf, wf = (t.detach().float().requires_grad_() for t in (x, r, w))
        hf = (xf + rf).bfloat16().float()
        yf = F.rms_norm(xf + rf, (cols,), wf, 1e-5)
        (yf * g.float()).sum().backward()
        assert torch.equal(h.float(), hf)
        assert torch.allclose(y.float(), yf, atol=2e-2, rtol=2e-2)
        assert torch.allclose(x.grad.float(), xf.grad, atol=3e-2, rtol=3e-2)
        assert torch.allclose(w.grad.float(), wf.grad, atol=0.15, rtol=3e-2)
        y2 = norm.rms_norm(x.detach(), w.detach(), 1e-5)
        assert torch.allclose(y2.float(), F.rms_norm(x.detach().float(), (cols,), w.detach().float(), 1e-5), atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("rows,cols", [(1, 8), (700, 1024), (1300, 1024), (5, 1032), (461, 4096), (3, 4104), (301, 8192)])
def test_rmsnorm_walks_rows_of_every_width(rows, cols):
    """The widths at which the CTA changes, one vector more, and more rows than CTAs run at once.  Every result is rounded once
    from fp32 to eight bits: 2^-8 of a value at most (2^-8.6 of a norm of many), and the fp32 sums' 1e-5."""
    torch.manual_seed(rows + cols)
    x, r, g = (torch.randn(rows, cols, device=DEV).bfloat16() for _ in range(3))
    gh = torch.randn(rows, cols, device=DEV).bfloat16()
    w = (1 + 0.1 * torch.randn(cols, device=DEV)).bfloat16().requires_grad_()
    x.requires_grad_()
    y, h = norm.add_rms_norm(x, r, w, 1e-5)
    dx, dw = torch.autograd.grad([y, h], [x, w], [g, gh])
    assert torch.equal(h, (x.detach().float() + r.float()).bfloat16())
    hd, wd = h.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    yd = hd * (hd.pow(2).mean(-1, keepdim=True) + 1e-5).rsqrt() * wd
    dhd, dwd = torch.autograd.grad(yd, [hd, wd], g.double())
    for got, want in [(y, yd), (dx, dhd + gh.double()), (dw, dwd)]:
        assert ((got.double() - want).norm() / want.norm()).item() < 2 ** -8 + 1e-5


@pytest.mark.parametrize("rows,cols", [(888, 2048), (1480, 2048), (1481, 2048), (1481, 1032), (889, 8), (889, 1024), (890, 1032), (891, 2048), (1500, 2056), (1501, 3072), (889, 3080)])
@pytest.mark.parametrize("residual", [False, True])
def test_rmsnorm_of_many_rows_at_every_width(rows, cols, residual):
    """Either side of six and ten rows an SM of 148, of the widths at which a lane's vectors change and of the last one of a warp a row,
    with rows that do not fill a CTA.  The bounds of the test above."""
    torch.manual_seed(rows + cols)
    x, r, g = (torch.randn(rows, cols, device=DEV).bfloat16() for _ in range(3))
    w = (1 + 0.1 * torch.randn(cols, device=DEV)).bfloat16().requires_grad_()
    x.requires_grad_()
    y, h = norm.add_rms_norm(x, r, w, 1e-5) if residual else (norm.rms_norm(x, w, 1e-5), x)
    dx, dw = torch.autograd.grad(y, [x, w], g)
    if residual:
        assert torch.equal(h, (x.detach().float() + r.float()).bfloat16())
    hd, wd = h.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    yd = hd * (hd.pow(2).mean(-1, keepdim=True) + 1e-5).rsqrt() * wd
    for got, want in zip((y, dx, dw), (yd, *torch.autograd.grad(yd, [hd, wd], g.double()))):
        assert ((got.double() - want).norm() / want.norm()).item() < 2 ** -8 + 1e-5


@pytest.mark.parametrize("cols", [8, 264, 1024, 1032, 2048, 2056, 3072])
@pytest.mark.parametrize("residual", [False, True])
def test_rmsnorm_of_a_row_has_the_same_bits_among_few_and_many(cols, residual):
    """A warp adds a row's squares up in the order of the CTA that takes it where rows are few."""
    torch.manual_seed(cols)
    x, r = (torch.randn(3000, cols, device=DEV).bfloat16() for _ in range(2))
    w = torch.randn(cols, device=DEV).bfloat16()
    f = lambda a, b: norm.add_rms_norm(a, b, w, 1e-5)[0] if residual else norm.rms_norm(a, w, 1e-5)
    assert torch.equal(f(x, r), torch.cat([f(a, b) for a, b in zip(x.split(750), r.split(750))]))


@pytest.mark.parametrize("n", [8, 2048, 2056, 4096, 4104, 100_000])
def test_adamw_updates_every_vector_once(n):
    """Around a thread's second vector and a CTA's 512; elements are independent, so each size has the bits of the largest.
    Rounded once to eight bits: 2^-8 of a value at most."""
    torch.manual_seed(3)
    whole = [(torch.randn(100_000, device=DEV) * s).bfloat16() for s in (1.0, 0.1, 0.01)] + [torch.rand(100_000, device=DEV).bfloat16()]
    run = lambda t: _lib.check(_lib.cuda().zc_adamw(*(v.data_ptr() for v in t), t[0].numel(), 0, 0, 0, 1e-3, 0.9, 0.95, 1e-8, 0.01, 0.1,
                                                    0.05, 0, _lib.stream_ptr(t[0].device)), "zc_adamw")
    part = [v[:n].clone() for v in whole]
    p, g, m, v = (t.double() for t in part)
    run(part)
    run(whole)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b[:n]) for a, b in zip(part, whole))
    m, v = 0.9 * m + 0.1 * g, 0.95 * v + 0.05 * g * g
    p = p * (1 - 1e-3 * 0.01) - 1e-3 / 0.1 * m / (v.sqrt() / 0.05 ** 0.5 + 1e-8)
    for got, want in zip((part[0], part[2], part[3]), (p, m, v)):
        assert ((got.double() - want).norm() / want.norm()).item() < 2 ** -8 + 1e-5


@pytest.mark.parametrize("n", [8, 2048, 2056, 4096, 4104, 6152, 100_000])
def test_adamw_in_32_bits_updates_every_vector_once(n):
    """Streams of 32 bits, whose threads' second vectors are a grid further: each size has the bits of the largest.  A few roundings to
    24 bits, of sums of two terms with a difference in one of them."""
    torch.manual_seed(4)
    whole = [torch.randn(100_000, device=DEV) * s for s in (1.0, 0.1, 0.01)] + [torch.rand(100_000, device=DEV)]
    run = lambda t: _lib.check(_lib.cuda().zc_adamw(*(v.data_ptr() for v in t), t[0].numel(), 1, 1, 1, 1e-3, 0.9, 0.95, 1e-8, 0.01, 0.1,
                                                    0.05, 0, _lib.stream_ptr(t[0].device)), "zc_adamw")
    part = [v[:n].clone() for v in whole]
    p, g, m, v = (t.double() for t in part)
    run(part)
    run(whole)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b[:n]) for a, b in zip(part, whole))
    m, v = 0.9 * m + 0.1 * g, 0.95 * v + 0.05 * g * g
    p = p * (1 - 1e-3 * 0.01) - 1e-3 / 0.1 * m / (v.sqrt() / 0.05 ** 0.5 + 1e-8)
    for got, want in zip((part[0], part[2], part[3]), (p, m, v)):
        assert ((got.double() - want).norm() / want.norm()).item() < 2 ** -20


def test_swiglu_fwd_bwd():
    torch.manual_seed(1)
    gu = torch.randn(257, 2 * 1024, device=DEV).bfloat16().requires_grad_()
    out = swiglu.swiglu(gu)
    g = torch.randn_like(out)
    out.backward(g)
    gf = gu.detach().float().requires_grad_()
    ref = F.silu(gf[:, :1024]) * gf[:, 1024:]
    ref.backward(g.float())
    assert torch.allclose(out.float(), ref, atol=2e-2, rtol=2e-2)
    assert torch.allclose(gu.grad.float(), gf.grad, atol=3e-2, rtol=3e-2)


def test_rope_matches_cpu_path():
    torch.manual_seed(2)
    S, Hq, Hkv, D = 96, 4, 2, 128
    cos, sin = rope.rope_tables(S, D, 500000.0, DEV)
    x = torch.randn(2 * S, (Hq + 2 * Hkv) * D, device=DEV).bfloat16()
    ref = rope._rotate(x.cpu().float(), cos.cpu(), sin.cpu(), Hq + Hkv, D, S, 1.0)
    got = rope._rotate(x.clone(), cos, sin, Hq + Hkv, D, S, 1.0)
    assert torch.allclose(got.float().cpu(), ref, atol=2e-2, rtol=2e-2)
    back = rope._rotate(got.clone(), cos, sin, Hq + Hkv, D, S, -1.0)
    assert torch.allclose(back.float(), x.float(), atol=5e-2, rtol=5e-2)
    assert torch.equal(got[:, (Hq + Hkv) * D:], x[:, (Hq + Hkv) * D:])   # v heads untouched


@pytest.mark.parametrize("V", [8192, 50257, 128256])
def test_cross_entropy_fwd_bwd(V):
    torch.manual_seed(3)
    T = 64
    logits = (torch.randn(T, V, device=DEV) * 2).bfloat16()
    labels = torch.randint(0, V, (T,), device=DEV)
    labels[5] = -100
    lf = logits.float().requires_grad_()
    ref = F.cross_entropy(lf, labels, ignore_index=-100)
    ref.backward()
    work = logits.clone().requires_grad_()
    out = loss.cross_entropy(work * 1, labels)
    out.backward()
    assert abs(out.item() - ref.item()) < 2e-3
    assert torch.allclose(work.grad.float(), lf.grad, atol=2e-4, rtol=2e-2)


@pytest.mark.parametrize("V", [8, 36864, 36871, 36872, 73719, 73720, 100001])
def test_cross_entropy_at_the_edges_of_its_clusters(V):
    """The longest row of one and of two CTAs, the first that needs more, ragged rows whose label lies among the
    last V % 8 columns, in the first and the last share, masked logits, a row that is ignored.  fp32 against 64 bits: the loss to 1e-5, the
    gradient to half a bf16 unit (2^-9) of its value plus fp32 sums' 1e-5."""
    torch.manual_seed(V)
    T, ld = 7, (V + 7) // 8 * 8 + 8
    buf = (torch.randn(T, ld, device=DEV) * 2).bfloat16()
    buf[3, :V // 2] = float("-inf")                 # masked logits, whole threads' shares of them
    labels = torch.tensor([0, V - 1, V // 8 * 8 - 1, V // 2, -100, max(0, V - 2), V // 4 * 3], device=DEV)
    lf = buf[:, :V].double().requires_grad_()
    ref = F.cross_entropy(lf, labels, ignore_index=-100)
    ref.backward()
    work = buf.clone()
    logits = work[:, :V].requires_grad_()
    out = loss.cross_entropy(logits, labels)
    (grad,) = torch.autograd.grad(out, logits)
    assert abs(out.item() - ref.item()) <= 1e-5 * max(1.0, ref.item())
    assert ((grad.double() - lf.grad).abs() <= lf.grad.abs() * (2 ** -8 + 1e-5) + 1e-12).all()
    assert (work[:, V:] == 0).all()


@pytest.mark.parametrize("V", [8192, 1001, 50257, 100001])
def test_cross_entropy_of_a_label_outside_the_vocabulary_is_nan(V):
    """One CTA a row, a ragged row, two CTAs a row and the kernel for long rows: no logit outside the row is read and no row's
    loss is left unwritten; the other rows are as ever."""
    from fsdp_comm_opt_b200 import _lib

    torch.manual_seed(V)
    ld = (V + 7) // 8 * 8
    logits = torch.randn(6, ld, device=DEV).bfloat16()
    labels = torch.tensor([3, -1, V, V - 1, 1 << 40, -100], device=DEV)
    ref = torch.logsumexp(logits[:, :V].double(), 1)
    want = [ref[0] - logits[0, 3].double(), ref[3] - logits[3, V - 1].double()]
    rows = torch.full((6,), 7.0, device=DEV)
    inv = torch.ones(1, device=DEV)
    _lib.check(_lib.cuda().zc_ce_fwd_bwd_ld(logits.data_ptr(), labels.data_ptr(), rows.data_ptr(), inv.data_ptr(), 6, V, ld, -100,
                                            _lib.stream_ptr(logits.device)), "zc_ce_fwd_bwd")
    assert rows.isnan().tolist() == [False, True, True, False, True, False] and rows[5] == 0
    for got, w in zip((rows[0], rows[3]), want):
        assert abs(got.item() - w.item()) < 1e-4 * abs(w.item())       # fp32 sums of fast exponentials
    assert (logits[:, :V].float().sum(1)[[0, 3, 5]].abs() < 0.05).all()     # softmax minus one-hot, in bf16


def test_int8_quant_kernels():
    torch.manual_seed(4)
    n, world = 100003, 3
    buf = torch.zeros(world, quant.packed_bytes(n), dtype=torch.uint8, device=DEV)
    xs = [(torch.randn(n, device=DEV) * 0.01 * (r + 1)).bfloat16() for r in range(world)]
    for r in range(world):
        quant.quantize_pack(xs[r], buf[r])
    out = torch.zeros(world * n, dtype=torch.bfloat16, device=DEV)
    quant.dequantize_unpack(buf, n, out)
    for r in range(world):
        scale = xs[r].float().abs().max() / 127
        assert torch.allclose(buf[r, :4].view(torch.float32), scale.reshape(1))
        assert (out[r * n:(r + 1) * n].float() - xs[r].float()).abs().max() <= scale * 1.01


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("n,world", [(1, 1), (7, 3), (16, 2), (4099, 5), (1 << 19, 2), ((1 << 19) + 9, 3)])
def test_int8_vector_paths_and_their_edges(n, world, dt):
    """One-launch and three-launch quantiser, output rows at every alignment of the dequantiser."""
    torch.manual_seed(n)
    buf = torch.zeros(world, quant.packed_bytes(n), dtype=torch.uint8, device=DEV)
    xs = [(torch.randn(n, device=DEV) * 0.02).to(dt) for _ in range(world)]
    for r in range(world):
        quant.quantize_pack(xs[r], buf[r])
    out = torch.full((world * n + 8,), 7.0, dtype=dt, device=DEV)
    quant.dequantize_unpack(buf, n, out[:world * n])
    assert bool((out[world * n:] == 7.0).all())
    for r in range(world):
        scale = buf[r, :4].view(torch.float32)
        assert torch.allclose(scale, (xs[r].float().abs().max() / 127).clamp_min(1e-8).reshape(1))
        q = buf[r, 16:16 + n].view(torch.int8).float()
        # the approximate division may round a quotient that lies on a half the other way
        assert (q - xs[r].float() / scale).abs().max() <= 0.5 + 1e-4
        assert torch.equal(out[r * n:(r + 1) * n], (q * scale).to(dt))
        assert not buf[r, 16 + n:].any()


@pytest.mark.parametrize("world", [65535, 65536, 140_000])
def test_int8_contributions_beyond_a_grids_rows(world):
    n = 11
    g = torch.Generator(device=DEV).manual_seed(world)
    buf = torch.randint(0, 256, (world, quant.packed_bytes(n)), generator=g, device=DEV).to(torch.uint8)
    scale = torch.rand(world, generator=g, device=DEV) + 0.5
    buf[:, :4] = scale.view(world, 1).view(torch.uint8)
    out = torch.zeros(world * n, dtype=torch.float32, device=DEV)
    quant.dequantize_unpack(buf, n, out)
    ref = buf[:, 16:16 + n].contiguous().view(torch.int8).float() * scale[:, None]
    assert torch.equal(out.view(world, n), ref)


@pytest.mark.parametrize("pdt,sdt", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32)])
def test_fused_adamw_kernel(pdt, sdt):
    torch.manual_seed(5)
    p0 = torch.randn(100003, device=DEV)
    p1 = torch.nn.Parameter(p0.to(pdt))
    p2 = torch.nn.Parameter(p0.to(pdt).float())
    o1 = adamw.FusedAdamW([p1], lr=1e-2, weight_decay=0.1)
    o2 = torch.optim.AdamW([p2], lr=1e-2, weight_decay=0.1)
    for _ in range(4):
        g = torch.randn(100003, device=DEV).to(pdt)
        p1.grad, p2.grad = g.clone(), g.float()
        o1.step(), o2.step()
    tol = 3e-2 if pdt == torch.bfloat16 else 1e-5
    assert torch.allclose(p1.float(), p2, atol=tol, rtol=tol)
    assert o1.kernel_launches == 4


# ------------------------------------------------------------------ tensor cores
@pytest.mark.parametrize("a_major,b_major", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_umma_descriptor_conventions(a_major, b_major):
    torch.manual_seed(6)
    ksteps = 3
    K = 64 * ksteps
    A = torch.randn(128, K, device=DEV).bfloat16()
    B = torch.randn(128, K, device=DEV).bfloat16()
    Ag = A if a_major == 0 else A.t().contiguous()
    Bg = B if b_major == 0 else B.t().contiguous()
    D = torch.zeros(128, 128, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    rc = _lib.cuda().zc_umma_selftest(Ag.data_ptr(), Bg.data_ptr(), D.data_ptr(), a_major, b_major, ksteps,
                                      status.data_ptr(), _lib.stream_ptr())
    assert rc == 0
    torch.cuda.synchronize()
    assert int(status[0]) == 0, "bounded wait expired"
    ref = A.float() @ B.float().t()
    assert torch.allclose(D, ref, atol=1e-2, rtol=1e-3), (D - ref).abs().max().item()


def _attn_ref(qkv, Hq, Hkv):
    q, k, v = qkv[:, :, :Hq], qkv[:, :, Hq:Hq + Hkv], qkv[:, :, Hq + Hkv:]
    g = Hq // Hkv
    q, k, v = (t.transpose(1, 2).float() for t in (q, k, v))
    k, v = k.repeat_interleave(g, 1), v.repeat_interleave(g, 1)
    return F.scaled_dot_product_attention(q, k, v, is_causal=True).transpose(1, 2)


@pytest.mark.parametrize("impl", ["2q+kt", "ws+ws", "simple+simple"])
@pytest.mark.parametrize("B,S,Hq,Hkv,D", [(1, 128, 1, 1, 128), (2, 384, 4, 2, 128), (1, 200, 2, 2, 64), (1, 512, 8, 2, 128),
                                          (1, 1000, 4, 1, 128), (2, 2048, 8, 2, 128)])
def test_attention_fwd_bwd(B, S, Hq, Hkv, D, impl, monkeypatch):
    fwd_impl, bwd_impl = impl.split("+")
    monkeypatch.setattr(attention, "_FWD_IMPL", fwd_impl)
    monkeypatch.setattr(attention, "_BWD_IMPL", bwd_impl)
    torch.manual_seed(7)
    qkv = (torch.randn(B, S, Hq + 2 * Hkv, D, device=DEV) * 0.5).bfloat16().requires_grad_()
    o = attention.causal_attention(qkv * 1, Hq, Hkv)
    g = (torch.randn_like(o) * 0.5)
    o.backward(g)
    torch.cuda.synchronize()
    assert attention.status_read_and_clear() == 0
    qf = qkv.detach().float().requires_grad_()
    ref = _attn_ref(qf, Hq, Hkv)
    ref.backward(g.float())
    assert torch.allclose(o.float(), ref, atol=2e-2, rtol=2e-2), (o.float() - ref).abs().max().item()
    err = (qkv.grad.float() - qf.grad).abs().max().item()
    assert torch.allclose(qkv.grad.float(), qf.grad, atol=3e-2, rtol=3e-2), err


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,S,Hq,Hkv", [(1, 1, 1, 1), (2, 65, 2, 1), (1, 127, 3, 3), (1, 129, 4, 1), (3, 256, 2, 2),
                                        (1, 257, 8, 2), (1, 769, 2, 2), (2, 1024, 25, 25)])
def test_attention_at_the_edges_of_key_and_query_tiles(B, S, Hq, Hkv, D):
    """One, a part of one, exactly one and one more than a tile of 128 (and a pair of tiles); scores that rise
    along the sequence in the last heads, so that the accumulator is rescaled at both head sizes.  The bound:
    bf16 probabilities and score gradients (2^-9 relative each) summed over a row, against the result's norm."""
    torch.manual_seed(S * D)
    qkv = torch.randn(B, S, Hq + 2 * Hkv, D, device=DEV) * 0.5
    qkv[:, :, Hq - 1] = 1.0
    qkv[:, :, Hq + Hkv - 1] += torch.linspace(-2.0, 2.0, S, device=DEV)[None, :, None]
    qkv = qkv.bfloat16().requires_grad_()
    o = attention.causal_attention(qkv, Hq, Hkv)
    g = torch.randn_like(o)
    (dqkv,) = torch.autograd.grad(o, qkv, g)
    torch.cuda.synchronize()
    assert attention.status_read_and_clear() == 0
    qf = qkv.detach().double().requires_grad_()
    q, k, v = (t.transpose(1, 2) for t in qf.split([Hq, Hkv, Hkv], 2))
    k, v = (t.repeat_interleave(Hq // Hkv, 1) for t in (k, v))
    p = torch.matmul(q, k.transpose(2, 3)) / D ** 0.5
    p = p.masked_fill(torch.ones(S, S, dtype=torch.bool, device=DEV).triu(1), float("-inf")).softmax(-1)
    ref = torch.matmul(p, v).transpose(1, 2)
    (dref,) = torch.autograd.grad(ref, qf, g.double())
    assert ((o - ref).norm() / ref.norm()).item() < 6e-3
    assert ((dqkv - dref).norm() / dref.norm()).item() < 1e-2


@pytest.mark.parametrize("B,S,Hq,Hkv,D", [(1, 2048, 32, 8, 128), (1, 1920, 16, 8, 64), (2, 1000, 8, 2, 128), (1, 1100, 16, 2, 128),
                                          (1, 130, 8, 1, 64)])
def test_attention_backward_shared_by_a_cluster(B, S, Hq, Hkv, D):
    """Two, four and eight CTAs to a key block's query heads, at ragged lengths.  The bound of the test above: bf16
    probabilities and score gradients."""
    torch.manual_seed(S)
    qkv = (torch.randn(B, S, Hq + 2 * Hkv, D, device=DEV) * 0.5).bfloat16().requires_grad_()
    o = attention.causal_attention(qkv, Hq, Hkv)
    g = torch.randn_like(o)
    (dqkv,) = torch.autograd.grad(o, qkv, g)
    torch.cuda.synchronize()
    assert attention.status_read_and_clear() == 0
    qf = qkv.detach().float().requires_grad_()
    (dref,) = torch.autograd.grad(_attn_ref(qf, Hq, Hkv), qf, g.float())
    for part in (slice(0, Hq), slice(Hq, Hq + Hkv), slice(Hq + Hkv, None)):
        d, r = dqkv[:, :, part].float(), dref[:, :, part]
        assert ((d - r).norm() / r.norm()).item() < 1e-2


@pytest.mark.parametrize("B,S,Hq,Hkv,D,parts", [(1, 700, 16, 2, 64, 8), (1, 1100, 16, 2, 128, 4), (1, 1536, 8, 2, 128, 4), (1, 1024, 64, 8, 128, 2),
                                                (2, 1100, 8, 2, 128, 2), (1, 1024, 32, 8, 128, 2), (1, 900, 32, 8, 64, 2), (1, 1920, 16, 8, 64, 1)])
def test_attention_backward_is_shared_by_clusters_that_run_at_once(B, S, Hq, Hkv, D, parts):
    """dQ is added up in the order in which key blocks come to it.  That is the same at nearly every run while all clusters run at once, and
    another at every run where more CTAs to a key block take a second wave.  Against fp32 within the bound of the test above."""
    lib = _lib.cuda()
    assert lib.zc_attn_bwd_parts(S, Hq, Hkv, B, D) == parts
    assert (S + 127) // 128 * Hkv * B <= lib.zc_attn_bwd_blocks_at_once(parts, D)
    torch.manual_seed(S)
    qkv = torch.randn(B, S, Hq + 2 * Hkv, D, device=DEV).bfloat16().requires_grad_()
    o = attention.causal_attention(qkv, Hq, Hkv)
    g = torch.randn_like(o)
    weights = torch.randint(1 << 20, qkv.shape, device=DEV)
    runs = [torch.autograd.grad(o, qkv, g, retain_graph=True)[0] for _ in range(20)]
    assert attention.status_read_and_clear() == 0
    sums = [int((r.view(torch.int16) * weights).sum()) for r in runs]
    assert max(map(sums.count, sums)) > len(runs) // 2
    qf = qkv.detach().float().requires_grad_()
    (dref,) = torch.autograd.grad(_attn_ref(qf, Hq, Hkv), qf, g.float())
    assert ((runs[0].float() - dref).norm() / dref.norm()).item() < 1e-2


@pytest.mark.parametrize("impl", ["2q+kt", "ws+ws"])
def test_attention_rising_scores_rescale_the_accumulator(impl, monkeypatch):
    """Keys whose scores grow along the sequence raise the running row maximum again and again, so
    the forward kernel must rescale the output it has accumulated so far (the two-tile kernel does
    that in TMEM, and only when the maximum rose by more than a factor of 2^8)."""
    fwd_impl, bwd_impl = impl.split("+")
    monkeypatch.setattr(attention, "_FWD_IMPL", fwd_impl)
    monkeypatch.setattr(attention, "_BWD_IMPL", bwd_impl)
    torch.manual_seed(11)
    B, S, Hq, Hkv, D = 1, 1024, 2, 1, 128
    qkv = torch.randn(B, S, Hq + 2 * Hkv, D, device=DEV) * 0.5
    # q = +1 everywhere, k ramps from -3 to +3: scores rise by ~70 (in log2 units ~100) over the row
    qkv[:, :, :Hq] = 1.0 + 0.05 * torch.randn(B, S, Hq, D, device=DEV)
    ramp = torch.linspace(-3.0, 3.0, S, device=DEV)[None, :, None, None]
    qkv[:, :, Hq:Hq + Hkv] = ramp + 0.05 * torch.randn(B, S, Hkv, D, device=DEV)
    qkv = qkv.bfloat16().requires_grad_()
    o = attention.causal_attention(qkv * 1, Hq, Hkv)
    g = torch.randn_like(o) * 0.5
    o.backward(g)
    torch.cuda.synchronize()
    assert attention.status_read_and_clear() == 0
    qf = qkv.detach().float().requires_grad_()
    ref = _attn_ref(qf, Hq, Hkv)
    ref.backward(g.float())
    assert torch.allclose(o.float(), ref, atol=3e-2, rtol=3e-2), (o.float() - ref).abs().max().item()
    assert torch.allclose(qkv.grad.float(), qf.grad, atol=5e-2, rtol=5e-2), (qkv.grad.float() - qf.grad).abs().max().item()


@pytest.mark.parametrize("S", [1024, 3000])
def test_attention_forward_rounds_probabilities_of_the_running_maximum(S):
    """Head dimension 64: no further from 64 bits than probabilities that are rounded to bf16 relative to the running maximum
    of 128 keys at a time, with all else exact (the largest of a row are then exact ones).  Errors of so many values agree
    within a quarter of a percent; a reference that lags behind the maximum is 1.5 to 2 % further off."""
    H, D = 8, 64
    torch.manual_seed(S)
    qkv = torch.randn(1, S, 3 * H, D, device=DEV).bfloat16()
    o = attention.causal_attention(qkv, H, H)[0].transpose(0, 1).double()
    q, k, v = (t.transpose(0, 1).double() for t in qkv[0].split(H, dim=1))
    s = (q @ k.transpose(1, 2) / math.sqrt(D)).masked_fill(~torch.ones(S, S, dtype=torch.bool, device=DEV).tril(), -math.inf)
    exact = s.softmax(-1) @ v
    acc, total, top = torch.zeros_like(o), torch.zeros(H, S, 1, device=DEV).double(), torch.full((H, S, 1), -math.inf, device=DEV).double()
    for b in s.split(128, dim=-1):
        new = torch.maximum(top, b.amax(-1, keepdim=True))
        p = (b - new).exp()
        shrink = (top - new).exp()
        acc = acc * shrink + p.bfloat16().double() @ v[:, :b.shape[-1]]
        v = v[:, b.shape[-1]:]
        total = total * shrink + p.sum(-1, keepdim=True)
        top = new
    rounded = (acc / total).bfloat16().double()
    assert (o - exact).norm() <= 1.005 * (rounded - exact).norm()


def test_attention_with_fused_rope_matches_unfused():
    torch.manual_seed(8)
    B, S, Hq, Hkv, D = 1, 256, 4, 2, 128
    cos, sin = rope.rope_tables(S, D, 10000.0, DEV)
    qkv = (torch.randn(B, S, Hq + 2 * Hkv, D, device=DEV) * 0.5).bfloat16().requires_grad_()
    o = attention.causal_attention((qkv * 1).contiguous(), Hq, Hkv, None, cos, sin)
    g = torch.randn_like(o) * 0.5
    o.backward(g)
    qf = qkv.detach().float().requires_grad_()
    half = D // 2
    rot = qf[:, :, :Hq + Hkv]
    c, s = cos[None, :, None, :], sin[None, :, None, :]
    a, b = rot[..., :half], rot[..., half:]
    rotated = torch.cat([torch.cat([a * c - b * s, b * c + a * s], -1), qf[:, :, Hq + Hkv:]], 2)
    ref = _attn_ref(rotated, Hq, Hkv)
    ref.backward(g.float())
    assert torch.allclose(o.float(), ref, atol=3e-2, rtol=3e-2)
    assert torch.allclose(qkv.grad.float(), qf.grad, atol=4e-2, rtol=4e-2)


# ------------------------------------------------------------------ GPT-2 family ops
@pytest.mark.parametrize("rows,cols", [(64, 1600), (300, 256), (17, 4096), (8, 8192)])
def test_layernorm_fwd_bwd(rows, cols):
    torch.manual_seed(21)
    x = (torch.randn(rows, cols, device=DEV) * 2 + 0.5).bfloat16().requires_grad_()
    w = (1 + 0.1 * torch.randn(cols, device=DEV)).bfloat16().requires_grad_()
    b = (0.1 * torch.randn(cols, device=DEV)).bfloat16().requires_grad_()
    y = gpt2_ops.layer_norm(x, w, b, 1e-5)
    g = torch.randn_like(y)
    y.backward(g)
    xf, wf, bf = (t.detach().float().requires_grad_() for t in (x, w, b))
    ref = F.layer_norm(xf, (cols,), wf, bf, 1e-5)
    ref.backward(g.float())
    assert torch.allclose(y.float(), ref, atol=3e-2, rtol=2e-2)
    assert torch.allclose(x.grad.float(), xf.grad, atol=3e-2, rtol=3e-2), (x.grad.float() - xf.grad).abs().max().item()
    assert torch.allclose(w.grad.float(), wf.grad, atol=0.02 * rows ** 0.5 + 0.05, rtol=3e-2)
    assert torch.allclose(b.grad.float(), bf.grad, atol=0.02 * rows ** 0.5 + 0.05, rtol=3e-2)


@pytest.mark.parametrize("rows,cols", [(128, 6400), (33, 1024)])
def test_bias_gelu_fwd_bwd(rows, cols):
    torch.manual_seed(22)
    x = (torch.randn(rows, cols, device=DEV) * 1.5).bfloat16().requires_grad_()
    b = (0.2 * torch.randn(cols, device=DEV)).bfloat16().requires_grad_()
    y = gpt2_ops.bias_gelu(x, b)
    g = torch.randn_like(y)
    y.backward(g)
    xf, bf = (t.detach().float().requires_grad_() for t in (x, b))
    ref = F.gelu(xf + bf, approximate="tanh")
    ref.backward(g.float())
    assert torch.allclose(y.float(), ref, atol=2e-2, rtol=2e-2)
    assert torch.allclose(x.grad.float(), xf.grad, atol=2e-2, rtol=2e-2)
    assert torch.allclose(b.grad.float(), bf.grad, atol=0.02 * rows ** 0.5 + 0.05, rtol=3e-2)


@pytest.mark.parametrize("rows,cols,main_grad", [(64, 1600, None), (300, 256, torch.bfloat16), (2048, 1600, torch.float32)])
def test_add_layernorm_and_direct_gradient_delivery(rows, cols, main_grad):
    """LayerNorm fused with the residual add in front of it, the gradient arriving through the sum added
    inside the backward kernel, and dw / db written (or accumulated) straight into ``main_grad``."""
    torch.manual_seed(23)
    x = (torch.randn(rows, cols, device=DEV) * 2).bfloat16().requires_grad_()
    r = (torch.randn(rows, cols, device=DEV)).bfloat16().requires_grad_()
    w = (1 + 0.1 * torch.randn(cols, device=DEV)).bfloat16().requires_grad_()
    b = (0.1 * torch.randn(cols, device=DEV)).bfloat16().requires_grad_()
    if main_grad is not None:
        for p_ in (w, b):
            p_.main_grad = torch.full((cols,), 0.5, dtype=main_grad, device=DEV)
            p_.main_grad_written = True            # accumulate on top of the 0.5
    y, h = gpt2_ops.add_layer_norm(x, r, w, b, 1e-5)
    g, gh = torch.randn_like(y), torch.randn_like(h)
    torch.autograd.backward([y, h], [g, gh])
    xf, rf, wf, bf = (t.detach().float().requires_grad_() for t in (x, r, w, b))
    hf = (xf + rf)
    hq = hf.bfloat16().float()                     # the kernel normalises the stored (rounded) sum
    ref = F.layer_norm(hf + (hq - hf).detach(), (cols,), wf, bf, 1e-5)
    torch.autograd.backward([ref, hf], [g.float(), gh.float()])
    assert torch.equal(h.float(), hq)
    assert torch.allclose(y.float(), ref, atol=3e-2, rtol=2e-2)
    assert torch.allclose(x.grad.float(), xf.grad, atol=4e-2, rtol=3e-2)
    assert torch.equal(x.grad, r.grad)
    tol = dict(atol=0.02 * rows ** 0.5 + 0.05, rtol=3e-2)
    if main_grad is None:
        assert torch.allclose(w.grad.float(), wf.grad, **tol) and torch.allclose(b.grad.float(), bf.grad, **tol)
    else:
        assert w.grad is None and b.grad is None
        assert torch.allclose(w.main_grad.float() - 0.5, wf.grad, **tol)
        assert torch.allclose(b.main_grad.float() - 0.5, bf.grad, **tol)


@pytest.mark.parametrize("T,K,N", [(2048, 1600, 4800), (300, 256, 1000)])
def test_linear_with_bias_in_the_gemm_epilogue(T, K, N):
    from fsdp_comm_opt_b200.ops import gemm

    torch.manual_seed(24)
    x = (torch.randn(T, K, device=DEV) * 0.5).bfloat16().requires_grad_()
    w = (torch.randn(N, K, device=DEV) * 0.05).bfloat16().requires_grad_()
    b = torch.randn(N, device=DEV).bfloat16().requires_grad_()
    b.main_grad = torch.zeros(N, dtype=torch.bfloat16, device=DEV)
    b.main_grad_written = False
    g = torch.randn(T, N, device=DEV).bfloat16()
    before = _lib.launch_count()
    y = gemm.linear(x, w, b)
    y.backward(g)
    torch.cuda.synchronize()
    assert _lib.launch_count() - before >= 4          # three GEMMs and the column-sum kernel pair
    xf, wf, bf = (t.detach().float().requires_grad_() for t in (x, w, b))
    ref = xf @ wf.t() + bf
    ref.backward(g.float())
    assert torch.allclose(y.float(), ref, atol=2e-2 * float(ref.abs().max()), rtol=2e-2)
    assert b.grad is None and b.main_grad_written
    assert torch.allclose(b.main_grad.float(), bf.grad, atol=0.02 * T ** 0.5 + 0.1, rtol=3e-2)
    assert torch.allclose(x.grad.float(), xf.grad, atol=2e-2 * float(xf.grad.abs().max()), rtol=3e-2)
    assert torch.allclose(w.grad.float(), wf.grad, atol=2e-2 * float(wf.grad.abs().max()), rtol=3e-2)


# ------------------------------------------------------------------ embedding gradient
@pytest.mark.parametrize("n,dim,rows,accumulate", [(1, 8, 5, False), (31, 256, 64, True), (1025, 1600, 300, False),
                                                   (4096, 2056, 50257, True), (8192, 64, 3, False), (8192, 16, 1, True)])
def test_embedding_gradient_in_the_flat_buffer(n, dim, rows, accumulate):
    """One position, repeated ids (8192 positions of one row), widths below, at and past a block's 2048 columns, an old
    gradient to add to.  fp32 sums of m bf16 terms rounded once: 2^-9 relative plus m 2^-24 of the terms' magnitudes."""
    from fsdp_comm_opt_b200.ops.embedding import embedding

    torch.manual_seed(n)
    w = torch.nn.Parameter(torch.randn(rows, dim, device=DEV).bfloat16())
    w.main_grad = torch.randn(rows, dim, device=DEV).bfloat16()
    w.main_grad_written = accumulate
    old = w.main_grad.double() * accumulate
    ids = torch.randint(0, rows, (n,), device=DEV)
    out = embedding(ids, w)
    assert torch.equal(out, w.detach()[ids])
    g = torch.randn(n, dim, device=DEV).bfloat16()
    out.backward(g)
    assert w.grad is None and w.main_grad_written
    ref = old.index_add(0, ids, g.double())
    mag = old.abs().index_add(0, ids, g.double().abs())
    assert ((w.main_grad.double() - ref).abs() <= ref.abs() * 2 ** -8 + mag * n * 2 ** -24 + 1e-30).all()
    hook = w.register_hook(lambda t: None)     # a hook on the table still sees its gradient
    embedding(ids, w).backward(g)
    assert w.grad is not None
    hook.remove()


@pytest.mark.parametrize("draw", ["equal", "half", "zipf", "nine"])
@pytest.mark.parametrize("n,dim", [(4096, 4096), (8192, 8192), (4096, 1600), (8192, 200)])
def test_embedding_gradient_of_frequent_ids(n, dim, draw):
    """A padded batch, half of one, word frequencies, and ids just frequent enough to be divided over blocks: the sums, and
    no more time than PyTorch's sorted gradient and its copy take."""
    from fsdp_comm_opt_b200.ops.embedding import embedding

    torch.manual_seed(dim)
    rows = 2000
    ids = torch.randint(0, rows, (n,), device=DEV)
    if draw == "equal":
        ids.fill_(7)
    elif draw == "half":
        ids[n // 2:] = 7
    elif draw == "zipf":
        ids = torch.multinomial(1.0 / torch.arange(1, rows + 1, device=DEV), n, replacement=True)
    else:
        ids = torch.arange(n, device=DEV) // 9
    w = torch.nn.Parameter(torch.zeros(rows, dim, dtype=torch.bfloat16, device=DEV))
    w.main_grad = torch.ones_like(w)
    w.main_grad_written = False
    g = torch.randn(n, dim, device=DEV).bfloat16()
    out = embedding(ids, w)
    out.backward(g, retain_graph=True)
    ref = torch.zeros(rows, dim, dtype=torch.float64, device=DEV).index_add(0, ids, g.double())
    mag = torch.zeros(rows, dim, dtype=torch.float64, device=DEV).index_add(0, ids, g.double().abs())
    # m fp32 additions of bf16 terms, rounded once: 2^-9 relative plus m 2^-24 of the terms' magnitudes, m at most n
    assert ((w.main_grad.double() - ref).abs() <= ref.abs() * 2 ** -8 + mag * n * 2 ** -24 + 1e-30).all()

    def ours():
        w.main_grad_written = False
        out.backward(g, retain_graph=True)

    dense = torch.empty_like(w.main_grad)

    def sorted_gradient():
        dense.copy_(torch.ops.aten.embedding_dense_backward(g, ids, rows, -1, False))

    def best(fn):
        times = []
        for _ in range(8):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            torch.cuda._sleep(200_000)          # the host is ahead of the device: launches are not what is compared
            a.record()
            fn()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    assert best(ours) < best(sorted_gradient)


# ------------------------------------------------------------------ GEMM
@pytest.mark.parametrize("backend,M,N,K", [
    ("tcgen05", 128, 128, 128), ("tcgen05", 256, 512, 384), ("tcgen05", 4096, 1536, 1024), ("tcgen05", 384, 256, 4096),
    ("tcgen05", 128, 384, 128), ("tcgen05", 4096, 4096, 14336),
    # the two-SM kernel (the default backend): whole tiles, a split-K tail (4096 x 6144: 384 tiles on 74
    # clusters), and edge tiles in M, N and K
    ("tcgen05_2sm", 256, 256, 128), ("tcgen05_2sm", 512, 768, 256), ("tcgen05_2sm", 4096, 6144, 1024),
    ("tcgen05_2sm", 4096, 4096, 14336), ("tcgen05_2sm", 384, 640, 192), ("tcgen05_2sm", 2048, 1600, 1608),
    ("tcgen05_2sm", 136, 128, 136)])
def test_tcgen05_gemm_three_forms(backend, M, N, K):
    from fsdp_comm_opt_b200.ops import gemm

    torch.manual_seed(9)
    gemm.set_backend(backend)
    try:
        x = (torch.randn(M, K, device=DEV) * 0.5).bfloat16()
        w = (torch.randn(N, K, device=DEV) * 0.5).bfloat16()
        dy = (torch.randn(M, N, device=DEV) * 0.5).bfloat16()
        before = _lib.launch_count()
        y = gemm.gemm(x, w, False, True)            # forward
        dx = gemm.gemm(dy, w, False, False)         # dgrad:  [M,N] @ [N,K]
        dw = gemm.gemm(dy, x, True, False)          # wgrad:  [M,N]^T @ [M,K]  (needs N % 128 == 0 as "M")
        assert _lib.launch_count() - before == 3, "the hand-written kernel must have been taken"
        torch.cuda.synchronize()
        assert _lib.cuda().zc_gemm_status_read_and_clear() == 0
        for got, ref in ((y, x.float() @ w.float().t()), (dx, dy.float() @ w.float()), (dw, dy.float().t() @ x.float())):
            tol = 2e-2 * ref.abs().max().item()
            assert (got.float() - ref).abs().max().item() <= tol, (got.float() - ref).abs().max().item()
        acc = y.clone()
        gemm.gemm(x, w, False, True, out=acc, accumulate=True)
        assert torch.allclose(acc.float(), 2 * y.float(), atol=0.1, rtol=2e-2)
    finally:
        gemm.set_backend("auto")


@pytest.mark.parametrize("M,N,K", [(128, 128, 1792), (128, 128, 1856), (128, 128, 1920), (512, 256, 8192), (1024, 1024, 4096), (200, 137, 2056),
                                   (300, 520, 37 * 64), (2048, 1024, 4095), (256, 9472, 2560), (256, 9728, 2560)])
def test_gemm_split_along_k_when_tiles_are_few(M, N, K):
    """The longest K that is not split (1856) and the shortest that is (1920), slices of 8 K blocks, a K that does not divide into equal
    slices, ragged M / N / K, and the last size that is split (37 tiles) beside the first that is not.  Each is rounded once from fp32 sums: half
    a bf16 unit (2^-9) at most per value, so the relative error in the 2-norm is below 2^-9 plus the sums' 1e-5."""
    from fsdp_comm_opt_b200.ops import gemm

    assert (_lib.cuda().zc_gemm_2sm_split_bytes(M, N, K) > 0) == ((M, N, K) not in [(128, 128, 1792), (128, 128, 1856),
                                                                                    (256, 9728, 2560)])
    torch.manual_seed(K)
    pad = (K + 7) // 8 * 8
    x = torch.randn(M, pad, device=DEV).bfloat16()[:, :K]
    w = torch.randn(N, pad, device=DEV).bfloat16()[:, :K]
    bias = torch.randn(N, device=DEV).bfloat16()
    y = gemm.gemm(x, w, False, True, bias=bias)
    dw = gemm.gemm(x, x, True, False) if K <= 4096 else None          # K x K, summed over the M rows
    acc = y.clone() if N % 8 == 0 else None
    if acc is not None:
        gemm.gemm(x, w, False, True, out=acc, accumulate=True)
    torch.cuda.synchronize()
    assert _lib.cuda().zc_gemm_status_read_and_clear() == 0
    ref = x.double() @ w.double().t()
    assert ((y.double() - (ref + bias.double())).norm() / ref.norm()).item() < 2 ** -9 + 1e-5
    if dw is not None:
        rw = x.double().t() @ x.double()
        assert ((dw.double() - rw).norm() / rw.norm()).item() < 2 ** -9 + 1e-5
    if acc is not None:
        assert ((acc.double() - (ref + y.double())).norm() / ref.norm()).item() < 2 ** -8 + 1e-5


@pytest.mark.parametrize("M,N,K", [(128, 128, 128), (129, 136, 136), (300, 1000, 1000), (512, 256, 1024), (256, 129, 2040), (1024, 1024, 4096),
                                   (1536, 1500, 192), (128, 18944, 128), (128, 18945, 128)])
def test_products_of_few_tiles_run_on_one_sm_a_tile(M, N, K):
    """One tile, a row and a few columns more, ragged edges in every direction, K in two, four and eight parts, all SMs busy
    (148 tiles) and one tile more than that.  Rounded once from fp32 sums: 2^-9 and the sums' 1e-5."""
    from fsdp_comm_opt_b200.ops import gemm

    torch.manual_seed(M + N + K)
    mk = lambda r, c: torch.randn(r, (c + 7) // 8 * 8, device=DEV).bfloat16()[:, :c]
    x, w, dy, bias = mk(M, K), mk(N, K), mk(M, N), torch.randn(N, device=DEV).bfloat16()
    ref = x.double() @ w.double().t()
    y = gemm.gemm(x, w, False, True, bias=bias)
    whole = gemm.gemm(x, w, False, True, whole_k=True)
    acc = torch.empty(M, (N + 7) // 8 * 8, device=DEV, dtype=torch.bfloat16)[:, :N].copy_(dy)
    gemm.gemm(x, w, False, True, out=acc, accumulate=True)
    results = [(y, ref + bias.double()), (whole, ref), (acc, ref + dy.double()),
               (gemm.gemm(dy, w, False, False), dy.double() @ w.double()), (gemm.gemm(dy, x, True, False), dy.double().t() @ x.double())]
    torch.cuda.synchronize()
    assert _lib.cuda().zc_gemm_status_read_and_clear() == 0
    for got, want in results:
        assert ((got.double() - want).norm() / want.norm()).item() < 2 ** -9 + 1e-5


@pytest.mark.parametrize("K", [1000, 1024, 2048, 4096])
def test_products_are_cut_into_no_more_clusters_than_run_at_once(K):
    """A cluster lies within a GPC, so fewer fit than CTAs alone: the last number of tiles that is cut into so many parts and the
    first that is not.  Rounded once from fp32 sums: 2^-9 and the sums' 1e-5."""
    from fsdp_comm_opt_b200.ops import gemm

    lib = _lib.cuda()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    fit = {parts: lib.zc_gemm_small_tiles_at_once(parts) for parts in (1, 2, 4, 8)}
    assert fit[1] == sms and all(0 < parts * fit[parts] <= sms for parts in fit) and fit[8] < fit[4] < fit[2]
    chosen = {tiles: lib.zc_gemm_small_best_parts(128, 128 * tiles, K) for tiles in range(1, sms + 2)}
    assert chosen[sms + 1] == 0 and all(chosen[t] >= 1 and t <= fit[chosen[t]] for t in range(1, sms + 1))
    torch.manual_seed(K)
    x = torch.randn(128, K, device=DEV).bfloat16()
    for tiles in sorted({t for parts in (2, 4, 8) for t in (fit[parts], fit[parts] + 1)}):
        w = torch.randn(128 * tiles, K, device=DEV).bfloat16()
        ref = x.double() @ w.double().t()
        assert ((gemm.gemm(x, w, False, True).double() - ref).norm() / ref.norm()).item() < 2 ** -9 + 1e-5
    assert lib.zc_gemm_status_read_and_clear() == 0


def test_products_split_along_k_on_two_streams_have_partial_sums_of_their_own():
    """The tail of the last wave is split (4096 x 6144: 384 tiles on 74 clusters), and so is a product of few tiles; the slices
    are added by a second kernel, which other streams' products may run ahead of."""
    from fsdp_comm_opt_b200.ops import gemm

    torch.manual_seed(5)
    cases = [[(torch.randn(m, k, device=DEV).bfloat16(), torch.randn(n, k, device=DEV).bfloat16()) for _ in range(2)]
             for m, n, k in ((4096, 6144, 1024), (512, 512, 8192))]
    for m, n, k in ((4096, 6144, 1024), (512, 512, 8192)):
        assert _lib.cuda().zc_gemm_2sm_split_bytes(m, n, k) > 0
    for pair in cases:
        alone = [gemm.gemm(x, w, False, True) for x, w in pair]
        torch.cuda.synchronize()
        streams = [torch.cuda.Stream() for _ in pair]
        got = [[], []]
        for _ in range(20):
            for st, (x, w), out in zip(streams, pair, got):
                with torch.cuda.stream(st):
                    out.append(gemm.gemm(x, w, False, True))
        torch.cuda.synchronize()
        for ref, out in zip(alone, got):
            assert all(torch.equal(ref, y) for y in out)


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (1000, 3000, 200), (4096, 6144, 256)])
def test_products_beside_kernels_that_hold_tensor_memory_keep_their_bits(M, N, K):
    """Products of single SMs, of 48 pairs and of all, while other streams' attention and products take and free tensor memory."""
    from fsdp_comm_opt_b200.ops import gemm

    torch.manual_seed(M)
    x, w = torch.randn(M, K, device=DEV).bfloat16(), torch.randn(N, K, device=DEV).bfloat16()
    qkv = torch.randn(2, 700, 12, 64, device=DEV).bfloat16()
    ref = x.double() @ w.double().t()
    alone = gemm.gemm(x, w, False, True)
    other = attention.causal_attention(qkv, 8, 2)
    torch.cuda.synchronize()
    assert ((alone.double() - ref).norm() / ref.norm()).item() < 2 ** -9 + 1e-5
    streams = [torch.cuda.Stream() for _ in range(3)]
    got = [[], [], []]
    for _ in range(30):
        for st, out in zip(streams, got):
            with torch.cuda.stream(st):
                out.append(attention.causal_attention(qkv, 8, 2) if st is streams[0] else gemm.gemm(x, w, False, True))
    torch.cuda.synchronize()
    assert _lib.cuda().zc_gemm_status_read_and_clear() == 0 and attention.status_read_and_clear() == 0
    assert all(torch.equal(other, o) for o in got[0])
    assert all(torch.equal(alone, y) for out in got[1:] for y in out)


@pytest.mark.parametrize("M,N,K", [(1000, 3000, 64), (4096, 5120, 64), (2048, 1600, 4800), (128, 128, 16384), (8192, 8192, 64)])
def test_products_that_end_on_an_arrival_of_the_other_cta_repeat(M, N, K):
    """Pairs of one tile and of many (with the ring of tile numbers and without: a recorded launch), whole tiles, old values and
    slices of K, whose last arrivals at the even CTA are followed by its end; hundreds of launches have no time in between."""
    from fsdp_comm_opt_b200.ops import gemm

    torch.manual_seed(K)
    x, w = torch.randn(M, K, device=DEV).bfloat16(), torch.randn(N, K, device=DEV).bfloat16()
    c = torch.randn(M, N, device=DEV).bfloat16()
    run = lambda out, acc: gemm.gemm(x, w, False, True, out=out, accumulate=acc)
    ref = [run(torch.empty_like(c), False), run(c.clone(), True)]
    out = [torch.empty_like(c), c.clone()]
    for _ in range(100):
        run(out[0], False)
        run(out[1].copy_(c), True)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        recorded = [run(torch.empty_like(c), False), run(c.clone(), True)]
    for _ in range(20):
        graph.replay()
    torch.cuda.synchronize()
    assert _lib.cuda().zc_gemm_status_read_and_clear() == 0
    want = x.double() @ w.double().t()
    for got, whole in zip(ref, (want, want + c.double())):
        assert ((got.double() - whole).norm() / whole.norm()).item() < 2 ** -9 + 1e-5
    for got in (out, recorded):
        assert all(torch.equal(a, b) for a, b in zip(ref, got))


def test_products_behind_kernels_that_fill_shared_memory_report_no_failure():
    """Attention's backward leaves gradients and probabilities all over shared memory, where the products keep their abort flags: a
    flag that is read before it is cleared would end a wait and be reported."""
    from fsdp_comm_opt_b200.ops import gemm

    torch.manual_seed(2)
    qkv = torch.randn(1, 2048, 24, 128, device=DEV).bfloat16().requires_grad_()
    o = attention.causal_attention(qkv, 16, 4)
    cases = [(torch.randn(m, k, device=DEV).bfloat16(), torch.randn(n, k, device=DEV).bfloat16())
             for m, n, k in ((4096, 5120, 64), (512, 256, 1024), (256, 512, 256))]
    ref = [gemm.gemm(x, w, False, True) for x, w in cases]
    for _ in range(20):
        torch.autograd.grad(o, qkv, torch.ones_like(o), retain_graph=True)
        got = [gemm.gemm(x, w, False, True) for x, w in cases]
        assert _lib.cuda().zc_gemm_status_read_and_clear() == 0
        assert all(torch.equal(a, b) for a, b in zip(ref, got))


def _first_products_worker(rank, world):
    from fsdp_comm_opt_b200.ops import gemm

    x, w = torch.randn(4096, 256, device=DEV).bfloat16(), torch.randn(6144, 256, device=DEV).bfloat16()
    ref = x.double() @ w.double().t()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(8)]
    got = []
    for k in range(40):                        # the first of all on a stream that does not wait for the legacy stream
        with torch.cuda.stream(streams[k % 8]):
            got.append(gemm.gemm(x, w, False, True))
    torch.cuda.synchronize()
    assert all(torch.equal(got[0], y) for y in got)
    assert ((got[0].double() - ref).norm() / ref.norm()).item() < 2 ** -9 + 1e-5   # rounded once from fp32 sums


def test_the_first_products_of_a_process_run_on_side_streams():
    """Every stream hands out its tiles (384 on 74 clusters) from counters of its own."""
    from mp_util import run_ranks

    run_ranks(_first_products_worker, 1, init_pg=False, backend="nccl")


def test_gemm_with_leading_dimensions_and_odd_sizes():
    """Operands and results that are slices of wider buffers, and M / N / K that are not multiples of 8
    (GPT-2's vocabulary): the two-SM kernel takes row strides, zero-fills what lies outside a slice and
    hands back a [:, :N] view of aligned rows whose padding columns are zero."""
    from fsdp_comm_opt_b200.ops import gemm

    torch.manual_seed(11)
    M, N, K = 300, 1001, 520
    xb = (torch.randn(M, K + 8, device=DEV) * 0.5).bfloat16()
    x = xb[:, :K - 5]                                # K = 515, rows 528 elements apart
    Ke = K - 5
    w = (torch.randn(N, K, device=DEV) * 0.5).bfloat16()[:, :Ke]
    before = _lib.launch_count()
    y = gemm.gemm(x, w, False, True)                 # [300, 1001] view of [300, 1008]
    assert y.shape == (M, N) and y.stride(0) == 1008
    dx = gemm.gemm(y, w, False, False)               # dgrad form: K = 1001, A strided, B rows = K
    dw = gemm.gemm(y, x, True, False)                # wgrad form: M = 1001 rows out, both operands strided
    assert _lib.launch_count() - before == 3, "the hand-written kernel must have been taken"
    torch.cuda.synchronize()
    assert _lib.cuda().zc_gemm_status_read_and_clear() == 0
    yf = y.float()
    for got, ref in ((y, x.float() @ w.float().t()), (dx, yf @ w.float()), (dw, yf.t() @ x.float())):
        assert got.shape == ref.shape
        tol = 2e-2 * ref.abs().max().item()
        assert (got.float() - ref).abs().max().item() <= tol, (got.float() - ref).abs().max().item()
    pad = torch.as_strided(y, (M, 1008 - N), (1008, 1), y.storage_offset() + N)
    assert int(pad.float().abs().max().item()) == 0
    # a column block of a wider result, accumulated into
    big = torch.zeros(M, 2048, dtype=torch.bfloat16, device=DEV)
    gemm.gemm(x, w, False, True, out=big[:, 1024:1024 + N])
    gemm.gemm(x, w, False, True, out=big[:, 1024:1024 + N], accumulate=True)
    torch.cuda.synchronize()
    assert torch.allclose(big[:, 1024:1024 + N].float(), 2 * yf, atol=0.1, rtol=2e-2)
    assert float(big[:, :1024].float().abs().max()) == 0.0


def test_linear_and_loss_over_a_vocabulary_that_is_not_a_multiple_of_8():
    """lm_head + cross-entropy at an odd vocabulary run on the hand-written GEMM and the strided loss
    kernel; gradients against fp32 PyTorch."""
    from fsdp_comm_opt_b200.ops import gemm

    torch.manual_seed(12)
    T, D, V = 256, 192, 1001
    x = (torch.randn(T, D, device=DEV) * 0.5).bfloat16().requires_grad_()
    w = (torch.randn(V, D, device=DEV) * 0.1).bfloat16().requires_grad_()
    labels = torch.randint(0, V, (T,), device=DEV)
    labels[7] = -100
    before = _lib.launch_count()
    out = loss.cross_entropy(gemm.linear(x, w), labels)
    out.backward()
    torch.cuda.synchronize()
    assert _lib.launch_count() - before >= 4        # three GEMMs and the loss kernel
    xf, wf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    ref = F.cross_entropy((xf @ wf.t()).bfloat16().float(), labels, ignore_index=-100)
    ref2 = F.cross_entropy(xf @ wf.t(), labels, ignore_index=-100)
    ref2.backward()
    assert abs(out.item() - ref.item()) < 5e-3
    assert torch.allclose(x.grad.float(), xf.grad, atol=2e-2 * float(xf.grad.abs().max()), rtol=5e-2)
    assert torch.allclose(w.grad.float(), wf.grad, atol=2e-2 * float(wf.grad.abs().max()), rtol=5e-2)


def test_linear_autograd_on_tcgen05_matches_cublas():
    from fsdp_comm_opt_b200.ops import gemm

    torch.manual_seed(10)
    x = (torch.randn(2, 256, 512, device=DEV) * 0.5).bfloat16().requires_grad_()
    w = (torch.randn(768, 512, device=DEV) * 0.05).bfloat16().requires_grad_()
    g = torch.randn(2, 256, 768, device=DEV).bfloat16()
    gemm.set_backend("tcgen05")
    gemm.linear(x, w).backward(g)
    gx, gw = x.grad.clone(), w.grad.clone()
    x.grad = w.grad = None
    gemm.set_backend("cublas")
    gemm.linear(x, w).backward(g)
    gemm.set_backend("auto")
    assert torch.allclose(gx.float(), x.grad.float(), atol=3e-2, rtol=3e-2)
    assert torch.allclose(gw.float(), w.grad.float(), atol=0.3, rtol=3e-2)


# ------------------------------------------------------------------ whole models on the GPU
@pytest.mark.parametrize("shape", ["tiny", "gpt2-tiny"])
def test_model_forward_backward_matches_cpu(shape):
    """One forward + backward of a tiny model of each family on the GPU kernels against the same
    weights and tokens on the CPU reference paths of the ops."""
    from fsdp_comm_opt_b200.models import build_model, get_config

    cfg = get_config(shape)
    torch.manual_seed(3)
    ref = build_model(cfg).to(torch.bfloat16)
    ref.init_weights()
    gpu = build_model(cfg).to(torch.bfloat16)
    gpu.load_state_dict(ref.state_dict())
    gpu = gpu.to(DEV)
    ids = torch.randint(0, cfg.vocab_size, (2, 128))
    out_r = ref(input_ids=ids, labels=ids)
    out_r.loss.backward()
    out_g = gpu(input_ids=ids.to(DEV), labels=ids.to(DEV))
    out_g.loss.backward()
    torch.cuda.synchronize()
    assert abs(out_g.loss.item() - out_r.loss.item()) < 5e-2, (out_g.loss.item(), out_r.loss.item())
    checked = 0
    for (n, pr), (_, pg) in zip(ref.named_parameters(), gpu.named_parameters()):
        assert pg.grad is not None, n
        gr, gg = pr.grad.float(), pg.grad.float().cpu()
        assert torch.isfinite(gg).all(), n
        denom = gr.abs().max().item() + 1e-6
        assert (gg - gr).abs().max().item() / denom < 0.15, (n, (gg - gr).abs().max().item(), denom)
        checked += 1
    assert checked > 5


def test_device_status_check_is_clean_after_kernels():
    """The host-side health check reads every kernel family's status word; after normal launches it
    must find nothing (a wait that ran out would raise here instead of hanging the GPU)."""
    from fsdp_comm_opt_b200.utils.health import check_device_status

    qkv = (torch.randn(1, 256, 6, 128, device=DEV) * 0.5).bfloat16().requires_grad_()
    attention.causal_attention(qkv, 4, 1).sum().backward()
    torch.cuda.synchronize()
    check_device_status()


def test_adamw_is_skipped_while_the_health_word_is_set():
    """A step that follows a collective which gave up must not be applied: the guarded AdamW launch
    reads the library's health word on the device and leaves parameters and moments alone."""
    from fsdp_comm_opt_b200.ops.adamw import FusedAdamW

    lib = _lib.cuda()
    p = torch.nn.Parameter(torch.randn(1 << 16, device=DEV).bfloat16())
    p.grad = torch.randn_like(p)
    opt = FusedAdamW([p], lr=1e-2)
    before = p.detach().clone()
    assert lib.zc_health_set(2) == 0          # what an expired wait writes
    opt.step()
    torch.cuda.synchronize()
    assert torch.equal(p.detach(), before)
    assert float(opt.state[p]["exp_avg"].float().abs().sum()) == 0.0
    assert lib.zc_health_read_and_clear() == 2
    opt.step()
    torch.cuda.synchronize()
    assert not torch.equal(p.detach(), before)
    assert lib.zc_health_read_and_clear() == 0


def test_adamw_in_two_launches_equals_one():
    """``step(split_at=..., between=...)`` updates a prefix first, calls back, then updates the rest:
    same result as one launch (every element is independent)."""
    from fsdp_comm_opt_b200.ops.adamw import FusedAdamW

    torch.manual_seed(4)
    w = torch.randn(100_000, device=DEV).bfloat16()
    g = torch.randn_like(w)
    a, b = torch.nn.Parameter(w.clone()), torch.nn.Parameter(w.clone())
    a.grad, b.grad = g.clone(), g.clone()
    oa, ob = FusedAdamW([a], lr=1e-2), FusedAdamW([b], lr=1e-2)
    called = []
    for _ in range(3):
        oa.step()
        ob.step(split_at=33_333, between=lambda: called.append(1))
    torch.cuda.synchronize()
    assert len(called) == 3 and ob.kernel_launches == 6 and oa.kernel_launches == 3
    assert torch.equal(a.detach(), b.detach())
    assert torch.equal(oa.state[a]["exp_avg_sq"], ob.state[b]["exp_avg_sq"])


@pytest.mark.parametrize("N,K,M,slab_rows,ring", [(1024, 512, 256, 256, 3), (2048, 1024, 384, 512, 2), (512, 256, 128, 512, 2)])
def test_gemm_from_codec_records_matches_fp32_matmul(N, K, M, slab_rows, ring):
    """Decode fused with the consumer GEMM: the weight is given as v2 records, decoded slab by slab
    into an L2-resident ring beside the GEMM; same bits as decode-then-GEMM, close to fp32 matmul."""
    from fsdp_comm_opt_b200.ops.gemm_records import RecordLinear, linear_t_plain
    g = torch.Generator().manual_seed(N + K)
    w = (torch.randn(N, K, generator=g) * 0.02).bfloat16().cuda()
    w[::7, ::5] = 300.0                                   # escapes in most chunks
    x = torch.randn(M, K, generator=g).bfloat16().cuda()
    rec, hdr = codec.v2_encode(w.view(-1))
    rl = RecordLinear(N, K, "cuda", slab_rows=slab_rows, ring=ring)
    y1 = rl(x, rec, hdr).clone()
    y2 = rl(x, rec, hdr)                                  # second call runs over the first call's ring
    plain = linear_t_plain(x, rec, hdr, N, K)
    torch.cuda.synchronize()
    ref = w.float() @ x.float().t()
    assert torch.equal(y1, y2) and torch.equal(y1, plain)
    assert torch.allclose(y1.float(), ref, rtol=2e-2, atol=2e-2 * float(ref.abs().max()))


@pytest.mark.parametrize("heads,kv,D", [(4, 2, 128), (8, 2, 64)])
def test_recorded_launches_have_the_bits_of_launches_one_after_the_other(heads, kv, D):
    """Recorded kernels come up while the one before them still writes what they read.  Every kind of them behind another, behind a
    copy, behind a library kernel and on a branch that joins again, forward and backward, with other inputs at every replay:
    a value of the replay before would differ.  (Two key blocks: dQ has the same bits in either order.)"""
    from fsdp_comm_opt_b200.ops import embedding, gemm

    B, S, C, F_, V = 2, 256, 512, 1024, 1000
    T = B * S
    torch.manual_seed(D)
    mk = lambda *shape: (torch.randn(*shape, device=DEV) * shape[-1] ** -0.5).bfloat16().requires_grad_()
    table, w_qkv, w_o, w_gu, w_down, w_up, w_back, w_head = (
        mk(64, C), mk((heads + 2 * kv) * D, C), mk(C, heads * D), mk(2 * F_, C), mk(C, F_), mk(F_, C), mk(C, F_), mk(V, C))
    n1, n2, n3, nb, b_up, b_back = (torch.randn(n, device=DEV).bfloat16().requires_grad_() for n in (C, C, C, C, F_, C))
    weights = [w_qkv, w_o, w_gu, w_down, w_up, w_back, w_head, n1, n2, n3, nb, b_up, b_back]
    table.main_grad = torch.zeros_like(table)
    cos, sin = rope.rope_tables(S, D, 10000.0, torch.device(DEV, 0))
    side = torch.cuda.Stream()

    def step(ids, labels, extra, moments):
        table.main_grad_written = False
        x = embedding.embedding(ids, table) + extra
        q = gemm.linear(norm.rms_norm(x, n1), w_qkv).view(T, -1)
        q = rope.apply_rope(q, cos, sin, heads + kv, D, S) if D == 64 else q
        a = gemm.linear(attention.causal_attention(q.view(B, S, heads + 2 * kv, D), heads, kv).reshape(T, heads * D), w_o)
        y, h = norm.add_rms_norm(a, x.reshape(T, C), n2, 1e-5)
        m = gemm.linear(swiglu.swiglu(gemm.linear(y, w_gu)), w_down)
        z, h2 = gpt2_ops.add_layer_norm(m, h, n3, nb)
        g = gemm.linear(gpt2_ops.bias_gelu(gemm.linear(z, w_up), b_up), w_back, b_back) + h2
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        with torch.cuda.stream(side):
            branch = gemm.gemm(z.detach(), w_up.detach(), False, True)
        value = loss.cross_entropy(gemm.linear(g, w_head), labels)
        grads = torch.autograd.grad(value, weights + [table], allow_unused=True)[:-1]
        main.wait_stream(side)
        p, mean, sq = (t.clone() for t in moments)
        grad = grads[2].clone()
        _lib.check(_lib.cuda().zc_adamw(p.data_ptr(), grad.data_ptr(), mean.data_ptr(), sq.data_ptr(), p.numel(), 0, 0, 0, 1e-3, 0.9, 0.95,
                                        1e-8, 0.01, 0.1, 0.05, 0, _lib.stream_ptr(p.device)), "zc_adamw")
        return [value, branch, table.main_grad.clone(), p, mean, sq, *grads]

    def inputs(k):
        g = torch.Generator(DEV).manual_seed(k)
        return [torch.randint(0, 64, (B, S), device=DEV, generator=g), torch.randint(0, V, (T,), device=DEV, generator=g),
                torch.randn(B, S, C, device=DEV, generator=g).bfloat16(),
                [torch.rand(2 * F_, C, device=DEV, generator=g).bfloat16() for _ in range(3)]]

    def put(k):
        for a, b in zip(fixed[:3] + fixed[3], (lambda i: i[:3] + i[3])(inputs(k))):
            a.copy_(b)

    stream = torch.cuda.Stream()  # of all steps, recorded or not
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        fixed = inputs(0)
        want = [[t.detach() for t in step(*inputs(k))] for k in range(12)]
        again = [[t.detach() for t in step(*inputs(k))] for k in range(12)]
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for x, y in zip(want, again) for a, b in zip(x, y))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            ids, labels, extra = (t.clone() for t in fixed[:3])
            recorded = [t.detach() for t in step(ids, labels, extra, fixed[3])]
        for k in [*range(12), *range(12)]:
            put(k)
            graph.replay()
            assert all(torch.equal(a, b) for a, b in zip(want[k], recorded)), k
    assert _lib.cuda().zc_gemm_status_read_and_clear() == 0 and attention.status_read_and_clear() == 0


@pytest.mark.parametrize("N,K,M,slab_rows", [(4096, 1000, 520, 256), (2048, 1024, 2048, 128)])
def test_slabs_and_whole_products_of_different_kernels_have_the_same_bits(N, K, M, slab_rows):
    """A slab's few tiles run on one SM each, the whole product on pairs of SMs; both are one sum along K."""
    from fsdp_comm_opt_b200.ops import gemm_records

    lib = _lib.cuda()
    assert gemm_records._whole_k(N, M, K, 0) and gemm_records._whole_k(slab_rows, M, K, 0)
    assert lib.zc_gemm_small_best_parts(slab_rows, M, K) > 0 and lib.zc_gemm_small_best_parts(N, M, K) == 0
    g = torch.Generator().manual_seed(N)
    w, x = (torch.randn(n, K, generator=g).bfloat16().cuda() for n in (N, M))
    rec, hdr = codec.v2_encode(w.view(-1))
    slabs = gemm_records.RecordLinear(N, K, "cuda", slab_rows=slab_rows, ring=3)(x, rec, hdr)
    plain = gemm_records.linear_t_plain(x, rec, hdr, N, K)
    ref = w.double() @ x.double().t()
    assert torch.equal(slabs, plain)
    assert ((plain.double() - ref).norm() / ref.norm()).item() < 2 ** -9 + 1e-5


@pytest.mark.parametrize("N,K,M", [(4096, 4096, 128), (6144, 4096, 4096)])
def test_products_from_records_are_cut_along_k_where_other_products_are(N, K, M):
    """Few tiles, and a last wave of ten: the product of a decoded weight is the same launch as any other's."""
    from fsdp_comm_opt_b200.ops import gemm, gemm_records

    g = torch.Generator().manual_seed(M)
    w, x = (torch.randn(n, K, generator=g).bfloat16().cuda() for n in (N, M))
    rec, hdr = codec.v2_encode(w.view(-1))
    cut, whole = gemm.gemm(w, x, False, True), gemm.gemm(w, x, False, True, whole_k=True)
    assert not torch.equal(cut, whole)          # fp32 sums of other parts
    assert torch.equal(gemm_records.linear_t_plain(x, rec, hdr, N, K), cut)


@pytest.mark.parametrize("M,N,K", [(128, 128, 16384), (200, 137, 16390), (384, 512, 16384), (256, 2304, 4096), (256, 2290, 4090), (256, 9472, 3328),
                                   (2048, 1024, 4095)])
def test_products_whose_slices_of_k_a_second_kernel_adds(M, N, K):
    """Sixteen slices, a last slice of two K blocks, slices of eight, ragged edges, 37 tiles in two: sizes that still take the two-SM
    kernel and its workspace, alone and on two streams at once.  Rounded once from fp32 sums: 2^-9 and the sums' 1e-5."""
    from fsdp_comm_opt_b200.ops import gemm

    lib = _lib.cuda()
    assert lib.zc_gemm_ws_bytes(M, N, K) == lib.zc_gemm_2sm_split_bytes(M, N, K) > 0
    torch.manual_seed(K)
    mk = lambda r, c: torch.randn(r, (c + 7) // 8 * 8, device=DEV).bfloat16()[:, :c]
    pairs, old = [(mk(M, K), mk(N, K)) for _ in range(2)], mk(M, N)
    bias = torch.randn(N, device=DEV).bfloat16()
    alone = []
    for x, w in pairs:
        ref = x.double() @ w.double().t()
        acc = torch.empty(M, (N + 7) // 8 * 8, device=DEV, dtype=torch.bfloat16)[:, :N].copy_(old)
        alone.append(gemm.gemm(x, w, False, True))
        gemm.gemm(x, w, False, True, out=acc, accumulate=True)
        for got, want in ((alone[-1], ref), (gemm.gemm(x, w, False, True, bias=bias), ref + bias.double()), (acc, ref + old.double())):
            assert ((got.double() - want).norm() / want.norm()).item() < 2 ** -9 + 1e-5
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream() for _ in pairs], [[], []]
    for _ in range(20):
        for st, (x, w), out in zip(streams, pairs, got):
            with torch.cuda.stream(st):
                out.append(gemm.gemm(x, w, False, True))
    torch.cuda.synchronize()
    assert lib.zc_gemm_status_read_and_clear() == 0
    assert all(torch.equal(ref, y) for ref, out in zip(alone, got) for y in out)


@pytest.mark.parametrize("M,N,K,parts", [(129, 136, 136, 1), (300, 1001, 200, 1), (769, 650, 2040, 2), (129, 137, 900, 4), (130, 250, 2040, 8),
                                         (1100, 4301, 200, 0), (200, 137, 16390, 0), (4000, 6100, 1030, 0)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_products_into_a_part_of_a_buffer_leave_the_rest_alone(M, N, K, parts, accumulate):
    """Every element of a result in a buffer with longer rows and more of them, both kernels, K in one and in several parts.  An
    element is rounded once, by 2^-8 of itself at most, from a sum of K products, whose fp32 errors are below K 2^-22 of the sum of
    their sizes.  The columns up to the next multiple of eight are zeros (or what they were, when added to); all else is untouched."""
    from fsdp_comm_opt_b200.ops import gemm

    lib = _lib.cuda()
    if parts:
        assert lib.zc_gemm_small_best_parts(M, N, K) == parts and lib.zc_gemm_ws_bytes(M, N, K) == 0
    else:
        assert lib.zc_gemm_small_best_parts(M, N, K) == 0 or lib.zc_gemm_ws_bytes(M, N, K) > 0
    torch.manual_seed(M + K)
    pad = (N + 7) // 8 * 8
    mk = lambda r, c: torch.randn(r, (c + 7) // 8 * 8, device=DEV).bfloat16()[:, :c]
    x, w, bias = mk(M, K), mk(N, K), torch.randn(N, device=DEV).bfloat16()
    ref, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    for b in (None, bias):
        buf = torch.randn(M + 9, pad + 24, device=DEV).bfloat16()
        before = buf.clone()
        gemm.gemm(x, w, False, True, out=buf[4:4 + M, 8:8 + N], accumulate=accumulate, bias=b)
        torch.cuda.synchronize()
        assert lib.zc_gemm_status_read_and_clear() == 0
        want = ref + (before[4:4 + M, 8:8 + N].double() if accumulate else 0) + (b.double() if b is not None else 0)
        bound = want.abs() * 2 ** -8 + (size + want.abs() + 8) * K * 2 ** -22
        assert ((buf[4:4 + M, 8:8 + N].double() - want).abs() <= bound).all()
        padding = buf[4:4 + M, 8 + N:8 + pad]
        assert torch.equal(padding, before[4:4 + M, 8 + N:8 + pad]) if accumulate else not padding.any()
        buf[4:4 + M, 8:8 + pad] = before[4:4 + M, 8:8 + pad]
        assert torch.equal(buf, before)
