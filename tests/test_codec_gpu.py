"""sm_100a codec kernels against the plain PyTorch fp32 oracle (coccl_b200.ops.codec.reference_roundtrip)."""
import pytest
import torch

from coccl_b200 import _lib
from coccl_b200.ops import codec as C

pytestmark = pytest.mark.gpu

CFGS = [
    C.CodecConfig("sdp4bit", 4, 128, False, True),
    C.CodecConfig("sdp4bit", 4, 128, False, False),
    C.CodecConfig("sdp4bit", 8, 2048, False, False),
    C.CodecConfig("sdp4bit", 8, 512, False, True),
    C.CodecConfig("sdp4bit", 4, 64, True, False),
    C.CodecConfig("sdp4bit", 8, 128, True, True),
    C.CodecConfig("sdp4bit", 4, 32, False, True),
    C.MXFP8,
]


def _step(x, cfg):
    """Largest quantisation step of any group (bound on a single rounding flip)."""
    if cfg.kind == "mxfp8":
        return x.abs().max().item() / 8.0
    levels = (1 << (cfg.bits - 1)) - 1
    amax = x.abs().max().item() * (32 ** 0.5 * 4 if cfg.hadamard else 1.0)
    return 2.0 * amax / levels


@pytest.mark.parametrize("cfg", CFGS, ids=lambda c: f"{c.kind}{c.bits}g{c.group}{'a' if c.asym else 's'}{'h' if c.hadamard else ''}")
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("count,chunks", [(4096, 4), (1000, 3), (2048 * 5 + 136, 1), (8192 * 3 + 40, 2), (16384, 2)])
def test_roundtrip_matches_oracle(cuda, cfg, dtype, count, chunks):
    torch.manual_seed(0)
    x = (torch.randn(chunks * count, device=cuda) * 0.01).to(dtype)
    enc = C.encode(x, cfg, chunks)
    assert enc.shape == (chunks, cfg.encoded_chunk_bytes(count, dtype))
    y = C.decode(enc, cfg, count, dtype, chunks).reshape(-1).float()
    ref = C.reference_roundtrip(x, cfg, chunks).reshape(-1).to(dtype).float()
    diff = (y - ref).abs()
    # identical arithmetic up to fma contraction: almost every element matches to rounding of the
    # output type; a flipped rounding decision moves an element by at most one step
    tol = 1e-6 + 2e-3 * ref.abs().max().item()
    frac_bad = (diff > tol).float().mean().item()
    assert frac_bad < 2e-3, f"{frac_bad=} max={diff.max().item()}"
    assert diff.max().item() <= _step(x.float(), cfg) + tol


def test_encoded_sizes_match_reference_contract():
    # 1024 elements in 4 chunks, g128 q4: 544 B fp32, 576 B for 16-bit inputs
    cfg = C.CodecConfig("sdp4bit", 4, 128, False, True)
    assert 4 * cfg.encoded_chunk_bytes(256, torch.float32) == 544
    assert 4 * cfg.encoded_chunk_bytes(256, torch.bfloat16) == 576
    assert 4 * cfg.encoded_chunk_bytes(256, torch.float16) == 576


@pytest.mark.parametrize("cfg", [CFGS[0], CFGS[1], CFGS[2], CFGS[7]], ids=["q4h", "q4", "q8g2048", "mxfp8"])
def test_decode_reduce_and_drc(cuda, cfg):
    torch.manual_seed(1)
    n, count, chunks = 8, 5000, 2
    xs = [torch.randn(chunks * count, device=cuda) * 0.01 for _ in range(n)]
    enc = torch.cat([C.encode(x, cfg, chunks) for x in xs], dim=0)  # [n*chunks, B], copy i chunk j at i*chunks+j
    red = C.decode_reduce(enc, cfg, count, torch.float32, chunks, n).reshape(-1)
    ref = sum(C.reference_roundtrip(x, cfg, chunks).reshape(-1) for x in xs)
    assert torch.allclose(red, ref, atol=n * _step(xs[0], cfg) * 2e-3 + 1e-5, rtol=1e-4) or \
        ((red - ref).abs() > 1e-4).float().mean().item() < 2e-3
    # fused decode-reduce-encode == decode-reduce followed by encode without rotation; compare after decode
    drc = C.decode_reduce_encode(enc, cfg, count, torch.float32, chunks, n)
    back = C.decode(drc, cfg, count, torch.float32, chunks).reshape(-1)
    err = (back - ref).abs().max().item()
    bound = _step(ref, cfg)
    assert err <= bound, (err, bound)


def test_stochastic_rounding_is_unbiased_and_reproducible(cuda):
    cfg = C.CodecConfig("sdp4bit", 4, 128, False, False, True, seed=123)
    x = torch.full((1 << 20,), 0.3, device=cuda)
    x[::128] = 1.0  # absmax 1 -> scale 7, 0.3*7 = 2.1 -> rounds to 2 (p=.9) or 3 (p=.1)
    a = C.decode(C.encode(x, cfg), cfg, x.numel(), torch.float32).reshape(-1)
    b = C.decode(C.encode(x, cfg), cfg, x.numel(), torch.float32).reshape(-1)
    assert torch.equal(a, b)
    mask = torch.ones_like(x, dtype=torch.bool)
    mask[::128] = False
    assert abs(a[mask].mean().item() - 0.3) < 2e-3
    ref = C.reference_roundtrip(x, cfg)
    assert ((a - ref).abs() > 1e-6).float().mean().item() < 1e-3


@pytest.mark.parametrize("rate", [4, 8, 16])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("count,chunks", [(4096, 2), (1002, 3), (8192 * 2 + 36, 1)])
def test_zfp_tile_codec_is_bit_identical_to_the_cpu_coder(cuda, rate, dtype, count, chunks):
    """The tile codec writes the same stream as the CPU coder of csrc/oracle (block i at bit i * 4 * rate), and
    decodes to the same values; sums of several encoded copies equal the sum of the oracle's decodes."""
    import ctypes as CT
    from coccl_b200 import _lib
    cfg = C.CodecConfig("zfp", rate, 4, False, False)
    torch.manual_seed(11)
    x = (torch.randn(chunks * count, device=cuda) * 0.01).to(dtype)
    enc = C.encode(x, cfg, chunks)
    en = _lib.declare("cocclOracleZfpEncode", CT.c_int, [CT.c_void_p, CT.c_long, CT.c_int, CT.c_void_p])
    cb = _lib.declare("cocclOracleZfpChunkBytes", CT.c_long, [CT.c_long, CT.c_int])
    xc = x.float().cpu().reshape(chunks, count).contiguous()
    want = torch.zeros(cb(count, rate), dtype=torch.uint8)
    for ch in range(chunks):
        want.zero_()
        assert en(xc[ch].data_ptr(), count, rate, want.data_ptr()) == 0
        got = enc[ch].cpu()
        nbytes = (-(-count // 4) * 4 * rate + 7) // 8       # bits of the whole blocks, in bytes
        assert torch.equal(got[:nbytes], want[:nbytes]), (ch, (got[:nbytes] != want[:nbytes]).nonzero()[:4])
    ref = C.reference_roundtrip(x, cfg, chunks)
    y = C.decode(enc, cfg, count, dtype, chunks).reshape(-1)
    if dtype == torch.float32:
        assert torch.equal(y.cpu(), ref.cpu())
    else:
        assert ((y.float().cpu() - ref.cpu()).abs() <= ref.cpu().abs() * 2.0 ** -7 + 1e-12).all()
    if chunks > 1 and dtype == torch.float32:
        s = C.decode_reduce(enc, cfg, count, dtype, 1, chunks).reshape(-1)
        assert torch.allclose(s.cpu(), ref.cpu().reshape(chunks, count).sum(0), atol=1e-6)


@pytest.mark.parametrize("group", [32, 128, 512])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("count,chunks", [(4096, 2), (1000, 3), (8192 * 2 + 200, 1)])
def test_taco_tile_codec_matches_oracle(cuda, group, dtype, count, chunks):
    cfg = C.CodecConfig("taco", 8, group, False, False)
    torch.manual_seed(12)
    x = (torch.randn(chunks * count, device=cuda) * 0.05).to(dtype)
    enc = C.encode(x, cfg, chunks)
    assert enc.shape[1] == -(-count // group) * (group + 8)
    y = C.decode(enc, cfg, count, dtype, chunks).reshape(-1).float()
    ref = C.reference_roundtrip(x, cfg, chunks).reshape(-1).to(dtype).float()
    scale = ref.abs().max().item()
    assert ((y - ref).abs() > 2e-2 * scale).float().mean().item() < 5e-3   # a flipped FP8 rounding is spread over the group
    assert ((y - x.float()).norm() / x.float().norm()).item() < 0.05
    if chunks > 1:
        # copies with different adaptive scales add up in the rotated domain; one inverse transform serves the sum
        s = C.decode_reduce(enc, cfg, count, dtype, 1, chunks).reshape(-1).float()
        want = C.reference_roundtrip(x, cfg, chunks).reshape(chunks, count).sum(0)
        assert ((s - want).norm() / want.norm()).item() < 0.02
        drc = C.decode_reduce_encode(enc, cfg, count, dtype, 1, chunks)
        s2 = C.decode(drc, cfg, count, dtype, 1).reshape(-1).float()
        assert ((s2 - want).norm() / want.norm()).item() < 0.06


@pytest.mark.parametrize("cfg", [C.SDP4BIT_G128, C.MXFP8, C.TACO_G128, C.ZFP_RATE8], ids=lambda c: c.kind)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("count", [1, 5, 31, 1023, 1025, 3 * 1024 - 1, 8191, 8193, 2 * 8192 + 1031])
def test_misaligned_and_ragged_chunks_equal_aligned_ones(cuda, cfg, dtype, count):
    """Chunks that start at every distance from a 16-byte boundary (the start of the tensor shifted too) and end anywhere in a
    tile, a warp's window or a vector: the same bytes, and the same values back, as each chunk on its own in an aligned
    buffer. The chunks lie back to back, so a write outside one shows in its neighbour."""
    torch.manual_seed(count)
    chunks = 5
    for shift in (0, 1, 3):
        whole = (torch.randn(chunks * count + 8, device=cuda) * 0.01).to(dtype)
        x = whole[shift:shift + chunks * count]
        enc = C.encode(x, cfg, chunks)
        dec = C.decode(enc, cfg, count, dtype, chunks)
        for j in range(chunks):
            one = C.encode(x[j * count:(j + 1) * count].clone(), cfg, 1)
            assert torch.equal(enc[j], one[0]), (shift, j)
            assert torch.equal(dec[j], C.decode(one, cfg, count, dtype, 1)[0]), (shift, j)


@pytest.mark.parametrize("magnitude", [1e-30, 3e-33, 1e-36])
def test_sdp4bit_tiny_groups_decode_like_the_oracle(cuda, magnitude):
    """Groups whose scaled parameter would leave the normal range take the shifting decoder; next to ordinary groups."""
    torch.manual_seed(1)
    x = torch.randn(4, 128, device=cuda)
    x[1:3] *= magnitude
    cfg = C.CodecConfig("sdp4bit", 4, 128, False, False)
    y = C.decode(C.encode(x.reshape(-1), cfg, 1), cfg, 512, torch.float32, 1).reshape(4, 128)
    ref = C.reference_roundtrip(x.reshape(-1), cfg, 1).reshape(4, 128)
    step = x.abs().amax(1, keepdim=True) / 7
    assert ((y - ref).abs() <= 1e-4 * step + 1e-44).float().mean() > 0.99   # a flipped tie moves a value by one step
    assert ((y - ref).abs() <= 1.001 * step + 1e-44).all()


@pytest.mark.parametrize("groups", [1, 2, 3, 4, 7])
def test_mxfp8_chunk_padding_is_zero(cuda, groups):
    """The scale bytes of a chunk end anywhere in a word; the rest of the word is part of the stream and is written."""
    n = C.MXFP8.encoded_chunk_bytes(32 * groups, torch.bfloat16)
    x = torch.randn(64 * groups, device=cuda).to(torch.bfloat16)
    enc = torch.full((2, n), 255, dtype=torch.uint8, device=cuda)   # memory that held something else
    _lib.check(_lib.lib().cocclkEncode(x.data_ptr(), enc.data_ptr(), 32 * groups, 2, 32 * groups, n, C.DTYPE_CODE[x.dtype],
                                       C.MXFP8.to_c(x.dtype), _lib.cur_stream()), "cocclkEncode")
    assert torch.equal(enc, C.encode(x, C.MXFP8, 2))
    assert (enc[:, 33 * groups:] == 0).all()


@pytest.mark.parametrize("tiles", [1, 296, 297, 445, 593])
@pytest.mark.parametrize("cfg", [C.SDP4BIT_G128, C.CodecConfig("sdp4bit", 4, 8, False, False), C.CodecConfig("sdp4bit", 4, 16, True, False),
                                 C.CodecConfig("sdp4bit", 8, 8, True, False), C.CodecConfig("sdp4bit", 8, 512, False, True), C.MXFP8,
                                 C.TACO_G128, C.ZFP_RATE8, C.CodecConfig("zfp", 16, 4, False, False)],
                         ids=lambda c: f"{c.kind}{c.bits}g{c.group}{'a' if c.asym else 's'}")
def test_sums_on_both_sides_of_the_rounds_of_tiles(cuda, cfg, tiles):
    """One copy and the sum of three, with as many tiles as one more or less than the GPU's places for either kernel, the last
    tile ragged. The sum is formed in fp32 before the way out of the rotated domain: a few fp32 steps of the values' sizes."""
    torch.manual_seed(tiles)
    count = tiles * 8192 - 24
    x = torch.randn(3 * count, device=cuda)
    enc = C.encode(x, cfg, 3)
    one = C.decode(enc, cfg, count, torch.float32, 3).double()
    got = C.decode_reduce(enc, cfg, count, torch.float32, 1, 3)[0].double()
    size = one.abs().sum(0).amax()
    assert ((got - one.sum(0)).abs() <= 64 * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("offset", [0, 4, 8])
@pytest.mark.parametrize("cfg,dtype", [(C.SDP4BIT_G128, torch.float32), (C.SDP4BIT_G128, torch.bfloat16),
                                       (C.CodecConfig("sdp4bit", 4, 32, True, False), torch.float16),
                                       (C.CodecConfig("sdp4bit", 8, 128, False, True), torch.bfloat16),
                                       (C.CodecConfig("sdp4bit", 8, 64, True, True), torch.float32), (C.MXFP8, torch.bfloat16),
                                       (C.TACO_G128, torch.float32), (C.CodecConfig("taco", 8, 64, False, False), torch.float16),
                                       (C.CodecConfig("taco", 8, 32, False, False), torch.float32),
                                       (C.CodecConfig("taco", 8, 512, False, False, e5m2=True), torch.float32)],
                         ids=lambda v: f"{v.kind}{v.bits}g{v.group}{'a' if v.asym else 's'}" if isinstance(v, C.CodecConfig) else str(v)[6:])
@pytest.mark.parametrize("groups", [1, 3, 66])
def test_sums_at_every_alignment_and_number_of_copies(cuda, cfg, dtype, groups, offset):
    """Encoded copies that start on any word (the distance between them a multiple of 4, 8 or 16 bytes by the number of
    groups), 1 to 9 of them: the sum of what each decodes to on its own, to the rounding of fp32 sums (and of the output)."""
    torch.manual_seed(groups)
    count = groups * cfg.group - 5
    x = (torch.randn(9 * count, device=cuda)).to(dtype)
    enc = C.encode(x, cfg, 9)
    nb = enc.shape[1]
    room = torch.empty(9 * nb + 16, dtype=torch.uint8, device=cuda)
    room[offset:offset + 9 * nb] = enc.reshape(-1)
    one = C.decode(enc, cfg, count, torch.float32, 9) if cfg.param_bytes(dtype) == cfg.param_bytes(torch.float32) else None
    for n in range(1, 10):
        got = torch.full((count,), float("nan"), dtype=dtype, device=cuda)
        _lib.check(_lib.lib().cocclkDecodeReduce(room.data_ptr() + offset, got.data_ptr(), count, 1, n, count, nb, C.DTYPE_CODE[dtype],
                                                 cfg.to_c(dtype), _lib.cur_stream()), "cocclkDecodeReduce")
        each = [C.decode(enc[i:i + 1].clone(), cfg, count, dtype, 1)[0].double() for i in range(n)]
        want, size = sum(each), sum(e.abs() for e in each).amax()
        # fp32 roundings of the way out of the rotated domain, on values up to sqrt(group) larger than the results
        ulp = max(torch.finfo(dtype).eps, (cfg.group ** 0.5 * 16 * 2.0 ** -23 if cfg.kind == "taco" else 0.0))
        assert ((got.double() - want).abs() <= (n + 1) * max(ulp, 64 * 2.0 ** -24) * size).all()
        if one is not None:
            assert ((got.double() - one[:n].double().sum(0)).abs() <= max(ulp, 64 * 2.0 ** -24) * size).all()


@pytest.mark.parametrize("cfg", [C.SDP4BIT_G128, C.CodecConfig("sdp4bit", 4, 128, False, True, True), C.CodecConfig("sdp4bit", 4, 16, False, False),
                                 C.MXFP8, C.TACO_G128, C.ZFP_RATE8], ids=lambda c: f"{c.kind}g{c.group}{'r' if c.stochastic else ''}")
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("count", [8192 * 7 + 3, 8192 * 7, 41])
def test_several_tiles_a_cta_equal_one(cuda, cfg, dtype, count):
    """More tiles than the GPU has places, so that a CTA's tiles follow one another through its stages and over the ends of chunks
    (chunks of one tile: the walk steps over many chunks at once): the same bytes and values as a chunk on its own."""
    torch.manual_seed(2)
    chunks = 1900 if count < 8192 else 240
    x = (torch.randn(chunks * count, device=cuda) * 0.01).to(dtype)
    enc = C.encode(x, cfg, chunks)
    dec = C.decode(enc, cfg, count, dtype, chunks)
    for j in (0, 1, 83, 84, chunks // 2, chunks - 2, chunks - 1):
        if cfg.stochastic and j:
            continue   # the rounding stream is keyed by the chunk
        one = C.encode(x[j * count:(j + 1) * count].clone(), cfg, 1)
        assert torch.equal(enc[j], one[0]), j
    for j in (0, 1, 83, 84, chunks // 2, chunks - 2, chunks - 1):
        assert torch.equal(dec[j], C.decode(enc[j:j + 1].clone(), cfg, count, dtype, 1)[0]), j


@pytest.mark.parametrize("asym", [False, True])
def test_not_a_number_counts_in_no_maximum(cuda, asym):
    """A group's largest (and smallest) value is that of its numbers: groups with a NaN at any place keep the parameters they have
    with a zero there."""
    cfg = C.CodecConfig("sdp4bit", 4, 32, asym, False)
    x = torch.randn(32, 32, device=cuda)
    at = torch.arange(32, device=cuda)
    zero, nan = x.clone(), x.clone()
    zero[at, at] = 0.0
    nan[at, at] = float("nan")
    a, b = (C.encode(v.reshape(-1), cfg, 1)[0] for v in (zero, nan))
    payload = 32 * 16
    assert torch.equal(a[payload:], b[payload:])


@pytest.mark.parametrize("cfg", [C.SDP4BIT_G128, C.ZFP_RATE8], ids=lambda c: c.kind)
@pytest.mark.parametrize("count", [4099, 8192 * 300 + 5])
def test_launches_in_a_chain_see_one_another(cuda, cfg, count):
    """Back-to-back launches without a wait: a chain through the same two buffers, each read by one kernel and overwritten
    by the next but one, gives what it gives with a wait behind every launch; in a stream and in a graph."""
    x = torch.randn(6, count, device=cuda)
    nb = cfg.encoded_chunk_bytes(count, torch.float32)
    enc = torch.empty(1, nb, dtype=torch.uint8, device=cuda)
    y = torch.empty(count, device=cuda)
    lib, c = _lib.lib(), cfg.to_c(torch.float32)

    def chain(wait=lambda: None):
        outs = [torch.empty_like(y) for _ in range(6)]
        for i in range(6):
            src = y if i % 2 else x[i]
            _lib.check(lib.cocclkEncode(src.data_ptr(), enc.data_ptr(), count, 1, count, nb, 0, c, _lib.cur_stream()), "cocclkEncode")
            wait()
            _lib.check(lib.cocclkDecodeReduce(enc.data_ptr(), y.data_ptr(), count, 1, 1, count, nb, 0, c, _lib.cur_stream()), "cocclkDecodeReduce")
            wait()
            outs[i].copy_(y)
            wait()
        return outs
    want = chain(torch.cuda.synchronize)
    for _ in range(5):
        for a, b in zip(chain(), want):
            assert torch.equal(a, b)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = chain()
    for _ in range(3):
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(outs, want))


@pytest.mark.parametrize("cfg", [C.SDP4BIT_G128, C.CodecConfig("sdp4bit", 4, 128, True, True), C.CodecConfig("sdp4bit", 8, 128, False, True),
                                 C.CodecConfig("sdp4bit", 4, 8, False, False), C.MXFP8, *(C.CodecConfig("taco", 8, g, False, False) for g in (32, 64, 128, 512))],
                         ids=lambda c: f"{c.kind}{c.bits}g{c.group}{'a' if c.asym else 's'}")
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("chunks,count", [(3, 8192 * 3 + 512), (1, 512), (600, 8192)])
def test_one_copy_decodes_alike_wherever_it_is_put(cuda, cfg, dtype, chunks, count):
    """Aligned fp32 goes through another kernel than everything else: the same values, bit for bit, one element further on."""
    torch.manual_seed(count)
    x = torch.randn(chunks * count, device=cuda).to(dtype)
    enc = C.encode(x, cfg, chunks)
    room = torch.full((chunks * count + 16,), float("nan"), dtype=dtype, device=cuda)
    want = C.decode(enc, cfg, count, dtype, chunks).reshape(-1)
    for first in (0, 1, 3):
        out = room[first:first + chunks * count].fill_(float("nan"))
        _lib.check(_lib.lib().cocclkDecodeReduce(enc.data_ptr(), out.data_ptr(), count, chunks, 1, count, enc.shape[1], C.DTYPE_CODE[dtype],
                                                 cfg.to_c(dtype), _lib.cur_stream()), "cocclkDecodeReduce")
        assert torch.equal(out, want), first
        assert room[first + chunks * count:].isnan().all() and room[:first].isnan().all()
        room.fill_(float("nan"))
