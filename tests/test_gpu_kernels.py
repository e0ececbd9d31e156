"""GPU parity: every CUDA entry point, called through the C ABI, against the CPU oracles.

Decoders must be bit-exact (uint16 views, including -0.0).  The fused matvec and the layer forward
must agree with the oracle within relative L2 1e-3 (the fp16 budget of the path); the transforms,
being fp32, within 1e-5.
"""
import numpy as np
import pytest
import torch

import c_oracle as C
import qtip_oracle as O
from conftest import rel_l2
from qtip_b200 import ops, synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def dev(a):
    if a.dtype == np.uint16:
        return torch.from_numpy(a.view(np.int16)).to(DEV)
    return torch.from_numpy(a).to(DEV)


def u16(t):
    if torch.is_tensor(t):
        t = t.cpu().numpy()
    return np.ascontiguousarray(t).view(np.uint16)


# ---- decoders: bit exact ---------------------------------------------------------------------------
@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("shape", ["32x64", "64x96"])
def test_decode_hyb_golden(golden, K, shape):
    g = golden("decode_kernel")
    m, n = map(int, shape.split("x"))
    W = ops.decode_hyb(dev(g[f"codes_K{K}_{shape}"]), dev(g["tlut"]), K, m, n)
    assert np.array_equal(u16(W), u16(g[f"W_K{K}_{shape}"]))


@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("m,n", [(256, 256), (4096, 4096), (4096, 11008), (11008, 4096),
                                 (2048, 2048), (2080, 2048), (131104, 32), (32, 160000),
                                 # and of the one chosen for unsettled weights (16384 blocks)
                                 (4128, 4096), (524832, 32), (32, 524832)])
def test_decode_hyb_vs_oracle(K, m, n):
    lay = synth.make_layer(m, n, K, seed=2000 + K)
    codes, tlut = dev(lay["codes"]), dev(lay["tlut"])
    W = ops.decode_hyb(codes, tlut, K, m, n)
    assert np.array_equal(u16(W), u16(C.decode_kernel(lay["codes"], m, n, K, lay["tlut"])))
    torch.cuda.synchronize()
    assert torch.equal(W.view(torch.int16), ops.decode_hyb(codes, tlut, K, m, n, settled=True).view(torch.int16))


def write_early(dst, seed):
    """fp16 values into dst by a launch that lets the one after it start before it has written anything: 4096 or 1024 a row."""
    half = dst.view(torch.float16).view(-1)
    n = 4096 if half.numel() % 4096 == 0 else 1024
    x = torch.randn(half.numel() // n, n, device=DEV, generator=torch.Generator(DEV).manual_seed(seed)).half()
    torch.cuda.synchronize()
    ops.rht_fused(x, x.shape[0], n, half, scale=n**-0.5)


@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("m,n", [(1024, 1024), (16384, 4096)])
@pytest.mark.parametrize("operand", ["codes", "tlut"])
def test_decode_hyb_reads_what_the_launch_before_wrote(K, m, n, operand):
    for seed in range(3):
        codes = torch.full((K * m * n // 16,), -1, dtype=torch.int16, device=DEV)
        tlut = torch.full((512, 2), 7.0, dtype=torch.float16, device=DEV)
        write_early(codes if operand == "codes" else tlut, seed)
        W = ops.decode_hyb(codes, tlut, K, m, n)
        assert torch.equal(W.view(torch.int16), ops.decode_hyb(codes, tlut, K, m, n).view(torch.int16))


# ---- producers of the packed formats: bit exact ---------------------------------------------------------
@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("V", [1, 2])
def test_pack_trellis_golden(golden, K, V):
    g = golden("pack_trellis")
    states = torch.from_numpy(g[f"states_V{V}_K{K}"].astype(np.int32)).to(DEV)
    words = ops.pack_trellis(states, K, V)
    assert np.array_equal(u16(words), g[f"packed_V{V}_K{K}"])
    bad = states.clone()
    bad[1, 7] ^= 0x8000          # the top bit overlaps with the previous state only
    with pytest.raises(RuntimeError, match="1 consecutive state pairs"):
        ops.pack_trellis(bad, K, V)
    # check=False packs whatever it is given, like the arithmetic upstream without its assert
    ops.pack_trellis(bad, K, V, check=False)


VITERBI_CASES = [("quantlut_sym", 2, 2), ("quantlut_sym", 3, 2), ("quantlut_sym", 4, 2), ("3inst", 2, 1), ("1mad", 2, 1),
                 ("3inst", 3, 1), ("1mad", 4, 1)]


@pytest.mark.parametrize("mode,K,V", VITERBI_CASES)
def test_viterbi_quantize_golden(golden, mode, K, V):
    """The tail-biting Viterbi quantizer returns the very states upstream's bitshift_codebook.quantize returned."""
    g = golden("viterbi")
    X = torch.from_numpy(g[f"X_{mode}_K{K}"]).to(DEV)
    states = ops.viterbi_quantize(X, mode, K, tlut=torch.from_numpy(g["tlut32"]))
    assert np.array_equal(states.cpu().numpy().astype(np.uint16), g[f"states_{mode}_K{K}"])


@pytest.mark.parametrize("mode,K,V,N", [("quantlut_sym", 2, 2, 300), ("quantlut_sym", 3, 2, 40), ("quantlut_sym", 4, 2, 40),
                                        ("3inst", 2, 1, 24), ("1mad", 3, 1, 24), ("3inst", 4, 1, 24)])
def test_viterbi_quantize_vs_oracle(mode, K, V, N):
    """More sequences than CTAs can hold at once (the grid-stride loop), scaled inputs, against the C restatement of
    upstream's formulation (full cost vector per step); bit-exact states and final costs."""
    rng = np.random.default_rng(40 + K + V)
    code = ops.CODE_IDS[mode]
    tlut32 = (rng.standard_normal((512, 2)) * 0.97).astype(np.float32)
    X = (rng.standard_normal((N, 256)) * rng.uniform(0.2, 3.0, size=(N, 1))).astype(np.float16)
    X[1] = 0                                                    # all candidates tie on a constant sequence
    want, want_cost = C.viterbi_quantize(X, K, V, O.recons_table(code, tlut32))
    got, cost = ops.viterbi_quantize(torch.from_numpy(X).to(DEV), mode, K, tlut=torch.from_numpy(tlut32), return_cost=True)
    assert np.array_equal(got.cpu().numpy(), want)
    assert np.array_equal(cost.cpu().numpy().view(np.uint32), want_cost.view(np.uint32))


@pytest.mark.parametrize("N", [2, 5, 301, 1182])
def test_viterbi_sequences_sharing_a_place(N):
    """HYB K = 2: the least workspace makes two sequences share a place, anything up to the full one fewer; the same results."""
    from qtip_b200 import _lib
    g = torch.Generator(device=DEV).manual_seed(N)
    X, tlut = torch.randn(N, 64, generator=g, device=DEV).half(), torch.randn(512, 2, generator=g, device=DEV)
    want, want_cost = ops.viterbi_quantize(X, "quantlut_sym", 2, tlut=tlut, return_cost=True)
    lib = _lib.load()
    least, full = (f(_lib.CODE_HYB, 2, 64, N) for f in (lib.qtip_viterbi_workspace_bytes, lib.qtip_viterbi_workspace_bytes_full))
    assert least < full
    for size in (least, (least + full) // 2, full, 2 * full):
        ws = torch.empty(size, dtype=torch.uint8, device=DEV)
        states, cost = torch.zeros_like(want), torch.zeros_like(want_cost)
        _lib.check(lib.qtip_viterbi_quantize(states.data_ptr(), cost.data_ptr(), X.data_ptr(), N, 64, _lib.CODE_HYB, 2, tlut.data_ptr(),
                                             ws.data_ptr(), size, torch.cuda.current_stream().cuda_stream), "viterbi")
        assert torch.equal(states, want) and torch.equal(cost, want_cost)


@pytest.mark.parametrize("mode,K,T,N,limit", [("3inst", 3, 64, 11, 3 << 20), ("quantlut_sym", 2, 36, 700, 1 << 20), ("1mad", 4, 22, 5, 1 << 18)])
def test_viterbi_quantize_with_little_memory(monkeypatch, mode, K, T, N, limit):
    """Where the workspace for all sequences cannot be had the call takes fewer at a time; where not even one fits it raises."""
    g = torch.Generator(device=DEV).manual_seed(N)
    X, tlut = torch.randn(N, T, generator=g, device=DEV).half(), torch.randn(512, 2, generator=g, device=DEV)
    want, want_cost = ops.viterbi_quantize(X, mode, K, tlut=tlut, return_cost=True)
    real, sizes = torch.empty, []

    def empty(*size, **kw):
        if kw.get("dtype") == torch.uint8:
            sizes.append(size[0])
            if size[0] > limit:
                raise torch.OutOfMemoryError("not in this test")
        return real(*size, **kw)
    monkeypatch.setattr(ops.torch, "empty", empty)
    before = ops.launch_count
    got, cost = ops.viterbi_quantize(X, mode, K, tlut=tlut, return_cost=True)
    assert len(sizes) > 1 and sizes == sorted(set(sizes), reverse=True) and ops.launch_count - before > 1
    assert torch.equal(got, want) and torch.equal(cost, want_cost)
    limit = 1 << 10
    with pytest.raises(torch.OutOfMemoryError):
        ops.viterbi_quantize(X, mode, K, tlut=tlut)


@pytest.mark.parametrize("mode,K,V", VITERBI_CASES)
@pytest.mark.parametrize("T,N", [(16, 1), (256, 1500)])
def test_viterbi_wait_that_runs_out(mode, K, V, T, N):
    """No poll allowed: every wait for a stored row is given up.  The kernel ends, every sequence (also those a CTA had not begun)
    is marked by negative states that pack_trellis refuses and a cost that is no number, and the next call is right."""
    from qtip_b200 import _lib
    code = ops.CODE_IDS[mode]
    g = torch.Generator(device=DEV).manual_seed(T + K)
    X = torch.randn(N, T, generator=g, device=DEV).half()
    tlut = torch.randn(512, 2, generator=g, device=DEV)
    want, want_cost = ops.viterbi_quantize(X, mode, K, tlut=tlut, return_cost=True)
    lib = _lib.load()
    need = lib.qtip_viterbi_workspace_bytes(code, K, T, N)
    ws = torch.empty(need, dtype=torch.uint8, device=DEV)
    states, cost = torch.empty_like(want), torch.zeros(N, device=DEV)

    def call(polls):
        _lib.check(lib.qtip_viterbi_quantize_polls(states.data_ptr(), cost.data_ptr(), X.data_ptr(), N, T, code, K, tlut.data_ptr(),
                                                   ws.data_ptr(), need, polls, torch.cuda.current_stream().cuda_stream), "viterbi")
    call(0)
    assert bool((states < 0).all()) and bool(torch.isnan(cost).all())
    if T == 256:
        with pytest.raises(RuntimeError, match="do not overlap"):
            ops.pack_trellis(states, K, V)
    call(1 << 20)
    assert torch.equal(states, want) and torch.equal(cost, want_cost)


@pytest.mark.parametrize("mode,K,T,N", [("quantlut_sym", 2, 8, 3), ("quantlut_sym", 4, 16, 1), ("3inst", 2, 8, 2), ("1mad", 3, 64, 1),
                                        ("quantlut_sym", 3, 1024, 2)])
def test_viterbi_quantize_short_and_long_sequences(mode, K, T, N):
    """Sequence lengths other than a 16x16 tile - the shortest the tail-biting construction allows (16 stream bits), a single
    sequence, the longest the kernel takes (1024) - against the C restatement."""
    rng = np.random.default_rng(T + K)
    code = ops.CODE_IDS[mode]
    V = 2 if mode == "quantlut_sym" else 1
    tlut32 = rng.standard_normal((512, 2)).astype(np.float32)
    X = rng.standard_normal((N, T)).astype(np.float16)
    want, want_cost = C.viterbi_quantize(X, K, V, O.recons_table(code, tlut32))
    got, cost = ops.viterbi_quantize(torch.from_numpy(X).to(DEV), mode, K, tlut=torch.from_numpy(tlut32), return_cost=True)
    assert np.array_equal(got.cpu().numpy(), want)
    assert np.array_equal(cost.cpu().numpy().view(np.uint32), want_cost.view(np.uint32))


@pytest.mark.parametrize("mode,K,T", [("quantlut_sym", 2, 12), ("quantlut_sym", 2, 20), ("quantlut_sym", 3, 28), ("quantlut_sym", 4, 36),
                                      ("3inst", 2, 22), ("3inst", 3, 14), ("3inst", 4, 10), ("1mad", 2, 18), ("1mad", 3, 26), ("1mad", 4, 6)])
def test_viterbi_quantize_trace_depths(mode, K, T):
    """Walk lengths whose back-trace starts and stops inside a tree of stored rows (odd halves, partial depths), with tied
    candidates (repeated values), against the C restatement."""
    rng = np.random.default_rng(T * K)
    V = 2 if mode == "quantlut_sym" else 1
    tlut32 = np.round(rng.standard_normal((512, 2)) * 2).astype(np.float32) / 2
    X = (np.round(rng.standard_normal((5, T)) * 2) / 2).astype(np.float16)
    want, want_cost = C.viterbi_quantize(X, K, V, O.recons_table(ops.CODE_IDS[mode], tlut32))
    got, cost = ops.viterbi_quantize(torch.from_numpy(X).to(DEV), mode, K, tlut=torch.from_numpy(tlut32), return_cost=True)
    assert np.array_equal(got.cpu().numpy(), want)
    assert np.array_equal(cost.cpu().numpy().view(np.uint32), want_cost.view(np.uint32))


def test_producers_smallest_shapes():
    """One tile / one block: pack_trellis on a single tile, the layout shuffles on a single 32 x 32 block."""
    rng = np.random.default_rng(3)
    for K in (2, 3, 4):
        plain = rng.integers(0, 65536, size=(4, 16 * K), dtype=np.uint16)
        kern = ops.plain_to_kernel_layout(dev(plain), K, 32, 32)
        assert np.array_equal(u16(kern).reshape(-1), O.plain_words_to_kernel_layout(plain, 32, 32, K).reshape(-1))
        for V in (1, 2):
            st = O.states_plain_layout(plain[:1], 16, 16, K, V)
            words = ops.pack_trellis(torch.from_numpy(st.astype(np.int32)).to(DEV), K, V)
            assert np.array_equal(u16(words), plain[:1])


def test_viterbi_quantize_to_decoder():
    """The quantizer's tail on the GPU, end to end: sequences -> Viterbi states -> pack_trellis -> kernel layout -> fused
    decoder.  4096 sequences (a 1024 x 1024 matrix of 16x16 tiles); the table is fp16-representable so that the decoder
    (fp16 table) reproduces the quantizer's reconstruction exactly.  Checks that every walk bites its tail (pack_trellis
    counts violations), that the decoded matrix is the reconstruction the quantizer minimised over, and that the
    reported cost is its squared error."""
    K, m, n = 2, 1024, 1024
    rng = np.random.default_rng(9)
    tl16 = rng.standard_normal((512, 2)).astype(np.float16)
    W = rng.standard_normal((m, n)).astype(np.float32)
    # 16x16 tiles as sequences, row-major inside the tile (lib/algo/finetune.py:188-194 hands these rows to the quantizer)
    seqs = W.reshape(m // 16, 16, n // 16, 16).transpose(0, 2, 1, 3).reshape(-1, 256)
    Xd = torch.from_numpy(seqs).to(DEV)
    states, cost = ops.viterbi_quantize(Xd, "quantlut_sym", K, tlut=torch.from_numpy(tl16.astype(np.float32)), return_cost=True)
    words = ops.pack_trellis(states, K, 2)                  # raises if a walk does not overlap / bite its tail
    assert np.array_equal(O.states_plain_layout(u16(words), m, n, K, 2), states.cpu().numpy().astype(np.uint16))
    hat = ops.decode_plain(words, "quantlut_sym", K, m, n, tlut=dev(tl16)).float().cpu().numpy()
    x16 = seqs.astype(np.float16).astype(np.float64).reshape(m // 16, n // 16, 16, 16).transpose(0, 2, 1, 3).reshape(m, n)
    err_tiles = ((hat.astype(np.float64) - x16) ** 2).reshape(m // 16, 16, n // 16, 16).sum(axis=(1, 3)).reshape(-1)
    assert np.allclose(cost.cpu().numpy(), err_tiles, rtol=1e-5)
    # 2 bits per weight on N(0,1) data: the trellis code gets close to the rate-distortion bound (0.0625); a scalar
    # quantizer is at 0.118
    assert 0.06 < err_tiles.sum() / (m * n) < 0.085
    # a handful of sequences against the oracle
    want, _ = C.viterbi_quantize(seqs[:16].astype(np.float16), K, 2, O.recons_table(O.CODE_HYB, tl16.astype(np.float32)))
    assert np.array_equal(states[:16].cpu().numpy(), want)
    # the same codes through the kernel layout and the fused decoder
    kern = ops.plain_to_kernel_layout(words, K, m, n)
    Wk = ops.decode_hyb(kern, dev(tl16), K, m, n)
    assert np.array_equal(u16(Wk), u16(C.decode_kernel(u16(kern), m, n, K, tl16)))


@pytest.mark.parametrize("K,V,m,n", [(2, 2, 4096, 4096), (3, 2, 1024, 2048), (4, 2, 256, 512), (2, 1, 2048, 1024), (4, 1, 512, 512)])
def test_pack_trellis_round_trip(K, V, m, n):
    """pack(unpack(words)) == words on uniform code words (every 256*K-bit stream is a tail-biting walk), and against
    the numpy restatement on a sample of the tiles."""
    rng = np.random.default_rng(77 + K + V)
    codes = rng.integers(0, 65536, size=(m * n // 256, 16 * K), dtype=np.uint16)
    states = O.states_plain_layout(codes, m, n, K, V)
    words = ops.pack_trellis(torch.from_numpy(states.astype(np.int32)).to(DEV), K, V)
    assert np.array_equal(u16(words), codes)
    assert np.array_equal(O.pack_trellis(states[:64], K, V), codes[:64])


@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("m,n", [(32, 64), (64, 96), (4096, 4096), (4096, 11008)])
def test_layout_shuffle_vs_oracle(K, m, n):
    rng = np.random.default_rng(5 + K)
    plain = rng.integers(0, 65536, size=(m * n // 256, 16 * K), dtype=np.uint16)
    kern = ops.plain_to_kernel_layout(dev(plain), K, m, n)
    assert np.array_equal(u16(kern).reshape(-1), O.plain_words_to_kernel_layout(plain, m, n, K).reshape(-1))
    back = ops.kernel_to_plain_layout(kern, K, m, n)
    assert np.array_equal(u16(back), plain)
    assert np.array_equal(u16(ops.kernel_to_plain_layout(dev(plain), K, m, n)).reshape(-1),
                          O.kernel_layout_to_plain_words(plain, m, n, K).reshape(-1))


def test_quantizer_tail_to_decoder():
    """States -> pack_trellis -> kernel layout -> the fused decoder gives the plain-layout decode of the same states with
    the elements moved by the kernel's sequence permutation (what lib/algo/finetune.py:188-201 hands to the kernels)."""
    K, m, n = 2, 256, 512
    lay = synth.make_layer(m, n, K, seed=31)
    plain = O.kernel_layout_to_plain_words(lay["codes"], m, n, K)
    states = O.states_plain_layout(plain, m, n, K, 2)
    words = ops.pack_trellis(torch.from_numpy(states.astype(np.int32)).to(DEV), K, 2)
    kern = ops.plain_to_kernel_layout(words, K, m, n)
    assert np.array_equal(u16(kern).reshape(-1), lay["codes"].reshape(-1))
    W = ops.decode_hyb(kern, dev(lay["tlut"]), K, m, n)
    assert np.array_equal(u16(W), u16(C.decode_kernel(lay["codes"], m, n, K, lay["tlut"])))


@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("mode", ["3inst", "1mad", "quantlut_sym"])
def test_decode_plain_golden(golden, K, mode):
    g = golden("decode_plain")
    W = ops.decode_plain(dev(g[f"codes_{mode}_K{K}"]), mode, K, 32, 64, tlut=dev(g["tlut"]))
    # 3INST values are fp16-exact; 1MAD is upstream's fp32 value rounded once to fp16
    assert np.array_equal(u16(W), u16(g[f"W_{mode}_K{K}"].astype(np.float16)))


@pytest.mark.parametrize("code,V", [(O.CODE_3INST, 1), (O.CODE_1MAD, 1), (O.CODE_HYB, 2)])
@pytest.mark.parametrize("K,m,n", [(2, 64, 96), (3, 256, 256), (4, 64, 96), (2, 8192, 8192)])
def test_decode_plain_vs_oracle(code, V, K, m, n):
    lay = synth.make_layer(m, n, K, seed=2100 + K)
    W = ops.decode_plain(dev(lay["codes"]), code, K, m, n, tlut=dev(lay["tlut"]))
    want = C.decode_plain(lay["codes"], m, n, K, V, O.state_table(code, lay["tlut"]))
    assert np.array_equal(u16(W), u16(want))


def test_state_functions_all_65536_states():
    """Every state value through both compute codes and the HYB hash: a stream whose windows enumerate
    all 16-bit states (K=4, V=1 / V=2 tiles filled with a counter pattern would not cover them), so
    instead decode random tiles until every state was seen at least once."""
    K, m, n = 4, 512, 512
    lay = synth.make_layer(m, n, K, seed=5)
    st = O.states_plain_layout(lay["codes"], m, n, K, 1)
    assert np.unique(st).size > 64000
    for code in (O.CODE_3INST, O.CODE_1MAD):
        W = ops.decode_plain(dev(lay["codes"]), code, K, m, n)
        assert np.array_equal(u16(W), u16(O.decode_plain_layout(lay["codes"], m, n, K, 1, code)))


# ---- fused matvec ----------------------------------------------------------------------------------
def test_known_answer():
    """qtip-kernels/src/test.cu:22-58 upstream: zero codes, LUT 1.0, x 1.0 => every output is exactly n."""
    for (m, n) in ((8192, 8192), (64, 256)):
        codes = torch.zeros(m * n // 256, 32, dtype=torch.int16, device=DEV)
        tlut = torch.ones(512, 2, dtype=torch.float16, device=DEV)
        x = torch.ones(1, n, dtype=torch.float16, device=DEV)
        y = ops.decompress_matvec(codes, x, tlut, 2, m, n)
        assert torch.all(y == n)


@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("m,n,bs", [(32, 64, 1), (64, 96, 1), (256, 256, 1), (4096, 4096, 1), (4096, 11008, 1),
                                    (11008, 4096, 1), (1024, 8192, 1), (4096, 4096, 4), (512, 1024, 8)])
def test_matvec_hyb(K, m, n, bs):
    lay = synth.make_layer(m, n, K, seed=3000 + K, bs=bs)
    out = torch.full((bs, m), float("nan"), device=DEV)  # the op overwrites, it must not accumulate
    y = ops.decompress_matvec(dev(lay["codes"]), dev(lay["x"]), dev(lay["tlut"]), K, m, n, out=out)
    want = C.matvec_kernel(lay["codes"], m, n, K, lay["tlut"], lay["x"])
    assert rel_l2(y.cpu().numpy(), want) < 1e-3
    assert rel_l2(y.cpu().numpy(), want) < 2e-6  # fp32 accumulation of exact fp16 products: only summation order differs
    y2 = ops.decompress_matvec(dev(lay["codes"]), dev(lay["x"]), dev(lay["tlut"]), K, m, n)
    assert torch.equal(y, y2), "result must be deterministic run to run"


def test_matvec_hyb_upstream_test_inputs():
    """Inputs shaped like prepare_arguments of qtip-kernels/test_decompress_matvec.py:251-272 upstream
    (codebook and x ~ N(0,1)/16 clamped to [-1,1]); acceptance as there: allclose(atol=1e-5, rtol=1e-2) in fp16."""
    g = torch.Generator().manual_seed(42)
    for K in (2, 3, 4):
        for (m, n) in ((256, 256), (8192, 1024), (1024, 8192)):
            cb = (torch.randn(1024, generator=g).half() / 16).clamp(-1, 1)
            codes = torch.randint(-2**31, 2**31, (K * m * n // 32,), generator=g, dtype=torch.int64).to(torch.int32)
            x = (torch.randn(n, 1, generator=g).half() / 16).clamp(-1, 1)
            y = ops.decompress_matvec(codes.to(DEV), x.to(DEV).view(1, n), cb.to(DEV), K, m, n)
            W = C.decode_kernel(codes.numpy(), m, n, K, cb.numpy())
            ref = torch.from_numpy(C.matvec_dense(W, x.numpy().reshape(1, n)))
            assert torch.allclose(y.cpu().half(), ref.half(), atol=1e-5, rtol=0.01)


@pytest.mark.parametrize("code", [O.CODE_3INST, O.CODE_1MAD])
@pytest.mark.parametrize("K,m,n,bs", [(2, 32, 64, 1), (2, 256, 256, 1), (3, 64, 96, 2), (4, 128, 256, 8),
                                      (2, 8192, 8192, 1), (2, 8192, 8192, 4)])
def test_matvec_plain(code, K, m, n, bs):
    lay = synth.make_layer(m, n, K, seed=3100 + K, bs=bs, code="none")
    y = ops.decompress_matvec_plain(dev(lay["codes"]), dev(lay["x"]), code, K, m, n)
    W = C.decode_plain(lay["codes"], m, n, K, 1, O.state_table(code))
    want = C.matvec_dense(W, lay["x"])
    assert rel_l2(y.cpu().numpy(), want) < 1e-3
    assert rel_l2(y.cpu().numpy(), want) < 2e-6


# ---- Hadamard -----------------------------------------------------------------------------------------
@pytest.mark.parametrize("n", [128, 896, 2048, 4096, 6656, 11008])
def test_hadamard_golden(golden, n):
    g = golden("hadamard")
    hk, k = ops.get_hadK(n)
    x = dev(g[f"x_{n}"])
    hk = None if hk is None else hk.to(DEV)
    assert rel_l2(ops.hadamard(x, hk, k).cpu().numpy(), g[f"y_{n}"]) < 1e-5
    assert rel_l2(ops.hadamard(x, hk, k, transpose=True).cpu().numpy(), g[f"yt_{n}"]) < 1e-5


@pytest.mark.parametrize("n", [2, 64, 8192, 14336, 16384, 28672, 53248])
def test_rht_vs_oracle(n):
    rng = np.random.default_rng(n)
    rows = 3
    x = rng.standard_normal((rows, n)).astype(np.float32)
    su = np.sign(rng.standard_normal(n)).astype(np.float16)
    sv = (np.sign(rng.standard_normal(n)) * (0.5 + rng.random(n))).astype(np.float32)
    hk, k = ops.get_hadK(n)
    bits = None if hk is None else ops.pack_hadk(hk.to(DEV))
    hkn = None if hk is None else hk.numpy()
    # input side: fp32 in, fp16 out, sign in, transposed factor
    got = ops.rht(dev(x), sign_in=dev(su), hadk_bits=bits, kfac=k, transpose=True, scale=1 / np.sqrt(n) / 32,
                  out_dtype=torch.float16)
    want = O.hadamard(x * su.astype(np.float32), hkn, transpose=True) / 32
    assert rel_l2(got.float().cpu().numpy(), want) < 6e-4  # fp16 output rounding
    # output side: fp32 in, fp32 out, sign out
    got = ops.rht(dev(x), sign_out=dev(sv), hadk_bits=bits, kfac=k, scale=1 / np.sqrt(n))
    want = O.hadamard(x, hkn) * sv
    assert rel_l2(got.cpu().numpy(), want) < 1e-5
    # fp16 in
    xh = x.astype(np.float16)
    got = ops.rht(dev(xh), hadk_bits=bits, kfac=k, scale=1 / np.sqrt(n), out_dtype=torch.float32)
    assert rel_l2(got.cpu().numpy(), O.hadamard(xh.astype(np.float32), hkn)) < 1e-5


@pytest.mark.parametrize("n", [96, 1376, 2240, 2496, 3328, 5120, 11008, 13824, 14336, 22016, 24576, 28672, 53248])
@pytest.mark.parametrize("rows", [1, 3, 28, 75, 151])
@pytest.mark.parametrize("kind", ["fp16", "fp16-scales", "fp32", "wide"])
def test_rht_factor_rows(n, rows, kind):
    """Factor widths over every split of the work (rows of the view of 8..2048 columns, parts of a row, clusters, whole rows),
    both directions: fp16 activations with signs (exact operands), or with a scale among the signs, fp32 values, and fp32 rows whose magnitudes differ by
    many orders (scaled heads and remainders)."""
    g = torch.Generator(device=DEV).manual_seed(n + rows)
    k = ops.had_factor(n)
    H = ops.get_hadK(n)[0].to(DEV)
    bits = ops.pack_hadk(H)
    x = torch.randn(rows, n, generator=g, device=DEV)
    if kind == "wide":
        x = x * 10.0 ** torch.linspace(-30, 30, rows, device=DEV)[:, None] * 10.0 ** torch.linspace(-4, 0, n, device=DEV)
    x = x.half() if "fp16" in kind else x
    su = (torch.randn(n, generator=g, device=DEV).sign() + 1e-5).sign().half()
    if kind == "fp16-scales":
        su[n // 3] = 1.3
    sv = torch.randn(n, generator=g, device=DEV)
    hh = torch.ones(1, 1, dtype=torch.float64, device=DEV)
    while hh.shape[0] < n // k:
        hh = torch.cat([torch.cat([hh, hh], 1), torch.cat([hh, -hh], 1)], 0)
    for transpose in (False, True):
        F = (H.T if transpose else H).double()
        want = torch.einsum("ik,rkj,jl->ril", F, (x.double() * su.double()).view(rows, k, n // k), hh).reshape(rows, n) * sv.double() / n**0.5
        got = ops.rht(x, sign_in=su, sign_out=sv, hadk_bits=bits, kfac=k, transpose=transpose, scale=1 / n**0.5, out_dtype=torch.float32)
        err = (got.double() - want).norm(dim=1) / want.norm(dim=1)
        assert float(err.max()) < 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1376, 11008, 13824, 7168, 14336, 28672, 24576])
def test_rht_factor_fp16_results(n):
    """Every width of the stores (rows of the view of 8 to 2048 columns), with and without signs: the fp32 results rounded once."""
    bits, k = ops.pack_hadk(ops.get_hadK(n)[0].to(DEV)), ops.had_factor(n)
    x, sv = torch.randn(200, n, device=DEV).half(), torch.randn(n, device=DEV)
    for sign in (None, sv):
        y = [ops.rht(x, sign_out=sign, hadk_bits=bits, kfac=k, scale=1 / n**0.5, out_dtype=t) for t in (torch.float16, torch.float32)]
        assert torch.equal(y[0], y[1].half())


@pytest.mark.parametrize("n", [1024, 2048, 4096, 8192, 16384, 32768, 65536])
@pytest.mark.parametrize("rows", [1, 5, 28, 149])
def test_rht_pow2_rows(n, rows):
    """Power-of-two rows over every split (several rows per CTA with a partly filled last one, one row per CTA, clusters), with
    the whole prologue: residual add, RMSNorm, SwiGLU gate and signs."""
    g = torch.Generator(device=DEV).manual_seed(n + rows)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    x, res, gate = r(rows, n).half(), r(rows, n).half(), r(rows, n).half()
    w, su, sv = (1 + 0.1 * r(n)).half(), (r(n).sign() + 1e-5).sign().half(), r(n)

    def transform(v):
        v, h = v.double().clone(), 1
        while h < n:
            v = v.view(-1, n // (2 * h), 2, h)
            v = torch.stack((v[:, :, 0] + v[:, :, 1], v[:, :, 0] - v[:, :, 1]), 2).reshape(-1, n)
            h *= 2
        return v / n**0.5
    got = ops.rht(x.float(), sign_in=su, sign_out=sv, scale=1 / n**0.5)
    want = transform(x.double() * su.double()) * sv.double()
    assert float(((got - want).norm(dim=1) / want.norm(dim=1)).max()) < 1e-6
    out, res_out = torch.empty(rows, n, device=DEV), torch.empty_like(x)
    ops.rht_fused(x, rows, n, out, residual=res, residual_out=res_out, norm_weight=w, eps=1e-5, gate=gate, sign_in=su, scale=1 / n**0.5)
    s = x + res
    assert torch.equal(res_out, s)
    v = w * (s.float() * torch.rsqrt(s.float().pow(2).mean(-1, keepdim=True) + 1e-5)).half()
    v = torch.nn.functional.silu(gate.float()).half() * v
    want = transform(v.double() * su.double())
    assert float(((out - want).norm(dim=1) / want.norm(dim=1)).max()) < 1e-3


def test_rht_chunked_signs():
    """Per-chunk transforms of the tensor-parallel layouts: rows cycle through the chunks of the sign vector."""
    rng = np.random.default_rng(0)
    bs, tp, seg = 2, 8, 832  # 832 = 52 * 16
    x = rng.standard_normal((bs, tp * seg)).astype(np.float32)
    su = np.sign(rng.standard_normal(tp * seg)).astype(np.float32)
    hk, k = ops.get_hadK(seg)
    got = ops.rht(dev(x).reshape(bs * tp, seg), sign_in=dev(su), hadk_bits=ops.pack_hadk(hk.to(DEV)), kfac=k,
                  transpose=True, scale=1 / np.sqrt(seg)).reshape(bs, tp * seg)
    want = O.hadamard((x * su).reshape(bs * tp, seg), hk.numpy(), transpose=True).reshape(bs, tp * seg)
    assert rel_l2(got.cpu().numpy(), want) < 1e-5


# ---- tcgen05 decompress-GEMM ---------------------------------------------------------------------------------
@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("m,n,bs", [(128, 64, 16), (256, 256, 9), (1024, 2048, 32), (8192, 8192, 16), (4096, 11008, 64),
                                    (11008, 4096, 33), (1024, 2048, 65), (4096, 4096, 128), (8192, 8192, 100)])
def test_decompress_gemm(K, m, n, bs):
    """Tensor-core path against the dense product of the (bit-exact) decoded matrix, fp32 accumulation."""
    lay = synth.make_layer(m, n, K, seed=3300 + K, bs=bs)
    codes, x, tl = dev(lay["codes"]), dev(lay["x"]), dev(lay["tlut"])
    y = ops.decompress_gemm(codes, x, tl, K, m, n)
    W = ops.decode_hyb(codes, tl, K, m, n)
    want = x.float() @ W.float().T
    torch.cuda.synchronize()
    assert ops.gemm_status(DEV) == 0, "a bounded barrier wait inside the kernel gave up"
    assert rel_l2(y.cpu().numpy(), want.cpu().numpy()) < 1e-3
    assert rel_l2(y.cpu().numpy(), want.cpu().numpy()) < 1e-5
    y2 = ops.decompress_gemm(codes, x, tl, K, m, n)
    assert torch.equal(y, y2)


@pytest.mark.gpu
@pytest.mark.parametrize("code", [O.CODE_3INST, O.CODE_1MAD])
@pytest.mark.parametrize("K,m,n,bs", [(2, 128, 64, 16), (2, 1024, 2048, 32), (3, 256, 256, 9), (4, 512, 1024, 64),
                                      (2, 8192, 8192, 16), (2, 1024, 2048, 128), (3, 512, 1024, 72)])
def test_decompress_gemm_plain_vs_oracle(code, K, m, n, bs):
    """Compute codes (V = 1, plain layout) on the tensor-core path against the CPU oracle: bit-exact decode
    (C.decode_plain with the oracle's state table) + dense product with fp32 accumulation."""
    lay = synth.make_layer(m, n, K, seed=3500 + K, bs=bs, code="none")
    y = ops.decompress_gemm_plain(dev(lay["codes"]), dev(lay["x"]), code, K, m, n)
    torch.cuda.synchronize()
    want = C.matvec_dense(C.decode_plain(lay["codes"], m, n, K, 1, O.state_table(code)), lay["x"])
    assert ops.gemm_status(DEV) == 0, "a bounded barrier wait inside the kernel gave up"
    assert rel_l2(y.cpu().numpy(), want) < 1e-5
    assert torch.equal(y, ops.decompress_gemm_plain(dev(lay["codes"]), dev(lay["x"]), code, K, m, n))


@pytest.mark.gpu
@pytest.mark.parametrize("K,m,n,bs", [(2, 1024, 2048, 16), (4, 256, 256, 40), (3, 1024, 1024, 128), (2, 256, 512, 90)])
def test_decompress_gemm_vs_oracle(K, m, n, bs):
    """The tensor-core path directly against the CPU oracle (decode of the kernel layout + dense product), with no
    CUDA kernel of this library on the reference side."""
    lay = synth.make_layer(m, n, K, seed=3400 + K, bs=bs)
    y = ops.decompress_gemm(dev(lay["codes"]), dev(lay["x"]), dev(lay["tlut"]), K, m, n)
    torch.cuda.synchronize()
    want = C.matvec_dense(C.decode_kernel(lay["codes"], m, n, K, lay["tlut"]), lay["x"])
    assert ops.gemm_status(DEV) == 0
    assert rel_l2(y.cpu().numpy(), want) < 1e-5


@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("code", [O.CODE_HYB, O.CODE_3INST, O.CODE_1MAD])
@pytest.mark.parametrize("m,n,bs", [(128, 192, 1), (128, 256, 49), (384, 320, 64), (128, 832, 65), (256, 1216, 128)])
def test_decompress_gemm_ring_edges(K, code, m, n, bs):
    """Step counts around the groups and the depth of the stage ring, batches around the 32-row copies of x."""
    lay = synth.make_layer(m, n, K, seed=3600 + K, bs=bs, **({} if code == O.CODE_HYB else {"code": "none"}))
    codes, x = dev(lay["codes"]), dev(lay["x"])
    if code == O.CODE_HYB:
        tl = dev(lay["tlut"])
        y, W = ops.decompress_gemm(codes, x, tl, K, m, n), ops.decode_hyb(codes, tl, K, m, n)
    else:
        y, W = ops.decompress_gemm_plain(codes, x, code, K, m, n), ops.decode_plain(codes, code, K, m, n)
    want = C.matvec_dense(W.cpu().numpy(), lay["x"])
    assert ops.gemm_status(DEV) == 0
    assert rel_l2(y.cpu().numpy(), want) < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("m,n,bs", [(64, 8192, 8), (4096, 8192, 5), (1024, 16384, 3), (320, 32768, 8), (32, 65536, 1)])
def test_transform_in_fragment_order(K, m, n, bs):
    """The transform's fragment order and the matvec that takes it: the bits of the row-major transform and its own re-ordering."""
    lay = synth.make_layer(m, n, K, seed=3900 + K, bs=bs, device=DEV)
    assert ops.matvec_takes_fragments(K, m, n, bs)
    x, su = lay["x"].to(torch.float16), lay["SU"].to(torch.float16)
    rows, frag = (torch.empty(bs, n, dtype=torch.float16, device=DEV) for _ in range(2))
    ops.rht_fused(x, bs, n, rows, sign_in=su, scale=n**-0.5)
    ops.rht_fused(x, bs, n, frag, sign_in=su, scale=n**-0.5, fragments=True)
    # block of 32 columns, row, thread t, pairs 2t + 8i
    want = rows.view(bs, n // 32, 4, 4, 2).permute(1, 0, 3, 2, 4).reshape(bs, n)
    assert torch.equal(frag, want)
    y = ops.decompress_matvec(lay["codes"], frag, lay["tlut"], K, m, n, fragments=True)
    assert torch.equal(y, ops.decompress_matvec(lay["codes"], rows, lay["tlut"], K, m, n))
    with pytest.raises(RuntimeError):
        ops.rht_fused(x[:, :4096].contiguous(), bs, 4096, frag, fragments=True)      # a width whose kernel does not write it


@pytest.mark.gpu
@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("code", [O.CODE_HYB, O.CODE_3INST, O.CODE_1MAD])
@pytest.mark.parametrize("m,n,bs", [(1024, 1024, 9), (8192, 4096, 27), (8192, 4096, 200)])
def test_decompress_gemm_reads_what_the_launch_before_wrote(K, code, m, n, bs):
    hyb = code == O.CODE_HYB
    x = torch.randn(bs, n, device=DEV, generator=torch.Generator(DEV).manual_seed(9)).half()
    codes = torch.zeros(K * m * n // 16, dtype=torch.int16, device=DEV)
    tlut = torch.zeros(512, 2, dtype=torch.float16, device=DEV)

    def product():
        if bs > ops.MAX_GEMM_BATCH:
            return ops.decompress_gemm_f16(codes, x, code, K, m, n, tlut=tlut if hyb else None)
        return ops.decompress_gemm(codes, x, tlut, K, m, n) if hyb else ops.decompress_gemm_plain(codes, x, code, K, m, n)

    product()
    for seed in range(3):
        for t in (codes, tlut) if hyb else (codes,):
            codes.fill_(-1)
            write_early(t, seed)
            y = product()
            assert torch.equal(y, product())
            if bs <= ops.MAX_GEMM_BATCH:
                assert torch.equal(y, ops.decompress_gemm(codes, x, tlut, K, m, n, settled=True) if hyb
                                   else ops.decompress_gemm_plain(codes, x, code, K, m, n, settled=True))
    assert ops.gemm_status(DEV) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("bs", [33, 75, 97, 113])
def test_decompress_gemm_x_ring_depths(bs):
    """The depths of the ring of x (6, 4, 4 and 3 stages) with several rounds in one CTA and a last step of one tile."""
    K, m, n = 2, 9600, 1600
    lay = synth.make_layer(m, n, K, seed=3700 + bs, bs=bs, device=DEV)
    y, W = ops.decompress_gemm(lay["codes"], lay["x"], lay["tlut"], K, m, n), ops.decode_hyb(lay["codes"], lay["tlut"], K, m, n)
    want = lay["x"].double() @ W.double().T
    assert ops.gemm_status(DEV) == 0
    assert rel_l2(y.cpu().numpy(), want.cpu().numpy()) < 1e-5      # 1600 fp32 additions, the bound of the tests above


@pytest.mark.gpu
@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("code", [O.CODE_HYB, O.CODE_3INST, O.CODE_1MAD])
@pytest.mark.parametrize("m,n,bs", [(128, 64, 129), (384, 320, 256), (256, 832, 257), (19200, 192, 300), (2560, 1216, 1000),
                                    (38016, 704, 1), (38016, 704, 16), (38016, 704, 17), (38016, 704, 128)])
def test_decompress_gemm_f16(K, code, m, n, bs):
    """One to several batch groups and tiles per CTA, an odd number of 64-column tiles, one step per tile, ragged last groups, few rows
    (all eight stages of x, several times round); against the dense product of the (bit-exact) decoded
    matrix in 64 bits: rounding to fp16 is 2^-11 of a value at most, uniform."""
    lay = synth.make_layer(m, n, K, seed=3800 + K, bs=bs, device=DEV, **({} if code == O.CODE_HYB else {"code": "none"}))
    hyb = code == O.CODE_HYB
    y = ops.decompress_gemm_f16(lay["codes"], lay["x"], code, K, m, n, tlut=lay["tlut"] if hyb else None)
    W = ops.decode_hyb(lay["codes"], lay["tlut"], K, m, n) if hyb else ops.decode_plain(lay["codes"], code, K, m, n)
    want = lay["x"].double() @ W.double().T
    assert ops.gemm_status(DEV) == 0
    assert float((y.double() - want).norm() / want.norm()) < 2.0**-11
    assert torch.equal(y, ops.decompress_gemm_f16(lay["codes"], lay["x"], code, K, m, n, tlut=lay["tlut"] if hyb else None))


@pytest.mark.gpu
@pytest.mark.parametrize("ctx", [1, 7, 200, 257, 2048, 2049, 5000])
@pytest.mark.parametrize("heads", [(8, 8), (16, 2)])
def test_attn_decode_matches_fp32_softmax(ctx, heads):
    """Single-query attention over a cache of `ctx` rows against an fp32 torch reference (tolerance:
    fp16 rounding of the output, 2e-3 absolute on values of order 1)."""
    n_heads, n_kv = heads
    hd = 128
    g = torch.Generator(device="cuda").manual_seed(ctx * 31 + n_heads)
    q = torch.randn(n_heads, hd, generator=g, device="cuda").half()
    ck = torch.randn(ctx + 3, n_kv * hd, generator=g, device="cuda").half()
    cv = torch.randn(ctx + 3, n_kv * hd, generator=g, device="cuda").half()
    pos = torch.tensor([ctx - 1], dtype=torch.int32, device="cuda")
    out = torch.empty(n_heads, hd, dtype=torch.float16, device="cuda")
    ops.attn_decode(out, q, ck, cv, pos, n_heads, n_kv, hd)
    rep = n_heads // n_kv
    k = ck[:ctx].float().view(ctx, n_kv, hd).repeat_interleave(rep, dim=1)     # (ctx, heads, hd)
    v = cv[:ctx].float().view(ctx, n_kv, hd).repeat_interleave(rep, dim=1)
    s = torch.einsum("hd,thd->ht", q.float(), k) / hd ** 0.5
    ref = torch.einsum("ht,thd->hd", torch.softmax(s, dim=-1), v)
    torch.testing.assert_close(out.float(), ref, atol=2e-3, rtol=2e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(4096, 32000), (512, 1001), (16384, 2048)])
def test_lm_head_matches_torch(shape):
    """Final RMSNorm + fp16 head against torch (fp32 accumulation; tolerance 1e-3 relative L2)."""
    hidden, vocab = shape
    g = torch.Generator(device="cuda").manual_seed(hidden + vocab)
    res = torch.randn(hidden, generator=g, device="cuda").half()
    delta = (0.3 * torch.randn(hidden, generator=g, device="cuda")).half()
    w_norm = (1 + 0.1 * torch.randn(hidden, generator=g, device="cuda")).half()
    W = (0.02 * torch.randn(vocab, hidden, generator=g, device="cuda")).half()
    logits = torch.zeros(vocab, device="cuda")
    ops.lm_head(logits, res, delta, w_norm, W, 1e-5)
    h = (res + delta).float()
    h = (h * torch.rsqrt(h.pow(2).mean() + 1e-5)).half() * w_norm
    want = h.float() @ W.float().T
    assert rel_l2(logits.cpu().numpy(), want.cpu().numpy()) < 1e-3


@pytest.mark.gpu
def test_embed_and_sampler():
    """Embedding lookup is a copy; the sampler returns one of the top-k logits, is reproducible for a seed and a
    position, follows softmax(top / temperature) over many positions, and advances the position."""
    vocab, hidden, k = 5000, 256, 5
    g = torch.Generator(device="cuda").manual_seed(5)
    embed = torch.randn(vocab, hidden, generator=g, device="cuda").half()
    tok = torch.tensor([1234], dtype=torch.int64, device="cuda")
    res = torch.zeros(hidden, dtype=torch.float16, device="cuda")
    delta = torch.ones(hidden, dtype=torch.float16, device="cuda")
    ops.embed_token(res, delta, embed, tok)
    assert torch.equal(res, embed[1234]) and torch.count_nonzero(delta) == 0

    logits = torch.randn(vocab, generator=g, device="cuda")
    top = torch.topk(logits, k)
    n_draws = 4000
    out = torch.full((n_draws + 2,), -1, dtype=torch.int64, device="cuda")
    pos = torch.zeros(1, dtype=torch.int32, device="cuda")
    for _ in range(n_draws):
        ops.sample_top_k(tok, out, pos, logits, temperature=0.6, top_k=k, seed=77)
    torch.cuda.synchronize()
    assert int(pos) == n_draws and int(out[0]) == -1 and int(tok) == int(out[n_draws])
    drawn = out[1:n_draws + 1]
    assert bool(torch.isin(drawn, top.indices).all())
    want = torch.softmax(top.values / 0.6, dim=0)
    freq = torch.stack([(drawn == i).float().mean() for i in top.indices])
    assert torch.allclose(freq, want, atol=0.03)
    # same seed and positions -> same tokens
    out2 = torch.full_like(out, -1)
    pos.zero_()
    for _ in range(50):
        ops.sample_top_k(tok, out2, pos, logits, temperature=0.6, top_k=k, seed=77)
    assert torch.equal(out2[1:51], out[1:51])


@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("m,n,bs", [(32, 32, 1), (32, 992, 1), (64, 32, 3), (9600, 64, 1), (4736, 1024, 1), (4768, 1056, 1), (9472, 1024, 2),
                                    (5000 * 32, 32, 1), (64, 65536, 1), (96, 32768, 8), (14208, 4096, 7), (512, 16384, 5),
                                    (9504, 4768, 8), (12288, 4096, 8), (28672, 8192, 8), (53248, 8192, 8), (65536, 8192, 7)])
def test_matvec_hyb_partitions(K, m, n, bs):
    """Every way of cutting the work: rows shorter than a warp each, pieces and contiguous runs, several rounds of row blocks,
    shared row blocks, x staged and x through the ring - against the decoded matrix."""
    lay = synth.make_layer(m, n, K, seed=m + n + bs, bs=bs, device=DEV)
    codes = lay["codes"].view(torch.int16)
    got = ops.decompress_matvec(codes, lay["x"], lay["tlut"], K, m, n)
    want = lay["x"].double() @ ops.decode_hyb(codes, lay["tlut"], K, m, n).double().T
    assert float((got.double() - want).norm() / want.norm()) < 2e-6
    assert torch.equal(got, ops.decompress_matvec(codes, lay["x"], lay["tlut"], K, m, n))


@pytest.mark.parametrize("K,m,n,bs", [(2, 28672, 8192, 1), (2, 28672, 8192, 5), (3, 53248, 8192, 8), (4, 53248, 4096, 2), (2, 16384, 16384, 8)])
def test_matvec_hyb_error_of_long_runs(K, m, n, bs):
    """A warp that decodes a run of many blocks must not add all of them in one tensor-core accumulator, whose additions truncate.
    Bound: an accumulator takes a 32nd of a row, n / 512 additions of at most 2^-23 of the partial sum and 2^-24 on average, and 32 parts
    are added with rounding (about 6 units of 2^-24 as a random walk)."""
    lay = synth.make_layer(m, n, K, seed=m + n + bs, bs=bs, device=DEV)
    codes = lay["codes"].view(torch.int16)
    got = ops.decompress_matvec(codes, lay["x"], lay["tlut"], K, m, n).double()
    W = ops.decode_hyb(codes, lay["tlut"], K, m, n)
    want = torch.cat([lay["x"].double() @ W[i:i + 8192].double().T for i in range(0, m, 8192)], dim=1)
    assert float((got - want).norm() / want.norm()) < 2.0**-24 * (n / 512 + 6)


@pytest.mark.parametrize("n", [1152, 6656, 11008, 17920, 28672, 53248, 55296])
@pytest.mark.parametrize("rows", [1, 300])
def test_factor_transform_error_of_fp32_rows(n, rows):
    """fp32 rows are split into two fp16 parts (2^-23 of a value, uniform: 2^-23 / sqrt(3) in the norm); the additions of the factor
    (truncating, at most 11 of them on the heads) and the stages stay below that again: 1.25 * 2^-23 in all, which the fp32 additions
    of a plain evaluation take as well."""
    hk, k = ops.get_hadK(n)
    x = torch.randn(rows, n, generator=torch.Generator(device=DEV).manual_seed(n), device=DEV)
    for transpose in (False, True):
        got = ops.rht(x, hadk_bits=ops.pack_hadk(hk.to(DEV)), kfac=k, transpose=transpose, scale=n**-0.5).double()
        v, h = x.double().view(rows, k, -1), 1
        while h < n // k:
            v = v.reshape(rows, k, -1, 2, h)
            v = torch.stack([v[:, :, :, 0] + v[:, :, :, 1], v[:, :, :, 0] - v[:, :, :, 1]], dim=3)
            h *= 2
        hd = hk.double().to(DEV)
        want = ((hd.T if transpose else hd) @ v.reshape(rows, k, -1)).view(rows, n) * n**-0.5
        assert float((got - want).norm() / want.norm()) < 1.25 * 2.0**-23
