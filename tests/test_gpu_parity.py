"""GPU parity: every kernel of the X-engine against the CPU oracle (bit-exact for
all integer work) and against the reference's own kernels compiled from its
sources (k_packAB + cgemm_blk_t, src/rx_host_corr.cu:61-72, src/cgemm.cuh:28-69).

Floating-point tolerances, stated here and used below:
  * FP32 dump cube vs exact int64: each entry is the single correctly rounded
    FP32 value (bit-exact against numpy's float32 cast).
  * FP32 image vs FP64 oracle: max |img - img64| <= 1e-5 * max |img64|.
"""
import numpy as np
import pytest

import mixer
import oracle

pytestmark = pytest.mark.gpu


def _t(arr, cuda):
    import torch
    return torch.from_numpy(np.ascontiguousarray(arr)).to(cuda)


def _zeros(n, dtype, cuda):
    import torch
    return torch.zeros(n, dtype=dtype, device=cuda)


def _sync():
    import torch
    torch.cuda.synchronize()


# ---------------------------------------------------------------- packet source

@pytest.mark.parametrize("nant,nch,tpkt,nheaps,mode,sigma", [
    (256, 128, 32, 4, 0, 16.0),
    (40, 64, 64, 3, 0, 12.0),
    (32, 256, 16, 2, 1, 0.0),
])
def test_gen_packets_match_oracle(cuda, nant, nch, tpkt, nheaps, mode, sigma):
    import torch
    sky = oracle.sky_table(nant, nch, 16, [(0.10, -0.05, 6.0, 0.0), (0.2, 0.0, 0.0, 1.5)])
    sky_m = mixer.sky_table(nant, nch, 16, [(0.10, -0.05, 6.0, 0.0), (0.2, 0.0, 0.0, 1.5)])
    assert np.array_equal(sky, sky_m)
    stride = 64 + 2 * nch * tpkt
    dev = _zeros(nheaps * nant * stride, torch.uint8, cuda)
    dsky = _t(sky, cuda)
    mixer.gen_packets(dev, stride, 64, nant, nch, tpkt, nheaps, 3, 77, 4096, dsky, sigma, 1234, mode)
    _sync()
    ref = oracle.gen_packets(nant, nch, tpkt, nheaps, heap0=3, seq0=77, sky=sky, sigma=sigma,
                             seed=1234, mode=mode)
    assert np.array_equal(dev.cpu().numpy(), ref)


# ------------------------------------------------------------------ corner-turn

@pytest.mark.parametrize("nant,nch,tpkt,nheaps,k0,extra", [
    (256, 128, 32, 8, 0, 0),      # wire default, one 256-sample sub-integration
    (96, 64, 64, 4, 128, 64),     # offset into a wider plane
    (128, 256, 16, 16, 0, 0),     # 256-channel packets
    (40, 16, 16, 3, 16, 32),      # heaps not a multiple of any group
])
def test_corner_turn_matches_oracle(cuda, nant, nch, tpkt, nheaps, k0, extra):
    import torch
    pk = oracle.gen_packets(nant, nch, tpkt, nheaps, seq0=9, seed=5, sigma=30.0)
    stride = 64 + 2 * nch * tpkt
    kt = k0 + nheaps * tpkt + extra
    dpk = _t(pk, cuda)
    planes = torch.full((2, nch, nant, kt), 7, dtype=torch.int8, device=cuda)
    seq_err = _zeros(1, torch.int32, cuda)
    err = _zeros(1, torch.int32, cuda)
    mixer.corner_turn(dpk, stride, 64, nant, nch, tpkt, nheaps, 9, planes, kt, k0, seq_err, err)
    _sync()
    got = planes.cpu().numpy()
    ref = oracle.corner_turn(pk, nant, nch, tpkt, nheaps)
    assert np.array_equal(got[:, :, :, k0:k0 + nheaps * tpkt], ref)
    assert np.all(got[:, :, :, :k0] == 7) and np.all(got[:, :, :, k0 + nheaps * tpkt:] == 7)
    assert int(seq_err.item()) == 0 and int(err.item()) == 0


def test_corner_turn_counts_seq_errors(cuda):
    import torch
    nant, nch, tpkt, nheaps = 64, 128, 32, 4
    stride = 64 + 2 * nch * tpkt
    pk = oracle.gen_packets(nant, nch, tpkt, nheaps, seq0=100)
    v = pk.reshape(-1, stride)
    v[5, 51] ^= 0x10          # one corrupted seq
    v[[70, 71]] = v[[71, 70]]  # two packets swapped
    planes = _zeros(2 * nch * nant * nheaps * tpkt, torch.int8, cuda)
    seq_err = _zeros(1, torch.int32, cuda)
    mixer.corner_turn(_t(pk, cuda), stride, 64, nant, nch, tpkt, nheaps, 100, planes,
                      nheaps * tpkt, 0, seq_err)
    _sync()
    assert int(seq_err.item()) == 3 == oracle.seq_errors(pk, nheaps * nant, 100, stride)


# --------------------------------------------------------- tensor-core triangle GEMM

def _rand_planes(rng, nch, nant, kt, lo=-128, hi=128):
    return rng.integers(lo, hi, size=(2, nch, nant, kt), dtype=np.int8)


@pytest.mark.parametrize("nant,nch,kt,kbeg,klen", [
    (128, 2, 128, 0, 128),
    (256, 3, 512, 0, 512),
    (200, 2, 384, 0, 384),      # N not a multiple of the tile
    (40, 5, 64, 0, 64),         # K shorter than one stage
    (384, 2, 256, 0, 256),      # 6 tiles per channel, 3 diagonal
    (256, 2, 512, 128, 256),    # sample sub-range
    (130, 1, 208, 16, 176),     # ragged: N = 128 + 2, K not a multiple of 128
])
def test_xcorr_store_i32_matches_oracle(cuda, nant, nch, kt, kbeg, klen):
    import torch
    rng = np.random.default_rng(nant * 7 + kt)
    planes = _rand_planes(rng, nch, nant, kt)
    vis = _zeros(mixer.vis_elems(nant, nch), torch.int32, cuda)
    err = _zeros(1, torch.int32, cuda)
    mixer.xcorr_tri(_t(planes, cuda), nant, nch, kt, kbeg, klen, mixer.VIS_STORE_I32, vis, err)
    _sync()
    assert int(err.item()) == 0
    full = oracle.correlate(planes, kbeg=kbeg, klen=klen)
    ref = oracle.vis_tile_pack(full).reshape(-1)
    got = vis.cpu().numpy().astype(np.int64)
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("nant", [1, 15, 16, 17, 100, 129, 143, 160, 241, 255, 257, 300, 383, 1000])
@pytest.mark.parametrize("mode", ["store", "acc32", "acc64"])
def test_xcorr_ragged_last_block_matches_oracle(cuda, nant, mode):
    """N not a multiple of 128: the last block's tiles run with that block on
    the MMA's N side (N = 2 r16, r16 = rows rounded up to 16), the tiles left
    of the diagonal as conjugate transposes written back transposed.  Every
    rounding class of the last block, each mode, -128 rows in the ragged
    block; store mode rewrites the padding rows (the cube starts as junk),
    the accumulate modes add twice."""
    import torch
    rng = np.random.default_rng(nant * 3 + len(mode))
    nch, kt = 2, 384
    planes = _rand_planes(rng, nch, nant, kt)
    planes[:, :, -min(nant, 5):, ::3] = -128
    dpl = _t(planes, cuda)
    n = mixer.vis_elems(nant, nch)
    err = _zeros(1, torch.int32, cuda)
    ref = oracle.vis_tile_pack(oracle.correlate(planes)).reshape(-1)
    if mode == "store":
        vis = torch.full((n,), 0x5A5A5A5A, dtype=torch.int32, device=cuda)
        mixer.xcorr_tri(dpl, nant, nch, kt, 0, kt, mixer.VIS_STORE_I32, vis, err)
        times = 1
    else:
        dt = torch.int64 if mode == "acc64" else torch.int32
        md = mixer.VIS_ACC_I64 if mode == "acc64" else mixer.VIS_ACC_I32
        vis = _zeros(n, dt, cuda)
        for _ in range(2):
            mixer.xcorr_tri(dpl, nant, nch, kt, 0, kt, md, vis, err)
        times = 2
    _sync()
    assert int(err.item()) == 0
    assert np.array_equal(vis.cpu().numpy().astype(np.int64), times * ref)


def test_xcorr_accumulate_modes(cuda):
    import torch
    rng = np.random.default_rng(11)
    nant, nch, kt = 256, 4, 1024
    planes = _rand_planes(rng, nch, nant, kt)
    dpl = _t(planes, cuda)
    n = mixer.vis_elems(nant, nch)
    v32 = _zeros(n, torch.int32, cuda)
    v64 = _zeros(n, torch.int64, cuda)
    for k in range(0, kt, 256):
        mixer.xcorr_tri(dpl, nant, nch, kt, k, 256, mixer.VIS_ACC_I32, v32)
        mixer.xcorr_tri(dpl, nant, nch, kt, k, 256, mixer.VIS_ACC_I64, v64)
    _sync()
    ref = oracle.vis_tile_pack(oracle.correlate(planes)).reshape(-1)
    assert np.array_equal(v32.cpu().numpy().astype(np.int64), ref)
    assert np.array_equal(v64.cpu().numpy(), ref)
    # flush: v64 += v32, v32 = 0  (k_flush_cube, exact)
    mixer.vis_flush(v32, v64, n)
    _sync()
    assert np.array_equal(v64.cpu().numpy(), 2 * ref)
    assert int(v32.abs().max().item()) == 0


@pytest.mark.parametrize("pairs", ["0", "1"])
@pytest.mark.parametrize("max_ctas", [1, 7, 100000])
def test_xcorr_cta_cap_is_exact(cuda, monkeypatch, max_ctas, pairs):
    """mixer_xcorr_tri_ex: fewer persistent CTAs walk more items each, same cube
    (one-SM kernel, and the pair kernel with max_ctas / 2 clusters)."""
    import torch
    monkeypatch.setenv("MIXER_XCORR_PAIRS", pairs)
    rng = np.random.default_rng(31 + max_ctas)
    nant, nch, kt = 384, 3, 512
    planes = _rand_planes(rng, nch, nant, kt)
    v64 = _zeros(mixer.vis_elems(nant, nch), torch.int64, cuda)
    err = _zeros(1, torch.int32, cuda)
    mixer.xcorr_tri(_t(planes, cuda), nant, nch, kt, 0, kt, mixer.VIS_ACC_I64, v64, err,
                    max_ctas=max_ctas)
    _sync()
    assert int(err.item()) == 0
    ref = oracle.vis_tile_pack(oracle.correlate(planes)).reshape(-1)
    assert np.array_equal(v64.cpu().numpy(), ref)


@pytest.mark.parametrize("nant,nch,kt,kbeg,klen,mode", [
    (384, 3, 512, 0, 512, "store"),      # 3 row blocks: 3 pairs, one leftover pair
    (512, 2, 256, 0, 256, "acc64"),      # 4 blocks: 5 pairs
    (640, 2, 384, 128, 256, "store"),    # 5 blocks: last leftover pair has one tile
    (1000, 2, 208, 16, 176, "acc64"),    # 8 blocks, ragged N and K
    (1024, 4, 1024, 0, 1024, "acc32"),   # 8 blocks, 18 pairs per channel
])
def test_xcorr_pairs_match_oracle(cuda, monkeypatch, nant, nch, kt, kbeg, klen, mode):
    """MIXER_XCORR_PAIRS=1: from three 128-row blocks up the GEMM runs on pairs
    of SMs (tcgen05 cta_group::2): two tiles that share a column block per
    cluster, leftover tiles as conjugate-transposed products.  Every mode is
    exact."""
    import torch
    monkeypatch.setenv("MIXER_XCORR_PAIRS", "1")
    rng = np.random.default_rng(nant + kt + klen)
    planes = _rand_planes(rng, nch, nant, kt)
    dt = torch.int64 if mode == "acc64" else torch.int32
    vis = _zeros(mixer.vis_elems(nant, nch), dt, cuda)
    err = _zeros(1, torch.int32, cuda)
    md = {"store": mixer.VIS_STORE_I32, "acc32": mixer.VIS_ACC_I32, "acc64": mixer.VIS_ACC_I64}[mode]
    mixer.xcorr_tri(_t(planes, cuda), nant, nch, kt, kbeg, klen, md, vis, err)
    _sync()
    assert int(err.item()) == 0
    ref = oracle.vis_tile_pack(oracle.correlate(planes, kbeg=kbeg, klen=klen)).reshape(-1)
    assert np.array_equal(vis.cpu().numpy().astype(np.int64), ref)


def test_xcorr_pairs_equal_single_sm(cuda, monkeypatch):
    """The pair kernel (MIXER_XCORR_PAIRS=1) and the one-SM kernel give the same
    cube, including -128 inputs and the int32 bound of one launch."""
    import torch
    rng = np.random.default_rng(77)
    nant, nch, kt = 768, 2, 65408
    planes = rng.integers(-128, 128, size=(2, nch, nant, kt), dtype=np.int8)
    planes[:, :, :128] = -128                        # one row block at the extreme
    dpl = _t(planes, cuda)
    n = mixer.vis_elems(nant, nch)
    out = []
    for env in ("1", "0"):
        monkeypatch.setenv("MIXER_XCORR_PAIRS", env)
        v = _zeros(n, torch.int32, cuda)
        err = _zeros(1, torch.int32, cuda)
        mixer.xcorr_tri(dpl, nant, nch, kt, 0, kt, mixer.VIS_STORE_I32, v, err)
        _sync()
        assert int(err.item()) == 0
        out.append(v.cpu().numpy())
    assert np.array_equal(out[0], out[1])
    ref = oracle.vis_tile_pack(oracle.correlate(planes, nc=1)).reshape(-1)
    assert np.array_equal(out[0][:ref.size].astype(np.int64), ref)


def test_xcorr_partial_last_round_is_exact(cuda):
    """256 elements x 128 channels = 384 tile items on 148 persistent CTAs: the
    last round is partly empty and two thirds of the tiles are diagonal.  The
    int64 accumulate and int32 store launches give the same cube, equal to the
    oracle's exact sums on the first channels."""
    import torch
    rng = np.random.default_rng(41)
    nant, nch, kt = 256, 128, 16384
    planes = _rand_planes(rng, nch, nant, kt)
    dpl = _t(planes, cuda)
    n = mixer.vis_elems(nant, nch)
    v32 = _zeros(n, torch.int32, cuda)
    v64 = _zeros(n, torch.int64, cuda)
    err = _zeros(1, torch.int32, cuda)
    mixer.xcorr_tri(dpl, nant, nch, kt, 0, kt, mixer.VIS_STORE_I32, v32, err)
    mixer.xcorr_tri(dpl, nant, nch, kt, 0, kt, mixer.VIS_ACC_I64, v64, err)
    _sync()
    assert int(err.item()) == 0
    assert np.array_equal(v64.cpu().numpy(), v32.cpu().numpy().astype(np.int64))
    sub = 4                                                # oracle on the first channels
    ref = oracle.vis_tile_pack(oracle.correlate(planes, nc=sub)).reshape(-1)
    assert np.array_equal(v64[:ref.size].cpu().numpy(), ref)


@pytest.mark.parametrize("pairs", ["0", "1"])
def test_xcorr_large_array_matches_oracle(cuda, monkeypatch, pairs):
    """4096 elements (32 row blocks, 528 tiles per channel, tile indices past
    the float decode's easy range) and 4000 (ragged last block), int64 mode,
    one-SM and pair kernels."""
    import torch
    monkeypatch.setenv("MIXER_XCORR_PAIRS", pairs)
    for nant in (4096, 4000):
        rng = np.random.default_rng(nant)
        nch, kt = 1, 384
        planes = _rand_planes(rng, nch, nant, kt)
        v64 = _zeros(mixer.vis_elems(nant, nch), torch.int64, cuda)
        err = _zeros(1, torch.int32, cuda)
        mixer.xcorr_tri(_t(planes, cuda), nant, nch, kt, 0, kt, mixer.VIS_ACC_I64, v64, err)
        _sync()
        assert int(err.item()) == 0
        ref = oracle.vis_tile_pack(oracle.correlate(planes)).reshape(-1)
        assert np.array_equal(v64.cpu().numpy(), ref), nant


def test_mma_peak_probe(cuda):
    """The tensor-core rate probe runs its MMA stream to completion."""
    import torch
    err = _zeros(1, torch.int32, cuda)
    mixer.mma_peak(200, 0, err)
    mixer.mma_peak(50, 3, err)
    _sync()
    assert int(err.item()) == 0


def test_xcorr_extreme_inputs(cuda):
    """-128 everywhere: exact here; the reference's -A_im (src/cgemm.cuh:52) wraps."""
    import torch
    nant, nch, kt = 128, 1, 65408                      # largest int32-safe launch
    planes = np.full((2, nch, nant, kt), -128, dtype=np.int8)
    planes[1, 0, ::2] = 127
    vis = _zeros(mixer.vis_elems(nant, nch), torch.int32, cuda)
    mixer.xcorr_tri(_t(planes, cuda), nant, nch, kt, 0, kt, mixer.VIS_STORE_I32, vis)
    _sync()
    ref = oracle.vis_tile_pack(oracle.correlate(planes)).reshape(-1)
    assert np.array_equal(vis.cpu().numpy().astype(np.int64), ref)
    assert ref.max() == 2 * 128 * 128 * kt


def test_xcorr_long_integration_splits(cuda):
    """I64 mode over more samples than one int32-safe launch."""
    import torch
    rng = np.random.default_rng(2)
    nant, nch, kt = 128, 1, 65408 + 1024
    planes = rng.integers(-128, 128, size=(2, nch, nant, kt), dtype=np.int8)
    v64 = _zeros(mixer.vis_elems(nant, nch), torch.int64, cuda)
    mixer.xcorr_tri(_t(planes, cuda), nant, nch, kt, 0, kt, mixer.VIS_ACC_I64, v64)
    _sync()
    ref = oracle.vis_tile_pack(oracle.correlate(planes)).reshape(-1)
    assert np.array_equal(v64.cpu().numpy(), ref)


# ------------------------------------------------------------- cube outputs

def test_unpack_and_dump(cuda):
    import torch
    rng = np.random.default_rng(8)
    nant, nch, kt = 300, 3, 256
    planes = _rand_planes(rng, nch, nant, kt)
    full = oracle.correlate(planes) * 40000               # values beyond 2^24
    packed = _t(oracle.vis_tile_pack(full).reshape(-1), cuda)
    out64 = _zeros(nch * 2 * nant * nant, torch.int64, cuda)
    out32 = _zeros(nch * 2 * nant * nant, torch.float32, cuda)
    mixer.vis_unpack_i64(packed, nant, nch, out64)
    mixer.vis_dump_f32(packed, nant, nch, out32)
    _sync()
    assert np.array_equal(out64.cpu().numpy().reshape(full.shape), full)
    assert np.array_equal(out32.cpu().numpy().reshape(full.shape), full.astype(np.float32))


# ------------------------------------------------------------- context pipeline

def _config0_packets(nheaps, heap0=0, seed=99, nant=256, nch=128, tpkt=32, side=16):
    sky = oracle.sky_table(nant, nch, side, [(0.10, -0.05, 6.0, 0.0), (0.2, 0.0, 0.0, 1.5)])
    return oracle.gen_packets(nant, nch, tpkt, nheaps, heap0=heap0, seq0=heap0 * nant, sky=sky,
                              sigma=16.0, seed=seed)


def test_context_device_and_host_packets(cuda):
    import torch
    nheaps = 24
    pk = _config0_packets(nheaps)
    full = oracle.correlate(oracle.corner_turn(pk, 256, 128, 32, nheaps))
    with mixer.ArrayContext(max_heaps=8) as ctx:
        ctx.correlate(_t(pk, cuda), nheaps, seq0=0, on_device=True)       # 3 chunks
        out = _zeros(full.size, torch.int64, cuda)
        ctx.read_vis_i64(out, full_square=True)
        _sync()
        assert np.array_equal(out.cpu().numpy().reshape(full.shape), full)
        # same packets again from pageable and pinned host memory: doubles V
        ctx.correlate(pk, nheaps, seq0=0, on_device=False)
        pinned = torch.from_numpy(pk).pin_memory()
        ctx.correlate(pinned, nheaps, seq0=0, on_device=False)
        host = np.zeros(full.size, dtype=np.int64)
        ctx.read_vis_i64(host, full_square=True, on_device=False)
        _sync()
        assert np.array_equal(host.reshape(full.shape), 3 * full)
        st = ctx.stats()
        assert st["seq_errors"] == 0 and st["kernel_err"] == 0
        assert st["samples"] == 3 * nheaps * 32


def test_context_int32_split_and_dump(cuda, tmp_path):
    import torch
    nheaps = 16
    pk = _config0_packets(nheaps, seed=4)
    full = oracle.correlate(oracle.corner_turn(pk, 256, 128, 32, nheaps))
    with mixer.ArrayContext(max_heaps=16) as ctx:
        dpk = _t(pk, cuda)
        ctx.correlate_i32(dpk, 8, seq0=0)
        ctx.correlate_i32(dpk[8 * 256 * 8256:], 8, seq0=8 * 256)
        ctx.integrate()
        with pytest.raises(mixer.MixerError) as e:     # int32 headroom is enforced
            for _ in range(300):
                ctx.correlate_i32(dpk, 16, seq0=0)
        assert e.value.rc == mixer.EOVERFLOW
        ctx.reset()
        ctx.correlate_i32(dpk, 16, seq0=0)
        ctx.integrate()
        cube = torch.zeros(full.size, dtype=torch.float32, device=cuda)
        ctx.dump(cube)
        path = str(tmp_path / "v.f32")
        ctx.dump_to_file(path)
        ctx.dump_to_file(path)
        _sync()
        ref32 = full.astype(np.float32)
        assert np.array_equal(cube.cpu().numpy().reshape(full.shape), ref32)
        rec = np.fromfile(path, dtype=np.float32)
        assert rec.size == 2 * full.size
        assert np.array_equal(rec[:full.size].reshape(full.shape), ref32)


def test_context_detects_misordered_packets(cuda):
    nheaps = 8
    pk = _config0_packets(nheaps, seed=3).reshape(-1, 8256).copy()
    pk[[3, 4]] = pk[[4, 3]]
    with mixer.ArrayContext(max_heaps=8) as ctx:
        ctx.correlate(pk.reshape(-1), nheaps, seq0=0, on_device=False)
        assert ctx.stats()["seq_errors"] == 2


# ------------------------------------------------------------------- imaging

@pytest.mark.parametrize("nant,side,G,nch", [(256, 16, 32, 8), (1024, 32, 64, 2), (64, 8, 16, 3),
                                             (4096, 64, 128, 1)])
def test_grid_and_image(cuda, nant, side, G, nch):
    import torch
    rng = np.random.default_rng(nant)
    kt = 64
    planes = rng.integers(-100, 100, size=(2, nch, nant, kt), dtype=np.int8)
    full = oracle.correlate(planes)
    packed = _t(oracle.vis_tile_pack(full).reshape(-1), cuda)
    g = _zeros(nch * G * G * 2, torch.int64, cuda)
    mixer.grid(packed, nant, nch, side, G, g)
    img = _zeros(nch * G * G, torch.float32, cuda)
    vmax = _zeros(nch, torch.float32, cuda)
    vmin = _zeros(nch, torch.float32, cuda)
    mixer.image_fft(g, nch, G, img, vmax, vmin)
    _sync()
    gref = oracle.grid(full, side, G)
    assert np.array_equal(g.cpu().numpy().reshape(gref.shape), gref)
    i64 = oracle.image64(gref)
    got = img.cpu().numpy().reshape(i64.shape)
    for c in range(nch):
        err = np.abs(got[c] - i64[c]).max() / np.abs(i64[c]).max()
        assert err <= 1e-5, (c, err)
    assert np.array_equal(vmax.cpu().numpy(), got.reshape(nch, -1).max(1))
    assert np.array_equal(vmin.cpu().numpy(), got.reshape(nch, -1).min(1))


def test_delta_image_and_context_image(cuda):
    import torch
    pk = _config0_packets(8, seed=21)
    with mixer.ArrayContext(max_heaps=8) as ctx:
        img = torch.zeros(128 * 32 * 32, dtype=torch.float32, device=cuda)
        ctx.correlate(_t(pk, cuda), 8, seq0=0)
        ctx.image(img, delta=True)
        _sync()
        first = img.cpu().numpy().copy()
        ctx.correlate(_t(pk, cuda), 8, seq0=0)
        ctx.image(img, delta=True)                      # change since last image == first
        _sync()
        assert np.array_equal(img.cpu().numpy(), first)
        ctx.image(img, delta=False)                     # integrated == 2 x first
        _sync()
        full = 2 * oracle.correlate(oracle.corner_turn(pk, 256, 128, 32, 8))
        ref = oracle.image64(oracle.grid(full, 16, 32))
        got = img.cpu().numpy().reshape(ref.shape)
        assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()


# ------------------------------------------------- the reference's own GPU kernels

def _ref_v_update(cuda, pk):
    """k_packAB + cgemm_blk_t<false> on one V-update (32 heaps x 256 antennas)."""
    import torch
    if not oracle.ref_gpu_available():
        pytest.skip("oracle/_ref/libref_gpu.so not built")
    ref = oracle.ref_gpu()
    assert ref.ref_const(3) == 32 and ref.ref_const(4) == 1024
    bb = torch.from_numpy(pk.reshape(32 * 256, 8256)[:, 64:].copy()).to(cuda)   # header strip
    planes = [torch.zeros(128 * 256 * 1024, dtype=torch.int8, device=cuda) for _ in range(4)]
    cre = torch.zeros(128 * 256 * 256, dtype=torch.int32, device=cuda)
    cim = torch.zeros_like(cre)
    s = torch.cuda.current_stream().cuda_stream
    assert ref.ref_pack(bb.data_ptr(), *[p.data_ptr() for p in planes], s) == 0
    assert ref.ref_cgemm(0, 256, 256, 1024, 128, *[p.data_ptr() for p in planes], cre.data_ptr(),
                         cim.data_ptr(), s) == 0
    _sync()
    return planes, cre, cim


def test_matches_reference_gpu_kernels(cuda):
    import torch
    pk = _config0_packets(32, seed=2024)
    planes, cre, cim = _ref_v_update(cuda, pk)
    # corner-turn: our re / im planes equal the reference's A planes
    ours = torch.zeros(2 * 128 * 256 * 1024, dtype=torch.int8, device=cuda)
    mixer.corner_turn(_t(pk, cuda), 8256, 64, 256, 128, 32, 32, 0, ours, 1024, 0)
    _sync()
    o = ours.view(2, -1)
    assert torch.equal(o[0], planes[0]) and torch.equal(o[1], planes[1])
    # visibilities: bit-exact against cgemm_blk_t<false> (full square)
    with mixer.ArrayContext(max_heaps=32) as ctx:
        ctx.correlate(_t(pk, cuda), 32, seq0=0)
        v = torch.zeros(128 * 2 * 256 * 256, dtype=torch.int64, device=cuda)
        ctx.read_vis_i64(v, full_square=True)
        _sync()
        v = v.view(128, 2, 256, 256)
        assert torch.equal(v[:, 0], cre.view(128, 256, 256).to(torch.int64))
        assert torch.equal(v[:, 1], cim.view(128, 256, 256).to(torch.int64))


def test_image_matches_reference_publish_path(cuda):
    """k_flush_cube -> k_diff -> k_grid_cube -> cuFFT -> host fftshift (reference)
    against mixer_image on the same V; agreement to float rounding."""
    import torch
    pk = _config0_packets(32, seed=7)
    planes, cre, cim = _ref_v_update(cuda, pk)
    ref = oracle.ref_gpu()
    s = torch.cuda.current_stream().cuda_stream
    vcube = torch.zeros(128 * 2 * 256 * 256, dtype=torch.float32, device=cuda)
    vprev = torch.zeros_like(vcube)
    dv = torch.zeros_like(vcube)
    G = torch.zeros(128 * 32 * 32 * 2, dtype=torch.float32, device=cuda)
    im = torch.zeros_like(G)
    assert ref.ref_flush(vcube.data_ptr(), cre.data_ptr(), cim.data_ptr(), s) == 0
    assert ref.ref_diff(vcube.data_ptr(), vprev.data_ptr(), dv.data_ptr(), vcube.numel(), s) == 0
    assert ref.ref_grid(dv.data_ptr(), G.data_ptr(), s) == 0
    assert ref.ref_fft(G.data_ptr(), im.data_ptr(), s) == 0
    _sync()
    f = im.cpu().numpy().reshape(128, 32, 32, 2)[..., 0]
    ref_img = np.roll(f, (-16, -16), axis=(1, 2))            # host loop at :233
    with mixer.ArrayContext(max_heaps=32) as ctx:
        ctx.correlate(_t(pk, cuda), 32, seq0=0)
        img = torch.zeros(128 * 32 * 32, dtype=torch.float32, device=cuda)
        ctx.image(img)
        _sync()
        got = img.cpu().numpy().reshape(128, 32, 32)
    scale = np.abs(ref_img).max(axis=(1, 2), keepdims=True)
    assert np.all(np.abs(got - ref_img) <= 1e-4 * scale)


# ------------------------------------------- items taken over while a launch runs

@pytest.mark.parametrize("nant,nch,klen", [
    (24, 592, 96),       # 4 items per SM: the last round-robin launch
    (24, 593, 96),       # the first whose CTAs take over the waiting ones' items
    (24, 2000, 256),     # many rounds of short items
    (130, 198, 144),     # ragged tiles among them
])
def test_xcorr_items_taken_over(cuda, nant, nch, klen):
    import torch
    rng = np.random.default_rng(nch)
    planes = _rand_planes(rng, nch, nant, klen)
    ref = oracle.vis_tile_pack(oracle.correlate(planes)).reshape(-1)
    dpl = _t(planes, cuda)
    err = _zeros(1, torch.int32, cuda)
    for mode, dtype, times in ((mixer.VIS_STORE_I32, torch.int32, 1),
                               (mixer.VIS_ACC_I32, torch.int32, 2),
                               (mixer.VIS_ACC_I64, torch.int64, 2)):
        vis = _zeros(ref.size, dtype, cuda)
        for _ in range(2):
            mixer.xcorr_tri(dpl, nant, nch, klen, 0, klen, mode, vis, err)
        _sync()
        assert np.array_equal(vis.cpu().numpy().astype(np.int64), times * ref), mode
    assert int(err.item()) == 0


# ------------------------------------- corner-turn groups that do not divide evenly

@pytest.mark.parametrize("nant,nch,tpkt,nheaps,k0", [
    (3, 5, 16, 1, 0),        # one heap
    (5, 7, 32, 9, 16),       # last group of one heap
    (4, 127, 32, 15, 0),     # last groups of heaps and of channels both short
    (6, 43, 48, 7, 48),      # rows of 12 vectors: the block is no multiple of them
    (2, 3, 4112, 2, 0),      # rows wider than the block (257 vectors)
    (700, 16, 16, 3, 0),     # more CTAs than a short grid
])
def test_corner_turn_remainders(cuda, nant, nch, tpkt, nheaps, k0):
    import torch
    rng = np.random.default_rng(nant)
    stride = 64 + 2 * nch * tpkt
    pk = rng.integers(0, 256, size=nheaps * nant * stride, dtype=np.uint8)
    kt = (k0 + nheaps * tpkt + 16 + 15) // 16 * 16
    planes = torch.full((2, nch, nant, kt), 7, dtype=torch.int8, device=cuda)
    dpk = _t(pk, cuda)
    seq_err = _zeros(1, torch.int32, cuda)
    err = _zeros(1, torch.int32, cuda)
    mixer.restamp_seq(dpk, nheaps * nant, stride, 11)
    mixer.corner_turn(dpk, stride, 64, nant, nch, tpkt, nheaps, 11, planes, kt, k0, seq_err, err)
    mixer.corner_turn(dpk, stride, 64, nant, nch, tpkt, nheaps, 12, planes, kt, k0, seq_err, err)
    _sync()
    got = planes.cpu().numpy()
    ref = oracle.corner_turn(pk, nant, nch, tpkt, nheaps)
    assert np.array_equal(got[:, :, :, k0:k0 + nheaps * tpkt], ref)
    assert np.all(got[:, :, :, :k0] == 7) and np.all(got[:, :, :, k0 + nheaps * tpkt:] == 7)
    assert int(seq_err.item()) == nheaps * nant and int(err.item()) == 0


# ---------------------------------- context calls longer than max_heaps, in chunks

@pytest.mark.parametrize("nheaps", [2, 3, 1024, 1025])   # the planes hold 1024 heaps of 16
@pytest.mark.parametrize("on_device", [True, False])
@pytest.mark.parametrize("i32", [False, True])
def test_context_long_calls(cuda, nheaps, on_device, i32):
    import torch
    nant, nch, tpkt = 5, 3, 16
    stride = 64 + 2 * nch * tpkt
    rng = np.random.default_rng(nheaps)
    pk = torch.from_numpy(rng.integers(0, 256, size=nheaps * nant * stride, dtype=np.uint8)).to(cuda)
    mixer.restamp_seq(pk, nheaps * nant, stride, 7)
    _sync()
    ref = oracle.correlate(oracle.corner_turn(pk.cpu().numpy(), nant, nch, tpkt, nheaps))
    src = pk if on_device else pk.cpu().pin_memory()
    with mixer.ArrayContext(nant=nant, nch=nch, tpkt=tpkt, ksub=tpkt, side_x=3, grid=16,
                            pkt_stride=stride, max_heaps=2) as ctx:
        if i32:
            ctx.correlate_i32(src, nheaps, 7, on_device=on_device)
            ctx.integrate()
        else:
            ctx.correlate(src, nheaps, 7, on_device=on_device)
        out = torch.empty(nch * 2 * nant * nant, dtype=torch.int64, device=cuda)
        ctx.read_vis_i64(out)
        _sync()
        assert np.array_equal(out.cpu().numpy().reshape(ref.shape), ref)
        st = ctx.stats()
        assert st["samples"] == nheaps * tpkt and st["seq_errors"] == 0 and st["kernel_err"] == 0


# ------------------------------------------------ K ranges split over idle SMs

@pytest.mark.parametrize("nant,nch,klen,max_ctas", [
    (40, 1, 384, 0),       # one part of two chunks at most: not split
    (40, 1, 400, 0),       # four chunks, the last one short: two parts
    (60, 7, 1296, 0),      # parts of unequal length
    (70, 74, 512, 0),      # 148 items: two parts a tile
    (70, 75, 512, 0),      # more than half the SMs: not split
    (200, 3, 1280, 0),     # ragged tiles, plain and transposed
    (40, 2, 2048, 7),      # parts bounded by the CTA limit
    (40, 8, 1024, 7),      # one tile behind a round of seven CTAs, too short to split
    (24, 150, 1536, 0),    # two tiles behind a whole round, in two parts of six chunks
    (24, 150, 1408, 0),    # eleven chunks: not split
    (24, 222, 1664, 0),    # 74 tiles behind a round, parts of seven and six chunks
    (130, 200, 1536, 0),   # 600 items and 8 tiles in parts, taken over while they run
])
def test_xcorr_k_parts(cuda, nant, nch, klen, max_ctas):
    import torch
    rng = np.random.default_rng(klen + nch)
    planes = _rand_planes(rng, nch, nant, klen)
    ref = oracle.vis_tile_pack(oracle.correlate(planes)).reshape(-1)
    dpl = _t(planes, cuda)
    err = _zeros(1, torch.int32, cuda)
    for mode, dtype in ((mixer.VIS_STORE_I32, torch.int32), (mixer.VIS_ACC_I32, torch.int32),
                        (mixer.VIS_ACC_I64, torch.int64)):
        vis = torch.full((ref.size,), 5, dtype=dtype, device=cuda)
        mixer.xcorr_tri(dpl, nant, nch, klen, 0, klen, mode, vis, err, max_ctas=max_ctas)
        _sync()
        start = 0 if mode == mixer.VIS_STORE_I32 else 5
        assert np.array_equal(vis.cpu().numpy().astype(np.int64), ref + start), mode
    assert int(err.item()) == 0


# ------------------------------------------------- the stream a call without one uses

def test_default_stream_is_torchs_current(cuda):
    import threading
    import torch
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    seen = {}

    def thread():
        seen["thread"] = mixer._stream(None)
        with torch.cuda.stream(other):
            seen["thread side"] = mixer._stream(None)

    for _ in range(2):      # the first call binds, the second uses it
        assert mixer._stream(None) == torch.cuda.current_stream().cuda_stream
        with torch.cuda.stream(side):
            assert mixer._stream(None) == side.cuda_stream
            t = threading.Thread(target=thread)
            t.start()
            t.join()
    assert seen == {"thread": torch.cuda.default_stream().cuda_stream,
                    "thread side": other.cuda_stream}
    assert mixer._stream(side) == side.cuda_stream and mixer._stream(7) == 7


# ------------------------ dependent launches: captured, forked over streams, replayed

def test_dependent_launches_captured(cuda):
    import torch
    nant, nch, tpkt, nheaps, G = 72, 6, 16, 24, 32
    stride, k = 64 + 2 * nch * tpkt, nheaps * tpkt
    rng = np.random.default_rng(5)
    pk = torch.from_numpy(rng.integers(0, 256, size=nheaps * nant * stride, dtype=np.uint8)).to(cuda)
    n = mixer.vis_elems(nant, nch)

    def buffers():
        return dict(planes=torch.zeros((2, nch, nant, k), dtype=torch.int8, device=cuda),
                    v32=torch.zeros(n, dtype=torch.int32, device=cuda),
                    v64=torch.zeros(n, dtype=torch.int64, device=cuda),
                    dump=torch.zeros((nch, 2, nant, nant), device=cuda),
                    grid=torch.zeros((nch, G, G, 2), dtype=torch.int64, device=cuda),
                    img=torch.zeros((nch, G, G), device=cuda))

    def chain(b, st, side):
        with torch.cuda.stream(st):
            b["v64"].zero_()
            mixer.corner_turn(pk, stride, 64, nant, nch, tpkt, nheaps, 0, b["planes"], k)
            mixer.xcorr_tri(b["planes"], nant, nch, k, 0, k, mixer.VIS_ACC_I32, b["v32"])
            mixer.vis_flush(b["v32"], b["v64"], n)
            mixer.xcorr_tri(b["planes"], nant, nch, k, 0, k, mixer.VIS_ACC_I64, b["v64"])
            side.wait_stream(st)
            mixer.grid(b["v64"], nant, nch, 9, G, b["grid"])
            mixer.image_fft(b["grid"], nch, G, b["img"])
        with torch.cuda.stream(side):
            mixer.vis_dump_f32(b["v64"], nant, nch, b["dump"])
        st.wait_stream(side)

    st, side = torch.cuda.Stream(), torch.cuda.Stream()
    eager, graphed = buffers(), buffers()
    torch.cuda.synchronize()
    chain(eager, st, side)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        chain(graphed, st, side)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    ref = 2 * oracle.correlate(oracle.corner_turn(pk.cpu().numpy(), nant, nch, tpkt, nheaps))
    assert np.array_equal(eager["dump"].cpu().numpy(), ref.astype(np.float32))
    for name in eager:
        assert torch.equal(eager[name], graphed[name]), name


# -------------------------------------------- the forms of the gridding kernel

@pytest.mark.parametrize("nant,side,G,nch,shift", [
    (128, 16, 31, 3, 0),     # one tile, the grid just holds its baselines: written whole
    (128, 16, 30, 3, 0),     # one less: baselines wrap
    (128, 16, 32, 3, 8),     # grids on an 8-byte boundary
    (7, 9, 18, 2, 0),        # array wider than its elements
    (90, 1, 179, 2, 0),      # one column
    (129, 16, 32, 2, 0),     # three tiles
    (130, 12, 32, 197, 0),   # 591 tiles, the last launch with eight loads a thread
    (130, 12, 32, 198, 0),   # 594 tiles
])
def test_grid_forms(cuda, nant, side, G, nch, shift):
    import torch
    rng = np.random.default_rng(nant)
    planes = rng.integers(-128, 128, size=(2, nch, nant, 16), dtype=np.int8)
    full = oracle.correlate(planes)
    vis = _t(oracle.vis_tile_pack(full).reshape(-1), cuda)
    ref = oracle.grid(full, side, G)
    n, off = nch * G * G * 2, shift // 8
    grid = torch.full((n + 2,), 7, dtype=torch.int64, device=cuda)[off:off + n]
    mixer.grid(vis, nant, nch, side, G, grid)
    _sync()
    assert np.array_equal(grid.cpu().numpy().reshape(ref.shape), ref)
    old = rng.integers(-1000, 1000, size=n)
    prev = torch.full((n + 2,), 0, dtype=torch.int64, device=cuda)[off:off + n]
    prev.copy_(_t(old, cuda))
    mixer.grid(vis, nant, nch, side, G, grid, prev)
    _sync()
    assert np.array_equal(grid.cpu().numpy(), ref.reshape(-1) - old)
    assert np.array_equal(prev.cpu().numpy(), ref.reshape(-1))


# ------------------------------------------------------ a context's state zeroed

@pytest.mark.parametrize("i32", [False, True])       # with the int32 cube or without
@pytest.mark.parametrize("nant,nch", [(3, 1), (140, 5), (1000, 20)])   # 190 MB: by memset
def test_context_reset(cuda, nant, nch, i32):
    import torch
    tpkt, nheaps, G = 16, 2, 16
    stride = 64 + 2 * nch * tpkt
    rng = np.random.default_rng(nant)
    pk = torch.from_numpy(rng.integers(0, 256, size=nheaps * nant * stride, dtype=np.uint8)).to(cuda)
    ref = oracle.correlate(oracle.corner_turn(pk.cpu().numpy(), nant, nch, tpkt, nheaps))
    with mixer.ArrayContext(nant=nant, nch=nch, tpkt=tpkt, ksub=tpkt, side_x=32, grid=G,
                            pkt_stride=stride, max_heaps=nheaps) as ctx:
        img = torch.zeros(nch * G * G, device=cuda)
        out = torch.empty(nch * 2 * nant * nant, dtype=torch.int64, device=cuda)
        images = []
        for _ in range(2):              # the second pass starts from what the first left
            if i32:
                ctx.correlate_i32(pk, nheaps, 5)      # left in the int32 cube
            ctx.correlate(pk, nheaps, 5)
            ctx.image(img, delta=True)
            ctx.reset()
            ctx.integrate()
            ctx.read_vis_i64(out)
            _sync()
            assert int(out.abs().max()) == 0
            assert ctx.stats() == {"samples": 0, "seq_errors": 0, "kernel_err": 0}
            ctx.correlate(pk, nheaps, 5)
            ctx.read_vis_i64(out)
            ctx.image(img, delta=True)
            _sync()
            assert np.array_equal(out.cpu().numpy().reshape(ref.shape), ref)
            images.append(img.clone())
        # the delta image starts anew after a reset
        assert torch.equal(images[0], images[1])


# --------------------------- a ragged diagonal tile with both operands from one box

@pytest.mark.parametrize("nant", [16, 17, 33, 50, 65, 81, 97, 112, 144, 200])
@pytest.mark.parametrize("klen", [80, 512, 1152, 1408, 1520, 2480])   # 1 to 20 chunks
def test_xcorr_ragged_diagonal(cuda, nant, klen):
    import torch
    nch = 75 if nant <= 128 else 50       # one item a tile, no K ranges
    rng = np.random.default_rng(nant)
    planes = _rand_planes(rng, nch, nant, klen)
    ref = oracle.vis_tile_pack(oracle.correlate(planes)).reshape(-1)
    dpl = _t(planes, cuda)
    err = _zeros(1, torch.int32, cuda)
    for mode, dtype in ((mixer.VIS_STORE_I32, torch.int32), (mixer.VIS_ACC_I32, torch.int32),
                        (mixer.VIS_ACC_I64, torch.int64)):
        vis = torch.full((ref.size,), 3, dtype=dtype, device=cuda)
        mixer.xcorr_tri(dpl, nant, nch, klen, 0, klen, mode, vis, err)
        _sync()
        start = 0 if mode == mixer.VIS_STORE_I32 else 3
        assert np.array_equal(vis.cpu().numpy().astype(np.int64), ref + start), mode
    assert int(err.item()) == 0


def test_context_gives_long_planes_back(cuda):
    """A buffer made on first use that no longer fits takes the long planes' place."""
    import torch
    nant, nch, tpkt, nheaps = 1000, 20, 16, 2
    stride = 64 + 2 * nch * tpkt
    rng = np.random.default_rng(3)
    pk = torch.from_numpy(rng.integers(0, 256, size=nheaps * nant * stride, dtype=np.uint8)).to(cuda)
    ref = oracle.correlate(oracle.corner_turn(pk.cpu().numpy(), nant, nch, tpkt, nheaps))
    torch.cuda.empty_cache()
    with mixer.ArrayContext(nant=nant, nch=nch, tpkt=tpkt, ksub=tpkt, side_x=32, grid=64,
                            pkt_stride=stride, max_heaps=nheaps) as ctx:
        ctx.correlate(pk, nheaps)
        _sync()
        # leave 100 MB: less than the 160 MB dump, which the 655 MB planes make room for
        fill = torch.empty(max(0, torch.cuda.mem_get_info()[0] - (100 << 20)), dtype=torch.uint8,
                           device=cuda)
        dump = np.zeros(ref.shape, dtype=np.float32)
        ctx.dump(dump, on_device=False)
        _sync()
        assert np.array_equal(dump, ref.astype(np.float32))
        ctx.correlate(pk, nheaps)                      # with the short planes
        ctx.dump(dump, on_device=False)
        _sync()
        assert np.array_equal(dump, (2 * ref).astype(np.float32))
        del fill
    torch.cuda.empty_cache()


# ------------------------------------- context chunks that the corner-turn accepts

def test_context_chunks_of_max_heaps(cuda):
    """One heap more than a long max_heaps: chunks of 131 072 and 1, not two of 65 537."""
    import torch
    nant, nch, tpkt, max_heaps = 1, 1, 16, 131072
    nheaps, stride = max_heaps + 1, 64 + 2 * nch * tpkt
    rng = np.random.default_rng(11)
    pk = torch.from_numpy(rng.integers(0, 256, size=nheaps * nant * stride, dtype=np.uint8)).to(cuda)
    mixer.restamp_seq(pk, nheaps * nant, stride, 3)
    _sync()
    ref = oracle.correlate(oracle.corner_turn(pk.cpu().numpy(), nant, nch, tpkt, nheaps))
    with mixer.ArrayContext(nant=nant, nch=nch, tpkt=tpkt, ksub=tpkt, side_x=1, grid=16,
                            pkt_stride=stride, max_heaps=max_heaps) as ctx:
        ctx.correlate(pk, nheaps, 3)
        out = torch.empty(nch * 2 * nant * nant, dtype=torch.int64, device=cuda)
        ctx.read_vis_i64(out)
        _sync()
        assert np.array_equal(out.cpu().numpy().reshape(ref.shape), ref)
        st = ctx.stats()
        assert st["samples"] == nheaps * tpkt and st["seq_errors"] == 0 and st["kernel_err"] == 0


# ----------------------------- a captured call, after the context gave memory back

def test_captured_correlate_outlives_long_planes(cuda):
    """Replays of a captured call write only to buffers the context still owns."""
    import torch
    nant, nch, tpkt, nheaps = 1000, 20, 16, 5
    stride = 64 + 2 * nch * tpkt
    rng = np.random.default_rng(4)
    pk = torch.from_numpy(rng.integers(0, 256, size=nheaps * nant * stride, dtype=np.uint8)).to(cuda)
    ref = oracle.correlate(oracle.corner_turn(pk.cpu().numpy(), nant, nch, tpkt, nheaps))
    torch.cuda.empty_cache()
    with mixer.ArrayContext(nant=nant, nch=nch, tpkt=tpkt, ksub=tpkt, side_x=32, grid=64,
                            pkt_stride=stride, max_heaps=2) as ctx:
        ctx.correlate(pk, nheaps)                   # through the long planes
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            ctx.correlate(pk, nheaps)
        g.replay()
        _sync()
        # leave 100 MB: the 160 MB dump makes the context give its 655 MB back
        fill = torch.empty(max(0, torch.cuda.mem_get_info()[0] - (100 << 20)), dtype=torch.uint8,
                           device=cuda)
        dump = np.zeros(ref.shape, dtype=np.float32)
        ctx.dump(dump, on_device=False)
        _sync()
        assert np.array_equal(dump, (2 * ref).astype(np.float32))
        room = torch.cuda.mem_get_info()[0] - (100 << 20)
        assert room > 300 << 20                     # where the long planes were
        other = torch.full((room,), 7, dtype=torch.uint8, device=cuda)
        g.replay()
        ctx.correlate(pk, nheaps)                   # in chunks of max_heaps
        ctx.dump(dump, on_device=False)
        _sync()
        assert np.array_equal(dump, (4 * ref).astype(np.float32))
        assert int(other.min()) == 7 and int(other.max()) == 7
        assert ctx.stats()["kernel_err"] == 0
        del fill, other, g
    torch.cuda.empty_cache()


# ------------------------------------------- when a context holds the long planes

def _held(fn):
    """Device memory that a call leaves allocated."""
    import torch
    _sync()
    before = torch.cuda.mem_get_info()[0]
    fn()
    _sync()
    return before - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("i32", [False, True])
def test_context_long_planes_on_first_use(cuda, i32):
    """Calls that do not use them leave no long planes behind; three uneven long chunks."""
    import torch
    nant, nch, tpkt, nheaps, short = 96, 24, 16, 2501, 3     # 75 MB for 1024 heaps
    stride, long_bytes = 64 + 2 * nch * tpkt, 2 * nch * nant * 16384
    rng = np.random.default_rng(nant)
    pk = torch.from_numpy(rng.integers(0, 256, size=nheaps * nant * stride, dtype=np.uint8)).to(cuda)
    mixer.restamp_seq(pk, nheaps * nant, stride, 9)
    _sync()
    host = pk.cpu()

    def ref(n):
        return oracle.correlate(oracle.corner_turn(host[:n * nant * stride].numpy(), nant, nch, tpkt, n))

    with mixer.ArrayContext(nant=nant, nch=nch, tpkt=tpkt, ksub=tpkt, side_x=12, grid=32,
                            pkt_stride=stride, max_heaps=short) as ctx:
        call = ctx.correlate_i32 if i32 else ctx.correlate
        out = torch.empty(nch * 2 * nant * nant, dtype=torch.int64, device=cuda)
        call(pk, 1, 9)                                       # makes the int32 cube
        quiet = [_held(lambda: call(pk, short, 9)),
                 _held(lambda: call(host.pin_memory(), 2 * short, 9, on_device=False))]
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            call(pk, 2 * short, 9)
        quiet.append(_held(g.replay))
        assert max(quiet) < long_bytes // 2, quiet
        ctx.reset()
        assert long_bytes <= _held(lambda: call(pk, nheaps, 9)) < long_bytes + (16 << 20)
        assert _held(lambda: call(pk, 1500, 9)) < long_bytes // 2
        ctx.integrate()
        ctx.read_vis_i64(out)
        _sync()
        expect = ref(nheaps) + ref(1500)
        assert np.array_equal(out.cpu().numpy().reshape(expect.shape), expect)
        assert ctx.stats()["seq_errors"] == 0 and ctx.stats()["kernel_err"] == 0
        del g


def test_context_planes_longer_than_the_long_ones(cuda):
    """max_heaps past 16 384 samples: no second planes."""
    import torch
    nant, nch, tpkt, max_heaps, nheaps = 64, 16, 16, 1025, 2100
    stride = 64 + 2 * nch * tpkt
    rng = np.random.default_rng(nant)
    pk = torch.from_numpy(rng.integers(0, 256, size=nheaps * nant * stride, dtype=np.uint8)).to(cuda)
    ref = oracle.correlate(oracle.corner_turn(pk.cpu().numpy(), nant, nch, tpkt, nheaps))
    with mixer.ArrayContext(nant=nant, nch=nch, tpkt=tpkt, ksub=tpkt, side_x=8, grid=16,
                            pkt_stride=stride, max_heaps=max_heaps) as ctx:
        out = torch.empty(nch * 2 * nant * nant, dtype=torch.int64, device=cuda)
        ctx.correlate(pk, 1)
        ctx.reset()
        assert _held(lambda: ctx.correlate(pk, nheaps)) < 16 << 20
        ctx.read_vis_i64(out)
        _sync()
        assert np.array_equal(out.cpu().numpy().reshape(ref.shape), ref)


def test_context_of_host_packets_holds_no_long_planes(cuda):
    import torch
    nant, nch, tpkt, nheaps = 300, 40, 16, 2
    stride = 64 + 2 * nch * tpkt
    kw = dict(nant=nant, nch=nch, tpkt=tpkt, ksub=tpkt, side_x=20, grid=64, pkt_stride=stride,
              max_heaps=nheaps)
    pk = torch.zeros(nheaps * nant * stride, dtype=torch.uint8).pin_memory()
    first = mixer.ArrayContext(**kw)
    more = []
    try:
        each = _held(lambda: more.append(mixer.ArrayContext(**kw)))
        # cube, planes, grids and image (in blocks of 2 MB), without long planes (393 MB)
        own = mixer.vis_elems(nant, nch) * 8 + 2 * nch * nant * nheaps * tpkt + nch * 64 * 64 * 36
        assert own - (8 << 20) <= each < own + (64 << 20)
        assert _held(lambda: first.correlate(pk, 1, on_device=False)) < 64 << 20
    finally:
        for ctx in [first] + more:
            ctx.close()


@pytest.mark.parametrize("read", ["dump", "read_vis_i64"])
def test_context_host_output_in_pieces(cuda, read):
    """A full square whose device buffer does not fit comes out through a smaller one."""
    import torch
    nant, nch, tpkt, nheaps = 700, 41, 16, 2
    stride = 64 + 2 * nch * tpkt
    rng = np.random.default_rng(8)
    pk = torch.from_numpy(rng.integers(0, 256, size=nheaps * nant * stride, dtype=np.uint8)).to(cuda)
    ref = oracle.correlate(oracle.corner_turn(pk.cpu().numpy(), nant, nch, tpkt, nheaps))
    torch.cuda.empty_cache()
    with mixer.ArrayContext(nant=nant, nch=nch, tpkt=tpkt, ksub=tpkt, side_x=30, grid=64,
                            pkt_stride=stride, max_heaps=nheaps) as ctx:
        ctx.correlate(pk, nheaps)
        warm = torch.empty(nch * 2 * nant * nant, dtype=torch.float32, device=cuda)
        ctx.dump(warm)
        del warm
        torch.cuda.empty_cache()
        _sync()
        # leave 100 MB: less than the square of all 41 channels (161 MB, 321 MB in int64)
        fill = torch.empty(max(0, torch.cuda.mem_get_info()[0] - (100 << 20)), dtype=torch.uint8,
                           device=cuda)
        out = np.zeros(ref.shape, dtype=np.float32 if read == "dump" else np.int64)
        for times in (1, 2):                        # the second through the buffer of the first
            getattr(ctx, read)(out, on_device=False)
            _sync()
            assert np.array_equal(out, (times * ref).astype(out.dtype))
            ctx.correlate(pk, nheaps)
        del fill
    torch.cuda.empty_cache()


def test_context_long_call_beside_a_capture(cuda):
    """The first long call allocates without ending a capture on another stream."""
    import torch
    nant, nch, tpkt, nheaps = 24, 4, 16, 40
    stride = 64 + 2 * nch * tpkt
    rng = np.random.default_rng(6)
    pk = torch.from_numpy(rng.integers(0, 256, size=nheaps * nant * stride, dtype=np.uint8)).to(cuda)
    ref = oracle.correlate(oracle.corner_turn(pk.cpu().numpy(), nant, nch, tpkt, nheaps))
    kw = dict(nant=nant, nch=nch, tpkt=tpkt, ksub=tpkt, side_x=6, grid=16, pkt_stride=stride,
              max_heaps=8)
    with mixer.ArrayContext(**kw) as ctx, mixer.ArrayContext(**kw) as recorded:
        side = torch.cuda.Stream()
        _sync()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            recorded.correlate(pk, nheaps)
            ctx.correlate(pk, nheaps, stream=side)
        g.replay()
        _sync()
        for c in (ctx, recorded):
            out = torch.empty(nch * 2 * nant * nant, dtype=torch.int64, device=cuda)
            c.read_vis_i64(out)
            _sync()
            assert np.array_equal(out.cpu().numpy().reshape(ref.shape), ref)
        del g


# ------------------------- adds beside a next tile that is shorter than their own

@pytest.mark.parametrize("nch,klen", [
    (760, 2048),      # 20 tiles behind five rounds, in parts too short to be paced beside
    (760, 7424),      # parts of nine chunks, the last of four
])
def test_xcorr_paced_before_parts(cuda, nch, klen):
    import torch
    nant = 128
    g = torch.Generator(device=cuda).manual_seed(nch)
    planes = torch.randint(-128, 128, (2, nch, nant, klen), dtype=torch.int8, device=cuda, generator=g)
    n = mixer.vis_elems(nant, nch)
    err = _zeros(1, torch.int32, cuda)
    ref = _zeros(n, torch.int32, cuda)
    mixer.xcorr_tri(planes, nant, nch, klen, 0, klen, mixer.VIS_STORE_I32, ref, err)
    for mode, dtype in ((mixer.VIS_ACC_I32, torch.int32), (mixer.VIS_ACC_I64, torch.int64)):
        vis = torch.full((n,), 5, dtype=dtype, device=cuda)
        mixer.xcorr_tri(planes, nant, nch, klen, 0, klen, mode, vis, err)
        _sync()
        assert torch.equal(vis - 5, ref.to(dtype)), mode
    assert int(err.item()) == 0


def test_batch_items_of_falling_length(cuda):
    import torch
    g = torch.Generator(device=cuda).manual_seed(2)
    shapes = [(128, 300, 2176), (128, 300, 2048), (256, 40, 1024), (128, 200, 128)]
    err = _zeros(1, torch.int32, cuda)
    probs, refs = [], []
    for nant, nch, k in shapes:
        planes = torch.randint(-128, 128, (2, nch, nant, k), dtype=torch.int8, device=cuda, generator=g)
        refs.append(_zeros(mixer.vis_elems(nant, nch), torch.int32, cuda))
        mixer.xcorr_tri(planes, nant, nch, k, 0, k, mixer.VIS_STORE_I32, refs[-1], err)
        probs.append(dict(planes=planes, nant=nant, nch=nch, kt=k, mode=mixer.VIS_ACC_I64,
                          vis=_zeros(mixer.vis_elems(nant, nch), torch.int64, cuda)))
    batch = mixer.Batch(probs)
    for _ in range(3):
        batch.run()
    _sync()
    for prob, ref in zip(probs, refs):
        assert torch.equal(prob["vis"], 3 * ref.to(torch.int64))
    assert int(err.item()) == 0
