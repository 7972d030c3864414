"""Kernel variants at the sizes where their tiles, remainders and dispatch rules can go wrong, against the CPU oracle."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def oracle_rows(oracle, param, bin_, x):
    m = oracle.Model(param, bin_)
    return np.stack([m.run([xi])[0] for xi in x])


@pytest.mark.parametrize("cin,cout,k,stride,h,w,n", [
    (3, 5, 3, 1, 9, 7, 2),       # single-element loads of both operands, one tile
    (4, 64, 3, 2, 17, 16, 1),    # the narrowest whole pieces, chunk of 36
    (68, 66, 3, 1, 8, 8, 1),     # 612 = three chunks split over blocks, two column tiles, exactly one row tile
    (64, 62, 1, 1, 13, 5, 1),    # 65 rows: one past a tile; columns in pairs but not in fours
    (16, 64, 3, 1, 200, 200, 1), # 128-row tiles
])
def test_fp32_cuda_core_tiles(pkg, oracle, tmp_path, cin, cout, k, stride, h, w, n):
    param, bin_ = pkg.zoo.single_conv(str(tmp_path / "c"), h=h, w=w, cin=cin, cout=cout, k=k, stride=stride, pad=k // 2)
    x = np.random.default_rng(3).uniform(-1, 1, (n, cin, h, w)).astype(np.float32)
    m = pkg.Model(param, bin_, accuracy_mode=pkg.FP32_CUDA)
    got = m.run(x)[0]
    assert rel_l2(got, oracle_rows(oracle, param, bin_, x)) <= 2e-6
    many = m.run(np.concatenate([x] * 5))[0]  # more tiles, the chunks in one block or in several: the same bits
    assert np.array_equal(many[:n], got) and np.array_equal(many[-n:], got)


@pytest.mark.parametrize("m,k,n", [(1, 513, 1), (65, 7, 130), (3, 1001, 1537), (129, 2050, 63)])
def test_fp32_inner_product_of_odd_extents(pkg, oracle, tmp_path, m, k, n):
    param, bin_ = pkg.zoo.inner_product(str(tmp_path / "ip"), k, n)
    x = np.random.default_rng(4).uniform(-1, 1, (m, 1, 1, k)).astype(np.float32)
    want = oracle_rows(oracle, param, bin_, x)
    assert rel_l2(pkg.Model(param, bin_).run(x)[0], want) <= 1e-5
    assert rel_l2(pkg.Model(param, bin_, accuracy_mode=pkg.FP32_CUDA).run(x)[0], want) <= 2e-6


@pytest.mark.parametrize("m,k,n", [(1, 17, 3), (127, 31, 130), (200, 1001, 1537), (2, 4099, 2053), (8, 4097, 2051), (9, 4097, 2051)])
def test_int8_inner_product_of_odd_extents(pkg, oracle, tmp_path, m, k, n):
    """Rows that are no multiple of 16 bytes: padded by the Quantize step, or quantised by the rows kernel (M <= 8)."""
    param, bin_ = pkg.zoo.inner_product(str(tmp_path / "ip"), k, n, int8=True)
    x = np.random.default_rng(5).uniform(-1, 1, (m, 1, 1, k)).astype(np.float32)
    rows = sorted({0, m // 2, m - 1})
    got = pkg.Model(param, bin_).run(x)[0]
    assert np.array_equal(got[rows], oracle_rows(oracle, param, bin_, x[rows]))


@pytest.mark.parametrize("m", [1, 8, 40])
@pytest.mark.parametrize("int8", [False, True])
def test_device_arrays_in_place_at_any_alignment(pkg, tmp_path, m, int8):
    """Aligned caller arrays are read and written in place, others through the edge launches; a handle that meets more
    sets of arrays than it remembers still answers the same."""
    import torch
    k, n = 2048, 4096
    param, bin_ = pkg.zoo.inner_product(str(tmp_path / "ip"), k, n, int8=int8)
    x = np.random.default_rng(6).uniform(-1, 1, (m, 1, 1, k)).astype(np.float32)
    model = pkg.Model(param, bin_)
    want = model.run(x)[0]
    src = torch.from_numpy(x.reshape(-1)).cuda()
    for round_ in range(2):
        for shift_in, shift_out in [(0, 0), (4, 0), (0, 4), (8, 8), (1, 0), (0, 3), (2, 1)]:
            xin = torch.zeros(m * k + 8, device="cuda")
            xin[shift_in:shift_in + m * k] = src
            y = torch.full((m * n + 8,), 7.0, device="cuda")
            model.run_device(m, [xin.data_ptr() + 4 * shift_in], [y.data_ptr() + 4 * shift_out], torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            got = y.cpu().numpy()
            ref = got[shift_out:shift_out + m * n].reshape(m, n)
            if int8 or m > 8:
                assert np.array_equal(ref, want.reshape(m, n))
            else:  # the rows kernel reads fp32 rows in place, bf16 pairs behind an edge launch
                assert rel_l2(ref, want.reshape(m, n)) <= 1e-5
            assert (got[:shift_out] == 7.0).all() and (got[shift_out + m * n:] == 7.0).all()


@pytest.mark.parametrize("mode,int8,k,m", [(0, False, 4096, 1), (0, False, 4096, 8), (0, True, 4096, 8), (2, False, 300, 1), (2, False, 300, 70)])
def test_device_arrays_may_share_memory(pkg, tmp_path, mode, int8, k, m):
    """An output in the memory of an input, wholly and in part: the results of arrays that lie apart."""
    import torch
    param, bin_ = pkg.zoo.inner_product(str(tmp_path / "ip"), k, k, int8=int8)
    model = pkg.Model(param, bin_, accuracy_mode=mode)
    x = np.random.default_rng(15).uniform(-1, 1, (m, 1, 1, k)).astype(np.float32)
    want = model.run(x)[0].reshape(-1)
    src, room = torch.from_numpy(x.reshape(-1)).cuda(), torch.empty(2 * m * k, device="cuda")
    launches = model.launch_count(m)
    for at_in, at_out in [(0, 0), (0, 4 * (k // 8)), (m * k - 4, 0)]:
        for _ in range(10):
            room[at_in:at_in + m * k] = src
            model.run_device(m, [room.data_ptr() + 4 * at_in], [room.data_ptr() + 4 * at_out], torch.cuda.current_stream().cuda_stream)
            got = room[at_out:at_out + m * k].cpu().numpy()
            assert rel_l2(got, want) <= 1e-5 and (not int8 or np.array_equal(got, want))
    assert launches == model.launch_count(m)


@pytest.mark.parametrize("mode", [0, 2])
def test_an_output_may_take_the_memory_of_an_input_that_is_read_again(pkg, tmp_path, mode):
    """Two layers read one flat input and the first one's result lies over it; two results in one array: the last stays."""
    import torch
    k = 1536
    net = pkg.zoo._Net(16)
    net.w.layer("Input", "input", [], ["data"], f"0=1 1=1 2={k}")
    net.w.layer("Split", "split", ["data"], ["a", "b"])
    net.inner_product("ip1", "a", "y1", k, k)
    net.inner_product("ip2", "b", "y2", k, k)
    model = pkg.Model(*net.w.save(str(tmp_path / "two")), accuracy_mode=mode)
    x = np.random.default_rng(17).uniform(-1, 1, (2, k, 1, 1)).astype(np.float32)
    want = [y.reshape(2, k) for y in model.run(x)]
    src, first, second = torch.from_numpy(x.reshape(2, k)).cuda(), torch.empty(2, k, device="cuda"), torch.empty(2, k, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    for _ in range(10):
        first.copy_(src)
        model.run_device(2, [first.data_ptr()], [first.data_ptr(), second.data_ptr()], stream)
        assert rel_l2(first.cpu(), want[0]) <= 1e-5 and rel_l2(second.cpu(), want[1]) <= 1e-5
    model.run_device(2, [src.data_ptr()], [second.data_ptr(), second.data_ptr()], stream)
    assert rel_l2(second.cpu(), want[1]) <= 1e-5


@pytest.mark.parametrize("cin,cout,k,stride,h,w,n", [
    (64, 64, 3, 1, 9, 7, 3),    # tiles that span images
    (32, 37, 1, 1, 5, 11, 2),   # channels in no whole 16-byte pieces
    (8, 3, 3, 2, 33, 16, 1),
    (64, 160, 3, 1, 16, 16, 9),
])
def test_convolution_writes_the_callers_order(pkg, oracle, tmp_path, cin, cout, k, stride, h, w, n):
    """A convolution that is a graph output writes [channel][pixel] order from its epilogue."""
    param, bin_ = pkg.zoo.single_conv(str(tmp_path / "c"), h=h, w=w, cin=cin, cout=cout, k=k, stride=stride, pad=k // 2)
    x = np.random.default_rng(8).uniform(-1, 1, (n, cin, h, w)).astype(np.float32)
    m = pkg.Model(param, bin_)
    assert not any(r["kernel"].startswith("k_nhwc_to_chw") for r in m.profile(n, repeat=1))
    assert rel_l2(m.run(x)[0], oracle_rows(oracle, param, bin_, x)) <= 3e-5


@pytest.mark.parametrize("m", [1, 16, 17, 511, 512])  # inputs of up to 64 KB and results of up to 4 MB go through pinned memory
def test_small_host_arrays_through_pinned_memory(pkg, tmp_path, m):
    import torch
    k, n = 1024, 2048
    param, bin_ = pkg.zoo.inner_product(str(tmp_path / "ip"), k, n)
    model = pkg.Model(param, bin_)
    for seed in range(2):
        x = np.random.default_rng(seed).uniform(-1, 1, (m, 1, 1, k)).astype(np.float32)
        got = model.run(x)[0]
        xd, y = torch.from_numpy(x).cuda(), torch.empty((m, n), device="cuda")
        model.run_device(m, [xd.data_ptr()], [y.data_ptr()], torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert np.array_equal(got.reshape(m, n), y.cpu().numpy())


@pytest.mark.parametrize("h,w,n", [(56, 56, 22), (64, 24, 29), (41, 16, 60)])
def test_patch_resident_convolution_by_default(pkg, tmp_path, monkeypatch, h, w, n):
    """64 -> 64 channels: from four tiles per SM on, where the tiles fit the image, with the bits of the im2col kernel."""
    param, bin_ = pkg.zoo.residual_block(str(tmp_path / "rb"), h=h, w=w, c=64, cout=64)
    x = np.random.default_rng(9).uniform(-1, 1, (n, 64, h, w)).astype(np.float32)
    m = pkg.Model(param, bin_)
    halo = any("tc_conv_halo_kernel:pairs" in r["kernel"] for r in m.profile(n, repeat=1))
    tiles = -(-h // 16) * -(-w // 8)
    assert halo == (n * tiles >= 4 * 148 and h * w >= 0.85 * 128 * tiles)
    got = m.run(x)[0]
    assert np.array_equal(m.run(x[:1])[0], got[:1])
    monkeypatch.setenv("NCNN_B200_HALO", "0")
    assert np.array_equal(pkg.Model(param, bin_).run(x)[0], got)


@pytest.mark.parametrize("cin,cout,k,h,w,many", [
    (512, 80, 3, 7, 7, 30),    # 72 K blocks = 4 chunks; several tiles per image row block, a ragged last column tile
    (328, 24, 5, 5, 9, 3),     # 64-byte operand rows, 275 blocks: chunks that do not divide them
    (1160, 256, 3, 8, 16, 100), # many images: whole tiles that add up the same chunks
    (448, 24, 3, 7, 7, 30),    # 63 blocks of 64 channels: four chunks, the last one short
    (56, 40, 8, 11, 9, 20),    # 128 blocks of 32 channels, the second of every tap half empty
])
def test_deep_convolutions_sum_in_chunks(pkg, oracle, tmp_path, cin, cout, k, h, w, many):
    """The chunks of a deep contraction run side by side for few images and one after the other for many: the same bits."""
    param, bin_ = pkg.zoo.single_conv(str(tmp_path / "c"), h=h, w=w, cin=cin, cout=cout, k=k, stride=1, pad=k // 2)
    x = np.random.default_rng(10).uniform(-1, 1, (many, cin, h, w)).astype(np.float32)
    m = pkg.Model(param, bin_)
    one = m.run(x[:1])[0]
    assert rel_l2(one, oracle_rows(oracle, param, bin_, x[:1])) <= 3e-5
    for n in (2, many):
        for _ in range(2):
            assert np.array_equal(m.run(x[:n])[0][:1], one)


@pytest.mark.parametrize("c,h,n,pairs", [
    (512, 7, 192, True),   # one wave of pair tiles against two of the one-CTA kernel's
    (512, 7, 208, False),  # two against three
    (392, 14, 64, True),   # two against three, operand rows of 64 bytes
])
def test_chunks_on_pairs_of_ctas(pkg, tmp_path, c, h, n, pairs):
    """Deep layers of large batches on CTA pairs, where these win, sum the chunks of a lone image."""
    param, bin_ = pkg.zoo.residual_block(str(tmp_path / "rb"), h=h, w=h, c=c, cout=64)
    x = np.random.default_rng(19).uniform(-1, 1, (n, c, h, h)).astype(np.float32)
    m = pkg.Model(param, bin_)
    kernels = {r["layer"]: r["kernel"] for r in m.profile(n, repeat=1)}
    assert ("tc_gemm2_kernel:pairs" in kernels["conv1"]) == pairs
    got = m.run(x)[0]
    for i in (0, n // 2, n - 1):
        assert np.array_equal(m.run(x[i:i + 1])[0], got[i:i + 1])


@pytest.mark.parametrize("size,n", [(32, 64), (32, 65), (64, 4), (64, 5), (224, 1)])
def test_depthwise_apart_from_the_projection_on_small_maps(pkg, tmp_path, monkeypatch, size, n):
    """Deep blocks on maps of up to 256 pixels run the two layers apart: the bits of a batch that runs them in one kernel."""
    param, bin_ = pkg.zoo.mobilenet_v2(str(tmp_path / "m"), size=size)
    x = np.random.default_rng(11).uniform(-1, 1, (n + 8, 3, size, size)).astype(np.float32)
    m = pkg.Model(param, bin_)
    got = m.run(x[:n])[0]
    assert np.array_equal(m.run(x)[0][:n], got)
    monkeypatch.setenv("NCNN_B200_FUSE_DW", "0")
    monkeypatch.setenv("NCNN_B200_FUSE_EXPAND", "0")
    assert rel_l2(got, pkg.Model(param, bin_).run(x[:n])[0]) <= 1e-5


@pytest.mark.parametrize("hidden,n,apart", [(192, 1, False), (200, 1, True), (200, 2, False)])
def test_depthwise_apart_from_seven_blocks_of_channels(pkg, tmp_path, hidden, n, apart):
    """16x16 pixels are the most; whichever form runs, the bits of the images in a larger batch."""
    param, bin_ = pkg.zoo.inverted_residual(str(tmp_path / "b"), 16, 16, 64, hidden, 64)
    x = np.random.default_rng(18).uniform(-1, 1, (5, 64, 16, 16)).astype(np.float32)
    m = pkg.Model(param, bin_)
    assert any("tc_dw_project" in r["kernel"] for r in m.profile(n, repeat=1)) != apart
    assert np.array_equal(m.run(x[:n])[0], m.run(x)[0][:n])


def test_depthwise_apart_keeps_its_result_while_other_convolutions_split(pkg, oracle, tmp_path, monkeypatch):
    """NCNN_B200_STREAMK=1 splits convolutions through the workspace that holds the depthwise result of small maps: the
    projections behind those depthwise layers must not be split, the others are."""
    param, bin_ = pkg.zoo.mobilenet_v2(str(tmp_path / "m"))
    x = np.random.default_rng(14).uniform(-1, 1, (1, 3, 224, 224)).astype(np.float32)
    monkeypatch.setenv("NCNN_B200_STREAMK", "1")
    m = pkg.Model(param, bin_)
    fused = {r["layer"].split("+")[-1] for r in m.profile(256, repeat=1) if r["layer"].count("+") == 1}
    kernels = {r["layer"]: r["kernel"] for r in m.profile(1, repeat=1)}
    apart = fused & kernels.keys()
    assert any("split" in k for k in kernels.values())
    assert apart and all(kernels[name] == "tc_gemm_kernel<bf16x3>" for name in apart)
    want = oracle_rows(oracle, param, bin_, x)
    for _ in range(20):
        assert rel_l2(m.run(x)[0], want) <= 2e-4


def test_int8_residuals_beyond_the_l2_cache(pkg, tmp_path):
    """165 images: layer 1's fp32 residuals exceed 126 MB and are requested a tile ahead, up to the last, partial tile."""
    param, bin_ = pkg.zoo.resnet18(str(tmp_path / "r"), int8=True, classes=16)
    x = np.random.default_rng(13).uniform(-1, 1, (165, 3, 224, 224)).astype(np.float32)
    m = pkg.Model(param, bin_)
    got = m.run(x)[0]
    for rows in (slice(0, 3), slice(80, 82), slice(162, 165)):
        assert np.array_equal(m.run(x[rows])[0], got[rows])


@pytest.mark.parametrize("cin,cout,k,stride,h,w,n", [
    (64, 64, 3, 1, 56, 56, 2),    # whole tiles
    (64, 48, 3, 1, 9, 13, 3),     # tiles that overhang both ways
    (8, 24, 3, 1, 17, 8, 1),      # one block of channels, most of it zero fill
    (40, 20, 2, 1, 11, 10, 5),    # 64-byte rows, a second block that is a quarter full, rows of 80 bytes out
    (96, 160, 3, 2, 15, 14, 2),   # stride 2 from odd and even columns
    (96, 128, 5, 2, 12, 21, 1),
    (64, 16, 7, 1, 7, 7, 2),      # groups of a filter row
    (256, 256, 3, 1, 14, 14, 40), # more tiles than SMs
    (512, 40, 3, 1, 5, 6, 1),     # chunks on different blocks
    (512, 512, 3, 2, 8, 8, 70),   # and one after the other
    (200, 64, 4, 1, 6, 40, 2),    # an even filter
])
def test_patch_kernel_equals_im2col_kernel(pkg, oracle, tmp_path, monkeypatch, cin, cout, k, stride, h, w, n):
    """Small tiles out of input patches: the same products in the same order as the im2col kernel, so the same bits."""
    param, bin_ = pkg.zoo.single_conv(str(tmp_path / "c"), h=h, w=w, cin=cin, cout=cout, k=k, stride=stride, pad=k // 2)
    x = np.random.default_rng(23).uniform(-1, 1, (n, cin, h, w)).astype(np.float32)
    got = {}
    for level in ("0", "1"):
        monkeypatch.setenv("NCNN_B200_PATCH", level)
        m = pkg.Model(param, bin_)
        got[level] = m.run(x)[0]
        assert any("tc_conv_patch_kernel" in r["kernel"] for r in m.profile(n, repeat=1)) == (level == "1")
        m.close()
    assert np.array_equal(got["1"], got["0"])
    assert rel_l2(got["1"][:1], oracle_rows(oracle, param, bin_, x[:1])) <= 3e-5


@pytest.mark.parametrize("c,cout,h,n", [(64, 96, 15, 2), (128, 64, 7, 9), (96, 32, 10, 3)])
def test_patch_kernel_with_residuals(pkg, tmp_path, monkeypatch, c, cout, h, n):
    """bf16-pair results and residuals of tiles that overhang the image."""
    param, bin_ = pkg.zoo.residual_block(str(tmp_path / "rb"), h=h, w=h, c=c, cout=cout)
    x = np.random.default_rng(24).uniform(-1, 1, (n, c, h, h)).astype(np.float32)
    monkeypatch.setenv("NCNN_B200_PATCH", "1")
    m = pkg.Model(param, bin_)
    got = m.run(x)[0]
    kernels = {r["layer"]: r["kernel"] for r in m.profile(n, repeat=1)}
    assert "tc_conv_patch_kernel" in kernels["conv1"] and "tc_conv_patch_kernel" in kernels["conv2"]
    monkeypatch.setenv("NCNN_B200_PATCH", "0")
    assert np.array_equal(pkg.Model(param, bin_).run(x)[0], got)


def test_patch_kernel_waits_that_run_out(pkg, tmp_path, monkeypatch):
    """A first patch that never comes: the bounded waits give up, the call answers 7, the handle recovers."""
    param, bin_ = pkg.zoo.single_conv(str(tmp_path / "c"), h=20, w=20, cin=128)
    x = np.random.default_rng(25).uniform(-1, 1, (1, 128, 20, 20)).astype(np.float32)
    m = pkg.Model(param, bin_)
    assert any("tc_conv_patch_kernel" in r["kernel"] for r in m.profile(1, repeat=1))
    good = m.run(x)[0].copy()
    monkeypatch.setenv("NCNN_B200_TEST_STALL", "1")
    with pytest.raises(pkg.NcnnB200Error) as err:
        m.run(x)
    assert err.value.status == 7
    monkeypatch.delenv("NCNN_B200_TEST_STALL")
    assert np.array_equal(m.run(x)[0], good)
    m.check_status()


@pytest.mark.parametrize("switch,net,n", [
    ("NCNN_B200_PATCH", "conv128", 1),
    ("NCNN_B200_HALO", "conv64", 22),
    ("NCNN_B200_CONV_I8", "resnet18", 16),
])
def test_an_empty_switch_is_no_switch(pkg, tmp_path, monkeypatch, switch, net, n):
    path = str(tmp_path / net)
    files = (pkg.zoo.single_conv(path, h=20, w=20, cin=128) if net == "conv128" else
             pkg.zoo.residual_block(path, h=56, w=56, c=64, cout=64) if net == "conv64" else
             pkg.zoo.resnet18(path, int8=True, classes=8))
    used = []
    for value in (None, "", "0"):
        if value is not None:
            monkeypatch.setenv(switch, value)
        used.append([r["kernel"] for r in pkg.Model(*files).profile(n, repeat=1)])
    assert used[1] == used[0] and used[2] != used[0]


@pytest.mark.parametrize("m,k,n,int8", [
    (9, 1472, 24, False),    # 23 K blocks: whole
    (9, 1728, 24, False),    # 27: the shallowest in chunks, one narrow tile column
    (100, 2048, 1000, False),
    (128, 3000, 40, False),  # a last K block and a last chunk that are not full
    (129, 1536, 72, False),
    (129, 1792, 72, False),  # a second tile of one row
    (384, 1600, 136, False),
    (384, 1984, 136, False),
    (385, 1600, 136, False),
    (385, 1984, 136, False), # past the line
    (3, 4096, 80, True),
    (256, 3600, 48, True),
    (12, 3584, 2000, True),
])
def test_inner_product_of_few_rows_in_chunks(pkg, oracle, tmp_path, m, k, n, int8):
    """Chunks of K on different blocks, added by whichever finishes last: the same bits call after call; int8 exact."""
    param, bin_ = pkg.zoo.inner_product(str(tmp_path / "ip"), k, n, int8=int8)
    x = np.random.default_rng(26).uniform(-1, 1, (m, 1, 1, k)).astype(np.float32)
    model = pkg.Model(param, bin_)
    got = model.run(x)[0]
    for _ in range(20):
        assert np.array_equal(model.run(x)[0], got)
    rows = sorted({0, m // 2, m - 1})
    want = oracle_rows(oracle, param, bin_, x[rows]).reshape(got[rows].shape)
    if int8:
        assert np.array_equal(got[rows], want)
    else:
        assert rel_l2(got[rows], want) <= 3e-5


@pytest.mark.parametrize("k,n", [
    (1472, 1000),  # 23 K blocks: whole in every call
    (1664, 1000),  # 26: the deepest of these
    (1728, 1000),  # 27: in chunks
    (1792, 1000),
    (2048, 1000),
    (4094, 520),   # a last K block that is not full
    (2816, 2816),
])
def test_inner_product_sums_alike_whatever_the_rows_of_a_tile(pkg, tmp_path, k, n):
    """Chunks of K follow from the layer: a row has the bits that it has among 128; where nothing is cut, those of any call."""
    param, bin_ = pkg.zoo.inner_product(str(tmp_path / "ip"), k, n)
    most = 400 if k <= 1664 else 128
    x = np.random.default_rng(27).uniform(-1, 1, (most, 1, 1, k)).astype(np.float32)
    model = pkg.Model(param, bin_)
    want = model.run(x)[0]
    first = 9 if 4 * k * n >= 8 << 20 else 1  # (up to eight rows of such weights take the rows kernel)
    for m in (first, 16, 32, 33, 64, 65, 100, 127, 128, 384):
        if m <= most:
            assert np.array_equal(model.run(x[:m])[0], want[:m]), m


@pytest.mark.parametrize("h,w,c,stride,pad,act,n", [
    (7, 7, 960, 1, 1, "clip", 18),     # bf16 pairs for the 1x1 layer behind it
    (7, 7, 960, 1, 1, "", 18),
    (5, 3, 512, 1, 0, "relu", 140),    # one column of results, no padding
    (4, 9, 512, 1, 2, "clip", 36),     # two columns and rows of zeros on each side
    (15, 14, 512, 2, 1, "clip", 33),   # stride 2, the last column is the last of its pair
    (8, 9, 640, 2, 0, "", 60),
    (9, 11, 512, 2, 2, "relu", 43),
    (1, 1, 992, 1, 1, "clip", 70),
    (6, 5, 36, 1, 1, "relu", 612),     # channels that no tensor-core layer takes as bf16 pairs: plain results only
])
def test_depthwise_by_columns(pkg, oracle, tmp_path, monkeypatch, h, w, c, stride, pad, act, n):
    """Many images take the kernel that walks down columns; few take the tile kernel: the same bits, and the oracle's values."""
    monkeypatch.setenv("NCNN_B200_FUSE_DW", "0")
    for tail in ((False, True) if c % 32 == 0 else (False,)):
        net = pkg.zoo._Net(31 + h)
        net.w.layer("Input", "input", [], ["data"], f"0={w} 1={h} 2={c}")
        top = "d" if act or tail else "output"
        net.depthwise("dw", "data", top, c, 3, stride, pad)
        if act:
            top, bottom = ("a" if tail else "output"), top
            if act == "relu":
                net.w.layer("ReLU", "act", [bottom], [top], "0=0.0")
            else:
                net.w.layer("Clip", "act", [bottom], [top], "0=-0.25 1=0.75")
        if tail:
            net.conv("project", top, "output", c, 32, 1, 1, 0, act=0, zero_bias=False)
        param, bin_ = net.w.save(str(tmp_path / f"m{int(tail)}"))
        x = np.random.default_rng(h * w + c).uniform(-2, 2, (n, c, h, w)).astype(np.float32)
        model = pkg.Model(param, bin_)
        kinds = lambda m: [r["kernel"] for r in model.profile(m, 1) if "depthwise" in r["kernel"]]
        assert kinds(n) == ["k_depthwise3x3_columns"] and kinds(2) == ["k_depthwise3x3_tile"]
        got = model.run(x)[0]
        assert np.array_equal(got[-2:], model.run(x[-2:])[0])
        assert rel_l2(got[0], oracle.Model(param, bin_).run([x[0]])[0]) <= (1e-4 if tail else 1e-6)


@pytest.mark.parametrize("h,w,cin", [(1, 1, 64), (1, 7, 96), (3, 3, 32), (7, 9, 64), (8, 8, 40), (5, 13, 64), (11, 11, 64), (8, 16, 64)])
def test_lone_tile_of_few_pixels(pkg, tmp_path, monkeypatch, h, w, cin):
    """A tile that is alone brings only the rows it has (1 to 128 of them): the bits of the same image in front of others."""
    monkeypatch.setenv("NCNN_B200_PATCH", "0")
    param, bin_ = pkg.zoo.single_conv(str(tmp_path / "c"), h=h, w=w, cin=cin, cout=72, k=1, stride=1, pad=0)
    x = np.random.default_rng(h * w).uniform(-1, 1, (300 // (h * w) + 2, cin, h, w)).astype(np.float32)
    model = pkg.Model(param, bin_)
    assert any(r["kernel"].startswith("tc_gemm_kernel") for r in model.profile(1, 1))
    want = model.run(x)[0]
    assert np.array_equal(model.run(x[:1])[0], want[:1])
    assert rel_l2(want, pkg.Model(param, bin_, accuracy_mode=pkg.FP32_CUDA).run(x)[0]) <= 3e-5


@pytest.mark.parametrize("m", [1, 7, 8, 9, 63, 64, 65, 121, 128])
@pytest.mark.parametrize("k,n", [(1001, 130), (512, 64)])
def test_lone_tile_of_few_int8_rows(pkg, oracle, tmp_path, m, k, n):
    param, bin_ = pkg.zoo.inner_product(str(tmp_path / "ip"), k, n, int8=True)
    x = np.random.default_rng(m).uniform(-1, 1, (m, 1, 1, k)).astype(np.float32)
    got = pkg.Model(param, bin_).run(x)[0]
    ref = oracle.Model(param, bin_)
    for i in sorted({0, m // 2, m - 1}):
        assert np.array_equal(got[i], ref.run([x[i]])[0])


@pytest.mark.parametrize("m,k,n", [
    (1, 2048, 1000),
    (33, 2048, 1000),
    (128, 3000, 40),   # a last K block and a last chunk that are not full, one narrow tile column
    (129, 3000, 700),  # a second tile of one row
    (300, 2048, 512),
    (300, 2816, 2816),
    (100, 3600, 48),
])
def test_chunks_in_one_cta_change_no_bit_of_an_inner_product(pkg, tmp_path, monkeypatch, m, k, n):
    """NCNN_B200_SPLIT_K=0 puts the chunks of a tile one after the other; the sums stay what they are."""
    param, bin_ = pkg.zoo.inner_product(str(tmp_path / "ip"), k, n)
    x = np.random.default_rng(28).uniform(-1, 1, (m, 1, 1, k)).astype(np.float32)
    want = pkg.Model(param, bin_).run(x)[0]
    monkeypatch.setenv("NCNN_B200_SPLIT_K", "0")
    assert np.array_equal(pkg.Model(param, bin_).run(x)[0], want)


@pytest.mark.parametrize("m,k,n", [
    (200, 3000, 700),   # chunks on different CTAs
    (300, 2816, 2816),  # one after the other
    (129, 2048, 2048),
    (384, 4096, 1000),
    (384, 1728, 1000),
])
def test_inner_product_of_two_and_three_tiles_of_rows(pkg, tmp_path, m, k, n):
    """Wherever its chunks run, a row has the bits that it has in a call of one tile."""
    param, bin_ = pkg.zoo.inner_product(str(tmp_path / "ip"), k, n)
    x = np.random.default_rng(29).uniform(-1, 1, (m, 1, 1, k)).astype(np.float32)
    model = pkg.Model(param, bin_)
    assert np.array_equal(model.run(x)[0][m - 128:], model.run(x[m - 128:])[0])


def _int8_pair(zoo, prefix, cin, mid, cout, k, h, w, act):
    """Two int8 Convolutions in a row: the first writes int8 (term 101), the second fp32."""
    net = zoo._Net(41, int8=True)
    net.w.layer("Input", "input", [], ["data"], f"0={w} 1={h} 2={cin}")
    net.conv("a", "data", "x", cin, mid, k, 1, k // 2, act=act, zero_bias=False, term=101)
    net.conv("b", "x", "output", mid, cout, k, 1, k // 2, zero_bias=False, term=1)
    return net.w.save(prefix)


@pytest.mark.parametrize("cin,mid,cout,k,h,w,act,n", [
    (64, 64, 64, 3, 16, 8, 1, 1),      # one whole tile
    (64, 80, 48, 3, 17, 9, 1, 3),      # tiles that overhang both ways, rows that are no multiple of 64 bytes
    (48, 96, 16, 3, 33, 20, 0, 2),     # a channel block that is three quarters full; results below zero
    (80, 128, 128, 3, 28, 28, 1, 21),  # 128-byte rows, a filter that leaves room for few patches, more tiles than SMs
    (192, 64, 272, 3, 15, 7, 0, 2),    # two channel blocks; several column blocks, the last one narrower
    (256, 256, 256, 3, 7, 7, 1, 40),   # four column blocks of all taps of two channel blocks
    (64, 64, 64, 2, 11, 12, 1, 2),     # filters that are no 3x3
    (128, 48, 64, 5, 13, 16, 0, 2),
])
def test_int8_convolution_with_its_filter_resident(pkg, oracle, tmp_path, monkeypatch, cin, mid, cout, k, h, w, act, n):
    """Whole-number sums: the same bits as the im2col kernel and the oracle."""
    param, bin_ = _int8_pair(pkg.zoo, str(tmp_path / "c"), cin, mid, cout, k, h, w, act)
    x = np.random.default_rng(42).uniform(-1, 1, (n, cin, h, w)).astype(np.float32)
    got = {}
    for level in ("0", "1"):
        monkeypatch.setenv("NCNN_B200_CONV_I8", level)
        m = pkg.Model(param, bin_)
        got[level] = m.run(x)[0]
        kernels = {r["layer"]: r["kernel"] for r in m.profile(n, repeat=1)}
        assert ("tc_conv_i8_kernel" in kernels["a"]) == (level == "1")
        m.close()
    assert np.array_equal(got["1"], got["0"])
    assert np.array_equal(got["1"][-1:], oracle_rows(oracle, param, bin_, x[-1:]))


@pytest.mark.parametrize("size,n", [(64, 5), (97, 2), (224, 20)])
def test_int8_network_with_resident_filters(pkg, oracle, tmp_path, monkeypatch, size, n):
    """fp32 residuals and results with one or two int8 copies, tiles that overhang; by default (None) on the layers it suits."""
    param, bin_ = pkg.zoo.resnet18(str(tmp_path / "r8"), int8=True, size=size, classes=40)
    x = np.random.default_rng(size).uniform(-1, 1, (n, 3, size, size)).astype(np.float32)
    got, used = {}, {}
    for level in ("0", "1", None):
        if level is None:
            monkeypatch.delenv("NCNN_B200_CONV_I8")
        else:
            monkeypatch.setenv("NCNN_B200_CONV_I8", level)
        m = pkg.Model(param, bin_)
        got[level] = m.run(x)[0]
        used[level] = sum("tc_conv_i8_kernel" in r["kernel"] for r in m.profile(n, repeat=1))
        m.close()
    assert used["0"] == 0 and used["1"] == 13 and used[None] > 0
    assert np.array_equal(got["1"], got["0"]) and np.array_equal(got[None], got["0"])
    assert np.array_equal(got["1"][:1], oracle_rows(oracle, param, bin_, x[:1]))


@pytest.mark.parametrize("cin,n", [
    (256, 2),   # two channel blocks, one tile to a CTA
    (64, 21),   # more tiles than CTAs
])
def test_int8_resident_filters_waits_that_run_out(pkg, tmp_path, monkeypatch, cin, n):
    """A first patch that never comes, in the one tensor-core kernel of the net: the waits give up, the call answers 7, the
    handle recovers."""
    net = pkg.zoo._Net(44, int8=True)
    net.w.layer("Input", "input", [], ["data"], f"0=28 1=28 2={cin}")
    net.conv("a", "data", "x", cin, 64, 3, 1, 1, act=1, zero_bias=False, term=1)
    net.w.layer("Pooling", "gap", ["x"], ["output"], "0=1 4=1")
    monkeypatch.setenv("NCNN_B200_CONV_I8", "1")
    m = pkg.Model(*net.w.save(str(tmp_path / "c")))
    x = np.random.default_rng(45).uniform(-1, 1, (n, cin, 28, 28)).astype(np.float32)
    assert [r["kernel"] for r in m.profile(n, repeat=1) if r["kernel"].startswith("tc_")] == ["tc_conv_i8_kernel<i8>"]
    good = m.run(x)[0].copy()
    monkeypatch.setenv("NCNN_B200_TEST_STALL", "1")
    with pytest.raises(pkg.NcnnB200Error) as err:
        m.run(x)
    assert err.value.status == 7
    monkeypatch.delenv("NCNN_B200_TEST_STALL")
    assert np.array_equal(m.run(x)[0], good)
    m.check_status()


@pytest.mark.parametrize("n,pays", [(74, True), (75, False)])
def test_int8_filters_of_128_channels_stay_resident_for_few_fp32_tiles(pkg, tmp_path, n, pays):
    """fp32 results, with a residual or not: up to four tiles of 16 x 8 pixels an SM; int8 results on either side."""
    param, bin_ = pkg.zoo.resnet18(str(tmp_path / "r8"), int8=True, classes=8)
    kernels = {r["layer"]: r["kernel"] for r in pkg.Model(param, bin_).profile(n, repeat=1)}
    for layer in ("l2b0_conv2", "l2b1_conv2"):
        assert ("tc_conv_i8_kernel" in kernels[layer]) == pays
    assert "tc_conv_i8_kernel" in kernels["l2b1_conv1"] and "tc_conv_i8_kernel" in kernels["l1b1_conv2"]


@pytest.mark.parametrize("m,k,n", [
    (1, 7, 5),       # one short chunk, most lanes without a column
    (3, 1001, 33),   # an odd K: its last pair is half there; one column past a block
    (8, 512, 64),    # whole chunks
    (9, 257, 31),    # two chunks, the second one shorter
    (16, 4097, 515), # as many rows as a warp takes, seventeen chunks
    (17, 300, 70),   # a second group of one row
    (128, 130, 40),  # as many rows as a call may have
    (1, 513, 20512), # 641 blocks of columns of three chunks
    (17, 1001, 10272), # 642 in two groups of rows
])
def test_fp32_inner_product_of_few_rows(pkg, oracle, tmp_path, monkeypatch, m, k, n):
    """A pass over the weights sums in the tiles' chunks and order: the same bits, so more rows change none."""
    param, bin_ = pkg.zoo.inner_product(str(tmp_path / "ip"), k, n)
    x = np.random.default_rng(43).uniform(-1, 1, (m, 1, 1, k)).astype(np.float32)
    model = pkg.Model(param, bin_, accuracy_mode=pkg.FP32_CUDA)
    got = model.run(x)[0]
    assert any(r["kernel"] == "k_rows_f32" for r in model.profile(m, repeat=1))
    many = model.run(np.concatenate([x] * (128 // m + 1)))[0]  # more rows than the kernel takes
    assert np.array_equal(many[:m], got) and np.array_equal(many[-m:], got)
    monkeypatch.setenv("NCNN_B200_ROWS_F32", "0")
    tiles = pkg.Model(param, bin_, accuracy_mode=pkg.FP32_CUDA)
    assert np.array_equal(tiles.run(x)[0], got)
    assert not any(r["kernel"] == "k_rows_f32" for r in tiles.profile(m, repeat=1))
    assert rel_l2(got, oracle_rows(oracle, param, bin_, x)) <= 2e-6


@pytest.mark.parametrize("m,k,n,takes", [
    (16, 300, 12000, True),    # one group of rows, always
    (17, 300, 12000, False),   # more: many columns of short chunks that come in whole pieces
    (48, 513, 7000, False),
    (48, 1001, 2501, True),    # operands of the tiles come element by element
    (128, 1001, 600, True),
    (129, 1001, 600, False),
])
def test_which_fp32_inner_products_are_a_pass_over_the_weights(pkg, tmp_path, m, k, n, takes):
    model = pkg.Model(*pkg.zoo.inner_product(str(tmp_path / "ip"), k, n), accuracy_mode=pkg.FP32_CUDA)
    assert any(r["kernel"] == "k_rows_f32" for r in model.profile(m, repeat=1)) == takes


def _one_launch(pkg, tmp_path, int8):
    """An InnerProduct whose call is one launch of the rows kernel, which goes to the caller's stream without a graph."""
    model = pkg.Model(*pkg.zoo.inner_product(str(tmp_path / "ip"), 4096, 2048, int8=int8))
    x = np.random.default_rng(51).uniform(-1, 1, (7, 1, 1, 4096)).astype(np.float32)
    want = np.stack([model.run(xi[None])[0].reshape(-1) for xi in x])
    assert model.launch_count(1) == 1
    return model, x.reshape(7, 4096), want


@pytest.mark.parametrize("int8", [False, True])
def test_one_launch_follows_what_precedes_it_on_the_stream(pkg, tmp_path, int8):
    """The input is written just before the call and again just after it; the result is read just after it."""
    import torch
    model, x, want = _one_launch(pkg, tmp_path, int8)
    source, busy, stream = torch.from_numpy(x).cuda(), torch.rand(1 << 25, device="cuda"), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        row, y, got = torch.zeros(4096, device="cuda"), torch.zeros(2048, device="cuda"), []
        for _ in range(5):
            for i in range(len(x)):
                busy.mul_(1.0)
                row.copy_(source[i])
                model.run_device(1, [row.data_ptr()], [y.data_ptr()], stream.cuda_stream)
                row.fill_(9.0)
                got.append(y.clone())
                y.fill_(5.0)
    stream.synchronize()
    assert np.array_equal(torch.stack(got).cpu().numpy(), np.concatenate([want] * 5))


@pytest.mark.parametrize("int8", [False, True])
def test_one_launch_with_arrays_in_turn(pkg, tmp_path, int8):
    """Back to back, each call's input the array that the call before wrote into; more sets of arrays than a plan remembers."""
    import torch
    model, x, want = _one_launch(pkg, tmp_path, int8)
    stream = torch.cuda.current_stream().cuda_stream
    xs, ys = torch.from_numpy(x).cuda(), torch.zeros(len(x), 2048, device="cuda")
    for order in (range(7), (0, 1) * 8, (6, 0, 5, 1, 4, 2, 3), range(7)):
        ys.zero_()
        for i in order:
            model.run_device(1, [xs[i].data_ptr()], [ys[i].data_ptr()], stream)
        used = sorted(set(order))
        assert np.array_equal(ys.cpu().numpy()[used], want[used])
    square = pkg.Model(*pkg.zoo.inner_product(str(tmp_path / "sq"), 4096, 4096, int8=int8))
    first = square.run(x[0].reshape(1, 1, 4096))[0].reshape(-1)
    second = square.run(first.reshape(1, 1, 4096))[0].reshape(-1)
    a, b, c = xs[0].clone(), torch.zeros(4096, device="cuda"), torch.zeros(4096, device="cuda")
    for _ in range(20):
        square.run_device(1, [a.data_ptr()], [b.data_ptr()], stream)
        square.run_device(1, [b.data_ptr()], [c.data_ptr()], stream)
    assert np.array_equal(b.cpu().numpy(), first) and np.array_equal(c.cpu().numpy(), second)


@pytest.mark.parametrize("int8", [False, True])
def test_one_launch_under_the_callers_capture(pkg, tmp_path, int8):
    """Captured between two kernels of the caller's; new values in the arrays for every replay, also after the pass was dropped."""
    import torch
    model, x, want = _one_launch(pkg, tmp_path, int8)
    source = torch.from_numpy(x).cuda()
    half, row, y, z = (torch.zeros(n, device="cuda") for n in (4096, 4096, 2048, 2048))
    model.run_device(1, [row.data_ptr()], [y.data_ptr()], torch.cuda.current_stream().cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        torch.mul(half, 2.0, out=row)
        model.run_device(1, [row.data_ptr()], [y.data_ptr()], torch.cuda.current_stream().cuda_stream)
        z.copy_(y)
    for i in range(len(x)):
        torch.mul(source[i], 0.5, out=half)  # (exact)
        graph.replay()
        assert np.array_equal(z.cpu().numpy(), want[i])
        other = torch.zeros(2048, device="cuda")
        model.run_device(1, [source[i].data_ptr()], [other.data_ptr()], torch.cuda.current_stream().cuda_stream)
        assert np.array_equal(other.cpu().numpy(), want[i])


@pytest.mark.parametrize("h,c,stride,n,kernel", [
    (32, 96, 1, 44, "tile"),       # 16 896 threads of the columns kernel with 32 rows each
    (32, 96, 1, 64, "columns"),    # 24 576
    (56, 96, 2, 71, "tile"),       # a third of a wave at stride 2
    (56, 96, 2, 223, "columns"),   # 0.99 of one
    (56, 96, 2, 250, "tile"),      # one and a ninth
    (28, 96, 2, 143, "columns"),   # short walks: as at stride 1
])
def test_depthwise_columns_where_they_are_faster(pkg, oracle, tmp_path, monkeypatch, h, c, stride, n, kernel):
    monkeypatch.setenv("NCNN_B200_FUSE_DW", "0")
    net = pkg.zoo._Net(7)
    net.w.layer("Input", "input", [], ["data"], f"0={h} 1={h} 2={c}")
    net.depthwise("dw", "data", "output", c, 3, stride, 1)
    param, bin_ = net.w.save(str(tmp_path / "m"))
    x = np.random.default_rng(n).uniform(-2, 2, (n, c, h, h)).astype(np.float32)
    model = pkg.Model(param, bin_)
    assert [r["kernel"] for r in model.profile(n, 1) if "depthwise" in r["kernel"]] == ["k_depthwise3x3_" + kernel]
    got = model.run(x)[0]
    assert rel_l2(got[-1], oracle.Model(param, bin_).run([x[-1]])[0]) <= 1e-6
