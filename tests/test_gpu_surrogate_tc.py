"""The surrogate's tcgen05 inference kernels (cpipe_b200/csrc/surrogate_tc.cu)
against its mma.sync kernels and the CPU oracle.

Both engines take the same BF16 operands and accumulate in FP32; they differ
in the order of the FP32 sums, so an activation on a bfloat16 rounding
boundary can land one bfloat16 ulp apart (in practice the two engines have
agreed bit for bit: both reduce each 16-wide K slice the same way).  Bounds:
PSNR >= 60 dB between the engines and against the oracle (rounded to binary16
like the frames), mean relative error <= 2e-4 between the engines and <= 5e-4
against the oracle (these random networks with a strong last layer amplify the
bfloat16 rounding flips), max <= 1e-2 (relative to max(1, |value|)); alpha
bit-exact; and no bounded wait inside the tcgen05
pipeline ran out (cpipe_surrogate_check)."""
import numpy as np
import oracle_surrogate as O
import os
import pytest
from cpipe_b200 import surrogate as S

pytestmark = pytest.mark.gpu


def close(got, want, what, mean_bound=2e-4):
    d = np.abs(got - want) / np.maximum(1.0, np.abs(want))
    p = 10.0 * np.log10(max(1.0, float(np.max(np.abs(want)))) ** 2 / max(float(np.mean((got - want) ** 2)), 1e-30))
    print(f"{what}: max rel {d.max():.2e}, mean {d.mean():.2e}, PSNR {p:.1f} dB")
    assert d.max() <= 1e-2 and d.mean() <= mean_bound and p >= 60.0, what


def run(sg, engine, x, ab, f16=True):
    n, h, w = x.shape[:3]
    din = S.DeviceArray(x.nbytes).upload(x)
    dout = S.DeviceArray(x.nbytes)
    sg.set_engine(engine)
    sg.denoise(din.ptr, dout.ptr, n, w, h, ab, f16=f16)
    sg.check()
    return dout.download(x.shape, x.dtype).astype(np.float32)


@pytest.mark.parametrize("n,h,w", [(2, 19, 35), (1, 64, 64), (1, 33, 130), (3, 16, 8), (1, 1, 1)])
def test_tcgen05_matches_mma_and_oracle(cuda_device, n, h, w):
    rng = np.random.default_rng(n * 1000 + h * 10 + w)
    x = rng.uniform(0.02, 0.95, (n, h, w, 4)).astype(np.float16)
    ab = np.array([(4e-3, 4e-5), (1e-3, 1e-5), (8e-3, 9e-5)][:n], np.float32)
    params = [(W, (b + rng.normal(0, 0.02, b.shape)).astype(np.float32)) for W, b in S.init_params(n + h)]
    params[-1] = (params[-1][0] * 10.0, params[-1][1])
    sg = S.Surrogate(S.to_blob(params))
    tc = run(sg, "tcgen05", x, ab)
    mma = run(sg, "mma", x, ab)
    np.testing.assert_array_equal(tc[..., 3], x[..., 3].astype(np.float32))
    close(tc[..., :3], mma[..., :3], f"tcgen05 vs mma {n}x{h}x{w}")
    want, _ = O.forward(params, x.astype(np.float32), ab, bf=True)
    want = want.astype(np.float16).astype(np.float64)  # the frames are binary16
    close(tc[..., :3], want, f"tcgen05 vs oracle {n}x{h}x{w}", mean_bound=5e-4)
    sg.close()


# strips of up to 122 columns and CTAs of at least 8 rows: one strip exactly, one column more, three strips, rows
# dealt out across frames and strips, fewer rows than a layer's reach, one row
@pytest.mark.parametrize("n,h,w", [(1, 9, 122), (2, 17, 123), (1, 40, 245), (3, 7, 260), (1, 2, 130), (1, 1, 300),
                                   (1, 301, 5)])
def test_tcgen05_strips_match_mma(cuda_device, n, h, w):
    rng = np.random.default_rng(h * 1000 + w)
    x = rng.uniform(0.02, 0.95, (n, h, w, 4)).astype(np.float16)
    ab = np.array([(4e-3, 4e-5), (1e-3, 1e-5), (8e-3, 9e-5)][:n], np.float32)
    params = [(W, (b + rng.normal(0, 0.02, b.shape)).astype(np.float32)) for W, b in S.init_params(n + h)]
    params[-1] = (params[-1][0] * 10.0, params[-1][1])
    sg = S.Surrogate(S.to_blob(params))
    tc, mma = run(sg, "tcgen05", x, ab), run(sg, "mma", x, ab)
    np.testing.assert_array_equal(tc[..., 3], x[..., 3].astype(np.float32))
    close(tc[..., :3], mma[..., :3], f"tcgen05 vs mma {n}x{h}x{w}")
    sg.close()


# frames of at most 63 columns and more than 1184 rows in all go by bands of rows side by side: just below and above that
# line, two bands to 64 of them (63, 62, 42 .. 1 columns), the widest that fits (63) and the first that does not (64),
# bands that end inside a frame and on the zeros after it, many frames, of one row too
@pytest.mark.parametrize("n,h,w", [(1, 1184, 2), (1, 1185, 2), (600, 1, 20), (3, 431, 62), (1, 2500, 63), (1, 3000, 64),
                                   (2, 1700, 42), (1, 5000, 31), (100, 16, 16), (7, 1300, 16), (1, 9001, 9),
                                   (2, 19000, 2), (1, 76000, 1), (25, 59, 5)])
@pytest.mark.parametrize("f16", [True, False])
def test_tcgen05_bands_match_mma(cuda_device, n, h, w, f16):
    rng = np.random.default_rng(h * 1000 + w)
    x = rng.uniform(0.02, 0.95, (n, h, w, 4)).astype(np.float16 if f16 else np.float32)
    ab = np.tile(np.array([(4e-3, 4e-5), (1e-3, 1e-5), (8e-3, 9e-5)], np.float32), (n // 3 + 1, 1))[:n]
    params = [(W, (b + rng.normal(0, 0.02, b.shape)).astype(np.float32)) for W, b in S.init_params(n + h)]
    params[-1] = (params[-1][0] * 10.0, params[-1][1])
    sg = S.Surrogate(S.to_blob(params))
    tc, mma = run(sg, "tcgen05", x, ab, f16), run(sg, "mma", x, ab, f16)
    np.testing.assert_array_equal(tc[..., 3], x[..., 3].astype(np.float32))
    close(tc[..., :3], mma[..., :3], f"tcgen05 vs mma {n}x{h}x{w}")
    sg.close()


def test_narrow_frames_fill_the_products(cuda_device):
    """A pixel of a 16-column frame costs at most 2.5 times one of a wide frame (a strip of 16 columns in products of
    128 pixels cost six times as much)."""
    sg = S.Surrogate(S.to_blob(S.init_params(1)))
    d = [S.DeviceArray(1200000 * 8), S.DeviceArray(1200000 * 8)]

    def ms(w, h):
        return min(sum(sg.profile(d[0].ptr, d[1].ptr, 1, w, h, [(1e-3, 1e-5)])) for _ in range(5))

    d[0].upload(np.zeros((1200000, 4), np.float16))
    wide, narrow = ms(1200, 1000), ms(16, 75000)
    print(f"1.2 MP: 1200 columns {wide:.3f} ms, 16 columns {narrow:.3f} ms")
    assert narrow <= 2.5 * wide
    sg.close()


def test_profile_reports_what_was_timed(cuda_device):
    """The tcgen05 engine has two kernels: two times.  The mma.sync engine has nine."""
    sg = S.Surrogate(S.to_blob(S.init_params(1)))
    x = np.full((2, 60, 150, 4), 0.5, np.float16)
    d = [S.DeviceArray(x.nbytes).upload(x), S.DeviceArray(x.nbytes)]
    for engine, places in (("tcgen05", [1, 5]), ("mma", list(range(9)))):
        sg.set_engine(engine)
        ms = sg.profile(d[0].ptr, d[1].ptr, 2, 150, 60, [(1e-3, 1e-5)] * 2)
        assert [k for k, v in enumerate(ms) if v != 0.0] == places, (engine, ms)
    sg.close()


def test_workspace_follows_the_engine(cuda_device):
    """Inference on tcgen05 keeps one hidden activation, 64 bytes a pixel; the mma.sync engine's 144 are allocated when
    it is asked for, a training step's too, and each engine's output stays its own."""
    import torch
    w, h = 2048, 2048
    rng = np.random.default_rng(9)
    x = np.tile(rng.uniform(0.02, 0.95, (1, 64, w, 4)), (1, h // 64, 1, 1)).astype(np.float16)
    ab = np.array([(4e-3, 4e-5)], np.float32)
    params = S.init_params(4)
    params[-1] = (params[-1][0] * 10.0, params[-1][1])
    sg = S.Surrogate(S.to_blob(params))
    small = x[:, :16, :16].copy()
    run(sg, "tcgen05", small, ab)  # (the kernels' own setup)
    dev = [S.DeviceArray(x.nbytes).upload(x), S.DeviceArray(x.nbytes)]
    before = torch.cuda.mem_get_info()[0]
    sg.denoise(dev[0].ptr, dev[1].ptr, 1, w, h, ab)
    sg.check()
    used = before - torch.cuda.mem_get_info()[0]
    assert 60 * w * h <= used <= 72 * w * h, used / (w * h)
    tc = dev[1].download(x.shape, x.dtype).astype(np.float32)
    mma = run(sg, "mma", x, ab)
    close(tc[..., :3], mma[..., :3], "after regrowing")
    d16 = S.DeviceArray(small.nbytes).upload(small)
    sg.train_step(d16.ptr, d16.ptr, ab, 1, 16, 16, 0.0, update=False)
    np.testing.assert_array_equal(run(sg, "tcgen05", x, ab), tc)
    sg.close()


def test_tcgen05_float32_frames(cuda_device):
    rng = np.random.default_rng(7)
    x = rng.uniform(0.02, 0.95, (1, 24, 40, 4)).astype(np.float32)
    sg = S.Surrogate(S.to_blob(S.init_params(7)))
    tc = run(sg, "tcgen05", x, [(4e-3, 4e-5)], f16=False)
    mma = run(sg, "mma", x, [(4e-3, 4e-5)], f16=False)
    close(tc[..., :3], mma[..., :3], "f32 frames")
    np.testing.assert_array_equal(tc[..., 3], x[..., 3])
    sg.close()


@pytest.mark.skipif(not os.path.exists(S.DEFAULT_WEIGHTS), reason="no trained weights committed")
def test_tcgen05_trained_network_12mp(cuda_device):
    from cpipe_b200.chain import Chain, ChainConfig
    front = Chain(ChainConfig.full_12mp(stop_after=1))
    cfg = front.config
    x = front.run_host(cfg.make_raw())[None]
    front.close()
    sg = S.Surrogate(S.load_weights())
    ab = [(cfg.noise_a, cfg.noise_b)]
    tc = run(sg, "tcgen05", x, ab)
    mma = run(sg, "mma", x, ab)
    close(tc[..., :3], mma[..., :3], "12 MP trained network")
    sg.close()
