"""How a decode step's attention is cut over the chip, against times measured for every cut. The cut is host arithmetic; what the
two ways of merging compute is tested on the GPU (test_parity_gpu.py). At the end the same for when a prompt's attention starts."""
import pytest

# clusters of 1 .. 8 blocks of the decode attention kernel that a B200 of 148 SMs holds at once
RESIDENT = [0, 148, 74, 45, 33, 26, 22, 15, 15]
# us per layer of a decode step (attention, its projections and a narrow feed-forward, 8 layers, graph replay) by head width,
# sequences x 2 kv heads and context: cN = N splits in a cluster, wN = N splits through the workspace
MEASURED = [
    (64, 2, 130, "c1:24.4 c2:25.0"),
    (64, 2, 1024, "c1:28.6 c2:27.4 c3:26.7 c4:26.6 c5:26.4 c6:26.2 c7:26.6 c8:26.7 w16:32.0"),
    (64, 2, 8192, "c1:69.5 c2:46.4 c3:39.6 c4:36.2 c5:34.2 c6:32.8 c7:31.9 c8:31.3 w16:33.9 w24:33.9"),
    (64, 2, 30000, "c1:200.0 c2:113.7 c3:83.9 c4:69.0 c5:59.7 c6:53.4 c7:49.1 c8:46.4 w16:41.8 w24:39.3"),
    (64, 10, 400, "c1:26.8 c2:27.3 c3:27.4 c4:26.7 c5:27.2 c6:27.5"),
    (64, 10, 16384, "c1:127.8 c2:77.1 c3:58.9 c4:50.3 c5:46.1 c6:43.0 c7:41.5 c8:40.0 w7:46.1 w10:42.9 w14:40.7"),
    (64, 10, 30000, "c1:218.1 c2:123.4 c3:90.4 c4:73.8 c5:64.4 c6:57.5 c7:53.4 c8:50.4 w7:58.8 w10:52.1 w14:48.0"),
    (64, 16, 2048, "c1:36.4 c2:32.8 c3:31.0 c4:30.6 c5:30.4 c6:30.0 c7:35.9 c8:35.7 w5:35.0 w6:34.6 w9:34.1"),
    (64, 16, 30000, "c1:226.7 c2:125.8 c3:92.8 c4:75.4 c5:66.4 c6:60.1 c7:84.5 c8:79.0 w5:72.1 w6:66.5 w9:56.5"),
    (64, 32, 400, "c1:28.5 c2:28.8 c3:29.4 c4:28.9 w2:34.0 w3:33.6 w4:33.0"),
    (64, 32, 8192, "c1:77.5 c2:51.7 c3:45.3 c4:42.1 w2:57.9 w3:50.1 w4:46.1"),
    (64, 32, 30000, "c1:227.6 c2:126.2 c3:92.9 c4:77.2 w2:132.9 w3:98.3 w4:81.3"),
    (64, 48, 8192, "c1:81.1 c2:55.9 c3:68.5 w2:60.9 w3:55.4"),
    (64, 64, 4096, "c1:52.6 c2:45.0 w2:49.3"),
    (64, 74, 8192, "c1:90.1 c2:64.9 w2:70.6"),
    (128, 2, 512, "c1:33.7 c2:33.4 c3:32.0 c4:32.0 c5:31.7 c6:31.7 c7:32.0 c8:32.0"),
    (128, 2, 16384, "c1:179.5 c2:106.7 c3:79.9 c4:67.5 c5:60.1 c6:55.6 c7:52.5 c8:49.7 w16:47.7 w24:46.5"),
    (128, 10, 8192, "c1:107.1 c2:69.6 c3:56.4 c4:50.8 c5:47.4 c6:45.0 c7:43.2 c8:42.1 w7:48.7 w10:47.2 w14:46.7"),
    (128, 10, 30000, "c1:326.6 c2:180.1 c3:128.8 c4:104.3 c5:91.1 c6:81.5 c7:76.3 c8:71.5 w7:82.6 w10:72.3 w14:67.6"),
    (128, 16, 16384, "c1:193.2 c2:111.9 c3:85.7 c4:73.4 c5:67.3 c6:62.3 c7:87.8 c8:83.0 w5:73.5 w6:69.2 w9:64.7"),
    (128, 24, 8192, "c1:111.4 c2:73.1 c3:62.1 c4:55.7 c5:52.9 c6:70.1 w3:67.8 w4:62.3 w6:59.4"),
    (128, 32, 8192, "c1:111.0 c2:73.9 c3:63.0 c4:57.9 w2:79.3 w3:68.0 w4:63.8"),
    (128, 64, 1024, "c1:44.9 c2:42.7 w2:47.4"),
    (128, 64, 8192, "c1:115.5 c2:79.0 w2:85.1"),
]


@pytest.mark.parametrize("width,units,ctx,times", MEASURED)
def test_cut_is_near_the_fastest(width, units, ctx, times):
    import tffn
    times = {k: float(v) for k, v in (x.split(":") for x in times.split())}
    heads = 14 if width == 64 else 12
    n, cluster = tffn.attention_cut(units // 2, heads, 2, width, ctx, 148, RESIDENT)
    # over all 198 points of the sweep the rule's choice is at most 3.9 % off the fastest
    assert times[("c" if cluster or n == 1 else "w") + str(n)] <= 1.04 * min(times.values()), (n, cluster)


@pytest.mark.parametrize("units", [1, 2, 3, 7, 15, 16, 22, 23, 33, 34, 74, 75, 148, 149])
@pytest.mark.parametrize("ctx", [1, 31, 129, 1025, 9000, 32768, 1 << 20])
@pytest.mark.parametrize("scratch", [0, 9000, 8 << 20])
def test_cut_fits_the_device_and_its_scratch(units, ctx, scratch):
    import tffn
    for heads, width in ((1, 64), (7, 64), (20, 128)):
        parts = (heads + 7) // 8
        n, cluster = tffn.attention_cut(units, heads, 1, width, ctx, 148, RESIDENT, scratch)
        assert n >= 1 and (n == 1 or n * units * parts <= 148)
        if cluster:
            assert 2 <= n <= 8 and units * parts <= RESIDENT[n]
        elif n > 1:
            assert units * parts * n * min(heads, 8) * (width + 2) <= scratch


@pytest.mark.parametrize("n", [1, 2, 3, 16, 40, 64, 80])
@pytest.mark.parametrize("heads,rank,rot", [(16, 512, 64), (14, 256, 32), (5, 72, 16), (40, 320, 32)])
def test_latent_steps_are_keyed_by_all_that_their_launch_depends_on(n, heads, rank, rot):
    """a step captured with one ring depth is not replayed where the rule asks for the other"""
    import tffn
    cuts = {tffn.latent_attention_cut(n, heads, rank, rot, ctx, 148) for ctx in list(range(1, 12000, 61)) + [32768]}
    assert len({c[3] for c in cuts}) == len({c[:3] for c in cuts}) == len(cuts)
    assert all(c[2] >= 1 and c[0] >= 1 and (not c[1] or c[0] in (2, 4, 8, 16)) for c in cuts)


# whole prompts, us: heads, kv heads, lengths, with the attention started ahead of the kernel before it and behind it
PROMPTS = [
    (14, 2, [1332], 3145, 3144), (14, 2, [1440], 3253, 3206), (14, 2, [720] * 2, 2904, 2921), (14, 2, [360] * 4, 2745, 2782),
    (14, 2, [144] * 10, 2686, 2700), (14, 2, [36] * 40, 2637, 2710), (14, 2, [1600], 3425, 3382), (14, 2, [800] * 2, 3038, 3053),
    (14, 2, [400] * 4, 2872, 2920), (14, 2, [200] * 8, 2815, 2864), (14, 2, [160] * 10, 2793, 2844), (14, 2, [1800], 3720, 3621),
    (14, 2, [900] * 2, 3279, 3256), (14, 2, [600] * 3, 3171, 3157), (14, 2, [450] * 4, 3123, 3149), (14, 2, [300] * 6, 3025, 3069),
    (14, 2, [180] * 10, 2901, 2976), (14, 2, [90] * 20, 2842, 2944), (14, 2, [36] * 50, 2858, 2961), (14, 2, [2016], 3814, 3707),
    (14, 2, [1008] * 2, 3311, 3295), (14, 2, [666] * 3, 3182, 3229), (14, 2, [504] * 4, 3089, 3148), (14, 2, [252] * 8, 2915, 3022),
    (14, 2, [126] * 16, 2867, 2973), (14, 2, [2100], 3963, 3899), (14, 2, [2340], 4205, 4170), (14, 2, [1170] * 2, 3671, 3749),
    (14, 2, [2700], 4669, 4644), (14, 2, [1500, 100, 100, 100], 3537, 3507), (14, 2, [1000, 400, 200, 100, 50], 3108, 3163),
    (14, 2, [1300, 450], 3291, 3281), (14, 2, [700, 500, 300, 200], 2997, 3027), (14, 2, [50, 100, 200, 1400], 3381, 3348),
    (14, 2, [1000, 800], 3290, 3274), (14, 2, [1200, 600], 3354, 3355),
    (12, 2, [1600], 1481, 1465), (12, 2, [2000], 1629, 1578), (12, 2, [1000] * 2, 1491, 1494), (12, 2, [500] * 4, 1429, 1452),
    (12, 2, [250] * 8, 1406, 1427), (12, 2, [126] * 16, 1386, 1408), (12, 2, [2300], 1739, 1699),
]


@pytest.mark.parametrize("heads,kv,lens,ahead,behind", PROMPTS)
def test_prompt_attention_starts_where_it_is_faster(heads, kv, lens, ahead, behind):
    import tffn
    chosen = behind if tffn.prompt_attention_waits(lens, heads, kv, 148) else ahead
    assert chosen <= 1.01 * min(ahead, behind)  # repeated measurements differ by about as much
