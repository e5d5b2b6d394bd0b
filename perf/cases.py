"""The calls this framework is used for, as cases that can be timed and compared.

Every case goes through the package's public entry points exactly as a program
would call them: the inputs, the context / batch object and (for a search) the
candidate list are what the program holds before the call; one pass is one
call with its results read back.

  kind      entry points                                        in real use
  pair      Ssimulacra2.compute_* + get_result                  the drop-in: one pair scored and waited for
  maps      Ssimulacra2.compute_linear + error_maps             a heat map of where an image differs
  batch     Ssim2Batch.submit + results                         frames of a video, or a corpus of images
  search    Ssim2Batch.set_reference + submit_with_reference    an encoder trying qualities against one original
  host      Ssim2Batch.submit_host + results                    frames that a CPU decoder left in pinned memory
  dssim     Dssim.compute_sync                                  the sibling metric on its own
  zensim    Zensim.set_reference + compute_with_reference       feature extraction for a quality model

Sizes: the images of the synthetic workloads of this repository (512x512,
1920x1080 NV12, uneven sRGB8 in [64, 2048], 3840x2160 10-bit RGB), a thumbnail,
and odd sizes between them.  Pictures are smooth gratings and noise; the
distorted side is 8x8 DCT quantisation, or blur and noise for 10-bit RGB.
"""
import importlib
import math

import numpy as np
import torch

tmb = importlib.import_module("turbo-metrics_b200")

#: kind -> the most scale-0 pixels (of one image, over all pairs of a pass) that a drawn case takes
MOST = {"pair": 1920 * 1080, "maps": 1920 * 1080, "batch": 64 * 1920 * 1080, "search": 16 * 1920 * 1080,
        "host": 16 * 1920 * 1080, "dssim": 1920 * 1080, "zensim": 2 * 1920 * 1080}


def listed():
    return [
        # the smallest call: one thumbnail; launches and latency are all of it
        {"name": "pair_srgb8_96x64", "kind": "pair", "fmt": "srgb8", "w": 96, "h": 64, "blur": "fir", "rule": "cpu"},
        # the drop-in call of a video tool: one 1080p frame pair at a time
        {"name": "pair_nv12_1080p", "kind": "pair", "fmt": "nv12", "w": 1920, "h": 1080, "blur": "fir", "rule": "cpu"},
        # the mode that reproduces the reference's own f32 recursion, for who compares against old scores
        {"name": "pair_iir_ref_1280x853", "kind": "pair", "fmt": "srgb8", "w": 1280, "h": 853, "blur": "iir_ref",
         "rule": "all6"},
        # linear float input of odd size, and the full-size error maps of it
        {"name": "maps_linear_1023x769", "kind": "maps", "fmt": "linear_f32", "w": 1023, "h": 769, "rule": "min8"},
        # the headline: 64 1080p frame pairs in one submission
        {"name": "batch_nv12_1080p_x64", "kind": "batch", "fmt": "nv12", "w": 1920, "h": 1080, "n": 64, "uneven": False,
         "metrics": "ssimulacra2"},
        # a corpus of images, every one of its own size
        {"name": "batch_uneven_srgb8_x64", "kind": "batch", "fmt": "srgb8", "w": 2048, "h": 2048, "n": 64,
         "uneven": True, "metrics": "ssimulacra2"},
        # 4K HDR frames
        {"name": "batch_rgb16_4k_x4", "kind": "batch", "fmt": "rgb16", "w": 3840, "h": 2160, "n": 4, "uneven": False,
         "metrics": "ssimulacra2"},
        # 10-bit video scored with both metrics from one preparation
        {"name": "batch_both_p016_720p_x16", "kind": "batch", "fmt": "p016", "w": 1280, "h": 720, "n": 16,
         "uneven": False, "metrics": "both"},
        # a quality search: one photo, 12 encodes of it
        {"name": "search_srgb8_1367x911_x12", "kind": "search", "fmt": "srgb8", "w": 1367, "h": 911, "n": 12},
        # frames in host memory, uploaded and scored
        {"name": "host_nv12_1080p_x16", "kind": "host", "fmt": "nv12", "w": 1920, "h": 1080, "n": 16},
        # DSSIM of one photo
        {"name": "dssim_srgb8_1600x1067", "kind": "dssim", "fmt": "srgb8", "w": 1600, "h": 1067},
        # features of one 1080p original against two encodes
        {"name": "zensim_srgb8_1080p_x2", "kind": "zensim", "fmt": "srgb8", "w": 1920, "h": 1080, "n": 2},
    ]


def draw(rng):
    kind = rng.choice(["pair", "pair", "maps", "batch", "batch", "batch", "search", "host", "dssim", "zensim"])
    fmt = {"pair": ["srgb8", "nv12", "rgb16", "p016", "linear_f32"], "maps": ["linear_f32"],
           "batch": ["nv12", "srgb8", "rgb16", "p016"], "search": ["srgb8", "nv12"], "host": ["nv12", "srgb8"],
           "dssim": ["srgb8"], "zensim": ["srgb8"]}[kind]
    case = {"kind": kind, "fmt": rng.choice(fmt)}
    side = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    w, h = side(64, 3840), side(64, 2160)
    while w * h > MOST[kind]:
        w, h = side(64, 3840), side(64, 2160)
    if case["fmt"] in ("nv12", "p016"):
        w, h = w & ~1, h & ~1
    case.update(w=w, h=h)
    if kind in ("pair", "maps"):
        case["rule"] = rng.choice(["cpu", "min8", "all6"])
    if kind == "pair":
        case["blur"] = "iir_ref" if rng.random() < 0.25 and w * h <= 1280 * 853 else "fir"
    if kind in ("batch", "search", "host", "zensim"):
        # at most 2 1080p reads per pass of the both-metrics kind as of the listed one
        both = kind == "batch" and rng.random() < 0.33
        most = MOST[kind] // 8 if both else MOST[kind]
        top = max(1, min({"batch": 64, "search": 16, "host": 16, "zensim": 3}[kind], most // (w * h)))
        case["n"] = int(round(math.exp(rng.uniform(0.0, math.log(top)))))
        if kind == "batch":
            case["uneven"] = case["fmt"] == "srgb8" and case["n"] > 1 and rng.random() < 0.6
            case["metrics"] = "both" if both else "ssimulacra2"
    return case


# --------------------------------------------------------------------------
# pictures
# --------------------------------------------------------------------------

def sizes(case):
    """(w, h) of each pair of a pass; an uneven batch spreads them over [64, w] x [64, h]."""
    n = case.get("n", 1)
    if not case.get("uneven"):
        return [(case["w"], case["h"])] * n
    rng = np.random.RandomState(1000 + n)
    lo = lambda v: min(64, v)  # noqa: E731
    return [(int(rng.randint(lo(case["w"]), case["w"] + 1)), int(rng.randint(lo(case["h"]), case["h"] + 1)))
            for _ in range(n)]


def _dct8():
    k, n = np.arange(8)[:, None], np.arange(8)[None, :]
    d = np.sqrt(2.0 / 8.0) * np.cos(np.pi * (2 * n + 1) * k / 16.0)
    d[0, :] = np.sqrt(1.0 / 8.0)
    return torch.tensor(d, dtype=torch.float32, device="cuda")


def _picture(gen, channels, h, w):
    """(channels, h, w) float32 in [0, 1]: four gratings a channel and a little noise."""
    r = torch.rand((channels, 4, 3), generator=gen, device="cuda")
    y = torch.arange(h, device="cuda", dtype=torch.float32)[None, :, None]
    x = torch.arange(w, device="cuda", dtype=torch.float32)[None, None, :]
    out = torch.full((channels, h, w), 0.5, device="cuda")
    for k in range(4):
        angle, period, phase = r[:, k, 0] * math.pi, 4 * 16 ** r[:, k, 1], r[:, k, 2] * 2 * math.pi
        fx, fy = torch.cos(angle) * 2 * math.pi / period, torch.sin(angle) * 2 * math.pi / period
        out += 0.11 * torch.sin(fx[:, None, None] * x + fy[:, None, None] * y + phase[:, None, None])
    out += 0.06 * (torch.rand((channels, h, w), generator=gen, device="cuda") - 0.5)
    return out.clamp_(0, 1)


def _quantised(p, step):
    """`p` (channels, h, w) in [0, 1] after 8x8 DCT quantisation with `step` / 255."""
    c, h, w = p.shape
    ph, pw = -h % 8, -w % 8
    q = torch.nn.functional.pad(p[None], (0, pw, 0, ph), mode="replicate")[0]
    d = _dct8()
    b = q.reshape(c, (h + ph) // 8, 8, (w + pw) // 8, 8).transpose(2, 3)
    s = step / 255.0
    b = d.T @ (torch.round(d @ b @ d.T / s) * s) @ d
    return b.transpose(2, 3).reshape(c, h + ph, w + pw)[:, :h, :w].clamp(0, 1)


def _distorted(gen, p, fmt, index):
    if fmt == "rgb16":
        k = torch.tensor([0.06, 0.24, 0.4, 0.24, 0.06], device="cuda")
        q = torch.nn.functional.pad(p[None], (2, 2, 2, 2), mode="replicate")[0]
        q = sum(k[i] * q[:, i:i + p.shape[1], :] for i in range(5))
        q = sum(k[i] * q[:, :, i:i + p.shape[2]] for i in range(5))
        return (q + 0.008 * torch.randn(q.shape, generator=gen, device="cuda")).clamp(0, 1)
    return _quantised(p, (4, 8, 16, 32)[index % 4])


def _rows(p, scale):
    """(channels, h, w) in [0, 1] as (h, w, channels) whole numbers up to `scale`."""
    v = torch.round(p.permute(1, 2, 0) * scale).to(torch.int32)
    return v.to(torch.uint8 if scale == 255 else torch.int16).contiguous()


def _yuv(gen, w, h, index, fmt):
    """A 4:2:0 pair: ((y, uv), (y, uv)), BT.709 limited range; 16-bit samples are 10-bit ones shifted up."""
    luma, chroma = _picture(gen, 1, h, w), 0.3 + 0.4 * _picture(gen, 2, h // 2, w // 2)
    pair = []
    for img in range(2):
        a = _distorted(gen, luma, fmt, index) if img else luma
        b = _distorted(gen, chroma, fmt, index) if img else chroma
        if fmt == "nv12":
            y, uv = torch.round(16 + 219 * a[0]).to(torch.uint8), torch.round(16 + 224 * b).to(torch.uint8)
        else:
            y = (torch.round(64 + 876 * a[0]).to(torch.int32) << 6).to(torch.int16)
            uv = (torch.round(64 + 896 * b).to(torch.int32) << 6).to(torch.int16)
        pair.append((y.contiguous(), uv.permute(1, 2, 0).reshape(h // 2, w).contiguous()))
    return pair


def _pair(gen, w, h, fmt, index):
    """One pair as the entry points take it: (reference, distorted), each a tuple of planes."""
    if fmt in ("nv12", "p016"):
        return _yuv(gen, w, h, index, fmt)
    ref = _picture(gen, 3, h, w)
    dis = _distorted(gen, ref, fmt, index)
    if fmt == "linear_f32":
        return [(p.permute(1, 2, 0).pow(2.2).contiguous(),) for p in (ref, dis)]
    return [(_rows(p, 255 if fmt == "srgb8" else 1023),) for p in (ref, dis)]


def _inputs(case, seed):
    """Every pair of the case on the GPU; a search or feature case has one reference and n distorted images."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1_000_003 * (int(seed) + 1))
    if case["kind"] not in ("search", "zensim"):
        return [_pair(gen, w, h, case["fmt"], i) for i, (w, h) in enumerate(sizes(case))]
    first = _pair(gen, case["w"], case["h"], case["fmt"], 0)
    pairs = [first]
    for i in range(1, case["n"]):
        planes = []
        for p in first[0]:  # another encode of the same original
            if case["fmt"] == "srgb8":
                q = _quantised(p.permute(2, 0, 1).float() / 255, 3.0 * (i + 1))
                planes.append(_rows(q, 255))
            else:
                q = _quantised(p[None].float() / 255, 3.0 * (i + 1))
                planes.append(torch.round(q[0] * 255).to(torch.uint8).contiguous())
        pairs.append((first[0], tuple(planes)))
    return pairs


# --------------------------------------------------------------------------
# the calls
# --------------------------------------------------------------------------

def prepare(case, seed):
    pairs = _inputs(case, seed)
    kind, w, h = case["kind"], case["w"], case["h"]
    state = {"case": case, "pairs": pairs}
    if kind in ("pair", "maps"):
        state["call"] = tmb.Ssimulacra2(w, h, blur=case.get("blur", "fir"), scale_rule=case["rule"])
    elif kind in ("batch", "search", "host"):
        pixels = sum(a * b for a, b in sizes(case))
        state["call"] = tmb.Ssim2Batch(len(pairs), pixels)
        if case.get("metrics") == "both":
            state["call"].set_metrics(("ssimulacra2", "dssim"))
        if kind == "host":
            state["pairs"] = [[tuple(p.cpu().pin_memory() for p in img) for img in pair] for pair in pairs]
    elif kind == "dssim":
        state["call"] = tmb.Dssim(w, h)
    else:
        state["call"] = tmb.Zensim(w, h)
    return state


def _descs(case, pairs):
    fmt = case["fmt"]
    if fmt in ("nv12", "p016"):
        return [tmb.PairDesc(r[0], d[0], fmt, r[1], d[1]) for r, d in pairs]
    return [tmb.PairDesc(r[0], d[0], fmt) for r, d in pairs]


def _read(results, dssim=False):
    out = {"score": np.array([r[0] for r in results]), "stats": np.stack([r[1] for r in results]),
           "sums": np.stack([r[2] for r in results]), "scales": np.array([r[3] for r in results]),
           "status": np.array([r[4] for r in results])}
    if dssim:
        out["dssim"] = np.array([r[5] for r in results])
        out["dssim_scale"] = np.stack([r[6] for r in results])
    return out


def run(state):
    case, pairs, call = state["case"], state["pairs"], state["call"]
    kind, fmt = case["kind"], case["fmt"]
    ref, dis = pairs[0]
    if kind in ("pair", "maps"):
        if fmt == "srgb8":
            call.compute_srgb(ref[0], dis[0])
        elif fmt == "nv12":
            call.compute_nv12(ref[0], ref[1], dis[0], dis[1])
        elif fmt == "p016":
            call.compute_p016(ref[0], ref[1], dis[0], dis[1])
        elif fmt == "rgb16":
            call.compute_rgb16(ref[0], dis[0], bits=10)
        else:
            call.compute_linear(ref[0], dis[0])
        score, stats, sums = call.get_result()
        out = {"score": score, "stats": stats, "sums": sums}
        if kind == "maps":
            out["maps"] = call.error_maps(0)
        return out
    if kind == "batch":
        call.submit(_descs(case, pairs))
        return _read(call.results(), case["metrics"] == "both")
    if kind == "host":
        call.submit_host(_descs(case, pairs))
        return _read(call.results())
    if kind == "search":
        if fmt == "nv12":
            call.set_reference(ref[0], fmt, ref_uv=ref[1])
            call.submit_with_reference([d[0] for _, d in pairs], fmt, dis_uv=[d[1] for _, d in pairs])
        else:
            call.set_reference(ref[0], fmt)
            call.submit_with_reference([d[0] for _, d in pairs], fmt)
        return _read(call.results())
    if kind == "dssim":
        return {"dssim": call.compute_sync(ref[0], dis[0])}
    call.set_reference(ref[0])
    return {"features": np.stack([call.compute_with_reference(d[0]) for _, d in pairs])}


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------

def work(case):
    """bytes: every input sample read once, the results written once.  flops: per pixel of an image's pyramid
    the colour conversion and cube roots (~90), per pixel and channel of a pair the four (FIR) or five
    (recursion) blurred planes in two directions and the error maps; DSSIM's 38 3x3 blurs; zensim's box sums."""
    fmt, kind = case["fmt"], case["kind"]
    per = {"srgb8": 3, "nv12": 1.5, "p016": 3, "rgb16": 6, "linear_f32": 12}[fmt]
    px = sum(a * b for a, b in sizes(case))
    n = case.get("n", 1)
    images = px + case["w"] * case["h"] if kind in ("search", "zensim") else 2 * px
    pyramid = 4.0 / 3.0
    if kind == "zensim":
        return {"bytes": images * per + 228 * 8 * n, "flops": images * 90 + px * 3 * pyramid * (4 * 15 + 60)}
    dssim = px * pyramid * (38 * 17 + 60) + images * pyramid * 60
    if kind == "dssim":
        return {"bytes": images * per + 8, "flops": dssim}
    blur = 5 * 2 * 15 if case.get("blur") == "iir_ref" else 4 * 2 * 14
    flops = images * pyramid * 90 + px * pyramid * 3 * (blur + 40)
    out = n * (1 + 108 + 108) * 8
    if kind == "maps":
        out += px * 9 * 4
        flops += px * 3 * (blur + 40)
    if case.get("metrics") == "both":
        flops += dssim
        out += n * 6 * 8
    return {"bytes": images * per + out, "flops": flops}


# --------------------------------------------------------------------------
# the same values in 64 bits, from the definitions of the metrics
# --------------------------------------------------------------------------

#: the reference's sRGB8 -> linear table (it defines the conversion)
LUT = """
    0 0.000303526991 0.000607053982 0.000910581031 0.00121410796 0.00151763496 0.00182116206 0.00212468905
    0.00242821593 0.00273174304 0.00303526991 0.00334653561 0.00367650692 0.00402471703 0.00439144205
    0.00477695325 0.00518151699 0.00560539169 0.00604883255 0.00651209103 0.00699541019 0.00749903172
    0.00802319217 0.00856812485 0.00913405698 0.00972121768 0.010329823 0.0109600937 0.0116122449 0.012286487
    0.0129830306 0.0137020806 0.0144438436 0.0152085144 0.0159962922 0.0168073755 0.0176419523 0.0185002182
    0.0193823613 0.0202885624 0.0212190095 0.0221738834 0.0231533647 0.0241576303 0.0251868572 0.0262412224
    0.0273208916 0.0284260381 0.0295568425 0.0307134502 0.0318960398 0.0331047736 0.0343398117 0.0356013253
    0.0368894525 0.0382043757 0.0395462476 0.0409152098 0.0423114225 0.0437350422 0.0451862141 0.0466650948
    0.0481718332 0.0497065745 0.0512694679 0.0528606549 0.0544802807 0.0561284944 0.0578054339 0.0595112406
    0.061246071 0.0630100295 0.0648032799 0.0666259527 0.068478182 0.0703601092 0.0722718611 0.0742135793
    0.0761853904 0.0781874284 0.0802198276 0.0822827145 0.0843762159 0.0865004659 0.0886556059 0.0908417329
    0.093058981 0.0953074843 0.0975873619 0.0998987406 0.102241747 0.104616493 0.107023112 0.109461717
    0.111932434 0.114435382 0.116970696 0.119538449 0.122138813 0.124771863 0.127437726 0.13013652 0.132868364
    0.135633364 0.138431653 0.141263321 0.144128501 0.147027299 0.149959818 0.152926177 0.155926496 0.158960864
    0.16202943 0.165132239 0.168269455 0.171441153 0.17464745 0.177888468 0.181164294 0.184475034 0.187820807
    0.191201717 0.194617867 0.198069349 0.201556295 0.205078766 0.208636895 0.212230787 0.215860531 0.219526231
    0.223227978 0.226965889 0.23074007 0.234550655 0.238397658 0.242281199 0.246201396 0.25015837 0.254152179
    0.258182913 0.262250721 0.266355664 0.270497859 0.274677366 0.278894335 0.283148795 0.287440896 0.291770697
    0.296138316 0.300543845 0.304987371 0.309468955 0.313988745 0.318546832 0.323143244 0.327778131 0.332451582
    0.337163657 0.341914445 0.346704096 0.351532698 0.356400251 0.361306876 0.366252691 0.371237785 0.376262218
    0.381326109 0.386429518 0.391572565 0.396755308 0.401977867 0.407240301 0.412542701 0.417885154 0.423267752
    0.428690553 0.434153706 0.439657241 0.445201248 0.450785846 0.456411064 0.462077051 0.467783839 0.473531544
    0.479320228 0.48514998 0.491020888 0.496933043 0.502886593 0.50888145 0.514917791 0.520995677 0.527115345
    0.533276618 0.539479673 0.54572469 0.552011609 0.558340609 0.56471169 0.571125031 0.577580631 0.58407861
    0.590619028 0.597202003 0.603827536 0.610495746 0.617206752 0.623960555 0.630757332 0.637597024 0.644479871
    0.651405811 0.658374965 0.665387452 0.67244333 0.679542601 0.686685443 0.693872035 0.701102138 0.70837605
    0.715693772 0.723055363 0.730461001 0.737910688 0.745404482 0.752942443 0.76052475 0.768151402 0.775822461
    0.783538043 0.791298151 0.799102962 0.806952477 0.814846814 0.822785974 0.830770075 0.838799238 0.846873462
    0.854992807 0.863157392 0.871367335 0.879622579 0.887923181 0.89626956 0.904661357 0.913098991 0.921582043
    0.93011117 0.938685894 0.947306871 0.955973506 0.964686573 0.973445475 0.982250869 0.991102219 1
"""

#: the weights of the 108 statistics
WEIGHTS = """
    0 0.0007376606707406586 0 0 0.0007793481682867309 0 0 0.0004371155730107379 0 1.1041726426657346
    0.00066284834129271 0.00015231632783718752 0 0.0016406437456599754 0 1.8422455520539298 11.441172603757666
    0 0.0007989109436015163 0.000176816438078653 0 1.8787594979546387 10.94906990605142 0 0.0007289346991508072
    0.9677937080626833 0 0.00014003424285435884 0.9981766977854967 0.00031949755934435053 0.0004550992113792063
    0 0 0.0013648766163243398 0 0 0 0 0 7.466890328078848 0 17.445833984131262 0.0006235601634041466 0 0
    6.683678146179332 0.00037724407979611296 1.027889937768264 225.20515300849274 0 0 19.213238186143016
    0.0011401524586618361 0.001237755635509985 176.39317598450694 0 0 24.43300999870476 0.28520802612117757
    0.0004485436923833408 0 0 0 34.77906344483772 44.835625328877896 0 0 0 0 0 0 0 0 0.0008680556573291698 0 0
    0 0 0 0.0005313191874358747 0 0.00016533814161379112 0 0 0 0 0 0.0004179171803251336 0.0017290828234722833
    0 0.0020827005846636437 0 0 8.826982764996862 23.19243343998926 0 95.1080498811086 0.9863978034400682
    0.9834382792465353 0.0012286405048278493 171.2667255897307 0.9807858872435379 0 0 0 0.0005130064588990679 0
    0.00010854057858411537
"""

#: the recursive Gaussian of sigma 1.5 in closed form: taps 0..4 of a symmetric 9-tap filter, zero padding
TAPS = [0.26462110548819856, 0.2129285920104222, 0.1093353727774603, 0.036011114658364374, 0.009414367809653656]


def _table():
    return torch.tensor([float(np.float32(v)) for v in LUT.split()], dtype=torch.float64, device="cuda")


def _eotf(v):
    alpha = 1.0 + 5.5 * 0.018053968510807
    high = ((v + (alpha - 1.0)) / alpha).clamp_min(0.0) ** (20.0 / 9.0)
    return torch.where(v >= 0.08124285829863521110029445797874, high, v / 4.5)


def _xyz_of(r, g, b, white):
    cols = np.array([[x / y, 1.0, (1 - x - y) / y] for x, y in (r, g, b)]).T
    x, y = white
    return cols * np.linalg.solve(cols, np.array([x / y, 1.0, (1 - x - y) / y]))[None, :]


_WHITE = (0.3127, 0.3290)


def _m709():
    return _xyz_of((0.64, 0.33), (0.30, 0.60), (0.15, 0.06), _WHITE)


def _linear64(planes, fmt):
    """(3, h, w) float64 linear RGB of one image."""
    if fmt == "linear_f32":
        return planes[0].cuda().double().permute(2, 0, 1)
    if fmt == "srgb8":
        return _table()[planes[0].cuda().long()].permute(2, 0, 1)
    if fmt == "rgb16":
        v = (planes[0].cuda().to(torch.int32) & 0xffff).double() / 1023.0
        m = np.linalg.solve(_m709(), _xyz_of((0.708, 0.292), (0.170, 0.797), (0.131, 0.046), _WHITE))
        return torch.einsum("kc,hwc->khw", torch.tensor(m, device="cuda"), _eotf(v)).clamp_min(0.0)
    bits = 8 if fmt == "nv12" else 16
    y, uv = ((p.cuda().to(torch.int32) & ((1 << bits) - 1)).double() for p in planes)
    kr, kb = _m709()[1, 0], _m709()[1, 2]
    kg = 1.0 - kr - kb
    luma_range, chroma_range = 219 << (bits - 8), 224 << (bits - 8)
    luma = (y.clamp_min(16 << (bits - 8)) - (16 << (bits - 8))) / luma_range
    c = (uv - (1 << (bits - 1))) / chroma_range
    up = lambda p: p.repeat_interleave(2, 0).repeat_interleave(2, 1)  # noqa: E731
    cb, cr = up(c[:, 0::2]), up(c[:, 1::2])
    r = luma + 2 * (1 - kr) * cr
    g = luma - 2 * (1 - kb) * kb / kg * cb - 2 * (1 - kr) * kr / kg * cr
    b = luma + 2 * (1 - kb) * cb
    return _eotf(torch.stack([r, g, b])).clamp(0.0, 1.0)


def _half(p, w, h):
    """2x2 mean of (c, sh, sw) to (c, h, w), source indexes clamped."""
    sh, sw = p.shape[1:]
    y, x = torch.arange(h, device="cuda") * 2, torch.arange(w, device="cuda") * 2
    y0, y1, x0, x1 = y.clamp_max(sh - 1), (y + 1).clamp_max(sh - 1), x.clamp_max(sw - 1), (x + 1).clamp_max(sw - 1)
    a, b = p[:, y0], p[:, y1]
    return (a[:, :, x0] + a[:, :, x1] + b[:, :, x0] + b[:, :, x1]) * 0.25


_F = lambda v: float(np.float32(v))  # noqa: E731
_BIAS = _F(0.0037930734)


def _opsin(lin):
    m = [[_F(0.30), 1 - _F(0.078) - _F(0.30), _F(0.078)], [_F(0.23), 1 - _F(0.078) - _F(0.23), _F(0.078)],
         [_F(0.24342269), _F(0.20476745), 1 - _F(0.24342269) - _F(0.20476745)]]
    v = torch.einsum("kc,chw->khw", torch.tensor(m, dtype=torch.float64, device="cuda"), lin) + _BIAS
    v = v.clamp_min(0.0) ** (1.0 / 3.0) - _BIAS ** (1.0 / 3.0)
    y = 0.5 * (v[0] + v[1])
    return torch.stack([0.5 * (v[0] - v[1]) * 14.0 + 0.42, y + 0.01, v[2] - y + 0.55])


def _blur9(p):
    for dim in (1, 2):
        n = p.shape[dim]
        q = torch.nn.functional.pad(p, (0, 0, 4, 4) if dim == 1 else (4, 4))
        p = sum(TAPS[abs(k - 4)] * q.narrow(dim, k, n) for k in range(9))
    return p


def _error_maps64(ref, dis):
    """(channel, map, h, w) of two XYB planes sets of one scale."""
    m1, m2 = _blur9(ref), _blur9(dis)
    s11, s22, s12 = _blur9(ref * ref) - m1 * m1, _blur9(dis * dis) - m2 * m2, _blur9(ref * dis) - m1 * m2
    num_s = 2 * s12 + 0.0009
    d = (1 - (1 - (m1 - m2) ** 2) * num_s / (s11 + s22 + 0.0009)).clamp_min(0.0)
    e = (1 + (dis - m2).abs()) / (1 + (ref - m1).abs()) - 1
    return torch.stack([d, e.clamp_min(0.0), (-e).clamp_min(0.0)], 1)


def _scales(w, h, rule):
    dims, n = [(w, h)], 1
    while len(dims) < 6:
        dims.append(((dims[-1][0] + 1) // 2, (dims[-1][1] + 1) // 2))
    if rule == "all6":
        return dims
    while n < 6 and min(dims[n if rule == "min8" else n - 1]) >= 8:
        n += 1
    return dims[:n]


def _ssimulacra2(ref, dis, rule, maps=False):
    stats, sums, first = np.zeros(108), np.zeros(108), None
    dims = _scales(ref.shape[2], ref.shape[1], rule)
    for s, (w, h) in enumerate(dims):
        if s:
            ref, dis = _half(ref, w, h), _half(dis, w, h)
        e = _error_maps64(_opsin(ref), _opsin(dis))
        first = e if maps and not s else first
        one, four = e.sum((2, 3)).cpu().numpy(), (e ** 4).sum((2, 3)).cpu().numpy()
        for c in range(3):
            at = c * 36 + s * 6
            sums[at:at + 3], sums[at + 3:at + 6] = one[c], four[c]
            stats[at:at + 3], stats[at + 3:at + 6] = one[c] / (w * h), (four[c] / (w * h)) ** 0.25
    t = float(np.dot([float(v) for v in WEIGHTS.split()], np.abs(stats))) * 0.9562382616834844
    t = 6.248496625763138e-5 * t ** 3 + 2.326765642916932 * t - 0.020884521182843837 * t * t
    out = {"score": 100.0 - 10.0 * t ** 0.6276336467831387 if t > 0 else 100.0, "stats": stats, "sums": sums}
    return (out, len(dims), first)


def _lab(lin):
    m = [[_F(0.4124), _F(0.3576), _F(0.1805)], [_F(0.2126), _F(0.7152), _F(0.0722)], [_F(0.0193), _F(0.1192), _F(0.9505)]]
    v = torch.einsum("kc,chw->khw", torch.tensor(m, dtype=torch.float64, device="cuda"), lin)
    v = v / torch.tensor([0.9505, 1.0, 1.089], dtype=torch.float64, device="cuda")[:, None, None]
    f = torch.where(v > 216.0 / 24389.0, v.clamp_min(0.0) ** (1.0 / 3.0), 24389.0 / (27.0 * 116.0) * v + 16.0 / 116.0)
    return torch.stack([(f[1] - 16.0 / 116.0) * 1.05, (f[0] - f[1]) * (500.0 / 220.0) + 86.2 / 220.0,
                        (f[1] - f[2]) * (200.0 / 220.0) + 107.9 / 220.0])


def _blur3(p):
    q = torch.nn.functional.pad(p[None], (1, 1, 1, 1), mode="replicate")[0]
    h, w = p.shape[1:]
    k = [_F(0.095332), _F(0.118095), _F(0.146293)]
    return sum(k[2 - (ky != 1) - (kx != 1)] * q[:, ky:ky + h, kx:kx + w] for ky in range(3) for kx in range(3))


def _dssim(ref, dis):
    two = lambda p: _blur3(_blur3(p))  # noqa: E731
    scale, w, h = [], ref.shape[2], ref.shape[1]
    for s in range(5):
        if s:
            w, h = max((w + 1) // 2, 8), max((h + 1) // 2, 8)
            ref, dis = _half(ref, w, h), _half(dis, w, h)
        a, b = _lab(ref), _lab(dis)
        a, b = (torch.cat([p[:1], two(p[1:])]) for p in (a, b))
        m1, m2 = two(a), two(b)
        mean = lambda p: p.mean(0)  # noqa: E731
        m11, m22, m12 = mean(m1 * m1), mean(m2 * m2), mean(m1 * m2)
        s11, s22, s12 = mean(two(a * a)) - m11, mean(two(b * b)) - m22, mean(two(a * b)) - m12
        ssim = (2 * m12 + 0.0001) * (2 * s12 + 0.0009) / ((m11 + m22 + 0.0001) * (s11 + s22 + 0.0009))
        avg = ssim.mean().clamp_min(0.0) ** (0.5 ** s)
        scale.append(float(1.0 - (avg - ssim).abs().mean()))
    weights = np.array([0.028, 0.197, 0.322, 0.298, 0.155])
    mean = float(np.dot(scale, weights) / weights.sum())
    return 1.0 / max(mean, 2.220446049250313e-16) - 1.0, np.array(scale)


def _box11(p):
    for dim in (1, 2):
        n = p.shape[dim]
        q = torch.nn.functional.pad(p[None], (0, 0, 5, 5) if dim == 1 else (5, 5, 0, 0), mode="reflect")[0]
        p = sum(q.narrow(dim, k, n) for k in range(11)) / 11.0
    return p


def _zensim(ref, dis):
    h, w = ref.shape[1:]
    n = (w + 15) & ~15
    n += 16 if n >= 512 and (n // 16) % 2 == 0 else 0
    at = torch.arange(n, device="cuda") % max(1, 2 * (w - 1))
    at = torch.where(at < w, at, 2 * (w - 1) - at)
    a, b = (_opsin(p)[:, :, at] for p in (ref, dis))
    basic, peaks = [], []
    while len(basic) < 4 and w >= 8 and h >= 8:
        if basic:
            a, b = _half(a, n, h), _half(b, n, h)
        m1, m2 = _box11(a), _box11(b)
        num_s = 2 * (_box11(a * b) - m1 * m2) + 0.0009
        den = _box11(a * a + b * b) - m1 * m1 - m2 * m2 + 0.0009
        d = (1 - (1 - (m1 - m2) ** 2) * num_s / den).clamp_min(0.0)
        e1, e2 = (a - m1).abs(), (b - m2).abs()
        e = (1 + e2) / (1 + e1) - 1
        maps = [d, e.clamp_min(0.0), (-e).clamp_min(0.0)]
        mean = lambda p: p.mean((1, 2))  # noqa: E731
        l2 = mean(e2 ** 2) / mean(e1 ** 2)
        l1 = mean(e2) / mean(e1)
        cols = [f(m) for m in maps for f in (mean, lambda p: mean(p ** 4) ** 0.25, lambda p: mean(p ** 2) ** 0.5)]
        cols += [mean((a - b) ** 2), (1 - l2).clamp_min(0.0), (1 - l1).clamp_min(0.0), (l2 - 1).clamp_min(0.0)]
        basic.append(torch.stack(cols, 1))
        peaks.append(torch.stack([m.amax((1, 2)) for m in maps] + [mean(m ** 8) ** 0.125 for m in maps], 1))
        w, n, h = (w + 1) // 2, n // 2, (h + 1) // 2
    got = torch.cat([torch.stack(basic).reshape(-1), torch.stack(peaks).reshape(-1)]).cpu().numpy()
    return np.concatenate([got, np.zeros(228 - got.size)])


def exact(case, seed):
    kind, fmt = case["kind"], case["fmt"]
    got = []
    for ref, dis in _inputs(case, seed):
        a, b = _linear64(ref, fmt), _linear64(dis, fmt)
        if kind == "zensim":
            got.append(_zensim(a, b))
        elif kind == "dssim":
            return {"dssim": _dssim(a, b)[0]}
        elif kind in ("pair", "maps"):
            out, _, maps = _ssimulacra2(a, b, case["rule"], kind == "maps")
            return {**out, "maps": maps} if kind == "maps" else out
        else:
            both = _dssim(a, b) if case.get("metrics") == "both" else None
            got.append((_ssimulacra2(a, b, "cpu"), both))
    if kind == "zensim":
        return {"features": np.stack(got)}
    out = {k: np.array([g[0][k] for g, _ in got]) for k in ("score", "stats", "sums")}
    out["scales"], out["status"] = np.array([g[1] for g, _ in got]), np.zeros(len(got), np.int64)
    if case.get("metrics") == "both":
        out["dssim"], out["dssim_scale"] = np.array([d[0] for _, d in got]), np.stack([d[1] for _, d in got])
    return out
