"""The workloads whose speed this library is judged by, as plain functions.

``listed()`` are the fixed cases, ``draw(rng)`` gives further ones of the same
ranges, ``prepare`` makes what a host model holds before the call (fields on
the GPU, or host arrays where the Fortran drop-in passes them), ``run`` is one
call of the public entry points and ``work`` the bytes and operations it
cannot do without.  ``exact`` restates the caller steps in 64 bits; the
radiation schemes and the training have no plain restatement short of the
schemes themselves (sixteen longwave and fourteen shortwave band routines), so
they have none.
"""
import ctypes
import math

import numpy as np
import torch

from ccpp_physics_b200 import abi, cloud_overlap, rad_time_vary, rrtmg_lw, rrtmg_lw_post, rrtmg_sw, surrogate, synthetic

_ready = {}       # what this process has set up: the scheme tables, the network
_F64 = dict(dtype=torch.float64, device="cuda")


def listed():
    return [
        # one physics block handed over by the Fortran host (host arrays), as a
        # host that does not batch its blocks calls the schemes: latency
        dict(name="lw_block_host", kind="lw", memory="host", cols=32, nlay=64, iovr=1, precision="fp64", clouds=True),
        dict(name="sw_block_host", kind="sw", memory="host", cols=57, nlay=127, iovr=1, night=0.4),
        # a small clear-sky set on the device
        dict(name="lw_clear_1024", kind="lw", memory="device", cols=1024, nlay=64, iovr=1, precision="fp64", clouds=False),
        # an ordinary rank's columns, all-sky McICA, each precision of the column path
        dict(name="lw_allsky_16384", kind="lw", memory="device", cols=16384, nlay=127, iovr=1, precision="fp64", clouds=True),
        dict(name="lw_fp32_16384", kind="lw", memory="device", cols=16384, nlay=127, iovr=1, precision="fp32", clouds=True),
        # the decorrelation-length overlap that GFS v16 runs, a ragged column count
        dict(name="lw_dcorr_5003", kind="lw", memory="device", cols=5003, nlay=127, iovr=3, precision="fp64", clouds=True),
        # a C384 face as uneven physics blocks in one call: the largest
        dict(name="lw_blocks_147456", kind="lw_blocks", cols=147456, nlay=127, iovr=1, precision="fp64"),
        dict(name="lw_learned_147456", kind="lw_blocks", cols=147456, nlay=127, iovr=1, precision="surrogate"),
        # the shortwave scheme: all daylit, and a ragged set with night columns and iovr 3
        dict(name="sw_allsky_16384", kind="sw", memory="device", cols=16384, nlay=127, iovr=1, night=0.0),
        dict(name="sw_dcorr_3001", kind="sw", memory="device", cols=3001, nlay=64, iovr=3, night=0.4),
        # seeds, overlap parameters and rrtmg_lw_post of a C384 face
        dict(name="steps_384", kind="steps", side=384, nlay=127),
        # one epoch of the learned gas optics' training: forward, backward, Adam
        dict(name="train_262144", kind="train", samples=262144, batch=8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("lw_host", "sw_host", "lw", "lw", "lw_blocks", "lw_blocks", "sw", "sw", "steps", "train"))
    iovr = rng.choice((1, 1, 3))
    if kind == "lw_host":
        return dict(kind="lw", memory="host", cols=rng.randint(8, 256), nlay=rng.randint(28, 127), iovr=iovr,
                    precision="fp64", clouds=True)
    if kind == "sw_host":
        return dict(kind="sw", memory="host", cols=rng.randint(8, 256), nlay=rng.randint(28, 127), iovr=iovr,
                    night=round(rng.uniform(0.0, 0.6), 3))
    if kind == "lw":
        return dict(kind="lw", memory="device", cols=_log_int(rng, 300, 16384), nlay=rng.randint(40, 127), iovr=iovr,
                    precision=rng.choice(("fp64", "fp64", "fp32")), clouds=rng.random() < 0.8)
    if kind == "lw_blocks":
        return dict(kind="lw_blocks", cols=_log_int(rng, 8192, 140000), nlay=rng.randint(60, 127), iovr=iovr,
                    precision=rng.choice(("fp64", "fp32", "surrogate")))
    if kind == "sw":
        return dict(kind="sw", memory="device", cols=_log_int(rng, 300, 16384), nlay=rng.randint(40, 127), iovr=iovr,
                    night=round(rng.uniform(0.0, 0.6), 3))
    if kind == "steps":
        return dict(kind="steps", side=rng.randint(48, 384), nlay=rng.randint(40, 127))
    return dict(kind="train", samples=rng.randint(65536, 262144), batch=8192)


def _once(key, value, call):
    """Sets up the process-wide state `key` unless it is already `value`."""
    if _ready.get(key) != value:
        call()
        _ready[key] = value


def _init_lw():
    errflg, msg = rrtmg_lw.rlwinit()
    if errflg:
        raise RuntimeError(msg)


def _check(msg, errflg):
    if errflg:
        raise RuntimeError(msg)


def _lw_profile(cols, nlay, seed, clouds):
    """Synthetic columns (``synthetic.make_profiles``) with a boundary-layer
    aerosol in every band."""
    p = synthetic.make_profiles(cols, nlay, seed=seed, cloudy=clouds, device="cuda")
    z = torch.cumsum(p["dzlyr"], 0)
    band = torch.linspace(0.2, 1.0, abi.NBANDS, **_F64)[:, None, None]
    p["aeraod"] = 0.05 * band * (torch.exp(-z / 2.0) * p["dzlyr"])
    p["aerssa"] = (0.3 + 0.3 * band).expand_as(p["aeraod"]).contiguous()
    return p


def _sw_profile(cols, nlay, seed, iovr, night):
    """The shortwave scheme's inputs on the same columns: solar angles with a
    share of night columns, albedos, aerosols, rain and snow in cloud."""
    p = synthetic.make_profiles(cols, nlay, seed=seed, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(seed)

    def u(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(shape, generator=g, **_F64)
    p["cosz"] = torch.where(u(0, 1, cols) < night, torch.zeros(cols, **_F64), u(0.05, 1, cols))
    p["cosz"][0] = 0.5
    p["idxday"] = (torch.nonzero(p["cosz"] >= 1e-4)[:, 0] + 1).to(torch.int32)
    p["solcon"] = 1361.0
    for n in ("sfcalb_nir_dir", "sfcalb_nir_dif", "sfcalb_uvis_dir", "sfcalb_uvis_dif"):
        p[n] = u(0.05, 0.35, cols)
    nb = rrtmg_sw.NBANDS
    z = torch.cumsum(p["dzlyr"], 0)
    p["aeraod"] = 0.1 * torch.exp(-z / 2.0) * p["dzlyr"] * u(0, 1, nb, nlay, cols)
    p["aerssa"], p["aerasy"] = u(0.8, 1.0, nb, nlay, cols), u(0.5, 0.8, nb, nlay, cols)
    cloud, zero = p["cld_cf"] > 0, torch.zeros_like(p["cld_cf"])
    p["cld_rwp"] = torch.where(cloud & (p["tlyr"] > 273.0), u(1.0, 10.0, nlay, cols), zero)
    p["cld_ref_rain"] = torch.full_like(zero, 500.0)
    p["cld_swp"] = torch.where(cloud & (p["tlyr"] < 263.0), u(1.0, 6.0, nlay, cols), zero)
    p["cld_ref_snow"] = u(20.0, 80.0, nlay, cols)
    p["sw_flags"] = dict(rrtmg_sw.DEFAULT_FLAGS, iovr=iovr)
    return p


def _to_host(d):
    return {k: np.ascontiguousarray(v.cpu().numpy()) if isinstance(v, torch.Tensor) else v for k, v in d.items()}


def _steps_inputs(case, seed):
    n, nlay = case["side"] ** 2, case["nlay"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    perm = torch.randperm(n, generator=g, device="cuda").to(torch.int32)
    cf = torch.rand((nlay, n), generator=g, **_F64)
    return dict(imap=(perm % case["side"] + 1).contiguous(), jmap=(perm // case["side"] + 1).contiguous(),
                sec=float(600 * (seed % 144)), lat=(torch.rand(n, generator=g, **_F64) - 0.5) * math.pi,
                dz=0.02 + 2.0 * torch.rand((nlay, n), generator=g, **_F64),
                cf=torch.where(cf < 0.5, torch.zeros_like(cf), cf),
                hlwc=torch.randn((nlay, n), generator=g, **_F64), hlw0=torch.randn((nlay, n), generator=g, **_F64),
                sfcflx=400 * torch.rand((n, 4), generator=g, **_F64), tsfa=260 + 50 * torch.rand(n, generator=g, **_F64))


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    _once("lw", True, _init_lw)
    if kind in ("lw", "lw_blocks"):
        s["prof"] = _lw_profile(case["cols"], case["nlay"], seed, case.get("clouds", True))
        s["prof"]["flags"]["iovr"] = case["iovr"]
    if kind == "lw":
        host = case["memory"] == "host"
        if host:
            s["prof"] = _to_host(s["prof"])
        s["out"] = abi.alloc_outputs(case["cols"], case["nlay"], like=None if host else "cuda")
    elif kind == "lw_blocks":
        if case["precision"] == "surrogate":
            _once("network", "shipped", surrogate.load)
        # every physics block its own contiguous arrays, described once
        sizes = synthetic.physics_blocks(case["cols"])
        s["prof"] = rrtmg_lw.pack_blocks(s["prof"], sizes, inplace=True)
        s["out"] = rrtmg_lw.pack_blocks(abi.alloc_outputs(case["cols"], case["nlay"], like="cuda"), sizes, inplace=True)
        s["args"], s["keep"] = rrtmg_lw.block_args(s["prof"], s["out"], sizes)
        s["exec"] = abi.ExecArgs(precision=rrtmg_lw.PRECISIONS[case["precision"]], memory=abi.DEVICE, sync=1)
        s["msg"] = ctypes.create_string_buffer(512)
    elif kind == "sw":
        _once("sw", True, rrtmg_sw.rswinit)
        s["prof"] = _sw_profile(case["cols"], case["nlay"], seed, case["iovr"], case["night"])
        if case["memory"] == "host":
            s["prof"] = _to_host(s["prof"])
        s["out"] = rrtmg_sw.alloc_outputs(case["cols"], case["nlay"],
                                          like=None if case["memory"] == "host" else s["prof"]["plyr"])
    elif kind == "steps":
        s.update(_steps_inputs(case, seed))
        n = case["side"] ** 2
        s["seeds"] = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2)]
        s["de_lgth"], s["alpha"] = torch.zeros(n, **_F64), torch.zeros_like(s["dz"])
        s["post"] = [torch.zeros(n, **_F64) for _ in range(2)] + [torch.zeros_like(s["dz"]) for _ in range(2)]
    elif kind == "train":
        _ready.pop("network", None)
        s["feats"], targets = surrogate.make_dataset(case["samples"], seed=seed)
        s["feats"], targets = s["feats"][:case["samples"]].contiguous(), targets[:case["samples"]]
        s["norm"] = surrogate.normalisation(s["feats"], targets)
        s["targets"] = surrogate.normalise_targets(targets, s["norm"])
    else:
        raise ValueError(kind)
    torch.cuda.synchronize()     # the library's calls do not all run on torch's stream
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "lw":
        _check(*rrtmg_lw.run_profile(s["prof"], s["out"], precision=case["precision"]))
        return s["out"]
    if kind == "lw_blocks":
        err = rrtmg_lw.lib().rrtmg_lw_gpu_run_blocks(s["args"], len(s["args"]), ctypes.byref(s["exec"]), None,
                                                     s["msg"], 512)
        _check(s["msg"].value.decode(), err)
        return {k: v for k, v in s["out"].items() if isinstance(v, torch.Tensor)}
    if kind == "sw":
        rrtmg_sw.rrtmg_sw_run(s["prof"], s["out"], device_memory=case["memory"] == "device")
        return s["out"]
    if kind == "steps":
        n, nlay, side = case["side"] ** 2, case["nlay"], case["side"]
        _check(*rad_time_vary.gfs_rad_time_vary_seeds(False, None, True, True, 2, 2, *s["seeds"], side, side, 1, 1,
                                                      s["imap"], s["jmap"], s["sec"], 35000, 100_000_000, sync=False))
        _check(*cloud_overlap.overlap_params(5, 1, s["dz"], s["cf"], s["de_lgth"], s["alpha"], xlat=s["lat"], sync=False))
        _check(*rrtmg_lw_post.rrtmg_lw_post_run(n, nlay, 0, nlay, 0, True, True, s["tsfa"], s["hlwc"], s["hlw0"],
                                                s["sfcflx"], *s["post"], sync=False))
        return dict(seeds=s["seeds"], de_lgth=s["de_lgth"], alpha=s["alpha"], post=s["post"])
    surrogate.init(s["norm"], seed=1)
    losses = surrogate.train(s["feats"], s["targets"], epochs=1, batch=case["batch"], lr=1e-3, lr_final=1e-4,
                             tau_weight=True)
    return dict(weights=surrogate.get_weights()[0], losses=losses)


def work(case):
    kind = case["kind"]
    if kind in ("lw", "lw_blocks"):
        # 56 input and 3 output doubles per layer, 138 per column; 12.6 kflop
        # per layer (gas optics and transfer of 140 g-points), 106 kflop for
        # the network in its place
        n, nlay = case["cols"], case["nlay"]
        flops = 106240 + 8000 if case["precision"] == "surrogate" else 12600
        return dict(bytes=n * (8 * (59 * nlay + 138) + 4), flops=n * nlay * flops)
    if kind == "sw":
        # 66 input and 3 output doubles per layer; gas optics, one two-stream
        # evaluation and both sweeps of 112 g-points: 23.5 kflop per layer
        n, nlay = max(1, int(case["cols"] * (1 - case["night"]))), case["nlay"]
        return dict(bytes=n * 8 * (69 * nlay + 24), flops=n * nlay * 23500)
    if kind == "steps":
        n, nlay = case["side"] ** 2, case["nlay"]
        return dict(bytes=n * (8 * (7 * nlay + 6) + 16), flops=n * nlay * 20)
    macs = 16 * 128 + 128 * 128 + 128 * 288
    return dict(bytes=case["samples"] * 4 * (8 + 288), flops=case["samples"] * 2 * (3 * macs - 16 * 128))


def exact(case, seed):
    if case["kind"] != "steps":
        return None
    x = _steps_inputs(case, seed)
    de = torch.clamp(2.78 - 4.6 * (x["lat"] / math.pi).abs(), min=0.6)
    alpha = torch.exp(-x["dz"] / de)
    alpha[1:][(x["cf"][1:] == 0.0) & (x["cf"][:-1] > 0.0)] = 0.0
    alpha[0] = 0.0
    return dict(seeds=[None, None], de_lgth=de, alpha=alpha,
                post=[x["tsfa"], x["sfcflx"][:, 2].contiguous(), x["hlwc"], x["hlw0"]])
