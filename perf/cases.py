"""Timed cases: what a user of this package has it do, through its public entry points.

A case is one call on one dataset.  Four kinds:

* ``plan``: a batched Whittle likelihood (``WhittleLikelihood``): lnL of one
  parameter mapping (``call`` "params"), of a batch ("lnl"), lnL with its
  gradient ("grad") or Fisher matrices ("fisher"), from the FP64 or the mixed
  plan, for IMRPhenomD or IMRPhenomHM, on one to three detectors.
* ``driver``: one sample through the plugins as a bilby sampler drives them
  (waveform, single-link response, TDI, lnL).
* ``td_tdi``: the time-domain TDI combination of six link series.

Sizes are those of the benchmark's workloads and of the tests (grids of
2^18 s to 2^23 s, batches of 1 to 1024, 8.4 million time samples).  ``draw``
takes others of the same ranges.

``exact`` restates the models in 64-bit torch: IMRPhenomD (arXiv:1508.07250,
1508.07253), IMRPhenomHM's maps (arXiv:1708.00404), the response of Marsat et
al. (2018) and equal-arm TDI.  Its only input from the package is the table of
quasi-normal-mode frequencies, read as numbers.
"""

import functools
import math
import os
import re

import numpy as np
import torch

PI = math.pi
C_SI, YEAR, AU = 299792458.0, 31557600.0, 149597870700.0
MRSUN, MTSUN, PC = 1.476625038050124729627979840144936351e3, 4.925490947641266978197229498498379006e-6, 3.085677581491367e16
EULER = 0.5772156649015329
DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64
DETECTORS = ("LISA", "Taiji", "TianQin")
ARM = {"LISA": 2.5e9, "Taiji": 3.0e9, "TianQin": math.sqrt(3.0) * 1e8}
NOISE = {"LISA": "LISA_SciRDv1", "Taiji": "Taiji_TDC", "TianQin": "Tianqin_GWSpace"}


# ------------------------------------------------------------------ the cases
def _plan(name, call, precision, batch, duration, dt, fmin, fmax, generation="1.5", detectors="LISA", approximant="D",
          nodes=1024, cut=1.2, samples="prior"):
    return {"name": name, "kind": "plan", "call": call, "precision": precision, "batch": batch, "duration": duration,
            "dt": dt, "fmin": fmin, "fmax": fmax, "generation": generation, "detectors": detectors,
            "approximant": approximant, "nodes": nodes, "cut": cut, "samples": samples}


def listed():
    return [
        # one step of a Metropolis chain, the reference's call with its default precision
        _plan("step_fp64", "params", "fp64", 1, 2.0 ** 20, 16.0, 1e-4, 0.03, cut=0.0, samples="posterior"),
        # a handful of chains on a short stretch of data (the tests' grid): latency and launches
        _plan("chains_short", "lnl", "mixed", 16, 2.0 ** 18, 8.0, 1e-4, 0.03, samples="posterior"),
        # the benchmark's batch of prior draws (nested sampling, SMC initialisation): lnL alone
        _plan("prior_lnl", "lnl", "mixed", 1024, 2.0 ** 22, 8.0, 1e-4, 0.03),
        # HMC chains on the three-detector network, whose inputs stream from DRAM
        _plan("chains_grad_network", "grad", "mixed", 24, 2.0 ** 23, 4.0, 3e-5, 0.1,
              detectors="LISA+Taiji+TianQin", nodes=2048, samples="posterior"),
        # the benchmark itself: lnL and gradient of 1024 prior draws
        _plan("prior_grad", "grad", "mixed", 1024, 2.0 ** 22, 8.0, 1e-4, 0.03),
        # Fisher matrices of an SMC sweep's particles
        _plan("fisher", "fisher", "mixed", 100, 2.0 ** 22, 8.0, 1e-4, 0.03, samples="posterior"),
        # the shape of the reference's published timings (65 471 bins, TDI 2.0) in FP64
        _plan("lnl_fp64", "lnl", "fp64", 37, 655360.0, 5.0, 1e-4, 0.1, generation="2.0"),
        # FP64 gradients on a heliocentric and a geocentric detector
        _plan("grad_fp64", "grad", "fp64", 12, 2.0 ** 20, 8.0, 1e-4, 0.03, detectors="LISA+TianQin"),
        # higher modes on the network (the six-mode configuration at a quarter of its duration)
        _plan("network_hm", "lnl", "mixed", 12, 2.0 ** 23, 4.0, 3e-5, 0.1, detectors="LISA+Taiji+TianQin",
              approximant="HM", nodes=2048),
        # one sample through the plugins (bilby)
        {"name": "bilby_d", "kind": "driver", "duration": 2.0 ** 22, "dt": 8.0, "fmin": 1e-4, "fmax": 0.03,
         "generation": "1.5", "detectors": "LISA", "approximant": "D"},
        {"name": "bilby_hm_network", "kind": "driver", "duration": 1500000.0, "dt": 5.0, "fmin": 1e-4, "fmax": 0.1,
         "generation": "2.0", "detectors": "LISA+Taiji+TianQin", "approximant": "HM"},
        # a year of time-domain links to A/E/T
        {"name": "td_tdi", "kind": "td_tdi", "n": 8388609, "dt": 4.0, "arm": "LISA", "generation": "2.0",
         "orthogonal": True, "precision": "mixed"},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


# the most (sample, detector, bin) evaluations of a drawn call: no more than the listed calls take
_LIMIT = {("mixed", "lnl"): 1.2e8, ("mixed", "grad"): 1.2e8, ("mixed", "fisher"): 1.25e7, ("fp64", "lnl"): 2.4e6,
          ("fp64", "grad"): 7.5e5, ("fp64", "params"): 1.0e6, ("mixed", "params"): 1.0e6, ("HM", "lnl"): 3.0e7}


def draw(rng):
    kind = rng.choices(("plan", "driver", "td_tdi"), (8, 2, 2))[0]
    if kind == "td_tdi":
        arm, dt = rng.choice(DETECTORS), rng.choice((0.5, 2.0, 4.0, 5.0))
        return {"kind": kind, "n": int(_log_uniform(rng, 3000, 8.3e6)), "dt": dt, "arm": arm,
                "generation": rng.choice(("1.5", "2.0")), "orthogonal": rng.random() < 0.7,
                "precision": rng.choice(("mixed", "mixed", "fp64"))}
    detectors = rng.choice(("LISA", "LISA", "Taiji", "LISA+Taiji", "LISA+TianQin", "LISA+Taiji+TianQin"))
    dt, fmax = rng.choice(((4.0, 0.1), (5.0, 0.08), (8.0, 0.03), (16.0, 0.03)))
    duration = round(_log_uniform(rng, 2.0 ** 18, 2.0 ** 22), 1)
    case = {"kind": kind, "duration": duration, "dt": dt, "fmin": rng.choice((3e-5, 1e-4)), "fmax": fmax,
            "generation": rng.choice(("1.5", "1.5", "2.0")), "detectors": detectors,
            "approximant": rng.choice(("D", "D", "D", "HM"))}
    if kind == "driver":
        return case
    if case["approximant"] == "HM":
        case.update(precision="mixed", call="lnl")
    else:
        case["precision"] = rng.choice(("mixed", "mixed", "fp64"))
        case["call"] = rng.choice(("params", "lnl", "lnl", "grad", "grad", "fisher"))
        if case["precision"] == "fp64" and case["call"] == "fisher":
            case["call"] = "lnl"
    per = fmax * duration * len(detectors.split("+"))
    most = _LIMIT[("HM" if case["approximant"] == "HM" else case["precision"], case["call"])] / per
    case.update(batch=1 if case["call"] == "params" else max(1, min(1024, int(_log_uniform(rng, 1, max(1.01, most))))),
                nodes=rng.choice((1024, 1024, 2048)), cut=rng.choice((0.0, 1.2)),
                samples=rng.choice(("prior", "posterior")))
    return case


# ------------------------------------------------------------------ inputs
def _grid(case):
    nt = int(case["duration"] // case["dt"] + 1)
    full = np.fft.rfftfreq(nt, case["dt"])
    return full[(full >= case["fmin"]) & (full <= case["fmax"])]


def _dets(case):
    return case["detectors"].split("+")


def _injection(case):
    """The injected source: 1e6 + 5e5 Msun at 10 Gpc, merging a little before the data end."""
    m1, m2 = 1e6, 5e5
    mc = (m1 * m2) ** 0.6 / (m1 + m2) ** 0.2
    return np.array([math.log(mc), 2.0, 0.5, -0.3, math.log(1e4), 0.5, 1.0, math.sin(0.3), 0.7, 0.0,
                     case["duration"] - min(86400.0, 0.08 * case["duration"])])


def _thetas(case, seed):
    rng = np.random.default_rng([seed, 3])
    inj, n = _injection(case), case.get("batch", 1)
    if case.get("samples") == "prior":
        mtot = np.exp(rng.uniform(math.log(1e5), math.log(1e7), n))
        q = rng.uniform(1.0, 8.0, n)
        mc = mtot * (q / (1 + q) ** 2) ** 0.6
        return np.stack([np.log(mc), q, rng.uniform(-0.99, 0.99, n), rng.uniform(-0.99, 0.99, n),
                         np.log(rng.uniform(1e3 ** 3, 3e4 ** 3, n) ** (1 / 3)), rng.uniform(-1, 1, n),
                         rng.uniform(0, 2 * PI, n), rng.uniform(-1, 1, n), rng.uniform(0, PI, n),
                         rng.uniform(0, 2 * PI, n), inj[10] + rng.uniform(-3600, 3600, n)], axis=1)
    wide = np.array([1e-5, 2e-3, 5e-3, 5e-3, 5e-3, 5e-3, 5e-3, 5e-3, 5e-3, 5e-3, 2.0])
    return inj + wide * rng.standard_normal((n, 11))


def _mapping(th):
    """A parameter row as the reference's parameter mapping."""
    q = th[1]
    return {"chirp_mass": math.exp(th[0]), "mass_ratio": q, "chi_1": th[2], "chi_2": th[3],
            "luminosity_distance": math.exp(th[4]), "inclination": math.acos(th[5]), "ecliptic_longitude": th[6],
            "ecliptic_latitude": math.asin(th[7]), "polarization": th[8], "reference_phase": th[9],
            "coalescence_time": th[10]}


def _psd(name, f, generation):
    """(3, n) A/E/T noise power of the preset models (arXiv:2108.01167, 2309.15020)."""
    w, x = 2 * PI * f / C_SI, PI * f / C_SI
    if name == "TianQin":
        oms, acc, L = 1e-24 * w ** 2, 1e-30 * (1 + 0.1e-3 / f) / (w * C_SI ** 2) ** 2, 1.7e8
    else:
        oms = ((15e-12 if name == "LISA" else 8e-12) ** 2) * (1 + (2e-3 / f) ** 4) * w ** 2
        acc, L = 9e-30 * (1 + (0.4e-3 / f) ** 2) * (1 + (f / 8e-3) ** 4) / (w * C_SI ** 2) ** 2, ARM[name]
    x = x * L
    c2, c4, s2, s1 = torch.cos(2 * x), torch.cos(4 * x), torch.sin(2 * x) ** 2, torch.sin(x) ** 2
    ae = 8 * s2 * ((2 + c2) * oms + (6 + 4 * c2 + 2 * c4) * acc)
    out = torch.stack([ae, ae, 32 * s2 * s1 * (oms + 4 * s1 * acc)])
    return out * (4 * torch.sin(4 * x) ** 2) if generation == "2.0" else out


def _noise(case, seed, k, f):
    """Gaussian noise of variance S / (2 df) per bin of detector k."""
    g = torch.Generator(device=DEV).manual_seed(1000003 * int(seed) + k)
    z = torch.randn((3, f.numel(), 2), generator=g, dtype=F64, device=DEV)
    S = _psd(_dets(case)[k], f, case["generation"])
    return torch.view_as_complex(z) * torch.sqrt(S * (0.25 * case["duration"]))


def _links(case, seed, added):
    """Six link series: a slow signal under white noise of a tenth of its amplitude."""
    n = case["n"] + added
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    t = torch.arange(n, dtype=F64, device=DEV) * case["dt"]
    ph = torch.rand(6, 1, generator=g, dtype=F64, device=DEV) * 2 * PI
    out = torch.randn((6, n), generator=g, dtype=F64, device=DEV)
    out.mul_(1e-22).add_(1e-21 * torch.sin(2 * PI * 3.1e-3 * t[None] + ph))
    return out


def _orbit(name):
    from pespace_gb300.detector.orbit import KaplerianHeliocentric, KeplerianGeocentric

    if name == "TianQin":
        return KeplerianGeocentric(ARM[name])
    return KaplerianHeliocentric(ARM[name], 0.0, -PI / 9 if name == "LISA" else PI / 9)


def prepare(case, seed):
    from pespace_gb300.detector.antenna import FDResponseModelMarset2018, InterferometerAntenna
    from pespace_gb300.detector.tdi import FDMichelsonConstantEqualArm, TDIChannelData, TDMichelsonConstantEqualArm
    from pespace_gb300.inference import LikelihoodBilbyInterface, WhittleLikelihood
    from pespace_gb300.waveform import IMRPhenomD, IMRPhenomHM

    if case["kind"] == "td_tdi":
        data = TDIChannelData()
        data.set_td_data_from_zero(("A", "E", "T"), (case["n"] - 1) * case["dt"], case["dt"], 0.0, 1e-4, 2e-4)
        tdi = TDMichelsonConstantEqualArm(case["generation"], case["orthogonal"], precision=case["precision"])
        det = InterferometerAntenna(case["arm"], data, _orbit(case["arm"]), FDResponseModelMarset2018(), tdi)
        det.single_link_response = _links(case, seed, tdi.added_time_samples_number)
        return {"kind": "td_tdi", "det": det, "tdi": tdi}

    inj = _injection(case)
    dets = []
    for k, name in enumerate(_dets(case)):
        data = TDIChannelData()
        data.set_fd_data_from_zero(("A", "E", "T"), case["duration"], case["dt"], 0.0, case["fmin"], case["fmax"])
        data.set_fd_noise_power_density_from_model(NOISE[name], tdi_generation=case["generation"])
        det = InterferometerAntenna(name, data, _orbit(name), FDResponseModelMarset2018(),
                                    FDMichelsonConstantEqualArm(case["generation"], True))
        data.add_into_fd_data(_noise(case, seed, k, data.frequency_samples))
        wf = (IMRPhenomHM if case["approximant"] == "HM" else IMRPhenomD)(data.data_info.frequency_samples_array, 1e-4)
        det.inject_signal(wf.from_theta(inj), inj[6], math.asin(inj[7]), inj[8], inj[10])
        dets.append(det)
    thetas = _thetas(case, seed)
    if case["kind"] == "driver":
        like = LikelihoodBilbyInterface(wf, tuple(dets), ("A", "E", "T"))
        return {"kind": "driver", "like": like, "params": _mapping(thetas[0]), "dets": dets}
    like = WhittleLikelihood(tuple(dets), precision=case["precision"], reference_frequency=1e-4,
                             cut_factor=case["cut"], max_batch=case["batch"], n_sparse=case["nodes"],
                             approximant="IMRPhenom" + case["approximant"])
    theta = _mapping(thetas[0]) if case["call"] == "params" else torch.as_tensor(thetas, device="cuda")
    return {"kind": case["call"], "like": like, "theta": theta}


def run(state):
    kind = state["kind"]
    if kind == "params":
        return state["like"].log_likelihood(state["theta"])
    if kind == "lnl":
        return state["like"].log_likelihood_batch(state["theta"])
    if kind == "grad":
        return state["like"].log_likelihood_and_grad(state["theta"])
    if kind == "fisher":
        return state["like"].fisher_matrix(state["theta"])
    if kind == "driver":
        logl = state["like"].log_likelihood(state["params"])
        return [logl] + [det.tdi_response for det in state["dets"]]
    state["tdi"].update_tdi_response()
    return state["det"].tdi_response


def work(case):
    """Bytes: the data, noise power and parameters read and the results written, each once.  Operations: those of
    the model per (sample, detector, bin), with the waveform's and response's functions counted as ten each."""
    if case["kind"] == "td_tdi":
        delays = 7 if case["generation"] == "2.0" else 3
        return {"bytes": 72.0 * case["n"], "flops": (6 + 24 + 6.0 * 3 * (delays + 1)) * case["n"]}
    n, nd = len(_grid(case)), len(_dets(case))
    modes = 6 if case["approximant"] == "HM" else 1
    if case["kind"] == "driver":  # the container, links and TDI response are written, and read by the next plugin
        waveform, response = 40.0 * modes * 2, 96.0 * 2 + 48.0 * 2
        return {"bytes": n * (waveform + nd * (response + 72.0)), "flops": n * (80.0 * modes + nd * (170.0 * modes + 60))}
    B, call = case["batch"], case["call"]
    per = {"params": 60, "lnl": 60, "grad": 180, "fisher": 600}[call]
    out = {"params": 8, "lnl": 8, "grad": 96, "fisher": 968}[call]
    return {"bytes": 72.0 * n * nd + B * (88 + out), "flops": float(B) * n * (80.0 * modes + nd * (170.0 * modes + per))}


# ------------------------------------------------------------------ the models in 64 bits
# Khan et al. 2016, Table V: v2, gamma 1-3, sigma 1-4, beta 1-3, alpha 1-5, rho 1-3
_FITS = [
    [0.8149838730507785, 2.5747553517454658, 1.1610198035496786, -2.3627771785551537, 6.771038707057573, 0.7570782938606834, -2.7256896890432474, 7.1140380397149965, 0.1766934149293479, -0.7978690983168183, 2.1162391502005153],
    [0.006927402739328343, 0.03020474290328911, 0.006308024337706171, -0.12074130661131138, 0.26271598905781324, 0.0034151773647198794, -0.10779338611188374, 0.27098966966891747, 0.0007374185938559283, -0.02749621038376281, 0.0733150789135702],
    [1.010344404799477, 0.0008993122007234548, 0.283949116804459, -4.049752962958005, 13.207828172665366, 0.10396278486805426, -7.025059158961947, 24.784892370130475, 0.03093202475605892, -2.6924023896851663, 9.609374464684983],
    [1.3081615607036106, -0.005537729694807678, -0.06782917938621007, -0.6689834970767117, 3.403147966134083, -0.05296577374411866, -0.9923793203111362, 4.820681208409587, -0.006134139870393713, -0.38429253308696365, 1.7561754421985984],
    [2096.551999295543, 1463.7493168261553, 1312.5493286098522, 18307.330017082117, -43534.1440746107, -833.2889543511114, 32047.31997183187, -108609.45037520859, 452.25136398112204, 8353.439546391714, -44531.3250037322],
    [-10114.056472621156, -44631.01109458185, -6541.308761668722, -266959.23419307504, 686328.3229317984, 3405.6372187679685, -437507.7208209015, 1.6318171307344697e6, -7462.648563007646, -114585.25177153319, 674402.4689098676],
    [22933.658273436497, 230960.00814979506, 14961.083974183695, 1.1940181342318142e6, -3.1042239693052764e6, -3038.166617199259, 1.8720322849093592e6, -7.309145012085539e6, 42738.22871475411, 467502.018616601, -3.064853498512499e6],
    [-14621.71522218357, -377812.8579387104, -9608.682631509726, -1.7108925257214056e6, 4.332924601416521e6, -22366.683262266528, -2.5019716386377467e6, 1.0274495902259542e7, -85360.30079034246, -570025.3441737515, 4.396844346849777e6],
    [97.89747327985583, -42.659730877489224, 153.48421037904913, -1417.0620760768954, 2752.8614143665027, 138.7406469558649, -1433.6585075135881, 2857.7418952430758, 41.025109467376126, -423.680737974639, 850.3594335657173],
    [-3.282701958759534, -9.051384468245866, -12.415449742258042, 55.4716447709787, -106.05109938966335, -11.953044553690658, 76.80704618365418, -155.33172948098394, -3.4129261592393263, 25.572377569952536, -54.408036707740465],
    [-0.000025156429818799565, 0.000019750256942201327, -0.000018370671469295915, 0.000021886317041311973, 0.00008250240316860033, 7.157371250566708e-6, -0.000055780000112270685, 0.00019142082884072178, 5.447166261464217e-6, -0.00003220610095021982, 0.00007974016714984341],
    [43.31514709695348, 638.6332679188081, -32.85768747216059, 2415.8938269370315, -5766.875169379177, -61.85459307173841, 2953.967762459948, -8986.29057591497, -21.571435779762044, 981.2158224673428, -3239.5664895930286],
    [-0.07020209449091723, -0.16269798450687084, -0.1872514685185499, 1.138313650449945, -2.8334196304430046, -0.17137955686840617, 1.7197549338119527, -4.539717148261272, -0.049983437357548705, 0.6062072055948309, -1.682769616644546],
    [9.5988072383479, -397.05438595557433, 16.202126189517813, -1574.8286986717037, 3600.3410843831093, 27.092429659075467, -1786.482357315139, 5152.919378666511, 11.175710130033895, -577.7999423177481, 1808.730762932043],
    [-0.02989487384493607, 1.4022106448583738, -0.07356049468633846, 0.8337006542278661, 0.2240008282397391, -0.055202870001177226, 0.5667186343606578, 0.7186931973380503, -0.015507437354325743, 0.15750322779277187, 0.21076815717176228],
    [0.9974408278363099, -0.007884449714907203, -0.059046901195591035, 1.3958712396764088, -4.516631601676276, -0.05585343136869692, 1.7516580039343603, -5.990208965347804, -0.017945336522161195, 0.5965097794825992, -2.0608879367971804],
    [3931.8979897196614, -17395.758706812805, 3132.375545898835, 343965.86092361377, -1.2162565819981997e6, -70698.00600428853, 1.383907177859705e6, -3.9662761890979446e6, -60017.52423652596, 803515.1181825735, -2.091710365941658e6],
    [-40105.47653771657, 112253.0169706701, 23561.696065836168, -3.476180699403351e6, 1.137593670849482e7, 754313.1127166454, -1.308476044625268e7, 3.6444584853928134e7, 596226.612472288, -7.4277901143564405e6, 1.8928977514040343e7],
    [83208.35471266537, -191237.7264145924, -210916.2454782992, 8.71797508352568e6, -2.6914942420669552e7, -1.9889806527362722e6, 3.0888029960154563e7, -8.390870279256162e7, -1.4535031953446497e6, 1.7063528990822166e7, -4.2748659731120914e7],
]
_MODES = ((2, 2, 0), (2, 1, 1), (3, 3, 3), (3, 2, 0), (4, 4, 2), (4, 3, 3))  # l, m, quarter turns of H_lm


@functools.lru_cache(maxsize=None)
def _qnm_table():
    """(modes, 4, nodes) spline table of the Kerr quasi-normal modes, its first node and spacing; None without it."""
    path = os.path.join("pespace_gb300", "csrc", "pes_qnm_table.h")
    if not os.path.isfile(path):
        return None
    text = open(path).read()
    value = {k: float(v) for k, v in re.findall(r"#define (PES_QNM_\w+) (\S+)", text) if "(" not in v and k != "PES_QNM_STORAGE"}
    body = re.sub(r"//.*", "", text[text.index("kQnmTable[PES_QNM_MODES]"):])
    numbers = np.array(re.findall(r"[-+]?\d+\.?\d*(?:[eE][-+]?\d+)?", body[body.index("{"):]), dtype=np.float64)
    return torch.as_tensor(numbers.reshape(6, 4, int(value["PES_QNM_NODES"])), device=DEV), value["PES_QNM_U0"], value["PES_QNM_DU"]


def _qnm(mode, af):
    tab, u0, h = _qnm_table()
    u = torch.sqrt(1.0 - af.clamp(-0.999, 0.999))
    i = ((u.detach() - u0) / h).floor().clamp(0, tab.shape[2] - 2)
    t = (u - (u0 + i * h)) / h
    i = i.long()
    s = 1.0 - t
    a, b = (s ** 3 - s) * (h * h / 6), (t ** 3 - t) * (h * h / 6)
    y, y2, z, z2 = tab[mode]
    return s * y[i] + t * y[i + 1] + a * y2[i] + b * y2[i + 1], s * z[i] + t * z[i + 1] + a * z2[i] + b * z2[i + 1]


def _fit(w, eta, xi):
    c = _FITS[w]
    return (c[0] + c[1] * eta + xi * (c[2] + eta * (c[3] + eta * c[4])) + xi ** 2 * (c[5] + eta * (c[6] + eta * c[7]))
            + xi ** 3 * (c[8] + eta * (c[9] + eta * c[10])))


def _psi_ins(c, Mf):
    """Inspiral phase and its derivative with respect to Mf."""
    u = Mf ** (1 / 3)
    lu = torch.log(u)
    p, r = c["pin11"], 2.0 * c["pin11"]
    for j in range(10, -1, -1):
        p, r = p * u + c[f"pin{j}"], r * u + c[f"pin{j}"] * ((j - 5) / 3)
    return (p / u ** 5 + (c["lg0"] + c["lg1"] * u) * lu,
            r / u ** 8 + (c["lg0"] / u + c["lg1"] * (lu + 1.0)) / (3 * u ** 2))


def _psi_int(c, Mf):
    return (c["int0"] + c["int1"] * Mf + c["int2"] / Mf ** 3 + c["int3"] * torch.log(Mf),
            c["int1"] - 3 * c["int2"] / Mf ** 4 + c["int3"] / Mf)


def _psi_mrd(c, fdm, Mf):
    x = Mf - c["pm5"]
    return (c["pm0"] + c["pm1"] * Mf + c["pm2"] / Mf + c["pm3"] * Mf ** 0.75 + c["pm4"] * torch.atan(x / fdm),
            c["pm1"] - c["pm2"] / Mf ** 2 + 0.75 * c["pm3"] * Mf ** -0.25 + c["pm4"] * fdm / (fdm ** 2 + x ** 2))


def _pieces(x, edges, parts):
    """parts[k] on the stretch of ascending x between edges[k-1] and edges[k] (last part from the last edge on)."""
    cuts = [0] + [int(torch.searchsorted(x.detach(), torch.as_tensor(e, dtype=F64, device=x.device).detach().reshape(()))) for e in edges] + [x.numel()]
    cuts = np.maximum.accumulate(cuts)
    got = [part(x[a:b]) for part, a, b in zip(parts, cuts[:-1], cuts[1:]) if b > a]
    return tuple(torch.cat(v) for v in zip(*got)) if isinstance(got[0], tuple) else torch.cat(got)


def _psi(c, Mf):
    return _pieces(Mf, (0.018, 0.5 * c["fRD"]),
                   (lambda x: _psi_ins(c, x), lambda x: _psi_int(c, x), lambda x: _psi_mrd(c, c["fDM"], x)))


def _poly(c, name, n, x):
    r = c[f"{name}{n - 1}"]
    for j in range(n - 2, -1, -1):
        r = r * x + c[f"{name}{j}"]
    return r


def _amp_ins(c, Mf):
    u = Mf ** (1 / 3)
    return 1.0 + u ** 2 * _poly(c, "ai", 8, u)


def _amp_mrd(c, w, Mf):
    x = Mf - c["fRD"]
    return c["g1"] * w / (x ** 2 + w ** 2) * torch.exp(-c["g2"] * x / w)


def _amp(c, Mf, w, fpeak, dl):
    hat = _pieces(Mf, (0.014, fpeak),
                  (lambda x: _amp_ins(c, x), lambda x: _poly(c, dl, 5, x), lambda x: _amp_mrd(c, w, x)))
    return c["scale"] * Mf ** (-7 / 6) * hat


def _intermediate(c, w, fpeak):
    """The quartic through the amplitude's joins (value and slope) and its collocation point."""
    f1 = torch.full_like(fpeak, 0.014)
    u1 = f1 ** (1 / 3)
    slope = sum((j + 2) * c[f"ai{j}"] * u1 ** (j + 1) for j in range(8)) / (3 * u1 ** 2)
    x3 = fpeak - c["fRD"]
    top = _amp_mrd(c, w, fpeak)
    dtop = top * (-c["g2"] / w - 2 * x3 / (x3 ** 2 + w ** 2))
    f2 = 0.5 * (f1 + fpeak)
    rows = [torch.stack([f ** j for j in range(5)], -1) for f in (f1, f2, fpeak)]
    rows += [torch.stack([j * f ** (j - 1) if j else torch.zeros_like(f) for j in range(5)], -1) for f in (f1, fpeak)]
    rhs = torch.stack([_amp_ins(c, f1), c["v2"], top, slope, dtop], -1)
    return torch.linalg.solve(torch.stack(rows, -2), rhs[..., None])[..., 0].unbind(-1)


def _peak(c, w):
    low = c["fRD"] + w * (torch.sqrt((1 - c["g2"] ** 2).clamp_min(1e-300)) - 1) / c["g2"]
    return torch.abs(torch.where(c["g2"] <= 1.0, low, c["fRD"] - w / c["g2"]))


def _phenomd(th):
    """IMRPhenomD's coefficients for (B, 11) parameters: a dict of (B,) tensors."""
    c = {}
    q, chi1, chi2 = th[:, 1], th[:, 2], th[:, 3]
    eta = q / (1 + q) ** 2
    m1, m2, seta = q / (1 + q), 1 / (1 + q), (q - 1) / (1 + q)
    M = torch.exp(th[:, 0]) * eta ** -0.6
    c["Msec"] = M * MTSUN
    chipn = m1 * chi1 + m2 * chi2 - (38 / 113) * eta * (chi1 + chi2)
    xi = chipn - 1
    s = m1 ** 2 * chi1 + m2 ** 2 * chi2
    af = eta * (3.4641016151377544 - 4.399247300629289 * eta + 9.397292189321194 * eta ** 2 - 13.180949901606242 * eta ** 3
                + s * ((1 / eta - 0.0850917821418767 - 5.837029316602263 * eta)
                       + s * ((0.1014665242971878 - 2.0967746996832157 * eta)
                              + s * ((-1.3546806617824356 + 4.108962025369336 * eta)
                                     + s * (-0.8676969352555539 + 2.064046835273906 * eta)))))
    sn = s / (m1 ** 2 + m2 ** 2)
    erad = ((0.055974469826360077 + 0.5809510763115132 * eta - 0.9606726679372312 * eta ** 2 + 3.352411249771192 * eta ** 3)
            * eta * (1 + (-0.0030302335878845507 - 2.0066110851351073 * eta + 7.7050567802399215 * eta ** 2) * sn)
            / (1 + (-0.6714403054720589 - 1.4756929437702908 * eta + 7.304676214885011 * eta ** 2) * sn))
    c["af"], c["erad"], c["eta"] = af, erad, eta
    wr, wi = _qnm(0, af)
    c["fRD"], c["fDM"] = wr / (2 * PI) / (1 - erad), wi / (2 * PI) / (1 - erad)
    c["v2"], c["g1"], c["g2"] = _fit(0, eta, xi), _fit(1, eta, xi), _fit(2, eta, xi)
    c["w"] = _fit(3, eta, xi) * c["fDM"]
    c["fpeak"] = _peak(c, c["w"])
    sp, sm, a2, d2, x12 = 1 + seta, 1 - seta, chi1 ** 2 + chi2 ** 2, chi1 ** 2 - chi2 ** 2, chi1 * chi2
    c["ai0"] = (-969 + 1804 * eta) * PI ** (2 / 3) / 672
    c["ai1"] = (chi1 * (81 * sp - 44 * eta) + chi2 * (81 * sm - 44 * eta)) * PI / 48
    sq = chi1 ** 2 * sp + chi2 ** 2 * sm
    c["ai2"] = (-27312085 - 10287648 * sq + 24 * (-1975055 + 857304 * a2 - 994896 * x12) * eta
                + 35371056 * eta ** 2) * PI ** (4 / 3) / 8128512
    c["ai3"] = (chi1 * (285197 * sp - 4 * (91902 + 1579 * seta) * eta - 35632 * eta ** 2)
                + chi2 * (285197 * sm - 4 * (91902 - 1579 * seta) * eta - 35632 * eta ** 2)
                + 42840 * PI * (-1 + 4 * eta)) * PI ** (5 / 3) / 32256
    c["ai4"] = (336 * (-3248849057 + 2943675504 * a2 - 3339284256 * x12) * eta ** 2 + 324322727232 * eta ** 3
                + 7 * (-177520268561 + 107414046432 * sq + 11087290368 * PI * (chi1 * sp + chi2 * sm))
                - 12 * eta * (-545384828789 - 176491177632 * x12 + 77616 * 2610335 * a2 + 77616 * 995766 * seta * d2
                              + 5841690624 * PI * (chi1 + chi2) + 21384760320 * PI ** 2)) * PI ** 2 / 60085960704
    for k in range(3):
        c[f"ai{5 + k}"] = _fit(16 + k, eta, xi)
    SL, dSL = s, seta * (m2 * chi2 - m1 * chi1)
    sigma = (474 / 48) * eta * x12 + (486 / 96) * (m1 ** 2 * chi1 ** 2 + m2 ** 2 * chi2 ** 2)
    gamma = (554345 / 1134 + (110 / 9) * eta) * SL + (13915 / 84 - (10 / 3) * eta) * dSL
    N = 3 / (128 * eta)
    v6 = (11583.231236531 / 4.694215680 - 640 / 3 * PI ** 2 - 6848 / 21 * EULER - 6848 / 21 * math.log(4.0)
          + eta * (-15737.765635 / 3.048192 + 2255 / 12 * PI ** 2) + eta ** 2 * 76055 / 1728 - eta ** 3 * 127825 / 1296
          + PI / 3 * (3760 * SL + 1490 * dSL))
    a7 = (PI * (77096675 / 254016 + 378515 / 1512 * eta - 74045 / 756 * eta ** 2)
          + (-8980424995 / 762048 + 6586595 / 756 * eta - 305 / 36 * eta ** 2) * SL
          - (170978035 / 48384 - 2876425 / 672 * eta - 4735 / 144 * eta ** 2) * dSL)
    ln = math.log(PI) / 3
    b5 = PI * (7729 / 84 - 13 * eta)
    c["pin0"], c["pin1"] = N * PI ** (-5 / 3), 0.0 * N
    c["pin2"] = N * (5 / 9) * (743 / 84 + 11 * eta) / PI
    c["pin3"] = N * (-16 * PI + (188 / 3) * SL + 25 * dSL) * PI ** (-2 / 3)
    c["pin4"] = N * ((5 / 72) * (3058.673 / 7.056 + (5429 / 7) * eta + 617 * eta ** 2) - 10 * sigma) * PI ** (-1 / 3)
    c["lg0"] = N * ((5 / 3) * b5 - 3 * gamma)
    c["lg1"] = N * (-6848 / 21) * PI ** (1 / 3)
    c["pin5"] = N * ((5 / 9) * b5 - gamma) + c["lg0"] * ln - PI / 4
    c["pin6"] = N * v6 * PI ** (1 / 3) + c["lg1"] * ln
    c["pin7"] = N * a7 * PI ** (2 / 3)
    for j, k in enumerate((1.0, 0.75, 0.6, 0.5)):
        c[f"pin{8 + j}"] = k * _fit(4 + j, eta, xi) / eta
    b1, b2, b3 = (_fit(8 + k, eta, xi) for k in range(3))
    c["int0"], c["int1"], c["int2"], c["int3"] = 0.0 * eta, b1 / eta, -b3 / (3 * eta), b2 / eta
    al = [_fit(11 + k, eta, xi) for k in range(5)]
    c["pm0"], c["pm1"], c["pm2"], c["pm3"], c["pm4"] = 0.0 * eta, al[0] / eta, -al[1] / eta, (4 / 3) * al[2] / eta, al[3] / eta
    c["pm5"] = al[4] * c["fRD"]
    f1 = torch.full_like(eta, 0.018)
    (pa, da), (pb, db) = _psi_ins(c, f1), _psi_int(c, f1)
    c["int1"] = c["int1"] + (da - db)
    c["int0"] = pa - pb - (da - db) * f1
    f2 = 0.5 * c["fRD"]
    (pa, da), (pb, db) = _psi_int(c, f2), _psi_mrd(c, c["fDM"], f2)
    c["pm1"] = c["pm1"] + (da - db)
    c["pm0"] = pa - pb - (da - db) * f2
    for j, v in enumerate(_intermediate(c, c["w"], c["fpeak"])):
        c[f"dl{j}"] = v

    def at(f):  # per sample: the branch that f lies in
        p = [_psi_ins(c, f), _psi_int(c, f), _psi_mrd(c, c["fDM"], f)]
        return [torch.where(f < 0.018, x, torch.where(f < 0.5 * c["fRD"], y, z)) for x, y, z in zip(*p)]

    t0 = at(c["fpeak"])[1]
    fr = c["Msec"] * 1e-4
    shift = t0 * fr - at(fr)[0] - 2 * th[:, 9]
    for name, by in (("pin5", shift), ("int0", shift), ("pm0", shift), ("pin8", -t0), ("int1", -t0), ("pm1", -t0)):
        c[name] = c[name] + by
    c["scale"] = (2 * math.sqrt(5 / (64 * PI)) / PI ** (1 / 6) * (M * MRSUN) * (M * MTSUN)
                  / (torch.exp(th[:, 4]) * 1e6 * PC) * torch.sqrt(eta * 2 / 3))
    c["P0"], c["C0"] = 0.5 * (1 + th[:, 5] ** 2), -th[:, 5]
    c["top"] = c["fRD"]
    return c


def _ylm(l, m, ci):
    """Spin -2 spherical harmonic at azimuth 0."""
    fac, ch, sh, total = math.factorial, torch.sqrt(0.5 * (1 + ci)), torch.sqrt(0.5 * (1 - ci)), 0.0
    for k in range(l + m + 1):
        if l - 2 - k >= 0 and k + 2 - m >= 0:
            total = total + ((-1) ** k * math.sqrt(fac(l + m) * fac(l - m) * fac(l + 2) * fac(l - 2))
                             / (fac(l + m - k) * fac(l - 2 - k) * fac(k) * fac(k + 2 - m))
                             * ch ** (2 * l + m - 2 * k - 2) * sh ** (2 * k + 2 - m))
    return math.sqrt((2 * l + 1) / (4 * PI)) * total


def _phenomhm(th, c):
    """Adds the modes' coefficients of IMRPhenomHM to IMRPhenomD's: keys with the mode's number at their end."""
    c["dlt"] = (th[:, 1] - 1) / (th[:, 1] + 1)
    c["chis"], c["chia"] = 0.5 * (th[:, 2] + th[:, 3]), 0.5 * (th[:, 2] - th[:, 3])
    nrm = 4 * math.sqrt(5 / (64 * PI))
    for k, (l, m, _) in enumerate(_MODES):
        yp, ym = _ylm(l, m, th[:, 5]), _ylm(l, -m, th[:, 5])
        c[f"P{k}"], c[f"C{k}"] = ((-1) ** l * ym + yp) / nrm, ((-1) ** l * ym - yp) / nrm
        if k == 0:
            continue
        wr, wi = _qnm(k, c["af"])
        frd, fdm = wr / (2 * PI) / (1 - c["erad"]), wi / (2 * PI) / (1 - c["erad"])
        c["top"] = torch.maximum(c["top"], frd)
        R = c["fRD"] / frd
        c[f"R{k}"], c[f"fDM{k}"] = R, R * fdm
        c[f"w{k}"] = c["w"] / c["fDM"] * c[f"fDM{k}"]
        c[f"fpeak{k}"] = _peak(c, c[f"w{k}"])
        for j, v in enumerate(_intermediate(c, c[f"w{k}"], c[f"fpeak{k}"])):
            c[f"dl{k}_{j}"] = v
        c[f"frA{k}"] = c[f"fpeak{k}"] / R
        fi, fr = 0.5 * m * 0.018 + 0 * R, 0.5 * c["fRD"] / R
        a = (0.5 * c["fRD"] - 0.018) / (fr - fi)
        b = 0.018 - a * fi
        c[f"frP{k}"], c[f"aP{k}"], c[f"bP{k}"] = fr, a, b
        # the maps' ends are the (2,2) phase's own joins, which it passes with continuous value and slope
        v1, d1 = _psi_ins(c, torch.full_like(R, 0.018))
        c[f"cI1{k}"] = d1 - d1
        c[f"cI0{k}"] = 0.5 * m * v1 - v1 / a
        vb, db = _psi_mrd(c, c["fDM"], 0.5 * c["fRD"])
        vr, dr = _psi_mrd(c, c[f"fDM{k}"], 0.5 * c["fRD"])
        c[f"cR1{k}"] = db - dr
        c[f"cR0{k}"] = vb / a + c[f"cI0{k}"] - vr / R - (db - dr) * fr
    return c


def _ratio(k, v, c):
    eta, d, v2 = c["eta"], c["dlt"], v * v
    h22 = 1 + v2 * (-107 / 42 + 55 / 42 * eta) + 2 * PI * v ** 3
    if k == 1:
        r = (d * v * (1 + v2 * (-17 / 28 + 5 / 7 * eta)) - 1.5 * (c["chia"] + d * c["chis"]) * v2) / 3 * math.sqrt(2)
    elif k == 2:
        r = 0.75 * math.sqrt(15 / 14) * d * v * (1 + v2 * (-4 + 2 * eta)) * math.sqrt(2 / 3)
    elif k == 3:
        r = math.sqrt(5 / 7) / 3 * v2 * (1 - 3 * eta)
    elif k == 4:
        r = 8 / 9 * math.sqrt(5 / 7) * v2 * (1 - 3 * eta) * math.sqrt(0.5)
    else:
        r = 9 / (4 * math.sqrt(70)) * d * v ** 3 * (1 - 2 * eta) * math.sqrt(2 / 3)
    return r / h22


def _mode(c, k, Mf):
    """(amplitude, phase, dPhase/dMf, mapped frequency) of mode k of one sample on ascending Mf."""
    if k == 0:
        p, d = _psi(c, Mf)
        return _amp(c, Mf, c["w"], c["fpeak"], "dl"), p, d, Mf
    m, R, fi, fr = _MODES[k][1], c[f"R{k}"], 0.5 * _MODES[k][1] * 0.014, c[f"frA{k}"]
    tm, h = 2 / m, fr - fi

    def blend(x):
        s = (x - fi) / h
        return ((2 * s ** 3 - 3 * s ** 2 + 1) * (tm * fi) + (s ** 3 - 2 * s ** 2 + s) * (h * tm)
                + (3 * s ** 2 - 2 * s ** 3) * (R * fr) + (s ** 3 - s ** 2) * (h * R))

    y = _pieces(Mf, (fi, fr), (lambda x: tm * x, blend, lambda x: R * x))
    fb = torch.where(Mf <= fi, Mf, fi * (2 - torch.exp(1 - Mf / fi)))
    amp = _ratio(k, (2 * PI / m * fb) ** (1 / 3), c) * _amp(c, y, c[f"w{k}"], c[f"fpeak{k}"], f"dl{k}_")

    def low(x):
        p, d = _psi(c, tm * x)
        return 0.5 * m * p, d

    def mid(x):
        p, d = _psi(c, c[f"aP{k}"] * x + c[f"bP{k}"])
        return p / c[f"aP{k}"] + c[f"cI0{k}"] + c[f"cI1{k}"] * x, d + c[f"cI1{k}"]

    def high(x):
        p, d = _psi_mrd(c, c[f"fDM{k}"], R * x)
        return p / R + c[f"cR0{k}"] + c[f"cR1{k}"] * x, d + c[f"cR1{k}"]

    p, d = _pieces(Mf, (0.5 * m * 0.018, c[f"frP{k}"]), (low, mid, high))
    return amp, p + 0.5 * PI * _MODES[k][2], d, y


def _nodes(name, t):
    """Node positions (3 nodes, 3 axes) in light-seconds at times t."""
    al = 2 * PI / YEAR * t + {"LISA": -PI / 9, "Taiji": PI / 9, "TianQin": 0.0}[name]
    c, s, L = torch.cos(al), torch.sin(al), ARM[name] / C_SI
    out = []
    for k in range(3):
        kap = 2 * PI * k / 3
        if name == "TianQin":
            ph = 2 * PI / (3.65 * 86400.0) * t + kap
            ck, sk, r, lr, br = torch.cos(ph), torch.sin(ph), L / math.sqrt(3), 120.5 / 180 * PI, -4.7 / 180 * PI
            x = [r * (math.sin(br) * math.cos(lr) * sk + math.sin(lr) * ck),
                 r * (math.sin(br) * math.sin(lr) * sk - math.cos(lr) * ck), -r * math.cos(br) * sk]
        else:
            ck, sk, r = math.cos(kap), math.sin(kap), L / (2 * math.sqrt(3))
            x = [r * (s * c * sk - (1 + s * s) * ck), r * (s * c * ck - (1 + c * c) * sk), -r * math.sqrt(3) * (c * ck + s * sk)]
        out.append([x[0], x[1], x[2]])
    return out, [c * (AU / C_SI), s * (AU / C_SI)]


def _combine(f, name, generation, L):
    """A/E/T from the links 12, 21, 23, 32, 31, 13."""
    D = torch.polar(torch.ones_like(f), -2 * PI * f * (ARM[name] / C_SI))
    pre = 1 - D ** 2 if generation == "1.5" else 1 - D ** 2 - D ** 4 + D ** 6
    X = pre * ((L[5] - L[0]) + D * (L[4] - L[1]))
    Y = pre * ((L[1] - L[2]) + D * (L[0] - L[3]))
    Z = pre * ((L[3] - L[4]) + D * (L[2] - L[5]))
    return torch.stack([(Z - X) / math.sqrt(2), (X - 2 * Y + Z) / math.sqrt(6), (X + Y + Z) / math.sqrt(3)])


def _respond(f, name, hp, hc, tf, th):
    """The six single-link responses of one mode (already shifted to t_c)."""
    x, x0 = _nodes(name, tf)
    L = ARM[name] / C_SI
    lam, sb, psi = th[6], th[7], th[8]
    cb, sl, cl, sp, cp = torch.sqrt(1 - sb * sb), torch.sin(lam), torch.cos(lam), torch.sin(psi), torch.cos(psi)
    p = [sl * cp - cl * sb * sp, -cl * cp - sl * sb * sp, cb * sp]
    q = [-sl * sp - cl * sb * cp, cl * sp - sl * sb * cp, cb * cp]
    k = [-cb * cl, -cb * sl, -sb]
    dot = lambda a, b: a[0] * b[0] + a[1] * b[1] + a[2] * b[2]  # noqa: E731
    kx0 = k[0] * x0[0] + k[1] * x0[1]
    out = []
    for a, b in ((0, 1), (1, 2), (2, 0)):  # links a+1 -> b+1 and back
        n = [(v - u) / L for u, v in zip(x[a], x[b])]
        np_, nq, kn = dot(n, p), dot(n, q), dot(n, k)
        strain = (np_ ** 2 - nq ** 2) * hp + 2 * np_ * nq * hc
        ph = -PI * f * (L + 2 * kx0 + dot(k, x[a]) + dot(k, x[b]))
        common = -1j * PI * f * L * strain * torch.polar(torch.ones_like(f), ph)
        out += [torch.sinc(f * L * (1 + kn)) * common, torch.sinc(f * L * (1 - kn)) * common]
    return out


def _model(case, f, c, th, dets):
    """A/E/T of every detector for one sample on the bins below its cut, f ascending; a list of (3, n) tensors."""
    Mf = c["Msec"] * f
    shift = torch.polar(torch.ones_like(f), -2 * PI * f * th[10])
    modes = []
    for k in range(6 if case["approximant"] == "HM" else 1):
        amp, psi, dpsi, y = _mode(c, k, Mf)
        h = torch.where(y <= 0.2, amp, 0.0 * amp) * torch.polar(torch.ones_like(f), -psi) * shift
        modes.append((c[f"P{k}"] * h, 1j * c[f"C{k}"] * h, c["Msec"] * dpsi / (2 * PI) + th[10]))
    out = []
    for name in dets:
        L = [sum(v) for v in zip(*(_respond(f, name, *m, th) for m in modes))]
        out.append(_combine(f, name, case["generation"], L))
    return out


def _live(case, f, c):
    """Bins of one sample that carry a model."""
    top = 0.2 / c["Msec"]
    if case["approximant"] == "HM":
        top = max(top, *(top / c[f"R{k}"] for k in range(1, 6)))
    if case.get("cut", 0.0) > 0:
        top = torch.minimum(top, case["cut"] * c["top"] / c["Msec"])
    return int(torch.searchsorted(f, top.detach().reshape(()), right=True))


def _coefficients(case, th):
    c = _phenomd(th)
    return _phenomhm(th, c) if case["approximant"] == "HM" else c


def _dataset(case, seed, f, dets):
    inj = torch.as_tensor(_injection(case), device=DEV)
    whole = {**case, "cut": 0.0}
    c = {k: v[0] for k, v in _coefficients(case, inj[None]).items()}
    n = _live(whole, f, c)
    h = _model(whole, f[:n], c, inj, dets)
    data, psd = [], []
    for k, name in enumerate(dets):
        d = _noise(case, seed, k, f)
        d[:, :n] += h[k]
        data.append(d)
        psd.append(_psd(name, f, case["generation"]))
    return data, psd


def _exact_td(case, seed):
    arm, dt, m = ARM[case["arm"]] / C_SI, case["dt"], 7 if case["generation"] == "2.0" else 3
    added, n = int(m * arm // dt + 1), case["n"]
    links = _links(case, seed, added)

    def term(l, k):  # link l delayed by k arms, linear between samples
        if k == 0:
            return links[l, added:added + n]
        s, w = int((m - k) * arm // dt), 1 - k * arm % dt / dt
        return links[l, s:s + n] + (links[l, s + 1:s + 1 + n] - links[l, s:s + n]) * w

    plus, minus = (5, 4, 0, 1, 0, 1, 5, 4), (0, 1, 5, 4, 5, 4, 0, 1)
    ch = [sum(term((plus[k] + 2 * c) % 6, k) - term((minus[k] + 2 * c) % 6, k) for k in range(m + 1)) for c in range(3)]
    X, Y, Z = ch
    if case["orthogonal"]:
        ch = [(Z - X) / math.sqrt(2), (X - 2 * Y + Z) / math.sqrt(6), (X + Y + Z) / math.sqrt(3)]
    return torch.stack(ch)


def exact(case, seed):
    if case["kind"] == "td_tdi":
        return _exact_td(case, seed)
    if _qnm_table() is None:
        return None
    dets = _dets(case)
    f = torch.as_tensor(_grid(case), device=DEV)
    th = torch.as_tensor(_thetas(case, seed), device=DEV)
    df = 1.0 / case["duration"]
    if case["kind"] == "driver":
        data, psd = _dataset(case, seed, f, dets)
        c = {k: v[0] for k, v in _coefficients(case, th).items()}
        n = _live(case, f, c)
        out, logl = [], 0.0
        for h, d, S in zip(_model(case, f[:n], c, th[0], dets), data, psd):
            full = torch.zeros_like(d)
            full[:, :n] = h
            out.append(full)
            logl += float(-2 * df * ((d - full).abs() ** 2 / S).sum())
        return [logl] + out
    if case["call"] == "fisher":
        return _exact_fisher(case, f, th, dets, df)
    data, psd = _dataset(case, seed, f, dets)
    grad = case["call"] == "grad"
    th = th.requires_grad_(grad)
    with torch.set_grad_enabled(grad):
        c = _coefficients(case, th)
    names = sorted(c)
    # every sample's bins hang on a copy of its coefficients, so that only one sample's graph is held at a time
    leaf = torch.stack([c[k].detach() for k in names], 1).requires_grad_(grad)
    own = th.detach().clone().requires_grad_(grad)
    # sums over the bins that a sample's model does not reach
    tail = [torch.cat([(d.abs() ** 2 / S).sum(0).flip(0).cumsum(0).flip(0), torch.zeros(1, dtype=F64, device=DEV)]) for d, S in zip(data, psd)]
    lnl = []
    for b in range(th.shape[0]):
        with torch.set_grad_enabled(grad):
            cb = dict(zip(names, leaf[b]))
            n = _live(case, f, cb)
            total = sum(t[n] for t in tail)
            if n > 0:
                for h, d, S in zip(_model(case, f[:n], cb, own[b], dets), data, psd):
                    r = d[:, :n] - h
                    total = total + ((r.real ** 2 + r.imag ** 2) / S[:, :n]).sum()
            value = -2 * df * total
            lnl.append(value.detach())
            if grad and n > 0:
                value.backward()
    lnl = torch.stack(lnl)
    if case["call"] == "params":
        return float(lnl[0])
    if not grad:
        return lnl
    through = torch.autograd.grad([c[k] for k in names], th, [leaf.grad[:, i] for i in range(len(names))], allow_unused=True)[0]
    return lnl, through + own.grad


def _exact_fisher(case, f, th, dets, df):
    import torch.autograd.forward_ad as fwd

    psd = [_psd(name, f, case["generation"]) for name in dets]
    jets = []
    with fwd.dual_level():
        for a in range(11):
            e = torch.zeros_like(th)
            e[:, a] = 1.0
            c = _coefficients(case, fwd.make_dual(th, e))
            jets.append({k: fwd.unpack_dual(v) for k, v in c.items()})
    out = torch.zeros((th.shape[0], 11, 11), dtype=F64, device=DEV)
    for b in range(th.shape[0]):
        n = _live(case, f, {k: v.primal[b] for k, v in jets[0].items()})
        rows = []
        for a in range(11):
            with fwd.dual_level():
                c = {k: fwd.make_dual(v.primal[b].clone(), v.tangent[b].clone()) if v.tangent is not None else v.primal[b]
                     for k, v in jets[a].items()}
                e = torch.zeros_like(th[b])
                e[a] = 1.0
                h = _model(case, f[:n], c, fwd.make_dual(th[b].clone(), e), dets)
                rows.append(torch.cat([fwd.unpack_dual(v).tangent / torch.sqrt(S[:, :n]) for v, S in zip(h, psd)]).reshape(-1))
        J = torch.view_as_real(torch.stack(rows)).reshape(11, -1)
        out[b] = 4 * df * (J @ J.T)
    return out
