"""Sampling calls that a user of gbsgmc makes, with their sizes, inputs and
exact values, for measuring the framework.

Three groups, all through the public entry points:

* whole sampler runs: ``alias.sgld / obabo / sghmc / re_sgld / amagold`` on
  the generalised-linear likelihoods, ``alias.obabo`` on the tanh network and
  the CNN, ``alias.re_sgld_ladder`` on the tanh network;
* one batched value and gradient of each likelihood family
  (``StochasticPotential.evaluate`` / ``value_and_grad``), which is what an
  integrator of a user's own calls;
* sizes from one chain on 32 features up to the shapes of the benchmark
  (256 logistic chains on 10^6 x 256, 64 chains of the 64-1024-1024-1
  network, 8 chains of the CNN), odd ones among them.
"""

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PACKAGE = str(Path(__file__).resolve().parents[1] / "jax-sgmc_gb300")
if _PACKAGE not in sys.path:
  sys.path.insert(0, _PACKAGE)

from gbsgmc import alias, data, likelihoods, potential  # noqa: E402


def listed():
  return [
      # Bayesian linear regression, one chain: the smallest run a user
      # starts (a first model, a convergence check); a step is a few
      # microseconds, so latency is all there is.
      dict(name="sgld_linear_1", kind="sgld", family="linear", chains=1,
           n_obs=10_000, features=32, batch=128, iterations=1000, kept=100,
           rms=True),
      # Bayesian logistic regression with many chains on data far larger
      # than L2: the framework's headline workload, as the whole call.
      dict(name="sgld_logistic_256", kind="sgld", family="logistic",
           chains=256, n_obs=1_000_000, features=256, batch=1024,
           iterations=200, kept=10, rms=True),
      # OBABO on a mid-sized logistic model with odd feature and batch
      # sizes, a couple of dozen chains (posterior with diagnostics).
      dict(name="obabo_logistic_24", kind="obabo", family="logistic",
           chains=24, n_obs=100_000, features=101, batch=500, iterations=20,
           kept=5, rms=False),
      # SGHMC on a small linear model, a handful of chains.
      dict(name="sghmc_linear_4", kind="sghmc", family="linear", chains=4,
           n_obs=20_000, features=57, batch=200, iterations=30, kept=10,
           rms=False),
      # Replica exchange with (normal, hot) pairs.
      dict(name="re_sgld_logistic_8", kind="re_sgld", family="logistic",
           chains=8, n_obs=50_000, features=64, batch=256, iterations=200,
           kept=20, rms=False),
      # AMAGOLD: minibatch proposals with a full-data correction for every
      # chain after each trajectory.
      dict(name="amagold_logistic_16", kind="amagold", family="logistic",
           chains=16, n_obs=100_000, features=64, batch=256, iterations=8,
           kept=8, rms=False),
      # One minibatch potential and gradient of one sample: the call in a
      # user's own integrator loop, all latency.
      dict(name="gradient_linear_1", kind="glm_grad", family="linear",
           chains=1, n_obs=10_000, features=33, batch=128),
      # One batched gradient of the benchmark's tanh network (64 chains of
      # 64-1024-1024-1, minibatch 2048): the tensor-core work of an OBABO
      # or SGHMC step.
      dict(name="gradient_mlp_64", kind="mlp_grad", chains=64,
           n_obs=500_000, d_in=64, h1=1024, h2=1024, batch=2048),
      # The same on a small network of unequal widths, few chains, a batch
      # that is no power of two: most user networks.
      dict(name="gradient_mlp_3", kind="mlp_grad", chains=3, n_obs=50_000,
           d_in=64, h1=512, h2=256, batch=384),
      # Replica exchange over a temperature ladder on the tanh network with
      # uneven minibatches (64 to 4096 rows): the tempering benchmark.
      dict(name="ladder_mlp_32", kind="mlp_ladder", chains=32,
           n_obs=500_000, d_in=64, h1=1024, h2=1024, batch=4096,
           iterations=50),
      # One batched gradient of the CNN classifier at the benchmark's size.
      dict(name="gradient_cnn_8", kind="cnn_grad", chains=8, n_obs=20_000,
           batch=256),
      # A short OBABO run of a few CNN chains at a small batch.
      dict(name="obabo_cnn_2", kind="cnn_obabo", chains=2, n_obs=10_000,
           batch=50, iterations=5),
  ]


def _log_int(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
  kind = rng.choice(["sgld", "sgld", "obabo", "sghmc", "re_sgld", "amagold",
                     "glm_grad", "glm_grad", "mlp_grad", "mlp_grad",
                     "mlp_ladder", "cnn_grad", "cnn_grad", "cnn_obabo"])
  if kind in ("mlp_grad", "mlp_ladder"):
    case = dict(kind=kind, n_obs=_log_int(rng, 20_000, 500_000),
                d_in=64 * rng.choice([1, 1, 2]),
                h1=256 * rng.randint(1, 4), h2=256 * rng.randint(1, 4))
    if kind == "mlp_grad":
      case["chains"] = _log_int(rng, 1, 48)
      case["batch"] = 128 * _log_int(rng, 1, 16)
    else:
      case["chains"] = _log_int(rng, 4, 24)
      case["batch"] = 128 * _log_int(rng, 4, 32)
      case["iterations"] = 10 * rng.randint(2, 5)
    return case
  if kind == "cnn_grad":
    return dict(kind=kind, chains=_log_int(rng, 1, 8),
                n_obs=_log_int(rng, 5_000, 20_000),
                batch=2 * _log_int(rng, 8, 128))
  if kind == "cnn_obabo":
    return dict(kind=kind, chains=_log_int(rng, 1, 4),
                n_obs=_log_int(rng, 5_000, 20_000),
                batch=2 * _log_int(rng, 8, 64), iterations=rng.randint(2, 5))
  case = dict(kind=kind, family=rng.choice(["linear", "logistic"]),
              n_obs=_log_int(rng, 5_000, 200_000),
              features=_log_int(rng, 8, 256))
  if kind == "glm_grad":
    case["chains"] = _log_int(rng, 1, 256)
    case["batch"] = _log_int(rng, 32, 1500)
    return case
  if kind == "amagold":
    case["family"] = "logistic"
    case["chains"] = _log_int(rng, 1, 32)
    case["features"] = _log_int(rng, 8, 128)
  elif kind == "re_sgld":
    case["chains"] = _log_int(rng, 1, 32)
  else:
    case["chains"] = _log_int(rng, 1, 256 if kind == "sgld" else 64)
  case["batch"] = _log_int(rng, 32, 1024 if kind == "sgld" else 512)
  case["iterations"] = {"sgld": rng.randint(50, 500), "re_sgld": rng.randint(50, 300),
                        "amagold": rng.randint(2, 8)}.get(kind, rng.randint(5, 30))
  case["kept"] = max(1, case["iterations"] // 10) if kind != "amagold" \
      else case["iterations"]
  case["rms"] = kind == "sgld" and rng.random() < 0.7
  return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

_SIGMA = 0.5          # noise of the linear model
_MLP_SIGMA = 0.1
_STEPS = 10           # integrator steps per iteration (alias's default)


def _gen(seed, stream):
  return torch.Generator(device="cuda").manual_seed(1_000_003 * seed + stream)


def _randn(g, *shape):
  return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)


def _glm_data(case, seed):
  """Standard normal features; targets from a teacher w* ~ N(0, 1/d)."""
  N, d = case["n_obs"], case["features"]
  g = _gen(seed, 1)
  X = _randn(g, N, d)
  z = (X * (_randn(g, d) / math.sqrt(d))).sum(1)
  if case["family"] == "linear":
    y = z + _SIGMA * _randn(g, N)
  else:
    y = (torch.rand(N, generator=g, device="cuda") < torch.sigmoid(z)).float()
  return X, y


def _glm_start(case, seed, rows):
  return 0.1 * _randn(_gen(seed, 2), rows, case["features"])


def _mlp_widths(case):
  return case["d_in"], case["h1"], case["h2"]


def _mlp_split(w, D, H1, H2):
  """The leaves of flat parameter rows [C, P]: W1, W2, W3, b1, b2, b3."""
  C, out, o = w.shape[0], [], 0
  for shape in ((D, H1), (H1, H2), (H2,), (H1,), (H2,), (1,)):
    k = math.prod(shape)
    out.append(w[:, o:o + k].reshape((C,) + shape))
    o += k
  return out


def _mlp_weights(g, C, D, H1, H2):
  return torch.cat([_randn(g, C, D * H1) / math.sqrt(D),
                    _randn(g, C, H1 * H2) / math.sqrt(H1),
                    _randn(g, C, H2) / math.sqrt(H2),
                    torch.zeros(C, H1 + H2 + 1, device="cuda")], 1)


def _mlp_data(case, seed):
  """Inputs ~ N(0, 1), targets from a random network of the same shape."""
  D, H1, H2 = _mlp_widths(case)
  g = _gen(seed, 3)
  X = _randn(g, case["n_obs"], D)
  W1, W2, W3, _, _, _ = (t[0] for t in _mlp_split(_mlp_weights(g, 1, D, H1, H2), D, H1, H2))
  y = torch.cat([torch.tanh(torch.tanh(x @ W1) @ W2) @ W3 for x in X.split(65536)])
  return X, y + _MLP_SIGMA * _randn(g, case["n_obs"])


def _cnn_data(case, seed):
  """Images ~ N(0, 1), labels uniform over ten classes."""
  g = _gen(seed, 4)
  return (_randn(g, case["n_obs"], 32, 32, 3),
          torch.randint(0, 10, (case["n_obs"],), generator=g, device="cuda").float())


_CNN_LEAVES = (("b", (32,)), ("w", (3, 3, 3, 32)), ("b", (64,)), ("w", (3, 3, 32, 64)),
               ("b", (128,)), ("w", (3, 3, 64, 128)), ("b", (10,)), ("w", (2048, 10)))


def _cnn_weights(g, C):
  parts = []
  for name, shape in _CNN_LEAVES:
    k = math.prod(shape)
    parts.append(0.01 * _randn(g, C, k) if name == "b" else
                 _randn(g, C, k) * math.sqrt(2.0 / math.prod(shape[:-1])))
  return torch.cat(parts, 1)


def _indices(case, seed):
  return torch.randint(0, case["n_obs"], (case["chains"], case["batch"]),
                       generator=_gen(seed, 5), device="cuda", dtype=torch.int32)


def _ladder(case):
  """Geometric temperatures 1 to 100 and uneven minibatch sizes."""
  R = case["chains"]
  temps = 100.0 ** (np.arange(R) / (R - 1))
  rows = np.random.default_rng(R).integers(64, case["batch"] + 1, R)
  return temps, rows.astype(np.int32)


def _glm_family(case):
  return likelihoods.LinearGaussian(sigma=_SIGMA) if case["family"] == "linear" \
      else likelihoods.Logistic()


# Step sizes (first, last): stable for unit-variance features at N
# observations, whose potential has curvature of about N / sigma^2 (linear)
# or N / 4 (logistic).
def _step_sizes(case):
  curvature = case["n_obs"] * (1 / _SIGMA ** 2 if case.get("family") == "linear" else 0.25)
  if case["kind"] in ("sgld", "re_sgld"):
    return (1e-3, 1e-4) if case["rms"] else (0.1 / curvature, 0.05 / curvature)
  h = 0.05 / math.sqrt(curvature)
  return (h, 0.5 * h) if case["kind"] in ("obabo", "sghmc") else (0.2 * h, 0.1 * h)


def _host(*tensors):
  return [t.cpu().numpy() for t in tensors]


def prepare(case, seed):
  kind, C = case["kind"], case["chains"]
  if kind.startswith("mlp"):
    D, H1, H2 = _mlp_widths(case)
    X, y = _host(*_mlp_data(case, seed))
    loader = data.NumpyDataLoader(copy=False, x=X, y=y)
    lik = likelihoods.MLPGaussian(d_in=D, h1=H1, h2=H2, sigma=_MLP_SIGMA)
    pot = potential.minibatch_potential(likelihoods.GaussianPrior(1.0), lik)
    dataset = loader.device_dataset()
    dataset.glm_view("x", "y")
    g = _gen(seed, 6)
    if kind == "mlp_grad":
      return dict(kind=kind, pot=pot, W=_mlp_weights(g, C, D, H1, H2),
                  idx=_indices(case, seed), dataset=dataset)
    temps, rows = _ladder(case)
    start = lik.unravel(_mlp_weights(g, 1, D, H1, H2)[0].cpu().numpy())
    sampler = alias.re_sgld_ladder(pot, loader, temps, batch_sizes=rows,
                                   exchange_every=10, first_step_size=1e-3,
                                   last_step_size=5e-4, rms_prop=True,
                                   burn_in=case["iterations"] - 10, accepted_samples=10)
    return dict(kind=kind, sampler=sampler, start=[start], iterations=case["iterations"])
  if kind.startswith("cnn"):
    images, labels = _host(*_cnn_data(case, seed))
    loader = data.NumpyDataLoader(copy=False, image=images, label=labels)
    lik = likelihoods.CNNSoftmax()
    pot = potential.minibatch_potential(likelihoods.GaussianPrior(1.0), lik)
    dataset = loader.device_dataset()
    dataset.glm_view("image", "label")
    W = _cnn_weights(_gen(seed, 6), C)
    if kind == "cnn_grad":
      return dict(kind=kind, pot=pot, W=W, idx=_indices(case, seed), dataset=dataset)
    sampler = alias.obabo(pot, loader, cache_size=50, batch_size=case["batch"],
                          integration_steps=_STEPS, first_step_size=1e-4,
                          last_step_size=5e-5, burn_in=case["iterations"] - 1,
                          accepted_samples=1, progress_bar=False)
    return dict(kind=kind, sampler=sampler, iterations=case["iterations"],
                start=[lik.unravel(w) for w in W.cpu().numpy()])
  X, y = _host(*_glm_data(case, seed))
  loader = data.NumpyDataLoader(copy=False, x=X, y=y)
  prior = likelihoods.GaussianPrior(1.0)
  pot = potential.minibatch_potential(prior, _glm_family(case))
  dataset = loader.device_dataset()
  dataset.matrix("x"), dataset.vector("y")
  if kind == "glm_grad":
    W, idx = _glm_start(case, seed, C), _indices(case, seed)
    if C == 1:
      info = data.MiniBatchInformation(case["n_obs"], None, case["batch"])
      return dict(kind="glm_value", pot=pot, w=W[0],
                  batch=(data.IndexedBatch(dataset, idx[0], loader), info))
    return dict(kind=kind, pot=pot, W=W, idx=idx, dataset=dataset)
  first, last = _step_sizes(case)
  its, kept = case["iterations"], case["kept"]
  opts = dict(cache_size=50, batch_size=case["batch"], first_step_size=first,
              last_step_size=last, burn_in=its - kept, accepted_samples=kept,
              progress_bar=False)
  pairs = 2 if kind == "re_sgld" else 1
  rows = _glm_start(case, seed, C * pairs).cpu().numpy()
  start = [{"w": w} for w in rows]
  if kind == "sgld":
    sampler = alias.sgld(pot, loader, rms_prop=case["rms"], **opts)
  elif kind == "re_sgld":
    sampler = alias.re_sgld(pot, loader, temperature=100.0, **opts)
    start = list(zip(start[0::2], start[1::2]))
  elif kind == "amagold":
    full = potential.full_potential(prior, _glm_family(case))
    sampler = alias.amagold(pot, full, loader, integration_steps=_STEPS,
                            friction=0.25, **opts)
  else:
    make = alias.obabo if kind == "obabo" else alias.sghmc
    sampler = make(pot, loader, integration_steps=_STEPS, **opts)
  return dict(kind=kind, sampler=sampler, start=start, iterations=its)


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def _leaves(tree):
  if isinstance(tree, dict):
    return [x for k in sorted(tree) for x in _leaves(tree[k])]
  return [tree]


def run(state):
  kind = state["kind"]
  if kind == "glm_value":
    (U, _), grad = state["pot"].value_and_grad(state["w"], state["batch"])
    return {"U": U, "grad": grad}
  if kind.endswith("_grad"):
    r = state["pot"].evaluate(state["W"], state["idx"], state["dataset"])
    return {"U": r.U, "grad": r.grad, "variance": r.lk_var}
  chains = state["sampler"](*state["start"], iterations=state["iterations"])
  # The chains' samples as one array per parameter, as a user's diagnostics
  # take them.  The potential along a chain is stored as float32, like the
  # samples it belongs to: chains run in float32, and their launch shapes
  # are timed anew in each process.
  samples = [_leaves(c["samples"]["variables"]) for c in chains]
  key = "likelihood" if "likelihood" in chains[0]["samples"] else "energy"
  return {"variables": [np.stack(leaf) for leaf in zip(*samples)],
          key: np.stack([c["samples"][key] for c in chains]).astype(np.float32)}


def work(case):
  """Bytes and flops of one pass: every gathered row, gradient and update
  the algorithm needs, once."""
  kind, C = case["kind"], case["chains"]
  if kind.startswith("mlp"):
    D, H1, H2 = _mlp_widths(case)
    P, mat = D * H1 + H1 * H2 + 2 * H2 + H1 + 1, D * H1 + H1 * H2 + H2
    if kind == "mlp_grad":
      rows, steps, per = C * case["batch"], 1, 8   # read w, write gradient
    else:
      rows, steps, per = int(_ladder(case)[1].sum()), case["iterations"], 16  # x and v
    return {"bytes": float(steps * (rows * (4 * D + 8) + per * C * P)),
            "flops": float(steps * 6 * rows * mat)}
  if kind.startswith("cnn"):
    P = sum(math.prod(s) for _, s in _CNN_LEAVES)
    mat = 1024 * 27 * 32 + 256 * 288 * 64 + 64 * 576 * 128 + 2048 * 10
    grads = 1 if kind == "cnn_grad" else 2 * _STEPS * case["iterations"]
    rows = C * case["batch"] * grads
    # The first layer needs no input gradient.
    return {"bytes": float(rows * (4 * 3072 + 8) + 8 * C * P * grads),
            "flops": float(rows * (6 * mat - 2 * 1024 * 27 * 32))}
  d, n = case["features"], case["batch"]
  row = 4 * d + 8   # features, target, index
  if kind == "glm_grad":
    return {"bytes": float(C * (n * row + 8 * d)), "flops": float(4 * C * n * d)}
  its = case["iterations"]
  grads = {"sgld": 1, "re_sgld": 2, "obabo": 2 * _STEPS}.get(kind, _STEPS) * its * C
  data_rows = grads * n
  flops = 4.0 * d * data_rows
  nbytes = float(data_rows * row + grads * 16 * d)
  if kind == "amagold":   # the full data once an iteration and at the start
    flops += 2.0 * d * C * case["n_obs"] * (its + 1)
    nbytes += case["n_obs"] * (4.0 * d + 4) * (its + 1)
  return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# Exact values in 64 bits
# ---------------------------------------------------------------------------

def _prior_grad_and_energy(w, scale=1.0):
  """-log N(w | 0, scale^2) summed over the row, and its gradient."""
  d = w.shape[1]
  return (0.5 * (w / scale) ** 2).sum(1) + d * math.log(scale * math.sqrt(2 * math.pi)), \
      w / scale ** 2


def _glm_exact(case, X, y, w, idx):
  """U, gradient and variance of the likelihoods of chains w [C, d]."""
  xb = X[idx]
  yb = y[idx].double()
  xb = xb.double()
  z = torch.einsum("cnd,cd->cn", xb, w)
  if case["family"] == "linear":
    lk = -0.5 * ((yb - z) / _SIGMA) ** 2 - math.log(_SIGMA * math.sqrt(2 * math.pi))
    dz = (yb - z) / _SIGMA ** 2
  else:
    lk = yb * z - torch.nn.functional.softplus(z, threshold=50.0)
    dz = yb - torch.sigmoid(z)
  scale = case["n_obs"] / idx.shape[1]
  e, ge = _prior_grad_and_energy(w)
  return (-scale * lk.sum(1) + e, ge - scale * torch.einsum("cn,cnd->cd", dz, xb),
          lk.var(1, unbiased=False))


def _normals(chains, step, tag, d):
  """Philox4x32-10 normals [C, d] of key 0: counter (group of four
  parameters, step, chain, tag), Box-Muller on the word pairs."""
  groups = (d + 3) // 4
  m = np.uint64(0xFFFFFFFF)
  c = [np.tile(np.arange(groups, dtype=np.uint64), (chains, 1)),
       np.full((chains, groups), step, np.uint64),
       np.repeat(np.arange(chains, dtype=np.uint64)[:, None], groups, 1),
       np.full((chains, groups), tag, np.uint64)]
  for r in range(10):
    k0, k1 = (np.uint64((r * w) & 0xFFFFFFFF) for w in (0x9E3779B9, 0xBB67AE85))
    p, q = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
    c = [(q >> np.uint64(32)) ^ c[1] ^ k0, q & m, (p >> np.uint64(32)) ^ c[3] ^ k1, p & m]
  u = [((v >> np.uint64(9)).astype(np.float64) + 0.5) / 2.0 ** 23 for v in c]
  out = np.empty((chains, groups, 4))
  for i in (0, 2):
    rad, ang = np.sqrt(-2 * np.log(u[i])), 2 * np.pi * u[i + 1]
    out[:, :, i], out[:, :, i + 1] = rad * np.cos(ang), rad * np.sin(ang)
  return torch.from_numpy(out.reshape(chains, -1)[:, :d].copy()).cuda()


def _chain_exact(case, seed):
  """The samples and potentials of a whole SGLD, OBABO or SGHMC run."""
  X, y = _glm_data(case, seed)
  kind, C, N, n, d = (case["kind"], case["chains"], case["n_obs"], case["batch"],
                      case["features"])
  x = _glm_start(case, seed, C).double()
  its, kept = case["iterations"], case["kept"]
  inner = 1 if kind == "sgld" else _STEPS
  draws = 2 if kind == "obabo" else 1
  if C * its * inner * draws * n * d > 2e10:
    return None
  idx = np.empty((C, its * inner * draws, n), np.int64)
  for c in range(C):
    rng = np.random.default_rng(np.random.SeedSequence(c).spawn(1)[0])
    idx[c] = rng.choice(N, size=(its * inner * draws, n))
  idx = torch.from_numpy(idx).cuda()
  first, last = _step_sizes(case)
  g = 0.33
  a1, a2 = first ** (-1 / g), last ** (-1 / g)
  slope = (a2 - a1) / (its - 1)
  hs = (a1 + slope * np.arange(its)) ** -g      # a (b + k)^-gamma through both ends
  v, p = torch.ones_like(x), torch.zeros_like(x)
  xs, es = [], []
  for it in range(its):
    h = float(hs[it])
    if kind == "sghmc":
      p = _normals(C, it * inner, 3, d)
    for j in range(inner):
      k = it * inner + j
      if kind == "sgld":
        U, grad, _ = _glm_exact(case, X, y, x, idx[:, k])
        energy, xi = -U, _normals(C, k, 0, d)
        if case["rms"]:
          v = 0.9 * v + 0.1 * grad ** 2
          G = 1 / (1e-5 + v.sqrt())
          x = x - h * G * grad + (2 * h * G).sqrt() * xi
        else:
          x = x - h * grad + math.sqrt(2 * h) * xi
      elif kind == "obabo":
        keep, inject = math.exp(-0.5 * h), math.sqrt(1 - math.exp(-h))
        U1, g1, _ = _glm_exact(case, X, y, x, idx[:, 2 * k])
        p = keep * p + inject * _normals(C, k, 1, d) - 0.5 * h * g1
        x = x + h * p
        U2, g2, _ = _glm_exact(case, X, y, x, idx[:, 2 * k + 1])
        p = keep * (p - 0.5 * h * g2) + inject * _normals(C, k, 2, d)
        energy = 0.5 * (U1 + U2)
      else:
        x = x + h * p
        p = (1 - h) * p
        energy, grad, _ = _glm_exact(case, X, y, x, idx[:, k])
        p = p - h * grad + math.sqrt(2 * h) * _normals(C, k, 4, d)
    if it >= its - kept:
      xs.append(x)
      es.append(energy)
  return {"variables": [torch.stack(xs, 1)],
          "likelihood" if kind == "sgld" else "energy": torch.stack(es, 1)}


def _mlp_exact(case, seed):
  D, H1, H2 = _mlp_widths(case)
  X, y = _mlp_data(case, seed)
  C, N, n = case["chains"], case["n_obs"], case["batch"]
  W = _mlp_weights(_gen(seed, 6), C, D, H1, H2)
  idx = _indices(case, seed).long()
  U, grad, var = [], [], []
  for c in range(C):
    w = W[c:c + 1].double()
    W1, W2, W3, b1, b2, b3 = (t[0] for t in _mlp_split(w, D, H1, H2))
    xb, yb = X[idx[c]].double(), y[idx[c]].double()
    Z1 = torch.tanh(xb @ W1 + b1)
    Z2 = torch.tanh(Z1 @ W2 + b2)
    res = yb - (Z2 @ W3 + b3)
    lk = -0.5 * (res / _MLP_SIGMA) ** 2 - math.log(_MLP_SIGMA * math.sqrt(2 * math.pi))
    g = -(N / n) * res / _MLP_SIGMA ** 2
    G2 = g[:, None] * W3 * (1 - Z2 ** 2)
    G1 = (G2 @ W2.T) * (1 - Z1 ** 2)
    e, ge = _prior_grad_and_energy(w)
    parts = (xb.T @ G1, Z1.T @ G2, Z2.T @ g, G1.sum(0), G2.sum(0), g.sum())
    U.append(-(N / n) * lk.sum() + e[0])
    grad.append(torch.cat([t.reshape(-1) for t in parts]) + ge[0])
    var.append(lk.var(unbiased=False))
  return {"U": torch.stack(U), "grad": torch.stack(grad), "variance": torch.stack(var)}


def _cnn_exact(case, seed):
  images, labels = _cnn_data(case, seed)
  C, N, n = case["chains"], case["n_obs"], case["batch"]
  W = _cnn_weights(_gen(seed, 6), C)
  idx = _indices(case, seed).long()
  F = torch.nn.functional
  U, grad, var = [], [], []
  for c in range(C):
    w = W[c].double().requires_grad_(True)
    leaves, o = [], 0
    for _, shape in _CNN_LEAVES:
      k = math.prod(shape)
      leaves.append(w[o:o + k].reshape(shape))
      o += k
    a = images[idx[c]].double().permute(0, 3, 1, 2)
    for l in range(3):
      a = F.conv2d(a, leaves[2 * l + 1].permute(3, 2, 0, 1), leaves[2 * l], padding=1)
      a = F.max_pool2d(torch.relu(a), 2)
    logits = a.permute(0, 2, 3, 1).reshape(n, -1) @ leaves[7] + leaves[6]
    lk = torch.log_softmax(logits, 1).gather(1, labels[idx[c]].long()[:, None])[:, 0]
    e, _ = _prior_grad_and_energy(w[None])
    u = -(N / n) * lk.sum() + e[0]
    grad.append(torch.autograd.grad(u, w)[0])
    U.append(u.detach())
    var.append(lk.detach().var(unbiased=False))
  return {"U": torch.stack(U), "grad": torch.stack(grad), "variance": torch.stack(var)}


def exact(case, seed):
  """What :func:`run` gives, in float64.  None for the runs whose samples
  hang on accept and exchange decisions, and for whole runs of the networks
  (their chains carry the BF16 rounding of every step before)."""
  kind = case["kind"]
  if kind == "mlp_grad":
    return _mlp_exact(case, seed)
  if kind == "cnn_grad":
    return _cnn_exact(case, seed)
  if kind == "glm_grad":
    X, y = _glm_data(case, seed)
    U, grad, var = _glm_exact(case, X, y, _glm_start(case, seed, case["chains"]).double(),
                              _indices(case, seed).long())
    if case["chains"] == 1:
      return {"U": U[0], "grad": grad[0]}
    return {"U": U, "grad": grad, "variance": var}
  if kind in ("sgld", "obabo", "sghmc"):
    return _chain_exact(case, seed)
  return None
