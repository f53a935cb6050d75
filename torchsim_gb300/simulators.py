"""The reference's simulator API on the GB300 path.

``MRFSimulator`` / ``FSESimulator`` keep the reference's call shape
(``src/torchsim/model/_signal.py:158-240``): properties and protocol are
given together, ``simulate(**values)`` returns the signal with the voxel axes
of the properties, and ``jacobian(diff, **values)`` returns ``(signal,
jacobian)`` with the parameter axis stacked before the samples (collapsed for
a single name). Unlike the reference, whose Jacobian is k separate
``torch.func.jvp`` calls each paying a forward and a tangent pass
(``model/_signal.py:233-268``), every column here comes out of ONE fused
kernel pass together with the signal.

``mrf_sim`` / ``fse_sim`` are the functional wrappers
(``_functional/_mrf.py:12-85``, ``_functional/_fse.py:12-96``).
"""

from __future__ import annotations

import copy
from collections.abc import Sequence
from dataclasses import dataclass
from typing import Any

import numpy as np
import torch
from torch.autograd import forward_ad

from . import _native, engine
from .sequence import (POST_SHIFT, PRE_SHIFT, SHIFT_AFTER, MrfEvents, PackedEvents, fse_events,
                       mrf_events, mrf_gradient_map, mrf_stream_on_device, mrf_stream_with_gradients,
                       played_flip_torch, program_for)


def _tracked(value: Any) -> bool:
    """A tensor that autograd follows: one that requires grad (with grad
    mode on), or one carrying a forward-mode tangent (``torch.func.jvp``,
    ``torch.autograd.forward_ad`` dual tensors)."""
    if not isinstance(value, torch.Tensor):
        return False
    if value.requires_grad and torch.is_grad_enabled():
        return True
    if torch._C._functorch.is_functorch_wrapped_tensor(value):
        return True
    return forward_ad.unpack_dual(value).tangent is not None


def _reverse_only(value: torch.Tensor) -> bool:
    """A tracked tensor that carries no forward-mode tangent, outside any
    function transform."""
    return (not torch._C._are_functorch_transforms_active()
            and not torch._C._functorch.is_functorch_wrapped_tensor(value)
            and forward_ad.unpack_dual(value).tangent is None)


def _plain_float(value: torch.Tensor, n: int) -> bool:
    """A float32 vector of ``n`` (or one value) under reverse mode alone."""
    return (_reverse_only(value) and value.dtype == torch.float32 and value.ndim <= 1
            and value.numel() in (1, n))


def _primal(value: Any) -> Any:
    """A tensor's value without any function-transform wrapper around it
    (``torch.func.jvp`` wraps its inputs), for the host-side steps that read
    values: packing the event stream, the real-subspace verdict."""
    if not isinstance(value, torch.Tensor):
        return value
    while torch._C._functorch.is_functorch_wrapped_tensor(value):
        value = torch._C._functorch.get_unwrapped(value)
    return value.detach()


def _tensorish(value: Any) -> bool:
    return isinstance(value, (torch.Tensor, np.ndarray, list, tuple))


def _as_tensor(value: Any) -> torch.Tensor:
    if isinstance(value, torch.Tensor):
        return value
    return torch.as_tensor(np.asarray(value, dtype=np.float32))


def _batch(held: dict[str, Any]) -> tuple[int, ...]:
    shapes = [tuple(_as_tensor(v).shape) for v in held.values() if v is not None]
    return tuple(torch.broadcast_shapes(*shapes)) if shapes else ()


def _numel(shape: tuple[int, ...]) -> int:
    n = 1
    for s in shape:
        n *= s
    return n


def _home(values: dict[str, Any]) -> torch.device:
    """Where results go back to: the first tensor argument's device."""
    for v in values.values():
        if isinstance(v, torch.Tensor):
            return v.device
    return torch.device("cpu")


def _nonzero(value: Any) -> bool:
    if value is None:
        return False
    if isinstance(value, torch.Tensor):
        return bool(_primal(value).ne(0).any())
    return bool(np.any(np.asarray(value) != 0))


def _turns(held: dict[str, Any]) -> bool:
    """True when a voxel carries off-resonance or a transmit phase."""
    return _nonzero(held.get("B0")) or _nonzero(held.get("B1phase"))


def _leaves_real_subspace(events: PackedEvents, held: dict[str, Any]) -> bool:
    """True when the stream's pulses and samples do not share one phase, or a
    voxel carries off-resonance or a transmit phase: the complex kernel runs
    (the reference's real_axis verdict, sequence/_accelerators.py:1953-2128)."""
    return events.real_axis() != 1 or _turns(held)


class _EpgSimulator:
    """Shared mechanics: split properties from protocol, run, reshape."""

    properties: dict[str, str] = {}
    states = 10

    def __init__(self, **protocol: Any) -> None:
        self.protocol = dict(protocol)

    # -- what is held (model/_state_machine.py:560-640) --------------------
    @property
    def exposes(self) -> tuple[str, ...]:
        """The tissue properties this simulator takes."""
        return tuple(self.properties)

    accepts = exposes

    @property
    def bound(self) -> dict[str, Any]:
        """The tissue properties fixed on this simulator (a value or a map)."""
        return {k: v for k, v in self.protocol.items() if k in self.properties}

    def bind(self, **values: Any) -> _EpgSimulator:
        """This simulator with more fixed on it: properties (a measured B1
        map, a known T1), protocol arguments or settings (``states``)
        alike, held for every later call (``Simulator.bind``,
        ``model/_state_machine.py:576-594``). A copy; this one is unchanged."""
        held = copy.copy(self)
        held.protocol = {**self.protocol, **values}
        return held

    def to(self, device: torch.device | str) -> _EpgSimulator:
        """A copy with every tensor it holds on ``device``."""
        held = copy.copy(self)
        held.protocol = {k: (v.to(device) if isinstance(v, torch.Tensor) else v)
                         for k, v in self.protocol.items()}
        return held

    # -- to be provided by a sequence ------------------------------------
    def events(self, **protocol: Any) -> PackedEvents:  # pragma: no cover - abstract
        raise NotImplementedError

    def _device_stream(self, protocol: dict[str, Any], repetitions: int, device: torch.device):
        """``(program, flip events, duration events)`` built on the device
        from device-resident protocol values, or None where the stream is
        built on the host."""
        return None

    def _device_stream_with_gradients(self, protocol: dict[str, Any], repetitions: int,
                                      device: torch.device):
        """The same with the event buffers carrying gradients to the
        protocol's tensors, or None where :meth:`_event_gradients` attaches
        them."""
        return None

    def _kernel_maps(self, held: dict[str, Any]) -> dict[str, Any]:
        return {
            "T1": held.get("T1"),
            "T2": held.get("T2"),
            "M0": held.get("M0"),
            "B1": held.get("B1"),
            "inv": held.get("inv_efficiency"),
            "B0": held.get("B0"),
            "B1phase": held.get("B1phase"),
        }

    def _post(self, signal, jacobian, names, held, protocol, device):
        return signal, jacobian

    def _post_untracked(self, signal, jacobian, names, held, protocol, device):
        """:meth:`_post` of a call that nothing is differentiated through."""
        return self._post(signal, jacobian, names, held, protocol, device)

    # -- machinery ---------------------------------------------------------
    def _split(self, values: dict[str, Any]):
        merged = {**self.protocol, **values}
        held = {k: merged.pop(k) for k in list(merged) if k in self.properties}
        states = int(merged.pop("states", self.states))
        device = merged.pop("device", None)
        repetitions = int(merged.pop("repetitions", merged.pop("nreps", 1)))
        return held, merged, states, device, repetitions

    def _run(self, values: dict[str, Any], names: Sequence[str] | None):
        held, protocol, states, device, repetitions = self._split(values)
        for required in ("T1", "T2"):
            if required not in held:
                raise ValueError(f"{required} is required")
        home = _home(values)
        dev = engine.require_cuda(torch.device(device) if device is not None else
                                  (home if home.type == "cuda" else None))
        on_device = self._device_stream(protocol, repetitions, dev)
        events = (on_device[0].events if on_device is not None
                  else self.events(repetitions=repetitions, **protocol))
        # A derivative along B0 or B1phase leaves the real subspace too, as
        # the reference's verdict counts the tangents (_accelerators.py:3953-3966).
        # (A stream built on the device has one phase, zero.)
        complex_path = ((_turns(held) if on_device is not None
                         else _leaves_real_subspace(events, held))
                        or bool(names and {"B0", "B1phase"} & set(names)))
        if complex_path and on_device is not None:
            on_device = None
            events = self.events(repetitions=repetitions, **protocol)
        batch = _batch(held)
        voxels = _numel(batch)
        maps = self._kernel_maps(held)
        if names:
            for name in names:
                if name not in held:
                    raise ValueError(
                        f"{name!r} is not among the properties this call gave "
                        f"{type(self).__name__}: {sorted(held)}")
        # Identity-valued scalars are left out of the kernel, as the
        # reference's feature mask does.
        def declared(key, value):
            if value is None:
                return None
            if key in {"M0", "B1", "inv"} and not _tensorish(value) and float(value) == 1.0:
                return None
            return value

        with torch.cuda.device(dev):
            tissue = engine.tissue_maps(dev, voxels, maps["T1"], maps["T2"],
                                        declared("M0", maps["M0"]), declared("B1", maps["B1"]),
                                        declared("inv", maps["inv"]))
            kernel_names = self._kernel_names(names) if names else None
            if complex_path:
                off, keep = engine.offaxis_maps(dev, voxels, maps.get("B1phase"), maps.get("B0"))
                program = program_for(events, dev, phased=True)
                if kernel_names:
                    signal, jac = engine.forward_tangents_complex(program, tissue, states,
                                                                  kernel_names, off)
                else:
                    signal, jac = engine.forward_complex(program, tissue, states, off), None
                del keep
                signal, jac = self._post_untracked(signal, jac, names, held, protocol, dev)
                signal = signal.reshape(*batch, signal.shape[-1]) if batch else signal.reshape(-1)
                if jac is not None:
                    jac = (jac.reshape(*batch, *jac.shape[-2:]) if batch
                           else jac.reshape(jac.shape[-2:]))
                if home.type != "cuda":
                    signal = signal.to(home)
                    jac = None if jac is None else jac.to(home)
                return signal, jac
            program = on_device[0] if on_device is not None else program_for(events, dev)
            if (home.type != "cuda" and program.trains == 1
                    and type(self)._post is _EpgSimulator._post):
                # Host tensors in, host tensors out: sweep in chunks whose
                # copies back overlap the next chunk's sweep.
                signal, jac = engine.sweep_to_host(program, tissue, states, kernel_names or ())
                signal = signal.reshape(*batch, signal.shape[-1]) if batch else signal.reshape(-1)
                if jac is not None:
                    jac = (jac.reshape(*batch, *jac.shape[-2:]) if batch
                           else jac.reshape(jac.shape[-2:]))
                return signal, jac
            if kernel_names:
                signal, jac = engine.forward_tangents(program, tissue, states, kernel_names)
            else:
                signal, jac = engine.forward(program, tissue, states), None
            signal, jac = self._post_untracked(signal, jac, names, held, protocol, dev)
        signal = signal.reshape(*batch, signal.shape[-1]) if batch else signal.reshape(-1)
        if jac is not None:
            jac = jac.reshape(*batch, *jac.shape[-2:]) if batch else jac.reshape(jac.shape[-2:])
        if home.type != "cuda":
            signal = signal.to(home)
            jac = None if jac is None else jac.to(home)
        return signal, jac

    def _kernel_names(self, names: Sequence[str]) -> list[str]:
        return list(names)

    def simulate(self, **values: Any) -> torch.Tensor:
        """Return the recorded signal, ``(*voxels, samples)`` complex64.

        Differentiable: when a property or a sequence argument requires grad,
        the result carries a backward that runs the checkpointed adjoint
        kernel (``engine.EpgFunction``); when one carries a forward-mode
        tangent (``torch.func.jvp``, dual tensors), its tangent comes from one
        general tangent sweep."""
        if any(_tracked(v) for v in {**self.protocol, **values}.values()):
            return self._run_differentiable(values)
        signal, _ = self._run(values, None)
        return signal

    def _event_gradients(self, protocol, events, flip_ev, dur_ev, repetitions, phase_ev=None):
        """Attach the protocol's differentiable arguments to the event buffers
        (flip, duration, phase; ``(trains, events)``)."""
        if any(_tracked(v) for v in protocol.values()):
            raise NotImplementedError(
                f"{type(self).__name__}: gradients w.r.t. its sequence arguments are not built")
        return flip_ev, dur_ev, phase_ev

    def _run_differentiable(self, values: dict[str, Any], names: Sequence[str] | None = None):
        """The signal (or, with ``names``, the signal and Jacobian) on the
        autograd route: the first-order adjoint kernel behind the signal, the
        second-order sweep behind a Jacobian."""
        held, protocol, states, device, repetitions = self._split(values)
        home = _home(values)
        dev = engine.require_cuda(torch.device(device) if device is not None else
                                  (home if home.type == "cuda" else None))
        plain = {k: _primal(v) for k, v in protocol.items()}
        # The event stream and the verdict are values, built outside any
        # function transform (torch.func.jvp wraps every tensor made inside).
        # Reverse mode alone reaches flips and TRs through the stream's own
        # transpose; forward mode and function transforms attach them below.
        attached = None
        moved = [v for v in protocol.values() if _tracked(v)]
        if moved and all(_reverse_only(v) for v in moved):
            attached = self._device_stream_with_gradients(protocol, repetitions, dev)
        with torch._C._DisableFuncTorch():
            on_device = (attached if attached is not None
                         else self._device_stream(plain, repetitions, dev))
            events = (on_device[0].events if on_device is not None
                      else self.events(repetitions=repetitions, **plain))
            complex_path = (_turns(held) if on_device is not None
                            else _leaves_real_subspace(events, held))
            if complex_path and on_device is not None:
                attached = on_device = None
                events = self.events(repetitions=repetitions, **plain)
        if complex_path and names:
            raise NotImplementedError(
                "a differentiable Jacobian on the complex path (RF phases, B0, B1phase) is not "
                "built; its signal is differentiable")
        batch = _batch(held)
        voxels = _numel(batch)
        maps = self._kernel_maps(held)

        def flat(value, clamp=False, optional=True):
            if value is None:
                return None
            if optional and not _tensorish(value) and float(value) == 1.0:
                return None
            t = value if isinstance(value, torch.Tensor) else torch.as_tensor(
                np.asarray(value, np.float32))
            t = t.to(device=dev, dtype=torch.float32)
            t = t.expand(batch).reshape(-1) if batch else t.reshape(1)
            return t.clamp_min(engine.MINIMUM_RELAXATION_TIME_MS) if clamp else t

        if names:
            for name in names:
                if name not in held:
                    raise ValueError(
                        f"{name!r} is not among the properties this call gave "
                        f"{type(self).__name__}: {sorted(held)}")
        def turn(value):
            # Transmit phase and off-resonance: absent (or a scalar 0) stays
            # out of the kernel.
            if value is None or (not _tensorish(value) and float(value) == 0.0):
                return None
            return flat(value, optional=False)

        with torch.cuda.device(dev):
            with torch._C._DisableFuncTorch():
                if on_device is not None and not complex_path:
                    program, flip_ev, dur_ev = on_device
                    phase_ev = None
                else:
                    program = program_for(events, dev, phased=complex_path)
                    flip_ev = torch.from_numpy(events.flip).to(dev)
                    dur_ev = torch.from_numpy(events.duration).to(dev)
                    phase_ev = torch.from_numpy(np.array(
                        np.broadcast_to(events.phase, events.duration.shape), np.float32)).to(dev)
            if attached is None:
                flip_ev, dur_ev, phase_ev = self._event_gradients(protocol, events, flip_ev,
                                                                  dur_ev, repetitions, phase_ev)
            tissue = (flat(maps["T1"], True, False), flat(maps["T2"], True, False),
                      flat(maps["M0"]), flat(maps["B1"]), flat(maps["inv"]))
            jac = None
            if complex_path:
                signal = engine.EpgComplexFunction.apply(
                    program, states, None, *tissue, turn(maps.get("B1phase")),
                    turn(maps.get("B0")), flip_ev, dur_ev, phase_ev)[0]
            elif names:
                kernel = tuple(self._kernel_names(names))
                signal, jac = engine.JacobianFunction.apply(program, states, kernel, None, *tissue,
                                                            flip_ev, dur_ev)
            else:
                signal = engine.EpgFunction.apply(program, states, None, *tissue, flip_ev,
                                                  dur_ev)[0]
            signal, jac = self._post(signal, jac, names, held, plain, dev)
        signal = signal.reshape(*batch, signal.shape[-1]) if batch else signal.reshape(-1)
        if jac is not None:
            jac = jac.reshape(*batch, *jac.shape[-2:]) if batch else jac.reshape(jac.shape[-2:])
        if home.type != "cuda":
            signal = signal.to(home)
            jac = None if jac is None else jac.to(home)
        return signal if names is None else (signal, jac)

    def jacobian(self, diff: str | Sequence[str], **values: Any):
        """Return ``(signal, jacobian)``; the Jacobian is ``(*voxels, k, samples)``
        (``(*voxels, samples)`` for a single name given as a string)."""
        names = (diff,) if isinstance(diff, str) else tuple(diff)
        if any(_tracked(v) and not v.requires_grad
               for v in {**self.protocol, **values}.values()):
            raise NotImplementedError("forward-mode derivatives of a Jacobian are not built; "
                                      "its reverse mode is")
        if torch.is_grad_enabled() and any(
                isinstance(v, torch.Tensor) and v.requires_grad
                for v in {**self.protocol, **values}.values()):
            # Differentiable: a cost of the Jacobian (a Cramer-Rao bound)
            # backs through the second-order sweep.
            signal, jac = self._run_differentiable(values, names)
        else:
            signal, jac = self._run(values, names)
        if isinstance(diff, str):
            jac = jac[..., 0, :]
        return signal, jac


_gradient_maps: dict[tuple, dict[str, torch.Tensor]] = {}


def _gradient_map_on(pulses: int, repetitions: int, device: torch.device) -> dict[str, torch.Tensor]:
    """:func:`mrf_gradient_map` as device index tensors, uploaded once per
    (pulses, repetitions, device) so that a design step uploads nothing."""
    key = (pulses, repetitions, str(device))
    hit = _gradient_maps.get(key)
    if hit is None:
        hit = {k: torch.from_numpy(v).to(device)
               for k, v in mrf_gradient_map(pulses, repetitions).items()}
        _gradient_maps[key] = hit
    return hit


class MRFSimulator(_EpgSimulator):
    """Inversion-prepared unbalanced-SSFP MR fingerprinting
    (``simulators/mrf.py:17-84``): protocol ``flip`` (deg), ``TR`` (ms),
    ``TI`` (ms), ``phases`` (deg); properties T1, T2, M0, B1,
    inv_efficiency. The signal is ``1j * i*m0*F+[0]`` at every repetition of
    the last playing."""

    properties = {"T1": "t1_ms", "T2": "t2_ms", "M0": "m0", "B1": "b1",
                  "inv_efficiency": "inversion_efficiency", "B0": "b0_hz",
                  "B1phase": "b1_phase_rad"}
    states = 10

    def events(self, *, flip, TR, TI=0.0, phases=0.0, repetitions=1) -> PackedEvents:
        return mrf_events(flip, TR, TI_ms=TI, phases_deg=phases, repetitions=repetitions)

    def _device_stream(self, protocol, repetitions, device):
        """Flips or TRs resident on the device: the stream and its program
        are rebound there (:func:`mrf_stream_on_device`), so a design loop
        that moves them pays no host round trip and no compile per step. One
        playing, TI a number, zero phases and two pulses or more."""
        flip, tr = protocol.get("flip"), protocol.get("TR")
        if not any(isinstance(v, torch.Tensor) and v.device.type == "cuda" for v in (flip, tr)):
            return None
        if repetitions != 1 or set(protocol) - {"flip", "TR", "TI", "phases"}:
            return None
        ti, phases = protocol.get("TI", 0.0), protocol.get("phases", 0.0)
        if _tensorish(ti) or _tensorish(phases) or float(phases) != 0.0:
            return None
        if not isinstance(flip, torch.Tensor) or flip.numel() < 2:
            return None
        return mrf_stream_on_device(flip, tr, float(ti), device)

    def _device_stream_with_gradients(self, protocol, repetitions, device):
        flip, ti, phases = (protocol.get("flip"), protocol.get("TI", 0.0),
                            protocol.get("phases", 0.0))
        if (not isinstance(flip, torch.Tensor) or repetitions != 1
                or set(protocol) - {"flip", "TR", "TI", "phases"} or _tensorish(ti)
                or _tensorish(phases) or float(phases) != 0.0):
            return None
        return mrf_stream_with_gradients(flip, protocol.get("TR"), float(ti), device)

    def _event_gradients(self, protocol, events, flip_ev, dur_ev, repetitions, phase_ev=None):
        flip = protocol.get("flip")
        tr = protocol.get("TR")
        ti = protocol.get("TI", 0.0)
        n = int(torch.atleast_1d(torch.as_tensor(
            _primal(flip) if isinstance(flip, torch.Tensor) else np.asarray(flip))).numel())
        dev = flip_ev.device
        if _tracked(protocol.get("phases")):
            raise NotImplementedError("MRFSimulator: gradients w.r.t. phases are not built")
        moved = [v for v in (flip, tr) if _tracked(v)]
        if (moved and repetitions == 1 and not _tracked(ti) and flip_ev.shape == (1, 1 + 4 * n)
                and all(_plain_float(v, n) for v in moved)):
            # Reverse mode alone: one transpose instead of a chain of
            # elementwise operations. (The flips are read for their sign.)
            at = flip if _tracked(flip) else flip_ev.new_zeros(n)
            flip_ev, dur_ev, _ = MrfEvents.apply(at, tr if _tracked(tr) else None, flip_ev, dur_ev)
            return flip_ev, dur_ev, phase_ev
        with torch._C._DisableFuncTorch():
            where = _gradient_map_on(n, repetitions, dev)
        if _tracked(flip):
            played = played_flip_torch(torch.atleast_1d(flip).to(dev))
            delta = (played - played.detach()).expand(repetitions, n).reshape(-1)
            flip_ev = flip_ev.index_add(1, where["flip"].reshape(-1), delta[None])
        if _tracked(tr):
            spacing = torch.atleast_1d(tr).to(dev, torch.float32).expand(n) * 1e-3
            pairs = where["tr"]
            delta = (spacing - spacing.detach())[pairs[:, 1]]
            dur_ev = dur_ev.index_add(1, pairs[:, 0], delta[None])
        if _tracked(ti):
            t = ti.to(dev, torch.float32).reshape(()) * 1e-3
            idx = where["ti"]
            dur_ev = dur_ev.index_add(1, idx, (t - t.detach()).expand(idx.numel())[None])
        return flip_ev, dur_ev, phase_ev


class FSESimulator(_EpgSimulator):
    """CPMG fast spin echo (``simulators/fse.py:17-133``): protocol ``flip``
    (refocusing, deg), ``ESP`` (ms), ``phases`` (deg), ``exc_flip``,
    ``exc_phase`` (deg), ``TR`` (ms); properties T1, T2, M0, B1. M0 and the
    recovery over what is left of the TR are applied to the recorded echo
    train afterwards, as the reference's ``evaluate`` does
    (``fse.py:110-133``); the Jacobian carries them through by the chain
    rule."""

    properties = {"T1": "t1_ms", "T2": "t2_ms", "M0": None, "B1": "b1", "B0": "b0_hz",
                  "B1phase": "b1_phase_rad"}
    states = 10

    def events(self, *, flip, ESP, phases=0.0, exc_flip=90.0, exc_phase=90.0, TR=1e6,
               repetitions=1) -> PackedEvents:
        if repetitions != 1:
            raise ValueError("FSESimulator plays a single train")
        return fse_events(flip, ESP, phases_deg=phases, exc_flip=exc_flip, exc_phase=exc_phase)

    def _kernel_maps(self, held):
        maps = super()._kernel_maps(held)
        maps["M0"] = None  # applied after the kernel
        return maps

    def _event_gradients(self, protocol, events, flip_ev, dur_ev, repetitions, phase_ev=None):
        """Refocusing flips (deg) and phases (deg) onto the train's events:
        echo j's pulse is event 1 + 3j and its ADC 2 + 3j
        (:func:`torchsim_gb300.sequence.fse_events`), the ADC sharing the
        pulse's phase."""
        other = [k for k in protocol if k not in ("flip", "phases")]
        if any(_tracked(protocol[k]) for k in other):
            raise NotImplementedError("FSESimulator: gradients w.r.t. ESP, TR and the excitation "
                                      "are not built")
        dev = flip_ev.device
        flip = protocol.get("flip")
        n = (events.events - 1) // 3
        with torch._C._DisableFuncTorch():
            pulses = torch.from_numpy(1 + 3 * np.arange(n)).to(dev)
        if _tracked(flip):
            played = played_flip_torch(torch.atleast_1d(flip).to(dev))
            flip_ev = flip_ev.index_add(1, pulses, (played - played.detach())[None])
        phases = protocol.get("phases")
        if _tracked(phases) and phase_ev is not None:
            turn = torch.deg2rad(torch.atleast_1d(phases).to(dev, torch.float32)).expand(n)
            delta = (turn - turn.detach())[None]
            phase_ev = phase_ev.index_add(1, pulses, delta).index_add(1, pulses + 1, delta)
        return flip_ev, dur_ev, phase_ev

    def _kernel_names(self, names):
        kernel = [n for n in names if n in ("T1", "T2", "B1", "B0", "B1phase")]
        if "T1" not in kernel:
            kernel.append("T1")  # the recovery term depends on T1 too
        return kernel

    def _post(self, signal, jacobian, names, held, protocol, device):
        # The kernel's value is 1j * s_raw; the reference's FSE returns s_raw.
        s = signal * -1j
        echoes = s.shape[-1]
        esp = float(protocol["ESP"])
        tr = protocol.get("TR", 1e6)
        t1 = torch.as_tensor(held["T1"], dtype=torch.float32, device=device).reshape(-1)
        t1 = t1.expand(s.shape[0]) if t1.numel() == 1 else t1
        left_ms = torch.as_tensor(tr, dtype=torch.float32, device=device) - esp * echoes
        rec = torch.exp(-1e3 / t1 * left_ms * 1e-3)[:, None]
        m0v = held.get("M0", 1.0)
        m0 = torch.as_tensor(m0v, dtype=torch.float32, device=device).reshape(-1)
        m0 = (m0.expand(s.shape[0]) if m0.numel() == 1 else m0)[:, None]
        denom = 1 - rec * s
        out = m0 * s * (1 - rec) / denom
        if jacobian is None:
            return out, None
        kernel = self._kernel_names(names)
        dj = jacobian * -1j
        dfds = m0 * (1 - rec) / denom**2
        dfdrec = m0 * s * (s - 1) / denom**2
        drec_dt1 = rec * (left_ms * 1e-3 * 1e3) / (t1[:, None] ** 2)
        cols = []
        for name in names:
            if name == "M0":
                cols.append(s * (1 - rec) / denom)
                continue
            col = dfds * dj[:, kernel.index(name)]
            if name == "T1":
                col = col + dfdrec * drec_dt1
            cols.append(col)
        return out, torch.stack(cols, dim=-2)

    def _post_untracked(self, signal, jacobian, names, held, protocol, device):
        # One kernel for the plain forms (csrc/fse_recovery.cu), against some
        # forty launches of _post: one TR, a value of T1 and M0 for each
        # voxel or for all.
        tr, names = protocol.get("TR", 1e6), names or ()
        t1 = torch.as_tensor(held["T1"], dtype=torch.float32, device=device).reshape(-1)
        m0 = held.get("M0", 1.0)
        if isinstance(m0, torch.Tensor):
            m0 = m0.to(device=device, dtype=torch.float32).reshape(-1)
        rows = signal.shape[0]
        if (type(self)._post is not FSESimulator._post or not isinstance(tr, (int, float))
                or t1.numel() not in (1, rows) or len(names) > 16 or len(set(names)) < len(names)
                or not (isinstance(m0, (int, float))
                        or isinstance(m0, torch.Tensor) and m0.numel() in (1, rows))
                or not signal.is_contiguous()
                or jacobian is not None and not jacobian.is_contiguous()):
            return self._post(signal, jacobian, names, held, protocol, device)
        kernel = self._kernel_names(names) if names else []
        left_ms = float(np.float32(tr) - np.float32(float(protocol["ESP"]) * signal.shape[-1]))
        t1_column = names.index("T1") if "T1" in names else -1
        return engine.fse_recovery(signal, jacobian,
                                   [-1 if n == "M0" else kernel.index(n) for n in names], t1_column,
                                   _native.readable(t1),
                                   _native.readable(m0) if isinstance(m0, torch.Tensor)
                                   else float(m0), left_ms)


def mrf_sim(flip, TR, T1, T2, diff: str | tuple[str, ...] | None = None, B1=1.0,
            inv_efficiency=1.0, M0=1.0, TI: float = 0.0, states: int = 10, nreps: int = 1,
            device: str | torch.device | None = None):
    """SSFP MR fingerprinting (``_functional/_mrf.py:12-85``): the signal
    ``(..., len(flip))`` or ``(signal, jacobian (..., len(diff), len(flip)))``."""
    model = MRFSimulator()
    values = dict(T1=T1, T2=T2, M0=M0, B1=B1, inv_efficiency=inv_efficiency, flip=flip, TR=TR,
                  TI=TI, states=states, repetitions=nreps)
    if device is not None:
        values["device"] = device
    if diff is None:
        return model.simulate(**values)
    return model.jacobian(diff, **values)


def fse_sim(flip, ESP: float, T1, T2, phases=0.0, TR=1e6, exc_flip: float = 90.0,
            exc_phase: float = 90.0, diff: str | tuple[str, ...] | None = None, B1=1.0, M0=1.0,
            states: int = 10, device: str | torch.device | None = None):
    """Fast spin echo (``_functional/_fse.py:12-96``). The GB300 path is the
    real subspace, which CPMG reaches with ``phases`` equal to ``exc_phase``
    (90 deg by default for the excitation)."""
    model = FSESimulator()
    values = dict(T1=T1, T2=T2, M0=M0, B1=B1, flip=flip, ESP=ESP, phases=phases, TR=TR,
                  exc_flip=exc_flip, exc_phase=exc_phase, states=states)
    if device is not None:
        values["device"] = device
    if diff is None:
        return model.simulate(**values)
    return model.jacobian(diff, **values)



# ---- the direct route: a packed stream on the fused kernels ----------------


@dataclass
class SimulationResult:
    """What one :meth:`EpgEngine.simulate` recorded (``sequence/_simulation.py:
    239-264``): ``signal`` ``(*voxels, samples)`` complex64 and, per sample,
    ``time_us``, ``event_index`` (the recording event of the stream),
    ``repetition`` (the playing it belongs to) and ``echo`` (a spin echo)."""

    signal: torch.Tensor
    time_us: torch.Tensor
    event_index: torch.Tensor
    repetition: torch.Tensor
    echo: torch.Tensor


_WINDING = PRE_SHIFT | POST_SHIFT | SHIFT_AFTER
_RECORD_MODES = ("all", "acquired", "echo")


class EpgEngine:
    """Runs a packed event stream on the fused EPG kernels: the role of the
    reference's ``EpgEngine`` (``sequence/_simulation.py:267-484``) for a
    stream a builder (:func:`mrf_events`, :func:`fse_events`) produced.
    Tissue is a mapping of ``T1``, ``T2`` (required), ``M0``, ``B1``,
    ``inv_efficiency``, ``B0`` (Hz), ``B1phase`` (rad); shapes broadcast to the
    voxel batch. Streams that leave the real subspace run the complex
    kernel."""

    def shifts_per_repetition(self, events: PackedEvents) -> int:
        """How far one playing winds the states (gradient actions counted
        once per bit, ``_simulation.py:284-295``)."""
        per_playing = events.events // max(events.repetitions, 1)
        bits = events.action[:per_playing] & _WINDING
        return int(sum(bin(int(b)).count("1") for b in bits))

    def simulate(self, events: PackedEvents, tissue: dict[str, Any], *, repetitions: int = 1,
                 record: str = "all", nstates: int | None = None,
                 device: str | torch.device | None = None) -> SimulationResult:
        """Simulate ``events`` for ``tissue`` and record its samples.

        ``record``: ``"all"`` and ``"acquired"`` keep every sample the stream
        records; ``"echo"`` keeps the spin echoes. ``nstates`` defaults to
        ``max(8, min(64, 1 + winding))`` over the stream's playings. A packed
        stream already carries its playings, so ``repetitions`` must be 1 (a
        builder takes ``repetitions=k``)."""
        if int(repetitions) != 1:
            raise ValueError("a packed stream carries its playings: build it with repetitions=k")
        if record not in _RECORD_MODES:
            raise ValueError("record must be 'all', 'acquired', or 'echo'")
        for required in ("T1", "T2"):
            if required not in tissue:
                raise ValueError(f"{required} is required")
        if nstates is None:
            winding = events.repetitions * self.shifts_per_repetition(events)
            nstates = max(8, min(64, 1 + winding))
        nstates = int(nstates)
        if nstates < 1:
            raise ValueError("nstates must be positive")
        held = {k: tissue.get(k) for k in ("T1", "T2", "M0", "B1", "inv_efficiency", "B0",
                                           "B1phase")}
        held = {k: v for k, v in held.items() if v is not None}
        complex_path = _leaves_real_subspace(events, held)
        home = _home(held)
        dev = engine.require_cuda(torch.device(device) if device is not None else
                                  (home if home.type == "cuda" else None))
        batch = _batch(held)
        voxels = _numel(batch)

        def declared(key):
            value = held.get(key)
            if value is None or (not _tensorish(value) and float(value) == 1.0):
                return None
            return value

        with torch.cuda.device(dev):
            maps = engine.tissue_maps(dev, voxels, held["T1"], held["T2"], declared("M0"),
                                      declared("B1"), declared("inv_efficiency"))
            if complex_path:
                off, keep = engine.offaxis_maps(dev, voxels, held.get("B1phase"), held.get("B0"))
                signal = engine.forward_complex(program_for(events, dev, phased=True), maps,
                                                nstates, off)
                del keep
            else:
                signal = engine.forward(program_for(events, dev), maps, nstates)
        signal = signal.reshape(*batch, signal.shape[-1]) if batch else signal.reshape(-1)
        outputs = events.outputs
        echo = events.echo if events.echo is not None else np.zeros(outputs, bool)
        keep = np.arange(outputs) if record != "echo" else np.flatnonzero(echo[:outputs])
        labels = dict(
            time_us=torch.from_numpy(events.time_us[keep].astype(np.float32)),
            event_index=torch.from_numpy(events.sample_events()[keep]),
            repetition=torch.full((keep.size,), events.repetitions - 1, dtype=torch.int64),
            echo=torch.from_numpy(echo[keep].copy()),
        )
        if record == "echo":
            signal = signal[..., torch.from_numpy(keep).to(signal.device)]
        if home.type != "cuda":
            signal = signal.to(home)
        return SimulationResult(signal=signal, **{k: v.to(signal.device) for k, v in labels.items()})
