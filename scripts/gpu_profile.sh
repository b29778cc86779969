#!/bin/bash
# Evidence for profiles/ from one GPU: a plain run first (its exit code gates the rest), then the ncu launch list of two decode
# steps (one metric, one pass).  Captures of more metrics replay every launch many times and save the device's memory around each
# pass: they belong on a small case of one kernel, not on these steps.
#   scripts/gpu_profile.sh [folder]
out=${1:-profile_out}
mkdir -p "$out"
timeout 300 python scripts/profile_decode.py --steps 2 > "$out/plain_decode.log" 2>&1 && tail -1 "$out/plain_decode.log" || exit 1
ncu --profile-from-start off --metrics gpu__time_duration.sum --clock-control none --csv --log-file "$out/launches_decode.csv" python scripts/profile_decode.py --steps 2 > "$out/ncu.log" 2>&1; echo "ncu exit $?"
