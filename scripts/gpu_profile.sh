#!/bin/bash
# Evidence for profiles/ from one GPU: plain runs first (their exit codes gate the rest), then the ncu launch list of two decode
# steps (one metric, one pass) and the CUPTI timelines (real overlap of dependent launches).  Captures of more metrics replay every
# launch many times and save the device's memory around each pass: they belong on a small case of one kernel, not on these steps.
#   scripts/gpu_profile.sh [folder]
out=${1:-profile_out}
mkdir -p "$out"
timeout 300 python scripts/timeline_prefill.py --sessions 4 --ctx 2048 --no-trace > "$out/plain_prefill.log" 2>&1 && tail -1 "$out/plain_prefill.log" || exit 1
timeout 300 python scripts/profile_decode.py --steps 2 > "$out/plain_decode.log" 2>&1 && tail -1 "$out/plain_decode.log" || exit 1
ncu --profile-from-start off --metrics gpu__time_duration.sum --clock-control none --csv --log-file "$out/launches_decode.csv" python scripts/profile_decode.py --steps 2 > "$out/ncu.log" 2>&1; echo "ncu exit $?"
timeout 300 python scripts/timeline_decode.py > "$out/timeline.txt" 2>&1; tail -12 "$out/timeline.txt"
timeout 300 python scripts/timeline_prefill.py --sessions 4 --ctx 2048 > "$out/timeline_prefill.txt" 2>&1; grep -v Warn "$out/timeline_prefill.txt" | tail -22
